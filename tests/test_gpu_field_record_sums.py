"""run_diag's field record of the mixed form, formed inside the field step where the slice is on
chip, and the record formed after a step, against FP64 sums of the field that the run leaves.

Tolerance: the sums are compensated, so what is left is the rounding of their FP32 terms (|u|^2
and its products with the coordinates, at most 1.5 units of 2^-24), random and averaged over the
cells that carry the field: (sum w)^2 / sum w^2 = pi (waist / dgrid)^2, over 700 here, so 9e-8 /
sqrt(700) = 3.4e-9 rms; 4.5 times that, the worst of a few hundred slices. Centroids are
compared in units of the size. The far field adds exact terms: the same bound holds."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GM, W0 = 1e-10, 11357.8, 1e-4, 30e-6


@pytest.mark.parametrize("ns,ngrid,nharm", [(200, 101, 1), (200, 151, 3), (3, 151, 1), (160, 201, 1), (20, 255, 3),
                                            (40, 128, 2)])
def test_field_record_of_a_run_is_that_of_its_field(lib, ns, ngrid, nharm):
    import g4gpu
    steps, npart = 2, 64
    rng = np.random.default_rng(ngrid)
    lat = T.undulator_lattice(1.7, 0.015, steps, 1, LAMBDA0, GAMMA0)
    lat[:, T.C["aw"]] = 0.0  # no source: the field stays the mode
    part = g4gpu.host_load_beam(T.slice_params(ns, GAMMA0, 1.0, 0.4e-6, 15.0), 0, npart, 4, 5, 1, LAMBDA0, 1.0)
    x = np.linspace(-GM, GM, ngrid)
    mode = np.exp(-(x[None] ** 2 + x[:, None] ** 2) / W0 ** 2) * np.exp(2e4j * x)[None]
    fld = mode[None] * np.exp(1j * rng.uniform(0, 6.28, ns))[:, None, None]
    with g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, gridmax=GM, lambda0=LAMBDA0, sample=1.0,
                                   gammaref=GAMMA0, precision=g4gpu.MIXED, time_run=0)) as h:
        h.set_lattice(lat)
        h.load_beam(part, np.full(ns, 3000.0))
        h.load_field(0, np.ascontiguousarray(fld.reshape(ns, -1)))
        _, fd = h.run_diag(0, steps, nharm=nharm)
        _, f2 = h.diag(nharm)
        u = h.get_field(0)[0].reshape(ns, ngrid, ngrid)
    w = np.abs(u) ** 2
    k = np.arange(ngrid) - 0.5 * (ngrid - 1)
    dg, ks = 2 * GM / (ngrid - 1), 2 * np.pi / LAMBDA0
    p = w.sum((1, 2))
    mx, my = (w * k).sum((1, 2)) / p, (w * k[:, None]).sum((1, 2)) / p
    sx = np.sqrt((w * k * k).sum((1, 2)) / p - mx * mx)
    sy = np.sqrt((w * (k * k)[:, None]).sum((1, 2)) / p - my * my)
    far = np.abs(u.sum((1, 2)))
    tol = 4.5 * 9e-8 / np.sqrt(np.pi) / (W0 / dg)
    for rec in (fd[-1, 0], f2[0]):
        assert np.max(np.abs(rec[:, 0] / ((dg * 510998.95069 / ks) ** 2 / 376.73) / p - 1)) <= tol
        assert np.max(np.abs(rec[:, 1] / dg - mx) / sx) <= tol
        assert np.max(np.abs(rec[:, 2] / dg / sx - 1)) <= tol
        assert np.max(np.abs(rec[:, 3] / dg - my) / sy) <= tol
        assert np.max(np.abs(rec[:, 4] / dg / sy - 1)) <= tol
        assert np.max(np.abs(np.sqrt(rec[:, 7]) / dg / far - 1)) <= tol
