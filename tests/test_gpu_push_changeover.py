"""The FP64 push around the energy where 1 / btpar0 changes from the integer series to the
corrected one (1 - btpar0^2 = 2^-22: gamma near 4040 at aw 1.7), against the oracle: energies on
both sides in one window, and particles whose field carries them across.

Tolerance: as for the push's phase elsewhere, theta advances by about 80 rad a step with a
rounding of xks (1 - 1/btpar0) that both sides share unless the field's last bits move it over a
boundary: 99 % of the particles within 1e-10 of the largest |theta|, all within 1e-6."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0 = 1e-10, 4040.0


@pytest.mark.parametrize("spread", [1e-9, 1e-5, 1e-2])
def test_push_on_both_sides_of_the_changeover(lib, oracle, spread):
    import g4gpu
    ns, npart, ng, gm, nstep = 2, 512, 33, 1e-4, 3
    lat = T.undulator_lattice(1.7, 0.015, nstep, 1, LAMBDA0, GAMMA0)
    rng = np.random.default_rng(7)
    part = np.zeros((ns, npart, 6))
    edge = np.sqrt((1 + 1.7 ** 2) * 2.0 ** 22)
    part[..., 0] = edge * (1 + spread * rng.uniform(-1, 1, (ns, npart)))
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2e-6, (ns, npart, 2))
    cur = np.full(ns, 1000.0)
    fld = np.stack([g4gpu.host_gauss_hermite(T.gauss_field_par(LAMBDA0, 1e6, 3e-5), gm, ng)] * ns)
    ref = oracle.run_steps(lat, GAMMA0, part, cur, LAMBDA0, 1.0, [1], [gm], fld[None], [0], time_run=0)[0]
    with g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=ng, gridmax=gm, lambda0=LAMBDA0, sample=1.0,
                                   gammaref=GAMMA0, precision=g4gpu.PLAIN, time_run=0)) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, fld)
        h.run(0, nstep)
        got = h.get_beam()
    for k in (0, 1):
        d = np.abs(got[..., k] - ref[..., k]) / np.max(np.abs(ref[..., k]))
        assert np.max(d) <= 1e-6
        assert np.mean(d <= 1e-10) >= 0.99
