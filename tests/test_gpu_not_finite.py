"""A value that is not finite in an FP64 field: the reference's sweeps carry it through every
line they cross, so that one step leaves its whole slice without a finite value, and the other
slices as they were. Over the shapes of the segmented solves (lines of 2, 4, 8 and 16) and one
thread per line."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GRIDMAX = 1e-10, 11357.8, 1e-4
XKS = 2 * np.pi / LAMBDA0


@pytest.mark.parametrize("ns,ngrid,r", [(2, 255, 0.03), (25, 101, 0.03), (70, 61, 0.03), (160, 33, 0.03), (90, 79, 0.4),
                                        (2, 60, 4.0)])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_a_value_that_is_not_finite_runs_through_its_slice(lib, ns, ngrid, r, value):
    import g4gpu
    rng = np.random.default_rng(ngrid)
    dgrid = 2 * GRIDMAX / (ngrid - 1)
    lat = T.undulator_lattice(1.7, r * 4 * XKS * dgrid * dgrid, 1, 1, LAMBDA0, GAMMA0)
    lat[:, T.C["aw"]] = 0.0
    part = np.zeros((ns, 32, 6))
    part[..., 0] = GAMMA0
    field = rng.normal(size=(ns, ngrid * ngrid)) + 1j * rng.normal(size=(ns, ngrid * ngrid))

    def step(f):
        with g4gpu.Handle(g4gpu.Config(nslice=ns, npart=32, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                                       gammaref=GAMMA0, precision=0, time_run=0)) as h:
            h.set_lattice(lat)
            h.load_beam(part, np.ones(ns))
            h.load_field(0, f)
            h.run(0, 1, g4gpu.STAGE_FIELD)
            return h.get_field(0)[0].copy()

    clean = step(field)
    hit = field.copy()
    hit[1, (ngrid // 3) * ngrid + ngrid // 2] = value
    got = step(hit)
    others = np.arange(ns) != 1
    assert np.array_equal(got[others], clean[others])
    assert not np.any(np.isfinite(got[1]))
