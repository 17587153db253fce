"""The tiled field step of the mixed form on grids of more columns than a CTA has threads
(256), against the oracle, with segmented solves and (large step factors) whole lines. Inputs
and tolerance are those of test_gpu_mixed_field."""
import numpy as np
import pytest

from test_gpu_mixed_field import GAMMA0, GRIDMAX, LAMBDA0, XKS, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,npart,ngrid,r", [(2, 32, 256, 2.0), (1, 32, 257, 2.0), (2, 30, 401, 2.0), (1, 32, 520, 0.03),
                                              (2, 32, 513, 0.1)])
def test_tiled_field_step_matches_oracle(lib, oracle, ns, npart, ngrid, r):
    import g4gpu
    lat, part, cur, _, src, field, dz, dgrid = setup(oracle, ns, npart, ngrid, r, True, False)
    ref = oracle.adi_advance(field, src, ns - 1, dz, dgrid, XKS)
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.MIXED, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, field, first=ns - 1)
        h.run(0, 1, g4gpu.STAGE_FIELD)
        got = h.get_field(0)[0]
    tol = 1.2e-5 * (1 + 4 * r) * np.max(np.abs(ref)) + (4 * ngrid * 6e-8 + 6e-6) * 2 * np.max(np.abs(src))
    assert np.max(np.abs(got - ref)) <= tol
