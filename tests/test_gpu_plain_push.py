"""The FP64 push's transverse maps at the edge of their series (|z| = |k1| (dz/2)^2 either
side of 2^-12), focusing and defocusing, and over the block sizes of small and large
windows, against the oracle.

Tolerance: a half step takes about ten roundings (1.1e-16) and its series omits less than
2^-63: coordinates within 4e-15 of the largest after one step of two half steps (the
calls' last-bit differences included)."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0 = 1e-10, 11357.8


@pytest.mark.parametrize("ns,npart", [(1, 64), (3, 100), (40, 2052)])
@pytest.mark.parametrize("k1", [0.0, 1e-6, 1.08, 1.09, 1.5, 40.0])
@pytest.mark.parametrize("helical", [False, True])
def test_plain_push_transverse_matches_oracle(lib, oracle, ns, npart, k1, helical):
    import g4gpu
    lat = T.undulator_lattice(1.7, 0.03, 1, 1, LAMBDA0, GAMMA0, helical=helical)
    lat[:, T.C["qf"]] = k1
    rng = np.random.default_rng(npart)
    part = np.empty((ns, npart, 6))
    part[..., 0] = GAMMA0 + rng.normal(0, 2, (ns, npart))
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    part[..., 4:6] = rng.normal(0, 0.05, (ns, npart, 2))
    cur = np.full(ns, 1000.0)
    ng, gm = 25, 1e-4
    fld = np.zeros((1, ns, ng * ng), dtype=np.complex128)
    ref = oracle.run_steps(lat, GAMMA0, part, cur, LAMBDA0, 1.0, [1], [gm], fld, [0], time_run=0)[0]
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=ng, gridmax=gm, lambda0=LAMBDA0, sample=1.0, gammaref=GAMMA0,
                       precision=g4gpu.PLAIN, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, fld[0])
        h.run(0, 1)
        got = h.get_beam()
    for k in (2, 3, 4, 5):
        assert np.max(np.abs(got[..., k] - ref[..., k])) <= 4e-15 * np.max(np.abs(ref[..., k]))
    assert np.max(np.abs(got[..., 1] - ref[..., 1])) <= 1e-9 * np.max(np.abs(ref[..., 1]))
