"""The mixed beam record against numpy on the stored state: slices that start off a 16-byte
boundary, fewer particles than a group or than the copies run ahead, remainders, one4one
slices down to none, one to sixteen harmonics.

Tolerance (u = 2^-24): compensated FP32 sums are good to 2 u of the sum of the magnitudes,
products add u: 3 u, and 4 u with what follows. A bunching factor's terms carry the fast
sine's 2^-21.2, the phase's conversion and scaling pi u each: under 1e-6, absolute."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GM = 1e-10, 11357.8, 1e-4
U4 = 4 * 2.0 ** -24


@pytest.mark.parametrize("ns,npart,nharm", [
    (1, 1, 1), (5, 3, 1), (7, 6, 2), (3, 127, 1), (3, 510, 3), (5, 513, 5), (2, 1537, 1), (3, 4101, 16), (2, 8192, 1)])
@pytest.mark.parametrize("counts", [False, True])
def test_mixed_beam_record_matches_numpy(lib, ns, npart, nharm, counts):
    import g4gpu
    rng = np.random.default_rng(ns + npart)
    part = np.empty((ns, npart, 6))
    part[..., 0] = GAMMA0 + rng.normal(0, 2, (ns, npart))
    part[..., 1] = rng.uniform(-40, 40, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    part[..., 4:6] = rng.normal(0, 0.02, (ns, npart, 2))
    cnt = rng.integers(0, npart + 1, ns).astype(np.int32) if counts else np.full(ns, npart, np.int32)
    if counts:
        cnt[-1] = 0
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=25, harm=[1], gridmax=GM, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.MIXED, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(T.undulator_lattice(1.7, 0.015, 4, 1, LAMBDA0, GAMMA0))
        if counts:
            h.load_beam_counts(part, np.full(ns, 1e3), cnt)
        else:
            h.load_beam(part, np.full(ns, 1e3))
        h.load_field(0, np.zeros((ns, 625), complex))
        bd, _ = h.diag(nharm)
        p = h.get_beam()
    for s in range(ns):
        q = p[s, :cnt[s]]
        if len(q) == 0:
            assert bd[s, 0] == 0 and bd[s, 24] == 0
            continue
        assert abs(bd[s, 0] - q[:, 0].mean()) <= U4 * np.abs(q[:, 0] - GAMMA0).mean() + 1e-11
        for c, k in ((2, 2), (4, 3), (6, 4), (7, 5)):
            assert abs(bd[s, c] - q[:, k].mean()) <= U4 * np.abs(q[:, k]).mean()
        for c, k in ((3, 2), (5, 3)):  # <v^2> = size^2 + mean^2
            assert abs(bd[s, c] ** 2 + bd[s, c - 1] ** 2 - (q[:, k] ** 2).mean()) <= U4 * (q[:, k] ** 2).mean()
        ext = [f(q[:, k]) for k in (2, 4, 3, 5, 0) for f in (np.min, np.max)]
        assert np.array_equal(bd[s, 14:24], ext)
        for m in range(1, nharm + 1):
            z = np.exp(1j * m * q[:, 1]).mean()
            got = bd[s, 24 + 2 * (m - 1)] * np.exp(1j * bd[s, 25 + 2 * (m - 1)])
            assert abs(got - z) <= 1e-6 + m * 1e-8  # m times the stored phase's 2^-32 turn
