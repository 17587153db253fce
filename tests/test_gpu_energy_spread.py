"""The energy and its spread in the beam record, of slices far above their own spread in gamma:
the sums are taken about gammaref, where sum g^2 - n <g>^2 would lose 2 gamma^2 / spread^2
(6e7) roundings.

Tolerance. FP64: differences from gammaref are exact, the sums of n squares carry at most
n / 8 + 40 roundings of 2^-53, the spread half of them; the mean is within two roundings of
gamma. Mixed: gamma is held as an FP32 difference (2^-24 of it), its square rounds once more:
3 2^-24 a term at most, random, over sqrt(n) of them five times that for the worst slice."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0 = 1e-10, 11357.8


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ns,npart,counts", [(1, 8192, False), (40, 1024, False), (7, 516, True)])
def test_energy_spread_keeps_its_digits(lib, precision, ns, npart, counts):
    import g4gpu
    rng = np.random.default_rng(ns + npart)
    part = np.zeros((ns, npart, 6))
    part[..., 0] = GAMMA0 + rng.normal(0, 2, (ns, npart))
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    part[..., 4:6] = rng.normal(0, 0.02, (ns, npart, 2))
    cnt = rng.integers(npart // 2, npart + 1, ns).astype(np.int32) if counts else np.full(ns, npart, np.int32)
    lat = T.undulator_lattice(1.7, 0.015, 2, 1, LAMBDA0, GAMMA0)
    with g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=41, gridmax=1e-4, lambda0=LAMBDA0, sample=1.0,
                                   gammaref=GAMMA0, precision=precision, time_run=0)) as h:
        h.set_lattice(lat)
        if counts:
            h.load_beam_counts(part, np.ones(ns), cnt)
        else:
            h.load_beam(part, np.ones(ns))
        h.load_field(0, np.zeros((ns, 41 * 41), dtype=complex))
        bd, _ = h.run_diag(0, 1, nharm=1)
        b2, _ = h.diag(1)
        got = h.get_beam()
    eps = 2.0 ** -53
    for rec in (bd[0], b2):
        for s in range(ns):
            g = got[s, :cnt[s], 0].astype(np.longdouble)
            spread = float(np.sqrt(np.mean((g - g.mean()) ** 2)))
            tol = (npart / 16 + 20) * eps if precision == 0 else 5 * 3 * 2.0 ** -24 / np.sqrt(npart // 2)
            assert abs(rec[s, 1] / spread - 1) <= tol
            assert abs(rec[s, 0] - float(g.mean())) <= 2 * eps * GAMMA0 + (0 if precision == 0 else tol * spread)
