"""The FP64 diagnostic kernel against numpy over its shapes: one or several CTAs a slice and
a grid, remainders of particles and rows, odd and even grids up to two columns a thread, one
to sixteen harmonics, phases from the push's phasors and (after a load) from theta, one4one
slices without particles.

Tolerance: sums of n terms are compared relative to the sum of the terms' magnitudes, whose
rounding is at most (n + 40) 1.1e-16 of it; bunching factors are compared absolutely, 1e-12
(a phase of 1e3 rad carries 1e-13)."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GM = 1e-10, 11357.8, 1e-4


@pytest.mark.parametrize("ns,npart,ng,harm,nharm,steps", [
    (1, 8192, 255, [1], 1, 2), (1, 100, 25, [1], 3, 0), (1, 4100, 128, [1, 3], 3, 1), (3, 2052, 101, [3, 1], 16, 1),
    (40, 516, 57, [1], 2, 1), (330, 1028, 33, [1], 1, 1), (2, 1024, 301, [1], 1, 0), (2, 1000, 45, [3], 4, 1)])
@pytest.mark.parametrize("counts", [False, True])
def test_plain_diag_matches_numpy(lib, ns, npart, ng, harm, nharm, steps, counts):
    import g4gpu
    rng = np.random.default_rng(ns + npart + ng)
    lat = T.undulator_lattice(1.7, 0.015, 4, 1, LAMBDA0, GAMMA0)
    part = np.empty((ns, npart, 6))
    part[..., 0] = GAMMA0 + rng.normal(0, 2, (ns, npart))
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    part[..., 4:6] = rng.normal(0, 0.02, (ns, npart, 2))
    cur = rng.uniform(500, 3000, ns)
    cnt = rng.integers(0, npart + 1, ns).astype(np.int32) if counts else np.full(ns, npart, np.int32)
    if counts:
        cnt[-1] = 0
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=ng, harm=harm, gridmax=GM, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.PLAIN, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        if counts:
            h.load_beam_counts(part, cur, cnt)
        else:
            h.load_beam(part, cur)
        for k in range(len(harm)):
            h.load_field(k, rng.normal(size=(ns, ng * ng)) + 1j * rng.normal(size=(ns, ng * ng)), first=ns - 1)
        h.run(0, steps)
        for _ in range(2):  # the tickets are left as they were found
            bd, fd = h.diag(nharm)
        p = h.get_beam()
        fields = [h.get_field(k)[0] for k in range(len(harm))]
    for s in range(ns):
        q = p[s, :cnt[s]]
        if len(q) == 0:
            assert bd[s, 0] == 0 and bd[s, 24] == 0
            continue
        eps = (len(q) + 40) * 1.1e-16
        for c, k in ((0, 0), (2, 2), (4, 3), (6, 4), (7, 5)):
            assert abs(bd[s, c] - q[:, k].mean()) <= eps * np.abs(q[:, k]).mean()
        for c, k in ((3, 2), (5, 3)):  # <v^2> = size^2 + mean^2
            assert abs(bd[s, c] ** 2 + bd[s, c - 1] ** 2 - (q[:, k] ** 2).mean()) <= 2 * eps * (q[:, k] ** 2).mean()
        ext = [f(q[:, k]) for k in (2, 4, 3, 5, 0) for f in (np.min, np.max)]
        assert np.array_equal(bd[s, 14:24], ext)
        for m in range(1, nharm + 1):
            z = np.exp(1j * m * q[:, 1]).mean()
            got = bd[s, 24 + 2 * (m - 1)] * np.exp(1j * bd[s, 25 + 2 * (m - 1)])
            assert abs(got - z) <= m * 1e-12
    grid = np.arange(ng) - 0.5 * (ng - 1)
    dg = 2 * GM / (ng - 1)
    for k, f in enumerate(fields):
        w = np.abs(f.reshape(ns, ng, ng)) ** 2
        ks = 2 * np.pi / (LAMBDA0 / harm[k])
        eps = (ng * ng + 40) * 1.1e-16
        w = np.roll(w, 1, axis=0) if ns > 1 else w  # window slice is in storage slot (is + first) % ns
        u = np.roll(f, 1, axis=0) if ns > 1 else f
        pw = w.sum((1, 2))
        assert np.all(np.abs(fd[k][:, 0] / (dg * 510998.95069 / ks) ** 2 * 376.73 - pw) <= 2 * eps * pw)
        assert np.all(np.abs(fd[k][:, 1] / dg - (w * grid).sum((1, 2)) / pw) <= 2 * eps * ng)
        assert np.all(np.abs(fd[k][:, 3] / dg - (w * grid[:, None]).sum((1, 2)) / pw) <= 2 * eps * ng)
        ff = u.sum(1)
        assert np.all(np.abs(np.sqrt(fd[k][:, 7]) / dg - np.abs(ff)) <= 2 * eps * np.abs(u).sum(1))
        mid = np.abs(u[:, (ng // 2) * ng + ng // 2]) ** 2 * (510998.95069 / ks) ** 2 / 376.73
        assert np.allclose(fd[k][:, 5], mid, rtol=1e-14)
