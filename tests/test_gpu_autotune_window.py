"""g4gpu_autotune against the automatic shapes: tuning a window does not slow it down, whatever
was tuned before it. Step times are compared as the best of several runs, the tuned and the
untuned handle in turn; 8 % is allowed, several times what such minima differ by."""
import time

import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0 = 1e-10, 11357.8


def window(precision, ns, npart, ngrid, steps):
    import g4gpu
    h = g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, gridmax=1e-4, lambda0=LAMBDA0, sample=1.0,
                                  gammaref=GAMMA0, precision=precision, time_run=0))
    rng = np.random.default_rng(ns)
    part = np.zeros((ns, npart, 6))
    part[..., 0] = GAMMA0
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    h.set_lattice(T.undulator_lattice(1.7, 0.015, steps, 1, LAMBDA0, GAMMA0))
    h.load_beam(part, np.full(ns, 1000.0))
    h.load_field(0, np.ones((ns, ngrid * ngrid), dtype=complex))
    return h


@pytest.mark.parametrize("precision,windows", [(1, [(4, 1024, 151), (300, 1024, 151)]), (1, [(4, 512, 117), (400, 512, 117)]),
                                               (0, [(1, 8192, 65)])])
def test_tuning_a_window_does_not_slow_it_down(lib, precision, windows):
    steps = 30
    for ns, npart, ngrid in windows:
        with window(precision, ns, npart, ngrid, steps) as plain, window(precision, ns, npart, ngrid, steps) as tuned:
            tuned.autotune()
            best = {}
            for _ in range(9):
                for name, h in (("plain", plain), ("tuned", tuned)):
                    h.synchronize()
                    t = time.perf_counter()
                    h.run(0, steps)
                    h.synchronize()
                    best[name] = min(best.get(name, 1e9), time.perf_counter() - t)
        assert best["tuned"] <= 1.08 * best["plain"], (ns, npart, ngrid, best)
