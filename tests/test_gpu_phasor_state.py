"""The FP64 push starts each step from the phasors the previous push left. A state copied
into a handle that already ran steps, or phases moved by a closure's correction, must not
meet phasors of other phases: the steps that follow give what a fresh handle gives (up to
the summation order of the deposition's atomics; stale phasors are off by order one)."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu

NS, NPART, NG, GM, LAMBDA0, GAMMA0 = 4, 512, 45, 1e-4, 1e-10, 11357.8


def window(g4gpu, beam):
    cfg = g4gpu.Config(nslice=NS, npart=NPART, ngrid=NG, gridmax=GM, lambda0=LAMBDA0, sample=1.0, gammaref=GAMMA0,
                       precision=g4gpu.PLAIN, time_run=1)
    h = g4gpu.Handle(cfg)
    h.set_lattice(T.undulator_lattice(1.7, 0.015, 6, 1, LAMBDA0, GAMMA0))
    h.load_beam(beam, np.full(NS, 3000.0))
    h.load_field(0, np.zeros((NS, NG * NG), dtype=np.complex128))
    return h


def beams(g4gpu):
    sp = T.slice_params(NS, GAMMA0, 1.0, 0.4e-6, 15.0)
    return [g4gpu.host_load_beam(sp, 0, NPART, 4, seed, 1, LAMBDA0, 1.0) for seed in (5, 9)]


def test_copied_state_restarts_the_phasors(lib):
    import g4gpu
    a, b = beams(g4gpu)
    with window(g4gpu, a) as h, window(g4gpu, b) as h0, window(g4gpu, b) as ref:
        h.run(0, 3)
        h.copy_state_from(h0)
        h.run(0, 6)
        ref.run(0, 6)
        assert np.allclose(h.get_beam(), ref.get_beam(), rtol=1e-9, atol=1e-12)


def test_closure_correction_restarts_the_phasors(lib):
    import g4gpu
    a, _ = beams(g4gpu)
    corr = np.zeros((NS, 4), dtype=np.float32)
    corr[:, 0] = [0.5, -0.25, 1.0, 2.0]
    with window(g4gpu, a) as h:
        mlp = g4gpu.MLP(seed=1)
        h.closure_attach(mlp, 30e-6)
        h.run(0, 3)
        h.closure_apply(corr)
        moved, (fld, first, acc) = h.get_beam(), h.get_field(0)
        h.run(3, 3)
        got = h.get_beam()
    with window(g4gpu, moved) as ref:
        ref.load_field(0, fld, first=first, accuslip=acc)
        ref.run(3, 3)
        assert np.allclose(got, ref.get_beam(), rtol=1e-9, atol=1e-12)
