"""The FFT solver on even grids, whose tiles in shared memory have gaps: first radices 4, 8
and 16 (and 2, without), two to four stages, both precisions; the far-field moments. A drift
step against numpy, the moments against the oracle.

Tolerance (of the largest value): two 2-D transforms of up to four stages of up to 17 terms a
dimension and a propagator: under 300 roundings, 300 x 1.1e-16 = 3.3e-14 in FP64 (1e-13 taken)
and 300 x 6e-8 = 1.8e-5 in FP32 if all agreed (the phase's 2e-7 and the fast sine's 4e-7 lie
below)."""
import numpy as np
import pytest

import g4cases as T
from test_oracle_pins import _k2_and_sigmoid

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GM = 1e-10, 11357.8, 6e-5
SIZES = [18, 20, 24, 32, 48, 64, 96, 100, 128, 144, 150, 200, 240, 250, 256]


def run(n, precision, u, diag=False):
    import g4gpu
    ns = len(u)
    lat = T.undulator_lattice(1.7, 0.015, 1, 1, LAMBDA0, GAMMA0)
    lat[0, T.C["aw"]] = 0.0
    part = g4gpu.host_load_beam(T.slice_params(ns, GAMMA0, 2.0, 0.4e-6, 15.0), 0, 32, 4, 1, 0, LAMBDA0, 1.0)
    cfg = g4gpu.Config(nslice=ns, npart=32, ngrid=n, harm=[1], gridmax=[GM], lambda0=LAMBDA0, sample=1.0, gammaref=GAMMA0,
                       precision=precision, solver=g4gpu.SOLVER_FFT, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, np.full(ns, 3000.0))
        h.load_field(0, u)
        if diag:
            return h.diag_fft()
        h.run(0, 1, g4gpu.STAGE_FIELD)
        return h.get_field(0)[0]


def random_field(n, ns=3):
    rng = np.random.default_rng(n)
    u = (rng.standard_normal((ns, n * n)) + 1j * rng.standard_normal((ns, n * n))) * 1e3
    return u.astype(np.complex64).astype(np.complex128)


@pytest.mark.parametrize("precision,tol", [(0, 1e-13), (1, 1.8e-5)])
@pytest.mark.parametrize("n", SIZES)
def test_drift_step_matches_numpy(lib, n, precision, tol):
    u = random_field(n)
    k2, _ = _k2_and_sigmoid(n, 2 * GM / (n - 1), 4.0 * np.arcsin(1.0) / LAMBDA0, 0.7, 0.9, 0.3)
    prop = np.exp(1j * k2 * 0.015)
    got = run(n, precision, u)
    for s in range(len(u)):
        want = np.fft.ifft2(np.fft.fft2(u[s].reshape(n, n)) * prop).ravel()
        assert np.max(np.abs(got[s] - want)) <= tol * np.max(np.abs(want))


@pytest.mark.parametrize("precision,tol", [(0, 1e-10), (1, 1e-4)])
@pytest.mark.parametrize("n", [20, 32, 128, 250])
def test_far_field_moments_match_oracle(lib, oracle, n, precision, tol):
    u = random_field(n)
    got = run(n, precision, u, diag=True)
    want = oracle.diag_field_fft(u, GM, LAMBDA0, 1, 0)
    got, want = np.asarray(got).reshape(len(u), -1), np.asarray(want).reshape(len(u), -1)
    assert got.shape == want.shape
    assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
