"""g4gpu_run_diag with the records formed beside the steps (one slice, few, many) and in line
(between them), against a record taken after every step run by itself: the same sums of the
same state. The deposition's atomics make two runs differ: 1e-9 of the largest value of a
column in FP64, 1e-4 in the mixed form (12 steps of FP32 rounding, as the oracle comparisons
of the mixed form allow)."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GM = 1e-10, 11357.8, 1e-4


@pytest.mark.parametrize("precision,ns,npart,ngrid,solver", [
    (0, 1, 512, 65, 0), (0, 5, 256, 41, 0), (0, 64, 128, 33, 0), (0, 70, 64, 32, 1), (1, 1, 512, 65, 0), (1, 20, 256, 49, 0),
    (1, 60, 128, 41, 0), (1, 610, 64, 33, 0), (1, 3, 128, 181, 0), (1, 2, 64, 341, 0), (1, 620, 64, 32, 1)])
def test_records_of_a_run_match_records_of_single_steps(lib, precision, ns, npart, ngrid, solver):
    import g4gpu
    rng = np.random.default_rng(ns + ngrid)
    steps = 12 if ngrid < 300 else 4
    lat = T.undulator_lattice(1.7, 0.015, steps, 1, LAMBDA0, GAMMA0)
    part = g4gpu.host_load_beam(T.slice_params(ns, GAMMA0, 1.0, 0.4e-6, 15.0), 0, npart, 4, 5, 1, LAMBDA0, 1.0)
    cur = np.linspace(1000.0, 3000.0, ns)
    fld = np.repeat(g4gpu.host_gauss_hermite(T.gauss_field_par(LAMBDA0, 1e5, 30e-6), GM, ngrid)[None, :], ns, axis=0)

    def handle():
        h = g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, gridmax=GM, lambda0=LAMBDA0, sample=1.0,
                                      gammaref=GAMMA0, precision=precision, time_run=1 if ns > 1 else 0, solver=solver))
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, fld)
        return h

    with handle() as h:
        bd, fd = h.run_diag(0, steps, nharm=2)
        end = h.get_beam()
    with handle() as h:
        one = []
        for i in range(steps):
            h.run(i, 1)
            one.append(h.diag(2))
        end1 = h.get_beam()
    tol = 1e-9 if precision == 0 else 1e-4
    phases = {25, 27}  # columns of a bunching factor's phase: compared as complex numbers

    def close(a, b, what):
        s = np.nanmax(np.abs(b))
        assert np.nanmax(np.abs(a - b)) <= tol * s if s > 0 else np.all(a == b), what

    for i in range(steps):
        b1, f1 = one[i]
        for c in range(14, bd.shape[-1]):
            if c in phases:
                close(bd[i][:, c - 1] * np.exp(1j * bd[i][:, c]), b1[:, c - 1] * np.exp(1j * b1[:, c]), (i, c))
            else:
                close(bd[i][:, c], b1[:, c], (i, c))
        close(bd[i][:, 0], b1[:, 0], (i, 0))
        close(bd[i][:, 3], b1[:, 3], (i, 3))
        close(fd[i, 0][:, 0], f1[0][:, 0], (i, "power"))
    close(end[..., 0], end1[..., 0], "gamma")
