"""Every column of g4gpu_run_diag's records, formed beside the steps that follow, against a record
taken after each step run by itself, on windows whose records overlap the next step's kernels.
A read of the state a step too late would show a record of the next step: the records of
consecutive steps are first seen to differ by far more than the tolerance.

Tolerance: the two runs differ by the order of the depositions' additions alone, which 6 steps
carry into the field (FP64 1e-12, mixed 2e-5 of the largest value) and from there into the beam.
Columns that are quotients and differences of others (emittances, Twiss parameters, sizes) are
compared on the scale of what they are formed from."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GM = 1e-10, 11357.8, 1e-4


@pytest.mark.parametrize("precision,ns,npart,ngrid,solver,harm", [
    (0, 1, 4096, 255, 0, [1]), (0, 160, 512, 65, 0, [1]), (0, 64, 1024, 96, 1, [1]), (0, 94, 256, 101, 0, [1, 3]),
    (1, 1, 8192, 151, 0, [1]), (1, 30, 4096, 101, 0, [1]), (1, 640, 1024, 101, 0, [1]), (1, 640, 512, 96, 1, [1, 3])])
def test_every_column_is_that_of_its_own_step(lib, precision, ns, npart, ngrid, solver, harm):
    import g4gpu
    rng = np.random.default_rng(ns + ngrid)
    steps = 6
    lat = T.undulator_lattice(1.7, 0.015, steps, 1, LAMBDA0, GAMMA0)
    part = g4gpu.host_load_beam(T.slice_params(ns, GAMMA0, 1.0, 0.4e-6, 15.0), 0, npart, 4, 5, 1, LAMBDA0, 1.0)
    part[..., 2:4] += 1e-5
    part[..., 4:6] += 0.1
    cur = np.linspace(1000.0, 3000.0, ns)
    mode = g4gpu.host_gauss_hermite(T.gauss_field_par(LAMBDA0, 1e9, 30e-6), GM, ngrid)
    fld = mode[None, :] * np.exp(1j * rng.uniform(0, 0.3, ns))[:, None]

    def handle():
        h = g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, harm=harm, gridmax=GM, lambda0=LAMBDA0,
                                      sample=1.0, gammaref=GAMMA0, precision=precision, time_run=1 if ns > 1 else 0,
                                      solver=solver))
        h.set_lattice(lat)
        h.load_beam(part, cur)
        for k in range(len(harm)):
            h.load_field(k, fld)
        return h

    with handle() as h:
        bd, fd = h.run_diag(0, steps, nharm=2)
    with handle() as h:
        one = []
        for i in range(steps):
            h.run(i, 1)
            one.append([v.copy() for v in h.diag(2)])
    tol = 1e-12 if precision == 0 else 2e-5

    def columns(b, f):
        """The columns as arrays and the scale each is compared on."""
        c = {n: i for i, n in enumerate(g4gpu.DB_COLS)}
        out = {}
        for n in ("energy", "energyspread", "xmin", "xmax", "pxmin", "pxmax", "ymin", "ymax", "pymin", "pymax", "emin", "emax"):
            out[n] = (b[:, c[n]], np.max(np.abs(b[:, c[n]])))
        for u in "xy":
            size = np.max(b[:, c[u + "size"]]) + np.max(np.abs(b[:, c[u + "position"]]))
            out[u + "position"] = (b[:, c[u + "position"]], size)
            out[u + "size"] = (b[:, c[u + "size"]], size * size / np.min(b[:, c[u + "size"]]))
            out["p" + u] = (b[:, c["p" + u + "position"]], np.max(np.abs(b[:, c["p" + u + "position"]])))
            for n in ("emit", "beta", "alpha"):
                out[n + u] = (b[:, c[n + u]], 100 * np.max(np.abs(b[:, c[n + u]])))
        for m in (0, 1):
            out["bunching%d" % m] = (b[:, 24 + 2 * m] * np.exp(1j * b[:, 25 + 2 * m]), 1.0)
        for k in range(len(harm)):
            p = f[k]
            dg = 2 * GM / (ngrid - 1)
            on = p[:, 0] > 0  # the slice that slipped in
            out["power%d" % k] = (p[on, 0], np.max(p[on, 0]))
            for j in (1, 2, 3, 4):
                out["centroid%d%d" % (k, j)] = (p[on, j], 10 * GM)
            out["axis%d" % k] = (np.sqrt(p[on, 5]) * np.exp(1j * p[on, 6]), np.max(np.sqrt(p[on, 5])))
            out["far%d" % k] = (np.sqrt(p[on, 7]) * np.exp(1j * p[on, 8]), ngrid * np.max(np.sqrt(p[on, 7])))
            out["slices%d" % k] = (on.astype(float), 1.0)
        return out

    for i in range(steps):
        got, want = columns(bd[i], fd[i]), columns(*one[i])
        for n, (v, scale) in want.items():
            assert np.max(np.abs(got[n][0] - v)) <= tol * scale, (i, n)
        if i:
            before = columns(*one[i - 1])
            for kind in (("xposition", "xmax", "energyspread"), ("power0", "axis0", "far0")):
                assert any(before[n][0].shape != want[n][0].shape or  # a slice slipped in
                           np.max(np.abs(before[n][0] - want[n][0])) > 10 * tol * want[n][1] for n in kind), (i, kind)
