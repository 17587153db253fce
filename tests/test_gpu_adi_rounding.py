"""The FP64 ADI half steps over many field-only steps against extended precision: what a step's
rounding leaves in the field. A rounded coefficient scales the field by the same factor in
every step, so its error grows with the number of steps and outgrows the random roundings.

Tolerance, for the error of the field after n steps over n, eps = 2^-53. Systematic: the column solve's coefficient, in [0.5, 1), is the one
number whose rounding is left, an error uniform within eps / 2 of relative size up to eps:
0.29 eps rms; the part of it that the row solve's own coefficient leaves (4 r of 2 eps / 3) and
the off-diagonal coefficient (3 r eps): below 0.2 eps rms. Random: about 4 eps a step, 4 eps /
sqrt(n) of the n. Together 0.48 eps rms over the step factors at n = 150; 1.5 times that is
allowed. (Three uncompensated roundings a step give 1.2 eps.)"""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GRIDMAX = 1e-10, 11357.8, 1e-4
XKS = 2 * np.pi / LAMBDA0


def thomas(r, c):
    """(I - i c D) x = r along axis 0"""
    n = r.shape[0]
    a, b = -1j * c, 1 + 2j * c
    cp, d = [a / b], [r[0] / b]
    for k in range(1, n):
        m = b - a * cp[-1]
        cp.append(a / m)
        d.append((r[k] - a * d[-1]) / m)
    for k in range(n - 2, -1, -1):
        d[k] = d[k] - cp[k] * d[k + 1]
    return np.stack(d)


def stencil(u, c):
    z = np.zeros_like(u[:1])
    return u + 1j * c * (np.concatenate([u[1:], z]) - 2 * u + np.concatenate([z, u[:-1]]))


@pytest.mark.parametrize("ns,ngrid", [(1, 64), (80, 48)])
def test_field_steps_keep_the_rounding_of_one_coefficient(lib, ns, ngrid):
    import g4gpu
    steps = 150
    ext, cext = np.longdouble, np.clongdouble
    dgrid = 2 * GRIDMAX / (ngrid - 1)
    rng = np.random.default_rng(ngrid)
    u0 = (rng.normal(size=(ngrid, ngrid)) + 1j * rng.normal(size=(ngrid, ngrid))).astype(np.complex64)
    part = np.zeros((ns, 32, 6))
    part[..., 0] = GAMMA0
    errs = []
    for r in (0.02, 0.025, 0.03, 0.034, 0.04, 0.047, 0.055, 0.064):
        dz = r * 4 * XKS * dgrid * dgrid
        lat = T.undulator_lattice(1.7, dz, steps, 1, LAMBDA0, GAMMA0)
        lat[:, T.C["aw"]] = 0.0
        with g4gpu.Handle(g4gpu.Config(nslice=ns, npart=32, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                                       gammaref=GAMMA0, precision=0, time_run=0)) as h:
            h.set_lattice(lat)
            h.load_beam(part, np.ones(ns))
            h.load_field(0, np.repeat(u0.reshape(1, -1).astype(complex), ns, 0))
            h.run(0, steps, g4gpu.STAGE_FIELD)
            got = h.get_field(0)[0][-1].reshape(ngrid, ngrid)
        c = ext(0.25 * lat[0, T.C["dz"]] / (XKS * dgrid * dgrid))
        u = u0.astype(cext)
        for _ in range(steps):
            v = thomas(stencil(u, c).T, c).T
            u = thomas(stencil(v.T, c).T, c)
        d = got.astype(cext) - u
        errs.append(float(np.sqrt(np.sum(np.abs(d) ** 2) / np.sum(np.abs(u) ** 2))) / steps)
    eps = 2.0 ** -53
    assert np.sqrt(np.mean(np.square(errs))) <= 1.5 * eps * np.sqrt(0.29 ** 2 + 0.2 ** 2 + 16 / steps), np.array(errs) / eps
