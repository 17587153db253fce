"""The FP64 ADI half steps on tiles of lines against the oracle, over the rules that choose
their shape: lines a CTA (2, 4, 8, 16), segments a line, one thread per line where the
recurrences fade too slowly, the line is too short or two lines do not fit shared memory;
last bands and segments with remainders, with and without a source, a ring start.

Tolerance: a cell takes about 40 rounded operations (1.1e-16 each) on values up to 1 + 4 r
times the field's largest (the norm of I + i r D), a source of 32 particles adds as many
roundings, and the segments' truncation is 2^-62: below 2e-14 (1 + 4 r) of the largest value.
The source is formed here with the deposition's own cell coordinate, fma(x, 1 / dgrid,
gridmax / dgrid) (the reference's (x + gridmax) / dgrid differs from it in the last bit of a
number as large as ngrid, and so do the weights), so that only the solve is compared."""
from fractions import Fraction

import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu

LAMBDA0, GAMMA0, GRIDMAX = 1e-10, 11357.8, 1e-4
XKS = 2 * np.pi / LAMBDA0


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def deposit(oracle, lat, part, cur, ngrid):
    """The source of lattice step 0 (FieldSolverADI.cpp:13-52), harmonic 1, no offsets."""
    ns, npart = part.shape[:2]
    dgrid = 2 * GRIDMAX / (ngrid - 1)
    out = np.zeros((ns, ngrid * ngrid), dtype=np.complex128)
    row = lat[0]
    scl = oracle.fc(row[T.C["aw"]], 0, 1) * 376.73 * cur * XKS * row[T.C["dz"]]
    scl = scl / (4 * 510998.95069 * npart * dgrid * dgrid)
    for s in range(ns):
        for g, th, x, y in part[s, :, :4]:
            if not (abs(x) < GRIDMAX and abs(y) < GRIDMAX):
                continue
            tx, ty = (fma(v, 1 / dgrid, GRIDMAX * (1 / dgrid)) for v in (x, y))
            ix, iy = int(tx), int(ty)
            ux, uy = tx - ix, ty - iy
            part_ = np.sqrt(1 + row[T.C["kx"]] * x * x + row[T.C["ky"]] * y * y) * scl[s] / g
            v = complex(np.sin(th), np.cos(th)) * part_
            i = ix + iy * ngrid
            out[s, i] += (1 - ux) * (1 - uy) * v
            out[s, i + 1] += ux * (1 - uy) * v
            out[s, i + ngrid] += (1 - ux) * uy * v
            out[s, i + ngrid + 1] += ux * uy * v
    return out


@pytest.mark.parametrize("ns,ngrid,r,source,first", [
    (1, 3, 0.03, True, 0), (1, 25, 0.03, True, 0), (1, 27, 0.03, True, 0), (1, 51, 0.03, False, 0),
    (3, 128, 0.03, True, 2), (1, 255, 0.02, True, 0), (1, 801, 0.03, True, 0), (1, 3199, 0.03, False, 0),
    (1, 3201, 0.03, True, 0), (25, 101, 0.03, True, 7), (80, 40, 0.03, True, 0), (60, 90, 0.03, False, 59),
    (70, 61, 0.03, True, 1), (160, 33, 0.03, True, 3), (2, 151, 0.4, True, 1), (90, 79, 0.4, True, 0),
    (90, 151, 0.4, True, 0), (2, 60, 4.0, True, 0), (200, 49, 4.0, False, 11)])
def test_plain_adi_matches_oracle(lib, oracle, ns, ngrid, r, source, first):
    import g4gpu
    npart = 32
    dgrid = 2 * GRIDMAX / (ngrid - 1)
    rng = np.random.default_rng(ns * 1000 + ngrid)
    dz = r * 4 * XKS * dgrid * dgrid
    lat = T.undulator_lattice(1.7, dz, 1, 1, LAMBDA0, GAMMA0)
    if not source:
        lat[:, T.C["aw"]] = 0.0
    part = np.empty((ns, npart, 6))
    part[..., 0] = GAMMA0
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    part[..., 4:6] = 0.0
    cur = rng.uniform(500, 3000, ns)
    field = rng.normal(size=(ns, ngrid * ngrid)) + 1j * rng.normal(size=(ns, ngrid * ngrid))
    field *= 1e-3
    src = None
    if source:
        src, osrc = deposit(oracle, lat, part, cur, ngrid), oracle.deposit_source(lat, 0, part, cur, LAMBDA0, 1, ngrid, GRIDMAX)
        assert np.max(np.abs(src - osrc)) <= 1e-11 * np.max(np.abs(osrc))
    ref = oracle.adi_advance(field, src, first, dz, dgrid, XKS)
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.PLAIN, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, field, first=first)
        h.run(0, 1, g4gpu.STAGE_FIELD)
        got = h.get_field(0)[0]
    assert np.max(np.abs(ref - field)) > 1e-5 * np.max(np.abs(field))  # the step does something
    assert np.max(np.abs(got - ref)) <= 2e-14 * (1 + 4 * r) * np.max(np.abs(ref))
