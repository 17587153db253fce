"""The mixed form's field step (deposition and ADI of a slice on chip) against the oracle,
over the grids, CTA sizes and step factors that choose its kernel and segments: odd and even
grids, the largest that keeps its stencil term in tensor memory (165) and beyond, short
segments, a factor too large for segments, particle counts that take the vector loads and
those that do not, and the field record formed in the step.

Tolerance (of the largest field value): a cell takes about 40 rounded FP32 operations (6e-8)
on values up to 1 + 4 r times the field's largest: 2.4e-6 (1 + 4 r), five times that for
their worst agreement. A source adds its own: weights from a cell coordinate of up to ngrid
in FP32 (2 ngrid 6e-8 in each direction), a fast sine of a reduced phase (4e-6) and 32
additions (2e-6), of the largest source value."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0, GRIDMAX = 1e-10, 11357.8, 1e-4
XKS = 2 * np.pi / LAMBDA0


def setup(oracle, ns, npart, ngrid, r, source, counts):
    dgrid = 2 * GRIDMAX / (ngrid - 1)
    rng = np.random.default_rng(ns * 1000 + ngrid)
    dz = r * 4 * XKS * dgrid * dgrid
    lat = T.undulator_lattice(1.7, dz, 1, 1, LAMBDA0, GAMMA0)
    lat[:, T.C["ky"]] = 175000.0
    if not source:
        lat[:, T.C["aw"]] = 0.0
    part = np.empty((ns, npart, 6))
    part[..., 0] = GAMMA0
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 2.5e-5, (ns, npart, 2))
    part[..., 4:6] = 0.0
    cur = rng.uniform(500, 3000, ns)
    cnt = rng.integers(1, npart + 1, ns).astype(np.int32) if counts else None
    src = None
    if source:
        src = np.concatenate([oracle.deposit_source(lat, 0, part[s:s + 1, :cnt[s] if counts else npart], cur[s:s + 1],
                                                    LAMBDA0, 1, ngrid, GRIDMAX) for s in range(ns)])
    field = rng.normal(size=(ns, ngrid * ngrid)) + 1j * rng.normal(size=(ns, ngrid * ngrid))
    field *= np.max(np.abs(src)) if source else 1.0
    return lat, part, cur, cnt, src, field.astype(np.complex64).astype(np.complex128), dz, dgrid


CASES = [(ns, npart, ng, r, source, counts, threads) for ns, npart, ng, r, source, counts, threads in [
    (2, 32, 25, 0.03, True, False, 0), (3, 32, 32, 0.03, False, False, 0), (1, 32, 45, 0.1, True, False, 0),
    (5, 31, 60, 0.03, True, False, 0), (2, 32, 101, 0.2, True, False, 0), (3, 30, 117, 0.03, True, True, 0),
    (2, 32, 128, 0.03, True, False, 0), (2, 32, 151, 0.034, True, False, 0), (2, 32, 151, 0.034, False, False, 512),
    (2, 32, 151, 0.034, True, False, 768), (2, 32, 151, 0.4, True, False, 1024), (1, 32, 160, 0.03, True, False, 0),
    (2, 32, 165, 0.03, True, False, 0), (2, 32, 166, 0.03, True, False, 0), (1, 32, 168, 0.03, False, False, 0),
    (2, 32, 64, 2.0, True, False, 0), (200, 32, 49, 0.03, True, False, 0)]]


@pytest.mark.parametrize("ns,npart,ngrid,r,source,counts,threads", CASES)
def test_mixed_field_step_matches_oracle(lib, oracle, ns, npart, ngrid, r, source, counts, threads):
    import g4gpu
    lat, part, cur, cnt, src, field, dz, dgrid = setup(oracle, ns, npart, ngrid, r, source, counts)
    first = ns - 1
    ref = oracle.adi_advance(field, src, first, dz, dgrid, XKS)
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.MIXED, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        if counts:
            h.load_beam_counts(part, cur, cnt)
        else:
            h.load_beam(part, cur)
        h.load_field(0, field, first=first)
        if threads:
            h.set_launch_shapes(128, threads, 0)
        h.run(0, 1, g4gpu.STAGE_FIELD)
        got = h.get_field(0)[0]
    tol = 1.2e-5 * (1 + 4 * r) * np.max(np.abs(ref))
    if source:
        tol += (4 * ngrid * 6e-8 + 6e-6) * 2 * np.max(np.abs(src))
    assert np.max(np.abs(got - ref)) <= tol


@pytest.mark.parametrize("ns,ngrid,threads", [(3, 45, 0), (2, 128, 0), (2, 151, 512), (2, 165, 0), (1, 168, 0)])
def test_record_formed_in_the_step_matches_the_record_after_it(lib, oracle, ns, ngrid, threads):
    """run_diag's field record (formed in the field kernel where it can) against a record
    of the same state formed by the diagnostic kernels: sums of ngrid^2 FP32 terms."""
    import g4gpu
    lat, part, cur, _, _, field, _, _ = setup(oracle, ns, 32, ngrid, 0.03, True, False)
    cfg = g4gpu.Config(nslice=ns, npart=32, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.MIXED, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, field, first=0)
        if threads:
            h.set_launch_shapes(128, threads, 0)
        bd, fd = h.run_diag(0, 1, nharm=3)
        b2, f2 = h.diag(3)
    dg = 2 * GRIDMAX / (ngrid - 1)
    assert np.allclose(bd[0], b2, rtol=1e-6, atol=1e-9, equal_nan=True)  # px = py = 0: no emittance
    p = fd[0, 0]
    assert np.allclose(p[:, 0], f2[0][:, 0], rtol=2e-6)                          # power
    assert np.max(np.abs(p[:, 1:5] - f2[0][:, 1:5])) <= 4e-6 * ngrid * dg         # centroid, size
    assert np.allclose(p[:, 5], f2[0][:, 5], rtol=1e-6)                          # on axis: the same value
    assert np.allclose(np.sqrt(p[:, 7]), np.sqrt(f2[0][:, 7]), rtol=0, atol=4e-6 * ngrid * np.sqrt(np.max(f2[0][:, 7])))
