"""The field step with a slice's rows split between the CTAs of a cluster, against the oracle:
windows of few slices (2 to 8 CTAs), a pair asked for, grids that do not fit one CTA, bands of
unequal and of the fewest rows, more clusters than run at once, particle counts that take the
vector loads and those that do not, one4one slices, one CTA a slice beside it, and the field
record formed in the step. Inputs and tolerance are those of test_gpu_mixed_field."""
import numpy as np
import pytest

from test_gpu_mixed_field import GAMMA0, GRIDMAX, LAMBDA0, XKS, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,npart,ngrid,r,source,counts,kernel", [
    (1, 32, 25, 0.01, True, False, 0), (1, 64, 90, 0.03, True, False, 0), (4, 30, 101, 0.03, True, True, 0),
    (2, 32, 151, 0.034, True, False, 0), (1, 31, 151, 0.2, True, False, 0), (30, 32, 128, 0.03, True, False, 0),
    (50, 32, 73, 0.03, True, False, 0), (3, 64, 151, 0.034, True, False, 1), (1, 32, 167, 0.03, True, False, 0),
    (2, 32, 201, 0.2, True, False, 0), (3, 512, 255, 0.034, True, False, 0), (1, 30, 256, 0.03, True, True, 0),
    (60, 32, 255, 0.03, True, False, 0), (1, 64, 301, 0.03, True, False, 0), (2, 32, 401, 0.1, True, False, 0),
    (1, 32, 460, 0.03, True, False, 0), (1, 32, 520, 0.03, True, False, 0), (2, 32, 255, 0.4, True, False, 0),
    (160, 32, 45, 0.03, True, False, 0), (160, 30, 101, 0.03, True, True, 0), (160, 32, 165, 0.03, True, False, 0)])
def test_cluster_field_step_matches_oracle(lib, oracle, ns, npart, ngrid, r, source, counts, kernel):
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
        if kernel:
            h.set_launch_shapes(128, 512, kernel)
        h.run(0, 1, g4gpu.STAGE_FIELD)
        got = h.get_field(0)[0]
    tol = 1.2e-5 * (1 + 4 * r) * np.max(np.abs(ref)) + (4 * ngrid * 6e-8 + 6e-6) * 2 * np.max(np.abs(src))
    assert np.max(np.abs(got - ref)) <= tol


@pytest.mark.parametrize("ns,ngrid", [(1, 45), (3, 151), (20, 100), (2, 255), (1, 401)])
def test_record_formed_in_a_cluster_matches_the_record_after_it(lib, oracle, ns, ngrid):
    import g4gpu
    lat, part, cur, _, _, field, _, _ = setup(oracle, ns, 32, ngrid, 0.03, True, False)
    cfg = g4gpu.Config(nslice=ns, npart=32, ngrid=ngrid, gridmax=GRIDMAX, lambda0=LAMBDA0, sample=1.0,
                       gammaref=GAMMA0, precision=g4gpu.MIXED, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        h.load_field(0, field, first=0)
        _, fd = h.run_diag(0, 1, nharm=3)
        _, f2 = h.diag(3)
    dg = 2 * GRIDMAX / (ngrid - 1)
    p = fd[0, 0]
    assert np.allclose(p[:, 0], f2[0][:, 0], rtol=2e-6)
    assert np.max(np.abs(p[:, 1:5] - f2[0][:, 1:5])) <= 4e-6 * ngrid * dg
    assert np.allclose(p[:, 5], f2[0][:, 5], rtol=1e-6)
    assert np.allclose(np.sqrt(p[:, 7]), np.sqrt(f2[0][:, 7]), rtol=0, atol=4e-6 * ngrid * np.sqrt(np.max(f2[0][:, 7])))
