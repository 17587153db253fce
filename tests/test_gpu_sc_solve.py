"""The radial solves of the space charge on the device against the oracle: grids around the
32 rows a warp takes at a time, one mode and as many as run a thread each, particle counts
around the batches of loads. Plain FP64 form, tolerance of test_gpu_space_charge (1e-9 of the
largest change of gamma and theta)."""
import pytest

from test_gpu_space_charge import assert_plain_like, made_case, run_made

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npart,efield", [
    (256, (1e-4, 3, 1, 0, False)), (252, (2e-4, 31, 1, 0, False)), (256, (2e-4, 32, 2, 1, True)),
    (1028, (2e-4, 33, 1, 0, False)), (1020, (2e-4, 64, 5, 3, True)), (256, (2e-4, 65, 3, 5, False)),
    (256, (2e-4, 100, 7, 2, False))])
def test_radial_solve_matches_oracle(lib, oracle, npart, efield):
    gref, ng, gm, lat, part, cur, fld = case = made_case(npart=npart)
    oracle.set_efield(*efield)
    try:
        rp, rf, rfirst, _ = oracle.run_steps(lat, gref, part, cur, 1e-10, 1.0, [1], [gm], fld[None], [0])
    finally:
        oracle.set_efield()
    p, (f, first) = run_made(0, efield, *case)
    assert_plain_like(p, [(f, first)], part, rp, rf, rfirst)
