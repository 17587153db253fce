"""The FP64 push's phase integration against the oracle where its short forms change over:
remainders of the nominal phase advance below 1/16, below 1/4 and beyond (energy offsets of
0 to 3 %), 1 / btpar0 from the integer series and (low energy) from the corrected one,
gamma changes that leave the reciprocal's series, one to three fields, phase offsets, offset
and tilted undulators, cached and fresh phasors, a chicane step.

Tolerance: theta advances by up to delz xks / gamma^2 ~ 10 rad a step with a rounding of
xks (1 - 1/btpar0) ~ 1e-16 xks delz = 1e-7 rad that both sides share bit for bit unless the
field's last bits move btper0 / gamma^2 over a rounding boundary (rare; one unit is 1e-7
rad). So 99 % of the particles agree within 1e-10 of the largest |theta| and all within
1e-6; gamma likewise through the field's phase."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0 = 1e-10


@pytest.mark.parametrize("harm", [[1], [1, 3], [3, 1, 5]])
@pytest.mark.parametrize("gamma0,spread", [(11357.8, 0.0), (11357.8, 2e-4), (11357.8, 5e-3), (11357.8, 3e-2),
                                           (2500.0, 1e-3)])
@pytest.mark.parametrize("offset", [False, True])
def test_plain_push_phase_matches_oracle(lib, oracle, harm, gamma0, spread, offset):
    import g4gpu
    ns, npart, ng, gm, nstep = 3, 256, 33, 1e-4, 4
    lat = T.undulator_lattice(1.7, 0.015, nstep, 1, LAMBDA0, gamma0)
    if offset:
        lat[:, T.C["ax"]], lat[:, T.C["ay"]] = 2e-5, -1e-5
        lat[:, T.C["gradx"]], lat[:, T.C["grady"]] = 0.3, -0.2
        lat[1, T.C["phase"]] = 0.7
    rng = np.random.default_rng(len(harm) + int(gamma0))
    part = np.empty((ns, npart, 6))
    part[..., 0] = gamma0 * (1 + spread * rng.uniform(-1, 1, (ns, npart)))
    part[..., 1] = rng.uniform(0, 6.28, (ns, npart))
    part[..., 2:4] = rng.normal(0, 3e-5, (ns, npart, 2))
    part[..., 4:6] = rng.normal(0, 0.02, (ns, npart, 2))
    cur = np.full(ns, 1000.0)
    gh = g4gpu.host_gauss_hermite(T.gauss_field_par(LAMBDA0, 1e9, 3e-5), gm, ng)
    fld = np.stack([np.stack([gh * (1 + 0.3j * s) / (k + 1) for s in range(ns)]) for k in range(len(harm))])
    ref = oracle.run_steps(lat, gamma0, part, cur, LAMBDA0, 1.0, harm, [gm] * len(harm), fld, [0] * len(harm), time_run=0)[0]
    cfg = g4gpu.Config(nslice=ns, npart=npart, ngrid=ng, harm=harm, gridmax=gm, lambda0=LAMBDA0, sample=1.0,
                       gammaref=gamma0, precision=g4gpu.PLAIN, time_run=0)
    with g4gpu.Handle(cfg) as h:
        h.set_lattice(lat)
        h.load_beam(part, cur)
        for k in range(len(harm)):
            h.load_field(k, fld[k])
        h.run(0, nstep)
        got = h.get_beam()
    for k in (0, 1):
        d = np.abs(got[..., k] - ref[..., k]) / np.max(np.abs(ref[..., k]))
        assert np.max(d) <= 1e-6
        assert np.mean(d <= 1e-10) >= 0.99
    for k in (2, 3, 4, 5):
        assert np.max(np.abs(got[..., k] - ref[..., k])) <= 1e-13 * np.max(np.abs(ref[..., k]))
