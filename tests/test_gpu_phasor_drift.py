"""The FP64 form's cached phasors against the stored phases over a long run: the bunching that a
record forms from them is that of the particles it describes. All particles of a slice are
alike, so that nothing averages out; off resonance the phases reach thousands of radians, whose
own rounding must not part the two.

Tolerance: a step's rotations (the step's phase offset where there is one, its nominal advance,
the remainder) each bring the rounding of a constant and of a complex product, at most 4e-16:
1.2e-15 a step, all of one sign; and 2^-53 of the sums."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0 = 1e-10, 11357.8


@pytest.mark.parametrize("harm,phase,steps", [([1], 0.0, 600), ([1], 0.7, 300), ([3, 1], 0.0, 300)])
def test_recorded_bunching_is_that_of_the_stored_phases(lib, harm, phase, steps):
    import g4gpu
    ns, npart = 3, 64
    lat = T.undulator_lattice(1.7, 0.015, steps, 1, LAMBDA0, GAMMA0)
    lat[:, T.C["phase"]] = phase
    part = np.zeros((ns, npart, 6))
    part[..., 0] = GAMMA0 + np.array([-3.0, 0.0, 2.5])[:, None]
    part[..., 1] = np.array([0.3, 2.1, 5.5])[:, None]
    part[..., 2] = 1e-5
    with g4gpu.Handle(g4gpu.Config(nslice=ns, npart=npart, ngrid=31, harm=harm, gridmax=1e-4, lambda0=LAMBDA0,
                                   sample=1.0, gammaref=GAMMA0, precision=0, time_run=0)) as h:
        h.set_lattice(lat)
        h.load_beam(part, np.ones(ns))
        for k in range(len(harm)):
            h.load_field(k, np.zeros((ns, 31 * 31), dtype=complex))
        h.run(0, steps, g4gpu.STAGE_PUSH)
        bd, _ = h.diag(1)
        th = h.get_beam()[:, 0, 1]
    z = bd[:, 24] * np.exp(1j * bd[:, 25])
    want = (np.cos(th.astype(np.longdouble)) + 1j * np.sin(th.astype(np.longdouble))).astype(complex)
    assert np.max(np.abs(th)) > 300
    assert np.max(np.abs(z - want)) <= 1.2e-15 * steps + 1e-15
