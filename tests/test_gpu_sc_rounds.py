"""Space charge of a mixed window whose CTAs take one round by twos and two by fours (700 slices),
and of one in a single round by either (300), against the same slices in a window of their own:
the particles' loads are grouped differently, their sums are the same.

Tolerance: FP32 sums of 256 particles (radial bins, 2^-24 each) in another order of the
shared-memory additions, a solve and a gather over 7 modes: 1e-5 of the largest change of gamma."""
import numpy as np
import pytest

import g4cases as T

pytestmark = pytest.mark.gpu
LAMBDA0, GAMMA0 = 1e-10, 11357.8


@pytest.mark.parametrize("ns", [300, 700])
@pytest.mark.parametrize("nz,nphi", [(1, 0), (2, 1), (1, 3)])
def test_window_size_does_not_change_the_space_charge(lib, ns, nz, nphi):
    import g4gpu
    npart = 256
    lat = T.undulator_lattice(1.7, 0.015, 1, 1, LAMBDA0, GAMMA0)
    part = g4gpu.host_load_beam(T.slice_params(ns, GAMMA0, 0.0, 0.4e-6, 15.0), 0, npart, 4, 5, 1, LAMBDA0, 1.0)
    part[..., 0] = GAMMA0

    def gammas(p):
        n = p.shape[0]
        with g4gpu.Handle(g4gpu.Config(nslice=n, npart=npart, ngrid=21, gridmax=1e-4, lambda0=LAMBDA0, sample=1.0,
                                       gammaref=GAMMA0, precision=1, time_run=0)) as h:
            h.set_lattice(lat)
            h.load_beam(p, np.full(n, 3e5))
            h.load_field(0, np.zeros((n, 21 * 21), dtype=complex))
            h.set_efield(rmax=4e-4, ngrid=100, nz=nz, nphi=nphi, longrange=False)
            h.run(0, 1, g4gpu.STAGE_PUSH)
            return h.get_beam()[..., 0] - GAMMA0

    whole = gammas(part)
    for a in (0, ns - 16):
        alone = gammas(part[a:a + 16])
        assert np.max(np.abs(alone)) > 0
        assert np.max(np.abs(whole[a:a + 16] - alone)) <= 1e-5 * np.max(np.abs(alone))
