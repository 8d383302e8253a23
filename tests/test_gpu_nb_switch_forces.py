"""Forces in the shell of an energy switch whose width FP32 does not hold: the distance
beyond the inner radius is a difference of two distances, not of two rounded multiples
of the width.

Isolated charged pairs with InnerCutoff = 10 (exact in FP32) and Cutoff = 11.04: as
r (1/w) - (10/w) in FP32 constants, the scaled distance is off by 7.3e-7 at 0.4 w for
every pair.  The mean force error may be what a bias of 2^-26 of the reciprocal root
makes of r (the slope's share of it) and six standard deviations of the mean of r's own
rounding; the planted shift is above twice that."""
import math

import numpy as np
import pytest

from test_gpu_nb_energy_constants import ECONV, KCAL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1])     # one switch for LJ and Coulomb, or one each
def test_mean_force_error_in_the_switching_shell(split):
    torch = pytest.importorskip("torch")
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    inner, cut, N, m = 10.0, 11.04, 4000, 16
    w = cut - inner
    rng = np.random.default_rng(2)
    pos = np.repeat(30.0 * np.stack(np.unravel_index(np.arange(N), (m, m, m)), 1), 2, axis=0)
    pos[1::2, 0] += inner + rng.uniform(0.3, 0.5, N) * w
    r = pos[1::2, 0] - pos[0::2, 0]
    im = SystemImage([2 * N], np.zeros(3), np.ones(2 * N), np.zeros(2 * N), np.zeros(2 * N), np.full(2 * N, 2e-26),
                     np.zeros((0, 3), np.int32), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(Cutoff=cut, InnerCutoff=inner, VdwCutoff=9.0 if split else cut, VdwInnerCutoff=8.0 if split else inner,
               Vdw14Scaling=1.0, Elec14Scaling=1.0, Dielectric=1.0, EnergySwitch=1, ForceSwitch=0, DoVdw=1, DoElec=1)
    ctx.set_positions(pos)
    fd = torch.zeros((2 * N, 3), dtype=torch.float64, device="cuda")
    ctx.compute_device(ffi.NB, fd.data_ptr())
    ctx.synchronize()
    got = fd.cpu().numpy()[1::2, 0] / (KCAL / 1e-10)
    ctx.close()
    F = np.float32
    econv = float(F(ECONV))                    # (the kernel's constant)

    def force(r, shift=0.0):
        u = (r - inner) / w + shift
        s = 1.0 - u * u
        return econv * (s * s / r ** 2 + 4.0 * u * s / (w * r))

    err = (got - force(r)) / force(r)
    h = 1e-4
    slope = np.abs(force(r + h) - force(r - h)).mean() / (2 * h) / force(r).mean()
    iw = 1.0 / w
    shift = r.mean() * (float(F(iw)) - iw) - (float(F(inner * iw)) - inner * iw)
    planted = abs((force(r, shift) / force(r) - 1.0).mean())
    tol = slope * (2.0 ** -26 * cut + 6.0 * 2.0 ** -24 * 16 / math.sqrt(12 * N)) + 2.0 ** -25
    assert planted > 2.0 * tol, (planted, tol)
    assert abs(err.mean()) <= tol, (err.mean(), err.std(), tol, planted)
