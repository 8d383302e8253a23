"""Sums of the FF_NonBonded parameter gradients: equal terms add up without error.

An atom with 102 partners of one kind at exactly one distance (the integer vectors of
length 9, on a grid of 0.5 A: every difference, square and r^2 is exact in FP32, so
all its terms are one number) has 102 times the gradient it has with one partner, up to
2^-33 kcal/mol per unit a flush into fixed point (eight at most of either kind here)."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KCAL = 4184.0 / 6.0221418e23


def _gradient(partners, radius):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    pos = 0.5 * np.concatenate([np.zeros((1, 3)), partners])
    n = len(pos)
    eps = 2.0e-11
    im = SystemImage([n], np.zeros(3), np.full(n, 0.37), np.full(n, radius), np.full(n, eps), np.full(n, 2e-26),
                     np.zeros((0, 3), np.int32), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(Cutoff=12.0, InnerCutoff=10.0, VdwCutoff=12.0, VdwInnerCutoff=10.0, Vdw14Scaling=1.0, Elec14Scaling=1.0,
               Dielectric=1.0, EnergySwitch=1, ForceSwitch=0, DoVdw=1, DoElec=1)
    ctx.set_positions(pos)
    g = ctx.param_grad(ffi.NB)[1]
    ctx.close()
    unit = {"charge": KCAL, "radius": KCAL, "epsilon": KCAL * np.sqrt(6.0221418e23 / 4184.0)}
    return {k: g[k][0] / unit[k] for k in unit}


@pytest.mark.parametrize("radius", [1.71, 1.83, 2.17])
def test_equal_terms_add_up(radius):
    v = np.array([p for p in itertools.product(range(-9, 10), repeat=3) if sum(x * x for x in p) == 81])
    assert len(v) == 102
    one, all_ = _gradient(v[:1], radius), _gradient(v, radius)
    for k in one:
        assert abs(all_[k] - 102 * one[k]) <= (16 + 102) * 2.0 ** -33, (k, all_[k], all_[k] - 102 * one[k])
