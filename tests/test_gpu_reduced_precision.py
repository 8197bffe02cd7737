"""What the reduced-precision forms change a state by, field by field: the FP32
form of the solver and the BF16 split products of the per-operator path.

At Mach 0.1 the energy is 180 and a step changes it by 1e-6 of that, so a
tolerance on the state says little about the step.  Here the change over two
steps is compared with the FP64 form's, and the unit is the part of it that the
viscous flux makes (FP64 with and without viscosity): a form that lost the
viscous flux is off by one unit in momentum and energy.

Bounds.  A form rounds fluxes of the size of the pressure (71) in momentum and
of the enthalpy flux (250) in energy, at 2^-24 (FP32) or about 2^-16 and 2^-24 of
the products' operands (BF16 x 3 and x 6), and the line derivative multiplies that
by 10 to 50; the viscous part is 0.01 times second derivatives of size 3 in
momentum, and of a temperature of size 1 in energy.  Measured on these meshes, in
units: FP32 0.004 in momentum and 0.03 in energy, BF16x3 0.02 and 0.35, BF16x6
0.001 and 0.006.  The bounds are about twice that, and below one unit."""
import numpy as np
import pytest

import hifiles_b200 as H
from hifiles_b200 import seam
from test_gpu_tiles import GAMMA, PR, _tgv

pytestmark = pytest.mark.gpu

PHYS = dict(gamma=GAMMA, prandtl=PR, mu_inf=0.01, rt_inf=1.0, c_sth=1.0, fix_vis=1.0, tau=1.0, pen_fact=0.5)
MOMENTUM, ENERGY = [1, 2], 4     # the third momentum component has no viscous part at first


def _box(P, n, **kw):
    L = 2 * np.pi
    return H.Solver.box(3, P, n, (0, 0, 0), (L, L, L), viscous=True, vcjh_scheme=1, **dict(PHYS, **kw))


def _change(s, u0, **kw):
    s.set_state(u0)
    s.advance(2, 1e-3, **kw)
    return s.get_state() - u0


def _fields(d):
    return np.sqrt((d * d).sum(axis=(0, 1)))


@pytest.mark.parametrize("P,n", [(2, (9, 8, 7)), (3, (8, 8, 8)), (4, (5, 5, 5))])
def test_change_of_each_field(P, n):
    s = _box(P, n)
    u0 = _tgv(s.geometry()["pos_upts"])
    d64 = _change(s, u0)
    unit = _fields(d64 - _change(_box(P, n, mu_inf=0.0), u0))
    # the viscous part shows in what the step does
    assert np.all(unit[MOMENTUM] > 0.02 * _fields(d64)[MOMENTUM]) and unit[ENERGY] > 0.01 * _fields(d64)[ENERGY]
    op = seam.OperatorStage(s, PHYS, P, vcjh_scheme=1)
    forms = [("fp32", _change(_box(P, n, precision=1), u0), 0.01, 0.06),
             ("bf16x3", _change(op, u0, gemm_precision=1), 0.045, 0.7),
             ("bf16x6", _change(op, u0, gemm_precision=2), 0.0025, 0.012)]
    for name, d, mom, en in forms:
        e = _fields(d - d64) / unit
        assert np.all(e[MOMENTUM] < mom) and e[ENERGY] < en, (name, e)
        # the inviscid change of the third momentum component
        w = _fields(d - d64)[3] / _fields(d64)[3]
        assert w < 2e-3, (name, w)


@pytest.mark.parametrize("P,n", [(2, (9, 8, 7)), (3, (8, 8, 8)), (4, (5, 5, 5))])
def test_fp32_norms(P, n):
    """Residual norms of the FP32 form: the residual's error is up to 1e-3 of
    the momentum and energy residuals and 1e-2 of the density's, which a
    divergence-free start keeps small."""
    s, s32 = _box(P, n), _box(P, n, precision=1)
    u0 = _tgv(s.geometry()["pos_upts"])
    s.set_state(u0)
    s32.set_state(u0)
    n64, n32 = s.advance(2, 1e-3, norms=True), s32.advance(2, 1e-3, norms=True)
    assert np.all(np.abs(n32 - n64) <= np.array([1e-2, 1e-3, 1e-3, 1e-3, 2e-3]) * n64), (n32, n64)
