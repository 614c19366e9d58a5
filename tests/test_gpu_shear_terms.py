"""No metric term of a real shear is left out, however small.  On a grid with one coordinate sheared by s
(x = X + s Y, or y = Y + s X), a flow along the other one, uniform velocity and pressure and a density that varies
along the sheared index alone, d rho/dt comes through the off-diagonal entry alone: it is of order s V drho, and
zero without that term.

Tolerance: everything else in the right-hand side is rounding, a few 1e-16 V rho, against s V drho of 6e-14 V rho
(s = 5e-13, drho up to 0.13 rho a cell): a fifth of the largest entry.
"""
import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu

SHEAR = 5e-13
SPEED = 100.0


def sheared_case(sheared, kw):
    case = oc.mixing_layer_2d(mx=25, my=21, ybc="outflow", **kw)
    _, j, i = np.meshgrid(np.arange(1), np.arange(21), np.arange(25), indexing="ij")
    x, y = (i - 12) / 16.0, (j - 10) / 16.0
    case.x, case.y = (x + SHEAR * y, y) if sheared == "x" else (x, y + SHEAR * x)
    n = i / 24 if sheared == "x" else j / 20
    case.bv[0] = case.bv[0, 0, 0, 0] * (1 + 0.5 * np.sin(2 * np.pi * n))
    case.bv[1], case.bv[2] = (0.0, SPEED) if sheared == "x" else (SPEED, 0.0)
    case.bv[5] = case.bv[4] / (oc.R_AIR * case.bv[0])
    return case


@pytest.mark.parametrize("sheared", ["x", "y"])
@pytest.mark.parametrize("kw", [dict(reconstruction=5, inviscid_scheme=4), dict(reconstruction=2, inviscid_scheme=4)],
                         ids=["weno7_hllc", "muscl_hllc"])
def test_small_shear_moves_the_density(built, tmp_path, sheared, kw):
    import ostc
    from oracle import Oracle

    case = sheared_case(sheared, kw)
    s = ostc.Solver(str(oc.write_case(case, tmp_path / "c")))
    s.set_state(case.bv)
    got = s.rhs(1)[0]
    s.close()
    o = Oracle(case)
    o.set_state(case.bv)
    want = o.rhs(1)[0]
    signal = SHEAR * SPEED * case.grid_scale / 16 * case.bv[4].max() / (oc.R_AIR * 300.0)
    assert 0.05 * signal < np.max(np.abs(want)) < 0.5 * signal, (np.max(np.abs(want)), signal)
    assert np.max(np.abs(got - want)) <= 0.2 * np.max(np.abs(want))
