"""Rectilinear blocks run kernels that leave the off-diagonal metric terms out; any other block runs the
general ones.  Stretched grids, grids with two axes reversed (a negative metric diagonal) and extents at the
edges of the sweeps' tiles against the CPU oracle, for every Riemann solver; and grids sheared by far less
than a grid spacing, which are not rectilinear.

Tolerance 1e-12 relative per conserved variable over two RK3 steps, as the other trajectory tests.
"""
import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu

SCHEMES = [(5, 4), (4, 3), (5, 1), (2, 4), (3, 3), (1, 1), (2, 2)]  # (reconstruction, inviscid scheme)
IDS = ["weno7_hllc", "weno5_ausm", "weno7_lf", "muscl_hllc", "nnd_ausm", "first_lf", "muscl_roe"]


def _case(dims, scheme):
    mx, my, mz = dims
    kw = dict(mx=mx, my=my, ybc="outflow", reconstruction=scheme[0], inviscid_scheme=scheme[1])
    return oc.mixing_layer_2d(**kw) if mz == 1 else oc.mixing_layer_3d(mz=mz, **kw)


def _check(case, tmp_path, steps=2):
    import ostc
    from oracle import Oracle

    s = ostc.Solver(str(oc.write_case(case, tmp_path / "case")))
    s.set_state(case.bv)
    s.step(steps)
    cv, _ = s.get_state()
    s.close()
    o = Oracle(case)
    o.set_state(case.bv)
    o.step(steps)
    co = o.get_state()[0]
    assert np.all(np.isfinite(co))
    err = oc.relative_errors(cv, co)
    assert max(max(e) for e in err) <= 1e-12, err


def _stretch(case):
    k, j, i = np.meshgrid(*(np.arange(n) for n in (case.mz, case.my, case.mx)), indexing="ij")
    h = case.x[0, 0, 1] - case.x[0, 0, 0]
    case.x = case.x + 0.3 * h * np.sin(0.5 * i)
    case.y = case.y + 0.3 * h * np.sin(0.4 * j + 0.2)
    if case.mz > 1:
        case.z = case.z + 0.3 * h * np.sin(0.6 * k)
    return case


@pytest.mark.parametrize("scheme", SCHEMES, ids=IDS)
@pytest.mark.parametrize("dims", [(35, 26, 1), (34, 17, 14)], ids=["2d", "3d"])
@pytest.mark.parametrize("reverse", [False, True], ids=["", "reversed"])
def test_stretched(built, tmp_path, scheme, dims, reverse):
    case = _stretch(_case(dims, scheme))
    if reverse:
        case.x, case.y = -case.x, -case.y
    _check(case, tmp_path)


@pytest.mark.parametrize("scheme", [SCHEMES[0], SCHEMES[3], SCHEMES[6]], ids=["weno7_hllc", "muscl_hllc", "muscl_roe"])
@pytest.mark.parametrize("dims", [(127, 15, 16), (128, 31, 33), (129, 32, 30), (16, 46, 17)])
def test_tile_edges(built, tmp_path, scheme, dims):
    _check(_case(dims, scheme), tmp_path, steps=1)


@pytest.mark.parametrize("scheme", [SCHEMES[0], SCHEMES[3]], ids=["weno7_hllc", "muscl_hllc"])
@pytest.mark.parametrize("shear", [1e-5, 1e-8])
def test_small_shear(built, tmp_path, scheme, shear):
    case = _case((30, 20, 12), scheme)
    case.x = case.x + shear * case.y
    _check(case, tmp_path)
