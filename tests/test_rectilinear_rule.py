"""Which blocks run the kernels without the off-diagonal metric terms (host side, no GPU): those whose grid lines
are the coordinate axes, bit for bit at their own nodes and to rounding in their ghost layers.  A shear of any size, or one node
off its line by one ulp, is not."""
import numpy as np
import pytest

import ostc
import ostc_cases as oc


def _count(case, tmp_path):
    return ostc.probe_case(str(oc.write_case(case, tmp_path / "c")))["n_rectilinear"]


def _case(mz=10):
    return oc.mixing_layer_2d(mx=24, my=18) if mz == 1 else oc.mixing_layer_3d(mx=24, my=18, mz=mz)


@pytest.mark.parametrize("mz", [1, 10])
@pytest.mark.parametrize("how", ["uniform", "stretched", "reversed", "offset"])
def test_axis_aligned(built, tmp_path, mz, how):
    case = _case(mz)
    if how == "stretched":
        case.x = case.x + 0.02 * np.sin(9.0 * case.x)
        case.y = case.y * (1 + 0.1 * case.y ** 2)
    elif how == "reversed":
        case.x, case.y = -case.x, -case.y
    elif how == "offset":
        case.x = case.x + 17.3
    assert _count(case, tmp_path) == 1


@pytest.mark.parametrize("mz", [1, 10])
@pytest.mark.parametrize("shear", [1e-3, 1e-8, 1e-11, 1e-12, 1e-13, 1e-14])
def test_any_shear_is_general(built, tmp_path, mz, shear):
    case = _case(mz)
    case.x = case.x + shear * case.y
    assert _count(case, tmp_path) == 0


@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_one_ulp_is_general(built, tmp_path, axis):
    case = _case()
    a = getattr(case, axis).copy()
    a[4, 9, 13] = np.nextafter(a[4, 9, 13], np.inf)
    setattr(case, axis, a)
    assert _count(case, tmp_path) == 0


def test_edge_rounding_beyond_the_bar_is_general(built, tmp_path):
    """Far from the origin the ghost grid's edges round by more than 1e-12 of a spacing."""
    case = _case()
    case.x = case.x + 1.0e4 / 3
    assert _count(case, tmp_path) == 0


def test_chain(built, tmp_path):
    case = oc.multiblock_mixing_layer_3d(nb=3, lo=10, hi=16, my=10, mz=8, seed=1)
    assert _count(case, tmp_path) == 3
    case.blocks[1].x = case.blocks[1].x + 1e-13 * case.blocks[1].y
    # the sheared block, and its neighbours, whose ghosts are its nodes
    assert _count(case, tmp_path) == 0


def test_chain_of_uneven_blocks(built, tmp_path):
    """Interfaces on parts of a side: the ghost layer holds the neighbour's coordinates beside reflected ones, which
    differ by rounding."""
    case = oc.multiblock_mixing_layer_3d(nb=6, lo=16, hi=40, seed=3, uneven_axes=True)
    assert _count(case, tmp_path) == 6
