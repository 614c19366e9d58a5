"""Grouped boundary faces (k_bc_group) at the smallest extents a block may have (ngg + 2, where the nodes
the two sides of an axis read and write lie closest) and a little beyond, every kind that shares a
launch, against the CPU oracle over two RK3 steps.

Tolerance as the other parity tests: 1e-12 per conserved variable, max norm and L2.
"""
import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu


def _check(case, tmp_path):
    import ostc
    from oracle import Oracle

    s = ostc.Solver(str(oc.write_case(case, tmp_path / "case")))
    s.set_state(case.bv, sv=case.sv)
    s.step(2)
    cv, _ = s.get_state()
    s.close()
    o = Oracle(case)
    o.set_state(case.bv) if case.sv is None else o.set_state(case.bv, case.sv)
    o.step(2)
    co = o.get_state()[0]
    assert np.all(np.isfinite(co))
    err = oc.relative_errors(cv, co)
    assert max(max(e) for e in err) <= 1e-12, err


@pytest.mark.parametrize("my", [5, 6, 9])
@pytest.mark.parametrize("ybc", ["symmetry", "outflow"])
def test_2d_small_y(built, tmp_path, my, ybc):
    """WENO5 (three ghost layers): my from ngg + 2 between two slip or outflow faces."""
    _check(oc.mixing_layer_2d(mx=24, my=my, ybc=ybc), tmp_path)


@pytest.mark.parametrize("mz", [6, 7, 11])
@pytest.mark.parametrize("ybc", ["farfield", "outflow"])
def test_3d_small_z(built, tmp_path, mz, ybc):
    """WENO7 (four ghost layers): periodic mz from ngg + 2 under far-field or outflow y faces."""
    _check(oc.mixing_layer_3d(mx=20, my=14, mz=mz, ybc=ybc), tmp_path)


@pytest.mark.parametrize("mx,my", [(6, 6), (7, 6), (19, 13)])
def test_mixture_small(built, tmp_path, mx, my):
    """9 species (four ghost layers): periodic x and outflow y from ngg + 2."""
    _check(oc.reacting_mixing_layer_3d(mx=mx, my=my, mz=12), tmp_path)
