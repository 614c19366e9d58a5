"""Boundary faces that share a launch (k_bc_group) or must not: several patches on one side, of one kind and of
several, and different kinds on the two sides of an axis at the smallest extent a block may have (ngg + 2), against
the CPU oracle over two RK3 steps.

Tolerance as the other parity tests: 1e-12 per conserved variable, max norm and L2.
"""
import dataclasses

import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu

SLIP = {"type": ("string", "symmetry"), "label": ("int", 3)}
OUT = {"type": ("string", "outflow"), "label": ("int", 6)}


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


def _patched(case, side, labels):
    """Splits a y face (2: low, 3: high) along i into patches of the given labels that meet at a node."""
    raw = case.faces[side].raw
    n = len(labels)
    cuts = [raw[0] + (raw[1] - raw[0]) * q // n for q in range(n + 1)]
    patches = [oc.Face((cuts[q], cuts[q + 1]) + raw[2:], labels[q]) for q in range(n)]
    case.faces[side:side + 1] = patches
    case.bc_structs.update({"slipwall": SLIP, "outflow": OUT})
    return case


@pytest.mark.parametrize("labels", [(6, 6), (6, 6, 6), (6, 3), (3, 6, 6), (3, 3)],
                         ids=["out2", "out3", "out_slip", "slip_out2", "slip2"])
@pytest.mark.parametrize("side", [2, 3], ids=["low", "high"])
@pytest.mark.parametrize("mz", [1, 8])
def test_patches_on_a_side(built, tmp_path, labels, side, mz):
    case = oc.mixing_layer_2d(mx=31, my=13, ybc="outflow") if mz == 1 else oc.mixing_layer_3d(mx=31, my=12, mz=mz, ybc="outflow")
    _check(_patched(case, side, labels), tmp_path)


def test_far_field_patches(built, tmp_path):
    """Two far-field patches and an outflow one on a side, far field opposite."""
    _check(_patched(oc.mixing_layer_3d(mx=31, my=12, mz=8), 3, (4, 6, 4)), tmp_path)


@pytest.mark.parametrize("low,high", [(41, 3), (3, 4), (41, 6), (6, 4), (6, 3), (3, 6)])
@pytest.mark.parametrize("my", [6, 9])
def test_kinds_across_an_axis(built, tmp_path, low, high, my):
    """WENO7 (four ghost layers): far field, slip wall and outflow opposite one another."""
    case = oc.mixing_layer_3d(mx=20, my=my, mz=7)
    case.faces[2] = dataclasses.replace(case.faces[2], label=low)
    case.faces[3] = dataclasses.replace(case.faces[3], label=high)
    case.bc_structs.update({"slipwall": SLIP, "outflow": OUT})
    _check(case, tmp_path)


@pytest.mark.parametrize("labels", [(6, 6), (6, 3)], ids=["out2", "out_slip"])
def test_mixture_patches(built, tmp_path, labels):
    """5 % noise on the mass fractions: a field constant along x takes weights from its rounding where patches of two
    kinds break that constancy (epsilon is ~1e-40 of the fluxes), and those of two builds differ."""
    case = oc.reacting_mixing_layer_3d(mx=19, my=8, mz=8)
    case.sv = case.sv * (1 + 0.05 * np.random.default_rng(1).random(case.sv.shape))
    case.sv /= case.sv.sum(axis=0)
    mw = 1 / np.einsum("l...,l->...", case.sv, 1 / case.mixture["tables"].mw)
    case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
    _check(_patched(case, 3, labels), tmp_path)
