"""The flux-split sweeps far from the usual grid sizes.  Their weights do not change when the grid is scaled (the
epsilon follows the split fluxes), so with a grid scaled by a power of two, which scales every metric entry without
rounding, the inviscid right-hand side is that of the plain grid times the square of the factor.

Tolerance: the operations are the same ones on scaled operands; what may differ is the rounding where a quotient
takes another of its equivalent forms: a few rounding errors of the terms that sum to an entry, 1e-6 (FP32) and 1e-12
(FP64, whose adjoint adds a node's ~200 terms in any order) of each variable's largest entry.
"""
import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu


def layer(scheme, power, zero_half=()):
    """9 species on a grid scaled by 2^power; species of zero_half are absent from the half with low i."""
    case = oc.reacting_mixing_layer_3d(18, 14, 10, inviscid_scheme=scheme, finite_rate=False)
    case.grid_scale = case.grid_scale * 2.0 ** power
    tb = case.mixture["tables"]
    for n in zero_half:
        l = tb.names.index(n)
        case.sv[tb.names.index("N2"), ..., :9] += case.sv[l, ..., :9]
        case.sv[l, ..., :9] = 0.0
    mw = 1 / np.einsum("l...,l->...", case.sv, 1 / tb.mw)
    case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
    return case


def relative(a, b):
    """Largest difference of each variable over its largest entry (the three momentum components share one)."""
    top = [np.max(np.abs(v)) for v in b]
    top[1:4] = [max(top[1:4])] * 3
    return max(np.max(np.abs(x - y)) / t for x, y, t in zip(a, b, top))


def solver(case, path):
    import ostc

    s = ostc.Solver(str(oc.write_case(case, path)))
    s.set_state(case.bv, sv=case.sv)
    return s


@pytest.mark.parametrize("scheme", [71, 72])
@pytest.mark.parametrize("power", [-25, 25])
def test_mixed_precision(built, tmp_path, scheme, power):
    """2^-25: face areas of 1e-23, whose squares FP32 cannot hold."""
    import ostc

    out = []
    for p in (0, power):
        s = solver(layer(scheme, p), tmp_path / f"p{p}")
        s.set_precision(ostc.PREC_MIXED)
        out.append(s.rhs(1))
        s.close()
    assert np.all(np.isfinite(out[1]))
    assert relative(out[1] * 2.0 ** (-2 * power), out[0]) <= 1e-6


@pytest.mark.parametrize("scheme", [71, 72])
@pytest.mark.parametrize("power", [-25, 70, 75])
def test_fp64_and_adjoint(built, tmp_path, scheme, power):
    """Radicals absent from half of the block: eps alone in the weights' denominators there.  2^-25 takes the product
    of four of them below the FP64 range; 2^70 and 2^75 take that of four indicators above it."""
    rhs, vjp = [], []
    for p in (0, power):
        s = solver(layer(scheme, p, ("OH", "O", "H", "HO2", "H2O2")), tmp_path / f"p{p}")
        rhs.append(s.rhs(1))
        vjp.append(s.rhs_vjp(np.random.default_rng(3).standard_normal(rhs[0].shape), 1))
        s.close()
    for out in (rhs, vjp):
        assert np.all(np.isfinite(out[1])) and np.any(out[0])
        assert relative(out[1] * 2.0 ** (-2 * power), out[0]) <= 1e-12


@pytest.mark.parametrize("scheme", [71, 72])
def test_vanishing_species_without_reference_state(built, tmp_path, scheme):
    """Without a reference state the epsilon is 0, and where a mass fraction falls from 1e-3 to 1e-50 within a stencil
    the weight sums of the two sides are near 1e190 each.  Against the oracle, 1e-12 as the other comparisons of one
    evaluation; every field carries noise and all faces are periodic, since a constant field (the ghosts of an
    outflow face, too) has indicators of 0 / 0 then."""
    from oracle import Oracle

    case = layer(scheme, 0)
    case.freestream = None
    case.faces = [oc.Face(f.raw, 8) for f in case.faces]
    rng = np.random.default_rng(8)
    tb = case.mixture["tables"]
    case.sv = case.sv * (1 + 0.1 * rng.random(case.sv.shape)) + 1e-3 * rng.random(case.sv.shape)
    l = tb.names.index("H2O2")
    case.sv[l, :, :, :9] = 1e-50 * (1 + 0.1 * rng.random(case.sv[l, :, :, :9].shape))
    case.sv /= case.sv.sum(axis=0)
    for q in (1, 2, 3):
        case.bv[q] += 5.0 * rng.standard_normal(case.bv[q].shape)
    case.bv[5] *= 1 + 0.01 * rng.standard_normal(case.bv[5].shape)
    case.bv[4] *= 1 + 0.01 * rng.standard_normal(case.bv[4].shape)
    mw = 1 / np.einsum("l...,l->...", case.sv, 1 / tb.mw)
    case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
    s = solver(case, tmp_path / "c")
    got = s.rhs(1)
    s.close()
    o = Oracle(case)
    o.set_state(case.bv, case.sv)
    want = o.rhs(1)
    assert np.all(np.isfinite(want)) and np.all(np.isfinite(got))
    assert relative(got, want) <= 1e-12
