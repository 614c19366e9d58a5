"""The adjoint of the chemical source over the reaction lists where no reaction takes the equilibrium constant:
backward rates from REV coefficients, with third-body sums of present colliders and of absent ones only (a sum of
zero, whose derivative is not), against the dense kernel, where every derivative is by dual numbers.  A
reaction with five molecules on a side does not fit the lists, so the mechanism with such a reaction at a
vanishing rate runs the dense kernel with the same result.

Tolerance as tests/test_gpu_adjoint_lists.py: the same reactions' terms, each a product of fewer than 30 rounded
factors, in another order.
"""
import shutil

import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu

NONE = " ".join(f"{n}/0.0/" for n in ("H", "H2", "H2O", "HO2", "O", "O2", "OH", "N2"))
REACTIONS = f"""REACTIONS
H+O2=>O+OH       3.55E+15    -0.40   1.66E+04
O+H2=H+OH        5.08E+04     2.70   6.29E+03
  REV/ 2.20E+04 2.60 4.40E+03 /
H2+M=H+H+M       4.58E+19    -1.40   2.00E+04
  REV/ 1.10E+18 -1.00 1.00E+03 /
  {NONE}
O+O+M=O2+M       6.16E+15    -0.50   0.00
  REV/ 3.00E+15 -0.30 2.00E+04 /
  H2/2.5/ H2O/12.0/
"""


@pytest.mark.parametrize("peroxide", [0.0, 1e-3], ids=["no_collider", "collider"])
def test_rev_coefficients(built, tmp_path, peroxide):
    """H2 + M has one collider, H2O2."""
    import ostc

    text = (oc.CHEM_FIXTURE / "H2_mech.inp").read_text()
    head = text[: text.index("REACTIONS")]
    out = []
    for extra in ("", "H+H+H+H+O2=>H2+H2+O+O   1.00E-200   0.00   0.00E+00\n"):
        mech = tmp_path / f"mech{len(out)}"
        shutil.copytree(oc.CHEM_FIXTURE, mech)
        (mech / "H2_mech.inp").write_text(head + REACTIONS + extra + "END\n")
        case = oc.reacting_mixing_layer_3d(18, 14, 10, chem_dir=mech)
        tb = case.mixture["tables"]
        y = np.abs(case.sv + 0.02 * np.random.default_rng(5).random(case.sv.shape))
        y[tb.names.index("H2O2")] *= peroxide
        case.sv = y / y.sum(axis=0)
        mw = 1 / np.einsum("l...,l->...", case.sv, 1 / tb.mw)
        case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
        s = ostc.Solver(str(oc.write_case(case, tmp_path / f"case{len(out)}")))
        s.set_state(case.bv, sv=case.sv)
        w = np.random.default_rng(6).standard_normal(s.get_state()[0].shape)
        out.append(s.rhs_vjp(w, 4))
        s.close()
    listed, dense = out
    l = 5 + tb.names.index("H2O2")
    assert np.all(np.isfinite(listed)) and np.any(dense[l])
    for l in range(listed.shape[0]):
        assert np.max(np.abs(listed[l] - dense[l])) <= 1e-11 * np.max(np.abs(dense[l])), l
