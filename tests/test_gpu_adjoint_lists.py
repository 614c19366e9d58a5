"""The adjoint of the chemical source over the reaction lists (derivatives of the rates written out) against
the dense one (every derivative by dual numbers).  A reaction with five molecules on a side does not fit the
lists, so a mechanism with such a reaction at a vanishing rate runs the dense kernel with the same result.

Tolerance: the two sum the same ~20 reactions' terms, each a product of fewer than 30 rounded factors, in
another order; 1e-11 of each variable's largest entry leaves room for their cancellation near equilibrium
(the Gibbs energies' sum is ~30 and enters an exponential).
"""
import shutil

import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(18, 14, 10), (33, 16, 1)], ids=["3d", "2d"])
@pytest.mark.parametrize("hot", [False, True], ids=["layer", "hot"])
def test_listed_source_matches_dense(built, tmp_path, dims, hot):
    import ostc

    mech = tmp_path / "mech"
    shutil.copytree(oc.CHEM_FIXTURE, mech)
    text = (mech / "H2_mech.inp").read_text().rstrip()
    assert text.endswith("END")
    (mech / "H2_mech.inp").write_text(text[:-3] + "H+H+H+H+O2=H2+H2+O+O   1.00E-200   0.00   0.00E+00\nEND\n")
    out = []
    for chem in (oc.CHEM_FIXTURE, mech):
        case = oc.reacting_mixing_layer_3d(*dims, chem_dir=chem)
        rng = np.random.default_rng(5)
        y = np.abs(case.sv + 0.02 * rng.random(case.sv.shape))
        case.sv = y / y.sum(axis=0)
        if hot:
            case.bv[5] = 2.2 * case.bv[5]
        mw = 1 / np.einsum("l...,l->...", case.sv, 1 / case.mixture["tables"].mw)
        case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
        s = ostc.Solver(str(oc.write_case(case, tmp_path / f"case{len(out)}")))
        s.set_state(case.bv, sv=case.sv)
        cv0, _ = s.get_state()
        out.append(s.rhs_vjp(np.random.default_rng(6).standard_normal(cv0.shape), 4))
        s.close()
    listed, dense = out
    assert np.all(np.isfinite(listed)) and np.any(listed)
    for l in range(listed.shape[0]):
        assert np.max(np.abs(listed[l] - dense[l])) <= 1e-11 * np.max(np.abs(dense[l])), l
