"""The point-implicit chemistry beyond 9 species: 13 species (two blocks an SM over the reaction lists), and 14 and 16
on a block of cells below and above one wave (over the lists, and over every species), against the CPU oracle.  The
species after the ninth are inert copies of N2 under other names.

Tolerance 1e-12 relative per conserved variable after a step, as the mode's other comparisons.
"""
import shutil

import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu


def mechanism(directory, n):
    """The 9-species mechanism with n - 9 copies of N2: the therm.dat entry's four lines and the tran.dat line."""
    shutil.copytree(oc.CHEM_FIXTURE, directory)
    names = [f"NX{chr(65 + q)}" for q in range(n - 9)]
    mech = (directory / "H2_mech.inp").read_text().split("\n")
    at = next(q for q, line in enumerate(mech) if line.split()[-1:] == ["N2"] and "H2O2" in line)
    mech.insert(at + 1, " " + " ".join(names))
    (directory / "H2_mech.inp").write_text("\n".join(mech))
    therm = (directory / "therm.dat").read_text().split("\n")
    at = next(q for q, line in enumerate(therm) if line.startswith("N2 "))
    entry = therm[at:at + 4]
    tran = (directory / "tran.dat").read_text().rstrip("\n").split("\n")
    line = next(t for t in tran if t.startswith("N2 "))
    for name in names:
        therm[at:at] = [name.ljust(18) + entry[0][18:]] + entry[1:]
        tran.append(name.ljust(18) + line[18:])
    (directory / "therm.dat").write_text("\n".join(therm))
    (directory / "tran.dat").write_text("\n".join(tran) + "\n")
    return directory


@pytest.mark.parametrize("n", [13, 14, 16])
@pytest.mark.parametrize("dims", [(18, 14, 10), (24, 21, 20)], ids=["one_wave", "more"])
def test_point_implicit(built, tmp_path, n, dims):
    import ostc
    from oracle import Oracle

    case = oc.reacting_mixing_layer_3d(*dims, chem_dir=mechanism(tmp_path / "mech", n))
    rng = np.random.default_rng(4)
    assert case.sv.shape[0] == n
    case.sv = case.sv * (1 + 0.05 * rng.random(case.sv.shape)) + 1e-4 * rng.random(case.sv.shape)
    case.sv /= case.sv.sum(axis=0)
    mw = 1 / np.einsum("l...,l->...", case.sv, 1 / case.mixture["tables"].mw)
    case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
    s = ostc.Solver(str(oc.write_case(case, tmp_path / "case")))
    s.set_chem_mode(1)
    s.set_state(case.bv, sv=case.sv)
    s.step(1)
    cv, _ = s.get_state()
    s.close()
    o = Oracle(case, 1)
    o.set_state(case.bv, case.sv)
    o.step(1)
    err = oc.relative_errors(cv, o.get_state()[0])
    assert max(max(e) for e in err) <= 1e-12, err
