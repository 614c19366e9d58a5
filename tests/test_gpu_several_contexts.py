"""Contexts of several species counts side by side: a kernel's shared-memory limit is the process's, so a context
created later, with fewer species or none, must not lower it under one that is alive.  A 9-species context steps
(explicit and point-implicit chemistry) and takes a VJP after an air and a 5-species context were created, and the
5-species one after it; each gives what it gives alone.

Tolerance: the same kernels on the same inputs; only the adds of a VJP's node planes may come in another order, a
dozen terms an entry, so 1e-12 of each variable's largest entry there and equality for the states.
"""
import shutil

import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu


def _five_species(tmp_path):
    mech = tmp_path / "mech5"
    shutil.copytree(oc.CHEM_FIXTURE, mech)
    text = (mech / "H2_mech.inp").read_text()
    head = text[: text.index("SPECIES")]
    (mech / "H2_mech.inp").write_text(head + "SPECIES\nH2 H2O O2 OH N2\nEND\nREACTIONS\n"
                                      "H2+O2=OH+OH 1.70E+13 0.00 4.78E+04\nEND\n")
    return oc.reacting_mixing_layer_3d(18, 14, 10, chem_dir=mech, fuel={"H2": 0.05, "N2": 0.95},
                                       oxidiser={"O2": 0.2, "H2O": 0.1, "OH": 1e-3, "N2": 0.699})


def _work(s, case):
    """States after an explicit and an implicit step, and a VJP."""
    out = []
    for mode in (0, 1):
        s.set_chem_mode(mode)
        s.set_state(case.bv, sv=case.sv)
        s.step(1)
        out.append(s.get_state()[0])
    s.set_chem_mode(0)
    s.set_state(case.bv, sv=case.sv)
    w = np.random.default_rng(2).standard_normal(out[0].shape)
    return out, s.rhs_vjp(w)


def test_later_context_keeps_the_limits(built, tmp_path):
    import ostc

    nine = oc.reacting_mixing_layer_3d(18, 14, 10)
    five = _five_species(tmp_path)
    air = oc.mixing_layer_3d(18, 14, 10, ybc="outflow")
    dirs = {}
    alone = {}
    for name, case in (("nine", nine), ("five", five)):
        dirs[name] = str(oc.write_case(case, tmp_path / name))
        s = ostc.Solver(dirs[name])
        alone[name] = _work(s, case)
        s.close()
    s9 = ostc.Solver(dirs["nine"])
    s5 = ostc.Solver(dirs["five"])
    s0 = ostc.Solver(str(oc.write_case(air, tmp_path / "air")))
    s0.set_state(air.bv)
    for name, s, case in (("nine", s9, nine), ("five", s5, five)):
        states, vjp = _work(s, case)
        for a, b in zip(states, alone[name][0]):
            assert np.array_equal(a, b)
        for a, b in zip(vjp, alone[name][1]):
            assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    s0.step(1)
    assert np.all(np.isfinite(s0.get_state()[0]))
    for s in (s9, s5, s0):
        s.close()
