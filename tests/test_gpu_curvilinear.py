"""Wavy (non-orthogonal) grids and tile edges against the CPU oracle: the general metric branch of the
mixture viscous faces (cross differences of T and the mass fractions, which a rectilinear grid skips),
the flux-split and AWENO sweeps with all three metric components, extents at the edges of the sweeps'
tiles, mass fractions far below rounding (the flux-split weights' epsilon) and reactions with
more species than the reaction lists hold (the dense chemistry).

Tolerances: 1e-12 relative per conserved variable over two RK3 steps as the other trajectory tests; the
adjoint as tests/test_gpu_adjoint.py.
"""
import shutil

import numpy as np
import pytest

import ostc_cases as oc

pytestmark = pytest.mark.gpu


def _wavy(case, amp=0.15):
    """The case on a smoothly distorted grid (displacements of amp grid spacings, every direction)."""
    k, j, i = np.meshgrid(*(np.arange(n) for n in (case.mz, case.my, case.mx)), indexing="ij")
    h = case.x[0, 0, 1] - case.x[0, 0, 0]
    fz = 0.5 * k if case.mz > 1 else 0.0
    case.x = case.x + amp * h * np.sin(0.45 * j + 0.3 + fz)
    case.y = case.y + amp * h * np.sin(0.4 * i + 0.2 + 0.7 * fz)
    if case.mz > 1:
        case.z = case.z + amp * h * np.sin(0.35 * i + 0.5 * j)
    return case


def _check(case, tmp_path, steps=2, tol=1e-12):
    import ostc
    from oracle import Oracle

    s = ostc.Solver(str(oc.write_case(case, tmp_path / "case")))
    s.set_state(case.bv, sv=case.sv)
    s.step(steps)
    cv, _ = s.get_state()
    s.close()
    o = Oracle(case)
    o.set_state(case.bv) if case.sv is None else o.set_state(case.bv, case.sv)
    o.step(steps)
    co = o.get_state()[0]
    assert np.all(np.isfinite(co))
    err = oc.relative_errors(cv, co)
    assert max(max(e) for e in err) <= tol, err


@pytest.mark.parametrize("kw", [dict(reconstruction=5, inviscid_scheme=4), dict(reconstruction=4, inviscid_scheme=3)],
                         ids=["weno7_hllc", "weno5_ausm"])
@pytest.mark.parametrize("mz", [1, 14])
def test_air_wavy(built, tmp_path, kw, mz):
    if mz == 1:
        case = oc.mixing_layer_2d(mx=34, my=25, ybc="outflow", **kw)
    else:
        case = oc.mixing_layer_3d(mx=33, my=18, mz=mz, ybc="outflow", **kw)
    _check(_wavy(case), tmp_path)


@pytest.mark.parametrize("mz", [1, 12])
def test_mixture_wavy(built, tmp_path, mz):
    _check(_wavy(oc.reacting_mixing_layer_3d(mx=21, my=18, mz=mz)), tmp_path)


@pytest.mark.parametrize("dims", [(127, 15, 16), (128, 16, 17), (129, 31, 9), (9, 17, 46)])
def test_mixture_tile_edges(built, tmp_path, dims):
    _check(oc.reacting_mixing_layer_3d(*dims), tmp_path, steps=1)


@pytest.mark.parametrize("scale", [1e-12, 1e-60])
def test_mixture_vanishing_species(built, tmp_path, scale):
    """Radicals scaled towards zero: their indicators fall towards epsilon (1e-12) and far below it (1e-60).  The
    four weights still share a division here; tests/test_gpu_fvs_range.py leaves that form at both ends."""
    case = oc.reacting_mixing_layer_3d(mx=20, my=18, mz=10, finite_rate=False)
    names = case.mixture["tables"].names
    for n in ("OH", "O", "H", "HO2", "H2O2"):
        l = names.index(n)
        kept = case.sv[l] * scale
        case.sv[names.index("N2")] += case.sv[l] - kept
        case.sv[l] = kept
    mw = 1 / np.einsum("l...,l->...", case.sv, 1 / case.mixture["tables"].mw)
    case.bv[0] = case.bv[4] * mw / (oc.R_U * case.bv[5])
    _check(case, tmp_path)


@pytest.mark.parametrize("chem_mode", [0, 1])
def test_dense_chemistry(built, tmp_path, chem_mode):
    """A reaction with five molecules on a side does not fit the reaction lists: every reaction then runs
    over all species, explicitly and in the point-implicit mode."""
    import ostc
    from oracle import Oracle

    mech = tmp_path / "mech"
    shutil.copytree(oc.CHEM_FIXTURE, mech)
    text = (mech / "H2_mech.inp").read_text().rstrip()
    assert text.endswith("END")
    (mech / "H2_mech.inp").write_text(text[:-3] + "H+H+H+H+O2=H2+H2+O+O   1.00E+10   0.00   1.00E+04\nEND\n")
    case = oc.reacting_mixing_layer_3d(mx=16, my=14, mz=10, chem_dir=mech)
    s = ostc.Solver(str(oc.write_case(case, tmp_path / "case")))
    s.set_chem_mode(chem_mode)
    s.set_state(case.bv, sv=case.sv)
    s.step(1)
    cv, _ = s.get_state()
    o = Oracle(case, chem_mode)
    o.set_state(case.bv, case.sv)
    o.step(1)
    err = oc.relative_errors(cv, o.get_state()[0])
    assert max(max(e) for e in err) <= 1e-12, err


@pytest.mark.parametrize("kw", [dict(reconstruction=5, inviscid_scheme=4), dict(reconstruction=4, inviscid_scheme=3),
                                dict(reconstruction=5, inviscid_scheme=1)], ids=["weno7_hllc", "weno5_ausm", "weno7_lf"])
@pytest.mark.parametrize("mz", [1, 10])
def test_air_vjp_wavy(built, tmp_path, kw, mz):
    """<w, J v> = <J^T w, v> on a wavy grid, J v from Richardson central differences, a state with 5 % noise
    on every primitive variable (the bar and step of tests/test_gpu_adjoint.py for air)."""
    import ostc

    if mz == 1:
        case = oc.mixing_layer_2d(mx=24, my=18, ybc="outflow", **kw)
    else:
        case = oc.mixing_layer_3d(mx=20, my=14, mz=mz, ybc="outflow", **kw)
    case = _wavy(case)
    rng = np.random.default_rng(11)
    c0 = np.sqrt(oc.GAMMA * oc.R_AIR * 300.0)
    for l in (4, 5):
        case.bv[l] = case.bv[l] * (1 + 0.05 * rng.standard_normal(case.bv[l].shape))
    for l in (1, 2, 3)[: 3 if mz > 1 else 2]:
        case.bv[l] = case.bv[l] + 0.1 * c0 * rng.standard_normal(case.bv[l].shape)
    case.bv[0] = case.bv[4] / (oc.R_AIR * case.bv[5])
    s = ostc.Solver(str(oc.write_case(case, tmp_path / "case")))
    s.set_state(case.bv)
    cv0, _ = s.get_state()
    w = rng.standard_normal(cv0.shape)
    g = s.rhs_vjp(w)
    for _ in range(4):
        v = rng.standard_normal(cv0.shape) * np.abs(cv0)
        best = np.inf
        for eps in (1e-7, 1e-8):
            d = []
            for h in (2 * eps, eps):
                s.set_conservative(cv0 + h * v)
                rp = s.rhs()
                s.set_conservative(cv0 - h * v)
                rm = s.rhs()
                d.append((rp - rm) / (2 * h))
            jv = (4 * d[1] - d[0]) / 3
            lhs, rhs = float(np.sum(w * jv)), float(np.sum(g * v))
            best = min(best, abs(lhs - rhs) / (1e-6 * abs(lhs) + 1e-9 * float(np.sum(np.abs(w * jv)))))
        s.set_conservative(cv0)
        assert best <= 1.0, best
