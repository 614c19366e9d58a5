"""The sweeps and the viscous kernel of blocks that are not rectilinear (all three metric components), on a wavy grid:
every tile shape of the AWENO y / z sweeps, pinned, in both precisions, and the mixed precision of every family.

Tolerances: two shapes form the same face fluxes by the same expressions, 1e-13 as tests/test_gpu_sweep_variants.py;
mixed precision against the FP64 oracle over ten steps, 1e-5 in L2 as tests/test_gpu_schemes.py.
"""
import numpy as np
import pytest

import ostc
import ostc_cases as oc
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _wavy(dims, scheme):
    mx, my, mz = dims
    kw = dict(mx=mx, my=my, ybc="outflow", reconstruction=scheme[0], inviscid_scheme=scheme[1])
    case = oc.mixing_layer_2d(**kw) if mz == 1 else oc.mixing_layer_3d(mz=mz, **kw)
    k, j, i = np.meshgrid(np.arange(mz), np.arange(my), np.arange(mx), indexing="ij")
    h = case.x[0, 0, 1] - case.x[0, 0, 0]
    case.x = case.x + 0.15 * h * np.sin(0.45 * j + 0.3 + 0.5 * k)
    case.y = case.y + 0.15 * h * np.sin(0.4 * i + 0.2 + 0.35 * k)
    if mz > 1:
        case.z = case.z + 0.15 * h * np.sin(0.35 * i + 0.5 * j)
    return case


def _run(d, case, prec, steps, pins=()):
    s = ostc.Solver(str(d))
    s.set_precision(prec)
    for dir_, v in pins:
        s.set_sweep_variant(dir_, v, precision=prec)
    s.set_state(case.bv)
    s.step(steps)
    cv, _ = s.get_state()
    assert s.error_flags() == 0
    s.close()
    return cv


@pytest.mark.parametrize("scheme", [(5, 4), (4, 3)], ids=["weno7_hllc", "weno5_ausm"])
@pytest.mark.parametrize("prec", [ostc.PREC_FP64, ostc.PREC_MIXED], ids=["fp64", "mixed"])
def test_tile_shapes_agree(built, tmp_path, scheme, prec):
    case = _wavy((70, 36, 20), scheme)
    d = oc.write_case(case, tmp_path / "c")
    assert ostc.probe_case(str(d))["n_rectilinear"] == 0
    base = _run(d, case, prec, 3, [(1, 0), (2, 0)])
    for v in range(1, 4):
        cv = _run(d, case, prec, 3, [(1, v), (2, v)])
        err = oc.relative_errors(cv, base)
        assert all(m < 1e-13 and l2 < 1e-13 for m, l2 in err), (v, err)
    if prec == ostc.PREC_FP64:
        o = Oracle(case)
        o.set_state(case.bv)
        o.step(3)
        err = oc.relative_errors(base, o.get_state()[0])
        assert all(m < 1e-12 and l2 < 1e-12 for m, l2 in err), err


@pytest.mark.parametrize("scheme", [(5, 4), (4, 3), (5, 1), (2, 4), (3, 3), (1, 1), (2, 2)],
                         ids=["weno7_hllc", "weno5_ausm", "weno7_lf", "muscl_hllc", "nnd_ausm", "first_lf", "muscl_roe"])
@pytest.mark.parametrize("dims", [(34, 25, 1), (33, 18, 14)], ids=["2d", "3d"])
def test_mixed_precision(built, tmp_path, scheme, dims):
    case = _wavy(dims, scheme)
    d = oc.write_case(case, tmp_path / "c")
    assert ostc.probe_case(str(d))["n_rectilinear"] == 0
    cv = _run(d, case, ostc.PREC_MIXED, 10)
    o = Oracle(case)
    o.set_state(case.bv)
    o.step(10)
    err = oc.relative_errors(cv, o.get_state()[0])
    assert all(l2 < 1e-5 for _, l2 in err), err
