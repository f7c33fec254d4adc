"""Mixed precision: quartets whose Schwarz bound is below tau use the FP32 kernel form (FP64
screening and accumulation).  Errors are stated against the plain-FP64 build
and, through the relinked reference program (which builds with difference densities each
SCF iteration), against the reference's FP64 SCF energy: the bar is 1e-6 Eh."""
import json
import os

import numpy as np
import pytest

from conftest import golden, golden_basis, load_sqb200, results_path
from test_dropin_scf import SQREF_GPU, _run

TAUS = [1e-3, 1e-4, 1e-5, 1e-6]


def _engine(g):
    sqb = load_sqb200()
    return sqb.JKEngine(golden_basis(g), schwarz=g["schwarz"])


@pytest.mark.gpu
def test_tau_zero_is_plain_fp64():
    g = golden("h2co_631gs")
    eng = _engine(g)
    J0, K0, _ = eng.build(g["PA"], scf_cutoff=1e-10)
    eng.set_precision(0.0)
    J1, K1, _ = eng.build(g["PA"], scf_cutoff=1e-10)
    # FP64 atomics accumulate in a varying order: equal up to rounding, not bit for bit
    assert np.abs(J0 - J1).max() < 1e-12 and np.abs(K0 - K1).max() < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["benzene_631gs", "oh_321g_uhf"])
def test_mixed_error_shrinks_with_tau(case, monkeypatch):
    # every class with quartets below tau takes its FP32 form, however few its FP32 work items
    # (by default a class with few of them stays in FP64)
    monkeypatch.setenv("SQB200_F32_MIN_ITEMS", "0")
    g = golden(case)
    restricted = bool(g["restricted"])
    eng = _engine(g)
    PB = None if restricted else g["PB"]
    J0, K0, KB0 = eng.build(g["PA"], PB, restricted=restricted, scf_cutoff=1e-10)
    q0 = eng.stats()["quartets"]
    errs = []
    for tau in TAUS:
        eng.set_precision(tau)
        J, K, KB = eng.build(g["PA"], PB, restricted=restricted, scf_cutoff=1e-10)
        assert eng.stats()["quartets"] == q0          # same screening, only precision moves
        errs.append(max(np.abs(J - J0).max(), np.abs(K - K0).max(), np.abs(KB - KB0).max()))
    with open(results_path("mixed_jk_err_%s.json" % case), "w") as f:
        json.dump(dict(zip(map(str, TAUS), errs)), f)
    assert errs[0] < 1e-4
    # monotone above FP64 rounding (1e-13 here); a molecule whose FP32 share is negligible at
    # every tau sits at rounding level throughout
    assert errs[-1] <= max(errs[0], 1e-13)
    assert errs[-1] < 1e-8
    if case == "benzene_631gs":
        assert errs[0] > 1e-12          # the FP32 forms did run


@pytest.mark.gpu
@pytest.mark.skipif(not os.path.exists(SQREF_GPU), reason="oracle/_ref/sqref_b200 not built")
@pytest.mark.parametrize("tau", [1e-4, 1e-6])
def test_mixed_scf_energy_within_1e6(tau, monkeypatch):
    """Whole SCF through the reference's own uhf() (1STEP), GPU Fock build in mixed precision."""
    g = golden("benzene_631gs")
    monkeypatch.setenv("SQB200_FP32_BELOW", str(tau))
    e = _run(SQREF_GPU, g["atoms"], str(g["basis"]), ["-SCFACC=1STEP", "-SCFCONV=1e-8"])
    err = abs(e - float(g["energy"]))
    with open(results_path("mixed_scf_err_%g.json" % tau), "w") as f:
        json.dump({"tau": tau, "energy": e, "reference": float(g["energy"]), "abs_err": err}, f)
    assert err <= 1e-6, err


# (heavy atoms, tau): the classes that launch their FP32 form for a 6-31G* organic
F32_CLASSES = {(5, 1e-5): set(), (9, 1e-5): {"LS|SS"}, (9, 1e-3): {"LS|SS"},
               (11, 1e-5): {"DS|LS", "DS|SS", "LS|LS", "LS|SS", "SS|SS"},
               (13, 1e-5): {"DL|LS", "DL|SS", "DS|LS", "DS|SS", "LL|LS", "LL|SS", "LS|LS", "LS|SS", "SS|SS"}}


@pytest.mark.gpu
@pytest.mark.parametrize("heavy,tau", sorted(F32_CLASSES))
def test_fp32_classes_do_not_depend_on_the_item_shape(heavy, tau):
    """A class runs quartets in FP32 from 2400 FP32 items of 64 threads on, counted in items of one
    fixed shape: the items that a build is cut into get narrower and more with smaller builds,
    which must not move quartets to FP32."""
    sqb = load_sqb200()
    atoms = sqb.molecules.to_bohr(sqb.molecules.random_organic(np.random.default_rng([3, heavy]), heavy))
    b = sqb.basis.build_basis(atoms, "6-31g*")
    eng = sqb.JKEngine(b)
    eng.set_precision(tau)
    eng.profile(True)
    eng.build(np.eye(b.nbf), scf_cutoff=1e-10)
    got = {r["class"] for r in eng.profile_read() if r["class"].endswith("f32")}
    eng.close()
    assert got == {c + " f32" for c in F32_CLASSES[heavy, tau]}
