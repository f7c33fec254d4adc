"""The generated class kernels of the two-electron gradient against the run-time kernel (one thread
per shell quartet): a basis with every shell type takes the class kernels; the same basis with
the functions of one d shell in another order is a layout outside the classes and takes the
run-time kernel.  Both apply the same screens to the same quartets, so they differ by rounding:
tolerance 1e-11 of the largest component.  Restricted and unrestricted densities (the gradient's
spin term), screened and with every quartet kept; contraction lengths with remainders, shells
sharing a centre (same-shell and same-pair degeneracies)."""
import numpy as np
import pytest

from conftest import load_sqb200
from test_split_gpu import _basis

SHELLS = [("S", 0, 5), ("L", 0, 3), ("P", 1, 2), ("D", 2, 2), ("D", 0, 1), ("L", 1, 1), ("S", 2, 1), ("P", 2, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("shells", [SHELLS, SHELLS[:1] + SHELLS[3:5], [("S", 0, 7), ("S", 1, 1), ("S", 2, 2), ("D", 1, 1)]],
                         ids=["all", "s_d", "s"])
@pytest.mark.parametrize("screen", ["1e-10", "0"])
@pytest.mark.parametrize("restricted", [True, False])
def test_class_gradient_matches_run_time_kernel(shells, screen, restricted, monkeypatch):
    monkeypatch.setenv("SQB200_GRAD_SCREEN", screen)
    sqb = load_sqb200()
    b = _basis(sqb, shells, 7)
    n = b.nbf
    rng = np.random.default_rng(8)
    PA, PB, W = (0.2 * (A + A.T) for A in rng.standard_normal((3, n, n)))
    PB = PA if restricted else PB
    # the permuted layout: the first and fourth functions of the first d shell (xx, xy) swapped
    d0 = next(i for i in range(n) if b.lmn[i].sum() == 2)
    perm = np.arange(n)
    perm[[d0, d0 + 3]] = perm[[d0 + 3, d0]]
    ex = [b.exps[o:o + k] for o, k in zip(b.offset, b.nprim)]
    co = [b.coefs[o:o + k] for o, k in zip(b.offset, b.nprim)]
    no = [b.norms[o:o + k] for o, k in zip(b.offset, b.nprim)]
    cat = lambda v: np.concatenate([v[i] for i in perm])
    b2 = sqb.basis.Basis(b.nprim[perm], b.lmn[perm], b.center[perm], cat(ex), cat(co), cat(no))
    Z = np.array([6.0, 8.0, 1.0])
    xyz = np.array([[0.0, 0.0, 0.1], [0.0, 1.9, -0.4], [1.3, -0.7, 1.1]])
    G = []
    for basis, p in ((b, np.arange(n)), (b2, perm)):
        eng = sqb.JKEngine(basis)
        ix = np.ix_(p, p)
        G.append(eng.gradient(Z, xyz, PA[ix], PB[ix], W[ix], terms=8))
        eng.close()
    assert np.abs(G[0]).max() > 0
    assert np.abs(G[0] - G[1]).max() <= 1e-11 * np.abs(G[1]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_class_gradient_of_a_density_that_is_not_finite_is_not_finite(bad):
    sqb = load_sqb200()
    b = _basis(sqb, SHELLS, 7)
    n = b.nbf
    P = 0.2 * np.ones((n, n))
    P[3, 2] = P[2, 3] = bad
    eng = sqb.JKEngine(b)
    G = eng.gradient(np.array([6.0, 8.0, 1.0]), np.array([[0.0, 0.0, 0.1], [0.0, 1.9, -0.4], [1.3, -0.7, 1.1]]), P, P, P,
                     terms=8)
    eng.close()
    assert not np.isfinite(G).all()


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_class_gradient_keeps_an_infinite_density_factor_of_either_sign(sign):
    """Two H2 molecules 40 bohr apart; one density element of the first is infinite, the second
    molecule's elements have one sign.  The only quartets that join the two are Coulomb ones, so
    every density factor that reaches the second molecule is an infinity of that sign."""
    sqb = load_sqb200()
    xyz = np.array([[0.0, 0.0, z] for z in (0.0, 1.4, 40.0, 41.4)])
    b = sqb.basis.build_basis([(1, *r) for r in xyz], "sto-3g")
    P = np.zeros((2, 4, 4))
    P[0, 0, 1] = P[0, 1, 0] = np.inf
    P[0, 2:, 2:], P[1, 2:, 2:] = 0.3 * sign, 0.1 * sign
    eng = sqb.JKEngine(b)
    G = eng.gradient(np.ones(4), xyz, P[0], P[1], P[1], terms=8)
    eng.close()
    assert not np.isfinite(G[2:]).all(axis=1).any()


@pytest.mark.gpu
def test_gradients_of_one_context_from_several_threads_beside_its_builds():
    """Two threads ask one context for gradients of densities of their own (one with a quarter of the
    pairs screened out, so that the calls' sizes differ) while a third builds with it, past the
    number of builds that makes a replay graph; each against its own call alone."""
    import threading

    import torch
    sqb = load_sqb200()
    atoms = sqb.molecules.to_bohr(sqb.molecules.random_organic(np.random.default_rng(3), 4))
    b = sqb.basis.build_basis(atoms, "6-31g*")
    n = b.nbf
    Z = np.array([a[0] for a in atoms], dtype=np.float64)
    xyz = np.array([a[1:] for a in atoms])
    rng = np.random.default_rng(4)
    P = [0.1 * (A + A.T) for A in rng.standard_normal((3, n, n))]
    P[1][:n // 2, :n // 2] = 0.0
    eng = sqb.JKEngine(b)
    ref = [eng.gradient(Z, xyz, p, p, P[2]) for p in P[:2]]
    st = torch.cuda.Stream()
    d = torch.tensor(P[2], device="cuda")
    out = [torch.empty((n, n), dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    eng.build_tensors(d, d, *out, scf_cutoff=1e-10, stream=st)
    st.synchronize()
    J, K = out[0].clone(), out[1].clone()
    torch.cuda.synchronize()
    bad = []

    def gradients(k):
        for _ in range(25):
            err = np.abs(eng.gradient(Z, xyz, P[k], P[k], P[2]) - ref[k]).max()
            if not err <= 1e-11 * np.abs(ref[k]).max():
                bad.append(("gradient", k, err))

    def builds():
        for k in range(60):
            eng.build_tensors(d, d, *out, scf_cutoff=1e-10, stream=st)
            if k % 10 == 9:
                st.synchronize()
                err = max((out[0] - J).abs().max().item(), (out[1] - K).abs().max().item())
                if not err <= 1e-11 * J.abs().max().item():
                    bad.append(("build", k, err))

    ts = [threading.Thread(target=gradients, args=(k,)) for k in (0, 1)] + [threading.Thread(target=builds)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
    assert eng.replays() > 0
    eng.close()
