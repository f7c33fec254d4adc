"""Quartets split over threads (si x sj of the bra and ket primitives, picked per pair of contraction
lengths) against the oracle: contractions of 1, 2, 3, 5, 6, 7 and 11 primitives, so that the loops
have every kind of remainder, in shells of each type, on a molecule small enough that every
long quartet is split.  Every FP64 form; the quartet and primitive-quartet counts are exact.
J/K tolerance 1e-10 max-abs, as every FP64 build against the oracle."""
import numpy as np
import pytest

from conftest import load_oracle, load_sqb200

FUNCS = {"S": [(0, 0, 0)], "L": [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)], "P": [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
         "D": [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)],
         "F": [(3, 0, 0), (0, 3, 0), (0, 0, 3), (2, 1, 0), (1, 2, 0), (2, 0, 1), (1, 0, 2), (0, 2, 1), (0, 1, 2), (1, 1, 1)]}


def _basis(sqb, shells, seed):
    """shells: [(type, centre index, primitives)]; exponents spread over 0.2 .. 200."""
    rng = np.random.default_rng(seed)
    centres = np.array([[0.0, 0.0, 0.1], [0.0, 1.9, -0.4], [1.3, -0.7, 1.1]])
    nprim, lmn, xyz, exps, coefs, norms = [], [], [], [], [], []
    for kind, at, n in shells:
        ex = np.sort(0.25 * (3.0 ** np.arange(n)) * rng.uniform(0.8, 1.2, n))[::-1] if n < 8 else np.geomspace(200.0, 0.2, n)
        w = rng.uniform(0.2, 1.0, (n, 2)) / np.sqrt(n)
        for l in FUNCS[kind]:
            nprim.append(n)
            lmn.append(l)
            xyz.append(centres[at])
            for k in range(n):
                exps.append(ex[k])
                coefs.append(w[k, 0 if sum(l) == 0 else 1])
                norms.append(sqb.basis.prim_norm(ex[k], *l))
    return sqb.basis.Basis(nprim, lmn, xyz, exps, coefs, norms)


SETS = {
    "s": [("S", 0, 7), ("S", 1, 11), ("S", 2, 5), ("S", 0, 1), ("S", 1, 2)],
    "sp": [("S", 0, 6), ("L", 0, 3), ("L", 1, 5), ("L", 2, 1), ("S", 2, 7)],
    "p": [("S", 0, 5), ("P", 0, 4), ("P", 1, 1), ("P", 2, 7), ("D", 0, 2)],
    "d": [("D", 0, 3), ("L", 1, 2), ("D", 2, 1), ("P", 1, 3), ("S", 2, 6)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SETS))
@pytest.mark.parametrize("restricted", [True, False])
def test_split_quartets_match_oracle(name, restricted):
    sqb, orc = load_sqb200(), load_oracle()
    b = _basis(sqb, SETS[name], 3)
    rng = np.random.default_rng(4)
    P = [0.3 * (A + A.T) for A in rng.standard_normal((2, b.nbf, b.nbf))]
    PA, PB = P[0], P[0] if restricted else P[1]
    sch = orc.schwarz(b)
    J0, KA0, KB0, st = orc.jk_build(b, sch, PA, PB, restricted=restricted, scf_cutoff=1e-10)
    eng = sqb.JKEngine(b, schwarz=sch)
    try:
        for form in range(3):
            eng.set_tiles(np.full(256, form, np.int32))
            J, KA, KB = eng.build(PA, PB, restricted=restricted, scf_cutoff=1e-10)
            s = eng.stats()
            assert (s["quartets"], s["prim_quartets"]) == (st[1], st[2]), form
            scale = max(1.0, np.abs(J0).max())
            assert max(np.abs(J - J0).max(), np.abs(KA - KA0).max()) <= 1e-10 * scale, form
            if not restricted:
                assert np.abs(KB - KB0).max() <= 1e-10 * scale, form
    finally:
        eng.close()
