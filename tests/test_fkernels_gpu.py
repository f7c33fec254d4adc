"""The f-shell kernels (gen_fshell_kernels.py) against the oracle: every class of the bra's second shell
(s, sp, p, d, f), kets of 1 to 100 function pairs (so that quartets fill a warp several at a time,
once, and in chunks), contraction lengths with remainders, shells sharing a centre (coinciding
shells and pairs), restricted and unrestricted.  Counts are exact; J/K to 1e-10 of the largest
element, as every FP64 build against the oracle."""
import numpy as np
import pytest

from conftest import load_oracle, load_sqb200
from test_split_gpu import _basis

SETS = {
    "f_s": [("F", 0, 2), ("S", 1, 5), ("S", 2, 1), ("F", 1, 1)],
    "f_sp": [("F", 0, 1), ("L", 1, 3), ("L", 2, 1), ("S", 0, 6)],
    "f_pd": [("F", 0, 1), ("P", 1, 2), ("D", 2, 2), ("P", 0, 1), ("S", 1, 3)],
    "f_ld": [("F", 2, 2), ("L", 1, 2), ("D", 0, 1)],
    "f_f": [("F", 0, 1), ("F", 0, 3), ("F", 2, 1), ("S", 1, 2)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SETS))
@pytest.mark.parametrize("restricted", [True, False])
def test_f_kernels_match_oracle(name, restricted):
    sqb, orc = load_sqb200(), load_oracle()
    b = _basis(sqb, SETS[name], 11)
    rng = np.random.default_rng(12)
    P = [0.3 * (A + A.T) for A in rng.standard_normal((2, b.nbf, b.nbf))]
    PA, PB = P[0], P[0] if restricted else P[1]
    sch = orc.schwarz(b)
    J0, KA0, KB0, st = orc.jk_build(b, sch, PA, PB, restricted=restricted, scf_cutoff=1e-10)
    eng = sqb.JKEngine(b, schwarz=sch)
    try:
        for _ in range(2):
            J, KA, KB = eng.build(PA, PB, restricted=restricted, scf_cutoff=1e-10)
            s = eng.stats()
            assert (s["quartets"], s["prim_quartets"]) == (st[1], st[2])
            scale = max(1.0, np.abs(J0).max())
            assert max(np.abs(J - J0).max(), np.abs(KA - KA0).max()) <= 1e-10 * scale
            if not restricted:
                assert np.abs(KB - KB0).max() <= 1e-10 * scale
    finally:
        eng.close()


@pytest.mark.gpu
def test_first_build_with_f_shells_takes_little_longer_than_the_next():
    """The first build of a context makes its work list: for benzene/QZP 7.7 million units of the f-shell
    kernels, which the list must not hold or sort one by one (that took three builds' time)."""
    import time
    sqb = load_sqb200()

    def times(atoms, builds):
        b = sqb.basis.build_basis(sqb.molecules.to_bohr(atoms), "qzp")
        P = 0.5 * np.eye(b.nbf)
        eng = sqb.JKEngine(b)
        out = []
        for _ in range(builds):
            t = time.perf_counter()
            eng.build(P, scf_cutoff=1e-10)
            out.append(time.perf_counter() - t)
        eng.close()
        return out

    times(sqb.molecules.water(), 2)                     # the kernels' code is loaded
    t = times(sqb.molecules.benzene(), 3)
    assert t[0] <= 2.0 * min(t[1:]), t
