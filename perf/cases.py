"""What this framework's time is measured on: the two-electron Fock build and the calls around it,
through the package's public entry points.

A case is one user-level call: a J/K build on device buffers (the SCF iteration's hot call), the
same build on host buffers (the call the relinked reference program makes), a batched build of
many molecules, a nuclear gradient, or a whole SCF solve.  Molecules and basis sets are the
package's own workloads: water, benzene, C60 and seeded random C/N/O organics in STO-3G to QZP.

The seed moves every atom by a few thousandths of an angstrom and draws the density, so another
seed is another molecule of the same size.  Densities have the scale and the decay with distance
of a converged density of an insulating molecule (or, with `delta`, of the difference densities
that SCF iterations build from); they need no SCF to make.

`exact` restates the J/K build in plain torch: every integral (no screen) by contracted Hermite
expansions, for molecules of up to about 130 functions.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EXACT_MAX_NBF = 130           # larger molecules take `exact` over its time limit


def package():
    """The package directory siam-quantum_b200/ as module `sqb200` (its name is no identifier)."""
    if "sqb200" not in sys.modules:
        pkg = os.path.join(ROOT, "siam-quantum_b200")
        spec = importlib.util.spec_from_file_location("sqb200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["sqb200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["sqb200"]


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call a user makes: latency and launches
        {"name": "build_water_321g", "kind": "build", "mol": "water", "basis": "3-21g"},
        # an open-shell fragment, restricted = False (both spin densities, K of each)
        {"name": "build_radical_631gs_uhf", "kind": "build", "mol": "organic", "heavy": 3, "pick": 5,
         "radical": True, "basis": "6-31g*"},
        # an ordinary molecule with d shells: the build of one SCF iteration
        {"name": "build_benzene_631gs", "kind": "build", "mol": "benzene", "basis": "6-31g*"},
        # separate s and p shells (no sp shells), long contractions, p functions on hydrogen
        {"name": "build_organic_dzp", "kind": "build", "mol": "organic", "heavy": 4, "pick": 11, "basis": "dzp"},
        # f shells
        {"name": "build_water_qzp", "kind": "build", "mol": "water", "basis": "qzp"},
        # the largest single build, forms autotuned as a long-running program does
        {"name": "build_c60_631g", "kind": "build", "mol": "c60", "basis": "6-31g", "tuned": True},
        # the same in mixed precision
        {"name": "build_c60_631g_mixed", "kind": "build", "mol": "c60", "basis": "6-31g", "tuned": True,
         "fp32_below": 1e-5},
        # host buffers in and out, default forms: the relinked reference program's call, on a
        # difference density of a later SCF iteration
        {"name": "host_organic_631gs", "kind": "host", "mol": "organic", "heavy": 9, "pick": 3, "basis": "6-31g*",
         "delta": 0.01},
        # many molecules of uneven size in one batched build
        {"name": "batch_organics_631gs", "kind": "batch", "count": 24, "heavy": 10, "pick": 20, "basis": "6-31g*",
         "delta": 0.1},
        # the nuclear gradient that ends a force or optimisation step
        {"name": "gradient_organic_631gs", "kind": "gradient", "mol": "organic", "heavy": 8, "pick": 7,
         "basis": "6-31g*"},
        # a whole solve: set-up, every SCF iteration, convergence
        {"name": "scf_benzene_631gs", "kind": "scf", "mol": "benzene", "basis": "6-31g*"},
    ]


def draw(rng):
    kind = rng.choices(["build", "host", "batch", "gradient", "scf", "qzp"], [8, 3, 3, 3, 2, 2])[0]
    bases = ["sto-3g", "3-21g", "6-31g", "6-31g*", "6-31g*", "dzp"]
    delta = rng.choice([1.0, 1.0, 0.1, 0.01])
    pick = rng.randrange(1000)
    if kind == "qzp":
        mol = rng.choice(["water", "ammonia", "hydroxyl"])
        return {"kind": "build", "mol": mol, "basis": "qzp", "radical": False, "delta": delta, "pick": pick,
                "uhf": mol == "hydroxyl" or rng.random() < 0.3}
    if kind in ("build", "host"):
        heavy = int(round(math.exp(rng.uniform(0.0, math.log(14.0)))))
        case = {"kind": kind, "mol": "organic", "heavy": heavy, "pick": pick, "basis": rng.choice(bases),
                "radical": rng.random() < 0.3, "delta": delta}
        if kind == "build":
            case["tuned"] = rng.random() < 0.3
            case["fp32_below"] = rng.choice([0.0, 0.0, 0.0, 1e-5, 1e-4])
        return case
    if kind == "batch":
        return {"kind": "batch", "count": int(round(math.exp(rng.uniform(math.log(2.0), math.log(32.0))))),
                "heavy": rng.randrange(2, 9), "pick": pick, "basis": rng.choice(["3-21g", "6-31g", "6-31g*", "6-31g*"]),
                "delta": delta}
    if kind == "gradient":
        return {"kind": "gradient", "mol": "organic", "heavy": rng.randrange(1, 6), "pick": pick,
                "basis": rng.choice(bases), "radical": rng.random() < 0.4}
    mol = rng.choice(["water", "water", "ammonia", "benzene"])
    return {"kind": "scf", "mol": mol, "pick": pick,
            "basis": rng.choice(["3-21g", "6-31g", "6-31g*"] if mol == "benzene" else ["3-21g", "6-31g", "6-31g*", "dzp"])}


# ---------------------------------------------------------------- inputs

def molecule(case, seed):
    """[(Z, x, y, z)] in angstrom: the case's molecule with every atom moved by the seed."""
    M = package().molecules
    mol = case.get("mol", "organic")
    if mol == "water":
        atoms = M.water()
    elif mol == "benzene":
        atoms = M.benzene()
    elif mol == "c60":
        atoms = M.c60()
    elif mol == "hydroxyl":
        atoms = [(8, 0.0, 0.0, 0.0), (1, 0.0, 0.0, 0.97)]
    elif mol == "ammonia":
        atoms = [(7, 0.0, 0.0, 0.1128)] + [(1, 0.9385 * math.cos(t), 0.9385 * math.sin(t), -0.2632)
                                          for t in (0.0, 2.0 * math.pi / 3.0, 4.0 * math.pi / 3.0)]
    else:
        rng = np.random.default_rng([case["pick"], case["heavy"]])
        atoms = M.random_organic(rng, case["heavy"])
        if case.get("radical") and any(a[0] == 1 for a in atoms):
            atoms = M.remove_one_h(atoms, rng)
    rng = np.random.default_rng([17, seed])
    return [(z, *(float(c + 0.004 * rng.standard_normal()) for c in xyz)) for z, *xyz in atoms]


def density(basis, rng, scale, occ):
    """A symmetric one-spin density: elements of the size of a molecule's, falling off with the
    distance between the functions' centres (0.5 e^-1 per bohr)."""
    c = basis.center
    d = np.sqrt(((c[:, None, :] - c[None, :, :]) ** 2).sum(-1))
    A = 0.35 * rng.standard_normal(d.shape) * np.exp(-0.5 * d)
    A = 0.5 * (A + A.T)
    A[np.diag_indices_from(A)] = occ * rng.uniform(0.1, 1.0, len(A))
    return np.ascontiguousarray(scale * A)


def inputs(case, seed):
    """(atoms in bohr, basis, PA, PB, restricted): made from the seed alone."""
    P = package()
    atoms = P.molecules.to_bohr(molecule(case, seed))
    basis = P.basis.build_basis(atoms, case["basis"])
    restricted = not (case.get("radical") or case.get("uhf"))
    rng = np.random.default_rng([29, seed])
    scale = case.get("delta", 1.0)
    PA = density(basis, rng, scale, 1.0)
    PB = PA if restricted else density(basis, rng, scale, 0.9)
    return atoms, basis, PA, PB, restricted


def batch_case(case, k):
    """Molecule k of a batch: 2 to `heavy` heavy atoms, every fourth one a radical."""
    heavy = 2 + (7 * k + case["pick"]) % max(1, case["heavy"] - 1)
    return {"mol": "organic", "heavy": heavy, "pick": case["pick"] + k, "radical": k % 4 == 3,
            "basis": case["basis"], "delta": case.get("delta", 1.0)}


def prepare(case, seed):
    P = package()
    dev = torch.device("cuda", 0)
    f64 = dict(dtype=torch.float64, device=dev)
    kind = case["kind"]
    if kind == "scf":
        return {"kind": kind, "atoms": molecule(case, seed), "basis": case["basis"]}
    stream = torch.cuda.Stream(dev)
    if kind == "batch":
        engines, pa, pb, restricted = [], [], [], []
        for k in range(case["count"]):
            _, basis, PA, PB, r = inputs(batch_case(case, k), 1000 * seed + k)
            engines.append(P.JKEngine(basis, device=0))
            pa.append(PA.reshape(-1))
            pb.append(PB.reshape(-1))
            restricted.append(r)
        batch = P.JKBatch(engines)
        st = {"kind": kind, "batch": batch, "stream": stream, "PA": torch.tensor(np.concatenate(pa), **f64),
              "PB": torch.tensor(np.concatenate(pb), **f64), "out": torch.empty((3, batch.total), **f64)}
        torch.cuda.synchronize()
        batch.set_step(restricted, 1e-10)
        batch.autotune(st["PA"].data_ptr(), st["PB"].data_ptr(), stream=stream.cuda_stream)
        return st
    atoms, basis, PA, PB, restricted = inputs(case, seed)
    n = basis.nbf
    eng = P.JKEngine(basis, device=0)
    if case.get("fp32_below"):
        eng.set_precision(case["fp32_below"])
    st = {"kind": kind, "eng": eng, "restricted": restricted, "stream": stream}
    if kind == "host":
        pin = lambda a: torch.from_numpy(a).pin_memory().numpy()
        st["PA"] = pin(PA)
        st["PB"] = st["PA"] if restricted else pin(PB)
        st["out"] = tuple(pin(np.zeros((n, n))) for _ in range(3))
        return st
    if kind == "gradient":
        rng = np.random.default_rng([31, seed])
        st["Z"] = np.array([a[0] for a in atoms], dtype=np.float64)
        st["xyz"] = np.array([a[1:] for a in atoms], dtype=np.float64)
        st["PA"], st["PB"], st["W"] = PA, PB, -density(basis, rng, 0.7, 1.0)
        return st
    st["PA"] = torch.tensor(PA, **f64)
    st["PB"] = st["PA"] if restricted else torch.tensor(PB, **f64)
    st["out"] = [torch.empty((n, n), **f64) for _ in range(2 if restricted else 3)]
    if case.get("tuned"):
        torch.cuda.synchronize()
        eng.autotune(st["PA"].data_ptr(), st["PB"].data_ptr(), restricted=restricted, scf_cutoff=1e-10,
                     stream=stream.cuda_stream)
    return st


# ---------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "scf":
        job = package().scf.SCFJob(state["atoms"], state["basis"], device=0)
        energy = job.run()
        out = {"energy": energy, "PA": job.PA, "FA": job.FA}
        job.close()
        return out
    if kind == "host":
        return state["eng"].build(state["PA"], state["PB"], restricted=state["restricted"], scf_cutoff=1e-10,
                                  out=state["out"])
    if kind == "gradient":
        return state["eng"].gradient(state["Z"], state["xyz"], state["PA"], state["PB"], state["W"])
    # device builds run on the program's own stream, ordered with torch's current one
    here, stream = torch.cuda.current_stream(), state["stream"]
    stream.wait_stream(here)
    if kind == "batch":
        JT, KA, KB = state["out"]
        state["batch"].build_device(state["PA"].data_ptr(), state["PB"].data_ptr(), JT.data_ptr(), KA.data_ptr(),
                                    KB.data_ptr(), stream=stream.cuda_stream)
    else:
        state["eng"].build_tensors(state["PA"], state["PB"], *state["out"], restricted=state["restricted"],
                                   scf_cutoff=1e-10, stream=stream)
    here.wait_stream(stream)
    return state["out"]


# ---------------------------------------------------------------- work a pass cannot do without

def _shells(basis):
    """[(first function, [(l, m, n)], centre, exponents, weights (nprim, nfunc))] of a basis."""
    out, i, n = [], 0, basis.nbf
    ex = lambda k: basis.exps[basis.offset[k]:basis.offset[k] + basis.nprim[k]]
    w = lambda k: basis.ncoef[basis.offset[k]:basis.offset[k] + basis.nprim[k]]
    while i < n:
        j = i + 1
        while (j < n and j - i < 10 and np.array_equal(basis.center[i], basis.center[j])
               and np.array_equal(ex(i), ex(j)) and not (basis.lmn[j].sum() < basis.lmn[j - 1].sum())):
            j += 1
        out.append((i, basis.lmn[i:j], basis.center[i], np.asarray(ex(i)), np.stack([w(k) for k in range(i, j)], 1)))
        i = j
    return out


def _quartet_flops(basis, scale):
    """Operations of one build: per surviving shell quartet the primitive integrals (Boys
    function, Hermite recursion, one side's contraction), the other side's contraction and the
    J/K digestion, in the cheapest order of one McMurchie-Davidson evaluation.  Survivors by
    an s-type estimate of the Schwarz bound times the density's scale."""
    sh = _shells(basis)
    groups = {}
    for a in range(len(sh)):
        for b in range(a + 1):
            A, B = sh[a], sh[b]
            p = A[3][:, None] + B[3][None, :]
            mu = A[3][:, None] * B[3][None, :] / p
            s = np.exp(-mu * ((A[2] - B[2]) ** 2).sum()) * np.abs(A[4]).max(1)[:, None] * np.abs(B[4]).max(1)[None, :]
            bound = float((s * p ** -1.25).sum()) * 5.9
            l = int(A[1].sum(1).max() + B[1].sum(1).max())
            groups.setdefault((l, len(A[1]) * len(B[1]), p.size), []).append(bound)
    keys = sorted(groups)
    nh = lambda l: (l + 1) * (l + 2) * (l + 3) // 6
    total = 0.0
    for i, x in enumerate(keys):
        bx = np.sort(groups[x])
        for y in keys[:i + 1]:
            by = np.sort(groups[y])
            count = int((len(by) - np.searchsorted(by, 1e-10 / np.maximum(scale * bx, 1e-300))).sum())
            if x == y:
                count = (count + 1) // 2
            L = x[0] + y[0]
            prim = 40 + 6 * L + 3 * nh(L) + 2 * nh(x[0]) * y[1] * min(4, 1 + y[0])
            flush = 2 * x[1] * y[1] * min(4, 1 + x[0])
            total += count * (x[2] * y[2] * prim + x[2] * flush + 12 * x[1] * y[1])
    return total


def work(case):
    P = package()
    if case["kind"] == "batch":
        parts = [work(dict(batch_case(case, k), kind="build")) for k in range(case["count"])]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    atoms = P.molecules.to_bohr(molecule(case, 1))
    basis = P.basis.build_basis(atoms, case["basis"])
    n2 = 8 * basis.nbf ** 2
    flops = _quartet_flops(basis, case.get("delta", 1.0))
    if case["kind"] == "gradient":
        return {"bytes": 3 * n2, "flops": 3.0 * flops}
    if case["kind"] == "scf":
        return {"bytes": 3 * n2, "flops": 12.0 * flops}
    spins = 2 if case.get("radical") or case.get("uhf") else 1
    return {"bytes": (2 * spins + 1) * n2, "flops": flops}


# ---------------------------------------------------------------- the build in plain torch

def _boys(T, M):
    """F_0 .. F_M: the series of the top order and downward recursion for T < 40, else erf and
    upward recursion."""
    small = T < 40.0
    Ts = torch.where(small, T, torch.zeros_like(T))
    e = torch.exp(-Ts)
    term = torch.full_like(Ts, 1.0 / (2 * M + 1))
    total = term.clone()
    for i in range(1, 190):
        term = term * (2.0 * Ts / (2 * M + 2 * i + 1))
        total += term
    F = [None] * (M + 1)
    F[M] = e * total
    for m in range(M - 1, -1, -1):
        F[m] = (2.0 * Ts * F[m + 1] + e) / (2 * m + 1)
    Tl = torch.where(small, torch.full_like(T, 40.0), T)
    el = torch.exp(-Tl)
    G = 0.5 * torch.sqrt(math.pi / Tl) * torch.erf(torch.sqrt(Tl))
    for m in range(M + 1):
        F[m] = torch.where(small, F[m], G)
        G = ((2 * m + 1) * G - el) / (2.0 * Tl)
    return F


def _tuv(L):
    return [(t, u, N - t - u) for N in range(L + 1) for t in range(N, -1, -1) for u in range(N - t, -1, -1)]


def _hermite_1d(p, xa, xb, i, j):
    """E^{ij}_t of one axis (t = 0 .. i+j), prefactor excluded."""
    E = {(0, 0): [1.0]}
    h = 0.5 / p

    def get(a, b):
        if (a, b) not in E:
            src, X = (get(a - 1, b), xa) if a > 0 else (get(a, b - 1), xb)
            n = a + b
            E[a, b] = [X * (src[t] if t < n else 0.0) + (h * src[t - 1] if t > 0 else 0.0)
                       + ((t + 1) * src[t + 1] if t + 1 < n else 0.0) for t in range(n + 1)]
        return E[a, b]
    return get(i, j)


def _integrals(basis, dev):
    """(pairs, ERI matrix over the function pairs p >= q), every integral, no screen."""
    sh = _shells(basis)
    n = basis.nbf
    index = np.full((n, n), -1)
    pairs = [(p, q) for p in range(n) for q in range(p + 1)]
    for k, (p, q) in enumerate(pairs):
        index[p, q] = index[q, p] = k
    groups = {}               # Hermite order -> [exponent sum, centre, {pair: coefficients}]
    for a in range(len(sh)):
        for b in range(a + 1):
            fa, la, A, ea, wa = sh[a]
            fb, lb, B, eb, wb = sh[b]
            L = int(la.sum(1).max() + lb.sum(1).max())
            where = {h: k for k, h in enumerate(_tuv(L))}
            for i, x in enumerate(ea):
                for j, y in enumerate(eb):
                    p = x + y
                    C = (x * A + y * B) / p
                    k0 = math.exp(-x * y / p * ((A - B) ** 2).sum())
                    rows = {}
                    for f, u in enumerate(la):
                        for g, v in enumerate(lb):
                            if fa + f < fb + g:
                                continue
                            c = np.zeros(len(where))
                            ex = [_hermite_1d(p, C[d] - A[d], C[d] - B[d], int(u[d]), int(v[d])) for d in range(3)]
                            for t, cx in enumerate(ex[0]):
                                for s, cy in enumerate(ex[1]):
                                    for r, cz in enumerate(ex[2]):
                                        c[where[t, s, r]] = cx * cy * cz
                            rows[int(index[fa + f, fb + g])] = c * (k0 * wa[i, f] * wb[j, g])
                    groups.setdefault(L, []).append((p, C, rows))
    blocks = []
    for L, prims in sorted(groups.items()):
        hs = _tuv(L)
        pidx = sorted({k for _, _, rows in prims for k in rows})
        col = {k: c for c, k in enumerate(pidx)}
        r, c, v = [], [], []
        for m, (_, _, rows) in enumerate(prims):
            for k, co in rows.items():
                for h in np.nonzero(co)[0]:
                    r.append(h * len(prims) + m)
                    c.append(col[k])
                    v.append(co[h])
        E = torch.sparse_coo_tensor(torch.tensor([c, r]), torch.tensor(v, dtype=torch.float64),
                                    (len(pidx), len(hs) * len(prims))).to(dev).coalesce()
        blocks.append((L, hs, torch.tensor([x[0] for x in prims], dtype=torch.float64, device=dev),
                       torch.tensor(np.array([x[1] for x in prims]), device=dev), E,
                       torch.tensor(pidx, device=dev)))
    G = torch.zeros((len(pairs), len(pairs)), dtype=torch.float64, device=dev)
    for bi, (La, ha, pa, Ca, Ea, ia) in enumerate(blocks):
        for Lb, hb, pb, Cb, Eb, ib in blocks[:bi + 1]:
            L, m = La + Lb, len(pa)
            step = max(1, int(4e8 / (8 * m * (len(ha) * len(hb) + 3 * len(_tuv(L))))))
            out = torch.zeros((len(ia), len(ib)), dtype=torch.float64, device=dev)
            nb, Ebd = len(pb), Eb.to_dense().reshape(len(ib), len(hb), len(pb))
            for s in range(0, nb, step):
                p, q = pa[:, None], pb[None, s:s + step]
                al = p * q / (p + q)
                D = Ca[:, None, :] - Cb[None, s:s + step, :]
                F = _boys(al * (D * D).sum(-1), L)
                pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
                R = {(k, 0, 0, 0): pre * (-2.0 * al) ** k * F[k] for k in range(L + 1)}
                for k in range(L - 1, -1, -1):          # level by level, order k needs k + 1
                    for (t, u, v) in _tuv(L - k)[1:]:
                        d = 0 if t else 1 if u else 2
                        h = [t, u, v]
                        h[d] -= 1
                        x = D[:, :, d] * R[(k + 1, *h)]
                        if h[d] > 0:
                            c = h[d]
                            h[d] -= 1
                            x = x + c * R[(k + 1, *h)]
                        R[k, t, u, v] = x
                    for key in [key for key in R if key[0] == k + 1]:
                        del R[key]
                w = q.shape[1]
                V = torch.empty((len(ha), m, len(hb), w), dtype=torch.float64, device=dev)
                for x, (t, u, v) in enumerate(ha):
                    for y, (a, b, c) in enumerate(hb):
                        V[x, :, y, :] = (-1.0) ** (a + b + c) * R[0, t + a, u + b, v + c]
                del R
                half = torch.sparse.mm(Ea, V.reshape(len(ha) * m, len(hb) * w))
                out += half @ Ebd[:, :, s:s + step].reshape(len(ib), -1).T
                del V, half
            # function pairs appear in several groups (sp shells): add the block both ways
            G.index_put_((ia[:, None], ib[None, :]), out, accumulate=True)
            if La != Lb:
                G.index_put_((ib[:, None], ia[None, :]), out.T.contiguous(), accumulate=True)
    return torch.tensor(index, device=dev), G


def exact(case, seed):
    if case["kind"] not in ("build", "host"):
        return None
    _, basis, PA, PB, restricted = inputs(case, seed)
    n = basis.nbf
    if n > EXACT_MAX_NBF or (n > 40 and not torch.cuda.is_available()):
        return None
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    index, G = _integrals(basis, dev)
    PA, PB = torch.tensor(PA, device=dev), torch.tensor(PB, device=dev)
    PT = PA + PB
    weight = torch.zeros(G.shape[0], dtype=torch.float64, device=dev)
    weight.index_add_(0, index.reshape(-1), PT.reshape(-1))
    J = (G @ weight)[index]
    KA, KB = torch.empty_like(J), torch.empty_like(J)
    for a in range(n):                        # K_ac = sum_bd (ab|cd) P_bd
        g = G[index[a]][:, index.reshape(-1)].reshape(n, n, n)       # [b][c][d] of this a
        KA[a] = -torch.einsum("bcd,bd->c", g, PA)
        KB[a] = -torch.einsum("bcd,bd->c", g, PB)
    J, KA, KB = J.cpu(), KA.cpu(), KB.cpu()
    if case["kind"] == "host":
        return (J.numpy(), KA.numpy(), (KA if restricted else KB).numpy())
    return [J, KA] if restricted else [J, KA, KB]
