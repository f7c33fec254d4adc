"""Generate the class kernels of the two-electron nuclear gradient (s, sp, p and d shells).

One kernel per quartet class (bra pair class | ket pair class).  The two-electron term is
sum over unique shell quartets and their primitive and function quartets of G d(ab|cd), with
G = deg * gamma * prefactor * weights, gamma the density factor 4 PT_ab PT_cd - (PT_ac PT_bd + PT_ad
PT_bc + PS_ac PS_bd + PS_ad PS_bc) (GradEri_ShellSet_Parallel, reference src/grad.c:1734-2150), and a
function quartet of a primitive quartet dropped when |gamma * function degeneracy * prefactor *
weights| is below the screen (src/grad.c:1982-1988).  That test takes the value of one primitive
function quartet, so the contraction cannot leave the primitive loop; the density can: a
primitive quartet is reduced to a few scalars in Hermite space,

    U[h]  = sum_ab G_ab E_ab[h]                      Y[h]  = sum_k (-1)^|k| E_cd[k] R[h + k]
    U'x[h] = the same with dE_ab/dX_AB               Y'x[h] = the same with dE_cd/dX_CD
    e = U.Y    FP_x = sum_h U[h] Y[h + 1x]    FAB_x = U'x.Y - 2 mu_ab X_AB e    FCD_x = U.Y'x - 2 mu_cd X_CD e
    dA = (a/p) FP + FAB    dB = (b/p) FP - FAB    dC = -(c/q) FP + FCD    dD = -(dA + dB + dC)

so no integral block is formed and no index is raised.  A CTA owns one bra pair (its 1-D Hermite
tables in shared memory, a chunk of primitives at a time), a thread one ket pair (or si x sj
threads share one ket and split the primitives), and a pass (grid.y) one ket function pair
(c, d): per thread gamma of the bra functions, U and Y stay in registers.  Ket function pairs that
differ only by a permutation of the axes share one code path: the pass permutes the coordinates,
the bra's tables and its function indices (x, y, z of a p shell, xx, yy, zz and xy, xz, yz of a d
shell), which keeps the code of a class small enough for the instruction cache.

The larger pair is the bra, except where both have at least 9 functions and the larger one more
than 18: there the smaller one is the bra, because a thread holds one gamma per bra function.

Usage: python gen_grad_kernels.py <outdir>
"""
import itertools
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from gen_jk_kernels import COMP, LMAX, PAIRS, Emitter, gen_R, pair_L, quartet_classes, write_if_changed  # noqa: E402

NHEAD = 9          # bra record header in shared memory: p, P (3), kp, a/p, 2 mu X_AB (3)
NFIELD = 15        # global record: p, P (3), kp, a/p, X_PA (3), X_PB (3), 2 mu X_AB (3), then the weights
CTA = 64


def simplex(L):
    return [(t, u, v) for N in range(L + 1) for t in range(N, -1, -1) for u in range(N - t, -1, -1) for v in [N - t - u]]


def roles(x, y):
    """(bra, ket) of the class of pairs x >= y (generator order: x the larger)."""
    nx, ny = (len(COMP[p[0]]) * len(COMP[p[1]]) for p in (x, y))
    return (y, x) if nx > 18 and 9 <= ny < nx else (x, y)


def ket_orbits(ket):
    """Per ket function pair (c, d): (orbit index, axis permutation pi); the representatives.
    In the permuted frame axis r is the molecule's axis pi[r]."""
    reps, out = [], []
    for c in COMP[ket[0]]:
        for d in COMP[ket[1]]:
            best = max((tuple(c[k] for k in pi), tuple(d[k] for k in pi), tuple(-k for k in pi))
                       for pi in itertools.permutations(range(3)))
            rep, pi = best[:2], tuple(-k for k in best[2])
            if rep not in reps:
                reps.append(rep)
            out.append((reps.index(rep), pi))
    return reps, out


def tab1d(pc):
    """Offsets of the 1-D tables of a bra class: E^{ij}_t (t <= i+j) and its X_AB derivative."""
    off, offd, n, nd = {}, {}, 0, 0
    for i in range(LMAX[pc[0]] + 1):
        for j in range(LMAX[pc[1]] + 1):
            off[i, j] = n
            n += i + j + 1
            offd[i, j] = nd
            nd += i + j
    return off, n, offd, nd


def emit_1d(em, pre, imax, jmax, xa, xb, h):
    """Emit E^{ij}_t for i <= imax, j <= jmax as named constants; returns {(i, j): [names]}."""
    E = {(0, 0): ["1.0"]}
    for i in range(imax + 1):
        for j in range(jmax + 1):
            if i == 0 and j == 0:
                continue
            si, sj, X = (i - 1, j, xa) if i > 0 else (i, j - 1, xb)
            src, names = E[si, sj], []
            for t in range(i + j + 1):
                terms = []
                if t < i + j:
                    terms.append((X, src[t]))
                if t > 0:
                    terms.append((h, src[t - 1]))
                if t + 1 < i + j:
                    terms.append(("%d.0" % (t + 1), src[t + 1]))
                expr = None
                for u, w in terms:
                    if expr is None:
                        expr = u if w == "1.0" else w if u == "1.0" else "%s * %s" % (u, w)
                    elif w == "1.0":
                        expr = "(%s) + %s" % (expr, u)
                    else:
                        expr = "fma(%s, %s, %s)" % (u, w, expr)
                nm = "%s%d%d_%d" % (pre, i, j, t)
                em("const double %s = %s;" % (nm, expr))
                names.append(nm)
            E[i, j] = names
    return E


def emit_d1d(em, pre, E, i, j, fa, fb):
    """Emit dE^{ij}_t/dX_AB = -(b/p) i E^{i-1,j}_t + (a/p) j E^{i,j-1}_t, t < i+j; names."""
    names = []
    for t in range(i + j):
        terms = []
        if i > 0:
            terms.append("-%s%s" % (fb, "" if E[i - 1, j][t] == "1.0" else " * " + E[i - 1, j][t]) + (" * %d.0" % i if i > 1 else ""))
        if j > 0:
            terms.append("%s%s" % (fa, "" if E[i, j - 1][t] == "1.0" else " * " + E[i, j - 1][t]) + (" * %d.0" % j if j > 1 else ""))
        nm = "%s%d%d_%d" % (pre, i, j, t)
        em("const double %s = %s;" % (nm, " + ".join(terms)))
        names.append(nm)
    return names


def func_perm(t, k):
    """Expression of the molecule-frame index of permuted-frame function k of shell type t."""
    if t == "S":
        return "0"
    if t == "L":
        return "0" if k == 0 else "1 + p%d" % (k - 1)
    if t == "P":
        return "p%d" % k
    return "p%d" % k if k < 3 else "2 + %s" % {3: "p0 + p1", 4: "p0 + p2", 5: "p1 + p2"}[k]


def gen_grad(bra, ket, only=None):
    """The kernel of a class, or of one orbit of its ket function pairs (`only`)."""
    ta, tb = bra
    tc, td = ket
    fA, fB, fC, fD = COMP[ta], COMP[tb], COMP[tc], COMP[td]
    na, nb, nc, nd = len(fA), len(fB), len(fC), len(fD)
    Lb, Lk = pair_L(bra), pair_L(ket)
    L = Lb + Lk + 1
    off, n1, offd, n1d = tab1d(bra)
    NB = NHEAD + na + nb + 3 * (n1 + n1d) + 1       # + the largest |weight| product
    NFB, NFK = NFIELD + na + nb, NFIELD + nc + nd
    WT = NHEAD                                        # weights
    T0 = NHEAD + na + nb                              # E tables, then derivative tables
    reps, orb = ket_orbits(ket)
    Hb, Hb1, Hbd = simplex(Lb), simplex(Lb + 1), simplex(max(0, Lb - 1))
    name = "grad_%s_%s" % (bra, ket) + ("" if only is None else "_%d" % only)
    cds = [k for k, (o, _) in enumerate(orb) if only is None or o == only]
    hn = lambda h: "%d%d%d" % h
    em = Emitter()
    out = ['static __constant__ unsigned char kCd_%s[%d] = {%s};' % (name, len(cds), ", ".join(str(k) for k in cds)),
           'static __constant__ unsigned char kOrb_%s[%d] = {%s};' % (name, len(cds), ", ".join(str(orb[k][0]) for k in cds)),
           'static __constant__ unsigned char kPerm_%s[%d] = {%s};' % (
               name, len(cds), ", ".join(str(orb[k][1][0] | orb[k][1][1] << 2 | orb[k][1][2] << 4) for k in cds)),
           # at least one CTA per SM: without it ptxas falls back to 32 registers and 18 KB of stack a thread in
           # the largest classes (a launch then takes 5 GB of local memory)
           'extern "C" __global__ void __launch_bounds__(%d, 1)' % CTA,
           "%s(const sqb::GradArgs a, const sqb::WorkItem* __restrict__ items) {" % name]
    em("extern __shared__ double sb[];                // [chunk][%d] bra primitive records" % NB)
    em("const sqb::WorkItem it = items[blockIdx.x];")
    em("const sqb::GradPair bp = a.bra_pairs[it.bra];")
    em("const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;")
    em("const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;")
    em("const int gj = grp / si, gi = grp - gj * si;")
    em("const int cd = kCd_%s[blockIdx.y], c = cd / %d, d = cd - c * %d;" % (name, nd, nd))
    em("const int orbit = kOrb_%s[blockIdx.y], pi = kPerm_%s[blockIdx.y];" % (name, name))
    em("const int p0 = pi & 3, p1 = (pi >> 2) & 3, p2 = pi >> 4;   // axis r of this pass = molecule axis p<r>")
    em("const bool have = kl < it.cnt;")
    em("const sqb::GradPair kp = a.ket_pairs[it.k0 + min(kl, it.cnt - 1)];")
    em("const double screen = a.screen;")
    em("const bool ok = have && !(bp.sch * kp.sch * bp.pm * kp.pm < screen);")
    em("if (!__syncthreads_or(ok)) return;")
    em("const int N = a.nbf, nbp = bp.nprim, nkp = kp.nprim;")
    em("const bool same_b = bp.P == bp.Q, same_k = kp.P == kp.Q, same_pair = a.same_class && it.bra == it.k0 + kl;")
    em("const double deg = (same_b ? 0.5 : 1.0) * (same_k ? 0.5 : 1.0) * (same_pair ? 0.5 : 1.0);")
    em("const double* __restrict__ PT = a.PT;")
    em("const double* __restrict__ PS = a.PS;")
    em("const int fc = kp.fP + c, fd = kp.fQ + d;")
    # gamma * deg of the bra functions (permuted order); the density rows of c and d
    for x, n, base, t in (("a", na, "bp.fP", ta), ("b", nb, "bp.fQ", tb)):
        for k in range(n):
            em("const int f%s%d = %s + %s;" % (x, k, base, func_perm(t, k)))
    for ab in range(na * nb):
        em("double g%d = 0.0;" % ab)
    em("double gmax = 0.0, gsum = 0.0;")
    em("if (ok) {")
    em.ind += 1
    em("const double ptk = 4.0 * PT[fc * N + fd];")
    for x, n in (("a", na), ("b", nb)):
        for k in range(n):
            for y in "cd":
                em("const double t%s%d%s = PT[f%s%d * N + f%s], s%s%d%s = PS[f%s%d * N + f%s];" % (x, k, y, x, k, y, x, k, y, x, k, y))
    for i in range(na):
        for j in range(nb):
            em("g%d = deg * (ptk * PT[fa%d * N + fb%d] - (ta%dc * tb%dd + ta%dd * tb%dc + sa%dc * sb%dd + sa%dd * sb%dc));" % (
                i * nb + j, i, j, i, j, i, j, i, j, i, j))
            em("gmax = fmax(gmax, fabs(g%d)); gsum += g%d;" % (i * nb + j, i * nb + j))
    em("if (!(gsum - gsum == 0.0)) gmax = fabs(gsum); // fmax drops a NaN: a density that is not finite skips nothing")
    em.ind -= 1
    em("}")
    # thresholds on |G|: screen times (shell degeneracy / function degeneracy) of the function quartet
    em("const double th = screen * (same_k && fc != fd ? 0.5 : 1.0), tho = same_b ? 0.5 * th : th;")
    em("const double hp = same_pair ? 0.5 : 1.0;    // function pairs of one shell pair that differ")
    em("const double thmin = screen * deg * (1.0 - 1e-12);")
    em("double A0 = 0.0, A1 = 0.0, A2 = 0.0, B0 = 0.0, B1 = 0.0, B2 = 0.0, C0 = 0.0, C1 = 0.0, C2 = 0.0;")
    em("const double* __restrict__ kprim = a.ket_prims + kp.poff;")
    em("const int kS = kp.kstride;")
    em("for (int i0 = 0; i0 < nbp; i0 += a.chunk) {")
    em.ind += 1
    em("const int ni = min(a.chunk, nbp - i0);")
    em("__syncthreads();                              // the previous chunk's readers are done")
    em("for (int x = threadIdx.x; x < 3 * ni; x += %d) {   // 1-D tables: one (primitive, axis) per thread" % CTA)
    em.ind += 1
    em("const int i = x / 3, ax = x - 3 * i;")
    em("const double* __restrict__ src = a.bra_prims + bp.poff + (long long)(i0 + i) * %d * bp.kstride;" % NFB)
    em("const int S = bp.kstride;")
    em("double* __restrict__ dst = sb + i * %d;" % NB)
    em("const double p = src[0], h = 0.5 / p, ra = src[5 * S], rb = 1.0 - ra, xa = src[(6 + ax) * S], xb = src[(9 + ax) * S];")
    em("dst[1 + ax] = src[(1 + ax) * S];")
    em("dst[6 + ax] = src[(12 + ax) * S];")
    em("if (ax == 0) {")
    em("  dst[0] = p; dst[4] = src[4 * S]; dst[5] = ra;")
    em("  double wa = 0.0, wb = 0.0;")
    em("  for (int f = 0; f < %d; ++f) { const double w = src[(%d + f) * S]; dst[%d + f] = w; wa = fmax(wa, fabs(w)); }" % (na, NFIELD, WT))
    em("  for (int f = 0; f < %d; ++f) { const double w = src[(%d + f) * S]; dst[%d + f] = w; wb = fmax(wb, fabs(w)); }" % (nb, NFIELD + na, WT + na))
    em("  dst[%d] = wa * wb;" % (NB - 1))
    em("}")
    E = emit_1d(em, "E", LMAX[ta], LMAX[tb], "xa", "xb", "h")
    em("double* __restrict__ te = dst + %d + ax * %d;" % (T0, n1))
    for (i, j), o in off.items():
        for t in range(i + j + 1):
            em("te[%d] = %s;" % (o + t, E[i, j][t]))
    if n1d:
        em("double* __restrict__ tde = dst + %d + ax * %d;" % (T0 + 3 * n1, n1d))
    for (i, j), o in offd.items():
        if i + j:
            for t, nm in enumerate(emit_d1d(em, "D", E, i, j, "ra", "rb")):
                em("tde[%d] = %s;" % (o + t, nm))
    em.ind -= 1
    em("}")
    em("__syncthreads();")
    em("if (ok) {")
    em.ind += 1
    em("switch (orbit) {")
    for oi, (lc, ld) in enumerate(reps):
        if only is not None and oi != only:
            continue
        em("case %d: {  // ket functions like %s %s" % (oi, lc, ld))
        em.ind += 1
        em("for (int i = (gi + si - i0 % si) % si; i < ni; i += si) {   // bra primitives gi, gi + si, ...")
        em.ind += 1
        em("const double* __restrict__ br = sb + i * %d;" % NB)
        em("const double p = br[0], P0 = br[1 + p0], P1 = br[1 + p1], P2 = br[1 + p2], kpb = br[4], wmax = br[%d];" % (NB - 1))
        for r in range(3):
            em("const double* __restrict__ e%d = br + %d + p%d * %d;" % (r, T0, r, n1))
            if n1d:
                em("const double* __restrict__ d%d = br + %d + p%d * %d;" % (r, T0 + 3 * n1, r, n1d))
        em("for (int j = gj; j < nkp; j += sj) {")
        em.ind += 1
        em("const double* __restrict__ kj = kprim + (long long)j * %d * kS;" % NFK)
        em("const double q = kj[0];")
        em("const double pq = p + q, rs = rsqrt(pq);")
        em("const double pre = TWO_PI_2_5 * kpb * kj[4 * kS] * rs;")
        em("if (pre < PRIM_CUTOFF) continue;")
        em("const double s = pre * (kj[(%d + c) * kS] * kj[(%d + d) * kS]);" % (NFIELD, NFIELD + nc))
        em("if (gmax * fabs(s) * wmax < thmin) continue;   // every function quartet is below the screen")
        # U and U' from the screened G
        for h in Hb:
            em("double U%s = 0.0;" % hn(h))
        daxes = [r for r in range(3) if Lb > 0]
        for r in daxes:
            for h in Hbd:
                em("double V%d_%s = 0.0;" % (r, hn(h)))
        em("{")
        em.ind += 1
        for k in range(na):
            em("const double wa%d = br[%d + fa%d - bp.fP];" % (k, WT, k))
        for k in range(nb):
            em("const double wb%d = s * br[%d + fb%d - bp.fQ];" % (k, WT + na, k))
        for ia, la in enumerate(fA):
            for ib, lb in enumerate(fB):
                ab = ia * nb + ib
                # same shells on both sides: the function degeneracy has its 1/2 only on the diagonal
                t = "th" if (ta == tb and la == lb) else ("tho" if ta == tb else "th")
                if bra == ket:
                    d1 = la == lc and lb == ld
                    d2 = la == ld and lb == lc
                    if d1:
                        pass
                    elif d2:
                        t = "(same_b ? %s : hp * %s)" % (t, t)
                    else:
                        t = "hp * %s" % t
                em("{ double G = g%d * (wa%d * wb%d); G = fabs(G) < %s ? 0.0 : G;" % (ab, ia, ib, t))
                E1 = [["1.0"] if la[r] + lb[r] == 0 else ["e%d[%d]" % (r, off[la[r], lb[r]] + x) for x in range(la[r] + lb[r] + 1)]
                      for r in range(3)]
                D1 = [["d%d[%d]" % (r, offd[la[r], lb[r]] + x) for x in range(la[r] + lb[r])] for r in range(3)]

                def accumulate(F, dst):
                    # dst[h] += G F0[t] F1[u] F2[v], factors of 1 left out
                    for t_, f0 in enumerate(F[0]):
                        g0 = "G" if f0 == "1.0" else "G * %s" % f0
                        for u_, f1 in enumerate(F[1]):
                            g1 = g0 if f1 == "1.0" else "%s * %s" % (g0, f1)
                            for v_, f2 in enumerate(F[2]):
                                dd = dst % hn((t_, u_, v_))
                                if f2 != "1.0":
                                    em("  %s = fma(%s, %s, %s);" % (dd, g1, f2, dd))
                                else:
                                    fs = g1.rsplit(" * ", 1)
                                    em("  %s = fma(%s, %s, %s);" % (dd, fs[0], fs[1], dd) if len(fs) > 1 else "  %s += %s;" % (dd, g1))

                accumulate(E1, "U%s")
                for r in range(3):
                    if D1[r]:
                        accumulate([D1[x] if x == r else E1[x] for x in range(3)], "V%d_%%s" % r)
                em("}")
        em.ind -= 1
        em("}")
        # Boys function, seeds, and Y, Y' from the Hermite integrals
        em("const double alpha = p * q * (rs * rs);")
        for r in range(3):
            em("const double %s = P%d - kj[(1 + p%d) * kS];" % ("XYZ"[r], r, r))
        em("double F[%d];" % (L + 1))
        em("sqb::boys<%d>(alpha * fma(X, X, fma(Y, Y, Z * Z)), a.boys_tab, F);" % L)
        em("const double m2a = -2.0 * alpha;")
        em("const double b0 = F[0];")
        em("double w = m2a;")
        for n in range(1, L + 1):
            em("const double b%d = w * F[%d];" % (n, n))
            if n < L:
                em("w *= m2a;")
        kax = [r for r in range(3) if lc[r] + ld[r] > 0]
        em("const double rc = kj[5 * kS], rd = 1.0 - rc%s;" % (", hq = 0.5 / q" if kax else ""))
        KE, KD = [["1.0"]] * 3, [None] * 3
        for r in kax:
            em("const double xc%d = kj[(6 + p%d) * kS], xd%d = kj[(9 + p%d) * kS];" % (r, r, r, r))
            T = emit_1d(em, "k%d_" % r, lc[r], ld[r], "xc%d" % r, "xd%d" % r, "hq")
            KE[r] = T[lc[r], ld[r]]
            KD[r] = emit_d1d(em, "kd%d_" % r, T, lc[r], ld[r], "rc", "rd")

        def prods(F, pre):
            """[(k, name)] of the products F0[t] F1[u] F2[v], signed by (-1)^|k|."""
            got = []
            for t_, f0 in enumerate(F[0]):
                for u_, f1 in enumerate(F[1]):
                    for v_, f2 in enumerate(F[2]):
                        fs = [f for f in (f0, f1, f2) if f != "1.0"]
                        nm = "%s%d%d%d" % (pre, t_, u_, v_)
                        em("const double %s = %s%s;" % (nm, "-" if (t_ + u_ + v_) % 2 else "", " * ".join(fs) or "1.0"))
                        got.append(((t_, u_, v_), nm, not fs))
            return got

        ke = prods(KE, "ke")
        kd = {r: prods([KD[x] if x == r else KE[x] for x in range(3)], "kd%d" % r) for r in kax}
        for h in Hb1:
            em("double Y%s = 0.0;" % hn(h))
        for r in kax:
            for h in Hb:
                em("double W%d_%s = 0.0;" % (r, hn(h)))
        cons, need = {}, set()
        add = lambda h, k: tuple(x + y for x, y in zip(h, k))
        for k, nm, one in ke:
            for h in Hb1:
                cons.setdefault(add(h, k), []).append(("Y%s" % hn(h), nm, one and sum(k) % 2 == 0))
        for r in kax:
            for k, nm, one in kd[r]:
                for h in Hb:
                    cons.setdefault(add(h, k), []).append(("W%d_%s" % (r, hn(h)), nm, False))
        need = set(cons)
        gen_R(em, L, need, emit_use=lambda key, rn: [
            em("%s += %s;" % (dst, rn) if one else "%s = fma(%s, %s, %s);" % (dst, nm, rn, dst)) for dst, nm, one in cons.get(key, [])])
        dot = lambda xs: "".join("fma(%s, %s, " % x for x in xs[:-1]) + "%s * %s" % xs[-1] + ")" * (len(xs) - 1)
        em("const double e = %s;" % dot([("U%s" % hn(h), "Y%s" % hn(h)) for h in Hb]))
        em("const double ra = br[5], rb = 1.0 - ra;")
        for r in range(3):
            em("{")
            em("  const double fp = %s;" % dot([("U%s" % hn(h), "Y%s" % hn(add(h, tuple(int(x == r) for x in range(3))))) for h in Hb]))
            em("  const double fab = %s;" % ("fma(-br[6 + p%d], e, %s)" % (r, dot([("V%d_%s" % (r, hn(h)), "Y%s" % hn(h)) for h in Hbd]))
                                             if r in daxes else "-br[6 + p%d] * e" % r))
            em("  const double fcd = %s;" % ("fma(-kj[(12 + p%d) * kS], e, %s)" % (r, dot([("U%s" % hn(h), "W%d_%s" % (r, hn(h))) for h in Hb]))
                                             if r in kax else "-kj[(12 + p%d) * kS] * e" % r))
            em("  A%d += fma(ra, fp, fab); B%d += fma(rb, fp, -fab); C%d += fma(-rc, fp, fcd);" % (r, r, r))
            em("}")
        em.ind -= 1
        em("}")
        em.ind -= 1
        em("}")
        em.ind -= 1
        em("} break;")
    em("}")
    em.ind -= 1
    em("}")
    em.ind -= 1
    em("}")
    # every lane shares the bra atoms: one atomic per warp and component; the sums go to one of
    # `ncopy` copies of the gradient, which has only 3 natom addresses
    em("double* __restrict__ g = a.grad + (size_t)((blockIdx.x + 5 * blockIdx.y) % a.ncopy) * a.stride;")
    for r in range(3):
        em("{ const double va = sqb::warp_sum(A%d), vb = sqb::warp_sum(B%d);" % (r, r))
        em("  if ((threadIdx.x & 31) == 0) { atomicAdd(g + 3 * bp.atP + p%d, va); atomicAdd(g + 3 * bp.atQ + p%d, vb); } }" % (r, r))
    em("if (ok) {")
    for r in range(3):
        em("  atomicAdd(g + 3 * kp.atP + p%d, C%d); atomicAdd(g + 3 * kp.atQ + p%d, -(A%d + B%d + C%d));" % (r, r, r, r, r, r))
    em("}")
    out += em.lines
    out.append("}")
    ops = 60 + 6 * L + 3 * len(simplex(L)) + 10 * na * nb + 4 * len(Hb) * na * nb // 2
    return "\n".join(out) + "\n", {"name": name, "bra": bra, "ket": ket, "nb": NB, "passes": len(cds), "ops": ops}


def main():
    outdir = sys.argv[1] if len(sys.argv) > 1 else os.path.join(os.path.dirname(os.path.abspath(__file__)), "gen_grad")
    os.makedirs(outdir, exist_ok=True)
    head = "// generated by gen_grad_kernels.py -- do not edit\n#include \"../grad_common.cuh\"\n\n"
    files, reg = [], []
    for x, y in quartet_classes():
        bra, ket = roles(x, y)
        # one kernel per orbit where the whole class is more code than ptxas allocates registers for
        # ((dd|dd) in one kernel: 18 KB of stack a thread, 1.07 ms for an organic of 8 heavy atoms)
        parts = range(len(ket_orbits(ket)[0])) if pair_L(bra) + pair_L(ket) >= 8 else [None]
        for only in parts:
            src, m = gen_grad(bra, ket, only)
            write_if_changed(os.path.join(outdir, m["name"] + ".cu"), head + src)
            files.append(m["name"] + ".cu")
            reg.append(m)
    text = head + "".join('extern "C" __global__ void %s(const sqb::GradArgs, const sqb::WorkItem*);\n' % m["name"] for m in reg)
    text += "\nnamespace sqb {\nconst GradKernel kGradKernels[%d] = {\n" % len(reg)
    for m in reg:
        text += "  {%d, %d, (const void*)%s, %d, %d, %d},\n" % (PAIRS.index(m["bra"]), PAIRS.index(m["ket"]), m["name"],
                                                              m["passes"], m["nb"], m["ops"])
    text += "};\nconst int kNumGradKernels = %d;\n}  // namespace sqb\n" % len(reg)
    write_if_changed(os.path.join(outdir, "grad_registry.cu"), text)
    files.append("grad_registry.cu")
    for fn in os.listdir(outdir):
        if fn.endswith(".cu") and fn not in files:
            os.remove(os.path.join(outdir, fn))
    write_if_changed(os.path.join(outdir, "files.txt"), "\n".join(files) + "\n")
    print("generated %d gradient kernels" % len(reg))


if __name__ == "__main__":
    main()
