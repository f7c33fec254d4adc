"""Generate the J/K kernels of shell quartets with an f shell in the canonical layouts.

One kernel per bra pair class (f shell | s, sp, p, d or f shell) and block of its function pairs;
the ket pair's angular momenta are run-time values.  A lane holds one ket function pair (c, d) of one
quartet, and a warp as many quartets as fit: 32 / g for kets of g function pairs (larger kets in
chunks), all with one bra pair, kets of one type and contraction length.  Per primitive quartet the
lanes of a quartet build its Hermite integrals R in shared memory (a box [t][u][v], in place, level
by level), and every lane sums its own function pair's ket side over them,

    G[h] += sum_k (-1)^|k| E_cd[k] R[h + k],

with the bra's Hermite indices h unrolled (G in registers, one shared-memory load and one FMA per
term) and the lane's k in a run-time loop; once per bra primitive G is transformed by the bra's
Hermite coefficients, straight-line code with the sparsity of each component, into the lane's
column of the contracted block.  The one-warp-per-quartet kernel (jk_generic.cu) ran both sums with
run-time loops on both sides, about one operation per warp instruction, and left most lanes of a
small quartet idle; it keeps the multipole mode and other shell layouts.

Usage: python gen_fshell_kernels.py <outdir>
"""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from gen_jk_kernels import COMP, Emitter, write_if_changed  # noqa: E402

F = [(3, 0, 0), (0, 3, 0), (0, 0, 3), (2, 1, 0), (1, 2, 0), (2, 0, 1), (1, 0, 2), (0, 2, 1), (0, 1, 2), (1, 1, 1)]
SHELL = dict(COMP, F=F)
LMAX = {"S": 0, "L": 1, "P": 1, "D": 2, "F": 3}
# function pairs of one pass: blocks of the f shell's functions, so that G and the block's
# accumulators take at most about 100 doubles of a thread
NBLOCK = {"S": 1, "L": 2, "P": 1, "D": 2, "F": 5}
WARPS = 4


def simplex(L):
    return [(n - m, m - v, v) for n in range(L + 1) for m in range(n + 1) for v in range(m + 1)]


def gen_kernel(qt, blk):
    B = SHELL[qt]
    nb, LA = len(B), 3 + LMAX[qt]
    per = 10 // NBLOCK[qt]
    fa = list(range(blk * per, (blk + 1) * per))
    H = simplex(LA)
    hn = lambda h: "%d%d%d" % h
    lq1, lt = LMAX[qt] + 1, 3 + LMAX[qt] + 1
    sz = 4 * lq1 * lt
    name = "jkf_F%s_%d" % (qt, blk)
    em = Emitter()
    em("extern __shared__ double fsm[];")
    em("const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;")
    em("const long long unit = u0 + (long long)blockIdx.x * %d + wp;" % WARPS)
    em("if (unit >= nunits) return;                   // whole warps leave")
    em("const sqb::FUnit it = sqb::f_unit(runs, first, nruns, unit);")
    em("const int g = it.cg >> 16, s = lane / g, cc = lane - s * g, cd = (it.cg & 0xffff) + cc;")
    em("const sqb::GenPairRec A = a.pairs[it.bra];")
    em("const int kb = a.klist[it.k0 + min(s, it.cnt - 1)];   // idle lanes shadow the last ket")
    em("const sqb::GenPairRec B = a.pairs[kb];")
    em("const double r = A.schwarz * B.schwarz;")
    em("bool ok = s < it.cnt && !(r < a.b.cut_outer) && !(r < a.b.cut_fixed);")
    em("if (ok && r < a.b.dscreen_rmax) {")
    em("  const bool bf = (A.P > B.P) || (A.P == B.P && A.Q >= B.Q);")
    em("  const int P = bf ? A.P : B.P, Q = bf ? A.Q : B.Q, I = bf ? B.P : A.P, J = bf ? B.Q : A.Q;")
    em("  const double* PM = a.b.PM; const int ns = a.b.ns;")
    em("  const double mp = PM[P * ns + Q] + PM[I * ns + J] + PM[P * ns + I] + PM[P * ns + J] + PM[Q * ns + I] + PM[Q * ns + J];")
    em("  ok = !(r * mp < a.b.cut_fixed);")
    em("}")
    em("if (!__any_sync(0xffffffffu, ok)) return;")
    em("const double deg = (A.P == A.Q ? 0.5 : 1.0) * (B.P == B.Q ? 0.5 : 1.0) * (kb == it.bra ? 0.5 : 1.0);")
    em("const int L = %d + B.lP + B.lQ, S1 = L + 1, S2 = S1 * S1;   // uniform over the warp" % LA)
    em("double* __restrict__ box = fsm + wp * sqb::kFWarpDoubles + min(s, it.cnt - 1) * sqb::f_slot(L);   // [t][u][v], then the seeds")
    em("double* __restrict__ base = box + S1 * S2;")
    em("const bool mine = s < it.cnt;")
    em("const unsigned d = __ldg(a.desc + B.doff + cd);")
    em("const int cx = sqb::dsc(d, 0), dx = sqb::dsc(d, 1), cy = sqb::dsc(d, 2), dy = sqb::dsc(d, 3), cz = sqb::dsc(d, 4), dz = sqb::dsc(d, 5);")
    em("const int n1 = cy + dy + 1, n2 = cz + dz + 1, nk = (cx + dx + 1) * n1 * n2;")
    em("unsigned long long npq = 0, nfl = 0;")
    for a_ in fa:
        for b_ in range(nb):
            em("double o%d_%d = 0.0;" % (a_, b_))
    em("const int gi = it.gi, gj = it.gj, si = it.si, sj = it.sj;")
    em("for (int i = gi; i < A.nprim; i += si) {      // this unit's part of the primitives")
    em.ind += 1
    em("const double* pa = a.prims + (size_t)(A.poff + i) * sqb::kGenPrimStride;")
    em("const double p = pa[0], Px = pa[1], Py = pa[2], Pz = pa[3], kpa = pa[4];")
    for h in H:
        em("double g%s = 0.0;" % hn(h))
    em("bool any = false;")
    em("for (int j = gj; j < B.nprim; j += sj) {     // one contraction length per warp")
    em.ind += 1
    em("const double* pb = a.prims + (size_t)(B.poff + j) * sqb::kGenPrimStride;")
    em("const double q = pb[0], pq = p + q, rs = rsqrt(pq);")
    em("const bool live = ok && !(TWO_PI_2_5 * kpa * pb[4] * rs < PRIM_CUTOFF);")
    em("if (!__any_sync(0xffffffffu, live)) continue;")
    em("any = true;")
    em("if (live && cd == 0%s) ++npq;" % ("" if blk == 0 else " && false"))
    em("const double X = Px - pb[1], Y = Py - pb[2], Z = Pz - pb[3];")
    em("__syncwarp();                                // the previous step is done with the box")
    em("if (mine) sqb::f_seeds(L, p * q * (rs * rs), rs, X, Y, Z, a.boys, base, cc, g);")
    em("__syncwarp();")
    em("sqb::f_box(L, X, Y, Z, base, box, cc, g, mine);")
    em("if (live) {")
    em.ind += 1
    em("const sqb::EView Ej(a.coef, pb, B);")
    em("const double *ex = Ej.ax(0, cx, dx), *ey = Ej.ax(1, cy, dy), *ez = Ej.ax(2, cz, dz);")
    em("const double w = Ej.w(cd);")
    em("int tau = 0, nu = 0, ph = 0;")
    em("for (int k = 0; k < nk; ++k) {")
    em.ind += 1
    em("const double e0 = w * (__ldg(ex + tau) * __ldg(ey + nu)) * __ldg(ez + ph);")
    em("const double e = ((tau + nu + ph) & 1) ? -e0 : e0;")
    em("const double* __restrict__ R = box + tau * S2 + nu * S1 + ph;")
    for t in range(LA + 1):
        for u in range(LA + 1 - t):
            em("{ const double* __restrict__ x = R + %d * S2 + %d * S1;" % (t, u))
            for v in range(LA + 1 - t - u):
                em("  g%s = fma(e, x[%d], g%s);" % (hn((t, u, v)), v, hn((t, u, v))))
            em("}")
    em("if (++ph == n2) { ph = 0; if (++nu == n1) { nu = 0; ++tau; } }")
    em.ind -= 1
    em("}")
    em("nfl += 2ull * %d * nk;" % len(H))
    em.ind -= 1
    em("}")
    em.ind -= 1
    em("}")
    em("if (!any) continue;")
    # bra transform: o[ab] += w_ab sum_t Ex[t] sum_u Ey[u] sum_v Ez[v] g[tuv]
    em("const sqb::EView Ei(a.coef, pa, A);")
    em("const double* __restrict__ E = Ei.e;")
    fl = 0
    for a_ in fa:
        la = F[a_]
        for b_ in range(nb):
            lb = B[b_]
            n = [la[x] + lb[x] for x in range(3)]
            e = lambda x, t: "__ldg(E + %d)" % (x * sz + (la[x] * lq1 + lb[x]) * lt + t)
            em("{ double z = 0.0;")
            for t in range(n[0] + 1):
                for u in range(n[1] + 1):
                    if n[2] == 0:
                        sv = "g%s" % hn((t, u, 0))
                    else:
                        sv = "%s * g%s" % (e(2, 0), hn((t, u, 0)))
                        for v in range(1, n[2] + 1):
                            sv = "fma(%s, g%s, %s)" % (e(2, v), hn((t, u, v)), sv)
                    f = " * ".join(([e(0, t)] if n[0] else []) + ([e(1, u)] if n[1] else []))
                    em("  z = fma(%s, %s, z);" % (f, sv) if f else "  z += %s;" % sv)
                    fl += 2 * (n[2] + 2)
            em("  o%d_%d = fma(Ei.w(%d), z, o%d_%d); }" % (a_, b_, a_ * nb + b_, a_, b_))
            fl += 2
    em("if (ok) nfl += %d;" % fl)
    em.ind -= 1
    em("}")
    # digestion
    em("const int N = a.b.nbf, fP = A.fP, fQ = A.fQ;")
    em("const int fc = B.fP + cd / B.nfQ, fd = B.fQ + cd %% B.nfQ;".replace("%%", "%"))
    em("const double* __restrict__ PT = a.b.PT;")
    em("const double s2 = 2.0 * deg;")
    ab = [(x, y) for x in fa for y in range(nb)]
    em("if (ok) {")
    em.ind += 1
    em("double z = 0.0;")
    for x, y in ab:
        em("z = fma(o%d_%d, __ldg(PT + (fP + %d) * N + fQ + %d), z);" % (x, y, x, y))
    em("atomicAdd(a.b.J + fc * N + fd, s2 * z);")
    em("for (int sp = 0; sp < (a.b.uhf ? 2 : 1); ++sp) {")
    em.ind += 1
    em("const double* __restrict__ D = sp ? a.b.PB : a.b.PA;")
    em("double* __restrict__ K = sp ? a.b.KB : a.b.KA;")
    for src, dst in (("d", "c"), ("c", "d")):
        em("{  // K[p][%s], K[q][%s] from D[.][%s]" % (dst, dst, src))
        for y in range(nb):
            em("  const double q%d = D[(fQ + %d) * N + f%s];" % (y, y, src))
            em("  double kq%d = 0.0;" % y)
        for x in fa:
            em("  { const double px = D[(fP + %d) * N + f%s]; double kp = 0.0;" % (x, src))
            for y in range(nb):
                em("    kp = fma(o%d_%d, q%d, kp); kq%d = fma(o%d_%d, px, kq%d);" % (x, y, y, y, x, y, y))
            em("    atomicAdd(K + (fP + %d) * N + f%s, deg * kp); }" % (x, dst))
        for y in range(nb):
            em("  atomicAdd(K + (fQ + %d) * N + f%s, deg * kq%d);" % (y, dst, y))
        em("}")
    em.ind -= 1
    em("}")
    em("nfl += 2ull * %d * (2 + 4 * (a.b.uhf ? 2 : 1));" % len(ab))
    em.ind -= 1
    em("}")
    em("{  // J[p][q]: every lane shares the bra pair")
    em("  const double w = ok ? s2 * __ldg(PT + fc * N + fd) : 0.0;")
    for s0 in range(0, len(ab), 32):
        part = ab[s0:s0 + 32]
        M = 1
        while M < len(part):
            M *= 2
        em("  { double v[%d] = {%s};" % (M, ", ".join(["w * o%d_%d" % x for x in part] + ["0.0"] * (M - len(part)))))
        em("    const double z = sqb::warp_sum_scatter<%d>(v); const int x = lane + %d;" % (M, s0))
        em("    if (lane < %d && z != 0.0) atomicAdd(a.b.J + (fP + %d + x / %d) * N + fQ + x %% %d, z); }" % (len(part), fa[0], nb, nb))
    em("}")
    em("sqb::count_add(a.counters + 0, ok && cd == 0%s ? 1ull : 0ull);" % (" && gi == 0 && gj == 0" if blk == 0 else " && false"))
    em("sqb::count_add(a.counters + 1, npq);")
    em("sqb::count_add(a.counters + 2, nfl);")
    out = ['extern "C" __global__ void __launch_bounds__(%d)' % (32 * WARPS),
           "%s(const sqb::FArgs a, const sqb::FRun* __restrict__ runs, const long long* __restrict__ first, int nruns," % name,
           "   long long u0, long long nunits) {"] + em.lines + ["}"]
    return name, "\n".join(out) + "\n"


def main():
    outdir = sys.argv[1] if len(sys.argv) > 1 else os.path.join(os.path.dirname(os.path.abspath(__file__)), "gen_fshell")
    os.makedirs(outdir, exist_ok=True)
    head = "// generated by gen_fshell_kernels.py -- do not edit\n#include \"../jk_generic_dev.cuh\"\n\n"
    files, reg = [], []
    for qt in "SLPDF":
        for blk in range(NBLOCK[qt]):
            name, src = gen_kernel(qt, blk)
            write_if_changed(os.path.join(outdir, name + ".cu"), head + src)
            files.append(name + ".cu")
            reg.append((qt, name))
    text = head + "".join('extern "C" __global__ void %s(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);\n' % n for _, n in reg)
    text += "\nnamespace sqb {\nconst FKernel kFKernels[%d] = {\n" % len(reg)
    for qt, n in reg:
        text += "  {%d, (const void*)%s},\n" % ("SLPDF".index(qt), n)
    text += "};\nconst int kNumFKernels = %d;\n}  // namespace sqb\n" % len(reg)
    write_if_changed(os.path.join(outdir, "jkf_registry.cu"), text)
    files.append("jkf_registry.cu")
    for fn in os.listdir(outdir):
        if fn.endswith(".cu") and fn not in files:
            os.remove(os.path.join(outdir, fn))
    write_if_changed(os.path.join(outdir, "files.txt"), "\n".join(files) + "\n")
    print("generated %d f-shell kernels" % len(reg))


if __name__ == "__main__":
    main()
