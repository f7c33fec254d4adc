"""Generate the per-class J/K CUDA kernels (McMurchie-Davidson ERI + fused digestion).

One kernel per quartet class (bra pair class | ket pair class) and spin mode (R: restricted,
K from PA only; U: unrestricted, K from PA and PB).  A CTA owns one bra shell pair and as many
ket shell pairs as it has threads (the runtime launches 32, 64 or 128; the bra staging strides
by blockDim.x): one shell quartet per thread, or per si x sj threads that each take a strided
subset of the bra and of the ket primitives (the digestion is linear, so each thread digests
its partial contraction).  For each quartet the threads evaluate

    (ab|cd) = sum_{bra prims i} sum_{tuv} Eb_i[ab][tuv] *
              sum_{ket prims j} sum_{tau nu phi} (-1)^(tau+nu+phi) Ek_j[cd][tau nu phi] R_ij[t+tau, u+nu, v+phi]

where Eb/Ek are Hermite expansion coefficients (with contraction coefficients, exp(-mu R^2)/p
and 1/q folded in, precomputed per primitive pair on the host) and R are the Hermite Coulomb
integrals built from the Boys function.  The inner sum over ket primitives is accumulated in
Hermite space (G[cd][tuv]); the bra transform runs once per bra primitive.  When the per-thread
state would not fit in registers the ket functions are split into blocks ("passes"); each pass
is a separate CTA (blockIdx.y) that repeats the primitive loop for its block.  The contracted
block is digested at once into

    Jacc[ab] += 2 deg PT[cd] v     Jacc[cd] += 2 deg PT[ab] v
    Kacc[ac] += deg P[bd] v        Kacc[bc] += deg P[ad] v
    Kacc[ad] += deg P[bc] v        Kacc[bd] += deg P[ac] v

(deg = 1/2 per coinciding bra shells, ket shells and bra==ket pair), so J = Jacc + Jacc^T and
K = Kacc + Kacc^T.  This reproduces what the reference's storeQuartetEE (src/matrix.c:2934)
accumulates for the six degeneracy cases.

The generator also counts the floating-point operations it emits per primitive quartet, per
bra-primitive flush and per quartet (FMA = 2) and writes that table (jk_flops.json) as the
algorithmic work W(class) used for roofline reporting.

Usage: python gen_jk_kernels.py <outdir>
"""
import itertools
import json
import os
import sys

COMP = {
    "S": [(0, 0, 0)],
    "L": [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)],
    "P": [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
    "D": [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)],
}
LMAX = {"S": 0, "L": 1, "P": 1, "D": 2}
TYPE_ID = {"S": 0, "L": 1, "P": 2, "D": 3}        # reference sort order (src/matrix.h:238-244)
# pair classes (type of the first shell >= type of the second in the reference order)
PAIRS = [a + b for a in "SLPD" for b in "SLPD" if TYPE_ID[a] >= TYPE_ID[b]]
# bra/ket orientation: the larger pair (by functions, then L) is the bra
PAIR_ORDER = sorted(PAIRS, key=lambda p: (len(COMP[p[0]]) * len(COMP[p[1]]), LMAX[p[0]] + LMAX[p[1]], p))
STATE_MAX = int(os.environ.get("SQB_STATE_MAX", "64"))   # doubles of G + out accumulators per pass
# the mixed (FP32) form: floats of G + out per pass (a float takes one register).  LL|LL: 64
# floats -> 8 passes at 188 registers, 96 -> 6 passes at 242, 128 -> 4 passes at 255 with 132 B
# of spills; on C60 (tau 1e-5) 128 floats took the build from 64.4 to 53.5 ms: as for the FP64
# forms, fewer passes pay more than the spills cost
STATE_MAX_F32 = int(os.environ.get("SQB_STATE_MAX_F32", "128"))
# the wide tile: a second FP64 form of every class whose passes it merges (fewer passes, each
# re-deriving the Boys function and R for more ket functions, at more registers); which form a
# class runs is chosen by measurement (sqb200_jk_autotune)
STATE_MAX_WIDE = int(os.environ.get("SQB_STATE_MAX_WIDE", "128"))
# the swapped-role form (outer loop over the thread's ket primitives, inner over the shared bra
# primitives in shared memory): emitted for every class, state budget of its passes
SWAP = int(os.environ.get("SQB_SWAP", "1"))
STATE_MAX_SWAP = int(os.environ.get("SQB_STATE_MAX_SWAP", "128"))
TILE_KETS = int(os.environ.get("SQB_TILE_KETS", "1"))    # passes over (c, d) tiles of the ket functions
F32_MAX_L = 6               # mixed-precision kernels for classes up to this total angular momentum
MIN_BLOCKS = int(os.environ.get("SQB_MINB", "0"))   # __launch_bounds__ min CTAs per SM (0 = none)
# the same bound for the FP64 narrow-tile form only (its state is smallest, so a register cap
# spills least there); 0 = none
MIN_BLOCKS_NARROW = int(os.environ.get("SQB_MINB_NARROW", "0"))
GROUP_MAX = 16             # function quartets of the classes whose split lanes sum before the atomics
CTA = 128
# Register caps (__maxnreg__) for kernels where a cap measured faster on B200: with fewer
# registers per thread more 64-thread CTAs share an SM, which pays where the spills it adds stay
# small.  C60/6-31G build, restricted forms (ms per build, uncapped -> capped): LL|LS wide
# 17.20 -> 16.19 at 128 registers (16.48 at 168, 17.70 at 144, 255 uncapped); LS|LS swapped
# 3.61 -> 3.12 at 128 (144 uncapped, no spills either way; 3.22 at 112).  LL|LL wide stays
# uncapped (40.4 ms; 42.3 at 168, 47.2 at 200).  The unrestricted forms are not capped.
REG_CAP = {"jk_LL_LS_R_w": 128, "jk_LS_LS_R_s": 128}


# The FP64 form a class runs without autotuning: 0 narrow, 1 wide, 2 swapped.  Measured on B200
# (us per launch, narrow / wide / swapped, equal where a class has no wide form):
#   an organic of 14 heavy atoms, 6-31G*: DL|LL 471 / 312 / 346, LL|LL 228 / 175 / 184, DL|DL 248 / 186 / 247,
#   DL|LS 241 / 173 / 222, LL|LS 227 / 182 / 188, LS|SS 111 / 111 / 81, LS|LS 111 / 112 / 94, SS|SS 68 / 67 / 51,
#   DS|LS 93 / 93 / 86, LL|SS 100 / 101 / 82, DS|SS 70 / 70 / 52, DL|DS 144 / 105 / 170, LL|DS 123 / 108 / 141,
#   DL|SS 82 / 83 / 72, DS|DS 57 / 67 / 54, DD|LS 81 / 83 / 138, DD|SS 58 / 58 / 82;
#   of 10 heavy atoms, DZP: DP|PP 397 / 238 / 281, DP|PS 318 / 213 / 291, DP|DP 203 / 175 / 206, DP|DS 197 / 133 /
#   221, PP|PS 352 / 352 / 321, PS|SS 367 / 367 / 308, PS|PS 362 / 362 / 280, PP|SS 161 / 162 / 145, DP|SS 101 /
#   101 / 104, PP|PP 200 / 156 / 173, PP|DS 174 / 164 / 226, DS|DS 74 / 73 / 71; C60/6-31G LL|LL 60 / 39 / 45 ms,
#   LL|LS with its register cap 16 ms wide.
# So: bras of at least 18 functions (DL, DP, DD) take the wide form, narrow where they have none
# (their swapped flush is large), but for DL|SS, swapped; smaller bras take the swapped form on SS, PS
# and LS kets (LL|LS: within 3% of wide), and on the others the wide one, narrow where they have
# none; but for DS|DS, whose second pass gains nothing, narrow.
def default_form(bra, ket, has_wide, has_swap):
    if bra in ("DL", "DP", "DD"):
        if (bra, ket) == ("DL", "SS"):
            return 2
        return 1 if has_wide else 0
    if ket in ("SS", "PS", "LS") and has_swap:
        return 2
    if (bra, ket) == ("DS", "DS"):
        return 0
    return 1 if has_wide else 0


def kernel_qualifiers(name, bounds):
    """The launch qualifier of kernel `name`: its register cap if it has one, else
    __launch_bounds__(bounds)."""
    if name in REG_CAP:
        return "__maxnreg__(%d)" % REG_CAP[name]
    return "__launch_bounds__(%s)" % bounds


def pair_funcs(pc):
    a, b = pc
    return [(ca, cb) for ca in COMP[a] for cb in COMP[b]]


def nz(f):
    (ax, ay, az), (bx, by, bz) = f
    return [(t, u, v) for t in range(ax + bx + 1) for u in range(ay + by + 1) for v in range(az + bz + 1)]


def etable(pc):
    """E-table layout: list of (function index, (t,u,v)) in storage order, and offsets."""
    fs = pair_funcs(pc)
    off, lay = [], []
    for fi, f in enumerate(fs):
        off.append(len(lay))
        for h in nz(f):
            lay.append((fi, h))
    return fs, off, lay


def pair_L(pc):
    return LMAX[pc[0]] + LMAX[pc[1]]


class Emitter:
    def __init__(self):
        self.lines = []
        self.ind = 1

    def __call__(self, s):
        self.lines.append("  " * self.ind + s)


def gen_R(em, L, need, cons=None, emit_use=None, rt="double", fma="fma"):
    """Emit R^{(0)}_{tuv} for (t,u,v) in need; returns flop count and name map.  When
    emit_use is given it is called right after each R^{(0)} value is produced, so its
    consumers follow it and the value dies early (lower register pressure)."""
    have = {}
    flops = [0]

    def get(n, t, u, v):
        key = (n, t, u, v)
        if key in have:
            return have[key]
        if t == 0 and u == 0 and v == 0:
            have[key] = "b%d" % n
            return have[key]
        name = "r%d_%d_%d_%d" % key
        if t > 0:
            d, ax, lo = t, "X", (n + 1, t - 2, u, v)
            hi = (n + 1, t - 1, u, v)
        elif u > 0:
            d, ax, lo = u, "Y", (n + 1, t, u - 2, v)
            hi = (n + 1, t, u - 1, v)
        else:
            d, ax, lo = v, "Z", (n + 1, t, u, v - 2)
            hi = (n + 1, t, u, v - 1)
        h = get(*hi)
        if d - 1 > 0:
            l_ = get(*lo)
            if d - 1 == 1:
                em("const %s %s = %s(%s, %s, %s);" % (rt, name, fma, ax, h, l_))
                flops[0] += 2
            else:
                em("const %s %s = %s(%s, %s, %d.0%s * %s);" % (rt, name, fma, ax, h, d - 1, "f" if rt == "float" else "", l_))
                flops[0] += 3
        else:
            em("const %s %s = %s * %s;" % (rt, name, ax, h))
            flops[0] += 1
        have[key] = name
        return name

    names = {}
    for (t, u, v) in sorted(need, key=lambda x: (sum(x), x)):
        names[(t, u, v)] = get(0, t, u, v)
        if emit_use is not None:
            emit_use((t, u, v), names[(t, u, v)])
    return names, flops[0]


def boys_flops(M):
    # Taylor Horner (9 terms: 8 fma + 8 mul), downward recursion (fma + mul per order),
    # argument setup not counted here
    return 8 * 3 + M * 3


def alg_prim_flops(fk, Hb, rt, fma):
    """Algorithmic operations per primitive quartet of a class: the pass-free algorithm (primitive
    setup, one Boys evaluation at the class's highest Hermite order, every R value once, every
    ket E contraction once).  Passes that re-derive the Boys function and R for another block
    of ket functions emit more operations than this; those repeats are not counted as work."""
    need, ncons = set(), 0
    for f in fk:
        for (tau, nu, phi) in nz(f):
            for h in Hb:
                need.add((h[0] + tau, h[1] + nu, h[2] + phi))
                ncons += 1
    L = max(sum(x) for x in need)
    _, rf = gen_R(Emitter(), L, need, rt=rt, fma=fma)
    return 9 + 2 + 3 + 5 + boys_flops(L) + 2 + L + (L + 1) + rf + 2 * ncons


def ket_per_pass(bra, ket, state_max):
    fb, _, _ = etable(bra)
    fk, _, _ = etable(ket)
    Hb = {h for f in fb for h in nz(f)}
    return min(max(1, state_max // (len(Hb) + len(fb))), len(fk))


def ket_blocks(ncd, nc, nd, per):
    """The ket function pairs cd = c*nd + d of each pass.  Every pass digests into K rows of the
    bra functions at the columns of its distinct c and its distinct d, one atomic per (bra
    function, column) and pass, so a pass covering a tc x td tile of (c, d) adds (tc + td) x
    (bra functions) instead of (1 + per) for a run of one c: tiles when they need no more passes
    than runs of consecutive pairs (TILE_KETS=0 keeps the runs)."""
    runs = [list(range(s, min(ncd, s + per))) for s in range(0, ncd, per)]
    if not TILE_KETS or nc < 2 or nd < 2 or per < 2:
        return runs
    best = None
    for tc in range(1, nc + 1):
        for td in range(1, nd + 1):
            if tc * td > per:
                continue
            npass = -(-nc // tc) * -(-nd // td)
            key = (npass, tc + td)
            if best is None or key < best[0]:
                best = (key, tc, td)
    (npass, _), tc, td = best
    if npass > len(runs):
        return runs
    return [[c * nd + d for c in range(c0, min(nc, c0 + tc)) for d in range(d0, min(nd, d0 + td))]
            for c0 in range(0, nc, tc) for d0 in range(0, nd, td)]


def n_passes(bra, ket, state_max):
    fk, _, _ = etable(ket)
    per = ket_per_pass(bra, ket, state_max)
    return (len(fk) + per - 1) // per


def gen_class(bra, ket, spin, prec="D", state_max=None, suffix=""):
    """Return (kernel source, metadata) for class (bra|ket) and spin 'R' or 'U'.  prec "F"
    emits the mixed form: primitive setup, prefactor cut and Boys function in FP64, Hermite
    integrals, E tables and contracted accumulators in FP32, digestion into the FP64 J/K
    accumulators in FP64."""
    F32 = prec == "F"
    RT = "float" if F32 else "double"
    FMA = "fmaf" if F32 else "fma"
    fb, offb, layb = etable(bra)
    fk, offk, layk = etable(ket)
    nab, ncd = len(fb), len(fk)
    Lb, Lk = pair_L(bra), pair_L(ket)
    Lt = Lb + Lk
    Hb = sorted({h for f in fb for h in nz(f)}, key=lambda x: (sum(x), x))
    hidx = {h: i for i, h in enumerate(Hb)}
    na, nb_ = len(COMP[bra[0]]), len(COMP[bra[1]])
    nc, nd = len(COMP[ket[0]]), len(COMP[ket[1]])
    NB = 5 + len(layb)
    NK = 5 + len(layk)
    per = ket_per_pass(bra, ket, (STATE_MAX_F32 if F32 else STATE_MAX) if state_max is None else state_max)
    blocks = ket_blocks(ncd, len(COMP[ket[0]]), len(COMP[ket[1]]), per)
    name = "jk_%s_%s_%s%s%s" % (bra, ket, spin, "_f32" if F32 else "", suffix)
    MP = not F32 and suffix == ""   # the narrow FP64 form carries the multipole mode
    fl = {"prim": 0, "flush": 0, "quartet": 0, "passes": len(blocks),
          "alg_prim": alg_prim_flops(fk, Hb, RT, FMA)}

    em = Emitter()
    out = []
    minb = MIN_BLOCKS_NARROW if (MIN_BLOCKS_NARROW and suffix == "" and not F32) else MIN_BLOCKS
    out.append('extern "C" __global__ void %s' % kernel_qualifiers(
        name, "%d, %d" % (CTA, minb) if minb else "%d" % CTA))
    out.append("%s(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {" % name)
    if F32:
        em("extern __shared__ float sbra_f32[];")
        em("float* __restrict__ sbra = sbra_f32;")
    else:
        em("extern __shared__ double sbra[];")
    em("const sqb::WorkItem it = items[blockIdx.x];")
    em("const sqb::PairRec bp = a.bra_pairs[it.bra];")
    em("const sqb::MolRec mr = a.mols[it.mol];        // the molecule of this work item")
    em("const long long acc0 = mr.moff + (blockIdx.x & a.copy_mask) * a.copy_stride;   // this item's copy")
    em("double* __restrict__ Jacc = a.Jacc + acc0;")
    em("double* __restrict__ KAacc = a.KAacc + acc0;")
    em("double* __restrict__ KBacc = a.KBacc + acc0;")
    em("const int N = mr.nbf;")
    em("for (int x = threadIdx.x; x < bp.nprim * %d; x += blockDim.x) sbra[x] = a.bra_prims%s[bp.poff + (long long)x * bp.kstride];" % (NB, "_f" if F32 else ""))
    em("__syncthreads();")
    em("// threads sharing one quartet: si strides over the bra primitives x sj over the ket primitives")
    em("const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;")
    em("const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;")
    em("const int gj = grp / si, gi = grp - gj * si;")
    em("const unsigned gmask = isplit >= 32 ? 0xffffffffu : ((1u << isplit) - 1u) << ((threadIdx.x & 31) & ~(isplit - 1));")
    em("const int pass = blockIdx.y;                   // block of ket functions handled by this CTA")
    em("bool ok = kl < it.cnt;")
    em("sqb::PairRec kp = bp;")
    em("double deg = 0.0;")
    if MP:
        em("bool mpq = false;                            // multipole mode: the quartet takes monopole values")
        em("int erx = -1, erexp = sqb::ERR_UNKNOWN;      // its error-bank slot and stored exponent")
    em("if (ok) {")
    em.ind += 1
    em("kp = a.ket_pairs[it.k0 + kl];")
    em("const double r = bp.schwarz * kp.schwarz;")
    em("ok = !(r < mr.cut_outer) && !(r < mr.cut_fixed);")
    if MP:
        em("if (ok && a.erbank) { erx = a.er_items[blockIdx.x] + kl; erexp = a.erbank[erx]; }")
        em("const bool mpc = erexp != sqb::ERR_UNKNOWN && r < a.mp_rmax;   // substitution candidate")
        em("if (ok && (r < mr.dscreen_rmax || mpc)) {")
    else:
        em("if (ok && r < mr.dscreen_rmax) {")
    em("  const bool bf = (bp.P > kp.P) || (bp.P == kp.P && bp.Q >= kp.Q);")
    em("  const int P = bf ? bp.P : kp.P, Q = bf ? bp.Q : kp.Q, I = bf ? kp.P : bp.P, J = bf ? kp.Q : bp.Q;")
    em("  const double* PM = a.PM + mr.pmoff; const int ns = mr.ns;")
    em("  const double mp = PM[P * ns + Q] + PM[I * ns + J] + PM[P * ns + I] + PM[P * ns + J] + PM[Q * ns + I] + PM[Q * ns + J];")
    if MP:
        em("  if (r < mr.dscreen_rmax) ok = !(r * mp < mr.cut_fixed);")
        em("  if (ok && mpc) mpq = a.pow15[erexp - sqb::ERR_MIN] * mp < mr.cut_fixed;")
    else:
        em("  ok = !(r * mp < mr.cut_fixed);")
    em("}")
    em("deg = (bp.P == bp.Q ? 0.5 : 1.0) * (kp.P == kp.Q ? 0.5 : 1.0) * ((a.same_class && it.bra == it.k0 + kl) ? 0.5 : 1.0);")
    em.ind -= 1
    em("}")
    for ab in range(nab):
        em("double jab%d = 0.0;" % ab)
    em("unsigned long long nprimq = 0, nflush = 0;")
    em("if (ok) {")
    em.ind += 1
    em("const %s* __restrict__ kprim = a.ket_prims%s + kp.poff;" % (RT, "_f" if F32 else ""))
    em("const int kS = kp.kstride;                   // distance between the fields of one ket record")
    em("const int nbp = %sbp.nprim, nkp = kp.nprim;" % ("mpq ? 0 : " if MP else ""))
    em("nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;")
    em("const double* __restrict__ PA = a.PA + mr.moff;")
    if spin == "U":
        em("const double* __restrict__ PB = a.PB + mr.moff;")
    em("const double* __restrict__ PT = a.PT + mr.moff;")
    em("switch (pass) {")
    for bi, blk in enumerate(blocks):
        em("case %d: {  // ket functions %s" % (bi, blk))
        em.ind += 1
        for ab in range(nab):
            for cd in blk:
                em("%s o%d_%d = 0;" % (RT, ab, cd))
        # ket E-table entries this block reads
        kent = []
        for cd in blk:
            for k, (tau, nu, phi) in enumerate(nz(fk[cd])):
                kent.append((cd, k, offk[cd] + k, -1 if (tau + nu + phi) % 2 else 1))
        em("for (int i = gi; i < nbp; i += si) {")
        em.ind += 1
        em("const %s* __restrict__ bi = sbra + i * %d;" % (RT, NB))
        em("const %s p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];" % RT)
        for cd in blk:
            for h in Hb:
                em("%s g%d_%d = 0;" % (RT, cd, hidx[h]))
        em("for (int j = gj; j < nkp; j += sj) {")
        em.ind += 1
        if F32:
            # the mixed form: every step in FP32 (records, set-up, Boys function, recursion,
            # contraction); only the digestion adds into the FP64 accumulators
            em("const float* __restrict__ kj = kprim + (long long)j * %d * kS;" % NK)
            em("const float q = kj[0];")
            em("const float pq = p + q;")
            em("const float rs = rsqrtf(pq);")
            em("if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;")
        else:
            em("const %s* __restrict__ kj = kprim + (long long)j * %d * kS;" % (RT, NK))
            em("const double q = kj[0];")
            em("const double pq = p + q;")
            em("const double rs = rsqrt(pq);")
            em("if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;")
        if bi == 0:
            em("++nprimq;")   # counted by the pass-0 CTAs only
        em("const %s alpha = p * q * (rs * rs);" % RT)
        em("const %s X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];" % RT)
        em("const %s T = alpha * %s(X, X, %s(Y, Y, Z * Z));" % (RT, FMA, FMA))
        need = set()
        for cd in blk:
            for (tau, nu, phi) in nz(fk[cd]):
                for h in Hb:
                    need.add((h[0] + tau, h[1] + nu, h[2] + phi))
        Lp = max(sum(x) for x in need)          # highest Hermite order this pass needs
        if F32:
            em("float F[%d];" % (Lp + 1))
            em("sqb::boysf<%d>(T, a.boys_tab_f, F);" % Lp)
            em("const float s0 = TWO_PI_2_5F * rs;")
            em("const float m2a = -2.0f * alpha;")
            em("float w = s0;")
        else:
            em("double F[%d];" % (Lp + 1))
            em("sqb::boys<%d>(T, a.boys_tab, F);" % Lp)
            em("const double s0 = TWO_PI_2_5 * rs;")
            em("const double m2a = -2.0 * alpha;")
            em("double w = s0;")
        pf = 9 + 2 + 3 + 5 + boys_flops(Lp) + 2  # setup: pq, alpha, XYZ diff, T, s0, m2a
        for n in range(Lp + 1):
            if n > 0:
                em("w *= m2a;")
                pf += 1
            em("const %s b%d = w * F[%d];" % (RT, n, n))
            pf += 1
        # ket E coefficients of this block, signed by (-1)^(tau+nu+phi)
        for (cd, k, e, sg) in kent:
            em("const %s ek%d_%d = %skj[%d * kS];" % (RT, cd, k, "-" if sg < 0 else "", 5 + e))
        # consumers of each R value: (cd, k, h) with h + (tau nu phi) = R index
        cons = {}
        for cd in blk:
            for k, (tau, nu, phi) in enumerate(nz(fk[cd])):
                for h in Hb:
                    cons.setdefault((h[0] + tau, h[1] + nu, h[2] + phi), []).append((cd, k, h))
        rn, rf = gen_R(em, Lp, need, cons=cons, emit_use=lambda key, name: [
            (em("g%d_%d = %s(ek%d_%d, %s, g%d_%d);" % (cd, hidx[h], FMA, cd, k, name, cd, hidx[h])))
            for (cd, k, h) in cons.get(key, [])], rt=RT, fma=FMA)
        pf += rf + 2 * sum(len(v) for v in cons.values())
        em.ind -= 1
        em("}")
        # flush: o[ab][cd] += sum_h Eb[ab][h] g[cd][h]
        ff = 0
        for ab in range(nab):
            for k, h in enumerate(nz(fb[ab])):
                e = offb[ab] + k
                em("{ const %s eb = bi[%d];" % (RT, 5 + e))
                for cd in blk:
                    em("  o%d_%d = %s(eb, g%d_%d, o%d_%d);" % (ab, cd, FMA, cd, hidx[h], ab, cd))
                    ff += 2
                em("}")
        em.ind -= 1
        em("}")
        fl["prim"] += pf
        fl["flush"] += ff
        if MP:
            emit_multipole(em, blk, nab, nb_, nd)
        # digestion of this block
        qf = emit_digest(em, spin, blk, nab, na, nb_, nd, ncd)
        fl["quartet"] += qf
        em.ind -= 1
        em("} break;")
    em("}")
    em.ind -= 1
    em("}")
    # bra J: warp reduce (every lane shares the bra pair)
    emit_bra_j(em, list(range(nab)), nb_)
    em("sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);")
    em("sqb::count_add(a.counters + 1, nprimq);")
    em("sqb::count_add(a.counters + 2, nflush);")
    em("sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);")
    out.extend(persistent_body(em.lines))
    out.append("}")
    meta = {"name": name, "bra": bra, "ket": ket, "spin": spin, "nab": nab, "ncd": ncd,
            "neb": len(layb), "nek": len(layk), "Lt": Lt, "flops": fl}
    return "\n".join(out) + "\n", meta


def persistent_body(lines):
    """Wrap a class kernel's body in the work loop of the persistent launch.  A work unit is one
    (work item, pass) pair.  With a.queue null the CTA runs the unit (blockIdx.x, blockIdx.y)
    and stops (one CTA per unit); otherwise a grid of about one CTA per resident slot takes
    units from the device counter a.queue until the a.nqueue units are taken.  Unit q is item
    q % nitems of pass q / nitems -- the order in which the hardware hands out the CTAs of a
    (items x passes) grid, heaviest items first in each pass -- so that the CTAs running at one
    time work on different items: the passes of one item digest into the same exchange
    elements, and running them side by side would queue their atomics on the same addresses."""
    body = [l.replace("blockIdx.x", "qi_").replace("blockIdx.y", "qp_") for l in lines]
    out = ["  __shared__ int q_next;",
           "  const bool persistent = a.queue != nullptr;",
           "  for (int round = 0;; ++round) {",
           "    int qi_, qp_;",
           "    if (persistent) {",
           "      __syncthreads();                  // the previous unit is done with shared memory",
           "      if (threadIdx.x == 0) q_next = (int)atomicAdd(a.queue, 1ull);",
           "      __syncthreads();",
           "      const int q = q_next;",
           "      if (q >= a.nqueue) break;",
           "      const int nitems = a.nqueue / a.npass;",
           "      qp_ = q / nitems;",
           "      qi_ = q - qp_ * nitems;",
           "    } else {",
           "      if (round > 0) break;",
           "      qi_ = blockIdx.x;",
           "      qp_ = blockIdx.y;",
           "    }",
           "    {"]
    out += ["    " + l for l in body]
    out += ["    }", "  }"]
    return out


def swap_worthwhile(bra, ket):
    """The swapped form is emitted where a pass can hold at least two bra functions (or the only
    one) and the class needs at most 8 passes (beyond that the code size grows past what ptxas
    compiles in reasonable time, and the form repeats the Boys function and R too often to pay)."""
    fb, _, _ = etable(bra)
    fk, _, _ = etable(ket)
    Hk = {h for f in fk for h in nz(f)}
    per = min(len(fb), STATE_MAX_SWAP // (len(Hk) + len(fk)))
    return per >= min(2, len(fb)) and (len(fb) + per - 1) // per <= 8


def gen_class_swap(bra, ket, spin, state_max):
    """The class kernel with the loop roles swapped (suffix _s): the outer loop runs over the
    primitives of the thread's own ket pair (each record read from global memory once per pass),
    the inner loop over the CTA-shared bra pair's primitives in shared memory (broadcast reads).
    The inner loop contracts the bra E tables, G[ab][k] = sum_i sum_h Eb_i[ab][h] R_{h+k}; after
    it, the ket E tables flush, out[ab][cd] += sum_k (-1)^|k| Ek_j[cd][k] G[ab][k].  Passes
    (grid.y) split the bra functions: G + out of one pass <= state_max doubles.  FP64 only."""
    fb, offb, layb = etable(bra)
    fk, offk, layk = etable(ket)
    nab, ncd = len(fb), len(fk)
    Hk = sorted({h for f in fk for h in nz(f)}, key=lambda x: (sum(x), x))
    kidx = {h: i for i, h in enumerate(Hk)}
    na, nb_ = len(COMP[bra[0]]), len(COMP[bra[1]])
    nc, nd = len(COMP[ket[0]]), len(COMP[ket[1]])
    NB = 5 + len(layb)
    NK = 5 + len(layk)
    per = max(1, min(nab, state_max // (len(Hk) + ncd)))
    blocks = [list(range(s0, min(nab, s0 + per))) for s0 in range(0, nab, per)]
    name = "jk_%s_%s_%s_s" % (bra, ket, spin)
    Hb_all = sorted({h for f in fb for h in nz(f)}, key=lambda x: (sum(x), x))
    fl = {"prim": 0, "flush": 0, "quartet": 0, "passes": len(blocks),
          "alg_prim": alg_prim_flops(fk, Hb_all, "double", "fma")}
    em = Emitter()
    out = ['extern "C" __global__ void %s' % kernel_qualifiers(name, "%d" % CTA),
           "%s(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {" % name]
    em("extern __shared__ double sbra[];")
    em("const sqb::WorkItem it = items[blockIdx.x];")
    em("const sqb::PairRec bp = a.bra_pairs[it.bra];")
    em("const sqb::MolRec mr = a.mols[it.mol];        // the molecule of this work item")
    em("const long long acc0 = mr.moff + (blockIdx.x & a.copy_mask) * a.copy_stride;   // this item's copy")
    em("double* __restrict__ Jacc = a.Jacc + acc0;")
    em("double* __restrict__ KAacc = a.KAacc + acc0;")
    em("double* __restrict__ KBacc = a.KBacc + acc0;")
    em("const int N = mr.nbf;")
    em("for (int x = threadIdx.x; x < bp.nprim * %d; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];" % NB)
    em("__syncthreads();")
    em("// threads sharing one quartet: si strides over the bra primitives x sj over the ket primitives")
    em("const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;")
    em("const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;")
    em("const int gj = grp / si, gi = grp - gj * si;")
    em("const unsigned gmask = isplit >= 32 ? 0xffffffffu : ((1u << isplit) - 1u) << ((threadIdx.x & 31) & ~(isplit - 1));")
    em("const int pass = blockIdx.y;                   // block of bra functions handled by this CTA")
    em("bool ok = kl < it.cnt;")
    em("sqb::PairRec kp = bp;")
    em("double deg = 0.0;")
    em("if (ok) {")
    em.ind += 1
    em("kp = a.ket_pairs[it.k0 + kl];")
    em("const double r = bp.schwarz * kp.schwarz;")
    em("ok = !(r < mr.cut_outer) && !(r < mr.cut_fixed);")
    em("if (ok && r < mr.dscreen_rmax) {")
    em("  const bool bf = (bp.P > kp.P) || (bp.P == kp.P && bp.Q >= kp.Q);")
    em("  const int P = bf ? bp.P : kp.P, Q = bf ? bp.Q : kp.Q, I = bf ? kp.P : bp.P, J = bf ? kp.Q : bp.Q;")
    em("  const double* PM = a.PM + mr.pmoff; const int ns = mr.ns;")
    em("  const double mp = PM[P * ns + Q] + PM[I * ns + J] + PM[P * ns + I] + PM[P * ns + J] + PM[Q * ns + I] + PM[Q * ns + J];")
    em("  ok = !(r * mp < mr.cut_fixed);")
    em("}")
    em("deg = (bp.P == bp.Q ? 0.5 : 1.0) * (kp.P == kp.Q ? 0.5 : 1.0) * ((a.same_class && it.bra == it.k0 + kl) ? 0.5 : 1.0);")
    em.ind -= 1
    em("}")
    for ab in range(nab):
        em("double jab%d = 0.0;" % ab)
    em("unsigned long long nprimq = 0, nflush = 0;")
    em("if (ok) {")
    em.ind += 1
    em("const double* __restrict__ kprim = a.ket_prims + kp.poff;")
    em("const int kS = kp.kstride;                   // distance between the fields of one ket record")
    em("const int nbp = bp.nprim, nkp = kp.nprim;")
    em("nflush = pass == 0 && gj < nkp ? (unsigned long long)((nkp - gj + sj - 1) / sj) : 0ull;")
    em("const double* __restrict__ PA = a.PA + mr.moff;")
    if spin == "U":
        em("const double* __restrict__ PB = a.PB + mr.moff;")
    em("const double* __restrict__ PT = a.PT + mr.moff;")
    em("switch (pass) {")
    for bi, blk in enumerate(blocks):
        em("case %d: {  // bra functions %s" % (bi, blk))
        em.ind += 1
        for ab in blk:
            for cd in range(ncd):
                em("double o%d_%d = 0;" % (ab, cd))
        em("for (int j = gj; j < nkp; j += sj) {")
        em.ind += 1
        em("const double* __restrict__ kj = kprim + (long long)j * %d * kS;" % NK)
        em("const double q = kj[0], Qx = kj[kS], Qy = kj[2 * kS], Qz = kj[3 * kS], kq = kj[4 * kS];")
        for ab in blk:
            for k in Hk:
                em("double g%d_%d = 0;" % (ab, kidx[k]))
        # bra E-table entries this block reads (from shared memory, inside the inner loop)
        bent = []
        for ab in blk:
            for e, h in enumerate(nz(fb[ab])):
                bent.append((ab, e, h))
        em("for (int i = gi; i < nbp; i += si) {")
        em.ind += 1
        em("const double* __restrict__ bi = sbra + i * %d;" % NB)
        em("const double p = bi[0];")
        em("const double pq = p + q;")
        em("const double rs = rsqrt(pq);")
        em("if (TWO_PI_2_5 * bi[4] * kq * rs < PRIM_CUTOFF) continue;")
        if bi == 0:
            em("++nprimq;")
        em("const double alpha = p * q * (rs * rs);")
        em("const double X = bi[1] - Qx, Y = bi[2] - Qy, Z = bi[3] - Qz;")
        em("const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));")
        need = set()
        cons = {}
        for (ab, e, h) in bent:
            for k in Hk:
                key = (h[0] + k[0], h[1] + k[1], h[2] + k[2])
                need.add(key)
                cons.setdefault(key, []).append((ab, e, k))
        Lp = max(sum(x) for x in need)
        em("double F[%d];" % (Lp + 1))
        em("sqb::boys<%d>(T, a.boys_tab, F);" % Lp)
        em("const double s0 = TWO_PI_2_5 * rs;")
        em("const double m2a = -2.0 * alpha;")
        em("double w = s0;")
        pf = 9 + 2 + 3 + 5 + boys_flops(Lp) + 2
        for n in range(Lp + 1):
            if n > 0:
                em("w *= m2a;")
                pf += 1
            em("const double b%d = w * F[%d];" % (n, n))
            pf += 1
        for (ab, e, h) in bent:
            em("const double eb%d_%d = bi[%d];" % (ab, e, 5 + offb[ab] + e))
        rn, rf = gen_R(em, Lp, need, cons=cons, emit_use=lambda key, nm: [
            em("g%d_%d = fma(eb%d_%d, %s, g%d_%d);" % (ab, kidx[k], ab, e, nm, ab, kidx[k]))
            for (ab, e, k) in cons.get(key, [])], rt="double", fma="fma")
        pf += rf + 2 * sum(len(v) for v in cons.values())
        em.ind -= 1
        em("}")
        # flush with the ket E tables (signed by (-1)^(tau+nu+phi))
        ff = 0
        for cd in range(ncd):
            for e, k in enumerate(nz(fk[cd])):
                sg = "-" if sum(k) % 2 else ""
                em("{ const double ek = %skj[%d * kS];" % (sg, 5 + offk[cd] + e))
                for ab in blk:
                    em("  o%d_%d = fma(ek, g%d_%d, o%d_%d);" % (ab, cd, ab, kidx[k], ab, cd))
                    ff += 2
                em("}")
        em.ind -= 1
        em("}")
        fl["prim"] += pf
        fl["flush"] += ff
        qf = emit_digest(em, spin, list(range(ncd)), nab, na, nb_, nd, ncd, ablk=blk)
        fl["quartet"] += qf
        em.ind -= 1
        em("} break;")
    em("}")
    em.ind -= 1
    em("}")
    em("switch (pass) {")
    for bi, blk in enumerate(blocks):
        em("case %d:" % bi)
        emit_bra_j(em, blk, nb_)
        em("break;")
    em("}")
    em("sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);")
    em("sqb::count_add(a.counters + 1, nprimq);")
    em("sqb::count_add(a.counters + 2, nflush);")
    em("sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);")
    out.extend(persistent_body(em.lines))
    out.append("}")
    meta = {"name": name, "bra": bra, "ket": ket, "spin": spin, "nab": nab, "ncd": ncd,
            "neb": len(layb), "nek": len(layk), "Lt": pair_L(bra) + pair_L(ket), "flops": fl}
    return "\n".join(out) + "\n", meta


def emit_bra_j(em, blk, nb_):
    """Add the bra-side Coulomb sums jab<ab> (ab in blk) of the warp's lanes, which all share the
    bra pair: warp sums of up to 32 values at once, each added by one lane."""
    for s0 in range(0, len(blk), 32):
        part = blk[s0:s0 + 32]
        M = 1
        while M < len(part):
            M *= 2
        em("{")
        em("  const double s2 = 2.0 * deg;")
        em("  double v[%d] = {%s};" % (M, ", ".join(["s2 * jab%d" % ab for ab in part] + ["0.0"] * (M - len(part)))))
        em("  const double s = sqb::warp_sum_scatter<%d>(v);" % M)
        em("  const int l = threadIdx.x & 31, ab = %s;" % ("l + %d" % part[0] if part == list(range(part[0], part[0] + len(part)))
                                                          else "0"))
        em("  if (l < %d && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / %d) * N + bp.fQ + ab %% %d, s);" % (len(part), nb_, nb_))
        em("}")


def emit_multipole(em, blk, nab, nb_, nd):
    """Multipole mode of the narrow FP64 form: a substituted quartet (mpq) takes the monopole
    values of computeQuartetMPole (reference src/matrix.c:2609-2647) for its block; an exactly
    computed quartet whose exponent is still unknown contributes the largest |exact - monopole|
    over its block (getErrExpQuartetMPole, src/matrix.c:2551-2600) to its error-bank slot,
    combined over the passes by an atomic maximum of the bits (non-negative doubles order as
    integers; bit 63 marks the slot as measured)."""
    em("if (mpq) {")
    em("  const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;")
    for ab in range(nab):
        aa, bb = divmod(ab, nb_)
        for cd in blk:
            c, d = divmod(cd, nd)
            em("  o%d_%d = sqb::mpole_value(a.mpole, N, fP + %d, fQ + %d, fI + %d, fJ + %d);" % (ab, cd, aa, bb, c, d))
    em("} else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {")
    em("  const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;")
    em("  double e = 0.0;")
    for ab in range(nab):
        aa, bb = divmod(ab, nb_)
        for cd in blk:
            c, d = divmod(cd, nd)
            em("  e = fmax(e, fabs(o%d_%d - sqb::mpole_value(a.mpole, N, fP + %d, fQ + %d, fI + %d, fJ + %d)));" % (ab, cd, aa, bb, c, d))
    em("  atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));")
    em("}")


def grouped(nab, ncd):
    """True where the digestion sums the lanes of a quartet before its atomics (group_add)."""
    return nab * ncd <= GROUP_MAX


def emit_digest(em, spin, blk, nab, na, nb_, nd, ncd_all, ablk=None):
    """Digest the contracted block o<ab>_<cd> (cd in blk, ab in ablk -- all bra functions by
    default) into the J/K accumulators.  Expects PA, PB (unrestricted), PT, N, bp, kp, deg and
    jab<ab> in scope; returns flops."""
    abs_ = list(range(nab)) if ablk is None else list(ablk)
    qf = 0
    # small blocks, whose long contractions are split over many lanes, sum those lanes' values before
    # the atomic; larger blocks have too many targets: the inlined sums grow the code past what the
    # instruction cache holds (every class with them: benzene/6-31G* 0.68 -> 0.75 ms per build)
    group = grouped(nab, ncd_all)
    add = lambda p, v: em("sqb::group_add(%s, %s, isplit, gmask, grp == 0);" % (p, v) if group else "atomicAdd(%s, %s);" % (p, v))
    cset = sorted({cd // nd for cd in blk})
    dset = sorted({cd % nd for cd in blk})
    em("{  // digest")
    em.ind += 1
    em("const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;")
    for cd in blk:
        c, d = divmod(cd, nd)
        em("const double ptk%d = PT[(fI + %d) * N + fJ + %d];" % (cd, c, d))
    for ab in abs_:
        aa, bb = divmod(ab, nb_)
        em("const double ptb%d = PT[(fP + %d) * N + fQ + %d];" % (ab, aa, bb))
    spins = [("A", "PA")] + ([("B", "PB")] if spin == "U" else [])
    for s, P_ in spins:
        for bb in range(nb_):
            for d in dset:
                em("const double %sbd%d_%d = %s[(fQ + %d) * N + fJ + %d];" % (s, bb, d, P_, bb, d))
        for aa in sorted({ab // nb_ for ab in abs_}):
            for d in dset:
                em("const double %sad%d_%d = %s[(fP + %d) * N + fJ + %d];" % (s, aa, d, P_, aa, d))
        for bb in range(nb_):
            for c in cset:
                em("const double %sbc%d_%d = %s[(fQ + %d) * N + fI + %d];" % (s, bb, c, P_, bb, c))
        for aa in range(na):
            for c in cset:
                em("const double %sac%d_%d = %s[(fP + %d) * N + fI + %d];" % (s, aa, c, P_, aa, c))
    for ab in abs_:
        terms = " + ".join("o%d_%d * ptk%d" % (ab, cd, cd) for cd in blk)
        em("jab%d += %s;" % (ab, terms))
        qf += 2 * len(blk)
    for cd in blk:
        c, d = divmod(cd, nd)
        terms = " + ".join("o%d_%d * ptb%d" % (ab, cd, ab) for ab in abs_)
        add("Jacc + (fI + %d) * N + fJ + %d" % (c, d), "2.0 * deg * (%s)" % terms)
        qf += 2 * len(abs_) + 2
    for s, _ in spins:
        acc = "KAacc" if s == "A" else "KBacc"
        tg = {}
        for ab in abs_:
            aa, bb = divmod(ab, nb_)
            for cd in blk:
                c, d = divmod(cd, nd)
                o = "o%d_%d" % (ab, cd)
                tg.setdefault(("P", aa, "I", c), []).append("%s * %sbd%d_%d" % (o, s, bb, d))
                tg.setdefault(("Q", bb, "I", c), []).append("%s * %sad%d_%d" % (o, s, aa, d))
                tg.setdefault(("P", aa, "J", d), []).append("%s * %sbc%d_%d" % (o, s, bb, c))
                tg.setdefault(("Q", bb, "J", d), []).append("%s * %sac%d_%d" % (o, s, aa, c))
        for (rs_, ri, cs_, ci), terms in tg.items():
            add("%s + (f%s + %d) * N + f%s + %d" % (acc, rs_, ri, cs_, ci), "deg * (%s)" % " + ".join(terms))
            qf += 2 * len(terms) + 1
    em.ind -= 1
    em("}")
    return qf


def write_if_changed(path, text):
    if os.path.exists(path) and open(path).read() == text:
        return
    with open(path, "w") as f:
        f.write(text)


def quartet_classes():
    cls = []
    for i, x in enumerate(PAIR_ORDER):
        for y in PAIR_ORDER[: i + 1]:
            cls.append((x, y))
    return cls


def main():
    outdir = sys.argv[1] if len(sys.argv) > 1 else os.path.join(os.path.dirname(__file__), "gen")
    os.makedirs(outdir, exist_ok=True)
    metas = []
    files = []
    head = ['// generated by gen_jk_kernels.py -- do not edit', '#include "../jk_common.cuh"', '']

    def emit(src, meta):
        # one kernel per file: the largest classes' kernels take ptxas minutes each, and
        # separate files compile in parallel
        fn = "%s.cu" % meta["name"]
        write_if_changed(os.path.join(outdir, fn), "\n".join(head + [src]))
        files.append(fn)

    for bra, ket in quartet_classes():
        for spin in ("R", "U"):
            s, m = gen_class(bra, ket, spin)
            emit(s, m)
            m["wide"] = None
            if n_passes(bra, ket, STATE_MAX_WIDE) < n_passes(bra, ket, STATE_MAX):
                s4, m4 = gen_class(bra, ket, spin, "D", STATE_MAX_WIDE, "_w")
                emit(s4, m4)
                m["wide"] = m4
            m["swap"] = None
            if SWAP and swap_worthwhile(bra, ket):
                s5, m5 = gen_class_swap(bra, ket, spin, STATE_MAX_SWAP)
                emit(s5, m5)
                m["swap"] = m5
            m["f32"] = None
            if pair_L(bra) + pair_L(ket) <= F32_MAX_L:
                s3, m3 = gen_class(bra, ket, spin, "F")
                emit(s3, m3)
                m["f32"] = m3
            metas.append(m)
    # registry
    reg = ['// generated by gen_jk_kernels.py -- do not edit', '#include "../jk_common.cuh"',
           '#include "../jk_registry.h"', '']
    for m in metas:
        reg.append('extern "C" __global__ void %s(const sqb::JKArgs, const sqb::WorkItem*);' % m["name"])
        if m["f32"]:
            reg.append('extern "C" __global__ void %s(const sqb::JKArgs, const sqb::WorkItem*);' % m["f32"]["name"])
        if m["wide"]:
            reg.append('extern "C" __global__ void %s(const sqb::JKArgs, const sqb::WorkItem*);' % m["wide"]["name"])
        if m["swap"]:
            reg.append('extern "C" __global__ void %s(const sqb::JKArgs, const sqb::WorkItem*);' % m["swap"]["name"])
    reg.append("")
    reg.append("namespace sqb {")
    reg.append("const char* const kPairClassNames[%d] = {%s};" % (len(PAIRS), ", ".join('"%s"' % p for p in PAIRS)))
    reg.append("const ClassKernel kClassKernels[%d] = {" % (len(metas) // 2))
    for i in range(0, len(metas), 2):
        r, u = metas[i], metas[i + 1]
        reg.append('  {%d, %d, %d, %d, %d, %d, %d, %d, (const void*)%s, (const void*)%s, %d, %d, %d,' % (
            PAIRS.index(r["bra"]), PAIRS.index(r["ket"]), r["nab"], r["ncd"], r["neb"], r["nek"],
            r["Lt"], r["flops"]["passes"], r["name"], u["name"], r["flops"]["prim"], r["flops"]["flush"],
            r["flops"]["quartet"]))
        fr, fu = r["f32"], u["f32"]
        if fr:
            reg.append('   %d, (const void*)%s, (const void*)%s, %d, %d, %d,' % (
                fr["flops"]["passes"], fr["name"], fu["name"], fr["flops"]["prim"], fr["flops"]["flush"],
                fr["flops"]["quartet"]))
        else:
            reg.append('   0, nullptr, nullptr, 0, 0, 0,')
        reg.append('   %d,' % r["flops"]["alg_prim"])
        wr, wu = r["wide"], u["wide"]
        if wr:
            reg.append('   %d, (const void*)%s, (const void*)%s, %d, %d, %d,' % (
                wr["flops"]["passes"], wr["name"], wu["name"], wr["flops"]["prim"], wr["flops"]["flush"],
                wr["flops"]["quartet"]))
        else:
            reg.append('   0, nullptr, nullptr, 0, 0, 0,')
        sr, su = r["swap"], u["swap"]
        if sr:
            reg.append('   %d, (const void*)%s, (const void*)%s, %d, %d, %d,' % (
                sr["flops"]["passes"], sr["name"], su["name"], sr["flops"]["prim"], sr["flops"]["flush"],
                sr["flops"]["quartet"]))
        else:
            reg.append('   0, nullptr, nullptr, 0, 0, 0,')
        reg.append('   %d, %d},' % (default_form(r["bra"], r["ket"], bool(wr), bool(sr)), grouped(r["nab"], r["ncd"])))
    reg.append("};")
    reg.append("const int kNumClassKernels = %d;" % (len(metas) // 2))
    reg.append("}  // namespace sqb")
    write_if_changed(os.path.join(outdir, "jk_registry.cu"), "\n".join(reg) + "\n")
    files.append("jk_registry.cu")
    fj = {m["name"]: m["flops"] for m in metas}
    fj.update({m["f32"]["name"]: m["f32"]["flops"] for m in metas if m["f32"]})
    fj.update({m["wide"]["name"]: m["wide"]["flops"] for m in metas if m["wide"]})
    fj.update({m["swap"]["name"]: m["swap"]["flops"] for m in metas if m["swap"]})
    write_if_changed(os.path.join(outdir, "jk_flops.json"), json.dumps(fj, indent=0))
    # sources of an earlier layout that this run did not write
    for fn in os.listdir(outdir):
        if fn.endswith(".cu") and fn not in files:
            os.remove(os.path.join(outdir, fn))
    write_if_changed(os.path.join(outdir, "files.txt"), "\n".join(files) + "\n")
    print("generated %d kernels in %d files" % (len(metas), len(files)))


if __name__ == "__main__":
    main()
