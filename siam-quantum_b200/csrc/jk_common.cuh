// Device-side records and the Boys function shared by every J/K class kernel.
//
// Boys function F_m(T) = int_0^1 u^(2m) exp(-T u^2) du  (role of fgamma_set, reference
// src/fgamma.c:172-206).  Written from the mathematics, not from any library:
//   T <  BOYS_TMAX : the top order F_M(T) by a 9-term Taylor expansion about the nearest grid
//                    point T0 (spacing BOYS_H), F_M(T0-x) = sum_k F_{M+k}(T0) x^k / k!,
//                    then the stable downward recursion F_m = (2T F_{m+1} + e^-T)/(2m+1), with
//                    e^-T = e^-T0 e^x from a tabulated e^-T0 and the Taylor series of e^x.
//   T >= BOYS_TMAX : F_0 = sqrt(pi/T)/2 (the erfc tail is below 1e-17 relative there) and the
//                    stable upward recursion F_{m+1} = ((2m+1) F_m - e^-T)/(2T).
// The grid values are computed on the host in extended precision (jk_engine.cu).
#pragma once
#include <cstdint>

#define BOYS_H      0.1
#define BOYS_INV_H  10.0
#define BOYS_TMAX   36.0
#define BOYS_NGRID  361      // grid points T0 = 0, 0.1, ..., 36.0
#define BOYS_MMAX   8        // highest order of the J/K kernels ((dd|dd)); the gradient's takes one more
#define BOYS_MROWS  (BOYS_MMAX + 2)   // orders of the FP64 row table: M = 0..9
#define BOYS_NTAY   9        // Taylor terms
// plain table of F_m(T0), m = 0..17 per grid row (the gradient kernels' table)
#define BOYS_NCOL   (BOYS_MMAX + BOYS_NTAY + 1)
// row table of boys<M> / boysf<M>: per order M (FP64 0..9, FP32 0..8) and grid point, the Taylor
// coefficients of F_M about T0 and e^-T0 (FP64: 9 + 1 of 16 doubles; FP32: 6 + 1 of 8 floats)
#define BOYS_ROW    16
#define BOYS_ROWF   8

#define TWO_PI_2_5  34.986836655249725     // 2 pi^(5/2)
#define PRIM_CUTOFF 1.0e-15                // reference src/int.h:19
#define TWO_PI_2_5F 34.986836655249725f    // the same in FP32 (mixed-precision forms)
#define PRIM_CUTOFF_F 1.0e-15f

namespace sqb {

// One shell pair (P >= Q in the reference's sorted shell order), 32 bytes.
struct PairRec {
  int P, Q;        // sorted shell indices
  int fP, fQ;      // first basis function of each shell
  int nprim;       // primitive pairs
  int poff;        // offset (elements) of field 0 of its first primitive record in the class array
  int kstride;     // elements between consecutive fields of one record: field f of primitive
                   // record j sits at poff + (j * fields + f) * kstride
  int pad_;
  double schwarz;  // max over the block of the basis-level Schwarz matrix
};

// A CTA's unit of work: one bra pair and a contiguous range of cnt ket pairs, each ket handled by
// si * sj threads: thread (gi, gj) takes the bra primitives gi, gi + si, ... and the ket
// primitives gj, gj + sj, ... (split = si | sj << 16; si, sj >= 1).
struct WorkItem {
  int bra, k0, cnt, split;
  int mol;         // index of the molecule (MolRec) the pairs belong to
};

// One molecule of a build: where its matrices sit in the packed device arrays, and the
// cutoffs of its current SCF step.  A single-molecule build has one record at offset 0; a
// batched build packs many molecules' nbf x nbf blocks back to back.
struct MolRec {
  long long moff;      // offset (doubles) of its nbf x nbf blocks in PA, PB, PT, Jacc, KAacc, KBacc
  long long pmoff;     // offset of its ns x ns block-maximum matrix in PM
  int nbf, ns;
  double cut_outer, cut_fixed, dscreen_rmax;
  int shoff;           // its first shell in the packed shell tables (batched block maxima)
  int uhf;             // 1 = unrestricted (KB from PB), 0 = restricted (KB = KA)
};

struct JKArgs {
  const PairRec* bra_pairs;
  const double* bra_prims;
  const PairRec* ket_pairs;
  const double* ket_prims;
  const double* PA;
  const double* PB;
  const double* PT;
  const double* PM;            // per molecule ns x ns shell-block max of |PT|,|PA|,|PB|
  double* Jacc;                // per molecule nbf x nbf, J = Jacc + Jacc^T
  double* KAacc;               // per molecule nbf x nbf, K[PA] = KAacc + KAacc^T
  double* KBacc;
  const double* boys_tab;      // row table of boys<M>: BOYS_MROWS x BOYS_NGRID x BOYS_ROW
  const float* boys_tab_f;     // the FP32 row table (mixed-precision forms), rows of BOYS_ROWF
  unsigned long long* counters;// [0] quartets computed, [1] primitive quartets evaluated,
                               // [2] bra-primitive flushes, [3] digestions
  const MolRec* mols;          // per-molecule offsets, sizes and cutoffs (WorkItem::mol)
  int same_class;              // bra and ket pairs come from one class (pair identity possible)
  const float* bra_prims_f;    // FP32 copies of the primitive records (mixed-precision kernels)
  const float* ket_prims_f;
  // Reference-parity multipole mode (erbank == nullptr: off; narrow FP64 form, isplit 1).
  // The reference's GTO_JK_Matrix_Quartet_Parallel (src/matrix.c:3914-3967) keeps, per shell
  // quartet surviving the outer Schwarz cutoff, the base-1.5 exponent of the largest error of
  // the monopole approximation (getErrExpQuartetMPole, src/matrix.c:2551), measured the first
  // time the quartet is computed; on later visits a quartet below its memory cutoff whose
  // 1.5^exponent * maxPShell is below the fixed cutoff takes the monopole values instead
  // (computeQuartetMPole, src/matrix.c:2609).
  signed char* erbank;         // per outer-cutoff survivor: exponent, or ERR_UNKNOWN
  unsigned long long* erscr;   // per survivor: bits of this build's largest error | 1 << 63
  const int* er_items;         // per work item: erbank index of its first ket
  const double* mpole;         // per function pair (p * nbf + q): charge q, centre x, y, z
  const double* pow15;         // 1.5^e, e = -120..120, as the host's pow computes it
  double mp_rmax;              // quartets with Sch(PQ)*Sch(IJ) >= this are never substituted
  // Persistent launch (queue != nullptr): a fixed grid takes the nqueue work units (item, pass)
  // of the launch from this device counter, zeroed before the launch; npass passes per item.
  unsigned long long* queue;
  int nqueue, npass;
  // Copies of the accumulators (a power of two, less one as a mask; `copy_stride` doubles apart):
  // work item i adds into copy i & copy_mask, so that the atomics of a small molecule's build do
  // not all meet on its few elements
  int copy_mask;
  long long copy_stride;
};

constexpr int ERR_MIN = -120;      // src/matrix.c:1745-1747
constexpr int ERR_MAX = 120;
constexpr int ERR_UNKNOWN = 121;
#define MULTIPOLE_R2_CUTOFF 1.0    // src/multipole.h:23: below this squared distance the term is 0

// Monopole-monopole value of the function-pair quartet (pq|rs) (computeQuartetMPole): charges
// times the inverse distance between the pairs' charge centres, 0 when the squared distance
// is below MULTIPOLE_R2_CUTOFF; the same operations in the same order, without contractions.
// Not inlined: the multipole mode is rare and its callers are unrolled over whole blocks.
static __device__ __noinline__ double mpole_value(const double* __restrict__ mp, int N, int p, int q, int r, int s) {
  const double* m1 = mp + 4 * ((long long)p * N + q);
  const double* m2 = mp + 4 * ((long long)r * N + s);
  const double dx = __dadd_rn(m1[1], -m2[1]), dy = __dadd_rn(m1[2], -m2[2]), dz = __dadd_rn(m1[3], -m2[3]);
  const double K = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  if (K < MULTIPOLE_R2_CUTOFF) return 0.0;
  return __dmul_rn(__dmul_rn(m1[0], m2[0]), __dsqrt_rn(__ddiv_rn(1.0, K)));
}

// F_0..F_M at T.  M is a compile-time order so the recursion unrolls.  `tab` is the row table
// (BOYS_ROW doubles per order and grid point): row (M, g) holds the Taylor coefficients
// F_{M+k}(T0) / k! of F_M(T0 - x), k < BOYS_NTAY, and e^-T0, so one aligned 128-byte line serves
// a lane in five 16-byte loads and neither series needs a multiplication per term.  Measured on
// B200 against rows of plain F_{M+k}(T0) with the 1/k! multiplied in the kernel, e^-T0 in a table of
// its own and a division and a square root above BOYS_TMAX (C60/6-31G, ms per launch): LL|LL wide
// 41.0 -> 38.7, LL|LS wide 16.9 -> 15.9, LS|LS swapped 3.3 -> 2.5, LS|SS swapped 0.80 -> 0.58.
template <int M>
__device__ __forceinline__ void boys(double T, const double* __restrict__ tab, double* F) {
  if (T < BOYS_TMAX) {
    const int g = __double2int_rn(T * BOYS_INV_H);
    const double x = fma((double)g, BOYS_H, -T);   // T0 - T, |x| <= BOYS_H/2
    const double2* r2 = reinterpret_cast<const double2*>(tab + (M * BOYS_NGRID + g) * BOYS_ROW);
    double v[BOYS_NTAY + 1];
#pragma unroll
    for (int q = 0; q < (BOYS_NTAY + 1) / 2; ++q) {
      const double2 t = __ldg(r2 + q);
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
    double s = v[BOYS_NTAY - 1];
#pragma unroll
    for (int k = BOYS_NTAY - 2; k >= 0; --k) s = fma(s, x, v[k]);
    F[M] = s;
    if (M > 0) {
      // e^-T = e^-T0 e^x: the row's e^-T0 times the Taylor series of e^x through x^8/8!
      // (the next term is below 6e-18)
      double ed = 1.0 / 40320.0;
      ed = fma(ed, x, 1.0 / 5040.0);
      ed = fma(ed, x, 1.0 / 720.0);
      ed = fma(ed, x, 1.0 / 120.0);
      ed = fma(ed, x, 1.0 / 24.0);
      ed = fma(ed, x, 1.0 / 6.0);
      ed = fma(ed, x, 0.5);
      ed = fma(ed, x, 1.0);
      ed = fma(ed, x, 1.0);
      const double e = v[BOYS_NTAY] * ed;
      const double t2 = T + T;
#pragma unroll
      for (int m = M - 1; m >= 0; --m) F[m] = fma(t2, F[m + 1], e) * (1.0 / (2 * m + 1));
    }
  } else {
    const double rt = rsqrt(T);
    F[0] = 0.88622692545275801365 * rt;          // sqrt(pi)/2 / sqrt(T)
    if (M > 0) {
      // e^-T is below 3e-18 of every (2m+1) F_m, m <= 8, for T >= 64
      const double e2 = T < 64.0 ? 0.5 * exp(-T) : 0.0;
      // 1/T = rt rt with one Newton step: its error enters every order anew (with rt rt alone F_8
      // has an rms error of 8.0 units of 2^-53 over T = 36..400, with the step 3.8, with a
      // division 4.0).  Measured on B200 without / with it: C60/6-31G 56.1 / 56.4 ms per build.
      const double q = rt * rt, it = fma(q, fma(-T, q, 1.0), q);
#pragma unroll
      for (int m = 0; m < M; ++m) F[m + 1] = fma(m + 0.5, F[m], -e2) * it;
    }
  }
}

// F_0..F_M at T in FP32, for the mixed-precision forms (quartets whose Schwarz bound is below
// the FP32 threshold): the scheme of boys<M> with rows of BOYS_ROWF floats, 6 Taylor terms
// (|x| <= BOYS_H/2: the next term is below 2e-11 of F_M, under FP32 rounding).
template <int M>
__device__ __forceinline__ void boysf(float T, const float* __restrict__ tab, float* F) {
  if (T < (float)BOYS_TMAX) {
    const int g = __float2int_rn(T * (float)BOYS_INV_H);
    const float x = fmaf((float)g, (float)BOYS_H, -T);
    const float4* r4 = reinterpret_cast<const float4*>(tab + (M * BOYS_NGRID + g) * BOYS_ROWF);
    const float4 u = __ldg(r4), w = __ldg(r4 + 1);   // c0..c3; c4, c5, e^-T0
    F[M] = fmaf(fmaf(fmaf(fmaf(fmaf(w.y, x, w.x), x, u.w), x, u.z), x, u.y), x, u.x);
    if (M > 0) {
      const float e = expf(-T);
      const float t2 = T + T;
#pragma unroll
      for (int m = M - 1; m >= 0; --m) F[m] = fmaf(t2, F[m + 1], e) * (1.0f / (float)(2 * m + 1));
    }
  } else {
    const float rt = rsqrtf(T);
    F[0] = 0.886226925f * rt;
    if (M > 0) {
      const float e2 = 0.5f * expf(-T);
      const float q = rt * rt, it = fmaf(q, fmaf(-T, q, 1.0f), q);   // as boys<M>
#pragma unroll
      for (int m = 0; m < M; ++m) F[m + 1] = fmaf(m + 0.5f, F[m], -e2) * it;
    }
  }
}

// Warp-aggregated 64-bit counter increment.
__device__ __forceinline__ void count_add(unsigned long long* c, unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(c, v);
}

// *p += v, summed first over the n lanes (a power of two, aligned: mask gmask) that share one
// quartet, whose targets are the same; one atomic per quartet instead of n on one address.
__device__ __forceinline__ void group_add(double* p, double v, int n, unsigned gmask, bool lead) {
  if (n > 1) {
    for (int o = n >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(gmask, v, o);
    if (!lead) return;
  }
  atomicAdd(p, v);
}

// Warp sums of M values (a power of two <= 32) at once: returns in lane l the warp's sum of
// v[l % M].  Every step halves the values a lane holds, M - 1 + log2(32 / M) exchanges in all
// where M separate sums take 5 M.
template <int M>
__device__ __forceinline__ double warp_sum_scatter(double (&v)[M]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = M / 2; s > 0; s >>= 1) {
    const bool hi = lane & s;
#pragma unroll
    for (int k = 0; k < s; ++k) {
      const double send = hi ? v[k] : v[k + s], keep = hi ? v[k + s] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
#pragma unroll
  for (int o = M; o < 32; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace sqb
