// Device side of the generic J/K path shared by its kernels (jk_generic.cu, the generated f-shell
// kernels): component descriptors, Hermite tables, the Boys function of one order.
#pragma once
#include "jk_common.cuh"
#include "jk_generic.cuh"

namespace sqb {

constexpr int kGenR = 455;                             // tetrahedral entries with t+u+v <= 12
static_assert(kGenMmax == 12 && (kGenMmax + 1) * (kGenMmax + 2) * (kGenMmax + 3) / 6 == kGenR, "R table size");

// (t, u, v) of tetrahedral index k: order n = t+u+v, then m = u+v, then v ascending
struct TuvTable {
  unsigned int v[kGenR];
  constexpr TuvTable() : v() {
    int k = 0;
    for (int n = 0; n <= sqb::kGenMmax; ++n)
      for (int m = 0; m <= n; ++m)
        for (int w = 0; w <= m; ++w) v[k++] = (unsigned)(n - m) | ((unsigned)(m - w) << 8) | ((unsigned)w << 16);
  }
};
static __device__ const TuvTable g_tuv = TuvTable();

__device__ __forceinline__ int gtet(int t, int u, int v) {
  const int n = t + u + v, m = u + v;
  return n * (n + 1) * (n + 2) / 6 + m * (m + 1) / 2 + v;
}

// A primitive pair's tables in `coef`: axis d, E^{ij}_t at e + d*sz + (i*lq1 + j)*lt + t
// (i <= lP, j <= lQ, t <= i+j; lq1 = lQ+1, lt = lP+lQ+1, sz = (lP+1) lq1 lt); then the weights
// c_a c_b exp(-ab|AB|^2/p)/p of its function pairs at e + 3*sz.
struct EView {
  const double* e;
  int lq1, lt, sz;
  __device__ EView(const double* coef, const double* rec, const GenPairRec& P)
      : e(coef + (long long)rec[11]), lq1(P.lQ + 1), lt(P.lP + P.lQ + 1), sz((P.lP + 1) * (P.lQ + 1) * (P.lP + P.lQ + 1)) {}
  __device__ __forceinline__ const double* ax(int d, int i, int j) const { return e + d * sz + (i * lq1 + j) * lt; }
  __device__ __forceinline__ double w(int ab) const { return __ldg(e + 3 * sz + ab); }
};

// component exponents of a function pair: a_x, b_x, a_y, b_y, a_z, b_z in 2 bits each
__device__ __forceinline__ int dsc(unsigned d, int k) { return (d >> (2 * k)) & 3; }

// F_n(T) for one order n <= 12: below BOYS_TMAX the 9-term Taylor expansion about the nearest
// grid point, F_n(T0+d) = sum_k F_{n+k}(T0) (-d)^k / k!, from the table's own column n; above,
// F_0 = sqrt(pi/T)/2 and the upward recursion F_{m+1} = ((2m+1) F_m - e^-T)/(2T).
static __device__ double gen_boys(int n, double T, const double* __restrict__ tab) {
  if (T < BOYS_TMAX) {
    const int g = __double2int_rn(T * BOYS_INV_H);
    const double d = T - g * BOYS_H;
    const double* row = tab + g * kGenBoysCols + n;
    double s = __ldg(row + BOYS_NTAY - 1);
    for (int k = BOYS_NTAY - 2; k >= 0; --k) s = fma(s, -d * (1.0 / (double)(k + 1)), __ldg(row + k));
    return s;
  }
  const double it = 1.0 / T;
  double F = 0.88622692545275801365 * sqrt(it);   // sqrt(pi)/2 / sqrt(T)
  if (n > 0) {
    const double e = exp(-T), h = 0.5 * it;
    for (int m = 0; m < n; ++m) F = ((2 * m + 1) * F - e) * h;
  }
  return F;
}

// The unit of a warp: its bra, its kets klist[k0 .. k0 + cnt), its function pairs and its part of the
// primitives.
struct FUnit {
  int bra, k0, cnt, cg, gi, gj, si, sj;
};

// Unit u of a class's runs (first[r] <= u < first[r + 1]; the last run ends with the class).  The
// warp looks for the run together, 32 starts at a time: at most three rounds of loads for up to 32,768
// runs (a class has up to 1,859 in water/QZP, 30,120 in benzene/QZP).
static __device__ __forceinline__ FUnit f_unit(const FRun* __restrict__ runs, const long long* __restrict__ first,
                                               int nruns, long long u) {
  const int lane = threadIdx.x & 31;
  int lo = 0;
  for (int n = nruns; n > 1;) {            // the run is one of lo .. lo + n - 1
    const int step = (n + 31) / 32, x = lane * step;
    const int k = __popc(__ballot_sync(0xffffffffu, x < n && first[lo + x] <= u)) - 1;   // lane 0's start is not above u
    lo += k * step;
    n = min(step, n - k * step);
  }
  const FRun r = runs[lo];
  const int si = r.split & 255, sj = (r.split >> 8) & 255, ng = r.split >> 16, parts = si * sj;
  const long long at = u - first[lo];
  const int kb = (int)(at / parts), part = (int)(at - (long long)kb * parts), gi = part / sj;
  return {r.bra, r.k0 + kb * ng, min(ng, r.cnt - kb * ng), r.cg, gi, part - gi * sj, si, sj};
}

// The f-shell kernels' seeds base[n] = 2 pi^(5/2)/sqrt(p+q) (-2 alpha)^n F_n(T), n <= L, by the g
// lanes of a quartet (cc = 0 .. g-1), each its own orders.
static __device__ __forceinline__ void f_seeds(int L, double alpha, double rs, double X, double Y, double Z,
                                               const double* tab, double* base, int cc, int g) {
  const double T = alpha * fma(X, X, fma(Y, Y, Z * Z)), m2a = -2.0 * alpha;
  double w = TWO_PI_2_5 * rs;
  int m = 0;
  for (int n = cc; n <= L; n += g) {
    for (; m < n; ++m) w *= m2a;
    base[n] = w * gen_boys(n, T, tab);
  }
}

// R^(0)_{tuv}, t+u+v <= L, in a box [t][u][v] of (L+1)^3, by the Hermite recursion
//   R^(n)_{t+1,u,v} = t R^(n+1)_{t-1,u,v} + X R^(n+1)_{t,u,v}   (likewise in u, v),
// in place: level n from level n + 1 by falling degree, an entry needing only entries one and two
// degrees below it, which still hold level n + 1.  The g lanes of a quartet share each degree; the
// whole warp takes the same steps (`mine`: the lane belongs to a quartet).
static __device__ __forceinline__ void f_box(int L, double X, double Y, double Z, const double* base, double* box,
                                             int cc, int g, bool mine) {
  const int S1 = L + 1, S2 = S1 * S1;
  if (mine && cc == 0) box[0] = base[L];
  __syncwarp();
  for (int n = L - 1; n >= 0; --n) {
    for (int N = L - n; N > 0; --N) {
      const int first = N * (N + 1) * (N + 2) / 6, cnt = (N + 1) * (N + 2) / 2;
      if (mine)
        for (int x = cc; x < cnt; x += g) {
          const unsigned e = g_tuv.v[first + x];
          const int t = e & 255, u = (e >> 8) & 255, v = e >> 16;
          const int at = t * S2 + u * S1 + v;
          const int st = t > 0 ? S2 : u > 0 ? S1 : 1, k = (t > 0 ? t : u > 0 ? u : v) - 1;
          const double D = t > 0 ? X : u > 0 ? Y : Z;
          double r = D * box[at - st];
          if (k > 0) r = fma((double)k, box[at - 2 * st], r);
          box[at] = r;
        }
      __syncwarp();
    }
    if (mine && cc == 0) box[0] = base[n];
    __syncwarp();
  }
}

}  // namespace sqb
