// generated by gen_fshell_kernels.py -- do not edit
#include "../jk_generic_dev.cuh"

extern "C" __global__ void __launch_bounds__(128)
jkf_FP_0(const sqb::FArgs a, const sqb::FRun* __restrict__ runs, const long long* __restrict__ first, int nruns,
   long long u0, long long nunits) {
  extern __shared__ double fsm[];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const long long unit = u0 + (long long)blockIdx.x * 4 + wp;
  if (unit >= nunits) return;                   // whole warps leave
  const sqb::FUnit it = sqb::f_unit(runs, first, nruns, unit);
  const int g = it.cg >> 16, s = lane / g, cc = lane - s * g, cd = (it.cg & 0xffff) + cc;
  const sqb::GenPairRec A = a.pairs[it.bra];
  const int kb = a.klist[it.k0 + min(s, it.cnt - 1)];   // idle lanes shadow the last ket
  const sqb::GenPairRec B = a.pairs[kb];
  const double r = A.schwarz * B.schwarz;
  bool ok = s < it.cnt && !(r < a.b.cut_outer) && !(r < a.b.cut_fixed);
  if (ok && r < a.b.dscreen_rmax) {
    const bool bf = (A.P > B.P) || (A.P == B.P && A.Q >= B.Q);
    const int P = bf ? A.P : B.P, Q = bf ? A.Q : B.Q, I = bf ? B.P : A.P, J = bf ? B.Q : A.Q;
    const double* PM = a.b.PM; const int ns = a.b.ns;
    const double mp = PM[P * ns + Q] + PM[I * ns + J] + PM[P * ns + I] + PM[P * ns + J] + PM[Q * ns + I] + PM[Q * ns + J];
    ok = !(r * mp < a.b.cut_fixed);
  }
  if (!__any_sync(0xffffffffu, ok)) return;
  const double deg = (A.P == A.Q ? 0.5 : 1.0) * (B.P == B.Q ? 0.5 : 1.0) * (kb == it.bra ? 0.5 : 1.0);
  const int L = 4 + B.lP + B.lQ, S1 = L + 1, S2 = S1 * S1;   // uniform over the warp
  double* __restrict__ box = fsm + wp * sqb::kFWarpDoubles + min(s, it.cnt - 1) * sqb::f_slot(L);   // [t][u][v], then the seeds
  double* __restrict__ base = box + S1 * S2;
  const bool mine = s < it.cnt;
  const unsigned d = __ldg(a.desc + B.doff + cd);
  const int cx = sqb::dsc(d, 0), dx = sqb::dsc(d, 1), cy = sqb::dsc(d, 2), dy = sqb::dsc(d, 3), cz = sqb::dsc(d, 4), dz = sqb::dsc(d, 5);
  const int n1 = cy + dy + 1, n2 = cz + dz + 1, nk = (cx + dx + 1) * n1 * n2;
  unsigned long long npq = 0, nfl = 0;
  double o0_0 = 0.0;
  double o0_1 = 0.0;
  double o0_2 = 0.0;
  double o1_0 = 0.0;
  double o1_1 = 0.0;
  double o1_2 = 0.0;
  double o2_0 = 0.0;
  double o2_1 = 0.0;
  double o2_2 = 0.0;
  double o3_0 = 0.0;
  double o3_1 = 0.0;
  double o3_2 = 0.0;
  double o4_0 = 0.0;
  double o4_1 = 0.0;
  double o4_2 = 0.0;
  double o5_0 = 0.0;
  double o5_1 = 0.0;
  double o5_2 = 0.0;
  double o6_0 = 0.0;
  double o6_1 = 0.0;
  double o6_2 = 0.0;
  double o7_0 = 0.0;
  double o7_1 = 0.0;
  double o7_2 = 0.0;
  double o8_0 = 0.0;
  double o8_1 = 0.0;
  double o8_2 = 0.0;
  double o9_0 = 0.0;
  double o9_1 = 0.0;
  double o9_2 = 0.0;
  const int gi = it.gi, gj = it.gj, si = it.si, sj = it.sj;
  for (int i = gi; i < A.nprim; i += si) {      // this unit's part of the primitives
    const double* pa = a.prims + (size_t)(A.poff + i) * sqb::kGenPrimStride;
    const double p = pa[0], Px = pa[1], Py = pa[2], Pz = pa[3], kpa = pa[4];
    double g000 = 0.0;
    double g100 = 0.0;
    double g010 = 0.0;
    double g001 = 0.0;
    double g200 = 0.0;
    double g110 = 0.0;
    double g101 = 0.0;
    double g020 = 0.0;
    double g011 = 0.0;
    double g002 = 0.0;
    double g300 = 0.0;
    double g210 = 0.0;
    double g201 = 0.0;
    double g120 = 0.0;
    double g111 = 0.0;
    double g102 = 0.0;
    double g030 = 0.0;
    double g021 = 0.0;
    double g012 = 0.0;
    double g003 = 0.0;
    double g400 = 0.0;
    double g310 = 0.0;
    double g301 = 0.0;
    double g220 = 0.0;
    double g211 = 0.0;
    double g202 = 0.0;
    double g130 = 0.0;
    double g121 = 0.0;
    double g112 = 0.0;
    double g103 = 0.0;
    double g040 = 0.0;
    double g031 = 0.0;
    double g022 = 0.0;
    double g013 = 0.0;
    double g004 = 0.0;
    bool any = false;
    for (int j = gj; j < B.nprim; j += sj) {     // one contraction length per warp
      const double* pb = a.prims + (size_t)(B.poff + j) * sqb::kGenPrimStride;
      const double q = pb[0], pq = p + q, rs = rsqrt(pq);
      const bool live = ok && !(TWO_PI_2_5 * kpa * pb[4] * rs < PRIM_CUTOFF);
      if (!__any_sync(0xffffffffu, live)) continue;
      any = true;
      if (live && cd == 0) ++npq;
      const double X = Px - pb[1], Y = Py - pb[2], Z = Pz - pb[3];
      __syncwarp();                                // the previous step is done with the box
      if (mine) sqb::f_seeds(L, p * q * (rs * rs), rs, X, Y, Z, a.boys, base, cc, g);
      __syncwarp();
      sqb::f_box(L, X, Y, Z, base, box, cc, g, mine);
      if (live) {
        const sqb::EView Ej(a.coef, pb, B);
        const double *ex = Ej.ax(0, cx, dx), *ey = Ej.ax(1, cy, dy), *ez = Ej.ax(2, cz, dz);
        const double w = Ej.w(cd);
        int tau = 0, nu = 0, ph = 0;
        for (int k = 0; k < nk; ++k) {
          const double e0 = w * (__ldg(ex + tau) * __ldg(ey + nu)) * __ldg(ez + ph);
          const double e = ((tau + nu + ph) & 1) ? -e0 : e0;
          const double* __restrict__ R = box + tau * S2 + nu * S1 + ph;
          { const double* __restrict__ x = R + 0 * S2 + 0 * S1;
            g000 = fma(e, x[0], g000);
            g001 = fma(e, x[1], g001);
            g002 = fma(e, x[2], g002);
            g003 = fma(e, x[3], g003);
            g004 = fma(e, x[4], g004);
          }
          { const double* __restrict__ x = R + 0 * S2 + 1 * S1;
            g010 = fma(e, x[0], g010);
            g011 = fma(e, x[1], g011);
            g012 = fma(e, x[2], g012);
            g013 = fma(e, x[3], g013);
          }
          { const double* __restrict__ x = R + 0 * S2 + 2 * S1;
            g020 = fma(e, x[0], g020);
            g021 = fma(e, x[1], g021);
            g022 = fma(e, x[2], g022);
          }
          { const double* __restrict__ x = R + 0 * S2 + 3 * S1;
            g030 = fma(e, x[0], g030);
            g031 = fma(e, x[1], g031);
          }
          { const double* __restrict__ x = R + 0 * S2 + 4 * S1;
            g040 = fma(e, x[0], g040);
          }
          { const double* __restrict__ x = R + 1 * S2 + 0 * S1;
            g100 = fma(e, x[0], g100);
            g101 = fma(e, x[1], g101);
            g102 = fma(e, x[2], g102);
            g103 = fma(e, x[3], g103);
          }
          { const double* __restrict__ x = R + 1 * S2 + 1 * S1;
            g110 = fma(e, x[0], g110);
            g111 = fma(e, x[1], g111);
            g112 = fma(e, x[2], g112);
          }
          { const double* __restrict__ x = R + 1 * S2 + 2 * S1;
            g120 = fma(e, x[0], g120);
            g121 = fma(e, x[1], g121);
          }
          { const double* __restrict__ x = R + 1 * S2 + 3 * S1;
            g130 = fma(e, x[0], g130);
          }
          { const double* __restrict__ x = R + 2 * S2 + 0 * S1;
            g200 = fma(e, x[0], g200);
            g201 = fma(e, x[1], g201);
            g202 = fma(e, x[2], g202);
          }
          { const double* __restrict__ x = R + 2 * S2 + 1 * S1;
            g210 = fma(e, x[0], g210);
            g211 = fma(e, x[1], g211);
          }
          { const double* __restrict__ x = R + 2 * S2 + 2 * S1;
            g220 = fma(e, x[0], g220);
          }
          { const double* __restrict__ x = R + 3 * S2 + 0 * S1;
            g300 = fma(e, x[0], g300);
            g301 = fma(e, x[1], g301);
          }
          { const double* __restrict__ x = R + 3 * S2 + 1 * S1;
            g310 = fma(e, x[0], g310);
          }
          { const double* __restrict__ x = R + 4 * S2 + 0 * S1;
            g400 = fma(e, x[0], g400);
          }
          if (++ph == n2) { ph = 0; if (++nu == n1) { nu = 0; ++tau; } }
        }
        nfl += 2ull * 35 * nk;
      }
    }
    if (!any) continue;
    const sqb::EView Ei(a.coef, pa, A);
    const double* __restrict__ E = Ei.e;
    { double z = 0.0;
      z = fma(__ldg(E + 35), g000, z);
      z = fma(__ldg(E + 36), g100, z);
      z = fma(__ldg(E + 37), g200, z);
      z = fma(__ldg(E + 38), g300, z);
      z = fma(__ldg(E + 39), g400, z);
      o0_0 = fma(Ei.w(0), z, o0_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 30) * __ldg(E + 45), g000, z);
      z = fma(__ldg(E + 30) * __ldg(E + 46), g010, z);
      z = fma(__ldg(E + 31) * __ldg(E + 45), g100, z);
      z = fma(__ldg(E + 31) * __ldg(E + 46), g110, z);
      z = fma(__ldg(E + 32) * __ldg(E + 45), g200, z);
      z = fma(__ldg(E + 32) * __ldg(E + 46), g210, z);
      z = fma(__ldg(E + 33) * __ldg(E + 45), g300, z);
      z = fma(__ldg(E + 33) * __ldg(E + 46), g310, z);
      o0_1 = fma(Ei.w(1), z, o0_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 30), fma(__ldg(E + 86), g001, __ldg(E + 85) * g000), z);
      z = fma(__ldg(E + 31), fma(__ldg(E + 86), g101, __ldg(E + 85) * g100), z);
      z = fma(__ldg(E + 32), fma(__ldg(E + 86), g201, __ldg(E + 85) * g200), z);
      z = fma(__ldg(E + 33), fma(__ldg(E + 86), g301, __ldg(E + 85) * g300), z);
      o0_2 = fma(Ei.w(2), z, o0_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 5) * __ldg(E + 70), g000, z);
      z = fma(__ldg(E + 5) * __ldg(E + 71), g010, z);
      z = fma(__ldg(E + 5) * __ldg(E + 72), g020, z);
      z = fma(__ldg(E + 5) * __ldg(E + 73), g030, z);
      z = fma(__ldg(E + 6) * __ldg(E + 70), g100, z);
      z = fma(__ldg(E + 6) * __ldg(E + 71), g110, z);
      z = fma(__ldg(E + 6) * __ldg(E + 72), g120, z);
      z = fma(__ldg(E + 6) * __ldg(E + 73), g130, z);
      o1_0 = fma(Ei.w(3), z, o1_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 75), g000, z);
      z = fma(__ldg(E + 76), g010, z);
      z = fma(__ldg(E + 77), g020, z);
      z = fma(__ldg(E + 78), g030, z);
      z = fma(__ldg(E + 79), g040, z);
      o1_1 = fma(Ei.w(4), z, o1_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 70), fma(__ldg(E + 86), g001, __ldg(E + 85) * g000), z);
      z = fma(__ldg(E + 71), fma(__ldg(E + 86), g011, __ldg(E + 85) * g010), z);
      z = fma(__ldg(E + 72), fma(__ldg(E + 86), g021, __ldg(E + 85) * g020), z);
      z = fma(__ldg(E + 73), fma(__ldg(E + 86), g031, __ldg(E + 85) * g030), z);
      o1_2 = fma(Ei.w(5), z, o1_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 5), fma(__ldg(E + 113), g003, fma(__ldg(E + 112), g002, fma(__ldg(E + 111), g001, __ldg(E + 110) * g000))), z);
      z = fma(__ldg(E + 6), fma(__ldg(E + 113), g103, fma(__ldg(E + 112), g102, fma(__ldg(E + 111), g101, __ldg(E + 110) * g100))), z);
      o2_0 = fma(Ei.w(6), z, o2_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 45), fma(__ldg(E + 113), g003, fma(__ldg(E + 112), g002, fma(__ldg(E + 111), g001, __ldg(E + 110) * g000))), z);
      z = fma(__ldg(E + 46), fma(__ldg(E + 113), g013, fma(__ldg(E + 112), g012, fma(__ldg(E + 111), g011, __ldg(E + 110) * g010))), z);
      o2_1 = fma(Ei.w(7), z, o2_1); }
    { double z = 0.0;
      z += fma(__ldg(E + 119), g004, fma(__ldg(E + 118), g003, fma(__ldg(E + 117), g002, fma(__ldg(E + 116), g001, __ldg(E + 115) * g000))));
      o2_2 = fma(Ei.w(8), z, o2_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 25) * __ldg(E + 50), g000, z);
      z = fma(__ldg(E + 25) * __ldg(E + 51), g010, z);
      z = fma(__ldg(E + 26) * __ldg(E + 50), g100, z);
      z = fma(__ldg(E + 26) * __ldg(E + 51), g110, z);
      z = fma(__ldg(E + 27) * __ldg(E + 50), g200, z);
      z = fma(__ldg(E + 27) * __ldg(E + 51), g210, z);
      z = fma(__ldg(E + 28) * __ldg(E + 50), g300, z);
      z = fma(__ldg(E + 28) * __ldg(E + 51), g310, z);
      o3_0 = fma(Ei.w(9), z, o3_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 20) * __ldg(E + 55), g000, z);
      z = fma(__ldg(E + 20) * __ldg(E + 56), g010, z);
      z = fma(__ldg(E + 20) * __ldg(E + 57), g020, z);
      z = fma(__ldg(E + 21) * __ldg(E + 55), g100, z);
      z = fma(__ldg(E + 21) * __ldg(E + 56), g110, z);
      z = fma(__ldg(E + 21) * __ldg(E + 57), g120, z);
      z = fma(__ldg(E + 22) * __ldg(E + 55), g200, z);
      z = fma(__ldg(E + 22) * __ldg(E + 56), g210, z);
      z = fma(__ldg(E + 22) * __ldg(E + 57), g220, z);
      o3_1 = fma(Ei.w(10), z, o3_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 20) * __ldg(E + 50), fma(__ldg(E + 86), g001, __ldg(E + 85) * g000), z);
      z = fma(__ldg(E + 20) * __ldg(E + 51), fma(__ldg(E + 86), g011, __ldg(E + 85) * g010), z);
      z = fma(__ldg(E + 21) * __ldg(E + 50), fma(__ldg(E + 86), g101, __ldg(E + 85) * g100), z);
      z = fma(__ldg(E + 21) * __ldg(E + 51), fma(__ldg(E + 86), g111, __ldg(E + 85) * g110), z);
      z = fma(__ldg(E + 22) * __ldg(E + 50), fma(__ldg(E + 86), g201, __ldg(E + 85) * g200), z);
      z = fma(__ldg(E + 22) * __ldg(E + 51), fma(__ldg(E + 86), g211, __ldg(E + 85) * g210), z);
      o3_2 = fma(Ei.w(11), z, o3_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 15) * __ldg(E + 60), g000, z);
      z = fma(__ldg(E + 15) * __ldg(E + 61), g010, z);
      z = fma(__ldg(E + 15) * __ldg(E + 62), g020, z);
      z = fma(__ldg(E + 16) * __ldg(E + 60), g100, z);
      z = fma(__ldg(E + 16) * __ldg(E + 61), g110, z);
      z = fma(__ldg(E + 16) * __ldg(E + 62), g120, z);
      z = fma(__ldg(E + 17) * __ldg(E + 60), g200, z);
      z = fma(__ldg(E + 17) * __ldg(E + 61), g210, z);
      z = fma(__ldg(E + 17) * __ldg(E + 62), g220, z);
      o4_0 = fma(Ei.w(12), z, o4_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 10) * __ldg(E + 65), g000, z);
      z = fma(__ldg(E + 10) * __ldg(E + 66), g010, z);
      z = fma(__ldg(E + 10) * __ldg(E + 67), g020, z);
      z = fma(__ldg(E + 10) * __ldg(E + 68), g030, z);
      z = fma(__ldg(E + 11) * __ldg(E + 65), g100, z);
      z = fma(__ldg(E + 11) * __ldg(E + 66), g110, z);
      z = fma(__ldg(E + 11) * __ldg(E + 67), g120, z);
      z = fma(__ldg(E + 11) * __ldg(E + 68), g130, z);
      o4_1 = fma(Ei.w(13), z, o4_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 10) * __ldg(E + 60), fma(__ldg(E + 86), g001, __ldg(E + 85) * g000), z);
      z = fma(__ldg(E + 10) * __ldg(E + 61), fma(__ldg(E + 86), g011, __ldg(E + 85) * g010), z);
      z = fma(__ldg(E + 10) * __ldg(E + 62), fma(__ldg(E + 86), g021, __ldg(E + 85) * g020), z);
      z = fma(__ldg(E + 11) * __ldg(E + 60), fma(__ldg(E + 86), g101, __ldg(E + 85) * g100), z);
      z = fma(__ldg(E + 11) * __ldg(E + 61), fma(__ldg(E + 86), g111, __ldg(E + 85) * g110), z);
      z = fma(__ldg(E + 11) * __ldg(E + 62), fma(__ldg(E + 86), g121, __ldg(E + 85) * g120), z);
      o4_2 = fma(Ei.w(14), z, o4_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 25), fma(__ldg(E + 91), g001, __ldg(E + 90) * g000), z);
      z = fma(__ldg(E + 26), fma(__ldg(E + 91), g101, __ldg(E + 90) * g100), z);
      z = fma(__ldg(E + 27), fma(__ldg(E + 91), g201, __ldg(E + 90) * g200), z);
      z = fma(__ldg(E + 28), fma(__ldg(E + 91), g301, __ldg(E + 90) * g300), z);
      o5_0 = fma(Ei.w(15), z, o5_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 20) * __ldg(E + 45), fma(__ldg(E + 91), g001, __ldg(E + 90) * g000), z);
      z = fma(__ldg(E + 20) * __ldg(E + 46), fma(__ldg(E + 91), g011, __ldg(E + 90) * g010), z);
      z = fma(__ldg(E + 21) * __ldg(E + 45), fma(__ldg(E + 91), g101, __ldg(E + 90) * g100), z);
      z = fma(__ldg(E + 21) * __ldg(E + 46), fma(__ldg(E + 91), g111, __ldg(E + 90) * g110), z);
      z = fma(__ldg(E + 22) * __ldg(E + 45), fma(__ldg(E + 91), g201, __ldg(E + 90) * g200), z);
      z = fma(__ldg(E + 22) * __ldg(E + 46), fma(__ldg(E + 91), g211, __ldg(E + 90) * g210), z);
      o5_1 = fma(Ei.w(16), z, o5_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 20), fma(__ldg(E + 97), g002, fma(__ldg(E + 96), g001, __ldg(E + 95) * g000)), z);
      z = fma(__ldg(E + 21), fma(__ldg(E + 97), g102, fma(__ldg(E + 96), g101, __ldg(E + 95) * g100)), z);
      z = fma(__ldg(E + 22), fma(__ldg(E + 97), g202, fma(__ldg(E + 96), g201, __ldg(E + 95) * g200)), z);
      o5_2 = fma(Ei.w(17), z, o5_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 15), fma(__ldg(E + 102), g002, fma(__ldg(E + 101), g001, __ldg(E + 100) * g000)), z);
      z = fma(__ldg(E + 16), fma(__ldg(E + 102), g102, fma(__ldg(E + 101), g101, __ldg(E + 100) * g100)), z);
      z = fma(__ldg(E + 17), fma(__ldg(E + 102), g202, fma(__ldg(E + 101), g201, __ldg(E + 100) * g200)), z);
      o6_0 = fma(Ei.w(18), z, o6_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 10) * __ldg(E + 45), fma(__ldg(E + 102), g002, fma(__ldg(E + 101), g001, __ldg(E + 100) * g000)), z);
      z = fma(__ldg(E + 10) * __ldg(E + 46), fma(__ldg(E + 102), g012, fma(__ldg(E + 101), g011, __ldg(E + 100) * g010)), z);
      z = fma(__ldg(E + 11) * __ldg(E + 45), fma(__ldg(E + 102), g102, fma(__ldg(E + 101), g101, __ldg(E + 100) * g100)), z);
      z = fma(__ldg(E + 11) * __ldg(E + 46), fma(__ldg(E + 102), g112, fma(__ldg(E + 101), g111, __ldg(E + 100) * g110)), z);
      o6_1 = fma(Ei.w(19), z, o6_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 10), fma(__ldg(E + 108), g003, fma(__ldg(E + 107), g002, fma(__ldg(E + 106), g001, __ldg(E + 105) * g000))), z);
      z = fma(__ldg(E + 11), fma(__ldg(E + 108), g103, fma(__ldg(E + 107), g102, fma(__ldg(E + 106), g101, __ldg(E + 105) * g100))), z);
      o6_2 = fma(Ei.w(20), z, o6_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 5) * __ldg(E + 60), fma(__ldg(E + 91), g001, __ldg(E + 90) * g000), z);
      z = fma(__ldg(E + 5) * __ldg(E + 61), fma(__ldg(E + 91), g011, __ldg(E + 90) * g010), z);
      z = fma(__ldg(E + 5) * __ldg(E + 62), fma(__ldg(E + 91), g021, __ldg(E + 90) * g020), z);
      z = fma(__ldg(E + 6) * __ldg(E + 60), fma(__ldg(E + 91), g101, __ldg(E + 90) * g100), z);
      z = fma(__ldg(E + 6) * __ldg(E + 61), fma(__ldg(E + 91), g111, __ldg(E + 90) * g110), z);
      z = fma(__ldg(E + 6) * __ldg(E + 62), fma(__ldg(E + 91), g121, __ldg(E + 90) * g120), z);
      o7_0 = fma(Ei.w(21), z, o7_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 65), fma(__ldg(E + 91), g001, __ldg(E + 90) * g000), z);
      z = fma(__ldg(E + 66), fma(__ldg(E + 91), g011, __ldg(E + 90) * g010), z);
      z = fma(__ldg(E + 67), fma(__ldg(E + 91), g021, __ldg(E + 90) * g020), z);
      z = fma(__ldg(E + 68), fma(__ldg(E + 91), g031, __ldg(E + 90) * g030), z);
      o7_1 = fma(Ei.w(22), z, o7_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 60), fma(__ldg(E + 97), g002, fma(__ldg(E + 96), g001, __ldg(E + 95) * g000)), z);
      z = fma(__ldg(E + 61), fma(__ldg(E + 97), g012, fma(__ldg(E + 96), g011, __ldg(E + 95) * g010)), z);
      z = fma(__ldg(E + 62), fma(__ldg(E + 97), g022, fma(__ldg(E + 96), g021, __ldg(E + 95) * g020)), z);
      o7_2 = fma(Ei.w(23), z, o7_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 5) * __ldg(E + 50), fma(__ldg(E + 102), g002, fma(__ldg(E + 101), g001, __ldg(E + 100) * g000)), z);
      z = fma(__ldg(E + 5) * __ldg(E + 51), fma(__ldg(E + 102), g012, fma(__ldg(E + 101), g011, __ldg(E + 100) * g010)), z);
      z = fma(__ldg(E + 6) * __ldg(E + 50), fma(__ldg(E + 102), g102, fma(__ldg(E + 101), g101, __ldg(E + 100) * g100)), z);
      z = fma(__ldg(E + 6) * __ldg(E + 51), fma(__ldg(E + 102), g112, fma(__ldg(E + 101), g111, __ldg(E + 100) * g110)), z);
      o8_0 = fma(Ei.w(24), z, o8_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 55), fma(__ldg(E + 102), g002, fma(__ldg(E + 101), g001, __ldg(E + 100) * g000)), z);
      z = fma(__ldg(E + 56), fma(__ldg(E + 102), g012, fma(__ldg(E + 101), g011, __ldg(E + 100) * g010)), z);
      z = fma(__ldg(E + 57), fma(__ldg(E + 102), g022, fma(__ldg(E + 101), g021, __ldg(E + 100) * g020)), z);
      o8_1 = fma(Ei.w(25), z, o8_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 50), fma(__ldg(E + 108), g003, fma(__ldg(E + 107), g002, fma(__ldg(E + 106), g001, __ldg(E + 105) * g000))), z);
      z = fma(__ldg(E + 51), fma(__ldg(E + 108), g013, fma(__ldg(E + 107), g012, fma(__ldg(E + 106), g011, __ldg(E + 105) * g010))), z);
      o8_2 = fma(Ei.w(26), z, o8_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 15) * __ldg(E + 50), fma(__ldg(E + 91), g001, __ldg(E + 90) * g000), z);
      z = fma(__ldg(E + 15) * __ldg(E + 51), fma(__ldg(E + 91), g011, __ldg(E + 90) * g010), z);
      z = fma(__ldg(E + 16) * __ldg(E + 50), fma(__ldg(E + 91), g101, __ldg(E + 90) * g100), z);
      z = fma(__ldg(E + 16) * __ldg(E + 51), fma(__ldg(E + 91), g111, __ldg(E + 90) * g110), z);
      z = fma(__ldg(E + 17) * __ldg(E + 50), fma(__ldg(E + 91), g201, __ldg(E + 90) * g200), z);
      z = fma(__ldg(E + 17) * __ldg(E + 51), fma(__ldg(E + 91), g211, __ldg(E + 90) * g210), z);
      o9_0 = fma(Ei.w(27), z, o9_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 10) * __ldg(E + 55), fma(__ldg(E + 91), g001, __ldg(E + 90) * g000), z);
      z = fma(__ldg(E + 10) * __ldg(E + 56), fma(__ldg(E + 91), g011, __ldg(E + 90) * g010), z);
      z = fma(__ldg(E + 10) * __ldg(E + 57), fma(__ldg(E + 91), g021, __ldg(E + 90) * g020), z);
      z = fma(__ldg(E + 11) * __ldg(E + 55), fma(__ldg(E + 91), g101, __ldg(E + 90) * g100), z);
      z = fma(__ldg(E + 11) * __ldg(E + 56), fma(__ldg(E + 91), g111, __ldg(E + 90) * g110), z);
      z = fma(__ldg(E + 11) * __ldg(E + 57), fma(__ldg(E + 91), g121, __ldg(E + 90) * g120), z);
      o9_1 = fma(Ei.w(28), z, o9_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 10) * __ldg(E + 50), fma(__ldg(E + 97), g002, fma(__ldg(E + 96), g001, __ldg(E + 95) * g000)), z);
      z = fma(__ldg(E + 10) * __ldg(E + 51), fma(__ldg(E + 97), g012, fma(__ldg(E + 96), g011, __ldg(E + 95) * g010)), z);
      z = fma(__ldg(E + 11) * __ldg(E + 50), fma(__ldg(E + 97), g102, fma(__ldg(E + 96), g101, __ldg(E + 95) * g100)), z);
      z = fma(__ldg(E + 11) * __ldg(E + 51), fma(__ldg(E + 97), g112, fma(__ldg(E + 96), g111, __ldg(E + 95) * g110)), z);
      o9_2 = fma(Ei.w(29), z, o9_2); }
    if (ok) nfl += 896;
  }
  const int N = a.b.nbf, fP = A.fP, fQ = A.fQ;
  const int fc = B.fP + cd / B.nfQ, fd = B.fQ + cd % B.nfQ;
  const double* __restrict__ PT = a.b.PT;
  const double s2 = 2.0 * deg;
  if (ok) {
    double z = 0.0;
    z = fma(o0_0, __ldg(PT + (fP + 0) * N + fQ + 0), z);
    z = fma(o0_1, __ldg(PT + (fP + 0) * N + fQ + 1), z);
    z = fma(o0_2, __ldg(PT + (fP + 0) * N + fQ + 2), z);
    z = fma(o1_0, __ldg(PT + (fP + 1) * N + fQ + 0), z);
    z = fma(o1_1, __ldg(PT + (fP + 1) * N + fQ + 1), z);
    z = fma(o1_2, __ldg(PT + (fP + 1) * N + fQ + 2), z);
    z = fma(o2_0, __ldg(PT + (fP + 2) * N + fQ + 0), z);
    z = fma(o2_1, __ldg(PT + (fP + 2) * N + fQ + 1), z);
    z = fma(o2_2, __ldg(PT + (fP + 2) * N + fQ + 2), z);
    z = fma(o3_0, __ldg(PT + (fP + 3) * N + fQ + 0), z);
    z = fma(o3_1, __ldg(PT + (fP + 3) * N + fQ + 1), z);
    z = fma(o3_2, __ldg(PT + (fP + 3) * N + fQ + 2), z);
    z = fma(o4_0, __ldg(PT + (fP + 4) * N + fQ + 0), z);
    z = fma(o4_1, __ldg(PT + (fP + 4) * N + fQ + 1), z);
    z = fma(o4_2, __ldg(PT + (fP + 4) * N + fQ + 2), z);
    z = fma(o5_0, __ldg(PT + (fP + 5) * N + fQ + 0), z);
    z = fma(o5_1, __ldg(PT + (fP + 5) * N + fQ + 1), z);
    z = fma(o5_2, __ldg(PT + (fP + 5) * N + fQ + 2), z);
    z = fma(o6_0, __ldg(PT + (fP + 6) * N + fQ + 0), z);
    z = fma(o6_1, __ldg(PT + (fP + 6) * N + fQ + 1), z);
    z = fma(o6_2, __ldg(PT + (fP + 6) * N + fQ + 2), z);
    z = fma(o7_0, __ldg(PT + (fP + 7) * N + fQ + 0), z);
    z = fma(o7_1, __ldg(PT + (fP + 7) * N + fQ + 1), z);
    z = fma(o7_2, __ldg(PT + (fP + 7) * N + fQ + 2), z);
    z = fma(o8_0, __ldg(PT + (fP + 8) * N + fQ + 0), z);
    z = fma(o8_1, __ldg(PT + (fP + 8) * N + fQ + 1), z);
    z = fma(o8_2, __ldg(PT + (fP + 8) * N + fQ + 2), z);
    z = fma(o9_0, __ldg(PT + (fP + 9) * N + fQ + 0), z);
    z = fma(o9_1, __ldg(PT + (fP + 9) * N + fQ + 1), z);
    z = fma(o9_2, __ldg(PT + (fP + 9) * N + fQ + 2), z);
    atomicAdd(a.b.J + fc * N + fd, s2 * z);
    for (int sp = 0; sp < (a.b.uhf ? 2 : 1); ++sp) {
      const double* __restrict__ D = sp ? a.b.PB : a.b.PA;
      double* __restrict__ K = sp ? a.b.KB : a.b.KA;
      {  // K[p][c], K[q][c] from D[.][d]
        const double q0 = D[(fQ + 0) * N + fd];
        double kq0 = 0.0;
        const double q1 = D[(fQ + 1) * N + fd];
        double kq1 = 0.0;
        const double q2 = D[(fQ + 2) * N + fd];
        double kq2 = 0.0;
        { const double px = D[(fP + 0) * N + fd]; double kp = 0.0;
          kp = fma(o0_0, q0, kp); kq0 = fma(o0_0, px, kq0);
          kp = fma(o0_1, q1, kp); kq1 = fma(o0_1, px, kq1);
          kp = fma(o0_2, q2, kp); kq2 = fma(o0_2, px, kq2);
          atomicAdd(K + (fP + 0) * N + fc, deg * kp); }
        { const double px = D[(fP + 1) * N + fd]; double kp = 0.0;
          kp = fma(o1_0, q0, kp); kq0 = fma(o1_0, px, kq0);
          kp = fma(o1_1, q1, kp); kq1 = fma(o1_1, px, kq1);
          kp = fma(o1_2, q2, kp); kq2 = fma(o1_2, px, kq2);
          atomicAdd(K + (fP + 1) * N + fc, deg * kp); }
        { const double px = D[(fP + 2) * N + fd]; double kp = 0.0;
          kp = fma(o2_0, q0, kp); kq0 = fma(o2_0, px, kq0);
          kp = fma(o2_1, q1, kp); kq1 = fma(o2_1, px, kq1);
          kp = fma(o2_2, q2, kp); kq2 = fma(o2_2, px, kq2);
          atomicAdd(K + (fP + 2) * N + fc, deg * kp); }
        { const double px = D[(fP + 3) * N + fd]; double kp = 0.0;
          kp = fma(o3_0, q0, kp); kq0 = fma(o3_0, px, kq0);
          kp = fma(o3_1, q1, kp); kq1 = fma(o3_1, px, kq1);
          kp = fma(o3_2, q2, kp); kq2 = fma(o3_2, px, kq2);
          atomicAdd(K + (fP + 3) * N + fc, deg * kp); }
        { const double px = D[(fP + 4) * N + fd]; double kp = 0.0;
          kp = fma(o4_0, q0, kp); kq0 = fma(o4_0, px, kq0);
          kp = fma(o4_1, q1, kp); kq1 = fma(o4_1, px, kq1);
          kp = fma(o4_2, q2, kp); kq2 = fma(o4_2, px, kq2);
          atomicAdd(K + (fP + 4) * N + fc, deg * kp); }
        { const double px = D[(fP + 5) * N + fd]; double kp = 0.0;
          kp = fma(o5_0, q0, kp); kq0 = fma(o5_0, px, kq0);
          kp = fma(o5_1, q1, kp); kq1 = fma(o5_1, px, kq1);
          kp = fma(o5_2, q2, kp); kq2 = fma(o5_2, px, kq2);
          atomicAdd(K + (fP + 5) * N + fc, deg * kp); }
        { const double px = D[(fP + 6) * N + fd]; double kp = 0.0;
          kp = fma(o6_0, q0, kp); kq0 = fma(o6_0, px, kq0);
          kp = fma(o6_1, q1, kp); kq1 = fma(o6_1, px, kq1);
          kp = fma(o6_2, q2, kp); kq2 = fma(o6_2, px, kq2);
          atomicAdd(K + (fP + 6) * N + fc, deg * kp); }
        { const double px = D[(fP + 7) * N + fd]; double kp = 0.0;
          kp = fma(o7_0, q0, kp); kq0 = fma(o7_0, px, kq0);
          kp = fma(o7_1, q1, kp); kq1 = fma(o7_1, px, kq1);
          kp = fma(o7_2, q2, kp); kq2 = fma(o7_2, px, kq2);
          atomicAdd(K + (fP + 7) * N + fc, deg * kp); }
        { const double px = D[(fP + 8) * N + fd]; double kp = 0.0;
          kp = fma(o8_0, q0, kp); kq0 = fma(o8_0, px, kq0);
          kp = fma(o8_1, q1, kp); kq1 = fma(o8_1, px, kq1);
          kp = fma(o8_2, q2, kp); kq2 = fma(o8_2, px, kq2);
          atomicAdd(K + (fP + 8) * N + fc, deg * kp); }
        { const double px = D[(fP + 9) * N + fd]; double kp = 0.0;
          kp = fma(o9_0, q0, kp); kq0 = fma(o9_0, px, kq0);
          kp = fma(o9_1, q1, kp); kq1 = fma(o9_1, px, kq1);
          kp = fma(o9_2, q2, kp); kq2 = fma(o9_2, px, kq2);
          atomicAdd(K + (fP + 9) * N + fc, deg * kp); }
        atomicAdd(K + (fQ + 0) * N + fc, deg * kq0);
        atomicAdd(K + (fQ + 1) * N + fc, deg * kq1);
        atomicAdd(K + (fQ + 2) * N + fc, deg * kq2);
      }
      {  // K[p][d], K[q][d] from D[.][c]
        const double q0 = D[(fQ + 0) * N + fc];
        double kq0 = 0.0;
        const double q1 = D[(fQ + 1) * N + fc];
        double kq1 = 0.0;
        const double q2 = D[(fQ + 2) * N + fc];
        double kq2 = 0.0;
        { const double px = D[(fP + 0) * N + fc]; double kp = 0.0;
          kp = fma(o0_0, q0, kp); kq0 = fma(o0_0, px, kq0);
          kp = fma(o0_1, q1, kp); kq1 = fma(o0_1, px, kq1);
          kp = fma(o0_2, q2, kp); kq2 = fma(o0_2, px, kq2);
          atomicAdd(K + (fP + 0) * N + fd, deg * kp); }
        { const double px = D[(fP + 1) * N + fc]; double kp = 0.0;
          kp = fma(o1_0, q0, kp); kq0 = fma(o1_0, px, kq0);
          kp = fma(o1_1, q1, kp); kq1 = fma(o1_1, px, kq1);
          kp = fma(o1_2, q2, kp); kq2 = fma(o1_2, px, kq2);
          atomicAdd(K + (fP + 1) * N + fd, deg * kp); }
        { const double px = D[(fP + 2) * N + fc]; double kp = 0.0;
          kp = fma(o2_0, q0, kp); kq0 = fma(o2_0, px, kq0);
          kp = fma(o2_1, q1, kp); kq1 = fma(o2_1, px, kq1);
          kp = fma(o2_2, q2, kp); kq2 = fma(o2_2, px, kq2);
          atomicAdd(K + (fP + 2) * N + fd, deg * kp); }
        { const double px = D[(fP + 3) * N + fc]; double kp = 0.0;
          kp = fma(o3_0, q0, kp); kq0 = fma(o3_0, px, kq0);
          kp = fma(o3_1, q1, kp); kq1 = fma(o3_1, px, kq1);
          kp = fma(o3_2, q2, kp); kq2 = fma(o3_2, px, kq2);
          atomicAdd(K + (fP + 3) * N + fd, deg * kp); }
        { const double px = D[(fP + 4) * N + fc]; double kp = 0.0;
          kp = fma(o4_0, q0, kp); kq0 = fma(o4_0, px, kq0);
          kp = fma(o4_1, q1, kp); kq1 = fma(o4_1, px, kq1);
          kp = fma(o4_2, q2, kp); kq2 = fma(o4_2, px, kq2);
          atomicAdd(K + (fP + 4) * N + fd, deg * kp); }
        { const double px = D[(fP + 5) * N + fc]; double kp = 0.0;
          kp = fma(o5_0, q0, kp); kq0 = fma(o5_0, px, kq0);
          kp = fma(o5_1, q1, kp); kq1 = fma(o5_1, px, kq1);
          kp = fma(o5_2, q2, kp); kq2 = fma(o5_2, px, kq2);
          atomicAdd(K + (fP + 5) * N + fd, deg * kp); }
        { const double px = D[(fP + 6) * N + fc]; double kp = 0.0;
          kp = fma(o6_0, q0, kp); kq0 = fma(o6_0, px, kq0);
          kp = fma(o6_1, q1, kp); kq1 = fma(o6_1, px, kq1);
          kp = fma(o6_2, q2, kp); kq2 = fma(o6_2, px, kq2);
          atomicAdd(K + (fP + 6) * N + fd, deg * kp); }
        { const double px = D[(fP + 7) * N + fc]; double kp = 0.0;
          kp = fma(o7_0, q0, kp); kq0 = fma(o7_0, px, kq0);
          kp = fma(o7_1, q1, kp); kq1 = fma(o7_1, px, kq1);
          kp = fma(o7_2, q2, kp); kq2 = fma(o7_2, px, kq2);
          atomicAdd(K + (fP + 7) * N + fd, deg * kp); }
        { const double px = D[(fP + 8) * N + fc]; double kp = 0.0;
          kp = fma(o8_0, q0, kp); kq0 = fma(o8_0, px, kq0);
          kp = fma(o8_1, q1, kp); kq1 = fma(o8_1, px, kq1);
          kp = fma(o8_2, q2, kp); kq2 = fma(o8_2, px, kq2);
          atomicAdd(K + (fP + 8) * N + fd, deg * kp); }
        { const double px = D[(fP + 9) * N + fc]; double kp = 0.0;
          kp = fma(o9_0, q0, kp); kq0 = fma(o9_0, px, kq0);
          kp = fma(o9_1, q1, kp); kq1 = fma(o9_1, px, kq1);
          kp = fma(o9_2, q2, kp); kq2 = fma(o9_2, px, kq2);
          atomicAdd(K + (fP + 9) * N + fd, deg * kp); }
        atomicAdd(K + (fQ + 0) * N + fd, deg * kq0);
        atomicAdd(K + (fQ + 1) * N + fd, deg * kq1);
        atomicAdd(K + (fQ + 2) * N + fd, deg * kq2);
      }
    }
    nfl += 2ull * 30 * (2 + 4 * (a.b.uhf ? 2 : 1));
  }
  {  // J[p][q]: every lane shares the bra pair
    const double w = ok ? s2 * __ldg(PT + fc * N + fd) : 0.0;
    { double v[32] = {w * o0_0, w * o0_1, w * o0_2, w * o1_0, w * o1_1, w * o1_2, w * o2_0, w * o2_1, w * o2_2, w * o3_0, w * o3_1, w * o3_2, w * o4_0, w * o4_1, w * o4_2, w * o5_0, w * o5_1, w * o5_2, w * o6_0, w * o6_1, w * o6_2, w * o7_0, w * o7_1, w * o7_2, w * o8_0, w * o8_1, w * o8_2, w * o9_0, w * o9_1, w * o9_2, 0.0, 0.0};
      const double z = sqb::warp_sum_scatter<32>(v); const int x = lane + 0;
      if (lane < 30 && z != 0.0) atomicAdd(a.b.J + (fP + 0 + x / 3) * N + fQ + x % 3, z); }
  }
  sqb::count_add(a.counters + 0, ok && cd == 0 && gi == 0 && gj == 0 ? 1ull : 0ull);
  sqb::count_add(a.counters + 1, npq);
  sqb::count_add(a.counters + 2, nfl);
}
