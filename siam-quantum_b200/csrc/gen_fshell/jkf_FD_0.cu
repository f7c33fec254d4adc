// generated by gen_fshell_kernels.py -- do not edit
#include "../jk_generic_dev.cuh"

extern "C" __global__ void __launch_bounds__(128)
jkf_FD_0(const sqb::FArgs a, const sqb::FRun* __restrict__ runs, const long long* __restrict__ first, int nruns,
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
  const int L = 5 + B.lP + B.lQ, S1 = L + 1, S2 = S1 * S1;   // uniform over the warp
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
  double o0_3 = 0.0;
  double o0_4 = 0.0;
  double o0_5 = 0.0;
  double o1_0 = 0.0;
  double o1_1 = 0.0;
  double o1_2 = 0.0;
  double o1_3 = 0.0;
  double o1_4 = 0.0;
  double o1_5 = 0.0;
  double o2_0 = 0.0;
  double o2_1 = 0.0;
  double o2_2 = 0.0;
  double o2_3 = 0.0;
  double o2_4 = 0.0;
  double o2_5 = 0.0;
  double o3_0 = 0.0;
  double o3_1 = 0.0;
  double o3_2 = 0.0;
  double o3_3 = 0.0;
  double o3_4 = 0.0;
  double o3_5 = 0.0;
  double o4_0 = 0.0;
  double o4_1 = 0.0;
  double o4_2 = 0.0;
  double o4_3 = 0.0;
  double o4_4 = 0.0;
  double o4_5 = 0.0;
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
    double g500 = 0.0;
    double g410 = 0.0;
    double g401 = 0.0;
    double g320 = 0.0;
    double g311 = 0.0;
    double g302 = 0.0;
    double g230 = 0.0;
    double g221 = 0.0;
    double g212 = 0.0;
    double g203 = 0.0;
    double g140 = 0.0;
    double g131 = 0.0;
    double g122 = 0.0;
    double g113 = 0.0;
    double g104 = 0.0;
    double g050 = 0.0;
    double g041 = 0.0;
    double g032 = 0.0;
    double g023 = 0.0;
    double g014 = 0.0;
    double g005 = 0.0;
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
            g005 = fma(e, x[5], g005);
          }
          { const double* __restrict__ x = R + 0 * S2 + 1 * S1;
            g010 = fma(e, x[0], g010);
            g011 = fma(e, x[1], g011);
            g012 = fma(e, x[2], g012);
            g013 = fma(e, x[3], g013);
            g014 = fma(e, x[4], g014);
          }
          { const double* __restrict__ x = R + 0 * S2 + 2 * S1;
            g020 = fma(e, x[0], g020);
            g021 = fma(e, x[1], g021);
            g022 = fma(e, x[2], g022);
            g023 = fma(e, x[3], g023);
          }
          { const double* __restrict__ x = R + 0 * S2 + 3 * S1;
            g030 = fma(e, x[0], g030);
            g031 = fma(e, x[1], g031);
            g032 = fma(e, x[2], g032);
          }
          { const double* __restrict__ x = R + 0 * S2 + 4 * S1;
            g040 = fma(e, x[0], g040);
            g041 = fma(e, x[1], g041);
          }
          { const double* __restrict__ x = R + 0 * S2 + 5 * S1;
            g050 = fma(e, x[0], g050);
          }
          { const double* __restrict__ x = R + 1 * S2 + 0 * S1;
            g100 = fma(e, x[0], g100);
            g101 = fma(e, x[1], g101);
            g102 = fma(e, x[2], g102);
            g103 = fma(e, x[3], g103);
            g104 = fma(e, x[4], g104);
          }
          { const double* __restrict__ x = R + 1 * S2 + 1 * S1;
            g110 = fma(e, x[0], g110);
            g111 = fma(e, x[1], g111);
            g112 = fma(e, x[2], g112);
            g113 = fma(e, x[3], g113);
          }
          { const double* __restrict__ x = R + 1 * S2 + 2 * S1;
            g120 = fma(e, x[0], g120);
            g121 = fma(e, x[1], g121);
            g122 = fma(e, x[2], g122);
          }
          { const double* __restrict__ x = R + 1 * S2 + 3 * S1;
            g130 = fma(e, x[0], g130);
            g131 = fma(e, x[1], g131);
          }
          { const double* __restrict__ x = R + 1 * S2 + 4 * S1;
            g140 = fma(e, x[0], g140);
          }
          { const double* __restrict__ x = R + 2 * S2 + 0 * S1;
            g200 = fma(e, x[0], g200);
            g201 = fma(e, x[1], g201);
            g202 = fma(e, x[2], g202);
            g203 = fma(e, x[3], g203);
          }
          { const double* __restrict__ x = R + 2 * S2 + 1 * S1;
            g210 = fma(e, x[0], g210);
            g211 = fma(e, x[1], g211);
            g212 = fma(e, x[2], g212);
          }
          { const double* __restrict__ x = R + 2 * S2 + 2 * S1;
            g220 = fma(e, x[0], g220);
            g221 = fma(e, x[1], g221);
          }
          { const double* __restrict__ x = R + 2 * S2 + 3 * S1;
            g230 = fma(e, x[0], g230);
          }
          { const double* __restrict__ x = R + 3 * S2 + 0 * S1;
            g300 = fma(e, x[0], g300);
            g301 = fma(e, x[1], g301);
            g302 = fma(e, x[2], g302);
          }
          { const double* __restrict__ x = R + 3 * S2 + 1 * S1;
            g310 = fma(e, x[0], g310);
            g311 = fma(e, x[1], g311);
          }
          { const double* __restrict__ x = R + 3 * S2 + 2 * S1;
            g320 = fma(e, x[0], g320);
          }
          { const double* __restrict__ x = R + 4 * S2 + 0 * S1;
            g400 = fma(e, x[0], g400);
            g401 = fma(e, x[1], g401);
          }
          { const double* __restrict__ x = R + 4 * S2 + 1 * S1;
            g410 = fma(e, x[0], g410);
          }
          { const double* __restrict__ x = R + 5 * S2 + 0 * S1;
            g500 = fma(e, x[0], g500);
          }
          if (++ph == n2) { ph = 0; if (++nu == n1) { nu = 0; ++tau; } }
        }
        nfl += 2ull * 56 * nk;
      }
    }
    if (!any) continue;
    const sqb::EView Ei(a.coef, pa, A);
    const double* __restrict__ E = Ei.e;
    { double z = 0.0;
      z = fma(__ldg(E + 66), g000, z);
      z = fma(__ldg(E + 67), g100, z);
      z = fma(__ldg(E + 68), g200, z);
      z = fma(__ldg(E + 69), g300, z);
      z = fma(__ldg(E + 70), g400, z);
      z = fma(__ldg(E + 71), g500, z);
      o0_0 = fma(Ei.w(0), z, o0_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 54) * __ldg(E + 84), g000, z);
      z = fma(__ldg(E + 54) * __ldg(E + 85), g010, z);
      z = fma(__ldg(E + 54) * __ldg(E + 86), g020, z);
      z = fma(__ldg(E + 55) * __ldg(E + 84), g100, z);
      z = fma(__ldg(E + 55) * __ldg(E + 85), g110, z);
      z = fma(__ldg(E + 55) * __ldg(E + 86), g120, z);
      z = fma(__ldg(E + 56) * __ldg(E + 84), g200, z);
      z = fma(__ldg(E + 56) * __ldg(E + 85), g210, z);
      z = fma(__ldg(E + 56) * __ldg(E + 86), g220, z);
      z = fma(__ldg(E + 57) * __ldg(E + 84), g300, z);
      z = fma(__ldg(E + 57) * __ldg(E + 85), g310, z);
      z = fma(__ldg(E + 57) * __ldg(E + 86), g320, z);
      o0_1 = fma(Ei.w(1), z, o0_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 54), fma(__ldg(E + 158), g002, fma(__ldg(E + 157), g001, __ldg(E + 156) * g000)), z);
      z = fma(__ldg(E + 55), fma(__ldg(E + 158), g102, fma(__ldg(E + 157), g101, __ldg(E + 156) * g100)), z);
      z = fma(__ldg(E + 56), fma(__ldg(E + 158), g202, fma(__ldg(E + 157), g201, __ldg(E + 156) * g200)), z);
      z = fma(__ldg(E + 57), fma(__ldg(E + 158), g302, fma(__ldg(E + 157), g301, __ldg(E + 156) * g300)), z);
      o0_2 = fma(Ei.w(2), z, o0_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 60) * __ldg(E + 78), g000, z);
      z = fma(__ldg(E + 60) * __ldg(E + 79), g010, z);
      z = fma(__ldg(E + 61) * __ldg(E + 78), g100, z);
      z = fma(__ldg(E + 61) * __ldg(E + 79), g110, z);
      z = fma(__ldg(E + 62) * __ldg(E + 78), g200, z);
      z = fma(__ldg(E + 62) * __ldg(E + 79), g210, z);
      z = fma(__ldg(E + 63) * __ldg(E + 78), g300, z);
      z = fma(__ldg(E + 63) * __ldg(E + 79), g310, z);
      z = fma(__ldg(E + 64) * __ldg(E + 78), g400, z);
      z = fma(__ldg(E + 64) * __ldg(E + 79), g410, z);
      o0_3 = fma(Ei.w(3), z, o0_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 60), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 61), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 62), fma(__ldg(E + 151), g201, __ldg(E + 150) * g200), z);
      z = fma(__ldg(E + 63), fma(__ldg(E + 151), g301, __ldg(E + 150) * g300), z);
      z = fma(__ldg(E + 64), fma(__ldg(E + 151), g401, __ldg(E + 150) * g400), z);
      o0_4 = fma(Ei.w(4), z, o0_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 54) * __ldg(E + 78), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 54) * __ldg(E + 79), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 55) * __ldg(E + 78), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 55) * __ldg(E + 79), fma(__ldg(E + 151), g111, __ldg(E + 150) * g110), z);
      z = fma(__ldg(E + 56) * __ldg(E + 78), fma(__ldg(E + 151), g201, __ldg(E + 150) * g200), z);
      z = fma(__ldg(E + 56) * __ldg(E + 79), fma(__ldg(E + 151), g211, __ldg(E + 150) * g210), z);
      z = fma(__ldg(E + 57) * __ldg(E + 78), fma(__ldg(E + 151), g301, __ldg(E + 150) * g300), z);
      z = fma(__ldg(E + 57) * __ldg(E + 79), fma(__ldg(E + 151), g311, __ldg(E + 150) * g310), z);
      o0_5 = fma(Ei.w(5), z, o0_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 12) * __ldg(E + 126), g000, z);
      z = fma(__ldg(E + 12) * __ldg(E + 127), g010, z);
      z = fma(__ldg(E + 12) * __ldg(E + 128), g020, z);
      z = fma(__ldg(E + 12) * __ldg(E + 129), g030, z);
      z = fma(__ldg(E + 13) * __ldg(E + 126), g100, z);
      z = fma(__ldg(E + 13) * __ldg(E + 127), g110, z);
      z = fma(__ldg(E + 13) * __ldg(E + 128), g120, z);
      z = fma(__ldg(E + 13) * __ldg(E + 129), g130, z);
      z = fma(__ldg(E + 14) * __ldg(E + 126), g200, z);
      z = fma(__ldg(E + 14) * __ldg(E + 127), g210, z);
      z = fma(__ldg(E + 14) * __ldg(E + 128), g220, z);
      z = fma(__ldg(E + 14) * __ldg(E + 129), g230, z);
      o1_0 = fma(Ei.w(6), z, o1_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 138), g000, z);
      z = fma(__ldg(E + 139), g010, z);
      z = fma(__ldg(E + 140), g020, z);
      z = fma(__ldg(E + 141), g030, z);
      z = fma(__ldg(E + 142), g040, z);
      z = fma(__ldg(E + 143), g050, z);
      o1_1 = fma(Ei.w(7), z, o1_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 126), fma(__ldg(E + 158), g002, fma(__ldg(E + 157), g001, __ldg(E + 156) * g000)), z);
      z = fma(__ldg(E + 127), fma(__ldg(E + 158), g012, fma(__ldg(E + 157), g011, __ldg(E + 156) * g010)), z);
      z = fma(__ldg(E + 128), fma(__ldg(E + 158), g022, fma(__ldg(E + 157), g021, __ldg(E + 156) * g020)), z);
      z = fma(__ldg(E + 129), fma(__ldg(E + 158), g032, fma(__ldg(E + 157), g031, __ldg(E + 156) * g030)), z);
      o1_2 = fma(Ei.w(8), z, o1_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 132), g000, z);
      z = fma(__ldg(E + 6) * __ldg(E + 133), g010, z);
      z = fma(__ldg(E + 6) * __ldg(E + 134), g020, z);
      z = fma(__ldg(E + 6) * __ldg(E + 135), g030, z);
      z = fma(__ldg(E + 6) * __ldg(E + 136), g040, z);
      z = fma(__ldg(E + 7) * __ldg(E + 132), g100, z);
      z = fma(__ldg(E + 7) * __ldg(E + 133), g110, z);
      z = fma(__ldg(E + 7) * __ldg(E + 134), g120, z);
      z = fma(__ldg(E + 7) * __ldg(E + 135), g130, z);
      z = fma(__ldg(E + 7) * __ldg(E + 136), g140, z);
      o1_3 = fma(Ei.w(9), z, o1_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 126), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 6) * __ldg(E + 127), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 6) * __ldg(E + 128), fma(__ldg(E + 151), g021, __ldg(E + 150) * g020), z);
      z = fma(__ldg(E + 6) * __ldg(E + 129), fma(__ldg(E + 151), g031, __ldg(E + 150) * g030), z);
      z = fma(__ldg(E + 7) * __ldg(E + 126), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 7) * __ldg(E + 127), fma(__ldg(E + 151), g111, __ldg(E + 150) * g110), z);
      z = fma(__ldg(E + 7) * __ldg(E + 128), fma(__ldg(E + 151), g121, __ldg(E + 150) * g120), z);
      z = fma(__ldg(E + 7) * __ldg(E + 129), fma(__ldg(E + 151), g131, __ldg(E + 150) * g130), z);
      o1_4 = fma(Ei.w(10), z, o1_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 132), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 133), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 134), fma(__ldg(E + 151), g021, __ldg(E + 150) * g020), z);
      z = fma(__ldg(E + 135), fma(__ldg(E + 151), g031, __ldg(E + 150) * g030), z);
      z = fma(__ldg(E + 136), fma(__ldg(E + 151), g041, __ldg(E + 150) * g040), z);
      o1_5 = fma(Ei.w(11), z, o1_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 12), fma(__ldg(E + 201), g003, fma(__ldg(E + 200), g002, fma(__ldg(E + 199), g001, __ldg(E + 198) * g000))), z);
      z = fma(__ldg(E + 13), fma(__ldg(E + 201), g103, fma(__ldg(E + 200), g102, fma(__ldg(E + 199), g101, __ldg(E + 198) * g100))), z);
      z = fma(__ldg(E + 14), fma(__ldg(E + 201), g203, fma(__ldg(E + 200), g202, fma(__ldg(E + 199), g201, __ldg(E + 198) * g200))), z);
      o2_0 = fma(Ei.w(12), z, o2_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 84), fma(__ldg(E + 201), g003, fma(__ldg(E + 200), g002, fma(__ldg(E + 199), g001, __ldg(E + 198) * g000))), z);
      z = fma(__ldg(E + 85), fma(__ldg(E + 201), g013, fma(__ldg(E + 200), g012, fma(__ldg(E + 199), g011, __ldg(E + 198) * g010))), z);
      z = fma(__ldg(E + 86), fma(__ldg(E + 201), g023, fma(__ldg(E + 200), g022, fma(__ldg(E + 199), g021, __ldg(E + 198) * g020))), z);
      o2_1 = fma(Ei.w(13), z, o2_1); }
    { double z = 0.0;
      z += fma(__ldg(E + 215), g005, fma(__ldg(E + 214), g004, fma(__ldg(E + 213), g003, fma(__ldg(E + 212), g002, fma(__ldg(E + 211), g001, __ldg(E + 210) * g000)))));
      o2_2 = fma(Ei.w(14), z, o2_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 78), fma(__ldg(E + 201), g003, fma(__ldg(E + 200), g002, fma(__ldg(E + 199), g001, __ldg(E + 198) * g000))), z);
      z = fma(__ldg(E + 6) * __ldg(E + 79), fma(__ldg(E + 201), g013, fma(__ldg(E + 200), g012, fma(__ldg(E + 199), g011, __ldg(E + 198) * g010))), z);
      z = fma(__ldg(E + 7) * __ldg(E + 78), fma(__ldg(E + 201), g103, fma(__ldg(E + 200), g102, fma(__ldg(E + 199), g101, __ldg(E + 198) * g100))), z);
      z = fma(__ldg(E + 7) * __ldg(E + 79), fma(__ldg(E + 201), g113, fma(__ldg(E + 200), g112, fma(__ldg(E + 199), g111, __ldg(E + 198) * g110))), z);
      o2_3 = fma(Ei.w(15), z, o2_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 6), fma(__ldg(E + 208), g004, fma(__ldg(E + 207), g003, fma(__ldg(E + 206), g002, fma(__ldg(E + 205), g001, __ldg(E + 204) * g000)))), z);
      z = fma(__ldg(E + 7), fma(__ldg(E + 208), g104, fma(__ldg(E + 207), g103, fma(__ldg(E + 206), g102, fma(__ldg(E + 205), g101, __ldg(E + 204) * g100)))), z);
      o2_4 = fma(Ei.w(16), z, o2_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 78), fma(__ldg(E + 208), g004, fma(__ldg(E + 207), g003, fma(__ldg(E + 206), g002, fma(__ldg(E + 205), g001, __ldg(E + 204) * g000)))), z);
      z = fma(__ldg(E + 79), fma(__ldg(E + 208), g014, fma(__ldg(E + 207), g013, fma(__ldg(E + 206), g012, fma(__ldg(E + 205), g011, __ldg(E + 204) * g010)))), z);
      o2_5 = fma(Ei.w(17), z, o2_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 48) * __ldg(E + 90), g000, z);
      z = fma(__ldg(E + 48) * __ldg(E + 91), g010, z);
      z = fma(__ldg(E + 49) * __ldg(E + 90), g100, z);
      z = fma(__ldg(E + 49) * __ldg(E + 91), g110, z);
      z = fma(__ldg(E + 50) * __ldg(E + 90), g200, z);
      z = fma(__ldg(E + 50) * __ldg(E + 91), g210, z);
      z = fma(__ldg(E + 51) * __ldg(E + 90), g300, z);
      z = fma(__ldg(E + 51) * __ldg(E + 91), g310, z);
      z = fma(__ldg(E + 52) * __ldg(E + 90), g400, z);
      z = fma(__ldg(E + 52) * __ldg(E + 91), g410, z);
      o3_0 = fma(Ei.w(18), z, o3_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 36) * __ldg(E + 102), g000, z);
      z = fma(__ldg(E + 36) * __ldg(E + 103), g010, z);
      z = fma(__ldg(E + 36) * __ldg(E + 104), g020, z);
      z = fma(__ldg(E + 36) * __ldg(E + 105), g030, z);
      z = fma(__ldg(E + 37) * __ldg(E + 102), g100, z);
      z = fma(__ldg(E + 37) * __ldg(E + 103), g110, z);
      z = fma(__ldg(E + 37) * __ldg(E + 104), g120, z);
      z = fma(__ldg(E + 37) * __ldg(E + 105), g130, z);
      z = fma(__ldg(E + 38) * __ldg(E + 102), g200, z);
      z = fma(__ldg(E + 38) * __ldg(E + 103), g210, z);
      z = fma(__ldg(E + 38) * __ldg(E + 104), g220, z);
      z = fma(__ldg(E + 38) * __ldg(E + 105), g230, z);
      o3_1 = fma(Ei.w(19), z, o3_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 36) * __ldg(E + 90), fma(__ldg(E + 158), g002, fma(__ldg(E + 157), g001, __ldg(E + 156) * g000)), z);
      z = fma(__ldg(E + 36) * __ldg(E + 91), fma(__ldg(E + 158), g012, fma(__ldg(E + 157), g011, __ldg(E + 156) * g010)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 90), fma(__ldg(E + 158), g102, fma(__ldg(E + 157), g101, __ldg(E + 156) * g100)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 91), fma(__ldg(E + 158), g112, fma(__ldg(E + 157), g111, __ldg(E + 156) * g110)), z);
      z = fma(__ldg(E + 38) * __ldg(E + 90), fma(__ldg(E + 158), g202, fma(__ldg(E + 157), g201, __ldg(E + 156) * g200)), z);
      z = fma(__ldg(E + 38) * __ldg(E + 91), fma(__ldg(E + 158), g212, fma(__ldg(E + 157), g211, __ldg(E + 156) * g210)), z);
      o3_2 = fma(Ei.w(20), z, o3_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 42) * __ldg(E + 96), g000, z);
      z = fma(__ldg(E + 42) * __ldg(E + 97), g010, z);
      z = fma(__ldg(E + 42) * __ldg(E + 98), g020, z);
      z = fma(__ldg(E + 43) * __ldg(E + 96), g100, z);
      z = fma(__ldg(E + 43) * __ldg(E + 97), g110, z);
      z = fma(__ldg(E + 43) * __ldg(E + 98), g120, z);
      z = fma(__ldg(E + 44) * __ldg(E + 96), g200, z);
      z = fma(__ldg(E + 44) * __ldg(E + 97), g210, z);
      z = fma(__ldg(E + 44) * __ldg(E + 98), g220, z);
      z = fma(__ldg(E + 45) * __ldg(E + 96), g300, z);
      z = fma(__ldg(E + 45) * __ldg(E + 97), g310, z);
      z = fma(__ldg(E + 45) * __ldg(E + 98), g320, z);
      o3_3 = fma(Ei.w(21), z, o3_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 42) * __ldg(E + 90), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 42) * __ldg(E + 91), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 43) * __ldg(E + 90), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 43) * __ldg(E + 91), fma(__ldg(E + 151), g111, __ldg(E + 150) * g110), z);
      z = fma(__ldg(E + 44) * __ldg(E + 90), fma(__ldg(E + 151), g201, __ldg(E + 150) * g200), z);
      z = fma(__ldg(E + 44) * __ldg(E + 91), fma(__ldg(E + 151), g211, __ldg(E + 150) * g210), z);
      z = fma(__ldg(E + 45) * __ldg(E + 90), fma(__ldg(E + 151), g301, __ldg(E + 150) * g300), z);
      z = fma(__ldg(E + 45) * __ldg(E + 91), fma(__ldg(E + 151), g311, __ldg(E + 150) * g310), z);
      o3_4 = fma(Ei.w(22), z, o3_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 36) * __ldg(E + 96), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 36) * __ldg(E + 97), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 36) * __ldg(E + 98), fma(__ldg(E + 151), g021, __ldg(E + 150) * g020), z);
      z = fma(__ldg(E + 37) * __ldg(E + 96), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 37) * __ldg(E + 97), fma(__ldg(E + 151), g111, __ldg(E + 150) * g110), z);
      z = fma(__ldg(E + 37) * __ldg(E + 98), fma(__ldg(E + 151), g121, __ldg(E + 150) * g120), z);
      z = fma(__ldg(E + 38) * __ldg(E + 96), fma(__ldg(E + 151), g201, __ldg(E + 150) * g200), z);
      z = fma(__ldg(E + 38) * __ldg(E + 97), fma(__ldg(E + 151), g211, __ldg(E + 150) * g210), z);
      z = fma(__ldg(E + 38) * __ldg(E + 98), fma(__ldg(E + 151), g221, __ldg(E + 150) * g220), z);
      o3_5 = fma(Ei.w(23), z, o3_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 30) * __ldg(E + 108), g000, z);
      z = fma(__ldg(E + 30) * __ldg(E + 109), g010, z);
      z = fma(__ldg(E + 30) * __ldg(E + 110), g020, z);
      z = fma(__ldg(E + 31) * __ldg(E + 108), g100, z);
      z = fma(__ldg(E + 31) * __ldg(E + 109), g110, z);
      z = fma(__ldg(E + 31) * __ldg(E + 110), g120, z);
      z = fma(__ldg(E + 32) * __ldg(E + 108), g200, z);
      z = fma(__ldg(E + 32) * __ldg(E + 109), g210, z);
      z = fma(__ldg(E + 32) * __ldg(E + 110), g220, z);
      z = fma(__ldg(E + 33) * __ldg(E + 108), g300, z);
      z = fma(__ldg(E + 33) * __ldg(E + 109), g310, z);
      z = fma(__ldg(E + 33) * __ldg(E + 110), g320, z);
      o4_0 = fma(Ei.w(24), z, o4_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 120), g000, z);
      z = fma(__ldg(E + 18) * __ldg(E + 121), g010, z);
      z = fma(__ldg(E + 18) * __ldg(E + 122), g020, z);
      z = fma(__ldg(E + 18) * __ldg(E + 123), g030, z);
      z = fma(__ldg(E + 18) * __ldg(E + 124), g040, z);
      z = fma(__ldg(E + 19) * __ldg(E + 120), g100, z);
      z = fma(__ldg(E + 19) * __ldg(E + 121), g110, z);
      z = fma(__ldg(E + 19) * __ldg(E + 122), g120, z);
      z = fma(__ldg(E + 19) * __ldg(E + 123), g130, z);
      z = fma(__ldg(E + 19) * __ldg(E + 124), g140, z);
      o4_1 = fma(Ei.w(25), z, o4_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 108), fma(__ldg(E + 158), g002, fma(__ldg(E + 157), g001, __ldg(E + 156) * g000)), z);
      z = fma(__ldg(E + 18) * __ldg(E + 109), fma(__ldg(E + 158), g012, fma(__ldg(E + 157), g011, __ldg(E + 156) * g010)), z);
      z = fma(__ldg(E + 18) * __ldg(E + 110), fma(__ldg(E + 158), g022, fma(__ldg(E + 157), g021, __ldg(E + 156) * g020)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 108), fma(__ldg(E + 158), g102, fma(__ldg(E + 157), g101, __ldg(E + 156) * g100)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 109), fma(__ldg(E + 158), g112, fma(__ldg(E + 157), g111, __ldg(E + 156) * g110)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 110), fma(__ldg(E + 158), g122, fma(__ldg(E + 157), g121, __ldg(E + 156) * g120)), z);
      o4_2 = fma(Ei.w(26), z, o4_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 24) * __ldg(E + 114), g000, z);
      z = fma(__ldg(E + 24) * __ldg(E + 115), g010, z);
      z = fma(__ldg(E + 24) * __ldg(E + 116), g020, z);
      z = fma(__ldg(E + 24) * __ldg(E + 117), g030, z);
      z = fma(__ldg(E + 25) * __ldg(E + 114), g100, z);
      z = fma(__ldg(E + 25) * __ldg(E + 115), g110, z);
      z = fma(__ldg(E + 25) * __ldg(E + 116), g120, z);
      z = fma(__ldg(E + 25) * __ldg(E + 117), g130, z);
      z = fma(__ldg(E + 26) * __ldg(E + 114), g200, z);
      z = fma(__ldg(E + 26) * __ldg(E + 115), g210, z);
      z = fma(__ldg(E + 26) * __ldg(E + 116), g220, z);
      z = fma(__ldg(E + 26) * __ldg(E + 117), g230, z);
      o4_3 = fma(Ei.w(27), z, o4_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 24) * __ldg(E + 108), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 24) * __ldg(E + 109), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 24) * __ldg(E + 110), fma(__ldg(E + 151), g021, __ldg(E + 150) * g020), z);
      z = fma(__ldg(E + 25) * __ldg(E + 108), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 25) * __ldg(E + 109), fma(__ldg(E + 151), g111, __ldg(E + 150) * g110), z);
      z = fma(__ldg(E + 25) * __ldg(E + 110), fma(__ldg(E + 151), g121, __ldg(E + 150) * g120), z);
      z = fma(__ldg(E + 26) * __ldg(E + 108), fma(__ldg(E + 151), g201, __ldg(E + 150) * g200), z);
      z = fma(__ldg(E + 26) * __ldg(E + 109), fma(__ldg(E + 151), g211, __ldg(E + 150) * g210), z);
      z = fma(__ldg(E + 26) * __ldg(E + 110), fma(__ldg(E + 151), g221, __ldg(E + 150) * g220), z);
      o4_4 = fma(Ei.w(28), z, o4_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 114), fma(__ldg(E + 151), g001, __ldg(E + 150) * g000), z);
      z = fma(__ldg(E + 18) * __ldg(E + 115), fma(__ldg(E + 151), g011, __ldg(E + 150) * g010), z);
      z = fma(__ldg(E + 18) * __ldg(E + 116), fma(__ldg(E + 151), g021, __ldg(E + 150) * g020), z);
      z = fma(__ldg(E + 18) * __ldg(E + 117), fma(__ldg(E + 151), g031, __ldg(E + 150) * g030), z);
      z = fma(__ldg(E + 19) * __ldg(E + 114), fma(__ldg(E + 151), g101, __ldg(E + 150) * g100), z);
      z = fma(__ldg(E + 19) * __ldg(E + 115), fma(__ldg(E + 151), g111, __ldg(E + 150) * g110), z);
      z = fma(__ldg(E + 19) * __ldg(E + 116), fma(__ldg(E + 151), g121, __ldg(E + 150) * g120), z);
      z = fma(__ldg(E + 19) * __ldg(E + 117), fma(__ldg(E + 151), g131, __ldg(E + 150) * g130), z);
      o4_5 = fma(Ei.w(29), z, o4_5); }
    if (ok) nfl += 1238;
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
    z = fma(o0_3, __ldg(PT + (fP + 0) * N + fQ + 3), z);
    z = fma(o0_4, __ldg(PT + (fP + 0) * N + fQ + 4), z);
    z = fma(o0_5, __ldg(PT + (fP + 0) * N + fQ + 5), z);
    z = fma(o1_0, __ldg(PT + (fP + 1) * N + fQ + 0), z);
    z = fma(o1_1, __ldg(PT + (fP + 1) * N + fQ + 1), z);
    z = fma(o1_2, __ldg(PT + (fP + 1) * N + fQ + 2), z);
    z = fma(o1_3, __ldg(PT + (fP + 1) * N + fQ + 3), z);
    z = fma(o1_4, __ldg(PT + (fP + 1) * N + fQ + 4), z);
    z = fma(o1_5, __ldg(PT + (fP + 1) * N + fQ + 5), z);
    z = fma(o2_0, __ldg(PT + (fP + 2) * N + fQ + 0), z);
    z = fma(o2_1, __ldg(PT + (fP + 2) * N + fQ + 1), z);
    z = fma(o2_2, __ldg(PT + (fP + 2) * N + fQ + 2), z);
    z = fma(o2_3, __ldg(PT + (fP + 2) * N + fQ + 3), z);
    z = fma(o2_4, __ldg(PT + (fP + 2) * N + fQ + 4), z);
    z = fma(o2_5, __ldg(PT + (fP + 2) * N + fQ + 5), z);
    z = fma(o3_0, __ldg(PT + (fP + 3) * N + fQ + 0), z);
    z = fma(o3_1, __ldg(PT + (fP + 3) * N + fQ + 1), z);
    z = fma(o3_2, __ldg(PT + (fP + 3) * N + fQ + 2), z);
    z = fma(o3_3, __ldg(PT + (fP + 3) * N + fQ + 3), z);
    z = fma(o3_4, __ldg(PT + (fP + 3) * N + fQ + 4), z);
    z = fma(o3_5, __ldg(PT + (fP + 3) * N + fQ + 5), z);
    z = fma(o4_0, __ldg(PT + (fP + 4) * N + fQ + 0), z);
    z = fma(o4_1, __ldg(PT + (fP + 4) * N + fQ + 1), z);
    z = fma(o4_2, __ldg(PT + (fP + 4) * N + fQ + 2), z);
    z = fma(o4_3, __ldg(PT + (fP + 4) * N + fQ + 3), z);
    z = fma(o4_4, __ldg(PT + (fP + 4) * N + fQ + 4), z);
    z = fma(o4_5, __ldg(PT + (fP + 4) * N + fQ + 5), z);
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
        const double q3 = D[(fQ + 3) * N + fd];
        double kq3 = 0.0;
        const double q4 = D[(fQ + 4) * N + fd];
        double kq4 = 0.0;
        const double q5 = D[(fQ + 5) * N + fd];
        double kq5 = 0.0;
        { const double px = D[(fP + 0) * N + fd]; double kp = 0.0;
          kp = fma(o0_0, q0, kp); kq0 = fma(o0_0, px, kq0);
          kp = fma(o0_1, q1, kp); kq1 = fma(o0_1, px, kq1);
          kp = fma(o0_2, q2, kp); kq2 = fma(o0_2, px, kq2);
          kp = fma(o0_3, q3, kp); kq3 = fma(o0_3, px, kq3);
          kp = fma(o0_4, q4, kp); kq4 = fma(o0_4, px, kq4);
          kp = fma(o0_5, q5, kp); kq5 = fma(o0_5, px, kq5);
          atomicAdd(K + (fP + 0) * N + fc, deg * kp); }
        { const double px = D[(fP + 1) * N + fd]; double kp = 0.0;
          kp = fma(o1_0, q0, kp); kq0 = fma(o1_0, px, kq0);
          kp = fma(o1_1, q1, kp); kq1 = fma(o1_1, px, kq1);
          kp = fma(o1_2, q2, kp); kq2 = fma(o1_2, px, kq2);
          kp = fma(o1_3, q3, kp); kq3 = fma(o1_3, px, kq3);
          kp = fma(o1_4, q4, kp); kq4 = fma(o1_4, px, kq4);
          kp = fma(o1_5, q5, kp); kq5 = fma(o1_5, px, kq5);
          atomicAdd(K + (fP + 1) * N + fc, deg * kp); }
        { const double px = D[(fP + 2) * N + fd]; double kp = 0.0;
          kp = fma(o2_0, q0, kp); kq0 = fma(o2_0, px, kq0);
          kp = fma(o2_1, q1, kp); kq1 = fma(o2_1, px, kq1);
          kp = fma(o2_2, q2, kp); kq2 = fma(o2_2, px, kq2);
          kp = fma(o2_3, q3, kp); kq3 = fma(o2_3, px, kq3);
          kp = fma(o2_4, q4, kp); kq4 = fma(o2_4, px, kq4);
          kp = fma(o2_5, q5, kp); kq5 = fma(o2_5, px, kq5);
          atomicAdd(K + (fP + 2) * N + fc, deg * kp); }
        { const double px = D[(fP + 3) * N + fd]; double kp = 0.0;
          kp = fma(o3_0, q0, kp); kq0 = fma(o3_0, px, kq0);
          kp = fma(o3_1, q1, kp); kq1 = fma(o3_1, px, kq1);
          kp = fma(o3_2, q2, kp); kq2 = fma(o3_2, px, kq2);
          kp = fma(o3_3, q3, kp); kq3 = fma(o3_3, px, kq3);
          kp = fma(o3_4, q4, kp); kq4 = fma(o3_4, px, kq4);
          kp = fma(o3_5, q5, kp); kq5 = fma(o3_5, px, kq5);
          atomicAdd(K + (fP + 3) * N + fc, deg * kp); }
        { const double px = D[(fP + 4) * N + fd]; double kp = 0.0;
          kp = fma(o4_0, q0, kp); kq0 = fma(o4_0, px, kq0);
          kp = fma(o4_1, q1, kp); kq1 = fma(o4_1, px, kq1);
          kp = fma(o4_2, q2, kp); kq2 = fma(o4_2, px, kq2);
          kp = fma(o4_3, q3, kp); kq3 = fma(o4_3, px, kq3);
          kp = fma(o4_4, q4, kp); kq4 = fma(o4_4, px, kq4);
          kp = fma(o4_5, q5, kp); kq5 = fma(o4_5, px, kq5);
          atomicAdd(K + (fP + 4) * N + fc, deg * kp); }
        atomicAdd(K + (fQ + 0) * N + fc, deg * kq0);
        atomicAdd(K + (fQ + 1) * N + fc, deg * kq1);
        atomicAdd(K + (fQ + 2) * N + fc, deg * kq2);
        atomicAdd(K + (fQ + 3) * N + fc, deg * kq3);
        atomicAdd(K + (fQ + 4) * N + fc, deg * kq4);
        atomicAdd(K + (fQ + 5) * N + fc, deg * kq5);
      }
      {  // K[p][d], K[q][d] from D[.][c]
        const double q0 = D[(fQ + 0) * N + fc];
        double kq0 = 0.0;
        const double q1 = D[(fQ + 1) * N + fc];
        double kq1 = 0.0;
        const double q2 = D[(fQ + 2) * N + fc];
        double kq2 = 0.0;
        const double q3 = D[(fQ + 3) * N + fc];
        double kq3 = 0.0;
        const double q4 = D[(fQ + 4) * N + fc];
        double kq4 = 0.0;
        const double q5 = D[(fQ + 5) * N + fc];
        double kq5 = 0.0;
        { const double px = D[(fP + 0) * N + fc]; double kp = 0.0;
          kp = fma(o0_0, q0, kp); kq0 = fma(o0_0, px, kq0);
          kp = fma(o0_1, q1, kp); kq1 = fma(o0_1, px, kq1);
          kp = fma(o0_2, q2, kp); kq2 = fma(o0_2, px, kq2);
          kp = fma(o0_3, q3, kp); kq3 = fma(o0_3, px, kq3);
          kp = fma(o0_4, q4, kp); kq4 = fma(o0_4, px, kq4);
          kp = fma(o0_5, q5, kp); kq5 = fma(o0_5, px, kq5);
          atomicAdd(K + (fP + 0) * N + fd, deg * kp); }
        { const double px = D[(fP + 1) * N + fc]; double kp = 0.0;
          kp = fma(o1_0, q0, kp); kq0 = fma(o1_0, px, kq0);
          kp = fma(o1_1, q1, kp); kq1 = fma(o1_1, px, kq1);
          kp = fma(o1_2, q2, kp); kq2 = fma(o1_2, px, kq2);
          kp = fma(o1_3, q3, kp); kq3 = fma(o1_3, px, kq3);
          kp = fma(o1_4, q4, kp); kq4 = fma(o1_4, px, kq4);
          kp = fma(o1_5, q5, kp); kq5 = fma(o1_5, px, kq5);
          atomicAdd(K + (fP + 1) * N + fd, deg * kp); }
        { const double px = D[(fP + 2) * N + fc]; double kp = 0.0;
          kp = fma(o2_0, q0, kp); kq0 = fma(o2_0, px, kq0);
          kp = fma(o2_1, q1, kp); kq1 = fma(o2_1, px, kq1);
          kp = fma(o2_2, q2, kp); kq2 = fma(o2_2, px, kq2);
          kp = fma(o2_3, q3, kp); kq3 = fma(o2_3, px, kq3);
          kp = fma(o2_4, q4, kp); kq4 = fma(o2_4, px, kq4);
          kp = fma(o2_5, q5, kp); kq5 = fma(o2_5, px, kq5);
          atomicAdd(K + (fP + 2) * N + fd, deg * kp); }
        { const double px = D[(fP + 3) * N + fc]; double kp = 0.0;
          kp = fma(o3_0, q0, kp); kq0 = fma(o3_0, px, kq0);
          kp = fma(o3_1, q1, kp); kq1 = fma(o3_1, px, kq1);
          kp = fma(o3_2, q2, kp); kq2 = fma(o3_2, px, kq2);
          kp = fma(o3_3, q3, kp); kq3 = fma(o3_3, px, kq3);
          kp = fma(o3_4, q4, kp); kq4 = fma(o3_4, px, kq4);
          kp = fma(o3_5, q5, kp); kq5 = fma(o3_5, px, kq5);
          atomicAdd(K + (fP + 3) * N + fd, deg * kp); }
        { const double px = D[(fP + 4) * N + fc]; double kp = 0.0;
          kp = fma(o4_0, q0, kp); kq0 = fma(o4_0, px, kq0);
          kp = fma(o4_1, q1, kp); kq1 = fma(o4_1, px, kq1);
          kp = fma(o4_2, q2, kp); kq2 = fma(o4_2, px, kq2);
          kp = fma(o4_3, q3, kp); kq3 = fma(o4_3, px, kq3);
          kp = fma(o4_4, q4, kp); kq4 = fma(o4_4, px, kq4);
          kp = fma(o4_5, q5, kp); kq5 = fma(o4_5, px, kq5);
          atomicAdd(K + (fP + 4) * N + fd, deg * kp); }
        atomicAdd(K + (fQ + 0) * N + fd, deg * kq0);
        atomicAdd(K + (fQ + 1) * N + fd, deg * kq1);
        atomicAdd(K + (fQ + 2) * N + fd, deg * kq2);
        atomicAdd(K + (fQ + 3) * N + fd, deg * kq3);
        atomicAdd(K + (fQ + 4) * N + fd, deg * kq4);
        atomicAdd(K + (fQ + 5) * N + fd, deg * kq5);
      }
    }
    nfl += 2ull * 30 * (2 + 4 * (a.b.uhf ? 2 : 1));
  }
  {  // J[p][q]: every lane shares the bra pair
    const double w = ok ? s2 * __ldg(PT + fc * N + fd) : 0.0;
    { double v[32] = {w * o0_0, w * o0_1, w * o0_2, w * o0_3, w * o0_4, w * o0_5, w * o1_0, w * o1_1, w * o1_2, w * o1_3, w * o1_4, w * o1_5, w * o2_0, w * o2_1, w * o2_2, w * o2_3, w * o2_4, w * o2_5, w * o3_0, w * o3_1, w * o3_2, w * o3_3, w * o3_4, w * o3_5, w * o4_0, w * o4_1, w * o4_2, w * o4_3, w * o4_4, w * o4_5, 0.0, 0.0};
      const double z = sqb::warp_sum_scatter<32>(v); const int x = lane + 0;
      if (lane < 30 && z != 0.0) atomicAdd(a.b.J + (fP + 0 + x / 6) * N + fQ + x % 6, z); }
  }
  sqb::count_add(a.counters + 0, ok && cd == 0 && gi == 0 && gj == 0 ? 1ull : 0ull);
  sqb::count_add(a.counters + 1, npq);
  sqb::count_add(a.counters + 2, nfl);
}
