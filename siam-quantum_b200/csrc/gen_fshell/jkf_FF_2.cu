// generated by gen_fshell_kernels.py -- do not edit
#include "../jk_generic_dev.cuh"

extern "C" __global__ void __launch_bounds__(128)
jkf_FF_2(const sqb::FArgs a, const sqb::FRun* __restrict__ runs, const long long* __restrict__ first, int nruns,
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
  const int L = 6 + B.lP + B.lQ, S1 = L + 1, S2 = S1 * S1;   // uniform over the warp
  double* __restrict__ box = fsm + wp * sqb::kFWarpDoubles + min(s, it.cnt - 1) * sqb::f_slot(L);   // [t][u][v], then the seeds
  double* __restrict__ base = box + S1 * S2;
  const bool mine = s < it.cnt;
  const unsigned d = __ldg(a.desc + B.doff + cd);
  const int cx = sqb::dsc(d, 0), dx = sqb::dsc(d, 1), cy = sqb::dsc(d, 2), dy = sqb::dsc(d, 3), cz = sqb::dsc(d, 4), dz = sqb::dsc(d, 5);
  const int n1 = cy + dy + 1, n2 = cz + dz + 1, nk = (cx + dx + 1) * n1 * n2;
  unsigned long long npq = 0, nfl = 0;
  double o4_0 = 0.0;
  double o4_1 = 0.0;
  double o4_2 = 0.0;
  double o4_3 = 0.0;
  double o4_4 = 0.0;
  double o4_5 = 0.0;
  double o4_6 = 0.0;
  double o4_7 = 0.0;
  double o4_8 = 0.0;
  double o4_9 = 0.0;
  double o5_0 = 0.0;
  double o5_1 = 0.0;
  double o5_2 = 0.0;
  double o5_3 = 0.0;
  double o5_4 = 0.0;
  double o5_5 = 0.0;
  double o5_6 = 0.0;
  double o5_7 = 0.0;
  double o5_8 = 0.0;
  double o5_9 = 0.0;
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
    double g600 = 0.0;
    double g510 = 0.0;
    double g501 = 0.0;
    double g420 = 0.0;
    double g411 = 0.0;
    double g402 = 0.0;
    double g330 = 0.0;
    double g321 = 0.0;
    double g312 = 0.0;
    double g303 = 0.0;
    double g240 = 0.0;
    double g231 = 0.0;
    double g222 = 0.0;
    double g213 = 0.0;
    double g204 = 0.0;
    double g150 = 0.0;
    double g141 = 0.0;
    double g132 = 0.0;
    double g123 = 0.0;
    double g114 = 0.0;
    double g105 = 0.0;
    double g060 = 0.0;
    double g051 = 0.0;
    double g042 = 0.0;
    double g033 = 0.0;
    double g024 = 0.0;
    double g015 = 0.0;
    double g006 = 0.0;
    bool any = false;
    for (int j = gj; j < B.nprim; j += sj) {     // one contraction length per warp
      const double* pb = a.prims + (size_t)(B.poff + j) * sqb::kGenPrimStride;
      const double q = pb[0], pq = p + q, rs = rsqrt(pq);
      const bool live = ok && !(TWO_PI_2_5 * kpa * pb[4] * rs < PRIM_CUTOFF);
      if (!__any_sync(0xffffffffu, live)) continue;
      any = true;
      if (live && cd == 0 && false) ++npq;
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
            g006 = fma(e, x[6], g006);
          }
          { const double* __restrict__ x = R + 0 * S2 + 1 * S1;
            g010 = fma(e, x[0], g010);
            g011 = fma(e, x[1], g011);
            g012 = fma(e, x[2], g012);
            g013 = fma(e, x[3], g013);
            g014 = fma(e, x[4], g014);
            g015 = fma(e, x[5], g015);
          }
          { const double* __restrict__ x = R + 0 * S2 + 2 * S1;
            g020 = fma(e, x[0], g020);
            g021 = fma(e, x[1], g021);
            g022 = fma(e, x[2], g022);
            g023 = fma(e, x[3], g023);
            g024 = fma(e, x[4], g024);
          }
          { const double* __restrict__ x = R + 0 * S2 + 3 * S1;
            g030 = fma(e, x[0], g030);
            g031 = fma(e, x[1], g031);
            g032 = fma(e, x[2], g032);
            g033 = fma(e, x[3], g033);
          }
          { const double* __restrict__ x = R + 0 * S2 + 4 * S1;
            g040 = fma(e, x[0], g040);
            g041 = fma(e, x[1], g041);
            g042 = fma(e, x[2], g042);
          }
          { const double* __restrict__ x = R + 0 * S2 + 5 * S1;
            g050 = fma(e, x[0], g050);
            g051 = fma(e, x[1], g051);
          }
          { const double* __restrict__ x = R + 0 * S2 + 6 * S1;
            g060 = fma(e, x[0], g060);
          }
          { const double* __restrict__ x = R + 1 * S2 + 0 * S1;
            g100 = fma(e, x[0], g100);
            g101 = fma(e, x[1], g101);
            g102 = fma(e, x[2], g102);
            g103 = fma(e, x[3], g103);
            g104 = fma(e, x[4], g104);
            g105 = fma(e, x[5], g105);
          }
          { const double* __restrict__ x = R + 1 * S2 + 1 * S1;
            g110 = fma(e, x[0], g110);
            g111 = fma(e, x[1], g111);
            g112 = fma(e, x[2], g112);
            g113 = fma(e, x[3], g113);
            g114 = fma(e, x[4], g114);
          }
          { const double* __restrict__ x = R + 1 * S2 + 2 * S1;
            g120 = fma(e, x[0], g120);
            g121 = fma(e, x[1], g121);
            g122 = fma(e, x[2], g122);
            g123 = fma(e, x[3], g123);
          }
          { const double* __restrict__ x = R + 1 * S2 + 3 * S1;
            g130 = fma(e, x[0], g130);
            g131 = fma(e, x[1], g131);
            g132 = fma(e, x[2], g132);
          }
          { const double* __restrict__ x = R + 1 * S2 + 4 * S1;
            g140 = fma(e, x[0], g140);
            g141 = fma(e, x[1], g141);
          }
          { const double* __restrict__ x = R + 1 * S2 + 5 * S1;
            g150 = fma(e, x[0], g150);
          }
          { const double* __restrict__ x = R + 2 * S2 + 0 * S1;
            g200 = fma(e, x[0], g200);
            g201 = fma(e, x[1], g201);
            g202 = fma(e, x[2], g202);
            g203 = fma(e, x[3], g203);
            g204 = fma(e, x[4], g204);
          }
          { const double* __restrict__ x = R + 2 * S2 + 1 * S1;
            g210 = fma(e, x[0], g210);
            g211 = fma(e, x[1], g211);
            g212 = fma(e, x[2], g212);
            g213 = fma(e, x[3], g213);
          }
          { const double* __restrict__ x = R + 2 * S2 + 2 * S1;
            g220 = fma(e, x[0], g220);
            g221 = fma(e, x[1], g221);
            g222 = fma(e, x[2], g222);
          }
          { const double* __restrict__ x = R + 2 * S2 + 3 * S1;
            g230 = fma(e, x[0], g230);
            g231 = fma(e, x[1], g231);
          }
          { const double* __restrict__ x = R + 2 * S2 + 4 * S1;
            g240 = fma(e, x[0], g240);
          }
          { const double* __restrict__ x = R + 3 * S2 + 0 * S1;
            g300 = fma(e, x[0], g300);
            g301 = fma(e, x[1], g301);
            g302 = fma(e, x[2], g302);
            g303 = fma(e, x[3], g303);
          }
          { const double* __restrict__ x = R + 3 * S2 + 1 * S1;
            g310 = fma(e, x[0], g310);
            g311 = fma(e, x[1], g311);
            g312 = fma(e, x[2], g312);
          }
          { const double* __restrict__ x = R + 3 * S2 + 2 * S1;
            g320 = fma(e, x[0], g320);
            g321 = fma(e, x[1], g321);
          }
          { const double* __restrict__ x = R + 3 * S2 + 3 * S1;
            g330 = fma(e, x[0], g330);
          }
          { const double* __restrict__ x = R + 4 * S2 + 0 * S1;
            g400 = fma(e, x[0], g400);
            g401 = fma(e, x[1], g401);
            g402 = fma(e, x[2], g402);
          }
          { const double* __restrict__ x = R + 4 * S2 + 1 * S1;
            g410 = fma(e, x[0], g410);
            g411 = fma(e, x[1], g411);
          }
          { const double* __restrict__ x = R + 4 * S2 + 2 * S1;
            g420 = fma(e, x[0], g420);
          }
          { const double* __restrict__ x = R + 5 * S2 + 0 * S1;
            g500 = fma(e, x[0], g500);
            g501 = fma(e, x[1], g501);
          }
          { const double* __restrict__ x = R + 5 * S2 + 1 * S1;
            g510 = fma(e, x[0], g510);
          }
          { const double* __restrict__ x = R + 6 * S2 + 0 * S1;
            g600 = fma(e, x[0], g600);
          }
          if (++ph == n2) { ph = 0; if (++nu == n1) { nu = 0; ++tau; } }
        }
        nfl += 2ull * 84 * nk;
      }
    }
    if (!any) continue;
    const sqb::EView Ei(a.coef, pa, A);
    const double* __restrict__ E = Ei.e;
    { double z = 0.0;
      z = fma(__ldg(E + 49) * __ldg(E + 168), g000, z);
      z = fma(__ldg(E + 49) * __ldg(E + 169), g010, z);
      z = fma(__ldg(E + 49) * __ldg(E + 170), g020, z);
      z = fma(__ldg(E + 50) * __ldg(E + 168), g100, z);
      z = fma(__ldg(E + 50) * __ldg(E + 169), g110, z);
      z = fma(__ldg(E + 50) * __ldg(E + 170), g120, z);
      z = fma(__ldg(E + 51) * __ldg(E + 168), g200, z);
      z = fma(__ldg(E + 51) * __ldg(E + 169), g210, z);
      z = fma(__ldg(E + 51) * __ldg(E + 170), g220, z);
      z = fma(__ldg(E + 52) * __ldg(E + 168), g300, z);
      z = fma(__ldg(E + 52) * __ldg(E + 169), g310, z);
      z = fma(__ldg(E + 52) * __ldg(E + 170), g320, z);
      z = fma(__ldg(E + 53) * __ldg(E + 168), g400, z);
      z = fma(__ldg(E + 53) * __ldg(E + 169), g410, z);
      z = fma(__ldg(E + 53) * __ldg(E + 170), g420, z);
      o4_0 = fma(Ei.w(40), z, o4_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 28) * __ldg(E + 189), g000, z);
      z = fma(__ldg(E + 28) * __ldg(E + 190), g010, z);
      z = fma(__ldg(E + 28) * __ldg(E + 191), g020, z);
      z = fma(__ldg(E + 28) * __ldg(E + 192), g030, z);
      z = fma(__ldg(E + 28) * __ldg(E + 193), g040, z);
      z = fma(__ldg(E + 28) * __ldg(E + 194), g050, z);
      z = fma(__ldg(E + 29) * __ldg(E + 189), g100, z);
      z = fma(__ldg(E + 29) * __ldg(E + 190), g110, z);
      z = fma(__ldg(E + 29) * __ldg(E + 191), g120, z);
      z = fma(__ldg(E + 29) * __ldg(E + 192), g130, z);
      z = fma(__ldg(E + 29) * __ldg(E + 193), g140, z);
      z = fma(__ldg(E + 29) * __ldg(E + 194), g150, z);
      o4_1 = fma(Ei.w(41), z, o4_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 28) * __ldg(E + 168), fma(__ldg(E + 248), g003, fma(__ldg(E + 247), g002, fma(__ldg(E + 246), g001, __ldg(E + 245) * g000))), z);
      z = fma(__ldg(E + 28) * __ldg(E + 169), fma(__ldg(E + 248), g013, fma(__ldg(E + 247), g012, fma(__ldg(E + 246), g011, __ldg(E + 245) * g010))), z);
      z = fma(__ldg(E + 28) * __ldg(E + 170), fma(__ldg(E + 248), g023, fma(__ldg(E + 247), g022, fma(__ldg(E + 246), g021, __ldg(E + 245) * g020))), z);
      z = fma(__ldg(E + 29) * __ldg(E + 168), fma(__ldg(E + 248), g103, fma(__ldg(E + 247), g102, fma(__ldg(E + 246), g101, __ldg(E + 245) * g100))), z);
      z = fma(__ldg(E + 29) * __ldg(E + 169), fma(__ldg(E + 248), g113, fma(__ldg(E + 247), g112, fma(__ldg(E + 246), g111, __ldg(E + 245) * g110))), z);
      z = fma(__ldg(E + 29) * __ldg(E + 170), fma(__ldg(E + 248), g123, fma(__ldg(E + 247), g122, fma(__ldg(E + 246), g121, __ldg(E + 245) * g120))), z);
      o4_2 = fma(Ei.w(42), z, o4_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 42) * __ldg(E + 175), g000, z);
      z = fma(__ldg(E + 42) * __ldg(E + 176), g010, z);
      z = fma(__ldg(E + 42) * __ldg(E + 177), g020, z);
      z = fma(__ldg(E + 42) * __ldg(E + 178), g030, z);
      z = fma(__ldg(E + 43) * __ldg(E + 175), g100, z);
      z = fma(__ldg(E + 43) * __ldg(E + 176), g110, z);
      z = fma(__ldg(E + 43) * __ldg(E + 177), g120, z);
      z = fma(__ldg(E + 43) * __ldg(E + 178), g130, z);
      z = fma(__ldg(E + 44) * __ldg(E + 175), g200, z);
      z = fma(__ldg(E + 44) * __ldg(E + 176), g210, z);
      z = fma(__ldg(E + 44) * __ldg(E + 177), g220, z);
      z = fma(__ldg(E + 44) * __ldg(E + 178), g230, z);
      z = fma(__ldg(E + 45) * __ldg(E + 175), g300, z);
      z = fma(__ldg(E + 45) * __ldg(E + 176), g310, z);
      z = fma(__ldg(E + 45) * __ldg(E + 177), g320, z);
      z = fma(__ldg(E + 45) * __ldg(E + 178), g330, z);
      o4_3 = fma(Ei.w(43), z, o4_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 35) * __ldg(E + 182), g000, z);
      z = fma(__ldg(E + 35) * __ldg(E + 183), g010, z);
      z = fma(__ldg(E + 35) * __ldg(E + 184), g020, z);
      z = fma(__ldg(E + 35) * __ldg(E + 185), g030, z);
      z = fma(__ldg(E + 35) * __ldg(E + 186), g040, z);
      z = fma(__ldg(E + 36) * __ldg(E + 182), g100, z);
      z = fma(__ldg(E + 36) * __ldg(E + 183), g110, z);
      z = fma(__ldg(E + 36) * __ldg(E + 184), g120, z);
      z = fma(__ldg(E + 36) * __ldg(E + 185), g130, z);
      z = fma(__ldg(E + 36) * __ldg(E + 186), g140, z);
      z = fma(__ldg(E + 37) * __ldg(E + 182), g200, z);
      z = fma(__ldg(E + 37) * __ldg(E + 183), g210, z);
      z = fma(__ldg(E + 37) * __ldg(E + 184), g220, z);
      z = fma(__ldg(E + 37) * __ldg(E + 185), g230, z);
      z = fma(__ldg(E + 37) * __ldg(E + 186), g240, z);
      o4_4 = fma(Ei.w(44), z, o4_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 42) * __ldg(E + 168), fma(__ldg(E + 232), g001, __ldg(E + 231) * g000), z);
      z = fma(__ldg(E + 42) * __ldg(E + 169), fma(__ldg(E + 232), g011, __ldg(E + 231) * g010), z);
      z = fma(__ldg(E + 42) * __ldg(E + 170), fma(__ldg(E + 232), g021, __ldg(E + 231) * g020), z);
      z = fma(__ldg(E + 43) * __ldg(E + 168), fma(__ldg(E + 232), g101, __ldg(E + 231) * g100), z);
      z = fma(__ldg(E + 43) * __ldg(E + 169), fma(__ldg(E + 232), g111, __ldg(E + 231) * g110), z);
      z = fma(__ldg(E + 43) * __ldg(E + 170), fma(__ldg(E + 232), g121, __ldg(E + 231) * g120), z);
      z = fma(__ldg(E + 44) * __ldg(E + 168), fma(__ldg(E + 232), g201, __ldg(E + 231) * g200), z);
      z = fma(__ldg(E + 44) * __ldg(E + 169), fma(__ldg(E + 232), g211, __ldg(E + 231) * g210), z);
      z = fma(__ldg(E + 44) * __ldg(E + 170), fma(__ldg(E + 232), g221, __ldg(E + 231) * g220), z);
      z = fma(__ldg(E + 45) * __ldg(E + 168), fma(__ldg(E + 232), g301, __ldg(E + 231) * g300), z);
      z = fma(__ldg(E + 45) * __ldg(E + 169), fma(__ldg(E + 232), g311, __ldg(E + 231) * g310), z);
      z = fma(__ldg(E + 45) * __ldg(E + 170), fma(__ldg(E + 232), g321, __ldg(E + 231) * g320), z);
      o4_5 = fma(Ei.w(45), z, o4_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 35) * __ldg(E + 168), fma(__ldg(E + 240), g002, fma(__ldg(E + 239), g001, __ldg(E + 238) * g000)), z);
      z = fma(__ldg(E + 35) * __ldg(E + 169), fma(__ldg(E + 240), g012, fma(__ldg(E + 239), g011, __ldg(E + 238) * g010)), z);
      z = fma(__ldg(E + 35) * __ldg(E + 170), fma(__ldg(E + 240), g022, fma(__ldg(E + 239), g021, __ldg(E + 238) * g020)), z);
      z = fma(__ldg(E + 36) * __ldg(E + 168), fma(__ldg(E + 240), g102, fma(__ldg(E + 239), g101, __ldg(E + 238) * g100)), z);
      z = fma(__ldg(E + 36) * __ldg(E + 169), fma(__ldg(E + 240), g112, fma(__ldg(E + 239), g111, __ldg(E + 238) * g110)), z);
      z = fma(__ldg(E + 36) * __ldg(E + 170), fma(__ldg(E + 240), g122, fma(__ldg(E + 239), g121, __ldg(E + 238) * g120)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 168), fma(__ldg(E + 240), g202, fma(__ldg(E + 239), g201, __ldg(E + 238) * g200)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 169), fma(__ldg(E + 240), g212, fma(__ldg(E + 239), g211, __ldg(E + 238) * g210)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 170), fma(__ldg(E + 240), g222, fma(__ldg(E + 239), g221, __ldg(E + 238) * g220)), z);
      o4_6 = fma(Ei.w(46), z, o4_6); }
    { double z = 0.0;
      z = fma(__ldg(E + 28) * __ldg(E + 182), fma(__ldg(E + 232), g001, __ldg(E + 231) * g000), z);
      z = fma(__ldg(E + 28) * __ldg(E + 183), fma(__ldg(E + 232), g011, __ldg(E + 231) * g010), z);
      z = fma(__ldg(E + 28) * __ldg(E + 184), fma(__ldg(E + 232), g021, __ldg(E + 231) * g020), z);
      z = fma(__ldg(E + 28) * __ldg(E + 185), fma(__ldg(E + 232), g031, __ldg(E + 231) * g030), z);
      z = fma(__ldg(E + 28) * __ldg(E + 186), fma(__ldg(E + 232), g041, __ldg(E + 231) * g040), z);
      z = fma(__ldg(E + 29) * __ldg(E + 182), fma(__ldg(E + 232), g101, __ldg(E + 231) * g100), z);
      z = fma(__ldg(E + 29) * __ldg(E + 183), fma(__ldg(E + 232), g111, __ldg(E + 231) * g110), z);
      z = fma(__ldg(E + 29) * __ldg(E + 184), fma(__ldg(E + 232), g121, __ldg(E + 231) * g120), z);
      z = fma(__ldg(E + 29) * __ldg(E + 185), fma(__ldg(E + 232), g131, __ldg(E + 231) * g130), z);
      z = fma(__ldg(E + 29) * __ldg(E + 186), fma(__ldg(E + 232), g141, __ldg(E + 231) * g140), z);
      o4_7 = fma(Ei.w(47), z, o4_7); }
    { double z = 0.0;
      z = fma(__ldg(E + 28) * __ldg(E + 175), fma(__ldg(E + 240), g002, fma(__ldg(E + 239), g001, __ldg(E + 238) * g000)), z);
      z = fma(__ldg(E + 28) * __ldg(E + 176), fma(__ldg(E + 240), g012, fma(__ldg(E + 239), g011, __ldg(E + 238) * g010)), z);
      z = fma(__ldg(E + 28) * __ldg(E + 177), fma(__ldg(E + 240), g022, fma(__ldg(E + 239), g021, __ldg(E + 238) * g020)), z);
      z = fma(__ldg(E + 28) * __ldg(E + 178), fma(__ldg(E + 240), g032, fma(__ldg(E + 239), g031, __ldg(E + 238) * g030)), z);
      z = fma(__ldg(E + 29) * __ldg(E + 175), fma(__ldg(E + 240), g102, fma(__ldg(E + 239), g101, __ldg(E + 238) * g100)), z);
      z = fma(__ldg(E + 29) * __ldg(E + 176), fma(__ldg(E + 240), g112, fma(__ldg(E + 239), g111, __ldg(E + 238) * g110)), z);
      z = fma(__ldg(E + 29) * __ldg(E + 177), fma(__ldg(E + 240), g122, fma(__ldg(E + 239), g121, __ldg(E + 238) * g120)), z);
      z = fma(__ldg(E + 29) * __ldg(E + 178), fma(__ldg(E + 240), g132, fma(__ldg(E + 239), g131, __ldg(E + 238) * g130)), z);
      o4_8 = fma(Ei.w(48), z, o4_8); }
    { double z = 0.0;
      z = fma(__ldg(E + 35) * __ldg(E + 175), fma(__ldg(E + 232), g001, __ldg(E + 231) * g000), z);
      z = fma(__ldg(E + 35) * __ldg(E + 176), fma(__ldg(E + 232), g011, __ldg(E + 231) * g010), z);
      z = fma(__ldg(E + 35) * __ldg(E + 177), fma(__ldg(E + 232), g021, __ldg(E + 231) * g020), z);
      z = fma(__ldg(E + 35) * __ldg(E + 178), fma(__ldg(E + 232), g031, __ldg(E + 231) * g030), z);
      z = fma(__ldg(E + 36) * __ldg(E + 175), fma(__ldg(E + 232), g101, __ldg(E + 231) * g100), z);
      z = fma(__ldg(E + 36) * __ldg(E + 176), fma(__ldg(E + 232), g111, __ldg(E + 231) * g110), z);
      z = fma(__ldg(E + 36) * __ldg(E + 177), fma(__ldg(E + 232), g121, __ldg(E + 231) * g120), z);
      z = fma(__ldg(E + 36) * __ldg(E + 178), fma(__ldg(E + 232), g131, __ldg(E + 231) * g130), z);
      z = fma(__ldg(E + 37) * __ldg(E + 175), fma(__ldg(E + 232), g201, __ldg(E + 231) * g200), z);
      z = fma(__ldg(E + 37) * __ldg(E + 176), fma(__ldg(E + 232), g211, __ldg(E + 231) * g210), z);
      z = fma(__ldg(E + 37) * __ldg(E + 177), fma(__ldg(E + 232), g221, __ldg(E + 231) * g220), z);
      z = fma(__ldg(E + 37) * __ldg(E + 178), fma(__ldg(E + 232), g231, __ldg(E + 231) * g230), z);
      o4_9 = fma(Ei.w(49), z, o4_9); }
    { double z = 0.0;
      z = fma(__ldg(E + 77), fma(__ldg(E + 253), g001, __ldg(E + 252) * g000), z);
      z = fma(__ldg(E + 78), fma(__ldg(E + 253), g101, __ldg(E + 252) * g100), z);
      z = fma(__ldg(E + 79), fma(__ldg(E + 253), g201, __ldg(E + 252) * g200), z);
      z = fma(__ldg(E + 80), fma(__ldg(E + 253), g301, __ldg(E + 252) * g300), z);
      z = fma(__ldg(E + 81), fma(__ldg(E + 253), g401, __ldg(E + 252) * g400), z);
      z = fma(__ldg(E + 82), fma(__ldg(E + 253), g501, __ldg(E + 252) * g500), z);
      o5_0 = fma(Ei.w(50), z, o5_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 56) * __ldg(E + 133), fma(__ldg(E + 253), g001, __ldg(E + 252) * g000), z);
      z = fma(__ldg(E + 56) * __ldg(E + 134), fma(__ldg(E + 253), g011, __ldg(E + 252) * g010), z);
      z = fma(__ldg(E + 56) * __ldg(E + 135), fma(__ldg(E + 253), g021, __ldg(E + 252) * g020), z);
      z = fma(__ldg(E + 56) * __ldg(E + 136), fma(__ldg(E + 253), g031, __ldg(E + 252) * g030), z);
      z = fma(__ldg(E + 57) * __ldg(E + 133), fma(__ldg(E + 253), g101, __ldg(E + 252) * g100), z);
      z = fma(__ldg(E + 57) * __ldg(E + 134), fma(__ldg(E + 253), g111, __ldg(E + 252) * g110), z);
      z = fma(__ldg(E + 57) * __ldg(E + 135), fma(__ldg(E + 253), g121, __ldg(E + 252) * g120), z);
      z = fma(__ldg(E + 57) * __ldg(E + 136), fma(__ldg(E + 253), g131, __ldg(E + 252) * g130), z);
      z = fma(__ldg(E + 58) * __ldg(E + 133), fma(__ldg(E + 253), g201, __ldg(E + 252) * g200), z);
      z = fma(__ldg(E + 58) * __ldg(E + 134), fma(__ldg(E + 253), g211, __ldg(E + 252) * g210), z);
      z = fma(__ldg(E + 58) * __ldg(E + 135), fma(__ldg(E + 253), g221, __ldg(E + 252) * g220), z);
      z = fma(__ldg(E + 58) * __ldg(E + 136), fma(__ldg(E + 253), g231, __ldg(E + 252) * g230), z);
      o5_1 = fma(Ei.w(51), z, o5_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 56), fma(__ldg(E + 277), g004, fma(__ldg(E + 276), g003, fma(__ldg(E + 275), g002, fma(__ldg(E + 274), g001, __ldg(E + 273) * g000)))), z);
      z = fma(__ldg(E + 57), fma(__ldg(E + 277), g104, fma(__ldg(E + 276), g103, fma(__ldg(E + 275), g102, fma(__ldg(E + 274), g101, __ldg(E + 273) * g100)))), z);
      z = fma(__ldg(E + 58), fma(__ldg(E + 277), g204, fma(__ldg(E + 276), g203, fma(__ldg(E + 275), g202, fma(__ldg(E + 274), g201, __ldg(E + 273) * g200)))), z);
      o5_2 = fma(Ei.w(52), z, o5_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 70) * __ldg(E + 119), fma(__ldg(E + 253), g001, __ldg(E + 252) * g000), z);
      z = fma(__ldg(E + 70) * __ldg(E + 120), fma(__ldg(E + 253), g011, __ldg(E + 252) * g010), z);
      z = fma(__ldg(E + 71) * __ldg(E + 119), fma(__ldg(E + 253), g101, __ldg(E + 252) * g100), z);
      z = fma(__ldg(E + 71) * __ldg(E + 120), fma(__ldg(E + 253), g111, __ldg(E + 252) * g110), z);
      z = fma(__ldg(E + 72) * __ldg(E + 119), fma(__ldg(E + 253), g201, __ldg(E + 252) * g200), z);
      z = fma(__ldg(E + 72) * __ldg(E + 120), fma(__ldg(E + 253), g211, __ldg(E + 252) * g210), z);
      z = fma(__ldg(E + 73) * __ldg(E + 119), fma(__ldg(E + 253), g301, __ldg(E + 252) * g300), z);
      z = fma(__ldg(E + 73) * __ldg(E + 120), fma(__ldg(E + 253), g311, __ldg(E + 252) * g310), z);
      z = fma(__ldg(E + 74) * __ldg(E + 119), fma(__ldg(E + 253), g401, __ldg(E + 252) * g400), z);
      z = fma(__ldg(E + 74) * __ldg(E + 120), fma(__ldg(E + 253), g411, __ldg(E + 252) * g410), z);
      o5_3 = fma(Ei.w(53), z, o5_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 63) * __ldg(E + 126), fma(__ldg(E + 253), g001, __ldg(E + 252) * g000), z);
      z = fma(__ldg(E + 63) * __ldg(E + 127), fma(__ldg(E + 253), g011, __ldg(E + 252) * g010), z);
      z = fma(__ldg(E + 63) * __ldg(E + 128), fma(__ldg(E + 253), g021, __ldg(E + 252) * g020), z);
      z = fma(__ldg(E + 64) * __ldg(E + 126), fma(__ldg(E + 253), g101, __ldg(E + 252) * g100), z);
      z = fma(__ldg(E + 64) * __ldg(E + 127), fma(__ldg(E + 253), g111, __ldg(E + 252) * g110), z);
      z = fma(__ldg(E + 64) * __ldg(E + 128), fma(__ldg(E + 253), g121, __ldg(E + 252) * g120), z);
      z = fma(__ldg(E + 65) * __ldg(E + 126), fma(__ldg(E + 253), g201, __ldg(E + 252) * g200), z);
      z = fma(__ldg(E + 65) * __ldg(E + 127), fma(__ldg(E + 253), g211, __ldg(E + 252) * g210), z);
      z = fma(__ldg(E + 65) * __ldg(E + 128), fma(__ldg(E + 253), g221, __ldg(E + 252) * g220), z);
      z = fma(__ldg(E + 66) * __ldg(E + 126), fma(__ldg(E + 253), g301, __ldg(E + 252) * g300), z);
      z = fma(__ldg(E + 66) * __ldg(E + 127), fma(__ldg(E + 253), g311, __ldg(E + 252) * g310), z);
      z = fma(__ldg(E + 66) * __ldg(E + 128), fma(__ldg(E + 253), g321, __ldg(E + 252) * g320), z);
      o5_4 = fma(Ei.w(54), z, o5_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 70), fma(__ldg(E + 261), g002, fma(__ldg(E + 260), g001, __ldg(E + 259) * g000)), z);
      z = fma(__ldg(E + 71), fma(__ldg(E + 261), g102, fma(__ldg(E + 260), g101, __ldg(E + 259) * g100)), z);
      z = fma(__ldg(E + 72), fma(__ldg(E + 261), g202, fma(__ldg(E + 260), g201, __ldg(E + 259) * g200)), z);
      z = fma(__ldg(E + 73), fma(__ldg(E + 261), g302, fma(__ldg(E + 260), g301, __ldg(E + 259) * g300)), z);
      z = fma(__ldg(E + 74), fma(__ldg(E + 261), g402, fma(__ldg(E + 260), g401, __ldg(E + 259) * g400)), z);
      o5_5 = fma(Ei.w(55), z, o5_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 63), fma(__ldg(E + 269), g003, fma(__ldg(E + 268), g002, fma(__ldg(E + 267), g001, __ldg(E + 266) * g000))), z);
      z = fma(__ldg(E + 64), fma(__ldg(E + 269), g103, fma(__ldg(E + 268), g102, fma(__ldg(E + 267), g101, __ldg(E + 266) * g100))), z);
      z = fma(__ldg(E + 65), fma(__ldg(E + 269), g203, fma(__ldg(E + 268), g202, fma(__ldg(E + 267), g201, __ldg(E + 266) * g200))), z);
      z = fma(__ldg(E + 66), fma(__ldg(E + 269), g303, fma(__ldg(E + 268), g302, fma(__ldg(E + 267), g301, __ldg(E + 266) * g300))), z);
      o5_6 = fma(Ei.w(56), z, o5_6); }
    { double z = 0.0;
      z = fma(__ldg(E + 56) * __ldg(E + 126), fma(__ldg(E + 261), g002, fma(__ldg(E + 260), g001, __ldg(E + 259) * g000)), z);
      z = fma(__ldg(E + 56) * __ldg(E + 127), fma(__ldg(E + 261), g012, fma(__ldg(E + 260), g011, __ldg(E + 259) * g010)), z);
      z = fma(__ldg(E + 56) * __ldg(E + 128), fma(__ldg(E + 261), g022, fma(__ldg(E + 260), g021, __ldg(E + 259) * g020)), z);
      z = fma(__ldg(E + 57) * __ldg(E + 126), fma(__ldg(E + 261), g102, fma(__ldg(E + 260), g101, __ldg(E + 259) * g100)), z);
      z = fma(__ldg(E + 57) * __ldg(E + 127), fma(__ldg(E + 261), g112, fma(__ldg(E + 260), g111, __ldg(E + 259) * g110)), z);
      z = fma(__ldg(E + 57) * __ldg(E + 128), fma(__ldg(E + 261), g122, fma(__ldg(E + 260), g121, __ldg(E + 259) * g120)), z);
      z = fma(__ldg(E + 58) * __ldg(E + 126), fma(__ldg(E + 261), g202, fma(__ldg(E + 260), g201, __ldg(E + 259) * g200)), z);
      z = fma(__ldg(E + 58) * __ldg(E + 127), fma(__ldg(E + 261), g212, fma(__ldg(E + 260), g211, __ldg(E + 259) * g210)), z);
      z = fma(__ldg(E + 58) * __ldg(E + 128), fma(__ldg(E + 261), g222, fma(__ldg(E + 260), g221, __ldg(E + 259) * g220)), z);
      o5_7 = fma(Ei.w(57), z, o5_7); }
    { double z = 0.0;
      z = fma(__ldg(E + 56) * __ldg(E + 119), fma(__ldg(E + 269), g003, fma(__ldg(E + 268), g002, fma(__ldg(E + 267), g001, __ldg(E + 266) * g000))), z);
      z = fma(__ldg(E + 56) * __ldg(E + 120), fma(__ldg(E + 269), g013, fma(__ldg(E + 268), g012, fma(__ldg(E + 267), g011, __ldg(E + 266) * g010))), z);
      z = fma(__ldg(E + 57) * __ldg(E + 119), fma(__ldg(E + 269), g103, fma(__ldg(E + 268), g102, fma(__ldg(E + 267), g101, __ldg(E + 266) * g100))), z);
      z = fma(__ldg(E + 57) * __ldg(E + 120), fma(__ldg(E + 269), g113, fma(__ldg(E + 268), g112, fma(__ldg(E + 267), g111, __ldg(E + 266) * g110))), z);
      z = fma(__ldg(E + 58) * __ldg(E + 119), fma(__ldg(E + 269), g203, fma(__ldg(E + 268), g202, fma(__ldg(E + 267), g201, __ldg(E + 266) * g200))), z);
      z = fma(__ldg(E + 58) * __ldg(E + 120), fma(__ldg(E + 269), g213, fma(__ldg(E + 268), g212, fma(__ldg(E + 267), g211, __ldg(E + 266) * g210))), z);
      o5_8 = fma(Ei.w(58), z, o5_8); }
    { double z = 0.0;
      z = fma(__ldg(E + 63) * __ldg(E + 119), fma(__ldg(E + 261), g002, fma(__ldg(E + 260), g001, __ldg(E + 259) * g000)), z);
      z = fma(__ldg(E + 63) * __ldg(E + 120), fma(__ldg(E + 261), g012, fma(__ldg(E + 260), g011, __ldg(E + 259) * g010)), z);
      z = fma(__ldg(E + 64) * __ldg(E + 119), fma(__ldg(E + 261), g102, fma(__ldg(E + 260), g101, __ldg(E + 259) * g100)), z);
      z = fma(__ldg(E + 64) * __ldg(E + 120), fma(__ldg(E + 261), g112, fma(__ldg(E + 260), g111, __ldg(E + 259) * g110)), z);
      z = fma(__ldg(E + 65) * __ldg(E + 119), fma(__ldg(E + 261), g202, fma(__ldg(E + 260), g201, __ldg(E + 259) * g200)), z);
      z = fma(__ldg(E + 65) * __ldg(E + 120), fma(__ldg(E + 261), g212, fma(__ldg(E + 260), g211, __ldg(E + 259) * g210)), z);
      z = fma(__ldg(E + 66) * __ldg(E + 119), fma(__ldg(E + 261), g302, fma(__ldg(E + 260), g301, __ldg(E + 259) * g300)), z);
      z = fma(__ldg(E + 66) * __ldg(E + 120), fma(__ldg(E + 261), g312, fma(__ldg(E + 260), g311, __ldg(E + 259) * g310)), z);
      o5_9 = fma(Ei.w(59), z, o5_9); }
    if (ok) nfl += 1224;
  }
  const int N = a.b.nbf, fP = A.fP, fQ = A.fQ;
  const int fc = B.fP + cd / B.nfQ, fd = B.fQ + cd % B.nfQ;
  const double* __restrict__ PT = a.b.PT;
  const double s2 = 2.0 * deg;
  if (ok) {
    double z = 0.0;
    z = fma(o4_0, __ldg(PT + (fP + 4) * N + fQ + 0), z);
    z = fma(o4_1, __ldg(PT + (fP + 4) * N + fQ + 1), z);
    z = fma(o4_2, __ldg(PT + (fP + 4) * N + fQ + 2), z);
    z = fma(o4_3, __ldg(PT + (fP + 4) * N + fQ + 3), z);
    z = fma(o4_4, __ldg(PT + (fP + 4) * N + fQ + 4), z);
    z = fma(o4_5, __ldg(PT + (fP + 4) * N + fQ + 5), z);
    z = fma(o4_6, __ldg(PT + (fP + 4) * N + fQ + 6), z);
    z = fma(o4_7, __ldg(PT + (fP + 4) * N + fQ + 7), z);
    z = fma(o4_8, __ldg(PT + (fP + 4) * N + fQ + 8), z);
    z = fma(o4_9, __ldg(PT + (fP + 4) * N + fQ + 9), z);
    z = fma(o5_0, __ldg(PT + (fP + 5) * N + fQ + 0), z);
    z = fma(o5_1, __ldg(PT + (fP + 5) * N + fQ + 1), z);
    z = fma(o5_2, __ldg(PT + (fP + 5) * N + fQ + 2), z);
    z = fma(o5_3, __ldg(PT + (fP + 5) * N + fQ + 3), z);
    z = fma(o5_4, __ldg(PT + (fP + 5) * N + fQ + 4), z);
    z = fma(o5_5, __ldg(PT + (fP + 5) * N + fQ + 5), z);
    z = fma(o5_6, __ldg(PT + (fP + 5) * N + fQ + 6), z);
    z = fma(o5_7, __ldg(PT + (fP + 5) * N + fQ + 7), z);
    z = fma(o5_8, __ldg(PT + (fP + 5) * N + fQ + 8), z);
    z = fma(o5_9, __ldg(PT + (fP + 5) * N + fQ + 9), z);
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
        const double q6 = D[(fQ + 6) * N + fd];
        double kq6 = 0.0;
        const double q7 = D[(fQ + 7) * N + fd];
        double kq7 = 0.0;
        const double q8 = D[(fQ + 8) * N + fd];
        double kq8 = 0.0;
        const double q9 = D[(fQ + 9) * N + fd];
        double kq9 = 0.0;
        { const double px = D[(fP + 4) * N + fd]; double kp = 0.0;
          kp = fma(o4_0, q0, kp); kq0 = fma(o4_0, px, kq0);
          kp = fma(o4_1, q1, kp); kq1 = fma(o4_1, px, kq1);
          kp = fma(o4_2, q2, kp); kq2 = fma(o4_2, px, kq2);
          kp = fma(o4_3, q3, kp); kq3 = fma(o4_3, px, kq3);
          kp = fma(o4_4, q4, kp); kq4 = fma(o4_4, px, kq4);
          kp = fma(o4_5, q5, kp); kq5 = fma(o4_5, px, kq5);
          kp = fma(o4_6, q6, kp); kq6 = fma(o4_6, px, kq6);
          kp = fma(o4_7, q7, kp); kq7 = fma(o4_7, px, kq7);
          kp = fma(o4_8, q8, kp); kq8 = fma(o4_8, px, kq8);
          kp = fma(o4_9, q9, kp); kq9 = fma(o4_9, px, kq9);
          atomicAdd(K + (fP + 4) * N + fc, deg * kp); }
        { const double px = D[(fP + 5) * N + fd]; double kp = 0.0;
          kp = fma(o5_0, q0, kp); kq0 = fma(o5_0, px, kq0);
          kp = fma(o5_1, q1, kp); kq1 = fma(o5_1, px, kq1);
          kp = fma(o5_2, q2, kp); kq2 = fma(o5_2, px, kq2);
          kp = fma(o5_3, q3, kp); kq3 = fma(o5_3, px, kq3);
          kp = fma(o5_4, q4, kp); kq4 = fma(o5_4, px, kq4);
          kp = fma(o5_5, q5, kp); kq5 = fma(o5_5, px, kq5);
          kp = fma(o5_6, q6, kp); kq6 = fma(o5_6, px, kq6);
          kp = fma(o5_7, q7, kp); kq7 = fma(o5_7, px, kq7);
          kp = fma(o5_8, q8, kp); kq8 = fma(o5_8, px, kq8);
          kp = fma(o5_9, q9, kp); kq9 = fma(o5_9, px, kq9);
          atomicAdd(K + (fP + 5) * N + fc, deg * kp); }
        atomicAdd(K + (fQ + 0) * N + fc, deg * kq0);
        atomicAdd(K + (fQ + 1) * N + fc, deg * kq1);
        atomicAdd(K + (fQ + 2) * N + fc, deg * kq2);
        atomicAdd(K + (fQ + 3) * N + fc, deg * kq3);
        atomicAdd(K + (fQ + 4) * N + fc, deg * kq4);
        atomicAdd(K + (fQ + 5) * N + fc, deg * kq5);
        atomicAdd(K + (fQ + 6) * N + fc, deg * kq6);
        atomicAdd(K + (fQ + 7) * N + fc, deg * kq7);
        atomicAdd(K + (fQ + 8) * N + fc, deg * kq8);
        atomicAdd(K + (fQ + 9) * N + fc, deg * kq9);
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
        const double q6 = D[(fQ + 6) * N + fc];
        double kq6 = 0.0;
        const double q7 = D[(fQ + 7) * N + fc];
        double kq7 = 0.0;
        const double q8 = D[(fQ + 8) * N + fc];
        double kq8 = 0.0;
        const double q9 = D[(fQ + 9) * N + fc];
        double kq9 = 0.0;
        { const double px = D[(fP + 4) * N + fc]; double kp = 0.0;
          kp = fma(o4_0, q0, kp); kq0 = fma(o4_0, px, kq0);
          kp = fma(o4_1, q1, kp); kq1 = fma(o4_1, px, kq1);
          kp = fma(o4_2, q2, kp); kq2 = fma(o4_2, px, kq2);
          kp = fma(o4_3, q3, kp); kq3 = fma(o4_3, px, kq3);
          kp = fma(o4_4, q4, kp); kq4 = fma(o4_4, px, kq4);
          kp = fma(o4_5, q5, kp); kq5 = fma(o4_5, px, kq5);
          kp = fma(o4_6, q6, kp); kq6 = fma(o4_6, px, kq6);
          kp = fma(o4_7, q7, kp); kq7 = fma(o4_7, px, kq7);
          kp = fma(o4_8, q8, kp); kq8 = fma(o4_8, px, kq8);
          kp = fma(o4_9, q9, kp); kq9 = fma(o4_9, px, kq9);
          atomicAdd(K + (fP + 4) * N + fd, deg * kp); }
        { const double px = D[(fP + 5) * N + fc]; double kp = 0.0;
          kp = fma(o5_0, q0, kp); kq0 = fma(o5_0, px, kq0);
          kp = fma(o5_1, q1, kp); kq1 = fma(o5_1, px, kq1);
          kp = fma(o5_2, q2, kp); kq2 = fma(o5_2, px, kq2);
          kp = fma(o5_3, q3, kp); kq3 = fma(o5_3, px, kq3);
          kp = fma(o5_4, q4, kp); kq4 = fma(o5_4, px, kq4);
          kp = fma(o5_5, q5, kp); kq5 = fma(o5_5, px, kq5);
          kp = fma(o5_6, q6, kp); kq6 = fma(o5_6, px, kq6);
          kp = fma(o5_7, q7, kp); kq7 = fma(o5_7, px, kq7);
          kp = fma(o5_8, q8, kp); kq8 = fma(o5_8, px, kq8);
          kp = fma(o5_9, q9, kp); kq9 = fma(o5_9, px, kq9);
          atomicAdd(K + (fP + 5) * N + fd, deg * kp); }
        atomicAdd(K + (fQ + 0) * N + fd, deg * kq0);
        atomicAdd(K + (fQ + 1) * N + fd, deg * kq1);
        atomicAdd(K + (fQ + 2) * N + fd, deg * kq2);
        atomicAdd(K + (fQ + 3) * N + fd, deg * kq3);
        atomicAdd(K + (fQ + 4) * N + fd, deg * kq4);
        atomicAdd(K + (fQ + 5) * N + fd, deg * kq5);
        atomicAdd(K + (fQ + 6) * N + fd, deg * kq6);
        atomicAdd(K + (fQ + 7) * N + fd, deg * kq7);
        atomicAdd(K + (fQ + 8) * N + fd, deg * kq8);
        atomicAdd(K + (fQ + 9) * N + fd, deg * kq9);
      }
    }
    nfl += 2ull * 20 * (2 + 4 * (a.b.uhf ? 2 : 1));
  }
  {  // J[p][q]: every lane shares the bra pair
    const double w = ok ? s2 * __ldg(PT + fc * N + fd) : 0.0;
    { double v[32] = {w * o4_0, w * o4_1, w * o4_2, w * o4_3, w * o4_4, w * o4_5, w * o4_6, w * o4_7, w * o4_8, w * o4_9, w * o5_0, w * o5_1, w * o5_2, w * o5_3, w * o5_4, w * o5_5, w * o5_6, w * o5_7, w * o5_8, w * o5_9, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      const double z = sqb::warp_sum_scatter<32>(v); const int x = lane + 0;
      if (lane < 20 && z != 0.0) atomicAdd(a.b.J + (fP + 4 + x / 10) * N + fQ + x % 10, z); }
  }
  sqb::count_add(a.counters + 0, ok && cd == 0 && false ? 1ull : 0ull);
  sqb::count_add(a.counters + 1, npq);
  sqb::count_add(a.counters + 2, nfl);
}
