// generated by gen_fshell_kernels.py -- do not edit
#include "../jk_generic_dev.cuh"

extern "C" __global__ void __launch_bounds__(128)
jkf_FD_1(const sqb::FArgs a, const sqb::FRun* __restrict__ runs, const long long* __restrict__ first, int nruns,
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
  double o5_0 = 0.0;
  double o5_1 = 0.0;
  double o5_2 = 0.0;
  double o5_3 = 0.0;
  double o5_4 = 0.0;
  double o5_5 = 0.0;
  double o6_0 = 0.0;
  double o6_1 = 0.0;
  double o6_2 = 0.0;
  double o6_3 = 0.0;
  double o6_4 = 0.0;
  double o6_5 = 0.0;
  double o7_0 = 0.0;
  double o7_1 = 0.0;
  double o7_2 = 0.0;
  double o7_3 = 0.0;
  double o7_4 = 0.0;
  double o7_5 = 0.0;
  double o8_0 = 0.0;
  double o8_1 = 0.0;
  double o8_2 = 0.0;
  double o8_3 = 0.0;
  double o8_4 = 0.0;
  double o8_5 = 0.0;
  double o9_0 = 0.0;
  double o9_1 = 0.0;
  double o9_2 = 0.0;
  double o9_3 = 0.0;
  double o9_4 = 0.0;
  double o9_5 = 0.0;
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
      z = fma(__ldg(E + 48), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 49), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 50), fma(__ldg(E + 163), g201, __ldg(E + 162) * g200), z);
      z = fma(__ldg(E + 51), fma(__ldg(E + 163), g301, __ldg(E + 162) * g300), z);
      z = fma(__ldg(E + 52), fma(__ldg(E + 163), g401, __ldg(E + 162) * g400), z);
      o5_0 = fma(Ei.w(30), z, o5_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 36) * __ldg(E + 84), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 36) * __ldg(E + 85), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 36) * __ldg(E + 86), fma(__ldg(E + 163), g021, __ldg(E + 162) * g020), z);
      z = fma(__ldg(E + 37) * __ldg(E + 84), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 37) * __ldg(E + 85), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 37) * __ldg(E + 86), fma(__ldg(E + 163), g121, __ldg(E + 162) * g120), z);
      z = fma(__ldg(E + 38) * __ldg(E + 84), fma(__ldg(E + 163), g201, __ldg(E + 162) * g200), z);
      z = fma(__ldg(E + 38) * __ldg(E + 85), fma(__ldg(E + 163), g211, __ldg(E + 162) * g210), z);
      z = fma(__ldg(E + 38) * __ldg(E + 86), fma(__ldg(E + 163), g221, __ldg(E + 162) * g220), z);
      o5_1 = fma(Ei.w(31), z, o5_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 36), fma(__ldg(E + 177), g003, fma(__ldg(E + 176), g002, fma(__ldg(E + 175), g001, __ldg(E + 174) * g000))), z);
      z = fma(__ldg(E + 37), fma(__ldg(E + 177), g103, fma(__ldg(E + 176), g102, fma(__ldg(E + 175), g101, __ldg(E + 174) * g100))), z);
      z = fma(__ldg(E + 38), fma(__ldg(E + 177), g203, fma(__ldg(E + 176), g202, fma(__ldg(E + 175), g201, __ldg(E + 174) * g200))), z);
      o5_2 = fma(Ei.w(32), z, o5_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 42) * __ldg(E + 78), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 42) * __ldg(E + 79), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 43) * __ldg(E + 78), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 43) * __ldg(E + 79), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 44) * __ldg(E + 78), fma(__ldg(E + 163), g201, __ldg(E + 162) * g200), z);
      z = fma(__ldg(E + 44) * __ldg(E + 79), fma(__ldg(E + 163), g211, __ldg(E + 162) * g210), z);
      z = fma(__ldg(E + 45) * __ldg(E + 78), fma(__ldg(E + 163), g301, __ldg(E + 162) * g300), z);
      z = fma(__ldg(E + 45) * __ldg(E + 79), fma(__ldg(E + 163), g311, __ldg(E + 162) * g310), z);
      o5_3 = fma(Ei.w(33), z, o5_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 42), fma(__ldg(E + 170), g002, fma(__ldg(E + 169), g001, __ldg(E + 168) * g000)), z);
      z = fma(__ldg(E + 43), fma(__ldg(E + 170), g102, fma(__ldg(E + 169), g101, __ldg(E + 168) * g100)), z);
      z = fma(__ldg(E + 44), fma(__ldg(E + 170), g202, fma(__ldg(E + 169), g201, __ldg(E + 168) * g200)), z);
      z = fma(__ldg(E + 45), fma(__ldg(E + 170), g302, fma(__ldg(E + 169), g301, __ldg(E + 168) * g300)), z);
      o5_4 = fma(Ei.w(34), z, o5_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 36) * __ldg(E + 78), fma(__ldg(E + 170), g002, fma(__ldg(E + 169), g001, __ldg(E + 168) * g000)), z);
      z = fma(__ldg(E + 36) * __ldg(E + 79), fma(__ldg(E + 170), g012, fma(__ldg(E + 169), g011, __ldg(E + 168) * g010)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 78), fma(__ldg(E + 170), g102, fma(__ldg(E + 169), g101, __ldg(E + 168) * g100)), z);
      z = fma(__ldg(E + 37) * __ldg(E + 79), fma(__ldg(E + 170), g112, fma(__ldg(E + 169), g111, __ldg(E + 168) * g110)), z);
      z = fma(__ldg(E + 38) * __ldg(E + 78), fma(__ldg(E + 170), g202, fma(__ldg(E + 169), g201, __ldg(E + 168) * g200)), z);
      z = fma(__ldg(E + 38) * __ldg(E + 79), fma(__ldg(E + 170), g212, fma(__ldg(E + 169), g211, __ldg(E + 168) * g210)), z);
      o5_5 = fma(Ei.w(35), z, o5_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 30), fma(__ldg(E + 182), g002, fma(__ldg(E + 181), g001, __ldg(E + 180) * g000)), z);
      z = fma(__ldg(E + 31), fma(__ldg(E + 182), g102, fma(__ldg(E + 181), g101, __ldg(E + 180) * g100)), z);
      z = fma(__ldg(E + 32), fma(__ldg(E + 182), g202, fma(__ldg(E + 181), g201, __ldg(E + 180) * g200)), z);
      z = fma(__ldg(E + 33), fma(__ldg(E + 182), g302, fma(__ldg(E + 181), g301, __ldg(E + 180) * g300)), z);
      o6_0 = fma(Ei.w(36), z, o6_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 84), fma(__ldg(E + 182), g002, fma(__ldg(E + 181), g001, __ldg(E + 180) * g000)), z);
      z = fma(__ldg(E + 18) * __ldg(E + 85), fma(__ldg(E + 182), g012, fma(__ldg(E + 181), g011, __ldg(E + 180) * g010)), z);
      z = fma(__ldg(E + 18) * __ldg(E + 86), fma(__ldg(E + 182), g022, fma(__ldg(E + 181), g021, __ldg(E + 180) * g020)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 84), fma(__ldg(E + 182), g102, fma(__ldg(E + 181), g101, __ldg(E + 180) * g100)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 85), fma(__ldg(E + 182), g112, fma(__ldg(E + 181), g111, __ldg(E + 180) * g110)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 86), fma(__ldg(E + 182), g122, fma(__ldg(E + 181), g121, __ldg(E + 180) * g120)), z);
      o6_1 = fma(Ei.w(37), z, o6_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 18), fma(__ldg(E + 196), g004, fma(__ldg(E + 195), g003, fma(__ldg(E + 194), g002, fma(__ldg(E + 193), g001, __ldg(E + 192) * g000)))), z);
      z = fma(__ldg(E + 19), fma(__ldg(E + 196), g104, fma(__ldg(E + 195), g103, fma(__ldg(E + 194), g102, fma(__ldg(E + 193), g101, __ldg(E + 192) * g100)))), z);
      o6_2 = fma(Ei.w(38), z, o6_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 24) * __ldg(E + 78), fma(__ldg(E + 182), g002, fma(__ldg(E + 181), g001, __ldg(E + 180) * g000)), z);
      z = fma(__ldg(E + 24) * __ldg(E + 79), fma(__ldg(E + 182), g012, fma(__ldg(E + 181), g011, __ldg(E + 180) * g010)), z);
      z = fma(__ldg(E + 25) * __ldg(E + 78), fma(__ldg(E + 182), g102, fma(__ldg(E + 181), g101, __ldg(E + 180) * g100)), z);
      z = fma(__ldg(E + 25) * __ldg(E + 79), fma(__ldg(E + 182), g112, fma(__ldg(E + 181), g111, __ldg(E + 180) * g110)), z);
      z = fma(__ldg(E + 26) * __ldg(E + 78), fma(__ldg(E + 182), g202, fma(__ldg(E + 181), g201, __ldg(E + 180) * g200)), z);
      z = fma(__ldg(E + 26) * __ldg(E + 79), fma(__ldg(E + 182), g212, fma(__ldg(E + 181), g211, __ldg(E + 180) * g210)), z);
      o6_3 = fma(Ei.w(39), z, o6_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 24), fma(__ldg(E + 189), g003, fma(__ldg(E + 188), g002, fma(__ldg(E + 187), g001, __ldg(E + 186) * g000))), z);
      z = fma(__ldg(E + 25), fma(__ldg(E + 189), g103, fma(__ldg(E + 188), g102, fma(__ldg(E + 187), g101, __ldg(E + 186) * g100))), z);
      z = fma(__ldg(E + 26), fma(__ldg(E + 189), g203, fma(__ldg(E + 188), g202, fma(__ldg(E + 187), g201, __ldg(E + 186) * g200))), z);
      o6_4 = fma(Ei.w(40), z, o6_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 78), fma(__ldg(E + 189), g003, fma(__ldg(E + 188), g002, fma(__ldg(E + 187), g001, __ldg(E + 186) * g000))), z);
      z = fma(__ldg(E + 18) * __ldg(E + 79), fma(__ldg(E + 189), g013, fma(__ldg(E + 188), g012, fma(__ldg(E + 187), g011, __ldg(E + 186) * g010))), z);
      z = fma(__ldg(E + 19) * __ldg(E + 78), fma(__ldg(E + 189), g103, fma(__ldg(E + 188), g102, fma(__ldg(E + 187), g101, __ldg(E + 186) * g100))), z);
      z = fma(__ldg(E + 19) * __ldg(E + 79), fma(__ldg(E + 189), g113, fma(__ldg(E + 188), g112, fma(__ldg(E + 187), g111, __ldg(E + 186) * g110))), z);
      o6_5 = fma(Ei.w(41), z, o6_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 12) * __ldg(E + 108), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 12) * __ldg(E + 109), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 12) * __ldg(E + 110), fma(__ldg(E + 163), g021, __ldg(E + 162) * g020), z);
      z = fma(__ldg(E + 13) * __ldg(E + 108), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 13) * __ldg(E + 109), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 13) * __ldg(E + 110), fma(__ldg(E + 163), g121, __ldg(E + 162) * g120), z);
      z = fma(__ldg(E + 14) * __ldg(E + 108), fma(__ldg(E + 163), g201, __ldg(E + 162) * g200), z);
      z = fma(__ldg(E + 14) * __ldg(E + 109), fma(__ldg(E + 163), g211, __ldg(E + 162) * g210), z);
      z = fma(__ldg(E + 14) * __ldg(E + 110), fma(__ldg(E + 163), g221, __ldg(E + 162) * g220), z);
      o7_0 = fma(Ei.w(42), z, o7_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 120), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 121), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 122), fma(__ldg(E + 163), g021, __ldg(E + 162) * g020), z);
      z = fma(__ldg(E + 123), fma(__ldg(E + 163), g031, __ldg(E + 162) * g030), z);
      z = fma(__ldg(E + 124), fma(__ldg(E + 163), g041, __ldg(E + 162) * g040), z);
      o7_1 = fma(Ei.w(43), z, o7_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 108), fma(__ldg(E + 177), g003, fma(__ldg(E + 176), g002, fma(__ldg(E + 175), g001, __ldg(E + 174) * g000))), z);
      z = fma(__ldg(E + 109), fma(__ldg(E + 177), g013, fma(__ldg(E + 176), g012, fma(__ldg(E + 175), g011, __ldg(E + 174) * g010))), z);
      z = fma(__ldg(E + 110), fma(__ldg(E + 177), g023, fma(__ldg(E + 176), g022, fma(__ldg(E + 175), g021, __ldg(E + 174) * g020))), z);
      o7_2 = fma(Ei.w(44), z, o7_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 114), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 6) * __ldg(E + 115), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 6) * __ldg(E + 116), fma(__ldg(E + 163), g021, __ldg(E + 162) * g020), z);
      z = fma(__ldg(E + 6) * __ldg(E + 117), fma(__ldg(E + 163), g031, __ldg(E + 162) * g030), z);
      z = fma(__ldg(E + 7) * __ldg(E + 114), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 7) * __ldg(E + 115), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 7) * __ldg(E + 116), fma(__ldg(E + 163), g121, __ldg(E + 162) * g120), z);
      z = fma(__ldg(E + 7) * __ldg(E + 117), fma(__ldg(E + 163), g131, __ldg(E + 162) * g130), z);
      o7_3 = fma(Ei.w(45), z, o7_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 108), fma(__ldg(E + 170), g002, fma(__ldg(E + 169), g001, __ldg(E + 168) * g000)), z);
      z = fma(__ldg(E + 6) * __ldg(E + 109), fma(__ldg(E + 170), g012, fma(__ldg(E + 169), g011, __ldg(E + 168) * g010)), z);
      z = fma(__ldg(E + 6) * __ldg(E + 110), fma(__ldg(E + 170), g022, fma(__ldg(E + 169), g021, __ldg(E + 168) * g020)), z);
      z = fma(__ldg(E + 7) * __ldg(E + 108), fma(__ldg(E + 170), g102, fma(__ldg(E + 169), g101, __ldg(E + 168) * g100)), z);
      z = fma(__ldg(E + 7) * __ldg(E + 109), fma(__ldg(E + 170), g112, fma(__ldg(E + 169), g111, __ldg(E + 168) * g110)), z);
      z = fma(__ldg(E + 7) * __ldg(E + 110), fma(__ldg(E + 170), g122, fma(__ldg(E + 169), g121, __ldg(E + 168) * g120)), z);
      o7_4 = fma(Ei.w(46), z, o7_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 114), fma(__ldg(E + 170), g002, fma(__ldg(E + 169), g001, __ldg(E + 168) * g000)), z);
      z = fma(__ldg(E + 115), fma(__ldg(E + 170), g012, fma(__ldg(E + 169), g011, __ldg(E + 168) * g010)), z);
      z = fma(__ldg(E + 116), fma(__ldg(E + 170), g022, fma(__ldg(E + 169), g021, __ldg(E + 168) * g020)), z);
      z = fma(__ldg(E + 117), fma(__ldg(E + 170), g032, fma(__ldg(E + 169), g031, __ldg(E + 168) * g030)), z);
      o7_5 = fma(Ei.w(47), z, o7_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 12) * __ldg(E + 90), fma(__ldg(E + 182), g002, fma(__ldg(E + 181), g001, __ldg(E + 180) * g000)), z);
      z = fma(__ldg(E + 12) * __ldg(E + 91), fma(__ldg(E + 182), g012, fma(__ldg(E + 181), g011, __ldg(E + 180) * g010)), z);
      z = fma(__ldg(E + 13) * __ldg(E + 90), fma(__ldg(E + 182), g102, fma(__ldg(E + 181), g101, __ldg(E + 180) * g100)), z);
      z = fma(__ldg(E + 13) * __ldg(E + 91), fma(__ldg(E + 182), g112, fma(__ldg(E + 181), g111, __ldg(E + 180) * g110)), z);
      z = fma(__ldg(E + 14) * __ldg(E + 90), fma(__ldg(E + 182), g202, fma(__ldg(E + 181), g201, __ldg(E + 180) * g200)), z);
      z = fma(__ldg(E + 14) * __ldg(E + 91), fma(__ldg(E + 182), g212, fma(__ldg(E + 181), g211, __ldg(E + 180) * g210)), z);
      o8_0 = fma(Ei.w(48), z, o8_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 102), fma(__ldg(E + 182), g002, fma(__ldg(E + 181), g001, __ldg(E + 180) * g000)), z);
      z = fma(__ldg(E + 103), fma(__ldg(E + 182), g012, fma(__ldg(E + 181), g011, __ldg(E + 180) * g010)), z);
      z = fma(__ldg(E + 104), fma(__ldg(E + 182), g022, fma(__ldg(E + 181), g021, __ldg(E + 180) * g020)), z);
      z = fma(__ldg(E + 105), fma(__ldg(E + 182), g032, fma(__ldg(E + 181), g031, __ldg(E + 180) * g030)), z);
      o8_1 = fma(Ei.w(49), z, o8_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 90), fma(__ldg(E + 196), g004, fma(__ldg(E + 195), g003, fma(__ldg(E + 194), g002, fma(__ldg(E + 193), g001, __ldg(E + 192) * g000)))), z);
      z = fma(__ldg(E + 91), fma(__ldg(E + 196), g014, fma(__ldg(E + 195), g013, fma(__ldg(E + 194), g012, fma(__ldg(E + 193), g011, __ldg(E + 192) * g010)))), z);
      o8_2 = fma(Ei.w(50), z, o8_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 96), fma(__ldg(E + 182), g002, fma(__ldg(E + 181), g001, __ldg(E + 180) * g000)), z);
      z = fma(__ldg(E + 6) * __ldg(E + 97), fma(__ldg(E + 182), g012, fma(__ldg(E + 181), g011, __ldg(E + 180) * g010)), z);
      z = fma(__ldg(E + 6) * __ldg(E + 98), fma(__ldg(E + 182), g022, fma(__ldg(E + 181), g021, __ldg(E + 180) * g020)), z);
      z = fma(__ldg(E + 7) * __ldg(E + 96), fma(__ldg(E + 182), g102, fma(__ldg(E + 181), g101, __ldg(E + 180) * g100)), z);
      z = fma(__ldg(E + 7) * __ldg(E + 97), fma(__ldg(E + 182), g112, fma(__ldg(E + 181), g111, __ldg(E + 180) * g110)), z);
      z = fma(__ldg(E + 7) * __ldg(E + 98), fma(__ldg(E + 182), g122, fma(__ldg(E + 181), g121, __ldg(E + 180) * g120)), z);
      o8_3 = fma(Ei.w(51), z, o8_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 6) * __ldg(E + 90), fma(__ldg(E + 189), g003, fma(__ldg(E + 188), g002, fma(__ldg(E + 187), g001, __ldg(E + 186) * g000))), z);
      z = fma(__ldg(E + 6) * __ldg(E + 91), fma(__ldg(E + 189), g013, fma(__ldg(E + 188), g012, fma(__ldg(E + 187), g011, __ldg(E + 186) * g010))), z);
      z = fma(__ldg(E + 7) * __ldg(E + 90), fma(__ldg(E + 189), g103, fma(__ldg(E + 188), g102, fma(__ldg(E + 187), g101, __ldg(E + 186) * g100))), z);
      z = fma(__ldg(E + 7) * __ldg(E + 91), fma(__ldg(E + 189), g113, fma(__ldg(E + 188), g112, fma(__ldg(E + 187), g111, __ldg(E + 186) * g110))), z);
      o8_4 = fma(Ei.w(52), z, o8_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 96), fma(__ldg(E + 189), g003, fma(__ldg(E + 188), g002, fma(__ldg(E + 187), g001, __ldg(E + 186) * g000))), z);
      z = fma(__ldg(E + 97), fma(__ldg(E + 189), g013, fma(__ldg(E + 188), g012, fma(__ldg(E + 187), g011, __ldg(E + 186) * g010))), z);
      z = fma(__ldg(E + 98), fma(__ldg(E + 189), g023, fma(__ldg(E + 188), g022, fma(__ldg(E + 187), g021, __ldg(E + 186) * g020))), z);
      o8_5 = fma(Ei.w(53), z, o8_5); }
    { double z = 0.0;
      z = fma(__ldg(E + 30) * __ldg(E + 90), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 30) * __ldg(E + 91), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 31) * __ldg(E + 90), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 31) * __ldg(E + 91), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 32) * __ldg(E + 90), fma(__ldg(E + 163), g201, __ldg(E + 162) * g200), z);
      z = fma(__ldg(E + 32) * __ldg(E + 91), fma(__ldg(E + 163), g211, __ldg(E + 162) * g210), z);
      z = fma(__ldg(E + 33) * __ldg(E + 90), fma(__ldg(E + 163), g301, __ldg(E + 162) * g300), z);
      z = fma(__ldg(E + 33) * __ldg(E + 91), fma(__ldg(E + 163), g311, __ldg(E + 162) * g310), z);
      o9_0 = fma(Ei.w(54), z, o9_0); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 102), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 18) * __ldg(E + 103), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 18) * __ldg(E + 104), fma(__ldg(E + 163), g021, __ldg(E + 162) * g020), z);
      z = fma(__ldg(E + 18) * __ldg(E + 105), fma(__ldg(E + 163), g031, __ldg(E + 162) * g030), z);
      z = fma(__ldg(E + 19) * __ldg(E + 102), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 19) * __ldg(E + 103), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 19) * __ldg(E + 104), fma(__ldg(E + 163), g121, __ldg(E + 162) * g120), z);
      z = fma(__ldg(E + 19) * __ldg(E + 105), fma(__ldg(E + 163), g131, __ldg(E + 162) * g130), z);
      o9_1 = fma(Ei.w(55), z, o9_1); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 90), fma(__ldg(E + 177), g003, fma(__ldg(E + 176), g002, fma(__ldg(E + 175), g001, __ldg(E + 174) * g000))), z);
      z = fma(__ldg(E + 18) * __ldg(E + 91), fma(__ldg(E + 177), g013, fma(__ldg(E + 176), g012, fma(__ldg(E + 175), g011, __ldg(E + 174) * g010))), z);
      z = fma(__ldg(E + 19) * __ldg(E + 90), fma(__ldg(E + 177), g103, fma(__ldg(E + 176), g102, fma(__ldg(E + 175), g101, __ldg(E + 174) * g100))), z);
      z = fma(__ldg(E + 19) * __ldg(E + 91), fma(__ldg(E + 177), g113, fma(__ldg(E + 176), g112, fma(__ldg(E + 175), g111, __ldg(E + 174) * g110))), z);
      o9_2 = fma(Ei.w(56), z, o9_2); }
    { double z = 0.0;
      z = fma(__ldg(E + 24) * __ldg(E + 96), fma(__ldg(E + 163), g001, __ldg(E + 162) * g000), z);
      z = fma(__ldg(E + 24) * __ldg(E + 97), fma(__ldg(E + 163), g011, __ldg(E + 162) * g010), z);
      z = fma(__ldg(E + 24) * __ldg(E + 98), fma(__ldg(E + 163), g021, __ldg(E + 162) * g020), z);
      z = fma(__ldg(E + 25) * __ldg(E + 96), fma(__ldg(E + 163), g101, __ldg(E + 162) * g100), z);
      z = fma(__ldg(E + 25) * __ldg(E + 97), fma(__ldg(E + 163), g111, __ldg(E + 162) * g110), z);
      z = fma(__ldg(E + 25) * __ldg(E + 98), fma(__ldg(E + 163), g121, __ldg(E + 162) * g120), z);
      z = fma(__ldg(E + 26) * __ldg(E + 96), fma(__ldg(E + 163), g201, __ldg(E + 162) * g200), z);
      z = fma(__ldg(E + 26) * __ldg(E + 97), fma(__ldg(E + 163), g211, __ldg(E + 162) * g210), z);
      z = fma(__ldg(E + 26) * __ldg(E + 98), fma(__ldg(E + 163), g221, __ldg(E + 162) * g220), z);
      o9_3 = fma(Ei.w(57), z, o9_3); }
    { double z = 0.0;
      z = fma(__ldg(E + 24) * __ldg(E + 90), fma(__ldg(E + 170), g002, fma(__ldg(E + 169), g001, __ldg(E + 168) * g000)), z);
      z = fma(__ldg(E + 24) * __ldg(E + 91), fma(__ldg(E + 170), g012, fma(__ldg(E + 169), g011, __ldg(E + 168) * g010)), z);
      z = fma(__ldg(E + 25) * __ldg(E + 90), fma(__ldg(E + 170), g102, fma(__ldg(E + 169), g101, __ldg(E + 168) * g100)), z);
      z = fma(__ldg(E + 25) * __ldg(E + 91), fma(__ldg(E + 170), g112, fma(__ldg(E + 169), g111, __ldg(E + 168) * g110)), z);
      z = fma(__ldg(E + 26) * __ldg(E + 90), fma(__ldg(E + 170), g202, fma(__ldg(E + 169), g201, __ldg(E + 168) * g200)), z);
      z = fma(__ldg(E + 26) * __ldg(E + 91), fma(__ldg(E + 170), g212, fma(__ldg(E + 169), g211, __ldg(E + 168) * g210)), z);
      o9_4 = fma(Ei.w(58), z, o9_4); }
    { double z = 0.0;
      z = fma(__ldg(E + 18) * __ldg(E + 96), fma(__ldg(E + 170), g002, fma(__ldg(E + 169), g001, __ldg(E + 168) * g000)), z);
      z = fma(__ldg(E + 18) * __ldg(E + 97), fma(__ldg(E + 170), g012, fma(__ldg(E + 169), g011, __ldg(E + 168) * g010)), z);
      z = fma(__ldg(E + 18) * __ldg(E + 98), fma(__ldg(E + 170), g022, fma(__ldg(E + 169), g021, __ldg(E + 168) * g020)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 96), fma(__ldg(E + 170), g102, fma(__ldg(E + 169), g101, __ldg(E + 168) * g100)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 97), fma(__ldg(E + 170), g112, fma(__ldg(E + 169), g111, __ldg(E + 168) * g110)), z);
      z = fma(__ldg(E + 19) * __ldg(E + 98), fma(__ldg(E + 170), g122, fma(__ldg(E + 169), g121, __ldg(E + 168) * g120)), z);
      o9_5 = fma(Ei.w(59), z, o9_5); }
    if (ok) nfl += 1274;
  }
  const int N = a.b.nbf, fP = A.fP, fQ = A.fQ;
  const int fc = B.fP + cd / B.nfQ, fd = B.fQ + cd % B.nfQ;
  const double* __restrict__ PT = a.b.PT;
  const double s2 = 2.0 * deg;
  if (ok) {
    double z = 0.0;
    z = fma(o5_0, __ldg(PT + (fP + 5) * N + fQ + 0), z);
    z = fma(o5_1, __ldg(PT + (fP + 5) * N + fQ + 1), z);
    z = fma(o5_2, __ldg(PT + (fP + 5) * N + fQ + 2), z);
    z = fma(o5_3, __ldg(PT + (fP + 5) * N + fQ + 3), z);
    z = fma(o5_4, __ldg(PT + (fP + 5) * N + fQ + 4), z);
    z = fma(o5_5, __ldg(PT + (fP + 5) * N + fQ + 5), z);
    z = fma(o6_0, __ldg(PT + (fP + 6) * N + fQ + 0), z);
    z = fma(o6_1, __ldg(PT + (fP + 6) * N + fQ + 1), z);
    z = fma(o6_2, __ldg(PT + (fP + 6) * N + fQ + 2), z);
    z = fma(o6_3, __ldg(PT + (fP + 6) * N + fQ + 3), z);
    z = fma(o6_4, __ldg(PT + (fP + 6) * N + fQ + 4), z);
    z = fma(o6_5, __ldg(PT + (fP + 6) * N + fQ + 5), z);
    z = fma(o7_0, __ldg(PT + (fP + 7) * N + fQ + 0), z);
    z = fma(o7_1, __ldg(PT + (fP + 7) * N + fQ + 1), z);
    z = fma(o7_2, __ldg(PT + (fP + 7) * N + fQ + 2), z);
    z = fma(o7_3, __ldg(PT + (fP + 7) * N + fQ + 3), z);
    z = fma(o7_4, __ldg(PT + (fP + 7) * N + fQ + 4), z);
    z = fma(o7_5, __ldg(PT + (fP + 7) * N + fQ + 5), z);
    z = fma(o8_0, __ldg(PT + (fP + 8) * N + fQ + 0), z);
    z = fma(o8_1, __ldg(PT + (fP + 8) * N + fQ + 1), z);
    z = fma(o8_2, __ldg(PT + (fP + 8) * N + fQ + 2), z);
    z = fma(o8_3, __ldg(PT + (fP + 8) * N + fQ + 3), z);
    z = fma(o8_4, __ldg(PT + (fP + 8) * N + fQ + 4), z);
    z = fma(o8_5, __ldg(PT + (fP + 8) * N + fQ + 5), z);
    z = fma(o9_0, __ldg(PT + (fP + 9) * N + fQ + 0), z);
    z = fma(o9_1, __ldg(PT + (fP + 9) * N + fQ + 1), z);
    z = fma(o9_2, __ldg(PT + (fP + 9) * N + fQ + 2), z);
    z = fma(o9_3, __ldg(PT + (fP + 9) * N + fQ + 3), z);
    z = fma(o9_4, __ldg(PT + (fP + 9) * N + fQ + 4), z);
    z = fma(o9_5, __ldg(PT + (fP + 9) * N + fQ + 5), z);
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
        { const double px = D[(fP + 5) * N + fd]; double kp = 0.0;
          kp = fma(o5_0, q0, kp); kq0 = fma(o5_0, px, kq0);
          kp = fma(o5_1, q1, kp); kq1 = fma(o5_1, px, kq1);
          kp = fma(o5_2, q2, kp); kq2 = fma(o5_2, px, kq2);
          kp = fma(o5_3, q3, kp); kq3 = fma(o5_3, px, kq3);
          kp = fma(o5_4, q4, kp); kq4 = fma(o5_4, px, kq4);
          kp = fma(o5_5, q5, kp); kq5 = fma(o5_5, px, kq5);
          atomicAdd(K + (fP + 5) * N + fc, deg * kp); }
        { const double px = D[(fP + 6) * N + fd]; double kp = 0.0;
          kp = fma(o6_0, q0, kp); kq0 = fma(o6_0, px, kq0);
          kp = fma(o6_1, q1, kp); kq1 = fma(o6_1, px, kq1);
          kp = fma(o6_2, q2, kp); kq2 = fma(o6_2, px, kq2);
          kp = fma(o6_3, q3, kp); kq3 = fma(o6_3, px, kq3);
          kp = fma(o6_4, q4, kp); kq4 = fma(o6_4, px, kq4);
          kp = fma(o6_5, q5, kp); kq5 = fma(o6_5, px, kq5);
          atomicAdd(K + (fP + 6) * N + fc, deg * kp); }
        { const double px = D[(fP + 7) * N + fd]; double kp = 0.0;
          kp = fma(o7_0, q0, kp); kq0 = fma(o7_0, px, kq0);
          kp = fma(o7_1, q1, kp); kq1 = fma(o7_1, px, kq1);
          kp = fma(o7_2, q2, kp); kq2 = fma(o7_2, px, kq2);
          kp = fma(o7_3, q3, kp); kq3 = fma(o7_3, px, kq3);
          kp = fma(o7_4, q4, kp); kq4 = fma(o7_4, px, kq4);
          kp = fma(o7_5, q5, kp); kq5 = fma(o7_5, px, kq5);
          atomicAdd(K + (fP + 7) * N + fc, deg * kp); }
        { const double px = D[(fP + 8) * N + fd]; double kp = 0.0;
          kp = fma(o8_0, q0, kp); kq0 = fma(o8_0, px, kq0);
          kp = fma(o8_1, q1, kp); kq1 = fma(o8_1, px, kq1);
          kp = fma(o8_2, q2, kp); kq2 = fma(o8_2, px, kq2);
          kp = fma(o8_3, q3, kp); kq3 = fma(o8_3, px, kq3);
          kp = fma(o8_4, q4, kp); kq4 = fma(o8_4, px, kq4);
          kp = fma(o8_5, q5, kp); kq5 = fma(o8_5, px, kq5);
          atomicAdd(K + (fP + 8) * N + fc, deg * kp); }
        { const double px = D[(fP + 9) * N + fd]; double kp = 0.0;
          kp = fma(o9_0, q0, kp); kq0 = fma(o9_0, px, kq0);
          kp = fma(o9_1, q1, kp); kq1 = fma(o9_1, px, kq1);
          kp = fma(o9_2, q2, kp); kq2 = fma(o9_2, px, kq2);
          kp = fma(o9_3, q3, kp); kq3 = fma(o9_3, px, kq3);
          kp = fma(o9_4, q4, kp); kq4 = fma(o9_4, px, kq4);
          kp = fma(o9_5, q5, kp); kq5 = fma(o9_5, px, kq5);
          atomicAdd(K + (fP + 9) * N + fc, deg * kp); }
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
        { const double px = D[(fP + 5) * N + fc]; double kp = 0.0;
          kp = fma(o5_0, q0, kp); kq0 = fma(o5_0, px, kq0);
          kp = fma(o5_1, q1, kp); kq1 = fma(o5_1, px, kq1);
          kp = fma(o5_2, q2, kp); kq2 = fma(o5_2, px, kq2);
          kp = fma(o5_3, q3, kp); kq3 = fma(o5_3, px, kq3);
          kp = fma(o5_4, q4, kp); kq4 = fma(o5_4, px, kq4);
          kp = fma(o5_5, q5, kp); kq5 = fma(o5_5, px, kq5);
          atomicAdd(K + (fP + 5) * N + fd, deg * kp); }
        { const double px = D[(fP + 6) * N + fc]; double kp = 0.0;
          kp = fma(o6_0, q0, kp); kq0 = fma(o6_0, px, kq0);
          kp = fma(o6_1, q1, kp); kq1 = fma(o6_1, px, kq1);
          kp = fma(o6_2, q2, kp); kq2 = fma(o6_2, px, kq2);
          kp = fma(o6_3, q3, kp); kq3 = fma(o6_3, px, kq3);
          kp = fma(o6_4, q4, kp); kq4 = fma(o6_4, px, kq4);
          kp = fma(o6_5, q5, kp); kq5 = fma(o6_5, px, kq5);
          atomicAdd(K + (fP + 6) * N + fd, deg * kp); }
        { const double px = D[(fP + 7) * N + fc]; double kp = 0.0;
          kp = fma(o7_0, q0, kp); kq0 = fma(o7_0, px, kq0);
          kp = fma(o7_1, q1, kp); kq1 = fma(o7_1, px, kq1);
          kp = fma(o7_2, q2, kp); kq2 = fma(o7_2, px, kq2);
          kp = fma(o7_3, q3, kp); kq3 = fma(o7_3, px, kq3);
          kp = fma(o7_4, q4, kp); kq4 = fma(o7_4, px, kq4);
          kp = fma(o7_5, q5, kp); kq5 = fma(o7_5, px, kq5);
          atomicAdd(K + (fP + 7) * N + fd, deg * kp); }
        { const double px = D[(fP + 8) * N + fc]; double kp = 0.0;
          kp = fma(o8_0, q0, kp); kq0 = fma(o8_0, px, kq0);
          kp = fma(o8_1, q1, kp); kq1 = fma(o8_1, px, kq1);
          kp = fma(o8_2, q2, kp); kq2 = fma(o8_2, px, kq2);
          kp = fma(o8_3, q3, kp); kq3 = fma(o8_3, px, kq3);
          kp = fma(o8_4, q4, kp); kq4 = fma(o8_4, px, kq4);
          kp = fma(o8_5, q5, kp); kq5 = fma(o8_5, px, kq5);
          atomicAdd(K + (fP + 8) * N + fd, deg * kp); }
        { const double px = D[(fP + 9) * N + fc]; double kp = 0.0;
          kp = fma(o9_0, q0, kp); kq0 = fma(o9_0, px, kq0);
          kp = fma(o9_1, q1, kp); kq1 = fma(o9_1, px, kq1);
          kp = fma(o9_2, q2, kp); kq2 = fma(o9_2, px, kq2);
          kp = fma(o9_3, q3, kp); kq3 = fma(o9_3, px, kq3);
          kp = fma(o9_4, q4, kp); kq4 = fma(o9_4, px, kq4);
          kp = fma(o9_5, q5, kp); kq5 = fma(o9_5, px, kq5);
          atomicAdd(K + (fP + 9) * N + fd, deg * kp); }
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
    { double v[32] = {w * o5_0, w * o5_1, w * o5_2, w * o5_3, w * o5_4, w * o5_5, w * o6_0, w * o6_1, w * o6_2, w * o6_3, w * o6_4, w * o6_5, w * o7_0, w * o7_1, w * o7_2, w * o7_3, w * o7_4, w * o7_5, w * o8_0, w * o8_1, w * o8_2, w * o8_3, w * o8_4, w * o8_5, w * o9_0, w * o9_1, w * o9_2, w * o9_3, w * o9_4, w * o9_5, 0.0, 0.0};
      const double z = sqb::warp_sum_scatter<32>(v); const int x = lane + 0;
      if (lane < 30 && z != 0.0) atomicAdd(a.b.J + (fP + 5 + x / 6) * N + fQ + x % 6, z); }
  }
  sqb::count_add(a.counters + 0, ok && cd == 0 && false ? 1ull : 0ull);
  sqb::count_add(a.counters + 1, npq);
  sqb::count_add(a.counters + 2, nfl);
}
