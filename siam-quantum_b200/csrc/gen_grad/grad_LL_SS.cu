// generated by gen_grad_kernels.py -- do not edit
#include "../grad_common.cuh"

static __constant__ unsigned char kCd_grad_LL_SS[1] = {0};
static __constant__ unsigned char kOrb_grad_LL_SS[1] = {0};
static __constant__ unsigned char kPerm_grad_LL_SS[1] = {36};
extern "C" __global__ void __launch_bounds__(64, 1)
grad_LL_SS(const sqb::GradArgs a, const sqb::WorkItem* __restrict__ items) {
  extern __shared__ double sb[];                // [chunk][54] bra primitive records
  const sqb::WorkItem it = items[blockIdx.x];
  const sqb::GradPair bp = a.bra_pairs[it.bra];
  const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;
  const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;
  const int gj = grp / si, gi = grp - gj * si;
  const int cd = kCd_grad_LL_SS[blockIdx.y], c = cd / 1, d = cd - c * 1;
  const int orbit = kOrb_grad_LL_SS[blockIdx.y], pi = kPerm_grad_LL_SS[blockIdx.y];
  const int p0 = pi & 3, p1 = (pi >> 2) & 3, p2 = pi >> 4;   // axis r of this pass = molecule axis p<r>
  const bool have = kl < it.cnt;
  const sqb::GradPair kp = a.ket_pairs[it.k0 + min(kl, it.cnt - 1)];
  const double screen = a.screen;
  const bool ok = have && !(bp.sch * kp.sch * bp.pm * kp.pm < screen);
  if (!__syncthreads_or(ok)) return;
  const int N = a.nbf, nbp = bp.nprim, nkp = kp.nprim;
  const bool same_b = bp.P == bp.Q, same_k = kp.P == kp.Q, same_pair = a.same_class && it.bra == it.k0 + kl;
  const double deg = (same_b ? 0.5 : 1.0) * (same_k ? 0.5 : 1.0) * (same_pair ? 0.5 : 1.0);
  const double* __restrict__ PT = a.PT;
  const double* __restrict__ PS = a.PS;
  const int fc = kp.fP + c, fd = kp.fQ + d;
  const int fa0 = bp.fP + 0;
  const int fa1 = bp.fP + 1 + p0;
  const int fa2 = bp.fP + 1 + p1;
  const int fa3 = bp.fP + 1 + p2;
  const int fb0 = bp.fQ + 0;
  const int fb1 = bp.fQ + 1 + p0;
  const int fb2 = bp.fQ + 1 + p1;
  const int fb3 = bp.fQ + 1 + p2;
  double g0 = 0.0;
  double g1 = 0.0;
  double g2 = 0.0;
  double g3 = 0.0;
  double g4 = 0.0;
  double g5 = 0.0;
  double g6 = 0.0;
  double g7 = 0.0;
  double g8 = 0.0;
  double g9 = 0.0;
  double g10 = 0.0;
  double g11 = 0.0;
  double g12 = 0.0;
  double g13 = 0.0;
  double g14 = 0.0;
  double g15 = 0.0;
  double gmax = 0.0, gsum = 0.0;
  if (ok) {
    const double ptk = 4.0 * PT[fc * N + fd];
    const double ta0c = PT[fa0 * N + fc], sa0c = PS[fa0 * N + fc];
    const double ta0d = PT[fa0 * N + fd], sa0d = PS[fa0 * N + fd];
    const double ta1c = PT[fa1 * N + fc], sa1c = PS[fa1 * N + fc];
    const double ta1d = PT[fa1 * N + fd], sa1d = PS[fa1 * N + fd];
    const double ta2c = PT[fa2 * N + fc], sa2c = PS[fa2 * N + fc];
    const double ta2d = PT[fa2 * N + fd], sa2d = PS[fa2 * N + fd];
    const double ta3c = PT[fa3 * N + fc], sa3c = PS[fa3 * N + fc];
    const double ta3d = PT[fa3 * N + fd], sa3d = PS[fa3 * N + fd];
    const double tb0c = PT[fb0 * N + fc], sb0c = PS[fb0 * N + fc];
    const double tb0d = PT[fb0 * N + fd], sb0d = PS[fb0 * N + fd];
    const double tb1c = PT[fb1 * N + fc], sb1c = PS[fb1 * N + fc];
    const double tb1d = PT[fb1 * N + fd], sb1d = PS[fb1 * N + fd];
    const double tb2c = PT[fb2 * N + fc], sb2c = PS[fb2 * N + fc];
    const double tb2d = PT[fb2 * N + fd], sb2d = PS[fb2 * N + fd];
    const double tb3c = PT[fb3 * N + fc], sb3c = PS[fb3 * N + fc];
    const double tb3d = PT[fb3 * N + fd], sb3d = PS[fb3 * N + fd];
    g0 = deg * (ptk * PT[fa0 * N + fb0] - (ta0c * tb0d + ta0d * tb0c + sa0c * sb0d + sa0d * sb0c));
    gmax = fmax(gmax, fabs(g0)); gsum += g0;
    g1 = deg * (ptk * PT[fa0 * N + fb1] - (ta0c * tb1d + ta0d * tb1c + sa0c * sb1d + sa0d * sb1c));
    gmax = fmax(gmax, fabs(g1)); gsum += g1;
    g2 = deg * (ptk * PT[fa0 * N + fb2] - (ta0c * tb2d + ta0d * tb2c + sa0c * sb2d + sa0d * sb2c));
    gmax = fmax(gmax, fabs(g2)); gsum += g2;
    g3 = deg * (ptk * PT[fa0 * N + fb3] - (ta0c * tb3d + ta0d * tb3c + sa0c * sb3d + sa0d * sb3c));
    gmax = fmax(gmax, fabs(g3)); gsum += g3;
    g4 = deg * (ptk * PT[fa1 * N + fb0] - (ta1c * tb0d + ta1d * tb0c + sa1c * sb0d + sa1d * sb0c));
    gmax = fmax(gmax, fabs(g4)); gsum += g4;
    g5 = deg * (ptk * PT[fa1 * N + fb1] - (ta1c * tb1d + ta1d * tb1c + sa1c * sb1d + sa1d * sb1c));
    gmax = fmax(gmax, fabs(g5)); gsum += g5;
    g6 = deg * (ptk * PT[fa1 * N + fb2] - (ta1c * tb2d + ta1d * tb2c + sa1c * sb2d + sa1d * sb2c));
    gmax = fmax(gmax, fabs(g6)); gsum += g6;
    g7 = deg * (ptk * PT[fa1 * N + fb3] - (ta1c * tb3d + ta1d * tb3c + sa1c * sb3d + sa1d * sb3c));
    gmax = fmax(gmax, fabs(g7)); gsum += g7;
    g8 = deg * (ptk * PT[fa2 * N + fb0] - (ta2c * tb0d + ta2d * tb0c + sa2c * sb0d + sa2d * sb0c));
    gmax = fmax(gmax, fabs(g8)); gsum += g8;
    g9 = deg * (ptk * PT[fa2 * N + fb1] - (ta2c * tb1d + ta2d * tb1c + sa2c * sb1d + sa2d * sb1c));
    gmax = fmax(gmax, fabs(g9)); gsum += g9;
    g10 = deg * (ptk * PT[fa2 * N + fb2] - (ta2c * tb2d + ta2d * tb2c + sa2c * sb2d + sa2d * sb2c));
    gmax = fmax(gmax, fabs(g10)); gsum += g10;
    g11 = deg * (ptk * PT[fa2 * N + fb3] - (ta2c * tb3d + ta2d * tb3c + sa2c * sb3d + sa2d * sb3c));
    gmax = fmax(gmax, fabs(g11)); gsum += g11;
    g12 = deg * (ptk * PT[fa3 * N + fb0] - (ta3c * tb0d + ta3d * tb0c + sa3c * sb0d + sa3d * sb0c));
    gmax = fmax(gmax, fabs(g12)); gsum += g12;
    g13 = deg * (ptk * PT[fa3 * N + fb1] - (ta3c * tb1d + ta3d * tb1c + sa3c * sb1d + sa3d * sb1c));
    gmax = fmax(gmax, fabs(g13)); gsum += g13;
    g14 = deg * (ptk * PT[fa3 * N + fb2] - (ta3c * tb2d + ta3d * tb2c + sa3c * sb2d + sa3d * sb2c));
    gmax = fmax(gmax, fabs(g14)); gsum += g14;
    g15 = deg * (ptk * PT[fa3 * N + fb3] - (ta3c * tb3d + ta3d * tb3c + sa3c * sb3d + sa3d * sb3c));
    gmax = fmax(gmax, fabs(g15)); gsum += g15;
    if (!(gsum - gsum == 0.0)) gmax = fabs(gsum); // fmax drops a NaN: a density that is not finite skips nothing
  }
  const double th = screen * (same_k && fc != fd ? 0.5 : 1.0), tho = same_b ? 0.5 * th : th;
  const double hp = same_pair ? 0.5 : 1.0;    // function pairs of one shell pair that differ
  const double thmin = screen * deg * (1.0 - 1e-12);
  double A0 = 0.0, A1 = 0.0, A2 = 0.0, B0 = 0.0, B1 = 0.0, B2 = 0.0, C0 = 0.0, C1 = 0.0, C2 = 0.0;
  const double* __restrict__ kprim = a.ket_prims + kp.poff;
  const int kS = kp.kstride;
  for (int i0 = 0; i0 < nbp; i0 += a.chunk) {
    const int ni = min(a.chunk, nbp - i0);
    __syncthreads();                              // the previous chunk's readers are done
    for (int x = threadIdx.x; x < 3 * ni; x += 64) {   // 1-D tables: one (primitive, axis) per thread
      const int i = x / 3, ax = x - 3 * i;
      const double* __restrict__ src = a.bra_prims + bp.poff + (long long)(i0 + i) * 23 * bp.kstride;
      const int S = bp.kstride;
      double* __restrict__ dst = sb + i * 54;
      const double p = src[0], h = 0.5 / p, ra = src[5 * S], rb = 1.0 - ra, xa = src[(6 + ax) * S], xb = src[(9 + ax) * S];
      dst[1 + ax] = src[(1 + ax) * S];
      dst[6 + ax] = src[(12 + ax) * S];
      if (ax == 0) {
        dst[0] = p; dst[4] = src[4 * S]; dst[5] = ra;
        double wa = 0.0, wb = 0.0;
        for (int f = 0; f < 4; ++f) { const double w = src[(15 + f) * S]; dst[9 + f] = w; wa = fmax(wa, fabs(w)); }
        for (int f = 0; f < 4; ++f) { const double w = src[(19 + f) * S]; dst[13 + f] = w; wb = fmax(wb, fabs(w)); }
        dst[53] = wa * wb;
      }
      const double E01_0 = xb;
      const double E01_1 = h;
      const double E10_0 = xa;
      const double E10_1 = h;
      const double E11_0 = fma(1.0, E01_1, xa * E01_0);
      const double E11_1 = fma(h, E01_0, xa * E01_1);
      const double E11_2 = h * E01_1;
      double* __restrict__ te = dst + 17 + ax * 8;
      te[0] = 1.0;
      te[1] = E01_0;
      te[2] = E01_1;
      te[3] = E10_0;
      te[4] = E10_1;
      te[5] = E11_0;
      te[6] = E11_1;
      te[7] = E11_2;
      double* __restrict__ tde = dst + 41 + ax * 4;
      const double D01_0 = ra;
      tde[0] = D01_0;
      const double D10_0 = -rb;
      tde[1] = D10_0;
      const double D11_0 = -rb * E01_0 + ra * E10_0;
      const double D11_1 = -rb * E01_1 + ra * E10_1;
      tde[2] = D11_0;
      tde[3] = D11_1;
    }
    __syncthreads();
    if (ok) {
      switch (orbit) {
      case 0: {  // ket functions like (0, 0, 0) (0, 0, 0)
        for (int i = (gi + si - i0 % si) % si; i < ni; i += si) {   // bra primitives gi, gi + si, ...
          const double* __restrict__ br = sb + i * 54;
          const double p = br[0], P0 = br[1 + p0], P1 = br[1 + p1], P2 = br[1 + p2], kpb = br[4], wmax = br[53];
          const double* __restrict__ e0 = br + 17 + p0 * 8;
          const double* __restrict__ d0 = br + 41 + p0 * 4;
          const double* __restrict__ e1 = br + 17 + p1 * 8;
          const double* __restrict__ d1 = br + 41 + p1 * 4;
          const double* __restrict__ e2 = br + 17 + p2 * 8;
          const double* __restrict__ d2 = br + 41 + p2 * 4;
          for (int j = gj; j < nkp; j += sj) {
            const double* __restrict__ kj = kprim + (long long)j * 17 * kS;
            const double q = kj[0];
            const double pq = p + q, rs = rsqrt(pq);
            const double pre = TWO_PI_2_5 * kpb * kj[4 * kS] * rs;
            if (pre < PRIM_CUTOFF) continue;
            const double s = pre * (kj[(15 + c) * kS] * kj[(16 + d) * kS]);
            if (gmax * fabs(s) * wmax < thmin) continue;   // every function quartet is below the screen
            double U000 = 0.0;
            double U100 = 0.0;
            double U010 = 0.0;
            double U001 = 0.0;
            double U200 = 0.0;
            double U110 = 0.0;
            double U101 = 0.0;
            double U020 = 0.0;
            double U011 = 0.0;
            double U002 = 0.0;
            double V0_000 = 0.0;
            double V0_100 = 0.0;
            double V0_010 = 0.0;
            double V0_001 = 0.0;
            double V1_000 = 0.0;
            double V1_100 = 0.0;
            double V1_010 = 0.0;
            double V1_001 = 0.0;
            double V2_000 = 0.0;
            double V2_100 = 0.0;
            double V2_010 = 0.0;
            double V2_001 = 0.0;
            {
              const double wa0 = br[9 + fa0 - bp.fP];
              const double wa1 = br[9 + fa1 - bp.fP];
              const double wa2 = br[9 + fa2 - bp.fP];
              const double wa3 = br[9 + fa3 - bp.fP];
              const double wb0 = s * br[13 + fb0 - bp.fQ];
              const double wb1 = s * br[13 + fb1 - bp.fQ];
              const double wb2 = s * br[13 + fb2 - bp.fQ];
              const double wb3 = s * br[13 + fb3 - bp.fQ];
              { double G = g0 * (wa0 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 += G;
              }
              { double G = g1 * (wa0 * wb1); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G, e0[1], U000);
                U100 = fma(G, e0[2], U100);
                V0_000 = fma(G, d0[0], V0_000);
              }
              { double G = g2 * (wa0 * wb2); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G, e1[1], U000);
                U010 = fma(G, e1[2], U010);
                V1_000 = fma(G, d1[0], V1_000);
              }
              { double G = g3 * (wa0 * wb3); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G, e2[1], U000);
                U001 = fma(G, e2[2], U001);
                V2_000 = fma(G, d2[0], V2_000);
              }
              { double G = g4 * (wa1 * wb0); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G, e0[3], U000);
                U100 = fma(G, e0[4], U100);
                V0_000 = fma(G, d0[1], V0_000);
              }
              { double G = g5 * (wa1 * wb1); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G, e0[5], U000);
                U100 = fma(G, e0[6], U100);
                U200 = fma(G, e0[7], U200);
                V0_000 = fma(G, d0[2], V0_000);
                V0_100 = fma(G, d0[3], V0_100);
              }
              { double G = g6 * (wa1 * wb2); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G * e0[3], e1[1], U000);
                U010 = fma(G * e0[3], e1[2], U010);
                U100 = fma(G * e0[4], e1[1], U100);
                U110 = fma(G * e0[4], e1[2], U110);
                V0_000 = fma(G * d0[1], e1[1], V0_000);
                V0_010 = fma(G * d0[1], e1[2], V0_010);
                V1_000 = fma(G * e0[3], d1[0], V1_000);
                V1_100 = fma(G * e0[4], d1[0], V1_100);
              }
              { double G = g7 * (wa1 * wb3); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G * e0[3], e2[1], U000);
                U001 = fma(G * e0[3], e2[2], U001);
                U100 = fma(G * e0[4], e2[1], U100);
                U101 = fma(G * e0[4], e2[2], U101);
                V0_000 = fma(G * d0[1], e2[1], V0_000);
                V0_001 = fma(G * d0[1], e2[2], V0_001);
                V2_000 = fma(G * e0[3], d2[0], V2_000);
                V2_100 = fma(G * e0[4], d2[0], V2_100);
              }
              { double G = g8 * (wa2 * wb0); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G, e1[3], U000);
                U010 = fma(G, e1[4], U010);
                V1_000 = fma(G, d1[1], V1_000);
              }
              { double G = g9 * (wa2 * wb1); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G * e0[1], e1[3], U000);
                U010 = fma(G * e0[1], e1[4], U010);
                U100 = fma(G * e0[2], e1[3], U100);
                U110 = fma(G * e0[2], e1[4], U110);
                V0_000 = fma(G * d0[0], e1[3], V0_000);
                V0_010 = fma(G * d0[0], e1[4], V0_010);
                V1_000 = fma(G * e0[1], d1[1], V1_000);
                V1_100 = fma(G * e0[2], d1[1], V1_100);
              }
              { double G = g10 * (wa2 * wb2); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G, e1[5], U000);
                U010 = fma(G, e1[6], U010);
                U020 = fma(G, e1[7], U020);
                V1_000 = fma(G, d1[2], V1_000);
                V1_010 = fma(G, d1[3], V1_010);
              }
              { double G = g11 * (wa2 * wb3); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G * e1[3], e2[1], U000);
                U001 = fma(G * e1[3], e2[2], U001);
                U010 = fma(G * e1[4], e2[1], U010);
                U011 = fma(G * e1[4], e2[2], U011);
                V1_000 = fma(G * d1[1], e2[1], V1_000);
                V1_001 = fma(G * d1[1], e2[2], V1_001);
                V2_000 = fma(G * e1[3], d2[0], V2_000);
                V2_010 = fma(G * e1[4], d2[0], V2_010);
              }
              { double G = g12 * (wa3 * wb0); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G, e2[3], U000);
                U001 = fma(G, e2[4], U001);
                V2_000 = fma(G, d2[1], V2_000);
              }
              { double G = g13 * (wa3 * wb1); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G * e0[1], e2[3], U000);
                U001 = fma(G * e0[1], e2[4], U001);
                U100 = fma(G * e0[2], e2[3], U100);
                U101 = fma(G * e0[2], e2[4], U101);
                V0_000 = fma(G * d0[0], e2[3], V0_000);
                V0_001 = fma(G * d0[0], e2[4], V0_001);
                V2_000 = fma(G * e0[1], d2[1], V2_000);
                V2_100 = fma(G * e0[2], d2[1], V2_100);
              }
              { double G = g14 * (wa3 * wb2); G = fabs(G) < tho ? 0.0 : G;
                U000 = fma(G * e1[1], e2[3], U000);
                U001 = fma(G * e1[1], e2[4], U001);
                U010 = fma(G * e1[2], e2[3], U010);
                U011 = fma(G * e1[2], e2[4], U011);
                V1_000 = fma(G * d1[0], e2[3], V1_000);
                V1_001 = fma(G * d1[0], e2[4], V1_001);
                V2_000 = fma(G * e1[1], d2[1], V2_000);
                V2_010 = fma(G * e1[2], d2[1], V2_010);
              }
              { double G = g15 * (wa3 * wb3); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G, e2[5], U000);
                U001 = fma(G, e2[6], U001);
                U002 = fma(G, e2[7], U002);
                V2_000 = fma(G, d2[2], V2_000);
                V2_001 = fma(G, d2[3], V2_001);
              }
            }
            const double alpha = p * q * (rs * rs);
            const double X = P0 - kj[(1 + p0) * kS];
            const double Y = P1 - kj[(1 + p1) * kS];
            const double Z = P2 - kj[(1 + p2) * kS];
            double F[4];
            sqb::boys<3>(alpha * fma(X, X, fma(Y, Y, Z * Z)), a.boys_tab, F);
            const double m2a = -2.0 * alpha;
            const double b0 = F[0];
            double w = m2a;
            const double b1 = w * F[1];
            w *= m2a;
            const double b2 = w * F[2];
            w *= m2a;
            const double b3 = w * F[3];
            const double rc = kj[5 * kS], rd = 1.0 - rc;
            const double ke000 = 1.0;
            double Y000 = 0.0;
            double Y100 = 0.0;
            double Y010 = 0.0;
            double Y001 = 0.0;
            double Y200 = 0.0;
            double Y110 = 0.0;
            double Y101 = 0.0;
            double Y020 = 0.0;
            double Y011 = 0.0;
            double Y002 = 0.0;
            double Y300 = 0.0;
            double Y210 = 0.0;
            double Y201 = 0.0;
            double Y120 = 0.0;
            double Y111 = 0.0;
            double Y102 = 0.0;
            double Y030 = 0.0;
            double Y021 = 0.0;
            double Y012 = 0.0;
            double Y003 = 0.0;
            Y000 += b0;
            const double r0_0_0_1 = Z * b1;
            Y001 += r0_0_0_1;
            const double r0_0_1_0 = Y * b1;
            Y010 += r0_0_1_0;
            const double r0_1_0_0 = X * b1;
            Y100 += r0_1_0_0;
            const double r1_0_0_1 = Z * b2;
            const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
            Y002 += r0_0_0_2;
            const double r0_0_1_1 = Y * r1_0_0_1;
            Y011 += r0_0_1_1;
            const double r1_0_1_0 = Y * b2;
            const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
            Y020 += r0_0_2_0;
            const double r0_1_0_1 = X * r1_0_0_1;
            Y101 += r0_1_0_1;
            const double r0_1_1_0 = X * r1_0_1_0;
            Y110 += r0_1_1_0;
            const double r1_1_0_0 = X * b2;
            const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
            Y200 += r0_2_0_0;
            const double r2_0_0_1 = Z * b3;
            const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
            const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
            Y003 += r0_0_0_3;
            const double r0_0_1_2 = Y * r1_0_0_2;
            Y012 += r0_0_1_2;
            const double r1_0_1_1 = Y * r2_0_0_1;
            const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
            Y021 += r0_0_2_1;
            const double r2_0_1_0 = Y * b3;
            const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
            const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
            Y030 += r0_0_3_0;
            const double r0_1_0_2 = X * r1_0_0_2;
            Y102 += r0_1_0_2;
            const double r0_1_1_1 = X * r1_0_1_1;
            Y111 += r0_1_1_1;
            const double r0_1_2_0 = X * r1_0_2_0;
            Y120 += r0_1_2_0;
            const double r1_1_0_1 = X * r2_0_0_1;
            const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
            Y201 += r0_2_0_1;
            const double r1_1_1_0 = X * r2_0_1_0;
            const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
            Y210 += r0_2_1_0;
            const double r2_1_0_0 = X * b3;
            const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
            const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
            Y300 += r0_3_0_0;
            const double e = fma(U000, Y000, fma(U100, Y100, fma(U010, Y010, fma(U001, Y001, fma(U200, Y200, fma(U110, Y110, fma(U101, Y101, fma(U020, Y020, fma(U011, Y011, U002 * Y002)))))))));
            const double ra = br[5], rb = 1.0 - ra;
            {
              const double fp = fma(U000, Y100, fma(U100, Y200, fma(U010, Y110, fma(U001, Y101, fma(U200, Y300, fma(U110, Y210, fma(U101, Y201, fma(U020, Y120, fma(U011, Y111, U002 * Y102)))))))));
              const double fab = fma(-br[6 + p0], e, fma(V0_000, Y000, fma(V0_100, Y100, fma(V0_010, Y010, V0_001 * Y001))));
              const double fcd = -kj[(12 + p0) * kS] * e;
              A0 += fma(ra, fp, fab); B0 += fma(rb, fp, -fab); C0 += fma(-rc, fp, fcd);
            }
            {
              const double fp = fma(U000, Y010, fma(U100, Y110, fma(U010, Y020, fma(U001, Y011, fma(U200, Y210, fma(U110, Y120, fma(U101, Y111, fma(U020, Y030, fma(U011, Y021, U002 * Y012)))))))));
              const double fab = fma(-br[6 + p1], e, fma(V1_000, Y000, fma(V1_100, Y100, fma(V1_010, Y010, V1_001 * Y001))));
              const double fcd = -kj[(12 + p1) * kS] * e;
              A1 += fma(ra, fp, fab); B1 += fma(rb, fp, -fab); C1 += fma(-rc, fp, fcd);
            }
            {
              const double fp = fma(U000, Y001, fma(U100, Y101, fma(U010, Y011, fma(U001, Y002, fma(U200, Y201, fma(U110, Y111, fma(U101, Y102, fma(U020, Y021, fma(U011, Y012, U002 * Y003)))))))));
              const double fab = fma(-br[6 + p2], e, fma(V2_000, Y000, fma(V2_100, Y100, fma(V2_010, Y010, V2_001 * Y001))));
              const double fcd = -kj[(12 + p2) * kS] * e;
              A2 += fma(ra, fp, fab); B2 += fma(rb, fp, -fab); C2 += fma(-rc, fp, fcd);
            }
          }
        }
      } break;
      }
    }
  }
  double* __restrict__ g = a.grad + (size_t)((blockIdx.x + 5 * blockIdx.y) % a.ncopy) * a.stride;
  { const double va = sqb::warp_sum(A0), vb = sqb::warp_sum(B0);
    if ((threadIdx.x & 31) == 0) { atomicAdd(g + 3 * bp.atP + p0, va); atomicAdd(g + 3 * bp.atQ + p0, vb); } }
  { const double va = sqb::warp_sum(A1), vb = sqb::warp_sum(B1);
    if ((threadIdx.x & 31) == 0) { atomicAdd(g + 3 * bp.atP + p1, va); atomicAdd(g + 3 * bp.atQ + p1, vb); } }
  { const double va = sqb::warp_sum(A2), vb = sqb::warp_sum(B2);
    if ((threadIdx.x & 31) == 0) { atomicAdd(g + 3 * bp.atP + p2, va); atomicAdd(g + 3 * bp.atQ + p2, vb); } }
  if (ok) {
    atomicAdd(g + 3 * kp.atP + p0, C0); atomicAdd(g + 3 * kp.atQ + p0, -(A0 + B0 + C0));
    atomicAdd(g + 3 * kp.atP + p1, C1); atomicAdd(g + 3 * kp.atQ + p1, -(A1 + B1 + C1));
    atomicAdd(g + 3 * kp.atP + p2, C2); atomicAdd(g + 3 * kp.atQ + p2, -(A2 + B2 + C2));
  }
}
