// generated by gen_grad_kernels.py -- do not edit
#include "../grad_common.cuh"

static __constant__ unsigned char kCd_grad_DS_PS[3] = {0, 1, 2};
static __constant__ unsigned char kOrb_grad_DS_PS[3] = {0, 0, 0};
static __constant__ unsigned char kPerm_grad_DS_PS[3] = {36, 33, 18};
extern "C" __global__ void __launch_bounds__(64, 1)
grad_DS_PS(const sqb::GradArgs a, const sqb::WorkItem* __restrict__ items) {
  extern __shared__ double sb[];                // [chunk][44] bra primitive records
  const sqb::WorkItem it = items[blockIdx.x];
  const sqb::GradPair bp = a.bra_pairs[it.bra];
  const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;
  const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;
  const int gj = grp / si, gi = grp - gj * si;
  const int cd = kCd_grad_DS_PS[blockIdx.y], c = cd / 1, d = cd - c * 1;
  const int orbit = kOrb_grad_DS_PS[blockIdx.y], pi = kPerm_grad_DS_PS[blockIdx.y];
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
  const int fa0 = bp.fP + p0;
  const int fa1 = bp.fP + p1;
  const int fa2 = bp.fP + p2;
  const int fa3 = bp.fP + 2 + p0 + p1;
  const int fa4 = bp.fP + 2 + p0 + p2;
  const int fa5 = bp.fP + 2 + p1 + p2;
  const int fb0 = bp.fQ + 0;
  double g0 = 0.0;
  double g1 = 0.0;
  double g2 = 0.0;
  double g3 = 0.0;
  double g4 = 0.0;
  double g5 = 0.0;
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
    const double ta4c = PT[fa4 * N + fc], sa4c = PS[fa4 * N + fc];
    const double ta4d = PT[fa4 * N + fd], sa4d = PS[fa4 * N + fd];
    const double ta5c = PT[fa5 * N + fc], sa5c = PS[fa5 * N + fc];
    const double ta5d = PT[fa5 * N + fd], sa5d = PS[fa5 * N + fd];
    const double tb0c = PT[fb0 * N + fc], sb0c = PS[fb0 * N + fc];
    const double tb0d = PT[fb0 * N + fd], sb0d = PS[fb0 * N + fd];
    g0 = deg * (ptk * PT[fa0 * N + fb0] - (ta0c * tb0d + ta0d * tb0c + sa0c * sb0d + sa0d * sb0c));
    gmax = fmax(gmax, fabs(g0)); gsum += g0;
    g1 = deg * (ptk * PT[fa1 * N + fb0] - (ta1c * tb0d + ta1d * tb0c + sa1c * sb0d + sa1d * sb0c));
    gmax = fmax(gmax, fabs(g1)); gsum += g1;
    g2 = deg * (ptk * PT[fa2 * N + fb0] - (ta2c * tb0d + ta2d * tb0c + sa2c * sb0d + sa2d * sb0c));
    gmax = fmax(gmax, fabs(g2)); gsum += g2;
    g3 = deg * (ptk * PT[fa3 * N + fb0] - (ta3c * tb0d + ta3d * tb0c + sa3c * sb0d + sa3d * sb0c));
    gmax = fmax(gmax, fabs(g3)); gsum += g3;
    g4 = deg * (ptk * PT[fa4 * N + fb0] - (ta4c * tb0d + ta4d * tb0c + sa4c * sb0d + sa4d * sb0c));
    gmax = fmax(gmax, fabs(g4)); gsum += g4;
    g5 = deg * (ptk * PT[fa5 * N + fb0] - (ta5c * tb0d + ta5d * tb0c + sa5c * sb0d + sa5d * sb0c));
    gmax = fmax(gmax, fabs(g5)); gsum += g5;
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
      const double* __restrict__ src = a.bra_prims + bp.poff + (long long)(i0 + i) * 22 * bp.kstride;
      const int S = bp.kstride;
      double* __restrict__ dst = sb + i * 44;
      const double p = src[0], h = 0.5 / p, ra = src[5 * S], rb = 1.0 - ra, xa = src[(6 + ax) * S], xb = src[(9 + ax) * S];
      dst[1 + ax] = src[(1 + ax) * S];
      dst[6 + ax] = src[(12 + ax) * S];
      if (ax == 0) {
        dst[0] = p; dst[4] = src[4 * S]; dst[5] = ra;
        double wa = 0.0, wb = 0.0;
        for (int f = 0; f < 6; ++f) { const double w = src[(15 + f) * S]; dst[9 + f] = w; wa = fmax(wa, fabs(w)); }
        for (int f = 0; f < 1; ++f) { const double w = src[(21 + f) * S]; dst[15 + f] = w; wb = fmax(wb, fabs(w)); }
        dst[43] = wa * wb;
      }
      const double E10_0 = xa;
      const double E10_1 = h;
      const double E20_0 = fma(1.0, E10_1, xa * E10_0);
      const double E20_1 = fma(h, E10_0, xa * E10_1);
      const double E20_2 = h * E10_1;
      double* __restrict__ te = dst + 16 + ax * 6;
      te[0] = 1.0;
      te[1] = E10_0;
      te[2] = E10_1;
      te[3] = E20_0;
      te[4] = E20_1;
      te[5] = E20_2;
      double* __restrict__ tde = dst + 34 + ax * 3;
      const double D10_0 = -rb;
      tde[0] = D10_0;
      const double D20_0 = -rb * E10_0 * 2.0;
      const double D20_1 = -rb * E10_1 * 2.0;
      tde[1] = D20_0;
      tde[2] = D20_1;
    }
    __syncthreads();
    if (ok) {
      switch (orbit) {
      case 0: {  // ket functions like (1, 0, 0) (0, 0, 0)
        for (int i = (gi + si - i0 % si) % si; i < ni; i += si) {   // bra primitives gi, gi + si, ...
          const double* __restrict__ br = sb + i * 44;
          const double p = br[0], P0 = br[1 + p0], P1 = br[1 + p1], P2 = br[1 + p2], kpb = br[4], wmax = br[43];
          const double* __restrict__ e0 = br + 16 + p0 * 6;
          const double* __restrict__ d0 = br + 34 + p0 * 3;
          const double* __restrict__ e1 = br + 16 + p1 * 6;
          const double* __restrict__ d1 = br + 34 + p1 * 3;
          const double* __restrict__ e2 = br + 16 + p2 * 6;
          const double* __restrict__ d2 = br + 34 + p2 * 3;
          for (int j = gj; j < nkp; j += sj) {
            const double* __restrict__ kj = kprim + (long long)j * 19 * kS;
            const double q = kj[0];
            const double pq = p + q, rs = rsqrt(pq);
            const double pre = TWO_PI_2_5 * kpb * kj[4 * kS] * rs;
            if (pre < PRIM_CUTOFF) continue;
            const double s = pre * (kj[(15 + c) * kS] * kj[(18 + d) * kS]);
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
              const double wa4 = br[9 + fa4 - bp.fP];
              const double wa5 = br[9 + fa5 - bp.fP];
              const double wb0 = s * br[15 + fb0 - bp.fQ];
              { double G = g0 * (wa0 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G, e0[3], U000);
                U100 = fma(G, e0[4], U100);
                U200 = fma(G, e0[5], U200);
                V0_000 = fma(G, d0[1], V0_000);
                V0_100 = fma(G, d0[2], V0_100);
              }
              { double G = g1 * (wa1 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G, e1[3], U000);
                U010 = fma(G, e1[4], U010);
                U020 = fma(G, e1[5], U020);
                V1_000 = fma(G, d1[1], V1_000);
                V1_010 = fma(G, d1[2], V1_010);
              }
              { double G = g2 * (wa2 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G, e2[3], U000);
                U001 = fma(G, e2[4], U001);
                U002 = fma(G, e2[5], U002);
                V2_000 = fma(G, d2[1], V2_000);
                V2_001 = fma(G, d2[2], V2_001);
              }
              { double G = g3 * (wa3 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G * e0[1], e1[1], U000);
                U010 = fma(G * e0[1], e1[2], U010);
                U100 = fma(G * e0[2], e1[1], U100);
                U110 = fma(G * e0[2], e1[2], U110);
                V0_000 = fma(G * d0[0], e1[1], V0_000);
                V0_010 = fma(G * d0[0], e1[2], V0_010);
                V1_000 = fma(G * e0[1], d1[0], V1_000);
                V1_100 = fma(G * e0[2], d1[0], V1_100);
              }
              { double G = g4 * (wa4 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G * e0[1], e2[1], U000);
                U001 = fma(G * e0[1], e2[2], U001);
                U100 = fma(G * e0[2], e2[1], U100);
                U101 = fma(G * e0[2], e2[2], U101);
                V0_000 = fma(G * d0[0], e2[1], V0_000);
                V0_001 = fma(G * d0[0], e2[2], V0_001);
                V2_000 = fma(G * e0[1], d2[0], V2_000);
                V2_100 = fma(G * e0[2], d2[0], V2_100);
              }
              { double G = g5 * (wa5 * wb0); G = fabs(G) < th ? 0.0 : G;
                U000 = fma(G * e1[1], e2[1], U000);
                U001 = fma(G * e1[1], e2[2], U001);
                U010 = fma(G * e1[2], e2[1], U010);
                U011 = fma(G * e1[2], e2[2], U011);
                V1_000 = fma(G * d1[0], e2[1], V1_000);
                V1_001 = fma(G * d1[0], e2[2], V1_001);
                V2_000 = fma(G * e1[1], d2[0], V2_000);
                V2_010 = fma(G * e1[2], d2[0], V2_010);
              }
            }
            const double alpha = p * q * (rs * rs);
            const double X = P0 - kj[(1 + p0) * kS];
            const double Y = P1 - kj[(1 + p1) * kS];
            const double Z = P2 - kj[(1 + p2) * kS];
            double F[5];
            sqb::boys<4>(alpha * fma(X, X, fma(Y, Y, Z * Z)), a.boys_tab, F);
            const double m2a = -2.0 * alpha;
            const double b0 = F[0];
            double w = m2a;
            const double b1 = w * F[1];
            w *= m2a;
            const double b2 = w * F[2];
            w *= m2a;
            const double b3 = w * F[3];
            w *= m2a;
            const double b4 = w * F[4];
            const double rc = kj[5 * kS], rd = 1.0 - rc, hq = 0.5 / q;
            const double xc0 = kj[(6 + p0) * kS], xd0 = kj[(9 + p0) * kS];
            const double k0_10_0 = xc0;
            const double k0_10_1 = hq;
            const double kd0_10_0 = -rd;
            const double ke000 = k0_10_0;
            const double ke100 = -k0_10_1;
            const double kd0000 = kd0_10_0;
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
            double W0_000 = 0.0;
            double W0_100 = 0.0;
            double W0_010 = 0.0;
            double W0_001 = 0.0;
            double W0_200 = 0.0;
            double W0_110 = 0.0;
            double W0_101 = 0.0;
            double W0_020 = 0.0;
            double W0_011 = 0.0;
            double W0_002 = 0.0;
            Y000 = fma(ke000, b0, Y000);
            W0_000 = fma(kd0000, b0, W0_000);
            const double r0_0_0_1 = Z * b1;
            Y001 = fma(ke000, r0_0_0_1, Y001);
            W0_001 = fma(kd0000, r0_0_0_1, W0_001);
            const double r0_0_1_0 = Y * b1;
            Y010 = fma(ke000, r0_0_1_0, Y010);
            W0_010 = fma(kd0000, r0_0_1_0, W0_010);
            const double r0_1_0_0 = X * b1;
            Y100 = fma(ke000, r0_1_0_0, Y100);
            Y000 = fma(ke100, r0_1_0_0, Y000);
            W0_100 = fma(kd0000, r0_1_0_0, W0_100);
            const double r1_0_0_1 = Z * b2;
            const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
            Y002 = fma(ke000, r0_0_0_2, Y002);
            W0_002 = fma(kd0000, r0_0_0_2, W0_002);
            const double r0_0_1_1 = Y * r1_0_0_1;
            Y011 = fma(ke000, r0_0_1_1, Y011);
            W0_011 = fma(kd0000, r0_0_1_1, W0_011);
            const double r1_0_1_0 = Y * b2;
            const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
            Y020 = fma(ke000, r0_0_2_0, Y020);
            W0_020 = fma(kd0000, r0_0_2_0, W0_020);
            const double r0_1_0_1 = X * r1_0_0_1;
            Y101 = fma(ke000, r0_1_0_1, Y101);
            Y001 = fma(ke100, r0_1_0_1, Y001);
            W0_101 = fma(kd0000, r0_1_0_1, W0_101);
            const double r0_1_1_0 = X * r1_0_1_0;
            Y110 = fma(ke000, r0_1_1_0, Y110);
            Y010 = fma(ke100, r0_1_1_0, Y010);
            W0_110 = fma(kd0000, r0_1_1_0, W0_110);
            const double r1_1_0_0 = X * b2;
            const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
            Y200 = fma(ke000, r0_2_0_0, Y200);
            Y100 = fma(ke100, r0_2_0_0, Y100);
            W0_200 = fma(kd0000, r0_2_0_0, W0_200);
            const double r2_0_0_1 = Z * b3;
            const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
            const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
            Y003 = fma(ke000, r0_0_0_3, Y003);
            const double r0_0_1_2 = Y * r1_0_0_2;
            Y012 = fma(ke000, r0_0_1_2, Y012);
            const double r1_0_1_1 = Y * r2_0_0_1;
            const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
            Y021 = fma(ke000, r0_0_2_1, Y021);
            const double r2_0_1_0 = Y * b3;
            const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
            const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
            Y030 = fma(ke000, r0_0_3_0, Y030);
            const double r0_1_0_2 = X * r1_0_0_2;
            Y102 = fma(ke000, r0_1_0_2, Y102);
            Y002 = fma(ke100, r0_1_0_2, Y002);
            const double r0_1_1_1 = X * r1_0_1_1;
            Y111 = fma(ke000, r0_1_1_1, Y111);
            Y011 = fma(ke100, r0_1_1_1, Y011);
            const double r0_1_2_0 = X * r1_0_2_0;
            Y120 = fma(ke000, r0_1_2_0, Y120);
            Y020 = fma(ke100, r0_1_2_0, Y020);
            const double r1_1_0_1 = X * r2_0_0_1;
            const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
            Y201 = fma(ke000, r0_2_0_1, Y201);
            Y101 = fma(ke100, r0_2_0_1, Y101);
            const double r1_1_1_0 = X * r2_0_1_0;
            const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
            Y210 = fma(ke000, r0_2_1_0, Y210);
            Y110 = fma(ke100, r0_2_1_0, Y110);
            const double r2_1_0_0 = X * b3;
            const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
            const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
            Y300 = fma(ke000, r0_3_0_0, Y300);
            Y200 = fma(ke100, r0_3_0_0, Y200);
            const double r3_0_0_1 = Z * b4;
            const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
            const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
            const double r0_1_0_3 = X * r1_0_0_3;
            Y003 = fma(ke100, r0_1_0_3, Y003);
            const double r1_0_1_2 = Y * r2_0_0_2;
            const double r0_1_1_2 = X * r1_0_1_2;
            Y012 = fma(ke100, r0_1_1_2, Y012);
            const double r2_0_1_1 = Y * r3_0_0_1;
            const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
            const double r0_1_2_1 = X * r1_0_2_1;
            Y021 = fma(ke100, r0_1_2_1, Y021);
            const double r3_0_1_0 = Y * b4;
            const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
            const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
            const double r0_1_3_0 = X * r1_0_3_0;
            Y030 = fma(ke100, r0_1_3_0, Y030);
            const double r1_1_0_2 = X * r2_0_0_2;
            const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
            Y102 = fma(ke100, r0_2_0_2, Y102);
            const double r1_1_1_1 = X * r2_0_1_1;
            const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
            Y111 = fma(ke100, r0_2_1_1, Y111);
            const double r1_1_2_0 = X * r2_0_2_0;
            const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
            Y120 = fma(ke100, r0_2_2_0, Y120);
            const double r2_1_0_1 = X * r3_0_0_1;
            const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
            const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
            Y201 = fma(ke100, r0_3_0_1, Y201);
            const double r2_1_1_0 = X * r3_0_1_0;
            const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
            const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
            Y210 = fma(ke100, r0_3_1_0, Y210);
            const double r3_1_0_0 = X * b4;
            const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
            const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
            const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
            Y300 = fma(ke100, r0_4_0_0, Y300);
            const double e = fma(U000, Y000, fma(U100, Y100, fma(U010, Y010, fma(U001, Y001, fma(U200, Y200, fma(U110, Y110, fma(U101, Y101, fma(U020, Y020, fma(U011, Y011, U002 * Y002)))))))));
            const double ra = br[5], rb = 1.0 - ra;
            {
              const double fp = fma(U000, Y100, fma(U100, Y200, fma(U010, Y110, fma(U001, Y101, fma(U200, Y300, fma(U110, Y210, fma(U101, Y201, fma(U020, Y120, fma(U011, Y111, U002 * Y102)))))))));
              const double fab = fma(-br[6 + p0], e, fma(V0_000, Y000, fma(V0_100, Y100, fma(V0_010, Y010, V0_001 * Y001))));
              const double fcd = fma(-kj[(12 + p0) * kS], e, fma(U000, W0_000, fma(U100, W0_100, fma(U010, W0_010, fma(U001, W0_001, fma(U200, W0_200, fma(U110, W0_110, fma(U101, W0_101, fma(U020, W0_020, fma(U011, W0_011, U002 * W0_002))))))))));
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
