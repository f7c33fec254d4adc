// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DP_PL_R_w(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
  __shared__ int q_next;
  const bool persistent = a.queue != nullptr;
  for (int round = 0;; ++round) {
    int qi_, qp_;
    if (persistent) {
      __syncthreads();                  // the previous unit is done with shared memory
      if (threadIdx.x == 0) q_next = (int)atomicAdd(a.queue, 1ull);
      __syncthreads();
      const int q = q_next;
      if (q >= a.nqueue) break;
      const int nitems = a.nqueue / a.npass;
      qp_ = q / nitems;
      qi_ = q - qp_ * nitems;
    } else {
      if (round > 0) break;
      qi_ = blockIdx.x;
      qp_ = blockIdx.y;
    }
    {
      extern __shared__ double sbra[];
      const sqb::WorkItem it = items[qi_];
      const sqb::PairRec bp = a.bra_pairs[it.bra];
      const sqb::MolRec mr = a.mols[it.mol];        // the molecule of this work item
      const long long acc0 = mr.moff + (qi_ & a.copy_mask) * a.copy_stride;   // this item's copy
      double* __restrict__ Jacc = a.Jacc + acc0;
      double* __restrict__ KAacc = a.KAacc + acc0;
      double* __restrict__ KBacc = a.KBacc + acc0;
      const int N = mr.nbf;
      for (int x = threadIdx.x; x < bp.nprim * 113; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];
      __syncthreads();
      // threads sharing one quartet: si strides over the bra primitives x sj over the ket primitives
      const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;
      const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;
      const int gj = grp / si, gi = grp - gj * si;
      const unsigned gmask = isplit >= 32 ? 0xffffffffu : ((1u << isplit) - 1u) << ((threadIdx.x & 31) & ~(isplit - 1));
      const int pass = qp_;                   // block of ket functions handled by this CTA
      bool ok = kl < it.cnt;
      sqb::PairRec kp = bp;
      double deg = 0.0;
      if (ok) {
        kp = a.ket_pairs[it.k0 + kl];
        const double r = bp.schwarz * kp.schwarz;
        ok = !(r < mr.cut_outer) && !(r < mr.cut_fixed);
        if (ok && r < mr.dscreen_rmax) {
          const bool bf = (bp.P > kp.P) || (bp.P == kp.P && bp.Q >= kp.Q);
          const int P = bf ? bp.P : kp.P, Q = bf ? bp.Q : kp.Q, I = bf ? kp.P : bp.P, J = bf ? kp.Q : bp.Q;
          const double* PM = a.PM + mr.pmoff; const int ns = mr.ns;
          const double mp = PM[P * ns + Q] + PM[I * ns + J] + PM[P * ns + I] + PM[P * ns + J] + PM[Q * ns + I] + PM[Q * ns + J];
          ok = !(r * mp < mr.cut_fixed);
        }
        deg = (bp.P == bp.Q ? 0.5 : 1.0) * (kp.P == kp.Q ? 0.5 : 1.0) * ((a.same_class && it.bra == it.k0 + kl) ? 0.5 : 1.0);
      }
      double jab0 = 0.0;
      double jab1 = 0.0;
      double jab2 = 0.0;
      double jab3 = 0.0;
      double jab4 = 0.0;
      double jab5 = 0.0;
      double jab6 = 0.0;
      double jab7 = 0.0;
      double jab8 = 0.0;
      double jab9 = 0.0;
      double jab10 = 0.0;
      double jab11 = 0.0;
      double jab12 = 0.0;
      double jab13 = 0.0;
      double jab14 = 0.0;
      double jab15 = 0.0;
      double jab16 = 0.0;
      double jab17 = 0.0;
      unsigned long long nprimq = 0, nflush = 0;
      if (ok) {
        const double* __restrict__ kprim = a.ket_prims + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // ket functions [0, 4, 8]
          double o0_0 = 0;
          double o0_4 = 0;
          double o0_8 = 0;
          double o1_0 = 0;
          double o1_4 = 0;
          double o1_8 = 0;
          double o2_0 = 0;
          double o2_4 = 0;
          double o2_8 = 0;
          double o3_0 = 0;
          double o3_4 = 0;
          double o3_8 = 0;
          double o4_0 = 0;
          double o4_4 = 0;
          double o4_8 = 0;
          double o5_0 = 0;
          double o5_4 = 0;
          double o5_8 = 0;
          double o6_0 = 0;
          double o6_4 = 0;
          double o6_8 = 0;
          double o7_0 = 0;
          double o7_4 = 0;
          double o7_8 = 0;
          double o8_0 = 0;
          double o8_4 = 0;
          double o8_8 = 0;
          double o9_0 = 0;
          double o9_4 = 0;
          double o9_8 = 0;
          double o10_0 = 0;
          double o10_4 = 0;
          double o10_8 = 0;
          double o11_0 = 0;
          double o11_4 = 0;
          double o11_8 = 0;
          double o12_0 = 0;
          double o12_4 = 0;
          double o12_8 = 0;
          double o13_0 = 0;
          double o13_4 = 0;
          double o13_8 = 0;
          double o14_0 = 0;
          double o14_4 = 0;
          double o14_8 = 0;
          double o15_0 = 0;
          double o15_4 = 0;
          double o15_8 = 0;
          double o16_0 = 0;
          double o16_4 = 0;
          double o16_8 = 0;
          double o17_0 = 0;
          double o17_4 = 0;
          double o17_8 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 113;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g0_0 = 0;
            double g0_1 = 0;
            double g0_2 = 0;
            double g0_3 = 0;
            double g0_4 = 0;
            double g0_5 = 0;
            double g0_6 = 0;
            double g0_7 = 0;
            double g0_8 = 0;
            double g0_9 = 0;
            double g0_10 = 0;
            double g0_11 = 0;
            double g0_12 = 0;
            double g0_13 = 0;
            double g0_14 = 0;
            double g0_15 = 0;
            double g0_16 = 0;
            double g0_17 = 0;
            double g0_18 = 0;
            double g0_19 = 0;
            double g4_0 = 0;
            double g4_1 = 0;
            double g4_2 = 0;
            double g4_3 = 0;
            double g4_4 = 0;
            double g4_5 = 0;
            double g4_6 = 0;
            double g4_7 = 0;
            double g4_8 = 0;
            double g4_9 = 0;
            double g4_10 = 0;
            double g4_11 = 0;
            double g4_12 = 0;
            double g4_13 = 0;
            double g4_14 = 0;
            double g4_15 = 0;
            double g4_16 = 0;
            double g4_17 = 0;
            double g4_18 = 0;
            double g4_19 = 0;
            double g8_0 = 0;
            double g8_1 = 0;
            double g8_2 = 0;
            double g8_3 = 0;
            double g8_4 = 0;
            double g8_5 = 0;
            double g8_6 = 0;
            double g8_7 = 0;
            double g8_8 = 0;
            double g8_9 = 0;
            double g8_10 = 0;
            double g8_11 = 0;
            double g8_12 = 0;
            double g8_13 = 0;
            double g8_14 = 0;
            double g8_15 = 0;
            double g8_16 = 0;
            double g8_17 = 0;
            double g8_18 = 0;
            double g8_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              ++nprimq;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[5];
              sqb::boys<4>(T, a.boys_tab, F);
              const double s0 = TWO_PI_2_5 * rs;
              const double m2a = -2.0 * alpha;
              double w = s0;
              const double b0 = w * F[0];
              w *= m2a;
              const double b1 = w * F[1];
              w *= m2a;
              const double b2 = w * F[2];
              w *= m2a;
              const double b3 = w * F[3];
              w *= m2a;
              const double b4 = w * F[4];
              const double ek0_0 = kj[5 * kS];
              const double ek0_1 = -kj[6 * kS];
              const double ek4_0 = kj[18 * kS];
              const double ek4_1 = -kj[19 * kS];
              const double ek8_0 = kj[31 * kS];
              const double ek8_1 = -kj[32 * kS];
              g0_0 = fma(ek0_0, b0, g0_0);
              g4_0 = fma(ek4_0, b0, g4_0);
              g8_0 = fma(ek8_0, b0, g8_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              g4_1 = fma(ek4_0, r0_0_0_1, g4_1);
              g8_1 = fma(ek8_0, r0_0_0_1, g8_1);
              g8_0 = fma(ek8_1, r0_0_0_1, g8_0);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              g4_2 = fma(ek4_0, r0_0_1_0, g4_2);
              g4_0 = fma(ek4_1, r0_0_1_0, g4_0);
              g8_2 = fma(ek8_0, r0_0_1_0, g8_2);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fma(ek0_1, r0_1_0_0, g0_0);
              g4_3 = fma(ek4_0, r0_1_0_0, g4_3);
              g8_3 = fma(ek8_0, r0_1_0_0, g8_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g0_4 = fma(ek0_0, r0_0_0_2, g0_4);
              g4_4 = fma(ek4_0, r0_0_0_2, g4_4);
              g8_4 = fma(ek8_0, r0_0_0_2, g8_4);
              g8_1 = fma(ek8_1, r0_0_0_2, g8_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fma(ek0_0, r0_0_1_1, g0_5);
              g4_5 = fma(ek4_0, r0_0_1_1, g4_5);
              g4_1 = fma(ek4_1, r0_0_1_1, g4_1);
              g8_5 = fma(ek8_0, r0_0_1_1, g8_5);
              g8_2 = fma(ek8_1, r0_0_1_1, g8_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g0_6 = fma(ek0_0, r0_0_2_0, g0_6);
              g4_6 = fma(ek4_0, r0_0_2_0, g4_6);
              g4_2 = fma(ek4_1, r0_0_2_0, g4_2);
              g8_6 = fma(ek8_0, r0_0_2_0, g8_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fma(ek0_0, r0_1_0_1, g0_7);
              g0_1 = fma(ek0_1, r0_1_0_1, g0_1);
              g4_7 = fma(ek4_0, r0_1_0_1, g4_7);
              g8_7 = fma(ek8_0, r0_1_0_1, g8_7);
              g8_3 = fma(ek8_1, r0_1_0_1, g8_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fma(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fma(ek0_1, r0_1_1_0, g0_2);
              g4_8 = fma(ek4_0, r0_1_1_0, g4_8);
              g4_3 = fma(ek4_1, r0_1_1_0, g4_3);
              g8_8 = fma(ek8_0, r0_1_1_0, g8_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g0_9 = fma(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fma(ek0_1, r0_2_0_0, g0_3);
              g4_9 = fma(ek4_0, r0_2_0_0, g4_9);
              g8_9 = fma(ek8_0, r0_2_0_0, g8_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g0_10 = fma(ek0_0, r0_0_0_3, g0_10);
              g4_10 = fma(ek4_0, r0_0_0_3, g4_10);
              g8_10 = fma(ek8_0, r0_0_0_3, g8_10);
              g8_4 = fma(ek8_1, r0_0_0_3, g8_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g0_11 = fma(ek0_0, r0_0_1_2, g0_11);
              g4_11 = fma(ek4_0, r0_0_1_2, g4_11);
              g4_4 = fma(ek4_1, r0_0_1_2, g4_4);
              g8_11 = fma(ek8_0, r0_0_1_2, g8_11);
              g8_5 = fma(ek8_1, r0_0_1_2, g8_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g0_12 = fma(ek0_0, r0_0_2_1, g0_12);
              g4_12 = fma(ek4_0, r0_0_2_1, g4_12);
              g4_5 = fma(ek4_1, r0_0_2_1, g4_5);
              g8_12 = fma(ek8_0, r0_0_2_1, g8_12);
              g8_6 = fma(ek8_1, r0_0_2_1, g8_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g0_13 = fma(ek0_0, r0_0_3_0, g0_13);
              g4_13 = fma(ek4_0, r0_0_3_0, g4_13);
              g4_6 = fma(ek4_1, r0_0_3_0, g4_6);
              g8_13 = fma(ek8_0, r0_0_3_0, g8_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g0_14 = fma(ek0_0, r0_1_0_2, g0_14);
              g0_4 = fma(ek0_1, r0_1_0_2, g0_4);
              g4_14 = fma(ek4_0, r0_1_0_2, g4_14);
              g8_14 = fma(ek8_0, r0_1_0_2, g8_14);
              g8_7 = fma(ek8_1, r0_1_0_2, g8_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g0_15 = fma(ek0_0, r0_1_1_1, g0_15);
              g0_5 = fma(ek0_1, r0_1_1_1, g0_5);
              g4_15 = fma(ek4_0, r0_1_1_1, g4_15);
              g4_7 = fma(ek4_1, r0_1_1_1, g4_7);
              g8_15 = fma(ek8_0, r0_1_1_1, g8_15);
              g8_8 = fma(ek8_1, r0_1_1_1, g8_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g0_16 = fma(ek0_0, r0_1_2_0, g0_16);
              g0_6 = fma(ek0_1, r0_1_2_0, g0_6);
              g4_16 = fma(ek4_0, r0_1_2_0, g4_16);
              g4_8 = fma(ek4_1, r0_1_2_0, g4_8);
              g8_16 = fma(ek8_0, r0_1_2_0, g8_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g0_17 = fma(ek0_0, r0_2_0_1, g0_17);
              g0_7 = fma(ek0_1, r0_2_0_1, g0_7);
              g4_17 = fma(ek4_0, r0_2_0_1, g4_17);
              g8_17 = fma(ek8_0, r0_2_0_1, g8_17);
              g8_9 = fma(ek8_1, r0_2_0_1, g8_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fma(ek0_0, r0_2_1_0, g0_18);
              g0_8 = fma(ek0_1, r0_2_1_0, g0_8);
              g4_18 = fma(ek4_0, r0_2_1_0, g4_18);
              g4_9 = fma(ek4_1, r0_2_1_0, g4_9);
              g8_18 = fma(ek8_0, r0_2_1_0, g8_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_19 = fma(ek0_0, r0_3_0_0, g0_19);
              g0_9 = fma(ek0_1, r0_3_0_0, g0_9);
              g4_19 = fma(ek4_0, r0_3_0_0, g4_19);
              g8_19 = fma(ek8_0, r0_3_0_0, g8_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g8_10 = fma(ek8_1, r0_0_0_4, g8_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g4_10 = fma(ek4_1, r0_0_1_3, g4_10);
              g8_11 = fma(ek8_1, r0_0_1_3, g8_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g4_11 = fma(ek4_1, r0_0_2_2, g4_11);
              g8_12 = fma(ek8_1, r0_0_2_2, g8_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g4_12 = fma(ek4_1, r0_0_3_1, g4_12);
              g8_13 = fma(ek8_1, r0_0_3_1, g8_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g4_13 = fma(ek4_1, r0_0_4_0, g4_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g0_10 = fma(ek0_1, r0_1_0_3, g0_10);
              g8_14 = fma(ek8_1, r0_1_0_3, g8_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g0_11 = fma(ek0_1, r0_1_1_2, g0_11);
              g4_14 = fma(ek4_1, r0_1_1_2, g4_14);
              g8_15 = fma(ek8_1, r0_1_1_2, g8_15);
              const double r0_1_2_1 = X * r1_0_2_1;
              g0_12 = fma(ek0_1, r0_1_2_1, g0_12);
              g4_15 = fma(ek4_1, r0_1_2_1, g4_15);
              g8_16 = fma(ek8_1, r0_1_2_1, g8_16);
              const double r0_1_3_0 = X * r1_0_3_0;
              g0_13 = fma(ek0_1, r0_1_3_0, g0_13);
              g4_16 = fma(ek4_1, r0_1_3_0, g4_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g0_14 = fma(ek0_1, r0_2_0_2, g0_14);
              g8_17 = fma(ek8_1, r0_2_0_2, g8_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g0_15 = fma(ek0_1, r0_2_1_1, g0_15);
              g4_17 = fma(ek4_1, r0_2_1_1, g4_17);
              g8_18 = fma(ek8_1, r0_2_1_1, g8_18);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g0_16 = fma(ek0_1, r0_2_2_0, g0_16);
              g4_18 = fma(ek4_1, r0_2_2_0, g4_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g0_17 = fma(ek0_1, r0_3_0_1, g0_17);
              g8_19 = fma(ek8_1, r0_3_0_1, g8_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g0_18 = fma(ek0_1, r0_3_1_0, g0_18);
              g4_19 = fma(ek4_1, r0_3_1_0, g4_19);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g0_19 = fma(ek0_1, r0_4_0_0, g0_19);
            }
            { const double eb = bi[5];
              o0_0 = fma(eb, g0_0, o0_0);
              o0_4 = fma(eb, g4_0, o0_4);
              o0_8 = fma(eb, g8_0, o0_8);
            }
            { const double eb = bi[6];
              o0_0 = fma(eb, g0_3, o0_0);
              o0_4 = fma(eb, g4_3, o0_4);
              o0_8 = fma(eb, g8_3, o0_8);
            }
            { const double eb = bi[7];
              o0_0 = fma(eb, g0_9, o0_0);
              o0_4 = fma(eb, g4_9, o0_4);
              o0_8 = fma(eb, g8_9, o0_8);
            }
            { const double eb = bi[8];
              o0_0 = fma(eb, g0_19, o0_0);
              o0_4 = fma(eb, g4_19, o0_4);
              o0_8 = fma(eb, g8_19, o0_8);
            }
            { const double eb = bi[9];
              o1_0 = fma(eb, g0_0, o1_0);
              o1_4 = fma(eb, g4_0, o1_4);
              o1_8 = fma(eb, g8_0, o1_8);
            }
            { const double eb = bi[10];
              o1_0 = fma(eb, g0_2, o1_0);
              o1_4 = fma(eb, g4_2, o1_4);
              o1_8 = fma(eb, g8_2, o1_8);
            }
            { const double eb = bi[11];
              o1_0 = fma(eb, g0_3, o1_0);
              o1_4 = fma(eb, g4_3, o1_4);
              o1_8 = fma(eb, g8_3, o1_8);
            }
            { const double eb = bi[12];
              o1_0 = fma(eb, g0_8, o1_0);
              o1_4 = fma(eb, g4_8, o1_4);
              o1_8 = fma(eb, g8_8, o1_8);
            }
            { const double eb = bi[13];
              o1_0 = fma(eb, g0_9, o1_0);
              o1_4 = fma(eb, g4_9, o1_4);
              o1_8 = fma(eb, g8_9, o1_8);
            }
            { const double eb = bi[14];
              o1_0 = fma(eb, g0_18, o1_0);
              o1_4 = fma(eb, g4_18, o1_4);
              o1_8 = fma(eb, g8_18, o1_8);
            }
            { const double eb = bi[15];
              o2_0 = fma(eb, g0_0, o2_0);
              o2_4 = fma(eb, g4_0, o2_4);
              o2_8 = fma(eb, g8_0, o2_8);
            }
            { const double eb = bi[16];
              o2_0 = fma(eb, g0_1, o2_0);
              o2_4 = fma(eb, g4_1, o2_4);
              o2_8 = fma(eb, g8_1, o2_8);
            }
            { const double eb = bi[17];
              o2_0 = fma(eb, g0_3, o2_0);
              o2_4 = fma(eb, g4_3, o2_4);
              o2_8 = fma(eb, g8_3, o2_8);
            }
            { const double eb = bi[18];
              o2_0 = fma(eb, g0_7, o2_0);
              o2_4 = fma(eb, g4_7, o2_4);
              o2_8 = fma(eb, g8_7, o2_8);
            }
            { const double eb = bi[19];
              o2_0 = fma(eb, g0_9, o2_0);
              o2_4 = fma(eb, g4_9, o2_4);
              o2_8 = fma(eb, g8_9, o2_8);
            }
            { const double eb = bi[20];
              o2_0 = fma(eb, g0_17, o2_0);
              o2_4 = fma(eb, g4_17, o2_4);
              o2_8 = fma(eb, g8_17, o2_8);
            }
            { const double eb = bi[21];
              o3_0 = fma(eb, g0_0, o3_0);
              o3_4 = fma(eb, g4_0, o3_4);
              o3_8 = fma(eb, g8_0, o3_8);
            }
            { const double eb = bi[22];
              o3_0 = fma(eb, g0_2, o3_0);
              o3_4 = fma(eb, g4_2, o3_4);
              o3_8 = fma(eb, g8_2, o3_8);
            }
            { const double eb = bi[23];
              o3_0 = fma(eb, g0_6, o3_0);
              o3_4 = fma(eb, g4_6, o3_4);
              o3_8 = fma(eb, g8_6, o3_8);
            }
            { const double eb = bi[24];
              o3_0 = fma(eb, g0_3, o3_0);
              o3_4 = fma(eb, g4_3, o3_4);
              o3_8 = fma(eb, g8_3, o3_8);
            }
            { const double eb = bi[25];
              o3_0 = fma(eb, g0_8, o3_0);
              o3_4 = fma(eb, g4_8, o3_4);
              o3_8 = fma(eb, g8_8, o3_8);
            }
            { const double eb = bi[26];
              o3_0 = fma(eb, g0_16, o3_0);
              o3_4 = fma(eb, g4_16, o3_4);
              o3_8 = fma(eb, g8_16, o3_8);
            }
            { const double eb = bi[27];
              o4_0 = fma(eb, g0_0, o4_0);
              o4_4 = fma(eb, g4_0, o4_4);
              o4_8 = fma(eb, g8_0, o4_8);
            }
            { const double eb = bi[28];
              o4_0 = fma(eb, g0_2, o4_0);
              o4_4 = fma(eb, g4_2, o4_4);
              o4_8 = fma(eb, g8_2, o4_8);
            }
            { const double eb = bi[29];
              o4_0 = fma(eb, g0_6, o4_0);
              o4_4 = fma(eb, g4_6, o4_4);
              o4_8 = fma(eb, g8_6, o4_8);
            }
            { const double eb = bi[30];
              o4_0 = fma(eb, g0_13, o4_0);
              o4_4 = fma(eb, g4_13, o4_4);
              o4_8 = fma(eb, g8_13, o4_8);
            }
            { const double eb = bi[31];
              o5_0 = fma(eb, g0_0, o5_0);
              o5_4 = fma(eb, g4_0, o5_4);
              o5_8 = fma(eb, g8_0, o5_8);
            }
            { const double eb = bi[32];
              o5_0 = fma(eb, g0_1, o5_0);
              o5_4 = fma(eb, g4_1, o5_4);
              o5_8 = fma(eb, g8_1, o5_8);
            }
            { const double eb = bi[33];
              o5_0 = fma(eb, g0_2, o5_0);
              o5_4 = fma(eb, g4_2, o5_4);
              o5_8 = fma(eb, g8_2, o5_8);
            }
            { const double eb = bi[34];
              o5_0 = fma(eb, g0_5, o5_0);
              o5_4 = fma(eb, g4_5, o5_4);
              o5_8 = fma(eb, g8_5, o5_8);
            }
            { const double eb = bi[35];
              o5_0 = fma(eb, g0_6, o5_0);
              o5_4 = fma(eb, g4_6, o5_4);
              o5_8 = fma(eb, g8_6, o5_8);
            }
            { const double eb = bi[36];
              o5_0 = fma(eb, g0_12, o5_0);
              o5_4 = fma(eb, g4_12, o5_4);
              o5_8 = fma(eb, g8_12, o5_8);
            }
            { const double eb = bi[37];
              o6_0 = fma(eb, g0_0, o6_0);
              o6_4 = fma(eb, g4_0, o6_4);
              o6_8 = fma(eb, g8_0, o6_8);
            }
            { const double eb = bi[38];
              o6_0 = fma(eb, g0_1, o6_0);
              o6_4 = fma(eb, g4_1, o6_4);
              o6_8 = fma(eb, g8_1, o6_8);
            }
            { const double eb = bi[39];
              o6_0 = fma(eb, g0_4, o6_0);
              o6_4 = fma(eb, g4_4, o6_4);
              o6_8 = fma(eb, g8_4, o6_8);
            }
            { const double eb = bi[40];
              o6_0 = fma(eb, g0_3, o6_0);
              o6_4 = fma(eb, g4_3, o6_4);
              o6_8 = fma(eb, g8_3, o6_8);
            }
            { const double eb = bi[41];
              o6_0 = fma(eb, g0_7, o6_0);
              o6_4 = fma(eb, g4_7, o6_4);
              o6_8 = fma(eb, g8_7, o6_8);
            }
            { const double eb = bi[42];
              o6_0 = fma(eb, g0_14, o6_0);
              o6_4 = fma(eb, g4_14, o6_4);
              o6_8 = fma(eb, g8_14, o6_8);
            }
            { const double eb = bi[43];
              o7_0 = fma(eb, g0_0, o7_0);
              o7_4 = fma(eb, g4_0, o7_4);
              o7_8 = fma(eb, g8_0, o7_8);
            }
            { const double eb = bi[44];
              o7_0 = fma(eb, g0_1, o7_0);
              o7_4 = fma(eb, g4_1, o7_4);
              o7_8 = fma(eb, g8_1, o7_8);
            }
            { const double eb = bi[45];
              o7_0 = fma(eb, g0_4, o7_0);
              o7_4 = fma(eb, g4_4, o7_4);
              o7_8 = fma(eb, g8_4, o7_8);
            }
            { const double eb = bi[46];
              o7_0 = fma(eb, g0_2, o7_0);
              o7_4 = fma(eb, g4_2, o7_4);
              o7_8 = fma(eb, g8_2, o7_8);
            }
            { const double eb = bi[47];
              o7_0 = fma(eb, g0_5, o7_0);
              o7_4 = fma(eb, g4_5, o7_4);
              o7_8 = fma(eb, g8_5, o7_8);
            }
            { const double eb = bi[48];
              o7_0 = fma(eb, g0_11, o7_0);
              o7_4 = fma(eb, g4_11, o7_4);
              o7_8 = fma(eb, g8_11, o7_8);
            }
            { const double eb = bi[49];
              o8_0 = fma(eb, g0_0, o8_0);
              o8_4 = fma(eb, g4_0, o8_4);
              o8_8 = fma(eb, g8_0, o8_8);
            }
            { const double eb = bi[50];
              o8_0 = fma(eb, g0_1, o8_0);
              o8_4 = fma(eb, g4_1, o8_4);
              o8_8 = fma(eb, g8_1, o8_8);
            }
            { const double eb = bi[51];
              o8_0 = fma(eb, g0_4, o8_0);
              o8_4 = fma(eb, g4_4, o8_4);
              o8_8 = fma(eb, g8_4, o8_8);
            }
            { const double eb = bi[52];
              o8_0 = fma(eb, g0_10, o8_0);
              o8_4 = fma(eb, g4_10, o8_4);
              o8_8 = fma(eb, g8_10, o8_8);
            }
            { const double eb = bi[53];
              o9_0 = fma(eb, g0_0, o9_0);
              o9_4 = fma(eb, g4_0, o9_4);
              o9_8 = fma(eb, g8_0, o9_8);
            }
            { const double eb = bi[54];
              o9_0 = fma(eb, g0_2, o9_0);
              o9_4 = fma(eb, g4_2, o9_4);
              o9_8 = fma(eb, g8_2, o9_8);
            }
            { const double eb = bi[55];
              o9_0 = fma(eb, g0_3, o9_0);
              o9_4 = fma(eb, g4_3, o9_4);
              o9_8 = fma(eb, g8_3, o9_8);
            }
            { const double eb = bi[56];
              o9_0 = fma(eb, g0_8, o9_0);
              o9_4 = fma(eb, g4_8, o9_4);
              o9_8 = fma(eb, g8_8, o9_8);
            }
            { const double eb = bi[57];
              o9_0 = fma(eb, g0_9, o9_0);
              o9_4 = fma(eb, g4_9, o9_4);
              o9_8 = fma(eb, g8_9, o9_8);
            }
            { const double eb = bi[58];
              o9_0 = fma(eb, g0_18, o9_0);
              o9_4 = fma(eb, g4_18, o9_4);
              o9_8 = fma(eb, g8_18, o9_8);
            }
            { const double eb = bi[59];
              o10_0 = fma(eb, g0_0, o10_0);
              o10_4 = fma(eb, g4_0, o10_4);
              o10_8 = fma(eb, g8_0, o10_8);
            }
            { const double eb = bi[60];
              o10_0 = fma(eb, g0_2, o10_0);
              o10_4 = fma(eb, g4_2, o10_4);
              o10_8 = fma(eb, g8_2, o10_8);
            }
            { const double eb = bi[61];
              o10_0 = fma(eb, g0_6, o10_0);
              o10_4 = fma(eb, g4_6, o10_4);
              o10_8 = fma(eb, g8_6, o10_8);
            }
            { const double eb = bi[62];
              o10_0 = fma(eb, g0_3, o10_0);
              o10_4 = fma(eb, g4_3, o10_4);
              o10_8 = fma(eb, g8_3, o10_8);
            }
            { const double eb = bi[63];
              o10_0 = fma(eb, g0_8, o10_0);
              o10_4 = fma(eb, g4_8, o10_4);
              o10_8 = fma(eb, g8_8, o10_8);
            }
            { const double eb = bi[64];
              o10_0 = fma(eb, g0_16, o10_0);
              o10_4 = fma(eb, g4_16, o10_4);
              o10_8 = fma(eb, g8_16, o10_8);
            }
            { const double eb = bi[65];
              o11_0 = fma(eb, g0_0, o11_0);
              o11_4 = fma(eb, g4_0, o11_4);
              o11_8 = fma(eb, g8_0, o11_8);
            }
            { const double eb = bi[66];
              o11_0 = fma(eb, g0_1, o11_0);
              o11_4 = fma(eb, g4_1, o11_4);
              o11_8 = fma(eb, g8_1, o11_8);
            }
            { const double eb = bi[67];
              o11_0 = fma(eb, g0_2, o11_0);
              o11_4 = fma(eb, g4_2, o11_4);
              o11_8 = fma(eb, g8_2, o11_8);
            }
            { const double eb = bi[68];
              o11_0 = fma(eb, g0_5, o11_0);
              o11_4 = fma(eb, g4_5, o11_4);
              o11_8 = fma(eb, g8_5, o11_8);
            }
            { const double eb = bi[69];
              o11_0 = fma(eb, g0_3, o11_0);
              o11_4 = fma(eb, g4_3, o11_4);
              o11_8 = fma(eb, g8_3, o11_8);
            }
            { const double eb = bi[70];
              o11_0 = fma(eb, g0_7, o11_0);
              o11_4 = fma(eb, g4_7, o11_4);
              o11_8 = fma(eb, g8_7, o11_8);
            }
            { const double eb = bi[71];
              o11_0 = fma(eb, g0_8, o11_0);
              o11_4 = fma(eb, g4_8, o11_4);
              o11_8 = fma(eb, g8_8, o11_8);
            }
            { const double eb = bi[72];
              o11_0 = fma(eb, g0_15, o11_0);
              o11_4 = fma(eb, g4_15, o11_4);
              o11_8 = fma(eb, g8_15, o11_8);
            }
            { const double eb = bi[73];
              o12_0 = fma(eb, g0_0, o12_0);
              o12_4 = fma(eb, g4_0, o12_4);
              o12_8 = fma(eb, g8_0, o12_8);
            }
            { const double eb = bi[74];
              o12_0 = fma(eb, g0_1, o12_0);
              o12_4 = fma(eb, g4_1, o12_4);
              o12_8 = fma(eb, g8_1, o12_8);
            }
            { const double eb = bi[75];
              o12_0 = fma(eb, g0_3, o12_0);
              o12_4 = fma(eb, g4_3, o12_4);
              o12_8 = fma(eb, g8_3, o12_8);
            }
            { const double eb = bi[76];
              o12_0 = fma(eb, g0_7, o12_0);
              o12_4 = fma(eb, g4_7, o12_4);
              o12_8 = fma(eb, g8_7, o12_8);
            }
            { const double eb = bi[77];
              o12_0 = fma(eb, g0_9, o12_0);
              o12_4 = fma(eb, g4_9, o12_4);
              o12_8 = fma(eb, g8_9, o12_8);
            }
            { const double eb = bi[78];
              o12_0 = fma(eb, g0_17, o12_0);
              o12_4 = fma(eb, g4_17, o12_4);
              o12_8 = fma(eb, g8_17, o12_8);
            }
            { const double eb = bi[79];
              o13_0 = fma(eb, g0_0, o13_0);
              o13_4 = fma(eb, g4_0, o13_4);
              o13_8 = fma(eb, g8_0, o13_8);
            }
            { const double eb = bi[80];
              o13_0 = fma(eb, g0_1, o13_0);
              o13_4 = fma(eb, g4_1, o13_4);
              o13_8 = fma(eb, g8_1, o13_8);
            }
            { const double eb = bi[81];
              o13_0 = fma(eb, g0_2, o13_0);
              o13_4 = fma(eb, g4_2, o13_4);
              o13_8 = fma(eb, g8_2, o13_8);
            }
            { const double eb = bi[82];
              o13_0 = fma(eb, g0_5, o13_0);
              o13_4 = fma(eb, g4_5, o13_4);
              o13_8 = fma(eb, g8_5, o13_8);
            }
            { const double eb = bi[83];
              o13_0 = fma(eb, g0_3, o13_0);
              o13_4 = fma(eb, g4_3, o13_4);
              o13_8 = fma(eb, g8_3, o13_8);
            }
            { const double eb = bi[84];
              o13_0 = fma(eb, g0_7, o13_0);
              o13_4 = fma(eb, g4_7, o13_4);
              o13_8 = fma(eb, g8_7, o13_8);
            }
            { const double eb = bi[85];
              o13_0 = fma(eb, g0_8, o13_0);
              o13_4 = fma(eb, g4_8, o13_4);
              o13_8 = fma(eb, g8_8, o13_8);
            }
            { const double eb = bi[86];
              o13_0 = fma(eb, g0_15, o13_0);
              o13_4 = fma(eb, g4_15, o13_4);
              o13_8 = fma(eb, g8_15, o13_8);
            }
            { const double eb = bi[87];
              o14_0 = fma(eb, g0_0, o14_0);
              o14_4 = fma(eb, g4_0, o14_4);
              o14_8 = fma(eb, g8_0, o14_8);
            }
            { const double eb = bi[88];
              o14_0 = fma(eb, g0_1, o14_0);
              o14_4 = fma(eb, g4_1, o14_4);
              o14_8 = fma(eb, g8_1, o14_8);
            }
            { const double eb = bi[89];
              o14_0 = fma(eb, g0_4, o14_0);
              o14_4 = fma(eb, g4_4, o14_4);
              o14_8 = fma(eb, g8_4, o14_8);
            }
            { const double eb = bi[90];
              o14_0 = fma(eb, g0_3, o14_0);
              o14_4 = fma(eb, g4_3, o14_4);
              o14_8 = fma(eb, g8_3, o14_8);
            }
            { const double eb = bi[91];
              o14_0 = fma(eb, g0_7, o14_0);
              o14_4 = fma(eb, g4_7, o14_4);
              o14_8 = fma(eb, g8_7, o14_8);
            }
            { const double eb = bi[92];
              o14_0 = fma(eb, g0_14, o14_0);
              o14_4 = fma(eb, g4_14, o14_4);
              o14_8 = fma(eb, g8_14, o14_8);
            }
            { const double eb = bi[93];
              o15_0 = fma(eb, g0_0, o15_0);
              o15_4 = fma(eb, g4_0, o15_4);
              o15_8 = fma(eb, g8_0, o15_8);
            }
            { const double eb = bi[94];
              o15_0 = fma(eb, g0_1, o15_0);
              o15_4 = fma(eb, g4_1, o15_4);
              o15_8 = fma(eb, g8_1, o15_8);
            }
            { const double eb = bi[95];
              o15_0 = fma(eb, g0_2, o15_0);
              o15_4 = fma(eb, g4_2, o15_4);
              o15_8 = fma(eb, g8_2, o15_8);
            }
            { const double eb = bi[96];
              o15_0 = fma(eb, g0_5, o15_0);
              o15_4 = fma(eb, g4_5, o15_4);
              o15_8 = fma(eb, g8_5, o15_8);
            }
            { const double eb = bi[97];
              o15_0 = fma(eb, g0_3, o15_0);
              o15_4 = fma(eb, g4_3, o15_4);
              o15_8 = fma(eb, g8_3, o15_8);
            }
            { const double eb = bi[98];
              o15_0 = fma(eb, g0_7, o15_0);
              o15_4 = fma(eb, g4_7, o15_4);
              o15_8 = fma(eb, g8_7, o15_8);
            }
            { const double eb = bi[99];
              o15_0 = fma(eb, g0_8, o15_0);
              o15_4 = fma(eb, g4_8, o15_4);
              o15_8 = fma(eb, g8_8, o15_8);
            }
            { const double eb = bi[100];
              o15_0 = fma(eb, g0_15, o15_0);
              o15_4 = fma(eb, g4_15, o15_4);
              o15_8 = fma(eb, g8_15, o15_8);
            }
            { const double eb = bi[101];
              o16_0 = fma(eb, g0_0, o16_0);
              o16_4 = fma(eb, g4_0, o16_4);
              o16_8 = fma(eb, g8_0, o16_8);
            }
            { const double eb = bi[102];
              o16_0 = fma(eb, g0_1, o16_0);
              o16_4 = fma(eb, g4_1, o16_4);
              o16_8 = fma(eb, g8_1, o16_8);
            }
            { const double eb = bi[103];
              o16_0 = fma(eb, g0_2, o16_0);
              o16_4 = fma(eb, g4_2, o16_4);
              o16_8 = fma(eb, g8_2, o16_8);
            }
            { const double eb = bi[104];
              o16_0 = fma(eb, g0_5, o16_0);
              o16_4 = fma(eb, g4_5, o16_4);
              o16_8 = fma(eb, g8_5, o16_8);
            }
            { const double eb = bi[105];
              o16_0 = fma(eb, g0_6, o16_0);
              o16_4 = fma(eb, g4_6, o16_4);
              o16_8 = fma(eb, g8_6, o16_8);
            }
            { const double eb = bi[106];
              o16_0 = fma(eb, g0_12, o16_0);
              o16_4 = fma(eb, g4_12, o16_4);
              o16_8 = fma(eb, g8_12, o16_8);
            }
            { const double eb = bi[107];
              o17_0 = fma(eb, g0_0, o17_0);
              o17_4 = fma(eb, g4_0, o17_4);
              o17_8 = fma(eb, g8_0, o17_8);
            }
            { const double eb = bi[108];
              o17_0 = fma(eb, g0_1, o17_0);
              o17_4 = fma(eb, g4_1, o17_4);
              o17_8 = fma(eb, g8_1, o17_8);
            }
            { const double eb = bi[109];
              o17_0 = fma(eb, g0_4, o17_0);
              o17_4 = fma(eb, g4_4, o17_4);
              o17_8 = fma(eb, g8_4, o17_8);
            }
            { const double eb = bi[110];
              o17_0 = fma(eb, g0_2, o17_0);
              o17_4 = fma(eb, g4_2, o17_4);
              o17_8 = fma(eb, g8_2, o17_8);
            }
            { const double eb = bi[111];
              o17_0 = fma(eb, g0_5, o17_0);
              o17_4 = fma(eb, g4_5, o17_4);
              o17_8 = fma(eb, g8_5, o17_8);
            }
            { const double eb = bi[112];
              o17_0 = fma(eb, g0_11, o17_0);
              o17_4 = fma(eb, g4_11, o17_4);
              o17_8 = fma(eb, g8_11, o17_8);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptk4 = PT[(fI + 1) * N + fJ + 0];
            const double ptk8 = PT[(fI + 2) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 1) * N + fQ + 0];
            const double ptb4 = PT[(fP + 1) * N + fQ + 1];
            const double ptb5 = PT[(fP + 1) * N + fQ + 2];
            const double ptb6 = PT[(fP + 2) * N + fQ + 0];
            const double ptb7 = PT[(fP + 2) * N + fQ + 1];
            const double ptb8 = PT[(fP + 2) * N + fQ + 2];
            const double ptb9 = PT[(fP + 3) * N + fQ + 0];
            const double ptb10 = PT[(fP + 3) * N + fQ + 1];
            const double ptb11 = PT[(fP + 3) * N + fQ + 2];
            const double ptb12 = PT[(fP + 4) * N + fQ + 0];
            const double ptb13 = PT[(fP + 4) * N + fQ + 1];
            const double ptb14 = PT[(fP + 4) * N + fQ + 2];
            const double ptb15 = PT[(fP + 5) * N + fQ + 0];
            const double ptb16 = PT[(fP + 5) * N + fQ + 1];
            const double ptb17 = PT[(fP + 5) * N + fQ + 2];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            jab0 += o0_0 * ptk0 + o0_4 * ptk4 + o0_8 * ptk8;
            jab1 += o1_0 * ptk0 + o1_4 * ptk4 + o1_8 * ptk8;
            jab2 += o2_0 * ptk0 + o2_4 * ptk4 + o2_8 * ptk8;
            jab3 += o3_0 * ptk0 + o3_4 * ptk4 + o3_8 * ptk8;
            jab4 += o4_0 * ptk0 + o4_4 * ptk4 + o4_8 * ptk8;
            jab5 += o5_0 * ptk0 + o5_4 * ptk4 + o5_8 * ptk8;
            jab6 += o6_0 * ptk0 + o6_4 * ptk4 + o6_8 * ptk8;
            jab7 += o7_0 * ptk0 + o7_4 * ptk4 + o7_8 * ptk8;
            jab8 += o8_0 * ptk0 + o8_4 * ptk4 + o8_8 * ptk8;
            jab9 += o9_0 * ptk0 + o9_4 * ptk4 + o9_8 * ptk8;
            jab10 += o10_0 * ptk0 + o10_4 * ptk4 + o10_8 * ptk8;
            jab11 += o11_0 * ptk0 + o11_4 * ptk4 + o11_8 * ptk8;
            jab12 += o12_0 * ptk0 + o12_4 * ptk4 + o12_8 * ptk8;
            jab13 += o13_0 * ptk0 + o13_4 * ptk4 + o13_8 * ptk8;
            jab14 += o14_0 * ptk0 + o14_4 * ptk4 + o14_8 * ptk8;
            jab15 += o15_0 * ptk0 + o15_4 * ptk4 + o15_8 * ptk8;
            jab16 += o16_0 * ptk0 + o16_4 * ptk4 + o16_8 * ptk8;
            jab17 += o17_0 * ptk0 + o17_4 * ptk4 + o17_8 * ptk8;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15 + o16_0 * ptb16 + o17_0 * ptb17));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_4 * ptb0 + o1_4 * ptb1 + o2_4 * ptb2 + o3_4 * ptb3 + o4_4 * ptb4 + o5_4 * ptb5 + o6_4 * ptb6 + o7_4 * ptb7 + o8_4 * ptb8 + o9_4 * ptb9 + o10_4 * ptb10 + o11_4 * ptb11 + o12_4 * ptb12 + o13_4 * ptb13 + o14_4 * ptb14 + o15_4 * ptb15 + o16_4 * ptb16 + o17_4 * ptb17));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_8 * ptb0 + o1_8 * ptb1 + o2_8 * ptb2 + o3_8 * ptb3 + o4_8 * ptb4 + o5_8 * ptb5 + o6_8 * ptb6 + o7_8 * ptb7 + o8_8 * ptb8 + o9_8 * ptb9 + o10_8 * ptb10 + o11_8 * ptb11 + o12_8 * ptb12 + o13_8 * ptb13 + o14_8 * ptb14 + o15_8 * ptb15 + o16_8 * ptb16 + o17_8 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o3_0 * Aad1_0 + o6_0 * Aad2_0 + o9_0 * Aad3_0 + o12_0 * Aad4_0 + o15_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o0_4 * Abc0_1 + o0_8 * Abc0_2 + o1_0 * Abc1_0 + o1_4 * Abc1_1 + o1_8 * Abc1_2 + o2_0 * Abc2_0 + o2_4 * Abc2_1 + o2_8 * Abc2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o0_4 * Aac0_1 + o0_8 * Aac0_2 + o3_0 * Aac1_0 + o3_4 * Aac1_1 + o3_8 * Aac1_2 + o6_0 * Aac2_0 + o6_4 * Aac2_1 + o6_8 * Aac2_2 + o9_0 * Aac3_0 + o9_4 * Aac3_1 + o9_8 * Aac3_2 + o12_0 * Aac4_0 + o12_4 * Aac4_1 + o12_8 * Aac4_2 + o15_0 * Aac5_0 + o15_4 * Aac5_1 + o15_8 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_4 * Abd0_0 + o1_4 * Abd1_0 + o2_4 * Abd2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_4 * Aad0_0 + o3_4 * Aad1_0 + o6_4 * Aad2_0 + o9_4 * Aad3_0 + o12_4 * Aad4_0 + o15_4 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_8 * Abd0_0 + o1_8 * Abd1_0 + o2_8 * Abd2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_8 * Aad0_0 + o3_8 * Aad1_0 + o6_8 * Aad2_0 + o9_8 * Aad3_0 + o12_8 * Aad4_0 + o15_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o4_0 * Aad1_0 + o7_0 * Aad2_0 + o10_0 * Aad3_0 + o13_0 * Aad4_0 + o16_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o1_4 * Aac0_1 + o1_8 * Aac0_2 + o4_0 * Aac1_0 + o4_4 * Aac1_1 + o4_8 * Aac1_2 + o7_0 * Aac2_0 + o7_4 * Aac2_1 + o7_8 * Aac2_2 + o10_0 * Aac3_0 + o10_4 * Aac3_1 + o10_8 * Aac3_2 + o13_0 * Aac4_0 + o13_4 * Aac4_1 + o13_8 * Aac4_2 + o16_0 * Aac5_0 + o16_4 * Aac5_1 + o16_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_4 * Aad0_0 + o4_4 * Aad1_0 + o7_4 * Aad2_0 + o10_4 * Aad3_0 + o13_4 * Aad4_0 + o16_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_8 * Aad0_0 + o4_8 * Aad1_0 + o7_8 * Aad2_0 + o10_8 * Aad3_0 + o13_8 * Aad4_0 + o16_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o5_0 * Aad1_0 + o8_0 * Aad2_0 + o11_0 * Aad3_0 + o14_0 * Aad4_0 + o17_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o2_4 * Aac0_1 + o2_8 * Aac0_2 + o5_0 * Aac1_0 + o5_4 * Aac1_1 + o5_8 * Aac1_2 + o8_0 * Aac2_0 + o8_4 * Aac2_1 + o8_8 * Aac2_2 + o11_0 * Aac3_0 + o11_4 * Aac3_1 + o11_8 * Aac3_2 + o14_0 * Aac4_0 + o14_4 * Aac4_1 + o14_8 * Aac4_2 + o17_0 * Aac5_0 + o17_4 * Aac5_1 + o17_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_4 * Aad0_0 + o5_4 * Aad1_0 + o8_4 * Aad2_0 + o11_4 * Aad3_0 + o14_4 * Aad4_0 + o17_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_8 * Aad0_0 + o5_8 * Aad1_0 + o8_8 * Aad2_0 + o11_8 * Aad3_0 + o14_8 * Aad4_0 + o17_8 * Aad5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o3_0 * Abd0_0 + o4_0 * Abd1_0 + o5_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o3_0 * Abc0_0 + o3_4 * Abc0_1 + o3_8 * Abc0_2 + o4_0 * Abc1_0 + o4_4 * Abc1_1 + o4_8 * Abc1_2 + o5_0 * Abc2_0 + o5_4 * Abc2_1 + o5_8 * Abc2_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o3_4 * Abd0_0 + o4_4 * Abd1_0 + o5_4 * Abd2_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o3_8 * Abd0_0 + o4_8 * Abd1_0 + o5_8 * Abd2_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o6_0 * Abd0_0 + o7_0 * Abd1_0 + o8_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o6_0 * Abc0_0 + o6_4 * Abc0_1 + o6_8 * Abc0_2 + o7_0 * Abc1_0 + o7_4 * Abc1_1 + o7_8 * Abc1_2 + o8_0 * Abc2_0 + o8_4 * Abc2_1 + o8_8 * Abc2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o6_4 * Abd0_0 + o7_4 * Abd1_0 + o8_4 * Abd2_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o6_8 * Abd0_0 + o7_8 * Abd1_0 + o8_8 * Abd2_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o9_0 * Abd0_0 + o10_0 * Abd1_0 + o11_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o9_0 * Abc0_0 + o9_4 * Abc0_1 + o9_8 * Abc0_2 + o10_0 * Abc1_0 + o10_4 * Abc1_1 + o10_8 * Abc1_2 + o11_0 * Abc2_0 + o11_4 * Abc2_1 + o11_8 * Abc2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o9_4 * Abd0_0 + o10_4 * Abd1_0 + o11_4 * Abd2_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o9_8 * Abd0_0 + o10_8 * Abd1_0 + o11_8 * Abd2_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o12_4 * Abc0_1 + o12_8 * Abc0_2 + o13_0 * Abc1_0 + o13_4 * Abc1_1 + o13_8 * Abc1_2 + o14_0 * Abc2_0 + o14_4 * Abc2_1 + o14_8 * Abc2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o12_4 * Abd0_0 + o13_4 * Abd1_0 + o14_4 * Abd2_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o12_8 * Abd0_0 + o13_8 * Abd1_0 + o14_8 * Abd2_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o15_0 * Abd0_0 + o16_0 * Abd1_0 + o17_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o15_0 * Abc0_0 + o15_4 * Abc0_1 + o15_8 * Abc0_2 + o16_0 * Abc1_0 + o16_4 * Abc1_1 + o16_8 * Abc1_2 + o17_0 * Abc2_0 + o17_4 * Abc2_1 + o17_8 * Abc2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o15_4 * Abd0_0 + o16_4 * Abd1_0 + o17_4 * Abd2_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o15_8 * Abd0_0 + o16_8 * Abd1_0 + o17_8 * Abd2_0));
          }
        } break;
        case 1: {  // ket functions [1, 5, 9]
          double o0_1 = 0;
          double o0_5 = 0;
          double o0_9 = 0;
          double o1_1 = 0;
          double o1_5 = 0;
          double o1_9 = 0;
          double o2_1 = 0;
          double o2_5 = 0;
          double o2_9 = 0;
          double o3_1 = 0;
          double o3_5 = 0;
          double o3_9 = 0;
          double o4_1 = 0;
          double o4_5 = 0;
          double o4_9 = 0;
          double o5_1 = 0;
          double o5_5 = 0;
          double o5_9 = 0;
          double o6_1 = 0;
          double o6_5 = 0;
          double o6_9 = 0;
          double o7_1 = 0;
          double o7_5 = 0;
          double o7_9 = 0;
          double o8_1 = 0;
          double o8_5 = 0;
          double o8_9 = 0;
          double o9_1 = 0;
          double o9_5 = 0;
          double o9_9 = 0;
          double o10_1 = 0;
          double o10_5 = 0;
          double o10_9 = 0;
          double o11_1 = 0;
          double o11_5 = 0;
          double o11_9 = 0;
          double o12_1 = 0;
          double o12_5 = 0;
          double o12_9 = 0;
          double o13_1 = 0;
          double o13_5 = 0;
          double o13_9 = 0;
          double o14_1 = 0;
          double o14_5 = 0;
          double o14_9 = 0;
          double o15_1 = 0;
          double o15_5 = 0;
          double o15_9 = 0;
          double o16_1 = 0;
          double o16_5 = 0;
          double o16_9 = 0;
          double o17_1 = 0;
          double o17_5 = 0;
          double o17_9 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 113;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g1_0 = 0;
            double g1_1 = 0;
            double g1_2 = 0;
            double g1_3 = 0;
            double g1_4 = 0;
            double g1_5 = 0;
            double g1_6 = 0;
            double g1_7 = 0;
            double g1_8 = 0;
            double g1_9 = 0;
            double g1_10 = 0;
            double g1_11 = 0;
            double g1_12 = 0;
            double g1_13 = 0;
            double g1_14 = 0;
            double g1_15 = 0;
            double g1_16 = 0;
            double g1_17 = 0;
            double g1_18 = 0;
            double g1_19 = 0;
            double g5_0 = 0;
            double g5_1 = 0;
            double g5_2 = 0;
            double g5_3 = 0;
            double g5_4 = 0;
            double g5_5 = 0;
            double g5_6 = 0;
            double g5_7 = 0;
            double g5_8 = 0;
            double g5_9 = 0;
            double g5_10 = 0;
            double g5_11 = 0;
            double g5_12 = 0;
            double g5_13 = 0;
            double g5_14 = 0;
            double g5_15 = 0;
            double g5_16 = 0;
            double g5_17 = 0;
            double g5_18 = 0;
            double g5_19 = 0;
            double g9_0 = 0;
            double g9_1 = 0;
            double g9_2 = 0;
            double g9_3 = 0;
            double g9_4 = 0;
            double g9_5 = 0;
            double g9_6 = 0;
            double g9_7 = 0;
            double g9_8 = 0;
            double g9_9 = 0;
            double g9_10 = 0;
            double g9_11 = 0;
            double g9_12 = 0;
            double g9_13 = 0;
            double g9_14 = 0;
            double g9_15 = 0;
            double g9_16 = 0;
            double g9_17 = 0;
            double g9_18 = 0;
            double g9_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[6];
              sqb::boys<5>(T, a.boys_tab, F);
              const double s0 = TWO_PI_2_5 * rs;
              const double m2a = -2.0 * alpha;
              double w = s0;
              const double b0 = w * F[0];
              w *= m2a;
              const double b1 = w * F[1];
              w *= m2a;
              const double b2 = w * F[2];
              w *= m2a;
              const double b3 = w * F[3];
              w *= m2a;
              const double b4 = w * F[4];
              w *= m2a;
              const double b5 = w * F[5];
              const double ek1_0 = kj[7 * kS];
              const double ek1_1 = -kj[8 * kS];
              const double ek1_2 = kj[9 * kS];
              const double ek5_0 = kj[20 * kS];
              const double ek5_1 = -kj[21 * kS];
              const double ek5_2 = -kj[22 * kS];
              const double ek5_3 = kj[23 * kS];
              const double ek9_0 = kj[33 * kS];
              const double ek9_1 = -kj[34 * kS];
              const double ek9_2 = -kj[35 * kS];
              const double ek9_3 = kj[36 * kS];
              g1_0 = fma(ek1_0, b0, g1_0);
              g5_0 = fma(ek5_0, b0, g5_0);
              g9_0 = fma(ek9_0, b0, g9_0);
              const double r0_0_0_1 = Z * b1;
              g1_1 = fma(ek1_0, r0_0_0_1, g1_1);
              g5_1 = fma(ek5_0, r0_0_0_1, g5_1);
              g9_1 = fma(ek9_0, r0_0_0_1, g9_1);
              g9_0 = fma(ek9_1, r0_0_0_1, g9_0);
              const double r0_0_1_0 = Y * b1;
              g1_2 = fma(ek1_0, r0_0_1_0, g1_2);
              g5_2 = fma(ek5_0, r0_0_1_0, g5_2);
              g5_0 = fma(ek5_1, r0_0_1_0, g5_0);
              g9_2 = fma(ek9_0, r0_0_1_0, g9_2);
              const double r0_1_0_0 = X * b1;
              g1_3 = fma(ek1_0, r0_1_0_0, g1_3);
              g1_0 = fma(ek1_1, r0_1_0_0, g1_0);
              g5_3 = fma(ek5_0, r0_1_0_0, g5_3);
              g5_0 = fma(ek5_2, r0_1_0_0, g5_0);
              g9_3 = fma(ek9_0, r0_1_0_0, g9_3);
              g9_0 = fma(ek9_2, r0_1_0_0, g9_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g1_4 = fma(ek1_0, r0_0_0_2, g1_4);
              g5_4 = fma(ek5_0, r0_0_0_2, g5_4);
              g9_4 = fma(ek9_0, r0_0_0_2, g9_4);
              g9_1 = fma(ek9_1, r0_0_0_2, g9_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g1_5 = fma(ek1_0, r0_0_1_1, g1_5);
              g5_5 = fma(ek5_0, r0_0_1_1, g5_5);
              g5_1 = fma(ek5_1, r0_0_1_1, g5_1);
              g9_5 = fma(ek9_0, r0_0_1_1, g9_5);
              g9_2 = fma(ek9_1, r0_0_1_1, g9_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g1_6 = fma(ek1_0, r0_0_2_0, g1_6);
              g5_6 = fma(ek5_0, r0_0_2_0, g5_6);
              g5_2 = fma(ek5_1, r0_0_2_0, g5_2);
              g9_6 = fma(ek9_0, r0_0_2_0, g9_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g1_7 = fma(ek1_0, r0_1_0_1, g1_7);
              g1_1 = fma(ek1_1, r0_1_0_1, g1_1);
              g5_7 = fma(ek5_0, r0_1_0_1, g5_7);
              g5_1 = fma(ek5_2, r0_1_0_1, g5_1);
              g9_7 = fma(ek9_0, r0_1_0_1, g9_7);
              g9_3 = fma(ek9_1, r0_1_0_1, g9_3);
              g9_1 = fma(ek9_2, r0_1_0_1, g9_1);
              g9_0 = fma(ek9_3, r0_1_0_1, g9_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g1_8 = fma(ek1_0, r0_1_1_0, g1_8);
              g1_2 = fma(ek1_1, r0_1_1_0, g1_2);
              g5_8 = fma(ek5_0, r0_1_1_0, g5_8);
              g5_3 = fma(ek5_1, r0_1_1_0, g5_3);
              g5_2 = fma(ek5_2, r0_1_1_0, g5_2);
              g5_0 = fma(ek5_3, r0_1_1_0, g5_0);
              g9_8 = fma(ek9_0, r0_1_1_0, g9_8);
              g9_2 = fma(ek9_2, r0_1_1_0, g9_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g1_9 = fma(ek1_0, r0_2_0_0, g1_9);
              g1_3 = fma(ek1_1, r0_2_0_0, g1_3);
              g1_0 = fma(ek1_2, r0_2_0_0, g1_0);
              g5_9 = fma(ek5_0, r0_2_0_0, g5_9);
              g5_3 = fma(ek5_2, r0_2_0_0, g5_3);
              g9_9 = fma(ek9_0, r0_2_0_0, g9_9);
              g9_3 = fma(ek9_2, r0_2_0_0, g9_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g1_10 = fma(ek1_0, r0_0_0_3, g1_10);
              g5_10 = fma(ek5_0, r0_0_0_3, g5_10);
              g9_10 = fma(ek9_0, r0_0_0_3, g9_10);
              g9_4 = fma(ek9_1, r0_0_0_3, g9_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g1_11 = fma(ek1_0, r0_0_1_2, g1_11);
              g5_11 = fma(ek5_0, r0_0_1_2, g5_11);
              g5_4 = fma(ek5_1, r0_0_1_2, g5_4);
              g9_11 = fma(ek9_0, r0_0_1_2, g9_11);
              g9_5 = fma(ek9_1, r0_0_1_2, g9_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g1_12 = fma(ek1_0, r0_0_2_1, g1_12);
              g5_12 = fma(ek5_0, r0_0_2_1, g5_12);
              g5_5 = fma(ek5_1, r0_0_2_1, g5_5);
              g9_12 = fma(ek9_0, r0_0_2_1, g9_12);
              g9_6 = fma(ek9_1, r0_0_2_1, g9_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g1_13 = fma(ek1_0, r0_0_3_0, g1_13);
              g5_13 = fma(ek5_0, r0_0_3_0, g5_13);
              g5_6 = fma(ek5_1, r0_0_3_0, g5_6);
              g9_13 = fma(ek9_0, r0_0_3_0, g9_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g1_14 = fma(ek1_0, r0_1_0_2, g1_14);
              g1_4 = fma(ek1_1, r0_1_0_2, g1_4);
              g5_14 = fma(ek5_0, r0_1_0_2, g5_14);
              g5_4 = fma(ek5_2, r0_1_0_2, g5_4);
              g9_14 = fma(ek9_0, r0_1_0_2, g9_14);
              g9_7 = fma(ek9_1, r0_1_0_2, g9_7);
              g9_4 = fma(ek9_2, r0_1_0_2, g9_4);
              g9_1 = fma(ek9_3, r0_1_0_2, g9_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g1_15 = fma(ek1_0, r0_1_1_1, g1_15);
              g1_5 = fma(ek1_1, r0_1_1_1, g1_5);
              g5_15 = fma(ek5_0, r0_1_1_1, g5_15);
              g5_7 = fma(ek5_1, r0_1_1_1, g5_7);
              g5_5 = fma(ek5_2, r0_1_1_1, g5_5);
              g5_1 = fma(ek5_3, r0_1_1_1, g5_1);
              g9_15 = fma(ek9_0, r0_1_1_1, g9_15);
              g9_8 = fma(ek9_1, r0_1_1_1, g9_8);
              g9_5 = fma(ek9_2, r0_1_1_1, g9_5);
              g9_2 = fma(ek9_3, r0_1_1_1, g9_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g1_16 = fma(ek1_0, r0_1_2_0, g1_16);
              g1_6 = fma(ek1_1, r0_1_2_0, g1_6);
              g5_16 = fma(ek5_0, r0_1_2_0, g5_16);
              g5_8 = fma(ek5_1, r0_1_2_0, g5_8);
              g5_6 = fma(ek5_2, r0_1_2_0, g5_6);
              g5_2 = fma(ek5_3, r0_1_2_0, g5_2);
              g9_16 = fma(ek9_0, r0_1_2_0, g9_16);
              g9_6 = fma(ek9_2, r0_1_2_0, g9_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g1_17 = fma(ek1_0, r0_2_0_1, g1_17);
              g1_7 = fma(ek1_1, r0_2_0_1, g1_7);
              g1_1 = fma(ek1_2, r0_2_0_1, g1_1);
              g5_17 = fma(ek5_0, r0_2_0_1, g5_17);
              g5_7 = fma(ek5_2, r0_2_0_1, g5_7);
              g9_17 = fma(ek9_0, r0_2_0_1, g9_17);
              g9_9 = fma(ek9_1, r0_2_0_1, g9_9);
              g9_7 = fma(ek9_2, r0_2_0_1, g9_7);
              g9_3 = fma(ek9_3, r0_2_0_1, g9_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g1_18 = fma(ek1_0, r0_2_1_0, g1_18);
              g1_8 = fma(ek1_1, r0_2_1_0, g1_8);
              g1_2 = fma(ek1_2, r0_2_1_0, g1_2);
              g5_18 = fma(ek5_0, r0_2_1_0, g5_18);
              g5_9 = fma(ek5_1, r0_2_1_0, g5_9);
              g5_8 = fma(ek5_2, r0_2_1_0, g5_8);
              g5_3 = fma(ek5_3, r0_2_1_0, g5_3);
              g9_18 = fma(ek9_0, r0_2_1_0, g9_18);
              g9_8 = fma(ek9_2, r0_2_1_0, g9_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g1_19 = fma(ek1_0, r0_3_0_0, g1_19);
              g1_9 = fma(ek1_1, r0_3_0_0, g1_9);
              g1_3 = fma(ek1_2, r0_3_0_0, g1_3);
              g5_19 = fma(ek5_0, r0_3_0_0, g5_19);
              g5_9 = fma(ek5_2, r0_3_0_0, g5_9);
              g9_19 = fma(ek9_0, r0_3_0_0, g9_19);
              g9_9 = fma(ek9_2, r0_3_0_0, g9_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g9_10 = fma(ek9_1, r0_0_0_4, g9_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g5_10 = fma(ek5_1, r0_0_1_3, g5_10);
              g9_11 = fma(ek9_1, r0_0_1_3, g9_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g5_11 = fma(ek5_1, r0_0_2_2, g5_11);
              g9_12 = fma(ek9_1, r0_0_2_2, g9_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g5_12 = fma(ek5_1, r0_0_3_1, g5_12);
              g9_13 = fma(ek9_1, r0_0_3_1, g9_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g5_13 = fma(ek5_1, r0_0_4_0, g5_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g1_10 = fma(ek1_1, r0_1_0_3, g1_10);
              g5_10 = fma(ek5_2, r0_1_0_3, g5_10);
              g9_14 = fma(ek9_1, r0_1_0_3, g9_14);
              g9_10 = fma(ek9_2, r0_1_0_3, g9_10);
              g9_4 = fma(ek9_3, r0_1_0_3, g9_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g1_11 = fma(ek1_1, r0_1_1_2, g1_11);
              g5_14 = fma(ek5_1, r0_1_1_2, g5_14);
              g5_11 = fma(ek5_2, r0_1_1_2, g5_11);
              g5_4 = fma(ek5_3, r0_1_1_2, g5_4);
              g9_15 = fma(ek9_1, r0_1_1_2, g9_15);
              g9_11 = fma(ek9_2, r0_1_1_2, g9_11);
              g9_5 = fma(ek9_3, r0_1_1_2, g9_5);
              const double r0_1_2_1 = X * r1_0_2_1;
              g1_12 = fma(ek1_1, r0_1_2_1, g1_12);
              g5_15 = fma(ek5_1, r0_1_2_1, g5_15);
              g5_12 = fma(ek5_2, r0_1_2_1, g5_12);
              g5_5 = fma(ek5_3, r0_1_2_1, g5_5);
              g9_16 = fma(ek9_1, r0_1_2_1, g9_16);
              g9_12 = fma(ek9_2, r0_1_2_1, g9_12);
              g9_6 = fma(ek9_3, r0_1_2_1, g9_6);
              const double r0_1_3_0 = X * r1_0_3_0;
              g1_13 = fma(ek1_1, r0_1_3_0, g1_13);
              g5_16 = fma(ek5_1, r0_1_3_0, g5_16);
              g5_13 = fma(ek5_2, r0_1_3_0, g5_13);
              g5_6 = fma(ek5_3, r0_1_3_0, g5_6);
              g9_13 = fma(ek9_2, r0_1_3_0, g9_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g1_14 = fma(ek1_1, r0_2_0_2, g1_14);
              g1_4 = fma(ek1_2, r0_2_0_2, g1_4);
              g5_14 = fma(ek5_2, r0_2_0_2, g5_14);
              g9_17 = fma(ek9_1, r0_2_0_2, g9_17);
              g9_14 = fma(ek9_2, r0_2_0_2, g9_14);
              g9_7 = fma(ek9_3, r0_2_0_2, g9_7);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g1_15 = fma(ek1_1, r0_2_1_1, g1_15);
              g1_5 = fma(ek1_2, r0_2_1_1, g1_5);
              g5_17 = fma(ek5_1, r0_2_1_1, g5_17);
              g5_15 = fma(ek5_2, r0_2_1_1, g5_15);
              g5_7 = fma(ek5_3, r0_2_1_1, g5_7);
              g9_18 = fma(ek9_1, r0_2_1_1, g9_18);
              g9_15 = fma(ek9_2, r0_2_1_1, g9_15);
              g9_8 = fma(ek9_3, r0_2_1_1, g9_8);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g1_16 = fma(ek1_1, r0_2_2_0, g1_16);
              g1_6 = fma(ek1_2, r0_2_2_0, g1_6);
              g5_18 = fma(ek5_1, r0_2_2_0, g5_18);
              g5_16 = fma(ek5_2, r0_2_2_0, g5_16);
              g5_8 = fma(ek5_3, r0_2_2_0, g5_8);
              g9_16 = fma(ek9_2, r0_2_2_0, g9_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g1_17 = fma(ek1_1, r0_3_0_1, g1_17);
              g1_7 = fma(ek1_2, r0_3_0_1, g1_7);
              g5_17 = fma(ek5_2, r0_3_0_1, g5_17);
              g9_19 = fma(ek9_1, r0_3_0_1, g9_19);
              g9_17 = fma(ek9_2, r0_3_0_1, g9_17);
              g9_9 = fma(ek9_3, r0_3_0_1, g9_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g1_18 = fma(ek1_1, r0_3_1_0, g1_18);
              g1_8 = fma(ek1_2, r0_3_1_0, g1_8);
              g5_19 = fma(ek5_1, r0_3_1_0, g5_19);
              g5_18 = fma(ek5_2, r0_3_1_0, g5_18);
              g5_9 = fma(ek5_3, r0_3_1_0, g5_9);
              g9_18 = fma(ek9_2, r0_3_1_0, g9_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g1_19 = fma(ek1_1, r0_4_0_0, g1_19);
              g1_9 = fma(ek1_2, r0_4_0_0, g1_9);
              g5_19 = fma(ek5_2, r0_4_0_0, g5_19);
              g9_19 = fma(ek9_2, r0_4_0_0, g9_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_1_0_4 = X * r1_0_0_4;
              g9_10 = fma(ek9_3, r0_1_0_4, g9_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g5_10 = fma(ek5_3, r0_1_1_3, g5_10);
              g9_11 = fma(ek9_3, r0_1_1_3, g9_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g5_11 = fma(ek5_3, r0_1_2_2, g5_11);
              g9_12 = fma(ek9_3, r0_1_2_2, g9_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g5_12 = fma(ek5_3, r0_1_3_1, g5_12);
              g9_13 = fma(ek9_3, r0_1_3_1, g9_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g5_13 = fma(ek5_3, r0_1_4_0, g5_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g1_10 = fma(ek1_2, r0_2_0_3, g1_10);
              g9_14 = fma(ek9_3, r0_2_0_3, g9_14);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g1_11 = fma(ek1_2, r0_2_1_2, g1_11);
              g5_14 = fma(ek5_3, r0_2_1_2, g5_14);
              g9_15 = fma(ek9_3, r0_2_1_2, g9_15);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g1_12 = fma(ek1_2, r0_2_2_1, g1_12);
              g5_15 = fma(ek5_3, r0_2_2_1, g5_15);
              g9_16 = fma(ek9_3, r0_2_2_1, g9_16);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g1_13 = fma(ek1_2, r0_2_3_0, g1_13);
              g5_16 = fma(ek5_3, r0_2_3_0, g5_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g1_14 = fma(ek1_2, r0_3_0_2, g1_14);
              g9_17 = fma(ek9_3, r0_3_0_2, g9_17);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g1_15 = fma(ek1_2, r0_3_1_1, g1_15);
              g5_17 = fma(ek5_3, r0_3_1_1, g5_17);
              g9_18 = fma(ek9_3, r0_3_1_1, g9_18);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g1_16 = fma(ek1_2, r0_3_2_0, g1_16);
              g5_18 = fma(ek5_3, r0_3_2_0, g5_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g1_17 = fma(ek1_2, r0_4_0_1, g1_17);
              g9_19 = fma(ek9_3, r0_4_0_1, g9_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g1_18 = fma(ek1_2, r0_4_1_0, g1_18);
              g5_19 = fma(ek5_3, r0_4_1_0, g5_19);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g1_19 = fma(ek1_2, r0_5_0_0, g1_19);
            }
            { const double eb = bi[5];
              o0_1 = fma(eb, g1_0, o0_1);
              o0_5 = fma(eb, g5_0, o0_5);
              o0_9 = fma(eb, g9_0, o0_9);
            }
            { const double eb = bi[6];
              o0_1 = fma(eb, g1_3, o0_1);
              o0_5 = fma(eb, g5_3, o0_5);
              o0_9 = fma(eb, g9_3, o0_9);
            }
            { const double eb = bi[7];
              o0_1 = fma(eb, g1_9, o0_1);
              o0_5 = fma(eb, g5_9, o0_5);
              o0_9 = fma(eb, g9_9, o0_9);
            }
            { const double eb = bi[8];
              o0_1 = fma(eb, g1_19, o0_1);
              o0_5 = fma(eb, g5_19, o0_5);
              o0_9 = fma(eb, g9_19, o0_9);
            }
            { const double eb = bi[9];
              o1_1 = fma(eb, g1_0, o1_1);
              o1_5 = fma(eb, g5_0, o1_5);
              o1_9 = fma(eb, g9_0, o1_9);
            }
            { const double eb = bi[10];
              o1_1 = fma(eb, g1_2, o1_1);
              o1_5 = fma(eb, g5_2, o1_5);
              o1_9 = fma(eb, g9_2, o1_9);
            }
            { const double eb = bi[11];
              o1_1 = fma(eb, g1_3, o1_1);
              o1_5 = fma(eb, g5_3, o1_5);
              o1_9 = fma(eb, g9_3, o1_9);
            }
            { const double eb = bi[12];
              o1_1 = fma(eb, g1_8, o1_1);
              o1_5 = fma(eb, g5_8, o1_5);
              o1_9 = fma(eb, g9_8, o1_9);
            }
            { const double eb = bi[13];
              o1_1 = fma(eb, g1_9, o1_1);
              o1_5 = fma(eb, g5_9, o1_5);
              o1_9 = fma(eb, g9_9, o1_9);
            }
            { const double eb = bi[14];
              o1_1 = fma(eb, g1_18, o1_1);
              o1_5 = fma(eb, g5_18, o1_5);
              o1_9 = fma(eb, g9_18, o1_9);
            }
            { const double eb = bi[15];
              o2_1 = fma(eb, g1_0, o2_1);
              o2_5 = fma(eb, g5_0, o2_5);
              o2_9 = fma(eb, g9_0, o2_9);
            }
            { const double eb = bi[16];
              o2_1 = fma(eb, g1_1, o2_1);
              o2_5 = fma(eb, g5_1, o2_5);
              o2_9 = fma(eb, g9_1, o2_9);
            }
            { const double eb = bi[17];
              o2_1 = fma(eb, g1_3, o2_1);
              o2_5 = fma(eb, g5_3, o2_5);
              o2_9 = fma(eb, g9_3, o2_9);
            }
            { const double eb = bi[18];
              o2_1 = fma(eb, g1_7, o2_1);
              o2_5 = fma(eb, g5_7, o2_5);
              o2_9 = fma(eb, g9_7, o2_9);
            }
            { const double eb = bi[19];
              o2_1 = fma(eb, g1_9, o2_1);
              o2_5 = fma(eb, g5_9, o2_5);
              o2_9 = fma(eb, g9_9, o2_9);
            }
            { const double eb = bi[20];
              o2_1 = fma(eb, g1_17, o2_1);
              o2_5 = fma(eb, g5_17, o2_5);
              o2_9 = fma(eb, g9_17, o2_9);
            }
            { const double eb = bi[21];
              o3_1 = fma(eb, g1_0, o3_1);
              o3_5 = fma(eb, g5_0, o3_5);
              o3_9 = fma(eb, g9_0, o3_9);
            }
            { const double eb = bi[22];
              o3_1 = fma(eb, g1_2, o3_1);
              o3_5 = fma(eb, g5_2, o3_5);
              o3_9 = fma(eb, g9_2, o3_9);
            }
            { const double eb = bi[23];
              o3_1 = fma(eb, g1_6, o3_1);
              o3_5 = fma(eb, g5_6, o3_5);
              o3_9 = fma(eb, g9_6, o3_9);
            }
            { const double eb = bi[24];
              o3_1 = fma(eb, g1_3, o3_1);
              o3_5 = fma(eb, g5_3, o3_5);
              o3_9 = fma(eb, g9_3, o3_9);
            }
            { const double eb = bi[25];
              o3_1 = fma(eb, g1_8, o3_1);
              o3_5 = fma(eb, g5_8, o3_5);
              o3_9 = fma(eb, g9_8, o3_9);
            }
            { const double eb = bi[26];
              o3_1 = fma(eb, g1_16, o3_1);
              o3_5 = fma(eb, g5_16, o3_5);
              o3_9 = fma(eb, g9_16, o3_9);
            }
            { const double eb = bi[27];
              o4_1 = fma(eb, g1_0, o4_1);
              o4_5 = fma(eb, g5_0, o4_5);
              o4_9 = fma(eb, g9_0, o4_9);
            }
            { const double eb = bi[28];
              o4_1 = fma(eb, g1_2, o4_1);
              o4_5 = fma(eb, g5_2, o4_5);
              o4_9 = fma(eb, g9_2, o4_9);
            }
            { const double eb = bi[29];
              o4_1 = fma(eb, g1_6, o4_1);
              o4_5 = fma(eb, g5_6, o4_5);
              o4_9 = fma(eb, g9_6, o4_9);
            }
            { const double eb = bi[30];
              o4_1 = fma(eb, g1_13, o4_1);
              o4_5 = fma(eb, g5_13, o4_5);
              o4_9 = fma(eb, g9_13, o4_9);
            }
            { const double eb = bi[31];
              o5_1 = fma(eb, g1_0, o5_1);
              o5_5 = fma(eb, g5_0, o5_5);
              o5_9 = fma(eb, g9_0, o5_9);
            }
            { const double eb = bi[32];
              o5_1 = fma(eb, g1_1, o5_1);
              o5_5 = fma(eb, g5_1, o5_5);
              o5_9 = fma(eb, g9_1, o5_9);
            }
            { const double eb = bi[33];
              o5_1 = fma(eb, g1_2, o5_1);
              o5_5 = fma(eb, g5_2, o5_5);
              o5_9 = fma(eb, g9_2, o5_9);
            }
            { const double eb = bi[34];
              o5_1 = fma(eb, g1_5, o5_1);
              o5_5 = fma(eb, g5_5, o5_5);
              o5_9 = fma(eb, g9_5, o5_9);
            }
            { const double eb = bi[35];
              o5_1 = fma(eb, g1_6, o5_1);
              o5_5 = fma(eb, g5_6, o5_5);
              o5_9 = fma(eb, g9_6, o5_9);
            }
            { const double eb = bi[36];
              o5_1 = fma(eb, g1_12, o5_1);
              o5_5 = fma(eb, g5_12, o5_5);
              o5_9 = fma(eb, g9_12, o5_9);
            }
            { const double eb = bi[37];
              o6_1 = fma(eb, g1_0, o6_1);
              o6_5 = fma(eb, g5_0, o6_5);
              o6_9 = fma(eb, g9_0, o6_9);
            }
            { const double eb = bi[38];
              o6_1 = fma(eb, g1_1, o6_1);
              o6_5 = fma(eb, g5_1, o6_5);
              o6_9 = fma(eb, g9_1, o6_9);
            }
            { const double eb = bi[39];
              o6_1 = fma(eb, g1_4, o6_1);
              o6_5 = fma(eb, g5_4, o6_5);
              o6_9 = fma(eb, g9_4, o6_9);
            }
            { const double eb = bi[40];
              o6_1 = fma(eb, g1_3, o6_1);
              o6_5 = fma(eb, g5_3, o6_5);
              o6_9 = fma(eb, g9_3, o6_9);
            }
            { const double eb = bi[41];
              o6_1 = fma(eb, g1_7, o6_1);
              o6_5 = fma(eb, g5_7, o6_5);
              o6_9 = fma(eb, g9_7, o6_9);
            }
            { const double eb = bi[42];
              o6_1 = fma(eb, g1_14, o6_1);
              o6_5 = fma(eb, g5_14, o6_5);
              o6_9 = fma(eb, g9_14, o6_9);
            }
            { const double eb = bi[43];
              o7_1 = fma(eb, g1_0, o7_1);
              o7_5 = fma(eb, g5_0, o7_5);
              o7_9 = fma(eb, g9_0, o7_9);
            }
            { const double eb = bi[44];
              o7_1 = fma(eb, g1_1, o7_1);
              o7_5 = fma(eb, g5_1, o7_5);
              o7_9 = fma(eb, g9_1, o7_9);
            }
            { const double eb = bi[45];
              o7_1 = fma(eb, g1_4, o7_1);
              o7_5 = fma(eb, g5_4, o7_5);
              o7_9 = fma(eb, g9_4, o7_9);
            }
            { const double eb = bi[46];
              o7_1 = fma(eb, g1_2, o7_1);
              o7_5 = fma(eb, g5_2, o7_5);
              o7_9 = fma(eb, g9_2, o7_9);
            }
            { const double eb = bi[47];
              o7_1 = fma(eb, g1_5, o7_1);
              o7_5 = fma(eb, g5_5, o7_5);
              o7_9 = fma(eb, g9_5, o7_9);
            }
            { const double eb = bi[48];
              o7_1 = fma(eb, g1_11, o7_1);
              o7_5 = fma(eb, g5_11, o7_5);
              o7_9 = fma(eb, g9_11, o7_9);
            }
            { const double eb = bi[49];
              o8_1 = fma(eb, g1_0, o8_1);
              o8_5 = fma(eb, g5_0, o8_5);
              o8_9 = fma(eb, g9_0, o8_9);
            }
            { const double eb = bi[50];
              o8_1 = fma(eb, g1_1, o8_1);
              o8_5 = fma(eb, g5_1, o8_5);
              o8_9 = fma(eb, g9_1, o8_9);
            }
            { const double eb = bi[51];
              o8_1 = fma(eb, g1_4, o8_1);
              o8_5 = fma(eb, g5_4, o8_5);
              o8_9 = fma(eb, g9_4, o8_9);
            }
            { const double eb = bi[52];
              o8_1 = fma(eb, g1_10, o8_1);
              o8_5 = fma(eb, g5_10, o8_5);
              o8_9 = fma(eb, g9_10, o8_9);
            }
            { const double eb = bi[53];
              o9_1 = fma(eb, g1_0, o9_1);
              o9_5 = fma(eb, g5_0, o9_5);
              o9_9 = fma(eb, g9_0, o9_9);
            }
            { const double eb = bi[54];
              o9_1 = fma(eb, g1_2, o9_1);
              o9_5 = fma(eb, g5_2, o9_5);
              o9_9 = fma(eb, g9_2, o9_9);
            }
            { const double eb = bi[55];
              o9_1 = fma(eb, g1_3, o9_1);
              o9_5 = fma(eb, g5_3, o9_5);
              o9_9 = fma(eb, g9_3, o9_9);
            }
            { const double eb = bi[56];
              o9_1 = fma(eb, g1_8, o9_1);
              o9_5 = fma(eb, g5_8, o9_5);
              o9_9 = fma(eb, g9_8, o9_9);
            }
            { const double eb = bi[57];
              o9_1 = fma(eb, g1_9, o9_1);
              o9_5 = fma(eb, g5_9, o9_5);
              o9_9 = fma(eb, g9_9, o9_9);
            }
            { const double eb = bi[58];
              o9_1 = fma(eb, g1_18, o9_1);
              o9_5 = fma(eb, g5_18, o9_5);
              o9_9 = fma(eb, g9_18, o9_9);
            }
            { const double eb = bi[59];
              o10_1 = fma(eb, g1_0, o10_1);
              o10_5 = fma(eb, g5_0, o10_5);
              o10_9 = fma(eb, g9_0, o10_9);
            }
            { const double eb = bi[60];
              o10_1 = fma(eb, g1_2, o10_1);
              o10_5 = fma(eb, g5_2, o10_5);
              o10_9 = fma(eb, g9_2, o10_9);
            }
            { const double eb = bi[61];
              o10_1 = fma(eb, g1_6, o10_1);
              o10_5 = fma(eb, g5_6, o10_5);
              o10_9 = fma(eb, g9_6, o10_9);
            }
            { const double eb = bi[62];
              o10_1 = fma(eb, g1_3, o10_1);
              o10_5 = fma(eb, g5_3, o10_5);
              o10_9 = fma(eb, g9_3, o10_9);
            }
            { const double eb = bi[63];
              o10_1 = fma(eb, g1_8, o10_1);
              o10_5 = fma(eb, g5_8, o10_5);
              o10_9 = fma(eb, g9_8, o10_9);
            }
            { const double eb = bi[64];
              o10_1 = fma(eb, g1_16, o10_1);
              o10_5 = fma(eb, g5_16, o10_5);
              o10_9 = fma(eb, g9_16, o10_9);
            }
            { const double eb = bi[65];
              o11_1 = fma(eb, g1_0, o11_1);
              o11_5 = fma(eb, g5_0, o11_5);
              o11_9 = fma(eb, g9_0, o11_9);
            }
            { const double eb = bi[66];
              o11_1 = fma(eb, g1_1, o11_1);
              o11_5 = fma(eb, g5_1, o11_5);
              o11_9 = fma(eb, g9_1, o11_9);
            }
            { const double eb = bi[67];
              o11_1 = fma(eb, g1_2, o11_1);
              o11_5 = fma(eb, g5_2, o11_5);
              o11_9 = fma(eb, g9_2, o11_9);
            }
            { const double eb = bi[68];
              o11_1 = fma(eb, g1_5, o11_1);
              o11_5 = fma(eb, g5_5, o11_5);
              o11_9 = fma(eb, g9_5, o11_9);
            }
            { const double eb = bi[69];
              o11_1 = fma(eb, g1_3, o11_1);
              o11_5 = fma(eb, g5_3, o11_5);
              o11_9 = fma(eb, g9_3, o11_9);
            }
            { const double eb = bi[70];
              o11_1 = fma(eb, g1_7, o11_1);
              o11_5 = fma(eb, g5_7, o11_5);
              o11_9 = fma(eb, g9_7, o11_9);
            }
            { const double eb = bi[71];
              o11_1 = fma(eb, g1_8, o11_1);
              o11_5 = fma(eb, g5_8, o11_5);
              o11_9 = fma(eb, g9_8, o11_9);
            }
            { const double eb = bi[72];
              o11_1 = fma(eb, g1_15, o11_1);
              o11_5 = fma(eb, g5_15, o11_5);
              o11_9 = fma(eb, g9_15, o11_9);
            }
            { const double eb = bi[73];
              o12_1 = fma(eb, g1_0, o12_1);
              o12_5 = fma(eb, g5_0, o12_5);
              o12_9 = fma(eb, g9_0, o12_9);
            }
            { const double eb = bi[74];
              o12_1 = fma(eb, g1_1, o12_1);
              o12_5 = fma(eb, g5_1, o12_5);
              o12_9 = fma(eb, g9_1, o12_9);
            }
            { const double eb = bi[75];
              o12_1 = fma(eb, g1_3, o12_1);
              o12_5 = fma(eb, g5_3, o12_5);
              o12_9 = fma(eb, g9_3, o12_9);
            }
            { const double eb = bi[76];
              o12_1 = fma(eb, g1_7, o12_1);
              o12_5 = fma(eb, g5_7, o12_5);
              o12_9 = fma(eb, g9_7, o12_9);
            }
            { const double eb = bi[77];
              o12_1 = fma(eb, g1_9, o12_1);
              o12_5 = fma(eb, g5_9, o12_5);
              o12_9 = fma(eb, g9_9, o12_9);
            }
            { const double eb = bi[78];
              o12_1 = fma(eb, g1_17, o12_1);
              o12_5 = fma(eb, g5_17, o12_5);
              o12_9 = fma(eb, g9_17, o12_9);
            }
            { const double eb = bi[79];
              o13_1 = fma(eb, g1_0, o13_1);
              o13_5 = fma(eb, g5_0, o13_5);
              o13_9 = fma(eb, g9_0, o13_9);
            }
            { const double eb = bi[80];
              o13_1 = fma(eb, g1_1, o13_1);
              o13_5 = fma(eb, g5_1, o13_5);
              o13_9 = fma(eb, g9_1, o13_9);
            }
            { const double eb = bi[81];
              o13_1 = fma(eb, g1_2, o13_1);
              o13_5 = fma(eb, g5_2, o13_5);
              o13_9 = fma(eb, g9_2, o13_9);
            }
            { const double eb = bi[82];
              o13_1 = fma(eb, g1_5, o13_1);
              o13_5 = fma(eb, g5_5, o13_5);
              o13_9 = fma(eb, g9_5, o13_9);
            }
            { const double eb = bi[83];
              o13_1 = fma(eb, g1_3, o13_1);
              o13_5 = fma(eb, g5_3, o13_5);
              o13_9 = fma(eb, g9_3, o13_9);
            }
            { const double eb = bi[84];
              o13_1 = fma(eb, g1_7, o13_1);
              o13_5 = fma(eb, g5_7, o13_5);
              o13_9 = fma(eb, g9_7, o13_9);
            }
            { const double eb = bi[85];
              o13_1 = fma(eb, g1_8, o13_1);
              o13_5 = fma(eb, g5_8, o13_5);
              o13_9 = fma(eb, g9_8, o13_9);
            }
            { const double eb = bi[86];
              o13_1 = fma(eb, g1_15, o13_1);
              o13_5 = fma(eb, g5_15, o13_5);
              o13_9 = fma(eb, g9_15, o13_9);
            }
            { const double eb = bi[87];
              o14_1 = fma(eb, g1_0, o14_1);
              o14_5 = fma(eb, g5_0, o14_5);
              o14_9 = fma(eb, g9_0, o14_9);
            }
            { const double eb = bi[88];
              o14_1 = fma(eb, g1_1, o14_1);
              o14_5 = fma(eb, g5_1, o14_5);
              o14_9 = fma(eb, g9_1, o14_9);
            }
            { const double eb = bi[89];
              o14_1 = fma(eb, g1_4, o14_1);
              o14_5 = fma(eb, g5_4, o14_5);
              o14_9 = fma(eb, g9_4, o14_9);
            }
            { const double eb = bi[90];
              o14_1 = fma(eb, g1_3, o14_1);
              o14_5 = fma(eb, g5_3, o14_5);
              o14_9 = fma(eb, g9_3, o14_9);
            }
            { const double eb = bi[91];
              o14_1 = fma(eb, g1_7, o14_1);
              o14_5 = fma(eb, g5_7, o14_5);
              o14_9 = fma(eb, g9_7, o14_9);
            }
            { const double eb = bi[92];
              o14_1 = fma(eb, g1_14, o14_1);
              o14_5 = fma(eb, g5_14, o14_5);
              o14_9 = fma(eb, g9_14, o14_9);
            }
            { const double eb = bi[93];
              o15_1 = fma(eb, g1_0, o15_1);
              o15_5 = fma(eb, g5_0, o15_5);
              o15_9 = fma(eb, g9_0, o15_9);
            }
            { const double eb = bi[94];
              o15_1 = fma(eb, g1_1, o15_1);
              o15_5 = fma(eb, g5_1, o15_5);
              o15_9 = fma(eb, g9_1, o15_9);
            }
            { const double eb = bi[95];
              o15_1 = fma(eb, g1_2, o15_1);
              o15_5 = fma(eb, g5_2, o15_5);
              o15_9 = fma(eb, g9_2, o15_9);
            }
            { const double eb = bi[96];
              o15_1 = fma(eb, g1_5, o15_1);
              o15_5 = fma(eb, g5_5, o15_5);
              o15_9 = fma(eb, g9_5, o15_9);
            }
            { const double eb = bi[97];
              o15_1 = fma(eb, g1_3, o15_1);
              o15_5 = fma(eb, g5_3, o15_5);
              o15_9 = fma(eb, g9_3, o15_9);
            }
            { const double eb = bi[98];
              o15_1 = fma(eb, g1_7, o15_1);
              o15_5 = fma(eb, g5_7, o15_5);
              o15_9 = fma(eb, g9_7, o15_9);
            }
            { const double eb = bi[99];
              o15_1 = fma(eb, g1_8, o15_1);
              o15_5 = fma(eb, g5_8, o15_5);
              o15_9 = fma(eb, g9_8, o15_9);
            }
            { const double eb = bi[100];
              o15_1 = fma(eb, g1_15, o15_1);
              o15_5 = fma(eb, g5_15, o15_5);
              o15_9 = fma(eb, g9_15, o15_9);
            }
            { const double eb = bi[101];
              o16_1 = fma(eb, g1_0, o16_1);
              o16_5 = fma(eb, g5_0, o16_5);
              o16_9 = fma(eb, g9_0, o16_9);
            }
            { const double eb = bi[102];
              o16_1 = fma(eb, g1_1, o16_1);
              o16_5 = fma(eb, g5_1, o16_5);
              o16_9 = fma(eb, g9_1, o16_9);
            }
            { const double eb = bi[103];
              o16_1 = fma(eb, g1_2, o16_1);
              o16_5 = fma(eb, g5_2, o16_5);
              o16_9 = fma(eb, g9_2, o16_9);
            }
            { const double eb = bi[104];
              o16_1 = fma(eb, g1_5, o16_1);
              o16_5 = fma(eb, g5_5, o16_5);
              o16_9 = fma(eb, g9_5, o16_9);
            }
            { const double eb = bi[105];
              o16_1 = fma(eb, g1_6, o16_1);
              o16_5 = fma(eb, g5_6, o16_5);
              o16_9 = fma(eb, g9_6, o16_9);
            }
            { const double eb = bi[106];
              o16_1 = fma(eb, g1_12, o16_1);
              o16_5 = fma(eb, g5_12, o16_5);
              o16_9 = fma(eb, g9_12, o16_9);
            }
            { const double eb = bi[107];
              o17_1 = fma(eb, g1_0, o17_1);
              o17_5 = fma(eb, g5_0, o17_5);
              o17_9 = fma(eb, g9_0, o17_9);
            }
            { const double eb = bi[108];
              o17_1 = fma(eb, g1_1, o17_1);
              o17_5 = fma(eb, g5_1, o17_5);
              o17_9 = fma(eb, g9_1, o17_9);
            }
            { const double eb = bi[109];
              o17_1 = fma(eb, g1_4, o17_1);
              o17_5 = fma(eb, g5_4, o17_5);
              o17_9 = fma(eb, g9_4, o17_9);
            }
            { const double eb = bi[110];
              o17_1 = fma(eb, g1_2, o17_1);
              o17_5 = fma(eb, g5_2, o17_5);
              o17_9 = fma(eb, g9_2, o17_9);
            }
            { const double eb = bi[111];
              o17_1 = fma(eb, g1_5, o17_1);
              o17_5 = fma(eb, g5_5, o17_5);
              o17_9 = fma(eb, g9_5, o17_9);
            }
            { const double eb = bi[112];
              o17_1 = fma(eb, g1_11, o17_1);
              o17_5 = fma(eb, g5_11, o17_5);
              o17_9 = fma(eb, g9_11, o17_9);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk1 = PT[(fI + 0) * N + fJ + 1];
            const double ptk5 = PT[(fI + 1) * N + fJ + 1];
            const double ptk9 = PT[(fI + 2) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 1) * N + fQ + 0];
            const double ptb4 = PT[(fP + 1) * N + fQ + 1];
            const double ptb5 = PT[(fP + 1) * N + fQ + 2];
            const double ptb6 = PT[(fP + 2) * N + fQ + 0];
            const double ptb7 = PT[(fP + 2) * N + fQ + 1];
            const double ptb8 = PT[(fP + 2) * N + fQ + 2];
            const double ptb9 = PT[(fP + 3) * N + fQ + 0];
            const double ptb10 = PT[(fP + 3) * N + fQ + 1];
            const double ptb11 = PT[(fP + 3) * N + fQ + 2];
            const double ptb12 = PT[(fP + 4) * N + fQ + 0];
            const double ptb13 = PT[(fP + 4) * N + fQ + 1];
            const double ptb14 = PT[(fP + 4) * N + fQ + 2];
            const double ptb15 = PT[(fP + 5) * N + fQ + 0];
            const double ptb16 = PT[(fP + 5) * N + fQ + 1];
            const double ptb17 = PT[(fP + 5) * N + fQ + 2];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            jab0 += o0_1 * ptk1 + o0_5 * ptk5 + o0_9 * ptk9;
            jab1 += o1_1 * ptk1 + o1_5 * ptk5 + o1_9 * ptk9;
            jab2 += o2_1 * ptk1 + o2_5 * ptk5 + o2_9 * ptk9;
            jab3 += o3_1 * ptk1 + o3_5 * ptk5 + o3_9 * ptk9;
            jab4 += o4_1 * ptk1 + o4_5 * ptk5 + o4_9 * ptk9;
            jab5 += o5_1 * ptk1 + o5_5 * ptk5 + o5_9 * ptk9;
            jab6 += o6_1 * ptk1 + o6_5 * ptk5 + o6_9 * ptk9;
            jab7 += o7_1 * ptk1 + o7_5 * ptk5 + o7_9 * ptk9;
            jab8 += o8_1 * ptk1 + o8_5 * ptk5 + o8_9 * ptk9;
            jab9 += o9_1 * ptk1 + o9_5 * ptk5 + o9_9 * ptk9;
            jab10 += o10_1 * ptk1 + o10_5 * ptk5 + o10_9 * ptk9;
            jab11 += o11_1 * ptk1 + o11_5 * ptk5 + o11_9 * ptk9;
            jab12 += o12_1 * ptk1 + o12_5 * ptk5 + o12_9 * ptk9;
            jab13 += o13_1 * ptk1 + o13_5 * ptk5 + o13_9 * ptk9;
            jab14 += o14_1 * ptk1 + o14_5 * ptk5 + o14_9 * ptk9;
            jab15 += o15_1 * ptk1 + o15_5 * ptk5 + o15_9 * ptk9;
            jab16 += o16_1 * ptk1 + o16_5 * ptk5 + o16_9 * ptk9;
            jab17 += o17_1 * ptk1 + o17_5 * ptk5 + o17_9 * ptk9;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 1, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 1, 2.0 * deg * (o0_5 * ptb0 + o1_5 * ptb1 + o2_5 * ptb2 + o3_5 * ptb3 + o4_5 * ptb4 + o5_5 * ptb5 + o6_5 * ptb6 + o7_5 * ptb7 + o8_5 * ptb8 + o9_5 * ptb9 + o10_5 * ptb10 + o11_5 * ptb11 + o12_5 * ptb12 + o13_5 * ptb13 + o14_5 * ptb14 + o15_5 * ptb15 + o16_5 * ptb16 + o17_5 * ptb17));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 1, 2.0 * deg * (o0_9 * ptb0 + o1_9 * ptb1 + o2_9 * ptb2 + o3_9 * ptb3 + o4_9 * ptb4 + o5_9 * ptb5 + o6_9 * ptb6 + o7_9 * ptb7 + o8_9 * ptb8 + o9_9 * ptb9 + o10_9 * ptb10 + o11_9 * ptb11 + o12_9 * ptb12 + o13_9 * ptb13 + o14_9 * ptb14 + o15_9 * ptb15 + o16_9 * ptb16 + o17_9 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_1 * Abd0_1 + o1_1 * Abd1_1 + o2_1 * Abd2_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_1 * Aad0_1 + o3_1 * Aad1_1 + o6_1 * Aad2_1 + o9_1 * Aad3_1 + o12_1 * Aad4_1 + o15_1 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_1 * Abc0_0 + o0_5 * Abc0_1 + o0_9 * Abc0_2 + o1_1 * Abc1_0 + o1_5 * Abc1_1 + o1_9 * Abc1_2 + o2_1 * Abc2_0 + o2_5 * Abc2_1 + o2_9 * Abc2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_1 * Aac0_0 + o0_5 * Aac0_1 + o0_9 * Aac0_2 + o3_1 * Aac1_0 + o3_5 * Aac1_1 + o3_9 * Aac1_2 + o6_1 * Aac2_0 + o6_5 * Aac2_1 + o6_9 * Aac2_2 + o9_1 * Aac3_0 + o9_5 * Aac3_1 + o9_9 * Aac3_2 + o12_1 * Aac4_0 + o12_5 * Aac4_1 + o12_9 * Aac4_2 + o15_1 * Aac5_0 + o15_5 * Aac5_1 + o15_9 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_5 * Abd0_1 + o1_5 * Abd1_1 + o2_5 * Abd2_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_5 * Aad0_1 + o3_5 * Aad1_1 + o6_5 * Aad2_1 + o9_5 * Aad3_1 + o12_5 * Aad4_1 + o15_5 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_9 * Abd0_1 + o1_9 * Abd1_1 + o2_9 * Abd2_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_9 * Aad0_1 + o3_9 * Aad1_1 + o6_9 * Aad2_1 + o9_9 * Aad3_1 + o12_9 * Aad4_1 + o15_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_1 * Aad0_1 + o4_1 * Aad1_1 + o7_1 * Aad2_1 + o10_1 * Aad3_1 + o13_1 * Aad4_1 + o16_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_1 * Aac0_0 + o1_5 * Aac0_1 + o1_9 * Aac0_2 + o4_1 * Aac1_0 + o4_5 * Aac1_1 + o4_9 * Aac1_2 + o7_1 * Aac2_0 + o7_5 * Aac2_1 + o7_9 * Aac2_2 + o10_1 * Aac3_0 + o10_5 * Aac3_1 + o10_9 * Aac3_2 + o13_1 * Aac4_0 + o13_5 * Aac4_1 + o13_9 * Aac4_2 + o16_1 * Aac5_0 + o16_5 * Aac5_1 + o16_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_5 * Aad0_1 + o4_5 * Aad1_1 + o7_5 * Aad2_1 + o10_5 * Aad3_1 + o13_5 * Aad4_1 + o16_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_9 * Aad0_1 + o4_9 * Aad1_1 + o7_9 * Aad2_1 + o10_9 * Aad3_1 + o13_9 * Aad4_1 + o16_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_1 * Aad0_1 + o5_1 * Aad1_1 + o8_1 * Aad2_1 + o11_1 * Aad3_1 + o14_1 * Aad4_1 + o17_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_1 * Aac0_0 + o2_5 * Aac0_1 + o2_9 * Aac0_2 + o5_1 * Aac1_0 + o5_5 * Aac1_1 + o5_9 * Aac1_2 + o8_1 * Aac2_0 + o8_5 * Aac2_1 + o8_9 * Aac2_2 + o11_1 * Aac3_0 + o11_5 * Aac3_1 + o11_9 * Aac3_2 + o14_1 * Aac4_0 + o14_5 * Aac4_1 + o14_9 * Aac4_2 + o17_1 * Aac5_0 + o17_5 * Aac5_1 + o17_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_5 * Aad0_1 + o5_5 * Aad1_1 + o8_5 * Aad2_1 + o11_5 * Aad3_1 + o14_5 * Aad4_1 + o17_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_9 * Aad0_1 + o5_9 * Aad1_1 + o8_9 * Aad2_1 + o11_9 * Aad3_1 + o14_9 * Aad4_1 + o17_9 * Aad5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o3_1 * Abd0_1 + o4_1 * Abd1_1 + o5_1 * Abd2_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o3_1 * Abc0_0 + o3_5 * Abc0_1 + o3_9 * Abc0_2 + o4_1 * Abc1_0 + o4_5 * Abc1_1 + o4_9 * Abc1_2 + o5_1 * Abc2_0 + o5_5 * Abc2_1 + o5_9 * Abc2_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o3_5 * Abd0_1 + o4_5 * Abd1_1 + o5_5 * Abd2_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o3_9 * Abd0_1 + o4_9 * Abd1_1 + o5_9 * Abd2_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o6_1 * Abd0_1 + o7_1 * Abd1_1 + o8_1 * Abd2_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o6_1 * Abc0_0 + o6_5 * Abc0_1 + o6_9 * Abc0_2 + o7_1 * Abc1_0 + o7_5 * Abc1_1 + o7_9 * Abc1_2 + o8_1 * Abc2_0 + o8_5 * Abc2_1 + o8_9 * Abc2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o6_5 * Abd0_1 + o7_5 * Abd1_1 + o8_5 * Abd2_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o6_9 * Abd0_1 + o7_9 * Abd1_1 + o8_9 * Abd2_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o9_1 * Abd0_1 + o10_1 * Abd1_1 + o11_1 * Abd2_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o9_1 * Abc0_0 + o9_5 * Abc0_1 + o9_9 * Abc0_2 + o10_1 * Abc1_0 + o10_5 * Abc1_1 + o10_9 * Abc1_2 + o11_1 * Abc2_0 + o11_5 * Abc2_1 + o11_9 * Abc2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o9_5 * Abd0_1 + o10_5 * Abd1_1 + o11_5 * Abd2_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o9_9 * Abd0_1 + o10_9 * Abd1_1 + o11_9 * Abd2_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o12_1 * Abd0_1 + o13_1 * Abd1_1 + o14_1 * Abd2_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o12_1 * Abc0_0 + o12_5 * Abc0_1 + o12_9 * Abc0_2 + o13_1 * Abc1_0 + o13_5 * Abc1_1 + o13_9 * Abc1_2 + o14_1 * Abc2_0 + o14_5 * Abc2_1 + o14_9 * Abc2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o12_5 * Abd0_1 + o13_5 * Abd1_1 + o14_5 * Abd2_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o12_9 * Abd0_1 + o13_9 * Abd1_1 + o14_9 * Abd2_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o15_1 * Abd0_1 + o16_1 * Abd1_1 + o17_1 * Abd2_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o15_1 * Abc0_0 + o15_5 * Abc0_1 + o15_9 * Abc0_2 + o16_1 * Abc1_0 + o16_5 * Abc1_1 + o16_9 * Abc1_2 + o17_1 * Abc2_0 + o17_5 * Abc2_1 + o17_9 * Abc2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o15_5 * Abd0_1 + o16_5 * Abd1_1 + o17_5 * Abd2_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o15_9 * Abd0_1 + o16_9 * Abd1_1 + o17_9 * Abd2_1));
          }
        } break;
        case 2: {  // ket functions [2, 6, 10]
          double o0_2 = 0;
          double o0_6 = 0;
          double o0_10 = 0;
          double o1_2 = 0;
          double o1_6 = 0;
          double o1_10 = 0;
          double o2_2 = 0;
          double o2_6 = 0;
          double o2_10 = 0;
          double o3_2 = 0;
          double o3_6 = 0;
          double o3_10 = 0;
          double o4_2 = 0;
          double o4_6 = 0;
          double o4_10 = 0;
          double o5_2 = 0;
          double o5_6 = 0;
          double o5_10 = 0;
          double o6_2 = 0;
          double o6_6 = 0;
          double o6_10 = 0;
          double o7_2 = 0;
          double o7_6 = 0;
          double o7_10 = 0;
          double o8_2 = 0;
          double o8_6 = 0;
          double o8_10 = 0;
          double o9_2 = 0;
          double o9_6 = 0;
          double o9_10 = 0;
          double o10_2 = 0;
          double o10_6 = 0;
          double o10_10 = 0;
          double o11_2 = 0;
          double o11_6 = 0;
          double o11_10 = 0;
          double o12_2 = 0;
          double o12_6 = 0;
          double o12_10 = 0;
          double o13_2 = 0;
          double o13_6 = 0;
          double o13_10 = 0;
          double o14_2 = 0;
          double o14_6 = 0;
          double o14_10 = 0;
          double o15_2 = 0;
          double o15_6 = 0;
          double o15_10 = 0;
          double o16_2 = 0;
          double o16_6 = 0;
          double o16_10 = 0;
          double o17_2 = 0;
          double o17_6 = 0;
          double o17_10 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 113;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g2_0 = 0;
            double g2_1 = 0;
            double g2_2 = 0;
            double g2_3 = 0;
            double g2_4 = 0;
            double g2_5 = 0;
            double g2_6 = 0;
            double g2_7 = 0;
            double g2_8 = 0;
            double g2_9 = 0;
            double g2_10 = 0;
            double g2_11 = 0;
            double g2_12 = 0;
            double g2_13 = 0;
            double g2_14 = 0;
            double g2_15 = 0;
            double g2_16 = 0;
            double g2_17 = 0;
            double g2_18 = 0;
            double g2_19 = 0;
            double g6_0 = 0;
            double g6_1 = 0;
            double g6_2 = 0;
            double g6_3 = 0;
            double g6_4 = 0;
            double g6_5 = 0;
            double g6_6 = 0;
            double g6_7 = 0;
            double g6_8 = 0;
            double g6_9 = 0;
            double g6_10 = 0;
            double g6_11 = 0;
            double g6_12 = 0;
            double g6_13 = 0;
            double g6_14 = 0;
            double g6_15 = 0;
            double g6_16 = 0;
            double g6_17 = 0;
            double g6_18 = 0;
            double g6_19 = 0;
            double g10_0 = 0;
            double g10_1 = 0;
            double g10_2 = 0;
            double g10_3 = 0;
            double g10_4 = 0;
            double g10_5 = 0;
            double g10_6 = 0;
            double g10_7 = 0;
            double g10_8 = 0;
            double g10_9 = 0;
            double g10_10 = 0;
            double g10_11 = 0;
            double g10_12 = 0;
            double g10_13 = 0;
            double g10_14 = 0;
            double g10_15 = 0;
            double g10_16 = 0;
            double g10_17 = 0;
            double g10_18 = 0;
            double g10_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[6];
              sqb::boys<5>(T, a.boys_tab, F);
              const double s0 = TWO_PI_2_5 * rs;
              const double m2a = -2.0 * alpha;
              double w = s0;
              const double b0 = w * F[0];
              w *= m2a;
              const double b1 = w * F[1];
              w *= m2a;
              const double b2 = w * F[2];
              w *= m2a;
              const double b3 = w * F[3];
              w *= m2a;
              const double b4 = w * F[4];
              w *= m2a;
              const double b5 = w * F[5];
              const double ek2_0 = kj[10 * kS];
              const double ek2_1 = -kj[11 * kS];
              const double ek2_2 = -kj[12 * kS];
              const double ek2_3 = kj[13 * kS];
              const double ek6_0 = kj[24 * kS];
              const double ek6_1 = -kj[25 * kS];
              const double ek6_2 = kj[26 * kS];
              const double ek10_0 = kj[37 * kS];
              const double ek10_1 = -kj[38 * kS];
              const double ek10_2 = -kj[39 * kS];
              const double ek10_3 = kj[40 * kS];
              g2_0 = fma(ek2_0, b0, g2_0);
              g6_0 = fma(ek6_0, b0, g6_0);
              g10_0 = fma(ek10_0, b0, g10_0);
              const double r0_0_0_1 = Z * b1;
              g2_1 = fma(ek2_0, r0_0_0_1, g2_1);
              g6_1 = fma(ek6_0, r0_0_0_1, g6_1);
              g10_1 = fma(ek10_0, r0_0_0_1, g10_1);
              g10_0 = fma(ek10_1, r0_0_0_1, g10_0);
              const double r0_0_1_0 = Y * b1;
              g2_2 = fma(ek2_0, r0_0_1_0, g2_2);
              g2_0 = fma(ek2_1, r0_0_1_0, g2_0);
              g6_2 = fma(ek6_0, r0_0_1_0, g6_2);
              g6_0 = fma(ek6_1, r0_0_1_0, g6_0);
              g10_2 = fma(ek10_0, r0_0_1_0, g10_2);
              g10_0 = fma(ek10_2, r0_0_1_0, g10_0);
              const double r0_1_0_0 = X * b1;
              g2_3 = fma(ek2_0, r0_1_0_0, g2_3);
              g2_0 = fma(ek2_2, r0_1_0_0, g2_0);
              g6_3 = fma(ek6_0, r0_1_0_0, g6_3);
              g10_3 = fma(ek10_0, r0_1_0_0, g10_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g2_4 = fma(ek2_0, r0_0_0_2, g2_4);
              g6_4 = fma(ek6_0, r0_0_0_2, g6_4);
              g10_4 = fma(ek10_0, r0_0_0_2, g10_4);
              g10_1 = fma(ek10_1, r0_0_0_2, g10_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g2_5 = fma(ek2_0, r0_0_1_1, g2_5);
              g2_1 = fma(ek2_1, r0_0_1_1, g2_1);
              g6_5 = fma(ek6_0, r0_0_1_1, g6_5);
              g6_1 = fma(ek6_1, r0_0_1_1, g6_1);
              g10_5 = fma(ek10_0, r0_0_1_1, g10_5);
              g10_2 = fma(ek10_1, r0_0_1_1, g10_2);
              g10_1 = fma(ek10_2, r0_0_1_1, g10_1);
              g10_0 = fma(ek10_3, r0_0_1_1, g10_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g2_6 = fma(ek2_0, r0_0_2_0, g2_6);
              g2_2 = fma(ek2_1, r0_0_2_0, g2_2);
              g6_6 = fma(ek6_0, r0_0_2_0, g6_6);
              g6_2 = fma(ek6_1, r0_0_2_0, g6_2);
              g6_0 = fma(ek6_2, r0_0_2_0, g6_0);
              g10_6 = fma(ek10_0, r0_0_2_0, g10_6);
              g10_2 = fma(ek10_2, r0_0_2_0, g10_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g2_7 = fma(ek2_0, r0_1_0_1, g2_7);
              g2_1 = fma(ek2_2, r0_1_0_1, g2_1);
              g6_7 = fma(ek6_0, r0_1_0_1, g6_7);
              g10_7 = fma(ek10_0, r0_1_0_1, g10_7);
              g10_3 = fma(ek10_1, r0_1_0_1, g10_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g2_8 = fma(ek2_0, r0_1_1_0, g2_8);
              g2_3 = fma(ek2_1, r0_1_1_0, g2_3);
              g2_2 = fma(ek2_2, r0_1_1_0, g2_2);
              g2_0 = fma(ek2_3, r0_1_1_0, g2_0);
              g6_8 = fma(ek6_0, r0_1_1_0, g6_8);
              g6_3 = fma(ek6_1, r0_1_1_0, g6_3);
              g10_8 = fma(ek10_0, r0_1_1_0, g10_8);
              g10_3 = fma(ek10_2, r0_1_1_0, g10_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g2_9 = fma(ek2_0, r0_2_0_0, g2_9);
              g2_3 = fma(ek2_2, r0_2_0_0, g2_3);
              g6_9 = fma(ek6_0, r0_2_0_0, g6_9);
              g10_9 = fma(ek10_0, r0_2_0_0, g10_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g2_10 = fma(ek2_0, r0_0_0_3, g2_10);
              g6_10 = fma(ek6_0, r0_0_0_3, g6_10);
              g10_10 = fma(ek10_0, r0_0_0_3, g10_10);
              g10_4 = fma(ek10_1, r0_0_0_3, g10_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g2_11 = fma(ek2_0, r0_0_1_2, g2_11);
              g2_4 = fma(ek2_1, r0_0_1_2, g2_4);
              g6_11 = fma(ek6_0, r0_0_1_2, g6_11);
              g6_4 = fma(ek6_1, r0_0_1_2, g6_4);
              g10_11 = fma(ek10_0, r0_0_1_2, g10_11);
              g10_5 = fma(ek10_1, r0_0_1_2, g10_5);
              g10_4 = fma(ek10_2, r0_0_1_2, g10_4);
              g10_1 = fma(ek10_3, r0_0_1_2, g10_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g2_12 = fma(ek2_0, r0_0_2_1, g2_12);
              g2_5 = fma(ek2_1, r0_0_2_1, g2_5);
              g6_12 = fma(ek6_0, r0_0_2_1, g6_12);
              g6_5 = fma(ek6_1, r0_0_2_1, g6_5);
              g6_1 = fma(ek6_2, r0_0_2_1, g6_1);
              g10_12 = fma(ek10_0, r0_0_2_1, g10_12);
              g10_6 = fma(ek10_1, r0_0_2_1, g10_6);
              g10_5 = fma(ek10_2, r0_0_2_1, g10_5);
              g10_2 = fma(ek10_3, r0_0_2_1, g10_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g2_13 = fma(ek2_0, r0_0_3_0, g2_13);
              g2_6 = fma(ek2_1, r0_0_3_0, g2_6);
              g6_13 = fma(ek6_0, r0_0_3_0, g6_13);
              g6_6 = fma(ek6_1, r0_0_3_0, g6_6);
              g6_2 = fma(ek6_2, r0_0_3_0, g6_2);
              g10_13 = fma(ek10_0, r0_0_3_0, g10_13);
              g10_6 = fma(ek10_2, r0_0_3_0, g10_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g2_14 = fma(ek2_0, r0_1_0_2, g2_14);
              g2_4 = fma(ek2_2, r0_1_0_2, g2_4);
              g6_14 = fma(ek6_0, r0_1_0_2, g6_14);
              g10_14 = fma(ek10_0, r0_1_0_2, g10_14);
              g10_7 = fma(ek10_1, r0_1_0_2, g10_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g2_15 = fma(ek2_0, r0_1_1_1, g2_15);
              g2_7 = fma(ek2_1, r0_1_1_1, g2_7);
              g2_5 = fma(ek2_2, r0_1_1_1, g2_5);
              g2_1 = fma(ek2_3, r0_1_1_1, g2_1);
              g6_15 = fma(ek6_0, r0_1_1_1, g6_15);
              g6_7 = fma(ek6_1, r0_1_1_1, g6_7);
              g10_15 = fma(ek10_0, r0_1_1_1, g10_15);
              g10_8 = fma(ek10_1, r0_1_1_1, g10_8);
              g10_7 = fma(ek10_2, r0_1_1_1, g10_7);
              g10_3 = fma(ek10_3, r0_1_1_1, g10_3);
              const double r0_1_2_0 = X * r1_0_2_0;
              g2_16 = fma(ek2_0, r0_1_2_0, g2_16);
              g2_8 = fma(ek2_1, r0_1_2_0, g2_8);
              g2_6 = fma(ek2_2, r0_1_2_0, g2_6);
              g2_2 = fma(ek2_3, r0_1_2_0, g2_2);
              g6_16 = fma(ek6_0, r0_1_2_0, g6_16);
              g6_8 = fma(ek6_1, r0_1_2_0, g6_8);
              g6_3 = fma(ek6_2, r0_1_2_0, g6_3);
              g10_16 = fma(ek10_0, r0_1_2_0, g10_16);
              g10_8 = fma(ek10_2, r0_1_2_0, g10_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g2_17 = fma(ek2_0, r0_2_0_1, g2_17);
              g2_7 = fma(ek2_2, r0_2_0_1, g2_7);
              g6_17 = fma(ek6_0, r0_2_0_1, g6_17);
              g10_17 = fma(ek10_0, r0_2_0_1, g10_17);
              g10_9 = fma(ek10_1, r0_2_0_1, g10_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g2_18 = fma(ek2_0, r0_2_1_0, g2_18);
              g2_9 = fma(ek2_1, r0_2_1_0, g2_9);
              g2_8 = fma(ek2_2, r0_2_1_0, g2_8);
              g2_3 = fma(ek2_3, r0_2_1_0, g2_3);
              g6_18 = fma(ek6_0, r0_2_1_0, g6_18);
              g6_9 = fma(ek6_1, r0_2_1_0, g6_9);
              g10_18 = fma(ek10_0, r0_2_1_0, g10_18);
              g10_9 = fma(ek10_2, r0_2_1_0, g10_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g2_19 = fma(ek2_0, r0_3_0_0, g2_19);
              g2_9 = fma(ek2_2, r0_3_0_0, g2_9);
              g6_19 = fma(ek6_0, r0_3_0_0, g6_19);
              g10_19 = fma(ek10_0, r0_3_0_0, g10_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g10_10 = fma(ek10_1, r0_0_0_4, g10_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g2_10 = fma(ek2_1, r0_0_1_3, g2_10);
              g6_10 = fma(ek6_1, r0_0_1_3, g6_10);
              g10_11 = fma(ek10_1, r0_0_1_3, g10_11);
              g10_10 = fma(ek10_2, r0_0_1_3, g10_10);
              g10_4 = fma(ek10_3, r0_0_1_3, g10_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g2_11 = fma(ek2_1, r0_0_2_2, g2_11);
              g6_11 = fma(ek6_1, r0_0_2_2, g6_11);
              g6_4 = fma(ek6_2, r0_0_2_2, g6_4);
              g10_12 = fma(ek10_1, r0_0_2_2, g10_12);
              g10_11 = fma(ek10_2, r0_0_2_2, g10_11);
              g10_5 = fma(ek10_3, r0_0_2_2, g10_5);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g2_12 = fma(ek2_1, r0_0_3_1, g2_12);
              g6_12 = fma(ek6_1, r0_0_3_1, g6_12);
              g6_5 = fma(ek6_2, r0_0_3_1, g6_5);
              g10_13 = fma(ek10_1, r0_0_3_1, g10_13);
              g10_12 = fma(ek10_2, r0_0_3_1, g10_12);
              g10_6 = fma(ek10_3, r0_0_3_1, g10_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g2_13 = fma(ek2_1, r0_0_4_0, g2_13);
              g6_13 = fma(ek6_1, r0_0_4_0, g6_13);
              g6_6 = fma(ek6_2, r0_0_4_0, g6_6);
              g10_13 = fma(ek10_2, r0_0_4_0, g10_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g2_10 = fma(ek2_2, r0_1_0_3, g2_10);
              g10_14 = fma(ek10_1, r0_1_0_3, g10_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g2_14 = fma(ek2_1, r0_1_1_2, g2_14);
              g2_11 = fma(ek2_2, r0_1_1_2, g2_11);
              g2_4 = fma(ek2_3, r0_1_1_2, g2_4);
              g6_14 = fma(ek6_1, r0_1_1_2, g6_14);
              g10_15 = fma(ek10_1, r0_1_1_2, g10_15);
              g10_14 = fma(ek10_2, r0_1_1_2, g10_14);
              g10_7 = fma(ek10_3, r0_1_1_2, g10_7);
              const double r0_1_2_1 = X * r1_0_2_1;
              g2_15 = fma(ek2_1, r0_1_2_1, g2_15);
              g2_12 = fma(ek2_2, r0_1_2_1, g2_12);
              g2_5 = fma(ek2_3, r0_1_2_1, g2_5);
              g6_15 = fma(ek6_1, r0_1_2_1, g6_15);
              g6_7 = fma(ek6_2, r0_1_2_1, g6_7);
              g10_16 = fma(ek10_1, r0_1_2_1, g10_16);
              g10_15 = fma(ek10_2, r0_1_2_1, g10_15);
              g10_8 = fma(ek10_3, r0_1_2_1, g10_8);
              const double r0_1_3_0 = X * r1_0_3_0;
              g2_16 = fma(ek2_1, r0_1_3_0, g2_16);
              g2_13 = fma(ek2_2, r0_1_3_0, g2_13);
              g2_6 = fma(ek2_3, r0_1_3_0, g2_6);
              g6_16 = fma(ek6_1, r0_1_3_0, g6_16);
              g6_8 = fma(ek6_2, r0_1_3_0, g6_8);
              g10_16 = fma(ek10_2, r0_1_3_0, g10_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g2_14 = fma(ek2_2, r0_2_0_2, g2_14);
              g10_17 = fma(ek10_1, r0_2_0_2, g10_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g2_17 = fma(ek2_1, r0_2_1_1, g2_17);
              g2_15 = fma(ek2_2, r0_2_1_1, g2_15);
              g2_7 = fma(ek2_3, r0_2_1_1, g2_7);
              g6_17 = fma(ek6_1, r0_2_1_1, g6_17);
              g10_18 = fma(ek10_1, r0_2_1_1, g10_18);
              g10_17 = fma(ek10_2, r0_2_1_1, g10_17);
              g10_9 = fma(ek10_3, r0_2_1_1, g10_9);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g2_18 = fma(ek2_1, r0_2_2_0, g2_18);
              g2_16 = fma(ek2_2, r0_2_2_0, g2_16);
              g2_8 = fma(ek2_3, r0_2_2_0, g2_8);
              g6_18 = fma(ek6_1, r0_2_2_0, g6_18);
              g6_9 = fma(ek6_2, r0_2_2_0, g6_9);
              g10_18 = fma(ek10_2, r0_2_2_0, g10_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g2_17 = fma(ek2_2, r0_3_0_1, g2_17);
              g10_19 = fma(ek10_1, r0_3_0_1, g10_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g2_19 = fma(ek2_1, r0_3_1_0, g2_19);
              g2_18 = fma(ek2_2, r0_3_1_0, g2_18);
              g2_9 = fma(ek2_3, r0_3_1_0, g2_9);
              g6_19 = fma(ek6_1, r0_3_1_0, g6_19);
              g10_19 = fma(ek10_2, r0_3_1_0, g10_19);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g2_19 = fma(ek2_2, r0_4_0_0, g2_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g10_10 = fma(ek10_3, r0_0_1_4, g10_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g6_10 = fma(ek6_2, r0_0_2_3, g6_10);
              g10_11 = fma(ek10_3, r0_0_2_3, g10_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g6_11 = fma(ek6_2, r0_0_3_2, g6_11);
              g10_12 = fma(ek10_3, r0_0_3_2, g10_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g6_12 = fma(ek6_2, r0_0_4_1, g6_12);
              g10_13 = fma(ek10_3, r0_0_4_1, g10_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g6_13 = fma(ek6_2, r0_0_5_0, g6_13);
              const double r0_1_1_3 = X * r1_0_1_3;
              g2_10 = fma(ek2_3, r0_1_1_3, g2_10);
              g10_14 = fma(ek10_3, r0_1_1_3, g10_14);
              const double r0_1_2_2 = X * r1_0_2_2;
              g2_11 = fma(ek2_3, r0_1_2_2, g2_11);
              g6_14 = fma(ek6_2, r0_1_2_2, g6_14);
              g10_15 = fma(ek10_3, r0_1_2_2, g10_15);
              const double r0_1_3_1 = X * r1_0_3_1;
              g2_12 = fma(ek2_3, r0_1_3_1, g2_12);
              g6_15 = fma(ek6_2, r0_1_3_1, g6_15);
              g10_16 = fma(ek10_3, r0_1_3_1, g10_16);
              const double r0_1_4_0 = X * r1_0_4_0;
              g2_13 = fma(ek2_3, r0_1_4_0, g2_13);
              g6_16 = fma(ek6_2, r0_1_4_0, g6_16);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g2_14 = fma(ek2_3, r0_2_1_2, g2_14);
              g10_17 = fma(ek10_3, r0_2_1_2, g10_17);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g2_15 = fma(ek2_3, r0_2_2_1, g2_15);
              g6_17 = fma(ek6_2, r0_2_2_1, g6_17);
              g10_18 = fma(ek10_3, r0_2_2_1, g10_18);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g2_16 = fma(ek2_3, r0_2_3_0, g2_16);
              g6_18 = fma(ek6_2, r0_2_3_0, g6_18);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g2_17 = fma(ek2_3, r0_3_1_1, g2_17);
              g10_19 = fma(ek10_3, r0_3_1_1, g10_19);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g2_18 = fma(ek2_3, r0_3_2_0, g2_18);
              g6_19 = fma(ek6_2, r0_3_2_0, g6_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g2_19 = fma(ek2_3, r0_4_1_0, g2_19);
            }
            { const double eb = bi[5];
              o0_2 = fma(eb, g2_0, o0_2);
              o0_6 = fma(eb, g6_0, o0_6);
              o0_10 = fma(eb, g10_0, o0_10);
            }
            { const double eb = bi[6];
              o0_2 = fma(eb, g2_3, o0_2);
              o0_6 = fma(eb, g6_3, o0_6);
              o0_10 = fma(eb, g10_3, o0_10);
            }
            { const double eb = bi[7];
              o0_2 = fma(eb, g2_9, o0_2);
              o0_6 = fma(eb, g6_9, o0_6);
              o0_10 = fma(eb, g10_9, o0_10);
            }
            { const double eb = bi[8];
              o0_2 = fma(eb, g2_19, o0_2);
              o0_6 = fma(eb, g6_19, o0_6);
              o0_10 = fma(eb, g10_19, o0_10);
            }
            { const double eb = bi[9];
              o1_2 = fma(eb, g2_0, o1_2);
              o1_6 = fma(eb, g6_0, o1_6);
              o1_10 = fma(eb, g10_0, o1_10);
            }
            { const double eb = bi[10];
              o1_2 = fma(eb, g2_2, o1_2);
              o1_6 = fma(eb, g6_2, o1_6);
              o1_10 = fma(eb, g10_2, o1_10);
            }
            { const double eb = bi[11];
              o1_2 = fma(eb, g2_3, o1_2);
              o1_6 = fma(eb, g6_3, o1_6);
              o1_10 = fma(eb, g10_3, o1_10);
            }
            { const double eb = bi[12];
              o1_2 = fma(eb, g2_8, o1_2);
              o1_6 = fma(eb, g6_8, o1_6);
              o1_10 = fma(eb, g10_8, o1_10);
            }
            { const double eb = bi[13];
              o1_2 = fma(eb, g2_9, o1_2);
              o1_6 = fma(eb, g6_9, o1_6);
              o1_10 = fma(eb, g10_9, o1_10);
            }
            { const double eb = bi[14];
              o1_2 = fma(eb, g2_18, o1_2);
              o1_6 = fma(eb, g6_18, o1_6);
              o1_10 = fma(eb, g10_18, o1_10);
            }
            { const double eb = bi[15];
              o2_2 = fma(eb, g2_0, o2_2);
              o2_6 = fma(eb, g6_0, o2_6);
              o2_10 = fma(eb, g10_0, o2_10);
            }
            { const double eb = bi[16];
              o2_2 = fma(eb, g2_1, o2_2);
              o2_6 = fma(eb, g6_1, o2_6);
              o2_10 = fma(eb, g10_1, o2_10);
            }
            { const double eb = bi[17];
              o2_2 = fma(eb, g2_3, o2_2);
              o2_6 = fma(eb, g6_3, o2_6);
              o2_10 = fma(eb, g10_3, o2_10);
            }
            { const double eb = bi[18];
              o2_2 = fma(eb, g2_7, o2_2);
              o2_6 = fma(eb, g6_7, o2_6);
              o2_10 = fma(eb, g10_7, o2_10);
            }
            { const double eb = bi[19];
              o2_2 = fma(eb, g2_9, o2_2);
              o2_6 = fma(eb, g6_9, o2_6);
              o2_10 = fma(eb, g10_9, o2_10);
            }
            { const double eb = bi[20];
              o2_2 = fma(eb, g2_17, o2_2);
              o2_6 = fma(eb, g6_17, o2_6);
              o2_10 = fma(eb, g10_17, o2_10);
            }
            { const double eb = bi[21];
              o3_2 = fma(eb, g2_0, o3_2);
              o3_6 = fma(eb, g6_0, o3_6);
              o3_10 = fma(eb, g10_0, o3_10);
            }
            { const double eb = bi[22];
              o3_2 = fma(eb, g2_2, o3_2);
              o3_6 = fma(eb, g6_2, o3_6);
              o3_10 = fma(eb, g10_2, o3_10);
            }
            { const double eb = bi[23];
              o3_2 = fma(eb, g2_6, o3_2);
              o3_6 = fma(eb, g6_6, o3_6);
              o3_10 = fma(eb, g10_6, o3_10);
            }
            { const double eb = bi[24];
              o3_2 = fma(eb, g2_3, o3_2);
              o3_6 = fma(eb, g6_3, o3_6);
              o3_10 = fma(eb, g10_3, o3_10);
            }
            { const double eb = bi[25];
              o3_2 = fma(eb, g2_8, o3_2);
              o3_6 = fma(eb, g6_8, o3_6);
              o3_10 = fma(eb, g10_8, o3_10);
            }
            { const double eb = bi[26];
              o3_2 = fma(eb, g2_16, o3_2);
              o3_6 = fma(eb, g6_16, o3_6);
              o3_10 = fma(eb, g10_16, o3_10);
            }
            { const double eb = bi[27];
              o4_2 = fma(eb, g2_0, o4_2);
              o4_6 = fma(eb, g6_0, o4_6);
              o4_10 = fma(eb, g10_0, o4_10);
            }
            { const double eb = bi[28];
              o4_2 = fma(eb, g2_2, o4_2);
              o4_6 = fma(eb, g6_2, o4_6);
              o4_10 = fma(eb, g10_2, o4_10);
            }
            { const double eb = bi[29];
              o4_2 = fma(eb, g2_6, o4_2);
              o4_6 = fma(eb, g6_6, o4_6);
              o4_10 = fma(eb, g10_6, o4_10);
            }
            { const double eb = bi[30];
              o4_2 = fma(eb, g2_13, o4_2);
              o4_6 = fma(eb, g6_13, o4_6);
              o4_10 = fma(eb, g10_13, o4_10);
            }
            { const double eb = bi[31];
              o5_2 = fma(eb, g2_0, o5_2);
              o5_6 = fma(eb, g6_0, o5_6);
              o5_10 = fma(eb, g10_0, o5_10);
            }
            { const double eb = bi[32];
              o5_2 = fma(eb, g2_1, o5_2);
              o5_6 = fma(eb, g6_1, o5_6);
              o5_10 = fma(eb, g10_1, o5_10);
            }
            { const double eb = bi[33];
              o5_2 = fma(eb, g2_2, o5_2);
              o5_6 = fma(eb, g6_2, o5_6);
              o5_10 = fma(eb, g10_2, o5_10);
            }
            { const double eb = bi[34];
              o5_2 = fma(eb, g2_5, o5_2);
              o5_6 = fma(eb, g6_5, o5_6);
              o5_10 = fma(eb, g10_5, o5_10);
            }
            { const double eb = bi[35];
              o5_2 = fma(eb, g2_6, o5_2);
              o5_6 = fma(eb, g6_6, o5_6);
              o5_10 = fma(eb, g10_6, o5_10);
            }
            { const double eb = bi[36];
              o5_2 = fma(eb, g2_12, o5_2);
              o5_6 = fma(eb, g6_12, o5_6);
              o5_10 = fma(eb, g10_12, o5_10);
            }
            { const double eb = bi[37];
              o6_2 = fma(eb, g2_0, o6_2);
              o6_6 = fma(eb, g6_0, o6_6);
              o6_10 = fma(eb, g10_0, o6_10);
            }
            { const double eb = bi[38];
              o6_2 = fma(eb, g2_1, o6_2);
              o6_6 = fma(eb, g6_1, o6_6);
              o6_10 = fma(eb, g10_1, o6_10);
            }
            { const double eb = bi[39];
              o6_2 = fma(eb, g2_4, o6_2);
              o6_6 = fma(eb, g6_4, o6_6);
              o6_10 = fma(eb, g10_4, o6_10);
            }
            { const double eb = bi[40];
              o6_2 = fma(eb, g2_3, o6_2);
              o6_6 = fma(eb, g6_3, o6_6);
              o6_10 = fma(eb, g10_3, o6_10);
            }
            { const double eb = bi[41];
              o6_2 = fma(eb, g2_7, o6_2);
              o6_6 = fma(eb, g6_7, o6_6);
              o6_10 = fma(eb, g10_7, o6_10);
            }
            { const double eb = bi[42];
              o6_2 = fma(eb, g2_14, o6_2);
              o6_6 = fma(eb, g6_14, o6_6);
              o6_10 = fma(eb, g10_14, o6_10);
            }
            { const double eb = bi[43];
              o7_2 = fma(eb, g2_0, o7_2);
              o7_6 = fma(eb, g6_0, o7_6);
              o7_10 = fma(eb, g10_0, o7_10);
            }
            { const double eb = bi[44];
              o7_2 = fma(eb, g2_1, o7_2);
              o7_6 = fma(eb, g6_1, o7_6);
              o7_10 = fma(eb, g10_1, o7_10);
            }
            { const double eb = bi[45];
              o7_2 = fma(eb, g2_4, o7_2);
              o7_6 = fma(eb, g6_4, o7_6);
              o7_10 = fma(eb, g10_4, o7_10);
            }
            { const double eb = bi[46];
              o7_2 = fma(eb, g2_2, o7_2);
              o7_6 = fma(eb, g6_2, o7_6);
              o7_10 = fma(eb, g10_2, o7_10);
            }
            { const double eb = bi[47];
              o7_2 = fma(eb, g2_5, o7_2);
              o7_6 = fma(eb, g6_5, o7_6);
              o7_10 = fma(eb, g10_5, o7_10);
            }
            { const double eb = bi[48];
              o7_2 = fma(eb, g2_11, o7_2);
              o7_6 = fma(eb, g6_11, o7_6);
              o7_10 = fma(eb, g10_11, o7_10);
            }
            { const double eb = bi[49];
              o8_2 = fma(eb, g2_0, o8_2);
              o8_6 = fma(eb, g6_0, o8_6);
              o8_10 = fma(eb, g10_0, o8_10);
            }
            { const double eb = bi[50];
              o8_2 = fma(eb, g2_1, o8_2);
              o8_6 = fma(eb, g6_1, o8_6);
              o8_10 = fma(eb, g10_1, o8_10);
            }
            { const double eb = bi[51];
              o8_2 = fma(eb, g2_4, o8_2);
              o8_6 = fma(eb, g6_4, o8_6);
              o8_10 = fma(eb, g10_4, o8_10);
            }
            { const double eb = bi[52];
              o8_2 = fma(eb, g2_10, o8_2);
              o8_6 = fma(eb, g6_10, o8_6);
              o8_10 = fma(eb, g10_10, o8_10);
            }
            { const double eb = bi[53];
              o9_2 = fma(eb, g2_0, o9_2);
              o9_6 = fma(eb, g6_0, o9_6);
              o9_10 = fma(eb, g10_0, o9_10);
            }
            { const double eb = bi[54];
              o9_2 = fma(eb, g2_2, o9_2);
              o9_6 = fma(eb, g6_2, o9_6);
              o9_10 = fma(eb, g10_2, o9_10);
            }
            { const double eb = bi[55];
              o9_2 = fma(eb, g2_3, o9_2);
              o9_6 = fma(eb, g6_3, o9_6);
              o9_10 = fma(eb, g10_3, o9_10);
            }
            { const double eb = bi[56];
              o9_2 = fma(eb, g2_8, o9_2);
              o9_6 = fma(eb, g6_8, o9_6);
              o9_10 = fma(eb, g10_8, o9_10);
            }
            { const double eb = bi[57];
              o9_2 = fma(eb, g2_9, o9_2);
              o9_6 = fma(eb, g6_9, o9_6);
              o9_10 = fma(eb, g10_9, o9_10);
            }
            { const double eb = bi[58];
              o9_2 = fma(eb, g2_18, o9_2);
              o9_6 = fma(eb, g6_18, o9_6);
              o9_10 = fma(eb, g10_18, o9_10);
            }
            { const double eb = bi[59];
              o10_2 = fma(eb, g2_0, o10_2);
              o10_6 = fma(eb, g6_0, o10_6);
              o10_10 = fma(eb, g10_0, o10_10);
            }
            { const double eb = bi[60];
              o10_2 = fma(eb, g2_2, o10_2);
              o10_6 = fma(eb, g6_2, o10_6);
              o10_10 = fma(eb, g10_2, o10_10);
            }
            { const double eb = bi[61];
              o10_2 = fma(eb, g2_6, o10_2);
              o10_6 = fma(eb, g6_6, o10_6);
              o10_10 = fma(eb, g10_6, o10_10);
            }
            { const double eb = bi[62];
              o10_2 = fma(eb, g2_3, o10_2);
              o10_6 = fma(eb, g6_3, o10_6);
              o10_10 = fma(eb, g10_3, o10_10);
            }
            { const double eb = bi[63];
              o10_2 = fma(eb, g2_8, o10_2);
              o10_6 = fma(eb, g6_8, o10_6);
              o10_10 = fma(eb, g10_8, o10_10);
            }
            { const double eb = bi[64];
              o10_2 = fma(eb, g2_16, o10_2);
              o10_6 = fma(eb, g6_16, o10_6);
              o10_10 = fma(eb, g10_16, o10_10);
            }
            { const double eb = bi[65];
              o11_2 = fma(eb, g2_0, o11_2);
              o11_6 = fma(eb, g6_0, o11_6);
              o11_10 = fma(eb, g10_0, o11_10);
            }
            { const double eb = bi[66];
              o11_2 = fma(eb, g2_1, o11_2);
              o11_6 = fma(eb, g6_1, o11_6);
              o11_10 = fma(eb, g10_1, o11_10);
            }
            { const double eb = bi[67];
              o11_2 = fma(eb, g2_2, o11_2);
              o11_6 = fma(eb, g6_2, o11_6);
              o11_10 = fma(eb, g10_2, o11_10);
            }
            { const double eb = bi[68];
              o11_2 = fma(eb, g2_5, o11_2);
              o11_6 = fma(eb, g6_5, o11_6);
              o11_10 = fma(eb, g10_5, o11_10);
            }
            { const double eb = bi[69];
              o11_2 = fma(eb, g2_3, o11_2);
              o11_6 = fma(eb, g6_3, o11_6);
              o11_10 = fma(eb, g10_3, o11_10);
            }
            { const double eb = bi[70];
              o11_2 = fma(eb, g2_7, o11_2);
              o11_6 = fma(eb, g6_7, o11_6);
              o11_10 = fma(eb, g10_7, o11_10);
            }
            { const double eb = bi[71];
              o11_2 = fma(eb, g2_8, o11_2);
              o11_6 = fma(eb, g6_8, o11_6);
              o11_10 = fma(eb, g10_8, o11_10);
            }
            { const double eb = bi[72];
              o11_2 = fma(eb, g2_15, o11_2);
              o11_6 = fma(eb, g6_15, o11_6);
              o11_10 = fma(eb, g10_15, o11_10);
            }
            { const double eb = bi[73];
              o12_2 = fma(eb, g2_0, o12_2);
              o12_6 = fma(eb, g6_0, o12_6);
              o12_10 = fma(eb, g10_0, o12_10);
            }
            { const double eb = bi[74];
              o12_2 = fma(eb, g2_1, o12_2);
              o12_6 = fma(eb, g6_1, o12_6);
              o12_10 = fma(eb, g10_1, o12_10);
            }
            { const double eb = bi[75];
              o12_2 = fma(eb, g2_3, o12_2);
              o12_6 = fma(eb, g6_3, o12_6);
              o12_10 = fma(eb, g10_3, o12_10);
            }
            { const double eb = bi[76];
              o12_2 = fma(eb, g2_7, o12_2);
              o12_6 = fma(eb, g6_7, o12_6);
              o12_10 = fma(eb, g10_7, o12_10);
            }
            { const double eb = bi[77];
              o12_2 = fma(eb, g2_9, o12_2);
              o12_6 = fma(eb, g6_9, o12_6);
              o12_10 = fma(eb, g10_9, o12_10);
            }
            { const double eb = bi[78];
              o12_2 = fma(eb, g2_17, o12_2);
              o12_6 = fma(eb, g6_17, o12_6);
              o12_10 = fma(eb, g10_17, o12_10);
            }
            { const double eb = bi[79];
              o13_2 = fma(eb, g2_0, o13_2);
              o13_6 = fma(eb, g6_0, o13_6);
              o13_10 = fma(eb, g10_0, o13_10);
            }
            { const double eb = bi[80];
              o13_2 = fma(eb, g2_1, o13_2);
              o13_6 = fma(eb, g6_1, o13_6);
              o13_10 = fma(eb, g10_1, o13_10);
            }
            { const double eb = bi[81];
              o13_2 = fma(eb, g2_2, o13_2);
              o13_6 = fma(eb, g6_2, o13_6);
              o13_10 = fma(eb, g10_2, o13_10);
            }
            { const double eb = bi[82];
              o13_2 = fma(eb, g2_5, o13_2);
              o13_6 = fma(eb, g6_5, o13_6);
              o13_10 = fma(eb, g10_5, o13_10);
            }
            { const double eb = bi[83];
              o13_2 = fma(eb, g2_3, o13_2);
              o13_6 = fma(eb, g6_3, o13_6);
              o13_10 = fma(eb, g10_3, o13_10);
            }
            { const double eb = bi[84];
              o13_2 = fma(eb, g2_7, o13_2);
              o13_6 = fma(eb, g6_7, o13_6);
              o13_10 = fma(eb, g10_7, o13_10);
            }
            { const double eb = bi[85];
              o13_2 = fma(eb, g2_8, o13_2);
              o13_6 = fma(eb, g6_8, o13_6);
              o13_10 = fma(eb, g10_8, o13_10);
            }
            { const double eb = bi[86];
              o13_2 = fma(eb, g2_15, o13_2);
              o13_6 = fma(eb, g6_15, o13_6);
              o13_10 = fma(eb, g10_15, o13_10);
            }
            { const double eb = bi[87];
              o14_2 = fma(eb, g2_0, o14_2);
              o14_6 = fma(eb, g6_0, o14_6);
              o14_10 = fma(eb, g10_0, o14_10);
            }
            { const double eb = bi[88];
              o14_2 = fma(eb, g2_1, o14_2);
              o14_6 = fma(eb, g6_1, o14_6);
              o14_10 = fma(eb, g10_1, o14_10);
            }
            { const double eb = bi[89];
              o14_2 = fma(eb, g2_4, o14_2);
              o14_6 = fma(eb, g6_4, o14_6);
              o14_10 = fma(eb, g10_4, o14_10);
            }
            { const double eb = bi[90];
              o14_2 = fma(eb, g2_3, o14_2);
              o14_6 = fma(eb, g6_3, o14_6);
              o14_10 = fma(eb, g10_3, o14_10);
            }
            { const double eb = bi[91];
              o14_2 = fma(eb, g2_7, o14_2);
              o14_6 = fma(eb, g6_7, o14_6);
              o14_10 = fma(eb, g10_7, o14_10);
            }
            { const double eb = bi[92];
              o14_2 = fma(eb, g2_14, o14_2);
              o14_6 = fma(eb, g6_14, o14_6);
              o14_10 = fma(eb, g10_14, o14_10);
            }
            { const double eb = bi[93];
              o15_2 = fma(eb, g2_0, o15_2);
              o15_6 = fma(eb, g6_0, o15_6);
              o15_10 = fma(eb, g10_0, o15_10);
            }
            { const double eb = bi[94];
              o15_2 = fma(eb, g2_1, o15_2);
              o15_6 = fma(eb, g6_1, o15_6);
              o15_10 = fma(eb, g10_1, o15_10);
            }
            { const double eb = bi[95];
              o15_2 = fma(eb, g2_2, o15_2);
              o15_6 = fma(eb, g6_2, o15_6);
              o15_10 = fma(eb, g10_2, o15_10);
            }
            { const double eb = bi[96];
              o15_2 = fma(eb, g2_5, o15_2);
              o15_6 = fma(eb, g6_5, o15_6);
              o15_10 = fma(eb, g10_5, o15_10);
            }
            { const double eb = bi[97];
              o15_2 = fma(eb, g2_3, o15_2);
              o15_6 = fma(eb, g6_3, o15_6);
              o15_10 = fma(eb, g10_3, o15_10);
            }
            { const double eb = bi[98];
              o15_2 = fma(eb, g2_7, o15_2);
              o15_6 = fma(eb, g6_7, o15_6);
              o15_10 = fma(eb, g10_7, o15_10);
            }
            { const double eb = bi[99];
              o15_2 = fma(eb, g2_8, o15_2);
              o15_6 = fma(eb, g6_8, o15_6);
              o15_10 = fma(eb, g10_8, o15_10);
            }
            { const double eb = bi[100];
              o15_2 = fma(eb, g2_15, o15_2);
              o15_6 = fma(eb, g6_15, o15_6);
              o15_10 = fma(eb, g10_15, o15_10);
            }
            { const double eb = bi[101];
              o16_2 = fma(eb, g2_0, o16_2);
              o16_6 = fma(eb, g6_0, o16_6);
              o16_10 = fma(eb, g10_0, o16_10);
            }
            { const double eb = bi[102];
              o16_2 = fma(eb, g2_1, o16_2);
              o16_6 = fma(eb, g6_1, o16_6);
              o16_10 = fma(eb, g10_1, o16_10);
            }
            { const double eb = bi[103];
              o16_2 = fma(eb, g2_2, o16_2);
              o16_6 = fma(eb, g6_2, o16_6);
              o16_10 = fma(eb, g10_2, o16_10);
            }
            { const double eb = bi[104];
              o16_2 = fma(eb, g2_5, o16_2);
              o16_6 = fma(eb, g6_5, o16_6);
              o16_10 = fma(eb, g10_5, o16_10);
            }
            { const double eb = bi[105];
              o16_2 = fma(eb, g2_6, o16_2);
              o16_6 = fma(eb, g6_6, o16_6);
              o16_10 = fma(eb, g10_6, o16_10);
            }
            { const double eb = bi[106];
              o16_2 = fma(eb, g2_12, o16_2);
              o16_6 = fma(eb, g6_12, o16_6);
              o16_10 = fma(eb, g10_12, o16_10);
            }
            { const double eb = bi[107];
              o17_2 = fma(eb, g2_0, o17_2);
              o17_6 = fma(eb, g6_0, o17_6);
              o17_10 = fma(eb, g10_0, o17_10);
            }
            { const double eb = bi[108];
              o17_2 = fma(eb, g2_1, o17_2);
              o17_6 = fma(eb, g6_1, o17_6);
              o17_10 = fma(eb, g10_1, o17_10);
            }
            { const double eb = bi[109];
              o17_2 = fma(eb, g2_4, o17_2);
              o17_6 = fma(eb, g6_4, o17_6);
              o17_10 = fma(eb, g10_4, o17_10);
            }
            { const double eb = bi[110];
              o17_2 = fma(eb, g2_2, o17_2);
              o17_6 = fma(eb, g6_2, o17_6);
              o17_10 = fma(eb, g10_2, o17_10);
            }
            { const double eb = bi[111];
              o17_2 = fma(eb, g2_5, o17_2);
              o17_6 = fma(eb, g6_5, o17_6);
              o17_10 = fma(eb, g10_5, o17_10);
            }
            { const double eb = bi[112];
              o17_2 = fma(eb, g2_11, o17_2);
              o17_6 = fma(eb, g6_11, o17_6);
              o17_10 = fma(eb, g10_11, o17_10);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 0) * N + fJ + 2];
            const double ptk6 = PT[(fI + 1) * N + fJ + 2];
            const double ptk10 = PT[(fI + 2) * N + fJ + 2];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 1) * N + fQ + 0];
            const double ptb4 = PT[(fP + 1) * N + fQ + 1];
            const double ptb5 = PT[(fP + 1) * N + fQ + 2];
            const double ptb6 = PT[(fP + 2) * N + fQ + 0];
            const double ptb7 = PT[(fP + 2) * N + fQ + 1];
            const double ptb8 = PT[(fP + 2) * N + fQ + 2];
            const double ptb9 = PT[(fP + 3) * N + fQ + 0];
            const double ptb10 = PT[(fP + 3) * N + fQ + 1];
            const double ptb11 = PT[(fP + 3) * N + fQ + 2];
            const double ptb12 = PT[(fP + 4) * N + fQ + 0];
            const double ptb13 = PT[(fP + 4) * N + fQ + 1];
            const double ptb14 = PT[(fP + 4) * N + fQ + 2];
            const double ptb15 = PT[(fP + 5) * N + fQ + 0];
            const double ptb16 = PT[(fP + 5) * N + fQ + 1];
            const double ptb17 = PT[(fP + 5) * N + fQ + 2];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            jab0 += o0_2 * ptk2 + o0_6 * ptk6 + o0_10 * ptk10;
            jab1 += o1_2 * ptk2 + o1_6 * ptk6 + o1_10 * ptk10;
            jab2 += o2_2 * ptk2 + o2_6 * ptk6 + o2_10 * ptk10;
            jab3 += o3_2 * ptk2 + o3_6 * ptk6 + o3_10 * ptk10;
            jab4 += o4_2 * ptk2 + o4_6 * ptk6 + o4_10 * ptk10;
            jab5 += o5_2 * ptk2 + o5_6 * ptk6 + o5_10 * ptk10;
            jab6 += o6_2 * ptk2 + o6_6 * ptk6 + o6_10 * ptk10;
            jab7 += o7_2 * ptk2 + o7_6 * ptk6 + o7_10 * ptk10;
            jab8 += o8_2 * ptk2 + o8_6 * ptk6 + o8_10 * ptk10;
            jab9 += o9_2 * ptk2 + o9_6 * ptk6 + o9_10 * ptk10;
            jab10 += o10_2 * ptk2 + o10_6 * ptk6 + o10_10 * ptk10;
            jab11 += o11_2 * ptk2 + o11_6 * ptk6 + o11_10 * ptk10;
            jab12 += o12_2 * ptk2 + o12_6 * ptk6 + o12_10 * ptk10;
            jab13 += o13_2 * ptk2 + o13_6 * ptk6 + o13_10 * ptk10;
            jab14 += o14_2 * ptk2 + o14_6 * ptk6 + o14_10 * ptk10;
            jab15 += o15_2 * ptk2 + o15_6 * ptk6 + o15_10 * ptk10;
            jab16 += o16_2 * ptk2 + o16_6 * ptk6 + o16_10 * ptk10;
            jab17 += o17_2 * ptk2 + o17_6 * ptk6 + o17_10 * ptk10;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 2, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 2, 2.0 * deg * (o0_6 * ptb0 + o1_6 * ptb1 + o2_6 * ptb2 + o3_6 * ptb3 + o4_6 * ptb4 + o5_6 * ptb5 + o6_6 * ptb6 + o7_6 * ptb7 + o8_6 * ptb8 + o9_6 * ptb9 + o10_6 * ptb10 + o11_6 * ptb11 + o12_6 * ptb12 + o13_6 * ptb13 + o14_6 * ptb14 + o15_6 * ptb15 + o16_6 * ptb16 + o17_6 * ptb17));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 2, 2.0 * deg * (o0_10 * ptb0 + o1_10 * ptb1 + o2_10 * ptb2 + o3_10 * ptb3 + o4_10 * ptb4 + o5_10 * ptb5 + o6_10 * ptb6 + o7_10 * ptb7 + o8_10 * ptb8 + o9_10 * ptb9 + o10_10 * ptb10 + o11_10 * ptb11 + o12_10 * ptb12 + o13_10 * ptb13 + o14_10 * ptb14 + o15_10 * ptb15 + o16_10 * ptb16 + o17_10 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_2 * Abd0_2 + o1_2 * Abd1_2 + o2_2 * Abd2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_2 * Aad0_2 + o3_2 * Aad1_2 + o6_2 * Aad2_2 + o9_2 * Aad3_2 + o12_2 * Aad4_2 + o15_2 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_2 * Abc0_0 + o0_6 * Abc0_1 + o0_10 * Abc0_2 + o1_2 * Abc1_0 + o1_6 * Abc1_1 + o1_10 * Abc1_2 + o2_2 * Abc2_0 + o2_6 * Abc2_1 + o2_10 * Abc2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_2 * Aac0_0 + o0_6 * Aac0_1 + o0_10 * Aac0_2 + o3_2 * Aac1_0 + o3_6 * Aac1_1 + o3_10 * Aac1_2 + o6_2 * Aac2_0 + o6_6 * Aac2_1 + o6_10 * Aac2_2 + o9_2 * Aac3_0 + o9_6 * Aac3_1 + o9_10 * Aac3_2 + o12_2 * Aac4_0 + o12_6 * Aac4_1 + o12_10 * Aac4_2 + o15_2 * Aac5_0 + o15_6 * Aac5_1 + o15_10 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_6 * Abd0_2 + o1_6 * Abd1_2 + o2_6 * Abd2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_6 * Aad0_2 + o3_6 * Aad1_2 + o6_6 * Aad2_2 + o9_6 * Aad3_2 + o12_6 * Aad4_2 + o15_6 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_10 * Abd0_2 + o1_10 * Abd1_2 + o2_10 * Abd2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_10 * Aad0_2 + o3_10 * Aad1_2 + o6_10 * Aad2_2 + o9_10 * Aad3_2 + o12_10 * Aad4_2 + o15_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_2 * Aad0_2 + o4_2 * Aad1_2 + o7_2 * Aad2_2 + o10_2 * Aad3_2 + o13_2 * Aad4_2 + o16_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_2 * Aac0_0 + o1_6 * Aac0_1 + o1_10 * Aac0_2 + o4_2 * Aac1_0 + o4_6 * Aac1_1 + o4_10 * Aac1_2 + o7_2 * Aac2_0 + o7_6 * Aac2_1 + o7_10 * Aac2_2 + o10_2 * Aac3_0 + o10_6 * Aac3_1 + o10_10 * Aac3_2 + o13_2 * Aac4_0 + o13_6 * Aac4_1 + o13_10 * Aac4_2 + o16_2 * Aac5_0 + o16_6 * Aac5_1 + o16_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_6 * Aad0_2 + o4_6 * Aad1_2 + o7_6 * Aad2_2 + o10_6 * Aad3_2 + o13_6 * Aad4_2 + o16_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_10 * Aad0_2 + o4_10 * Aad1_2 + o7_10 * Aad2_2 + o10_10 * Aad3_2 + o13_10 * Aad4_2 + o16_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_2 * Aad0_2 + o5_2 * Aad1_2 + o8_2 * Aad2_2 + o11_2 * Aad3_2 + o14_2 * Aad4_2 + o17_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_2 * Aac0_0 + o2_6 * Aac0_1 + o2_10 * Aac0_2 + o5_2 * Aac1_0 + o5_6 * Aac1_1 + o5_10 * Aac1_2 + o8_2 * Aac2_0 + o8_6 * Aac2_1 + o8_10 * Aac2_2 + o11_2 * Aac3_0 + o11_6 * Aac3_1 + o11_10 * Aac3_2 + o14_2 * Aac4_0 + o14_6 * Aac4_1 + o14_10 * Aac4_2 + o17_2 * Aac5_0 + o17_6 * Aac5_1 + o17_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_6 * Aad0_2 + o5_6 * Aad1_2 + o8_6 * Aad2_2 + o11_6 * Aad3_2 + o14_6 * Aad4_2 + o17_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_10 * Aad0_2 + o5_10 * Aad1_2 + o8_10 * Aad2_2 + o11_10 * Aad3_2 + o14_10 * Aad4_2 + o17_10 * Aad5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o3_2 * Abd0_2 + o4_2 * Abd1_2 + o5_2 * Abd2_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o3_2 * Abc0_0 + o3_6 * Abc0_1 + o3_10 * Abc0_2 + o4_2 * Abc1_0 + o4_6 * Abc1_1 + o4_10 * Abc1_2 + o5_2 * Abc2_0 + o5_6 * Abc2_1 + o5_10 * Abc2_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o3_6 * Abd0_2 + o4_6 * Abd1_2 + o5_6 * Abd2_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o3_10 * Abd0_2 + o4_10 * Abd1_2 + o5_10 * Abd2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o6_2 * Abd0_2 + o7_2 * Abd1_2 + o8_2 * Abd2_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o6_2 * Abc0_0 + o6_6 * Abc0_1 + o6_10 * Abc0_2 + o7_2 * Abc1_0 + o7_6 * Abc1_1 + o7_10 * Abc1_2 + o8_2 * Abc2_0 + o8_6 * Abc2_1 + o8_10 * Abc2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o6_6 * Abd0_2 + o7_6 * Abd1_2 + o8_6 * Abd2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o6_10 * Abd0_2 + o7_10 * Abd1_2 + o8_10 * Abd2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o9_2 * Abd0_2 + o10_2 * Abd1_2 + o11_2 * Abd2_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o9_2 * Abc0_0 + o9_6 * Abc0_1 + o9_10 * Abc0_2 + o10_2 * Abc1_0 + o10_6 * Abc1_1 + o10_10 * Abc1_2 + o11_2 * Abc2_0 + o11_6 * Abc2_1 + o11_10 * Abc2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o9_6 * Abd0_2 + o10_6 * Abd1_2 + o11_6 * Abd2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o9_10 * Abd0_2 + o10_10 * Abd1_2 + o11_10 * Abd2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o12_2 * Abd0_2 + o13_2 * Abd1_2 + o14_2 * Abd2_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o12_2 * Abc0_0 + o12_6 * Abc0_1 + o12_10 * Abc0_2 + o13_2 * Abc1_0 + o13_6 * Abc1_1 + o13_10 * Abc1_2 + o14_2 * Abc2_0 + o14_6 * Abc2_1 + o14_10 * Abc2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o12_6 * Abd0_2 + o13_6 * Abd1_2 + o14_6 * Abd2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o12_10 * Abd0_2 + o13_10 * Abd1_2 + o14_10 * Abd2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o15_2 * Abd0_2 + o16_2 * Abd1_2 + o17_2 * Abd2_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o15_2 * Abc0_0 + o15_6 * Abc0_1 + o15_10 * Abc0_2 + o16_2 * Abc1_0 + o16_6 * Abc1_1 + o16_10 * Abc1_2 + o17_2 * Abc2_0 + o17_6 * Abc2_1 + o17_10 * Abc2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o15_6 * Abd0_2 + o16_6 * Abd1_2 + o17_6 * Abd2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o15_10 * Abd0_2 + o16_10 * Abd1_2 + o17_10 * Abd2_2));
          }
        } break;
        case 3: {  // ket functions [3, 7, 11]
          double o0_3 = 0;
          double o0_7 = 0;
          double o0_11 = 0;
          double o1_3 = 0;
          double o1_7 = 0;
          double o1_11 = 0;
          double o2_3 = 0;
          double o2_7 = 0;
          double o2_11 = 0;
          double o3_3 = 0;
          double o3_7 = 0;
          double o3_11 = 0;
          double o4_3 = 0;
          double o4_7 = 0;
          double o4_11 = 0;
          double o5_3 = 0;
          double o5_7 = 0;
          double o5_11 = 0;
          double o6_3 = 0;
          double o6_7 = 0;
          double o6_11 = 0;
          double o7_3 = 0;
          double o7_7 = 0;
          double o7_11 = 0;
          double o8_3 = 0;
          double o8_7 = 0;
          double o8_11 = 0;
          double o9_3 = 0;
          double o9_7 = 0;
          double o9_11 = 0;
          double o10_3 = 0;
          double o10_7 = 0;
          double o10_11 = 0;
          double o11_3 = 0;
          double o11_7 = 0;
          double o11_11 = 0;
          double o12_3 = 0;
          double o12_7 = 0;
          double o12_11 = 0;
          double o13_3 = 0;
          double o13_7 = 0;
          double o13_11 = 0;
          double o14_3 = 0;
          double o14_7 = 0;
          double o14_11 = 0;
          double o15_3 = 0;
          double o15_7 = 0;
          double o15_11 = 0;
          double o16_3 = 0;
          double o16_7 = 0;
          double o16_11 = 0;
          double o17_3 = 0;
          double o17_7 = 0;
          double o17_11 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 113;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g3_0 = 0;
            double g3_1 = 0;
            double g3_2 = 0;
            double g3_3 = 0;
            double g3_4 = 0;
            double g3_5 = 0;
            double g3_6 = 0;
            double g3_7 = 0;
            double g3_8 = 0;
            double g3_9 = 0;
            double g3_10 = 0;
            double g3_11 = 0;
            double g3_12 = 0;
            double g3_13 = 0;
            double g3_14 = 0;
            double g3_15 = 0;
            double g3_16 = 0;
            double g3_17 = 0;
            double g3_18 = 0;
            double g3_19 = 0;
            double g7_0 = 0;
            double g7_1 = 0;
            double g7_2 = 0;
            double g7_3 = 0;
            double g7_4 = 0;
            double g7_5 = 0;
            double g7_6 = 0;
            double g7_7 = 0;
            double g7_8 = 0;
            double g7_9 = 0;
            double g7_10 = 0;
            double g7_11 = 0;
            double g7_12 = 0;
            double g7_13 = 0;
            double g7_14 = 0;
            double g7_15 = 0;
            double g7_16 = 0;
            double g7_17 = 0;
            double g7_18 = 0;
            double g7_19 = 0;
            double g11_0 = 0;
            double g11_1 = 0;
            double g11_2 = 0;
            double g11_3 = 0;
            double g11_4 = 0;
            double g11_5 = 0;
            double g11_6 = 0;
            double g11_7 = 0;
            double g11_8 = 0;
            double g11_9 = 0;
            double g11_10 = 0;
            double g11_11 = 0;
            double g11_12 = 0;
            double g11_13 = 0;
            double g11_14 = 0;
            double g11_15 = 0;
            double g11_16 = 0;
            double g11_17 = 0;
            double g11_18 = 0;
            double g11_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[6];
              sqb::boys<5>(T, a.boys_tab, F);
              const double s0 = TWO_PI_2_5 * rs;
              const double m2a = -2.0 * alpha;
              double w = s0;
              const double b0 = w * F[0];
              w *= m2a;
              const double b1 = w * F[1];
              w *= m2a;
              const double b2 = w * F[2];
              w *= m2a;
              const double b3 = w * F[3];
              w *= m2a;
              const double b4 = w * F[4];
              w *= m2a;
              const double b5 = w * F[5];
              const double ek3_0 = kj[14 * kS];
              const double ek3_1 = -kj[15 * kS];
              const double ek3_2 = -kj[16 * kS];
              const double ek3_3 = kj[17 * kS];
              const double ek7_0 = kj[27 * kS];
              const double ek7_1 = -kj[28 * kS];
              const double ek7_2 = -kj[29 * kS];
              const double ek7_3 = kj[30 * kS];
              const double ek11_0 = kj[41 * kS];
              const double ek11_1 = -kj[42 * kS];
              const double ek11_2 = kj[43 * kS];
              g3_0 = fma(ek3_0, b0, g3_0);
              g7_0 = fma(ek7_0, b0, g7_0);
              g11_0 = fma(ek11_0, b0, g11_0);
              const double r0_0_0_1 = Z * b1;
              g3_1 = fma(ek3_0, r0_0_0_1, g3_1);
              g3_0 = fma(ek3_1, r0_0_0_1, g3_0);
              g7_1 = fma(ek7_0, r0_0_0_1, g7_1);
              g7_0 = fma(ek7_1, r0_0_0_1, g7_0);
              g11_1 = fma(ek11_0, r0_0_0_1, g11_1);
              g11_0 = fma(ek11_1, r0_0_0_1, g11_0);
              const double r0_0_1_0 = Y * b1;
              g3_2 = fma(ek3_0, r0_0_1_0, g3_2);
              g7_2 = fma(ek7_0, r0_0_1_0, g7_2);
              g7_0 = fma(ek7_2, r0_0_1_0, g7_0);
              g11_2 = fma(ek11_0, r0_0_1_0, g11_2);
              const double r0_1_0_0 = X * b1;
              g3_3 = fma(ek3_0, r0_1_0_0, g3_3);
              g3_0 = fma(ek3_2, r0_1_0_0, g3_0);
              g7_3 = fma(ek7_0, r0_1_0_0, g7_3);
              g11_3 = fma(ek11_0, r0_1_0_0, g11_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g3_4 = fma(ek3_0, r0_0_0_2, g3_4);
              g3_1 = fma(ek3_1, r0_0_0_2, g3_1);
              g7_4 = fma(ek7_0, r0_0_0_2, g7_4);
              g7_1 = fma(ek7_1, r0_0_0_2, g7_1);
              g11_4 = fma(ek11_0, r0_0_0_2, g11_4);
              g11_1 = fma(ek11_1, r0_0_0_2, g11_1);
              g11_0 = fma(ek11_2, r0_0_0_2, g11_0);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g3_5 = fma(ek3_0, r0_0_1_1, g3_5);
              g3_2 = fma(ek3_1, r0_0_1_1, g3_2);
              g7_5 = fma(ek7_0, r0_0_1_1, g7_5);
              g7_2 = fma(ek7_1, r0_0_1_1, g7_2);
              g7_1 = fma(ek7_2, r0_0_1_1, g7_1);
              g7_0 = fma(ek7_3, r0_0_1_1, g7_0);
              g11_5 = fma(ek11_0, r0_0_1_1, g11_5);
              g11_2 = fma(ek11_1, r0_0_1_1, g11_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g3_6 = fma(ek3_0, r0_0_2_0, g3_6);
              g7_6 = fma(ek7_0, r0_0_2_0, g7_6);
              g7_2 = fma(ek7_2, r0_0_2_0, g7_2);
              g11_6 = fma(ek11_0, r0_0_2_0, g11_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g3_7 = fma(ek3_0, r0_1_0_1, g3_7);
              g3_3 = fma(ek3_1, r0_1_0_1, g3_3);
              g3_1 = fma(ek3_2, r0_1_0_1, g3_1);
              g3_0 = fma(ek3_3, r0_1_0_1, g3_0);
              g7_7 = fma(ek7_0, r0_1_0_1, g7_7);
              g7_3 = fma(ek7_1, r0_1_0_1, g7_3);
              g11_7 = fma(ek11_0, r0_1_0_1, g11_7);
              g11_3 = fma(ek11_1, r0_1_0_1, g11_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g3_8 = fma(ek3_0, r0_1_1_0, g3_8);
              g3_2 = fma(ek3_2, r0_1_1_0, g3_2);
              g7_8 = fma(ek7_0, r0_1_1_0, g7_8);
              g7_3 = fma(ek7_2, r0_1_1_0, g7_3);
              g11_8 = fma(ek11_0, r0_1_1_0, g11_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g3_9 = fma(ek3_0, r0_2_0_0, g3_9);
              g3_3 = fma(ek3_2, r0_2_0_0, g3_3);
              g7_9 = fma(ek7_0, r0_2_0_0, g7_9);
              g11_9 = fma(ek11_0, r0_2_0_0, g11_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g3_10 = fma(ek3_0, r0_0_0_3, g3_10);
              g3_4 = fma(ek3_1, r0_0_0_3, g3_4);
              g7_10 = fma(ek7_0, r0_0_0_3, g7_10);
              g7_4 = fma(ek7_1, r0_0_0_3, g7_4);
              g11_10 = fma(ek11_0, r0_0_0_3, g11_10);
              g11_4 = fma(ek11_1, r0_0_0_3, g11_4);
              g11_1 = fma(ek11_2, r0_0_0_3, g11_1);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g3_11 = fma(ek3_0, r0_0_1_2, g3_11);
              g3_5 = fma(ek3_1, r0_0_1_2, g3_5);
              g7_11 = fma(ek7_0, r0_0_1_2, g7_11);
              g7_5 = fma(ek7_1, r0_0_1_2, g7_5);
              g7_4 = fma(ek7_2, r0_0_1_2, g7_4);
              g7_1 = fma(ek7_3, r0_0_1_2, g7_1);
              g11_11 = fma(ek11_0, r0_0_1_2, g11_11);
              g11_5 = fma(ek11_1, r0_0_1_2, g11_5);
              g11_2 = fma(ek11_2, r0_0_1_2, g11_2);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g3_12 = fma(ek3_0, r0_0_2_1, g3_12);
              g3_6 = fma(ek3_1, r0_0_2_1, g3_6);
              g7_12 = fma(ek7_0, r0_0_2_1, g7_12);
              g7_6 = fma(ek7_1, r0_0_2_1, g7_6);
              g7_5 = fma(ek7_2, r0_0_2_1, g7_5);
              g7_2 = fma(ek7_3, r0_0_2_1, g7_2);
              g11_12 = fma(ek11_0, r0_0_2_1, g11_12);
              g11_6 = fma(ek11_1, r0_0_2_1, g11_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g3_13 = fma(ek3_0, r0_0_3_0, g3_13);
              g7_13 = fma(ek7_0, r0_0_3_0, g7_13);
              g7_6 = fma(ek7_2, r0_0_3_0, g7_6);
              g11_13 = fma(ek11_0, r0_0_3_0, g11_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g3_14 = fma(ek3_0, r0_1_0_2, g3_14);
              g3_7 = fma(ek3_1, r0_1_0_2, g3_7);
              g3_4 = fma(ek3_2, r0_1_0_2, g3_4);
              g3_1 = fma(ek3_3, r0_1_0_2, g3_1);
              g7_14 = fma(ek7_0, r0_1_0_2, g7_14);
              g7_7 = fma(ek7_1, r0_1_0_2, g7_7);
              g11_14 = fma(ek11_0, r0_1_0_2, g11_14);
              g11_7 = fma(ek11_1, r0_1_0_2, g11_7);
              g11_3 = fma(ek11_2, r0_1_0_2, g11_3);
              const double r0_1_1_1 = X * r1_0_1_1;
              g3_15 = fma(ek3_0, r0_1_1_1, g3_15);
              g3_8 = fma(ek3_1, r0_1_1_1, g3_8);
              g3_5 = fma(ek3_2, r0_1_1_1, g3_5);
              g3_2 = fma(ek3_3, r0_1_1_1, g3_2);
              g7_15 = fma(ek7_0, r0_1_1_1, g7_15);
              g7_8 = fma(ek7_1, r0_1_1_1, g7_8);
              g7_7 = fma(ek7_2, r0_1_1_1, g7_7);
              g7_3 = fma(ek7_3, r0_1_1_1, g7_3);
              g11_15 = fma(ek11_0, r0_1_1_1, g11_15);
              g11_8 = fma(ek11_1, r0_1_1_1, g11_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g3_16 = fma(ek3_0, r0_1_2_0, g3_16);
              g3_6 = fma(ek3_2, r0_1_2_0, g3_6);
              g7_16 = fma(ek7_0, r0_1_2_0, g7_16);
              g7_8 = fma(ek7_2, r0_1_2_0, g7_8);
              g11_16 = fma(ek11_0, r0_1_2_0, g11_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g3_17 = fma(ek3_0, r0_2_0_1, g3_17);
              g3_9 = fma(ek3_1, r0_2_0_1, g3_9);
              g3_7 = fma(ek3_2, r0_2_0_1, g3_7);
              g3_3 = fma(ek3_3, r0_2_0_1, g3_3);
              g7_17 = fma(ek7_0, r0_2_0_1, g7_17);
              g7_9 = fma(ek7_1, r0_2_0_1, g7_9);
              g11_17 = fma(ek11_0, r0_2_0_1, g11_17);
              g11_9 = fma(ek11_1, r0_2_0_1, g11_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g3_18 = fma(ek3_0, r0_2_1_0, g3_18);
              g3_8 = fma(ek3_2, r0_2_1_0, g3_8);
              g7_18 = fma(ek7_0, r0_2_1_0, g7_18);
              g7_9 = fma(ek7_2, r0_2_1_0, g7_9);
              g11_18 = fma(ek11_0, r0_2_1_0, g11_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g3_19 = fma(ek3_0, r0_3_0_0, g3_19);
              g3_9 = fma(ek3_2, r0_3_0_0, g3_9);
              g7_19 = fma(ek7_0, r0_3_0_0, g7_19);
              g11_19 = fma(ek11_0, r0_3_0_0, g11_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g3_10 = fma(ek3_1, r0_0_0_4, g3_10);
              g7_10 = fma(ek7_1, r0_0_0_4, g7_10);
              g11_10 = fma(ek11_1, r0_0_0_4, g11_10);
              g11_4 = fma(ek11_2, r0_0_0_4, g11_4);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g3_11 = fma(ek3_1, r0_0_1_3, g3_11);
              g7_11 = fma(ek7_1, r0_0_1_3, g7_11);
              g7_10 = fma(ek7_2, r0_0_1_3, g7_10);
              g7_4 = fma(ek7_3, r0_0_1_3, g7_4);
              g11_11 = fma(ek11_1, r0_0_1_3, g11_11);
              g11_5 = fma(ek11_2, r0_0_1_3, g11_5);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g3_12 = fma(ek3_1, r0_0_2_2, g3_12);
              g7_12 = fma(ek7_1, r0_0_2_2, g7_12);
              g7_11 = fma(ek7_2, r0_0_2_2, g7_11);
              g7_5 = fma(ek7_3, r0_0_2_2, g7_5);
              g11_12 = fma(ek11_1, r0_0_2_2, g11_12);
              g11_6 = fma(ek11_2, r0_0_2_2, g11_6);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g3_13 = fma(ek3_1, r0_0_3_1, g3_13);
              g7_13 = fma(ek7_1, r0_0_3_1, g7_13);
              g7_12 = fma(ek7_2, r0_0_3_1, g7_12);
              g7_6 = fma(ek7_3, r0_0_3_1, g7_6);
              g11_13 = fma(ek11_1, r0_0_3_1, g11_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g7_13 = fma(ek7_2, r0_0_4_0, g7_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g3_14 = fma(ek3_1, r0_1_0_3, g3_14);
              g3_10 = fma(ek3_2, r0_1_0_3, g3_10);
              g3_4 = fma(ek3_3, r0_1_0_3, g3_4);
              g7_14 = fma(ek7_1, r0_1_0_3, g7_14);
              g11_14 = fma(ek11_1, r0_1_0_3, g11_14);
              g11_7 = fma(ek11_2, r0_1_0_3, g11_7);
              const double r0_1_1_2 = X * r1_0_1_2;
              g3_15 = fma(ek3_1, r0_1_1_2, g3_15);
              g3_11 = fma(ek3_2, r0_1_1_2, g3_11);
              g3_5 = fma(ek3_3, r0_1_1_2, g3_5);
              g7_15 = fma(ek7_1, r0_1_1_2, g7_15);
              g7_14 = fma(ek7_2, r0_1_1_2, g7_14);
              g7_7 = fma(ek7_3, r0_1_1_2, g7_7);
              g11_15 = fma(ek11_1, r0_1_1_2, g11_15);
              g11_8 = fma(ek11_2, r0_1_1_2, g11_8);
              const double r0_1_2_1 = X * r1_0_2_1;
              g3_16 = fma(ek3_1, r0_1_2_1, g3_16);
              g3_12 = fma(ek3_2, r0_1_2_1, g3_12);
              g3_6 = fma(ek3_3, r0_1_2_1, g3_6);
              g7_16 = fma(ek7_1, r0_1_2_1, g7_16);
              g7_15 = fma(ek7_2, r0_1_2_1, g7_15);
              g7_8 = fma(ek7_3, r0_1_2_1, g7_8);
              g11_16 = fma(ek11_1, r0_1_2_1, g11_16);
              const double r0_1_3_0 = X * r1_0_3_0;
              g3_13 = fma(ek3_2, r0_1_3_0, g3_13);
              g7_16 = fma(ek7_2, r0_1_3_0, g7_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g3_17 = fma(ek3_1, r0_2_0_2, g3_17);
              g3_14 = fma(ek3_2, r0_2_0_2, g3_14);
              g3_7 = fma(ek3_3, r0_2_0_2, g3_7);
              g7_17 = fma(ek7_1, r0_2_0_2, g7_17);
              g11_17 = fma(ek11_1, r0_2_0_2, g11_17);
              g11_9 = fma(ek11_2, r0_2_0_2, g11_9);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g3_18 = fma(ek3_1, r0_2_1_1, g3_18);
              g3_15 = fma(ek3_2, r0_2_1_1, g3_15);
              g3_8 = fma(ek3_3, r0_2_1_1, g3_8);
              g7_18 = fma(ek7_1, r0_2_1_1, g7_18);
              g7_17 = fma(ek7_2, r0_2_1_1, g7_17);
              g7_9 = fma(ek7_3, r0_2_1_1, g7_9);
              g11_18 = fma(ek11_1, r0_2_1_1, g11_18);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g3_16 = fma(ek3_2, r0_2_2_0, g3_16);
              g7_18 = fma(ek7_2, r0_2_2_0, g7_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g3_19 = fma(ek3_1, r0_3_0_1, g3_19);
              g3_17 = fma(ek3_2, r0_3_0_1, g3_17);
              g3_9 = fma(ek3_3, r0_3_0_1, g3_9);
              g7_19 = fma(ek7_1, r0_3_0_1, g7_19);
              g11_19 = fma(ek11_1, r0_3_0_1, g11_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g3_18 = fma(ek3_2, r0_3_1_0, g3_18);
              g7_19 = fma(ek7_2, r0_3_1_0, g7_19);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g3_19 = fma(ek3_2, r0_4_0_0, g3_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g11_10 = fma(ek11_2, r0_0_0_5, g11_10);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g7_10 = fma(ek7_3, r0_0_1_4, g7_10);
              g11_11 = fma(ek11_2, r0_0_1_4, g11_11);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g7_11 = fma(ek7_3, r0_0_2_3, g7_11);
              g11_12 = fma(ek11_2, r0_0_2_3, g11_12);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g7_12 = fma(ek7_3, r0_0_3_2, g7_12);
              g11_13 = fma(ek11_2, r0_0_3_2, g11_13);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g7_13 = fma(ek7_3, r0_0_4_1, g7_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g3_10 = fma(ek3_3, r0_1_0_4, g3_10);
              g11_14 = fma(ek11_2, r0_1_0_4, g11_14);
              const double r0_1_1_3 = X * r1_0_1_3;
              g3_11 = fma(ek3_3, r0_1_1_3, g3_11);
              g7_14 = fma(ek7_3, r0_1_1_3, g7_14);
              g11_15 = fma(ek11_2, r0_1_1_3, g11_15);
              const double r0_1_2_2 = X * r1_0_2_2;
              g3_12 = fma(ek3_3, r0_1_2_2, g3_12);
              g7_15 = fma(ek7_3, r0_1_2_2, g7_15);
              g11_16 = fma(ek11_2, r0_1_2_2, g11_16);
              const double r0_1_3_1 = X * r1_0_3_1;
              g3_13 = fma(ek3_3, r0_1_3_1, g3_13);
              g7_16 = fma(ek7_3, r0_1_3_1, g7_16);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g3_14 = fma(ek3_3, r0_2_0_3, g3_14);
              g11_17 = fma(ek11_2, r0_2_0_3, g11_17);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g3_15 = fma(ek3_3, r0_2_1_2, g3_15);
              g7_17 = fma(ek7_3, r0_2_1_2, g7_17);
              g11_18 = fma(ek11_2, r0_2_1_2, g11_18);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g3_16 = fma(ek3_3, r0_2_2_1, g3_16);
              g7_18 = fma(ek7_3, r0_2_2_1, g7_18);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g3_17 = fma(ek3_3, r0_3_0_2, g3_17);
              g11_19 = fma(ek11_2, r0_3_0_2, g11_19);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g3_18 = fma(ek3_3, r0_3_1_1, g3_18);
              g7_19 = fma(ek7_3, r0_3_1_1, g7_19);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g3_19 = fma(ek3_3, r0_4_0_1, g3_19);
            }
            { const double eb = bi[5];
              o0_3 = fma(eb, g3_0, o0_3);
              o0_7 = fma(eb, g7_0, o0_7);
              o0_11 = fma(eb, g11_0, o0_11);
            }
            { const double eb = bi[6];
              o0_3 = fma(eb, g3_3, o0_3);
              o0_7 = fma(eb, g7_3, o0_7);
              o0_11 = fma(eb, g11_3, o0_11);
            }
            { const double eb = bi[7];
              o0_3 = fma(eb, g3_9, o0_3);
              o0_7 = fma(eb, g7_9, o0_7);
              o0_11 = fma(eb, g11_9, o0_11);
            }
            { const double eb = bi[8];
              o0_3 = fma(eb, g3_19, o0_3);
              o0_7 = fma(eb, g7_19, o0_7);
              o0_11 = fma(eb, g11_19, o0_11);
            }
            { const double eb = bi[9];
              o1_3 = fma(eb, g3_0, o1_3);
              o1_7 = fma(eb, g7_0, o1_7);
              o1_11 = fma(eb, g11_0, o1_11);
            }
            { const double eb = bi[10];
              o1_3 = fma(eb, g3_2, o1_3);
              o1_7 = fma(eb, g7_2, o1_7);
              o1_11 = fma(eb, g11_2, o1_11);
            }
            { const double eb = bi[11];
              o1_3 = fma(eb, g3_3, o1_3);
              o1_7 = fma(eb, g7_3, o1_7);
              o1_11 = fma(eb, g11_3, o1_11);
            }
            { const double eb = bi[12];
              o1_3 = fma(eb, g3_8, o1_3);
              o1_7 = fma(eb, g7_8, o1_7);
              o1_11 = fma(eb, g11_8, o1_11);
            }
            { const double eb = bi[13];
              o1_3 = fma(eb, g3_9, o1_3);
              o1_7 = fma(eb, g7_9, o1_7);
              o1_11 = fma(eb, g11_9, o1_11);
            }
            { const double eb = bi[14];
              o1_3 = fma(eb, g3_18, o1_3);
              o1_7 = fma(eb, g7_18, o1_7);
              o1_11 = fma(eb, g11_18, o1_11);
            }
            { const double eb = bi[15];
              o2_3 = fma(eb, g3_0, o2_3);
              o2_7 = fma(eb, g7_0, o2_7);
              o2_11 = fma(eb, g11_0, o2_11);
            }
            { const double eb = bi[16];
              o2_3 = fma(eb, g3_1, o2_3);
              o2_7 = fma(eb, g7_1, o2_7);
              o2_11 = fma(eb, g11_1, o2_11);
            }
            { const double eb = bi[17];
              o2_3 = fma(eb, g3_3, o2_3);
              o2_7 = fma(eb, g7_3, o2_7);
              o2_11 = fma(eb, g11_3, o2_11);
            }
            { const double eb = bi[18];
              o2_3 = fma(eb, g3_7, o2_3);
              o2_7 = fma(eb, g7_7, o2_7);
              o2_11 = fma(eb, g11_7, o2_11);
            }
            { const double eb = bi[19];
              o2_3 = fma(eb, g3_9, o2_3);
              o2_7 = fma(eb, g7_9, o2_7);
              o2_11 = fma(eb, g11_9, o2_11);
            }
            { const double eb = bi[20];
              o2_3 = fma(eb, g3_17, o2_3);
              o2_7 = fma(eb, g7_17, o2_7);
              o2_11 = fma(eb, g11_17, o2_11);
            }
            { const double eb = bi[21];
              o3_3 = fma(eb, g3_0, o3_3);
              o3_7 = fma(eb, g7_0, o3_7);
              o3_11 = fma(eb, g11_0, o3_11);
            }
            { const double eb = bi[22];
              o3_3 = fma(eb, g3_2, o3_3);
              o3_7 = fma(eb, g7_2, o3_7);
              o3_11 = fma(eb, g11_2, o3_11);
            }
            { const double eb = bi[23];
              o3_3 = fma(eb, g3_6, o3_3);
              o3_7 = fma(eb, g7_6, o3_7);
              o3_11 = fma(eb, g11_6, o3_11);
            }
            { const double eb = bi[24];
              o3_3 = fma(eb, g3_3, o3_3);
              o3_7 = fma(eb, g7_3, o3_7);
              o3_11 = fma(eb, g11_3, o3_11);
            }
            { const double eb = bi[25];
              o3_3 = fma(eb, g3_8, o3_3);
              o3_7 = fma(eb, g7_8, o3_7);
              o3_11 = fma(eb, g11_8, o3_11);
            }
            { const double eb = bi[26];
              o3_3 = fma(eb, g3_16, o3_3);
              o3_7 = fma(eb, g7_16, o3_7);
              o3_11 = fma(eb, g11_16, o3_11);
            }
            { const double eb = bi[27];
              o4_3 = fma(eb, g3_0, o4_3);
              o4_7 = fma(eb, g7_0, o4_7);
              o4_11 = fma(eb, g11_0, o4_11);
            }
            { const double eb = bi[28];
              o4_3 = fma(eb, g3_2, o4_3);
              o4_7 = fma(eb, g7_2, o4_7);
              o4_11 = fma(eb, g11_2, o4_11);
            }
            { const double eb = bi[29];
              o4_3 = fma(eb, g3_6, o4_3);
              o4_7 = fma(eb, g7_6, o4_7);
              o4_11 = fma(eb, g11_6, o4_11);
            }
            { const double eb = bi[30];
              o4_3 = fma(eb, g3_13, o4_3);
              o4_7 = fma(eb, g7_13, o4_7);
              o4_11 = fma(eb, g11_13, o4_11);
            }
            { const double eb = bi[31];
              o5_3 = fma(eb, g3_0, o5_3);
              o5_7 = fma(eb, g7_0, o5_7);
              o5_11 = fma(eb, g11_0, o5_11);
            }
            { const double eb = bi[32];
              o5_3 = fma(eb, g3_1, o5_3);
              o5_7 = fma(eb, g7_1, o5_7);
              o5_11 = fma(eb, g11_1, o5_11);
            }
            { const double eb = bi[33];
              o5_3 = fma(eb, g3_2, o5_3);
              o5_7 = fma(eb, g7_2, o5_7);
              o5_11 = fma(eb, g11_2, o5_11);
            }
            { const double eb = bi[34];
              o5_3 = fma(eb, g3_5, o5_3);
              o5_7 = fma(eb, g7_5, o5_7);
              o5_11 = fma(eb, g11_5, o5_11);
            }
            { const double eb = bi[35];
              o5_3 = fma(eb, g3_6, o5_3);
              o5_7 = fma(eb, g7_6, o5_7);
              o5_11 = fma(eb, g11_6, o5_11);
            }
            { const double eb = bi[36];
              o5_3 = fma(eb, g3_12, o5_3);
              o5_7 = fma(eb, g7_12, o5_7);
              o5_11 = fma(eb, g11_12, o5_11);
            }
            { const double eb = bi[37];
              o6_3 = fma(eb, g3_0, o6_3);
              o6_7 = fma(eb, g7_0, o6_7);
              o6_11 = fma(eb, g11_0, o6_11);
            }
            { const double eb = bi[38];
              o6_3 = fma(eb, g3_1, o6_3);
              o6_7 = fma(eb, g7_1, o6_7);
              o6_11 = fma(eb, g11_1, o6_11);
            }
            { const double eb = bi[39];
              o6_3 = fma(eb, g3_4, o6_3);
              o6_7 = fma(eb, g7_4, o6_7);
              o6_11 = fma(eb, g11_4, o6_11);
            }
            { const double eb = bi[40];
              o6_3 = fma(eb, g3_3, o6_3);
              o6_7 = fma(eb, g7_3, o6_7);
              o6_11 = fma(eb, g11_3, o6_11);
            }
            { const double eb = bi[41];
              o6_3 = fma(eb, g3_7, o6_3);
              o6_7 = fma(eb, g7_7, o6_7);
              o6_11 = fma(eb, g11_7, o6_11);
            }
            { const double eb = bi[42];
              o6_3 = fma(eb, g3_14, o6_3);
              o6_7 = fma(eb, g7_14, o6_7);
              o6_11 = fma(eb, g11_14, o6_11);
            }
            { const double eb = bi[43];
              o7_3 = fma(eb, g3_0, o7_3);
              o7_7 = fma(eb, g7_0, o7_7);
              o7_11 = fma(eb, g11_0, o7_11);
            }
            { const double eb = bi[44];
              o7_3 = fma(eb, g3_1, o7_3);
              o7_7 = fma(eb, g7_1, o7_7);
              o7_11 = fma(eb, g11_1, o7_11);
            }
            { const double eb = bi[45];
              o7_3 = fma(eb, g3_4, o7_3);
              o7_7 = fma(eb, g7_4, o7_7);
              o7_11 = fma(eb, g11_4, o7_11);
            }
            { const double eb = bi[46];
              o7_3 = fma(eb, g3_2, o7_3);
              o7_7 = fma(eb, g7_2, o7_7);
              o7_11 = fma(eb, g11_2, o7_11);
            }
            { const double eb = bi[47];
              o7_3 = fma(eb, g3_5, o7_3);
              o7_7 = fma(eb, g7_5, o7_7);
              o7_11 = fma(eb, g11_5, o7_11);
            }
            { const double eb = bi[48];
              o7_3 = fma(eb, g3_11, o7_3);
              o7_7 = fma(eb, g7_11, o7_7);
              o7_11 = fma(eb, g11_11, o7_11);
            }
            { const double eb = bi[49];
              o8_3 = fma(eb, g3_0, o8_3);
              o8_7 = fma(eb, g7_0, o8_7);
              o8_11 = fma(eb, g11_0, o8_11);
            }
            { const double eb = bi[50];
              o8_3 = fma(eb, g3_1, o8_3);
              o8_7 = fma(eb, g7_1, o8_7);
              o8_11 = fma(eb, g11_1, o8_11);
            }
            { const double eb = bi[51];
              o8_3 = fma(eb, g3_4, o8_3);
              o8_7 = fma(eb, g7_4, o8_7);
              o8_11 = fma(eb, g11_4, o8_11);
            }
            { const double eb = bi[52];
              o8_3 = fma(eb, g3_10, o8_3);
              o8_7 = fma(eb, g7_10, o8_7);
              o8_11 = fma(eb, g11_10, o8_11);
            }
            { const double eb = bi[53];
              o9_3 = fma(eb, g3_0, o9_3);
              o9_7 = fma(eb, g7_0, o9_7);
              o9_11 = fma(eb, g11_0, o9_11);
            }
            { const double eb = bi[54];
              o9_3 = fma(eb, g3_2, o9_3);
              o9_7 = fma(eb, g7_2, o9_7);
              o9_11 = fma(eb, g11_2, o9_11);
            }
            { const double eb = bi[55];
              o9_3 = fma(eb, g3_3, o9_3);
              o9_7 = fma(eb, g7_3, o9_7);
              o9_11 = fma(eb, g11_3, o9_11);
            }
            { const double eb = bi[56];
              o9_3 = fma(eb, g3_8, o9_3);
              o9_7 = fma(eb, g7_8, o9_7);
              o9_11 = fma(eb, g11_8, o9_11);
            }
            { const double eb = bi[57];
              o9_3 = fma(eb, g3_9, o9_3);
              o9_7 = fma(eb, g7_9, o9_7);
              o9_11 = fma(eb, g11_9, o9_11);
            }
            { const double eb = bi[58];
              o9_3 = fma(eb, g3_18, o9_3);
              o9_7 = fma(eb, g7_18, o9_7);
              o9_11 = fma(eb, g11_18, o9_11);
            }
            { const double eb = bi[59];
              o10_3 = fma(eb, g3_0, o10_3);
              o10_7 = fma(eb, g7_0, o10_7);
              o10_11 = fma(eb, g11_0, o10_11);
            }
            { const double eb = bi[60];
              o10_3 = fma(eb, g3_2, o10_3);
              o10_7 = fma(eb, g7_2, o10_7);
              o10_11 = fma(eb, g11_2, o10_11);
            }
            { const double eb = bi[61];
              o10_3 = fma(eb, g3_6, o10_3);
              o10_7 = fma(eb, g7_6, o10_7);
              o10_11 = fma(eb, g11_6, o10_11);
            }
            { const double eb = bi[62];
              o10_3 = fma(eb, g3_3, o10_3);
              o10_7 = fma(eb, g7_3, o10_7);
              o10_11 = fma(eb, g11_3, o10_11);
            }
            { const double eb = bi[63];
              o10_3 = fma(eb, g3_8, o10_3);
              o10_7 = fma(eb, g7_8, o10_7);
              o10_11 = fma(eb, g11_8, o10_11);
            }
            { const double eb = bi[64];
              o10_3 = fma(eb, g3_16, o10_3);
              o10_7 = fma(eb, g7_16, o10_7);
              o10_11 = fma(eb, g11_16, o10_11);
            }
            { const double eb = bi[65];
              o11_3 = fma(eb, g3_0, o11_3);
              o11_7 = fma(eb, g7_0, o11_7);
              o11_11 = fma(eb, g11_0, o11_11);
            }
            { const double eb = bi[66];
              o11_3 = fma(eb, g3_1, o11_3);
              o11_7 = fma(eb, g7_1, o11_7);
              o11_11 = fma(eb, g11_1, o11_11);
            }
            { const double eb = bi[67];
              o11_3 = fma(eb, g3_2, o11_3);
              o11_7 = fma(eb, g7_2, o11_7);
              o11_11 = fma(eb, g11_2, o11_11);
            }
            { const double eb = bi[68];
              o11_3 = fma(eb, g3_5, o11_3);
              o11_7 = fma(eb, g7_5, o11_7);
              o11_11 = fma(eb, g11_5, o11_11);
            }
            { const double eb = bi[69];
              o11_3 = fma(eb, g3_3, o11_3);
              o11_7 = fma(eb, g7_3, o11_7);
              o11_11 = fma(eb, g11_3, o11_11);
            }
            { const double eb = bi[70];
              o11_3 = fma(eb, g3_7, o11_3);
              o11_7 = fma(eb, g7_7, o11_7);
              o11_11 = fma(eb, g11_7, o11_11);
            }
            { const double eb = bi[71];
              o11_3 = fma(eb, g3_8, o11_3);
              o11_7 = fma(eb, g7_8, o11_7);
              o11_11 = fma(eb, g11_8, o11_11);
            }
            { const double eb = bi[72];
              o11_3 = fma(eb, g3_15, o11_3);
              o11_7 = fma(eb, g7_15, o11_7);
              o11_11 = fma(eb, g11_15, o11_11);
            }
            { const double eb = bi[73];
              o12_3 = fma(eb, g3_0, o12_3);
              o12_7 = fma(eb, g7_0, o12_7);
              o12_11 = fma(eb, g11_0, o12_11);
            }
            { const double eb = bi[74];
              o12_3 = fma(eb, g3_1, o12_3);
              o12_7 = fma(eb, g7_1, o12_7);
              o12_11 = fma(eb, g11_1, o12_11);
            }
            { const double eb = bi[75];
              o12_3 = fma(eb, g3_3, o12_3);
              o12_7 = fma(eb, g7_3, o12_7);
              o12_11 = fma(eb, g11_3, o12_11);
            }
            { const double eb = bi[76];
              o12_3 = fma(eb, g3_7, o12_3);
              o12_7 = fma(eb, g7_7, o12_7);
              o12_11 = fma(eb, g11_7, o12_11);
            }
            { const double eb = bi[77];
              o12_3 = fma(eb, g3_9, o12_3);
              o12_7 = fma(eb, g7_9, o12_7);
              o12_11 = fma(eb, g11_9, o12_11);
            }
            { const double eb = bi[78];
              o12_3 = fma(eb, g3_17, o12_3);
              o12_7 = fma(eb, g7_17, o12_7);
              o12_11 = fma(eb, g11_17, o12_11);
            }
            { const double eb = bi[79];
              o13_3 = fma(eb, g3_0, o13_3);
              o13_7 = fma(eb, g7_0, o13_7);
              o13_11 = fma(eb, g11_0, o13_11);
            }
            { const double eb = bi[80];
              o13_3 = fma(eb, g3_1, o13_3);
              o13_7 = fma(eb, g7_1, o13_7);
              o13_11 = fma(eb, g11_1, o13_11);
            }
            { const double eb = bi[81];
              o13_3 = fma(eb, g3_2, o13_3);
              o13_7 = fma(eb, g7_2, o13_7);
              o13_11 = fma(eb, g11_2, o13_11);
            }
            { const double eb = bi[82];
              o13_3 = fma(eb, g3_5, o13_3);
              o13_7 = fma(eb, g7_5, o13_7);
              o13_11 = fma(eb, g11_5, o13_11);
            }
            { const double eb = bi[83];
              o13_3 = fma(eb, g3_3, o13_3);
              o13_7 = fma(eb, g7_3, o13_7);
              o13_11 = fma(eb, g11_3, o13_11);
            }
            { const double eb = bi[84];
              o13_3 = fma(eb, g3_7, o13_3);
              o13_7 = fma(eb, g7_7, o13_7);
              o13_11 = fma(eb, g11_7, o13_11);
            }
            { const double eb = bi[85];
              o13_3 = fma(eb, g3_8, o13_3);
              o13_7 = fma(eb, g7_8, o13_7);
              o13_11 = fma(eb, g11_8, o13_11);
            }
            { const double eb = bi[86];
              o13_3 = fma(eb, g3_15, o13_3);
              o13_7 = fma(eb, g7_15, o13_7);
              o13_11 = fma(eb, g11_15, o13_11);
            }
            { const double eb = bi[87];
              o14_3 = fma(eb, g3_0, o14_3);
              o14_7 = fma(eb, g7_0, o14_7);
              o14_11 = fma(eb, g11_0, o14_11);
            }
            { const double eb = bi[88];
              o14_3 = fma(eb, g3_1, o14_3);
              o14_7 = fma(eb, g7_1, o14_7);
              o14_11 = fma(eb, g11_1, o14_11);
            }
            { const double eb = bi[89];
              o14_3 = fma(eb, g3_4, o14_3);
              o14_7 = fma(eb, g7_4, o14_7);
              o14_11 = fma(eb, g11_4, o14_11);
            }
            { const double eb = bi[90];
              o14_3 = fma(eb, g3_3, o14_3);
              o14_7 = fma(eb, g7_3, o14_7);
              o14_11 = fma(eb, g11_3, o14_11);
            }
            { const double eb = bi[91];
              o14_3 = fma(eb, g3_7, o14_3);
              o14_7 = fma(eb, g7_7, o14_7);
              o14_11 = fma(eb, g11_7, o14_11);
            }
            { const double eb = bi[92];
              o14_3 = fma(eb, g3_14, o14_3);
              o14_7 = fma(eb, g7_14, o14_7);
              o14_11 = fma(eb, g11_14, o14_11);
            }
            { const double eb = bi[93];
              o15_3 = fma(eb, g3_0, o15_3);
              o15_7 = fma(eb, g7_0, o15_7);
              o15_11 = fma(eb, g11_0, o15_11);
            }
            { const double eb = bi[94];
              o15_3 = fma(eb, g3_1, o15_3);
              o15_7 = fma(eb, g7_1, o15_7);
              o15_11 = fma(eb, g11_1, o15_11);
            }
            { const double eb = bi[95];
              o15_3 = fma(eb, g3_2, o15_3);
              o15_7 = fma(eb, g7_2, o15_7);
              o15_11 = fma(eb, g11_2, o15_11);
            }
            { const double eb = bi[96];
              o15_3 = fma(eb, g3_5, o15_3);
              o15_7 = fma(eb, g7_5, o15_7);
              o15_11 = fma(eb, g11_5, o15_11);
            }
            { const double eb = bi[97];
              o15_3 = fma(eb, g3_3, o15_3);
              o15_7 = fma(eb, g7_3, o15_7);
              o15_11 = fma(eb, g11_3, o15_11);
            }
            { const double eb = bi[98];
              o15_3 = fma(eb, g3_7, o15_3);
              o15_7 = fma(eb, g7_7, o15_7);
              o15_11 = fma(eb, g11_7, o15_11);
            }
            { const double eb = bi[99];
              o15_3 = fma(eb, g3_8, o15_3);
              o15_7 = fma(eb, g7_8, o15_7);
              o15_11 = fma(eb, g11_8, o15_11);
            }
            { const double eb = bi[100];
              o15_3 = fma(eb, g3_15, o15_3);
              o15_7 = fma(eb, g7_15, o15_7);
              o15_11 = fma(eb, g11_15, o15_11);
            }
            { const double eb = bi[101];
              o16_3 = fma(eb, g3_0, o16_3);
              o16_7 = fma(eb, g7_0, o16_7);
              o16_11 = fma(eb, g11_0, o16_11);
            }
            { const double eb = bi[102];
              o16_3 = fma(eb, g3_1, o16_3);
              o16_7 = fma(eb, g7_1, o16_7);
              o16_11 = fma(eb, g11_1, o16_11);
            }
            { const double eb = bi[103];
              o16_3 = fma(eb, g3_2, o16_3);
              o16_7 = fma(eb, g7_2, o16_7);
              o16_11 = fma(eb, g11_2, o16_11);
            }
            { const double eb = bi[104];
              o16_3 = fma(eb, g3_5, o16_3);
              o16_7 = fma(eb, g7_5, o16_7);
              o16_11 = fma(eb, g11_5, o16_11);
            }
            { const double eb = bi[105];
              o16_3 = fma(eb, g3_6, o16_3);
              o16_7 = fma(eb, g7_6, o16_7);
              o16_11 = fma(eb, g11_6, o16_11);
            }
            { const double eb = bi[106];
              o16_3 = fma(eb, g3_12, o16_3);
              o16_7 = fma(eb, g7_12, o16_7);
              o16_11 = fma(eb, g11_12, o16_11);
            }
            { const double eb = bi[107];
              o17_3 = fma(eb, g3_0, o17_3);
              o17_7 = fma(eb, g7_0, o17_7);
              o17_11 = fma(eb, g11_0, o17_11);
            }
            { const double eb = bi[108];
              o17_3 = fma(eb, g3_1, o17_3);
              o17_7 = fma(eb, g7_1, o17_7);
              o17_11 = fma(eb, g11_1, o17_11);
            }
            { const double eb = bi[109];
              o17_3 = fma(eb, g3_4, o17_3);
              o17_7 = fma(eb, g7_4, o17_7);
              o17_11 = fma(eb, g11_4, o17_11);
            }
            { const double eb = bi[110];
              o17_3 = fma(eb, g3_2, o17_3);
              o17_7 = fma(eb, g7_2, o17_7);
              o17_11 = fma(eb, g11_2, o17_11);
            }
            { const double eb = bi[111];
              o17_3 = fma(eb, g3_5, o17_3);
              o17_7 = fma(eb, g7_5, o17_7);
              o17_11 = fma(eb, g11_5, o17_11);
            }
            { const double eb = bi[112];
              o17_3 = fma(eb, g3_11, o17_3);
              o17_7 = fma(eb, g7_11, o17_7);
              o17_11 = fma(eb, g11_11, o17_11);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk3 = PT[(fI + 0) * N + fJ + 3];
            const double ptk7 = PT[(fI + 1) * N + fJ + 3];
            const double ptk11 = PT[(fI + 2) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 1) * N + fQ + 0];
            const double ptb4 = PT[(fP + 1) * N + fQ + 1];
            const double ptb5 = PT[(fP + 1) * N + fQ + 2];
            const double ptb6 = PT[(fP + 2) * N + fQ + 0];
            const double ptb7 = PT[(fP + 2) * N + fQ + 1];
            const double ptb8 = PT[(fP + 2) * N + fQ + 2];
            const double ptb9 = PT[(fP + 3) * N + fQ + 0];
            const double ptb10 = PT[(fP + 3) * N + fQ + 1];
            const double ptb11 = PT[(fP + 3) * N + fQ + 2];
            const double ptb12 = PT[(fP + 4) * N + fQ + 0];
            const double ptb13 = PT[(fP + 4) * N + fQ + 1];
            const double ptb14 = PT[(fP + 4) * N + fQ + 2];
            const double ptb15 = PT[(fP + 5) * N + fQ + 0];
            const double ptb16 = PT[(fP + 5) * N + fQ + 1];
            const double ptb17 = PT[(fP + 5) * N + fQ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            jab0 += o0_3 * ptk3 + o0_7 * ptk7 + o0_11 * ptk11;
            jab1 += o1_3 * ptk3 + o1_7 * ptk7 + o1_11 * ptk11;
            jab2 += o2_3 * ptk3 + o2_7 * ptk7 + o2_11 * ptk11;
            jab3 += o3_3 * ptk3 + o3_7 * ptk7 + o3_11 * ptk11;
            jab4 += o4_3 * ptk3 + o4_7 * ptk7 + o4_11 * ptk11;
            jab5 += o5_3 * ptk3 + o5_7 * ptk7 + o5_11 * ptk11;
            jab6 += o6_3 * ptk3 + o6_7 * ptk7 + o6_11 * ptk11;
            jab7 += o7_3 * ptk3 + o7_7 * ptk7 + o7_11 * ptk11;
            jab8 += o8_3 * ptk3 + o8_7 * ptk7 + o8_11 * ptk11;
            jab9 += o9_3 * ptk3 + o9_7 * ptk7 + o9_11 * ptk11;
            jab10 += o10_3 * ptk3 + o10_7 * ptk7 + o10_11 * ptk11;
            jab11 += o11_3 * ptk3 + o11_7 * ptk7 + o11_11 * ptk11;
            jab12 += o12_3 * ptk3 + o12_7 * ptk7 + o12_11 * ptk11;
            jab13 += o13_3 * ptk3 + o13_7 * ptk7 + o13_11 * ptk11;
            jab14 += o14_3 * ptk3 + o14_7 * ptk7 + o14_11 * ptk11;
            jab15 += o15_3 * ptk3 + o15_7 * ptk7 + o15_11 * ptk11;
            jab16 += o16_3 * ptk3 + o16_7 * ptk7 + o16_11 * ptk11;
            jab17 += o17_3 * ptk3 + o17_7 * ptk7 + o17_11 * ptk11;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 3, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5 + o6_3 * ptb6 + o7_3 * ptb7 + o8_3 * ptb8 + o9_3 * ptb9 + o10_3 * ptb10 + o11_3 * ptb11 + o12_3 * ptb12 + o13_3 * ptb13 + o14_3 * ptb14 + o15_3 * ptb15 + o16_3 * ptb16 + o17_3 * ptb17));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 3, 2.0 * deg * (o0_7 * ptb0 + o1_7 * ptb1 + o2_7 * ptb2 + o3_7 * ptb3 + o4_7 * ptb4 + o5_7 * ptb5 + o6_7 * ptb6 + o7_7 * ptb7 + o8_7 * ptb8 + o9_7 * ptb9 + o10_7 * ptb10 + o11_7 * ptb11 + o12_7 * ptb12 + o13_7 * ptb13 + o14_7 * ptb14 + o15_7 * ptb15 + o16_7 * ptb16 + o17_7 * ptb17));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 3, 2.0 * deg * (o0_11 * ptb0 + o1_11 * ptb1 + o2_11 * ptb2 + o3_11 * ptb3 + o4_11 * ptb4 + o5_11 * ptb5 + o6_11 * ptb6 + o7_11 * ptb7 + o8_11 * ptb8 + o9_11 * ptb9 + o10_11 * ptb10 + o11_11 * ptb11 + o12_11 * ptb12 + o13_11 * ptb13 + o14_11 * ptb14 + o15_11 * ptb15 + o16_11 * ptb16 + o17_11 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_3 * Abd0_3 + o1_3 * Abd1_3 + o2_3 * Abd2_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_3 * Aad0_3 + o3_3 * Aad1_3 + o6_3 * Aad2_3 + o9_3 * Aad3_3 + o12_3 * Aad4_3 + o15_3 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_3 * Abc0_0 + o0_7 * Abc0_1 + o0_11 * Abc0_2 + o1_3 * Abc1_0 + o1_7 * Abc1_1 + o1_11 * Abc1_2 + o2_3 * Abc2_0 + o2_7 * Abc2_1 + o2_11 * Abc2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_3 * Aac0_0 + o0_7 * Aac0_1 + o0_11 * Aac0_2 + o3_3 * Aac1_0 + o3_7 * Aac1_1 + o3_11 * Aac1_2 + o6_3 * Aac2_0 + o6_7 * Aac2_1 + o6_11 * Aac2_2 + o9_3 * Aac3_0 + o9_7 * Aac3_1 + o9_11 * Aac3_2 + o12_3 * Aac4_0 + o12_7 * Aac4_1 + o12_11 * Aac4_2 + o15_3 * Aac5_0 + o15_7 * Aac5_1 + o15_11 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_7 * Abd0_3 + o1_7 * Abd1_3 + o2_7 * Abd2_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_7 * Aad0_3 + o3_7 * Aad1_3 + o6_7 * Aad2_3 + o9_7 * Aad3_3 + o12_7 * Aad4_3 + o15_7 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_11 * Abd0_3 + o1_11 * Abd1_3 + o2_11 * Abd2_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_11 * Aad0_3 + o3_11 * Aad1_3 + o6_11 * Aad2_3 + o9_11 * Aad3_3 + o12_11 * Aad4_3 + o15_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_3 * Aad0_3 + o4_3 * Aad1_3 + o7_3 * Aad2_3 + o10_3 * Aad3_3 + o13_3 * Aad4_3 + o16_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_3 * Aac0_0 + o1_7 * Aac0_1 + o1_11 * Aac0_2 + o4_3 * Aac1_0 + o4_7 * Aac1_1 + o4_11 * Aac1_2 + o7_3 * Aac2_0 + o7_7 * Aac2_1 + o7_11 * Aac2_2 + o10_3 * Aac3_0 + o10_7 * Aac3_1 + o10_11 * Aac3_2 + o13_3 * Aac4_0 + o13_7 * Aac4_1 + o13_11 * Aac4_2 + o16_3 * Aac5_0 + o16_7 * Aac5_1 + o16_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_7 * Aad0_3 + o4_7 * Aad1_3 + o7_7 * Aad2_3 + o10_7 * Aad3_3 + o13_7 * Aad4_3 + o16_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_11 * Aad0_3 + o4_11 * Aad1_3 + o7_11 * Aad2_3 + o10_11 * Aad3_3 + o13_11 * Aad4_3 + o16_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_3 * Aad0_3 + o5_3 * Aad1_3 + o8_3 * Aad2_3 + o11_3 * Aad3_3 + o14_3 * Aad4_3 + o17_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_3 * Aac0_0 + o2_7 * Aac0_1 + o2_11 * Aac0_2 + o5_3 * Aac1_0 + o5_7 * Aac1_1 + o5_11 * Aac1_2 + o8_3 * Aac2_0 + o8_7 * Aac2_1 + o8_11 * Aac2_2 + o11_3 * Aac3_0 + o11_7 * Aac3_1 + o11_11 * Aac3_2 + o14_3 * Aac4_0 + o14_7 * Aac4_1 + o14_11 * Aac4_2 + o17_3 * Aac5_0 + o17_7 * Aac5_1 + o17_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_7 * Aad0_3 + o5_7 * Aad1_3 + o8_7 * Aad2_3 + o11_7 * Aad3_3 + o14_7 * Aad4_3 + o17_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_11 * Aad0_3 + o5_11 * Aad1_3 + o8_11 * Aad2_3 + o11_11 * Aad3_3 + o14_11 * Aad4_3 + o17_11 * Aad5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o3_3 * Abd0_3 + o4_3 * Abd1_3 + o5_3 * Abd2_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o3_3 * Abc0_0 + o3_7 * Abc0_1 + o3_11 * Abc0_2 + o4_3 * Abc1_0 + o4_7 * Abc1_1 + o4_11 * Abc1_2 + o5_3 * Abc2_0 + o5_7 * Abc2_1 + o5_11 * Abc2_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o3_7 * Abd0_3 + o4_7 * Abd1_3 + o5_7 * Abd2_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o3_11 * Abd0_3 + o4_11 * Abd1_3 + o5_11 * Abd2_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o6_3 * Abd0_3 + o7_3 * Abd1_3 + o8_3 * Abd2_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o6_3 * Abc0_0 + o6_7 * Abc0_1 + o6_11 * Abc0_2 + o7_3 * Abc1_0 + o7_7 * Abc1_1 + o7_11 * Abc1_2 + o8_3 * Abc2_0 + o8_7 * Abc2_1 + o8_11 * Abc2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o6_7 * Abd0_3 + o7_7 * Abd1_3 + o8_7 * Abd2_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o6_11 * Abd0_3 + o7_11 * Abd1_3 + o8_11 * Abd2_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o9_3 * Abd0_3 + o10_3 * Abd1_3 + o11_3 * Abd2_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o9_3 * Abc0_0 + o9_7 * Abc0_1 + o9_11 * Abc0_2 + o10_3 * Abc1_0 + o10_7 * Abc1_1 + o10_11 * Abc1_2 + o11_3 * Abc2_0 + o11_7 * Abc2_1 + o11_11 * Abc2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o9_7 * Abd0_3 + o10_7 * Abd1_3 + o11_7 * Abd2_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o9_11 * Abd0_3 + o10_11 * Abd1_3 + o11_11 * Abd2_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o12_3 * Abd0_3 + o13_3 * Abd1_3 + o14_3 * Abd2_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o12_3 * Abc0_0 + o12_7 * Abc0_1 + o12_11 * Abc0_2 + o13_3 * Abc1_0 + o13_7 * Abc1_1 + o13_11 * Abc1_2 + o14_3 * Abc2_0 + o14_7 * Abc2_1 + o14_11 * Abc2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o12_7 * Abd0_3 + o13_7 * Abd1_3 + o14_7 * Abd2_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o12_11 * Abd0_3 + o13_11 * Abd1_3 + o14_11 * Abd2_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o15_3 * Abd0_3 + o16_3 * Abd1_3 + o17_3 * Abd2_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o15_3 * Abc0_0 + o15_7 * Abc0_1 + o15_11 * Abc0_2 + o16_3 * Abc1_0 + o16_7 * Abc1_1 + o16_11 * Abc1_2 + o17_3 * Abc2_0 + o17_7 * Abc2_1 + o17_11 * Abc2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o15_7 * Abd0_3 + o16_7 * Abd1_3 + o17_7 * Abd2_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o15_11 * Abd0_3 + o16_11 * Abd1_3 + o17_11 * Abd2_3));
          }
        } break;
        }
      }
      {
        const double s2 = 2.0 * deg;
        double v[32] = {s2 * jab0, s2 * jab1, s2 * jab2, s2 * jab3, s2 * jab4, s2 * jab5, s2 * jab6, s2 * jab7, s2 * jab8, s2 * jab9, s2 * jab10, s2 * jab11, s2 * jab12, s2 * jab13, s2 * jab14, s2 * jab15, s2 * jab16, s2 * jab17, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const double s = sqb::warp_sum_scatter<32>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 18 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 3) * N + bp.fQ + ab % 3, s);
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
