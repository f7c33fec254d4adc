// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DL_DL_R_w(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 134; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];
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
      double jab18 = 0.0;
      double jab19 = 0.0;
      double jab20 = 0.0;
      double jab21 = 0.0;
      double jab22 = 0.0;
      double jab23 = 0.0;
      unsigned long long nprimq = 0, nflush = 0;
      if (ok) {
        const double* __restrict__ kprim = a.ket_prims + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // ket functions [0, 1]
          double o0_0 = 0;
          double o0_1 = 0;
          double o1_0 = 0;
          double o1_1 = 0;
          double o2_0 = 0;
          double o2_1 = 0;
          double o3_0 = 0;
          double o3_1 = 0;
          double o4_0 = 0;
          double o4_1 = 0;
          double o5_0 = 0;
          double o5_1 = 0;
          double o6_0 = 0;
          double o6_1 = 0;
          double o7_0 = 0;
          double o7_1 = 0;
          double o8_0 = 0;
          double o8_1 = 0;
          double o9_0 = 0;
          double o9_1 = 0;
          double o10_0 = 0;
          double o10_1 = 0;
          double o11_0 = 0;
          double o11_1 = 0;
          double o12_0 = 0;
          double o12_1 = 0;
          double o13_0 = 0;
          double o13_1 = 0;
          double o14_0 = 0;
          double o14_1 = 0;
          double o15_0 = 0;
          double o15_1 = 0;
          double o16_0 = 0;
          double o16_1 = 0;
          double o17_0 = 0;
          double o17_1 = 0;
          double o18_0 = 0;
          double o18_1 = 0;
          double o19_0 = 0;
          double o19_1 = 0;
          double o20_0 = 0;
          double o20_1 = 0;
          double o21_0 = 0;
          double o21_1 = 0;
          double o22_0 = 0;
          double o22_1 = 0;
          double o23_0 = 0;
          double o23_1 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              ++nprimq;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek0_0 = kj[5 * kS];
              const double ek0_1 = -kj[6 * kS];
              const double ek0_2 = kj[7 * kS];
              const double ek1_0 = kj[8 * kS];
              const double ek1_1 = -kj[9 * kS];
              const double ek1_2 = kj[10 * kS];
              const double ek1_3 = -kj[11 * kS];
              g0_0 = fma(ek0_0, b0, g0_0);
              g1_0 = fma(ek1_0, b0, g1_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              g1_1 = fma(ek1_0, r0_0_0_1, g1_1);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              g1_2 = fma(ek1_0, r0_0_1_0, g1_2);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fma(ek0_1, r0_1_0_0, g0_0);
              g1_3 = fma(ek1_0, r0_1_0_0, g1_3);
              g1_0 = fma(ek1_1, r0_1_0_0, g1_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g0_4 = fma(ek0_0, r0_0_0_2, g0_4);
              g1_4 = fma(ek1_0, r0_0_0_2, g1_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fma(ek0_0, r0_0_1_1, g0_5);
              g1_5 = fma(ek1_0, r0_0_1_1, g1_5);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g0_6 = fma(ek0_0, r0_0_2_0, g0_6);
              g1_6 = fma(ek1_0, r0_0_2_0, g1_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fma(ek0_0, r0_1_0_1, g0_7);
              g0_1 = fma(ek0_1, r0_1_0_1, g0_1);
              g1_7 = fma(ek1_0, r0_1_0_1, g1_7);
              g1_1 = fma(ek1_1, r0_1_0_1, g1_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fma(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fma(ek0_1, r0_1_1_0, g0_2);
              g1_8 = fma(ek1_0, r0_1_1_0, g1_8);
              g1_2 = fma(ek1_1, r0_1_1_0, g1_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g0_9 = fma(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fma(ek0_1, r0_2_0_0, g0_3);
              g0_0 = fma(ek0_2, r0_2_0_0, g0_0);
              g1_9 = fma(ek1_0, r0_2_0_0, g1_9);
              g1_3 = fma(ek1_1, r0_2_0_0, g1_3);
              g1_0 = fma(ek1_2, r0_2_0_0, g1_0);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g0_10 = fma(ek0_0, r0_0_0_3, g0_10);
              g1_10 = fma(ek1_0, r0_0_0_3, g1_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g0_11 = fma(ek0_0, r0_0_1_2, g0_11);
              g1_11 = fma(ek1_0, r0_0_1_2, g1_11);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g0_12 = fma(ek0_0, r0_0_2_1, g0_12);
              g1_12 = fma(ek1_0, r0_0_2_1, g1_12);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g0_13 = fma(ek0_0, r0_0_3_0, g0_13);
              g1_13 = fma(ek1_0, r0_0_3_0, g1_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g0_14 = fma(ek0_0, r0_1_0_2, g0_14);
              g0_4 = fma(ek0_1, r0_1_0_2, g0_4);
              g1_14 = fma(ek1_0, r0_1_0_2, g1_14);
              g1_4 = fma(ek1_1, r0_1_0_2, g1_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g0_15 = fma(ek0_0, r0_1_1_1, g0_15);
              g0_5 = fma(ek0_1, r0_1_1_1, g0_5);
              g1_15 = fma(ek1_0, r0_1_1_1, g1_15);
              g1_5 = fma(ek1_1, r0_1_1_1, g1_5);
              const double r0_1_2_0 = X * r1_0_2_0;
              g0_16 = fma(ek0_0, r0_1_2_0, g0_16);
              g0_6 = fma(ek0_1, r0_1_2_0, g0_6);
              g1_16 = fma(ek1_0, r0_1_2_0, g1_16);
              g1_6 = fma(ek1_1, r0_1_2_0, g1_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g0_17 = fma(ek0_0, r0_2_0_1, g0_17);
              g0_7 = fma(ek0_1, r0_2_0_1, g0_7);
              g0_1 = fma(ek0_2, r0_2_0_1, g0_1);
              g1_17 = fma(ek1_0, r0_2_0_1, g1_17);
              g1_7 = fma(ek1_1, r0_2_0_1, g1_7);
              g1_1 = fma(ek1_2, r0_2_0_1, g1_1);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fma(ek0_0, r0_2_1_0, g0_18);
              g0_8 = fma(ek0_1, r0_2_1_0, g0_8);
              g0_2 = fma(ek0_2, r0_2_1_0, g0_2);
              g1_18 = fma(ek1_0, r0_2_1_0, g1_18);
              g1_8 = fma(ek1_1, r0_2_1_0, g1_8);
              g1_2 = fma(ek1_2, r0_2_1_0, g1_2);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_19 = fma(ek0_0, r0_3_0_0, g0_19);
              g0_9 = fma(ek0_1, r0_3_0_0, g0_9);
              g0_3 = fma(ek0_2, r0_3_0_0, g0_3);
              g1_19 = fma(ek1_0, r0_3_0_0, g1_19);
              g1_9 = fma(ek1_1, r0_3_0_0, g1_9);
              g1_3 = fma(ek1_2, r0_3_0_0, g1_3);
              g1_0 = fma(ek1_3, r0_3_0_0, g1_0);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_1_0_3 = X * r1_0_0_3;
              g0_10 = fma(ek0_1, r0_1_0_3, g0_10);
              g1_10 = fma(ek1_1, r0_1_0_3, g1_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_1_1_2 = X * r1_0_1_2;
              g0_11 = fma(ek0_1, r0_1_1_2, g0_11);
              g1_11 = fma(ek1_1, r0_1_1_2, g1_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g0_12 = fma(ek0_1, r0_1_2_1, g0_12);
              g1_12 = fma(ek1_1, r0_1_2_1, g1_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g0_13 = fma(ek0_1, r0_1_3_0, g0_13);
              g1_13 = fma(ek1_1, r0_1_3_0, g1_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g0_14 = fma(ek0_1, r0_2_0_2, g0_14);
              g0_4 = fma(ek0_2, r0_2_0_2, g0_4);
              g1_14 = fma(ek1_1, r0_2_0_2, g1_14);
              g1_4 = fma(ek1_2, r0_2_0_2, g1_4);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g0_15 = fma(ek0_1, r0_2_1_1, g0_15);
              g0_5 = fma(ek0_2, r0_2_1_1, g0_5);
              g1_15 = fma(ek1_1, r0_2_1_1, g1_15);
              g1_5 = fma(ek1_2, r0_2_1_1, g1_5);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g0_16 = fma(ek0_1, r0_2_2_0, g0_16);
              g0_6 = fma(ek0_2, r0_2_2_0, g0_6);
              g1_16 = fma(ek1_1, r0_2_2_0, g1_16);
              g1_6 = fma(ek1_2, r0_2_2_0, g1_6);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g0_17 = fma(ek0_1, r0_3_0_1, g0_17);
              g0_7 = fma(ek0_2, r0_3_0_1, g0_7);
              g1_17 = fma(ek1_1, r0_3_0_1, g1_17);
              g1_7 = fma(ek1_2, r0_3_0_1, g1_7);
              g1_1 = fma(ek1_3, r0_3_0_1, g1_1);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g0_18 = fma(ek0_1, r0_3_1_0, g0_18);
              g0_8 = fma(ek0_2, r0_3_1_0, g0_8);
              g1_18 = fma(ek1_1, r0_3_1_0, g1_18);
              g1_8 = fma(ek1_2, r0_3_1_0, g1_8);
              g1_2 = fma(ek1_3, r0_3_1_0, g1_2);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g0_19 = fma(ek0_1, r0_4_0_0, g0_19);
              g0_9 = fma(ek0_2, r0_4_0_0, g0_9);
              g1_19 = fma(ek1_1, r0_4_0_0, g1_19);
              g1_9 = fma(ek1_2, r0_4_0_0, g1_9);
              g1_3 = fma(ek1_3, r0_4_0_0, g1_3);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g0_10 = fma(ek0_2, r0_2_0_3, g0_10);
              g1_10 = fma(ek1_2, r0_2_0_3, g1_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g0_11 = fma(ek0_2, r0_2_1_2, g0_11);
              g1_11 = fma(ek1_2, r0_2_1_2, g1_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g0_12 = fma(ek0_2, r0_2_2_1, g0_12);
              g1_12 = fma(ek1_2, r0_2_2_1, g1_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g0_13 = fma(ek0_2, r0_2_3_0, g0_13);
              g1_13 = fma(ek1_2, r0_2_3_0, g1_13);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g0_14 = fma(ek0_2, r0_3_0_2, g0_14);
              g1_14 = fma(ek1_2, r0_3_0_2, g1_14);
              g1_4 = fma(ek1_3, r0_3_0_2, g1_4);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g0_15 = fma(ek0_2, r0_3_1_1, g0_15);
              g1_15 = fma(ek1_2, r0_3_1_1, g1_15);
              g1_5 = fma(ek1_3, r0_3_1_1, g1_5);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g0_16 = fma(ek0_2, r0_3_2_0, g0_16);
              g1_16 = fma(ek1_2, r0_3_2_0, g1_16);
              g1_6 = fma(ek1_3, r0_3_2_0, g1_6);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g0_17 = fma(ek0_2, r0_4_0_1, g0_17);
              g1_17 = fma(ek1_2, r0_4_0_1, g1_17);
              g1_7 = fma(ek1_3, r0_4_0_1, g1_7);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g0_18 = fma(ek0_2, r0_4_1_0, g0_18);
              g1_18 = fma(ek1_2, r0_4_1_0, g1_18);
              g1_8 = fma(ek1_3, r0_4_1_0, g1_8);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g0_19 = fma(ek0_2, r0_5_0_0, g0_19);
              g1_19 = fma(ek1_2, r0_5_0_0, g1_19);
              g1_9 = fma(ek1_3, r0_5_0_0, g1_9);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g1_10 = fma(ek1_3, r0_3_0_3, g1_10);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g1_11 = fma(ek1_3, r0_3_1_2, g1_11);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g1_12 = fma(ek1_3, r0_3_2_1, g1_12);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g1_13 = fma(ek1_3, r0_3_3_0, g1_13);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g1_14 = fma(ek1_3, r0_4_0_2, g1_14);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g1_15 = fma(ek1_3, r0_4_1_1, g1_15);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g1_16 = fma(ek1_3, r0_4_2_0, g1_16);
              const double r4_1_0_1 = X * r5_0_0_1;
              const double r3_2_0_1 = fma(X, r4_1_0_1, r4_0_0_1);
              const double r2_3_0_1 = fma(X, r3_2_0_1, 2.0 * r3_1_0_1);
              const double r1_4_0_1 = fma(X, r2_3_0_1, 3.0 * r2_2_0_1);
              const double r0_5_0_1 = fma(X, r1_4_0_1, 4.0 * r1_3_0_1);
              g1_17 = fma(ek1_3, r0_5_0_1, g1_17);
              const double r4_1_1_0 = X * r5_0_1_0;
              const double r3_2_1_0 = fma(X, r4_1_1_0, r4_0_1_0);
              const double r2_3_1_0 = fma(X, r3_2_1_0, 2.0 * r3_1_1_0);
              const double r1_4_1_0 = fma(X, r2_3_1_0, 3.0 * r2_2_1_0);
              const double r0_5_1_0 = fma(X, r1_4_1_0, 4.0 * r1_3_1_0);
              g1_18 = fma(ek1_3, r0_5_1_0, g1_18);
              const double r5_1_0_0 = X * b6;
              const double r4_2_0_0 = fma(X, r5_1_0_0, b5);
              const double r3_3_0_0 = fma(X, r4_2_0_0, 2.0 * r4_1_0_0);
              const double r2_4_0_0 = fma(X, r3_3_0_0, 3.0 * r3_2_0_0);
              const double r1_5_0_0 = fma(X, r2_4_0_0, 4.0 * r2_3_0_0);
              const double r0_6_0_0 = fma(X, r1_5_0_0, 5.0 * r1_4_0_0);
              g1_19 = fma(ek1_3, r0_6_0_0, g1_19);
            }
            { const double eb = bi[5];
              o0_0 = fma(eb, g0_0, o0_0);
              o0_1 = fma(eb, g1_0, o0_1);
            }
            { const double eb = bi[6];
              o0_0 = fma(eb, g0_3, o0_0);
              o0_1 = fma(eb, g1_3, o0_1);
            }
            { const double eb = bi[7];
              o0_0 = fma(eb, g0_9, o0_0);
              o0_1 = fma(eb, g1_9, o0_1);
            }
            { const double eb = bi[8];
              o1_0 = fma(eb, g0_0, o1_0);
              o1_1 = fma(eb, g1_0, o1_1);
            }
            { const double eb = bi[9];
              o1_0 = fma(eb, g0_3, o1_0);
              o1_1 = fma(eb, g1_3, o1_1);
            }
            { const double eb = bi[10];
              o1_0 = fma(eb, g0_9, o1_0);
              o1_1 = fma(eb, g1_9, o1_1);
            }
            { const double eb = bi[11];
              o1_0 = fma(eb, g0_19, o1_0);
              o1_1 = fma(eb, g1_19, o1_1);
            }
            { const double eb = bi[12];
              o2_0 = fma(eb, g0_0, o2_0);
              o2_1 = fma(eb, g1_0, o2_1);
            }
            { const double eb = bi[13];
              o2_0 = fma(eb, g0_2, o2_0);
              o2_1 = fma(eb, g1_2, o2_1);
            }
            { const double eb = bi[14];
              o2_0 = fma(eb, g0_3, o2_0);
              o2_1 = fma(eb, g1_3, o2_1);
            }
            { const double eb = bi[15];
              o2_0 = fma(eb, g0_8, o2_0);
              o2_1 = fma(eb, g1_8, o2_1);
            }
            { const double eb = bi[16];
              o2_0 = fma(eb, g0_9, o2_0);
              o2_1 = fma(eb, g1_9, o2_1);
            }
            { const double eb = bi[17];
              o2_0 = fma(eb, g0_18, o2_0);
              o2_1 = fma(eb, g1_18, o2_1);
            }
            { const double eb = bi[18];
              o3_0 = fma(eb, g0_0, o3_0);
              o3_1 = fma(eb, g1_0, o3_1);
            }
            { const double eb = bi[19];
              o3_0 = fma(eb, g0_1, o3_0);
              o3_1 = fma(eb, g1_1, o3_1);
            }
            { const double eb = bi[20];
              o3_0 = fma(eb, g0_3, o3_0);
              o3_1 = fma(eb, g1_3, o3_1);
            }
            { const double eb = bi[21];
              o3_0 = fma(eb, g0_7, o3_0);
              o3_1 = fma(eb, g1_7, o3_1);
            }
            { const double eb = bi[22];
              o3_0 = fma(eb, g0_9, o3_0);
              o3_1 = fma(eb, g1_9, o3_1);
            }
            { const double eb = bi[23];
              o3_0 = fma(eb, g0_17, o3_0);
              o3_1 = fma(eb, g1_17, o3_1);
            }
            { const double eb = bi[24];
              o4_0 = fma(eb, g0_0, o4_0);
              o4_1 = fma(eb, g1_0, o4_1);
            }
            { const double eb = bi[25];
              o4_0 = fma(eb, g0_2, o4_0);
              o4_1 = fma(eb, g1_2, o4_1);
            }
            { const double eb = bi[26];
              o4_0 = fma(eb, g0_6, o4_0);
              o4_1 = fma(eb, g1_6, o4_1);
            }
            { const double eb = bi[27];
              o5_0 = fma(eb, g0_0, o5_0);
              o5_1 = fma(eb, g1_0, o5_1);
            }
            { const double eb = bi[28];
              o5_0 = fma(eb, g0_2, o5_0);
              o5_1 = fma(eb, g1_2, o5_1);
            }
            { const double eb = bi[29];
              o5_0 = fma(eb, g0_6, o5_0);
              o5_1 = fma(eb, g1_6, o5_1);
            }
            { const double eb = bi[30];
              o5_0 = fma(eb, g0_3, o5_0);
              o5_1 = fma(eb, g1_3, o5_1);
            }
            { const double eb = bi[31];
              o5_0 = fma(eb, g0_8, o5_0);
              o5_1 = fma(eb, g1_8, o5_1);
            }
            { const double eb = bi[32];
              o5_0 = fma(eb, g0_16, o5_0);
              o5_1 = fma(eb, g1_16, o5_1);
            }
            { const double eb = bi[33];
              o6_0 = fma(eb, g0_0, o6_0);
              o6_1 = fma(eb, g1_0, o6_1);
            }
            { const double eb = bi[34];
              o6_0 = fma(eb, g0_2, o6_0);
              o6_1 = fma(eb, g1_2, o6_1);
            }
            { const double eb = bi[35];
              o6_0 = fma(eb, g0_6, o6_0);
              o6_1 = fma(eb, g1_6, o6_1);
            }
            { const double eb = bi[36];
              o6_0 = fma(eb, g0_13, o6_0);
              o6_1 = fma(eb, g1_13, o6_1);
            }
            { const double eb = bi[37];
              o7_0 = fma(eb, g0_0, o7_0);
              o7_1 = fma(eb, g1_0, o7_1);
            }
            { const double eb = bi[38];
              o7_0 = fma(eb, g0_1, o7_0);
              o7_1 = fma(eb, g1_1, o7_1);
            }
            { const double eb = bi[39];
              o7_0 = fma(eb, g0_2, o7_0);
              o7_1 = fma(eb, g1_2, o7_1);
            }
            { const double eb = bi[40];
              o7_0 = fma(eb, g0_5, o7_0);
              o7_1 = fma(eb, g1_5, o7_1);
            }
            { const double eb = bi[41];
              o7_0 = fma(eb, g0_6, o7_0);
              o7_1 = fma(eb, g1_6, o7_1);
            }
            { const double eb = bi[42];
              o7_0 = fma(eb, g0_12, o7_0);
              o7_1 = fma(eb, g1_12, o7_1);
            }
            { const double eb = bi[43];
              o8_0 = fma(eb, g0_0, o8_0);
              o8_1 = fma(eb, g1_0, o8_1);
            }
            { const double eb = bi[44];
              o8_0 = fma(eb, g0_1, o8_0);
              o8_1 = fma(eb, g1_1, o8_1);
            }
            { const double eb = bi[45];
              o8_0 = fma(eb, g0_4, o8_0);
              o8_1 = fma(eb, g1_4, o8_1);
            }
            { const double eb = bi[46];
              o9_0 = fma(eb, g0_0, o9_0);
              o9_1 = fma(eb, g1_0, o9_1);
            }
            { const double eb = bi[47];
              o9_0 = fma(eb, g0_1, o9_0);
              o9_1 = fma(eb, g1_1, o9_1);
            }
            { const double eb = bi[48];
              o9_0 = fma(eb, g0_4, o9_0);
              o9_1 = fma(eb, g1_4, o9_1);
            }
            { const double eb = bi[49];
              o9_0 = fma(eb, g0_3, o9_0);
              o9_1 = fma(eb, g1_3, o9_1);
            }
            { const double eb = bi[50];
              o9_0 = fma(eb, g0_7, o9_0);
              o9_1 = fma(eb, g1_7, o9_1);
            }
            { const double eb = bi[51];
              o9_0 = fma(eb, g0_14, o9_0);
              o9_1 = fma(eb, g1_14, o9_1);
            }
            { const double eb = bi[52];
              o10_0 = fma(eb, g0_0, o10_0);
              o10_1 = fma(eb, g1_0, o10_1);
            }
            { const double eb = bi[53];
              o10_0 = fma(eb, g0_1, o10_0);
              o10_1 = fma(eb, g1_1, o10_1);
            }
            { const double eb = bi[54];
              o10_0 = fma(eb, g0_4, o10_0);
              o10_1 = fma(eb, g1_4, o10_1);
            }
            { const double eb = bi[55];
              o10_0 = fma(eb, g0_2, o10_0);
              o10_1 = fma(eb, g1_2, o10_1);
            }
            { const double eb = bi[56];
              o10_0 = fma(eb, g0_5, o10_0);
              o10_1 = fma(eb, g1_5, o10_1);
            }
            { const double eb = bi[57];
              o10_0 = fma(eb, g0_11, o10_0);
              o10_1 = fma(eb, g1_11, o10_1);
            }
            { const double eb = bi[58];
              o11_0 = fma(eb, g0_0, o11_0);
              o11_1 = fma(eb, g1_0, o11_1);
            }
            { const double eb = bi[59];
              o11_0 = fma(eb, g0_1, o11_0);
              o11_1 = fma(eb, g1_1, o11_1);
            }
            { const double eb = bi[60];
              o11_0 = fma(eb, g0_4, o11_0);
              o11_1 = fma(eb, g1_4, o11_1);
            }
            { const double eb = bi[61];
              o11_0 = fma(eb, g0_10, o11_0);
              o11_1 = fma(eb, g1_10, o11_1);
            }
            { const double eb = bi[62];
              o12_0 = fma(eb, g0_0, o12_0);
              o12_1 = fma(eb, g1_0, o12_1);
            }
            { const double eb = bi[63];
              o12_0 = fma(eb, g0_2, o12_0);
              o12_1 = fma(eb, g1_2, o12_1);
            }
            { const double eb = bi[64];
              o12_0 = fma(eb, g0_3, o12_0);
              o12_1 = fma(eb, g1_3, o12_1);
            }
            { const double eb = bi[65];
              o12_0 = fma(eb, g0_8, o12_0);
              o12_1 = fma(eb, g1_8, o12_1);
            }
            { const double eb = bi[66];
              o13_0 = fma(eb, g0_0, o13_0);
              o13_1 = fma(eb, g1_0, o13_1);
            }
            { const double eb = bi[67];
              o13_0 = fma(eb, g0_2, o13_0);
              o13_1 = fma(eb, g1_2, o13_1);
            }
            { const double eb = bi[68];
              o13_0 = fma(eb, g0_3, o13_0);
              o13_1 = fma(eb, g1_3, o13_1);
            }
            { const double eb = bi[69];
              o13_0 = fma(eb, g0_8, o13_0);
              o13_1 = fma(eb, g1_8, o13_1);
            }
            { const double eb = bi[70];
              o13_0 = fma(eb, g0_9, o13_0);
              o13_1 = fma(eb, g1_9, o13_1);
            }
            { const double eb = bi[71];
              o13_0 = fma(eb, g0_18, o13_0);
              o13_1 = fma(eb, g1_18, o13_1);
            }
            { const double eb = bi[72];
              o14_0 = fma(eb, g0_0, o14_0);
              o14_1 = fma(eb, g1_0, o14_1);
            }
            { const double eb = bi[73];
              o14_0 = fma(eb, g0_2, o14_0);
              o14_1 = fma(eb, g1_2, o14_1);
            }
            { const double eb = bi[74];
              o14_0 = fma(eb, g0_6, o14_0);
              o14_1 = fma(eb, g1_6, o14_1);
            }
            { const double eb = bi[75];
              o14_0 = fma(eb, g0_3, o14_0);
              o14_1 = fma(eb, g1_3, o14_1);
            }
            { const double eb = bi[76];
              o14_0 = fma(eb, g0_8, o14_0);
              o14_1 = fma(eb, g1_8, o14_1);
            }
            { const double eb = bi[77];
              o14_0 = fma(eb, g0_16, o14_0);
              o14_1 = fma(eb, g1_16, o14_1);
            }
            { const double eb = bi[78];
              o15_0 = fma(eb, g0_0, o15_0);
              o15_1 = fma(eb, g1_0, o15_1);
            }
            { const double eb = bi[79];
              o15_0 = fma(eb, g0_1, o15_0);
              o15_1 = fma(eb, g1_1, o15_1);
            }
            { const double eb = bi[80];
              o15_0 = fma(eb, g0_2, o15_0);
              o15_1 = fma(eb, g1_2, o15_1);
            }
            { const double eb = bi[81];
              o15_0 = fma(eb, g0_5, o15_0);
              o15_1 = fma(eb, g1_5, o15_1);
            }
            { const double eb = bi[82];
              o15_0 = fma(eb, g0_3, o15_0);
              o15_1 = fma(eb, g1_3, o15_1);
            }
            { const double eb = bi[83];
              o15_0 = fma(eb, g0_7, o15_0);
              o15_1 = fma(eb, g1_7, o15_1);
            }
            { const double eb = bi[84];
              o15_0 = fma(eb, g0_8, o15_0);
              o15_1 = fma(eb, g1_8, o15_1);
            }
            { const double eb = bi[85];
              o15_0 = fma(eb, g0_15, o15_0);
              o15_1 = fma(eb, g1_15, o15_1);
            }
            { const double eb = bi[86];
              o16_0 = fma(eb, g0_0, o16_0);
              o16_1 = fma(eb, g1_0, o16_1);
            }
            { const double eb = bi[87];
              o16_0 = fma(eb, g0_1, o16_0);
              o16_1 = fma(eb, g1_1, o16_1);
            }
            { const double eb = bi[88];
              o16_0 = fma(eb, g0_3, o16_0);
              o16_1 = fma(eb, g1_3, o16_1);
            }
            { const double eb = bi[89];
              o16_0 = fma(eb, g0_7, o16_0);
              o16_1 = fma(eb, g1_7, o16_1);
            }
            { const double eb = bi[90];
              o17_0 = fma(eb, g0_0, o17_0);
              o17_1 = fma(eb, g1_0, o17_1);
            }
            { const double eb = bi[91];
              o17_0 = fma(eb, g0_1, o17_0);
              o17_1 = fma(eb, g1_1, o17_1);
            }
            { const double eb = bi[92];
              o17_0 = fma(eb, g0_3, o17_0);
              o17_1 = fma(eb, g1_3, o17_1);
            }
            { const double eb = bi[93];
              o17_0 = fma(eb, g0_7, o17_0);
              o17_1 = fma(eb, g1_7, o17_1);
            }
            { const double eb = bi[94];
              o17_0 = fma(eb, g0_9, o17_0);
              o17_1 = fma(eb, g1_9, o17_1);
            }
            { const double eb = bi[95];
              o17_0 = fma(eb, g0_17, o17_0);
              o17_1 = fma(eb, g1_17, o17_1);
            }
            { const double eb = bi[96];
              o18_0 = fma(eb, g0_0, o18_0);
              o18_1 = fma(eb, g1_0, o18_1);
            }
            { const double eb = bi[97];
              o18_0 = fma(eb, g0_1, o18_0);
              o18_1 = fma(eb, g1_1, o18_1);
            }
            { const double eb = bi[98];
              o18_0 = fma(eb, g0_2, o18_0);
              o18_1 = fma(eb, g1_2, o18_1);
            }
            { const double eb = bi[99];
              o18_0 = fma(eb, g0_5, o18_0);
              o18_1 = fma(eb, g1_5, o18_1);
            }
            { const double eb = bi[100];
              o18_0 = fma(eb, g0_3, o18_0);
              o18_1 = fma(eb, g1_3, o18_1);
            }
            { const double eb = bi[101];
              o18_0 = fma(eb, g0_7, o18_0);
              o18_1 = fma(eb, g1_7, o18_1);
            }
            { const double eb = bi[102];
              o18_0 = fma(eb, g0_8, o18_0);
              o18_1 = fma(eb, g1_8, o18_1);
            }
            { const double eb = bi[103];
              o18_0 = fma(eb, g0_15, o18_0);
              o18_1 = fma(eb, g1_15, o18_1);
            }
            { const double eb = bi[104];
              o19_0 = fma(eb, g0_0, o19_0);
              o19_1 = fma(eb, g1_0, o19_1);
            }
            { const double eb = bi[105];
              o19_0 = fma(eb, g0_1, o19_0);
              o19_1 = fma(eb, g1_1, o19_1);
            }
            { const double eb = bi[106];
              o19_0 = fma(eb, g0_4, o19_0);
              o19_1 = fma(eb, g1_4, o19_1);
            }
            { const double eb = bi[107];
              o19_0 = fma(eb, g0_3, o19_0);
              o19_1 = fma(eb, g1_3, o19_1);
            }
            { const double eb = bi[108];
              o19_0 = fma(eb, g0_7, o19_0);
              o19_1 = fma(eb, g1_7, o19_1);
            }
            { const double eb = bi[109];
              o19_0 = fma(eb, g0_14, o19_0);
              o19_1 = fma(eb, g1_14, o19_1);
            }
            { const double eb = bi[110];
              o20_0 = fma(eb, g0_0, o20_0);
              o20_1 = fma(eb, g1_0, o20_1);
            }
            { const double eb = bi[111];
              o20_0 = fma(eb, g0_1, o20_0);
              o20_1 = fma(eb, g1_1, o20_1);
            }
            { const double eb = bi[112];
              o20_0 = fma(eb, g0_2, o20_0);
              o20_1 = fma(eb, g1_2, o20_1);
            }
            { const double eb = bi[113];
              o20_0 = fma(eb, g0_5, o20_0);
              o20_1 = fma(eb, g1_5, o20_1);
            }
            { const double eb = bi[114];
              o21_0 = fma(eb, g0_0, o21_0);
              o21_1 = fma(eb, g1_0, o21_1);
            }
            { const double eb = bi[115];
              o21_0 = fma(eb, g0_1, o21_0);
              o21_1 = fma(eb, g1_1, o21_1);
            }
            { const double eb = bi[116];
              o21_0 = fma(eb, g0_2, o21_0);
              o21_1 = fma(eb, g1_2, o21_1);
            }
            { const double eb = bi[117];
              o21_0 = fma(eb, g0_5, o21_0);
              o21_1 = fma(eb, g1_5, o21_1);
            }
            { const double eb = bi[118];
              o21_0 = fma(eb, g0_3, o21_0);
              o21_1 = fma(eb, g1_3, o21_1);
            }
            { const double eb = bi[119];
              o21_0 = fma(eb, g0_7, o21_0);
              o21_1 = fma(eb, g1_7, o21_1);
            }
            { const double eb = bi[120];
              o21_0 = fma(eb, g0_8, o21_0);
              o21_1 = fma(eb, g1_8, o21_1);
            }
            { const double eb = bi[121];
              o21_0 = fma(eb, g0_15, o21_0);
              o21_1 = fma(eb, g1_15, o21_1);
            }
            { const double eb = bi[122];
              o22_0 = fma(eb, g0_0, o22_0);
              o22_1 = fma(eb, g1_0, o22_1);
            }
            { const double eb = bi[123];
              o22_0 = fma(eb, g0_1, o22_0);
              o22_1 = fma(eb, g1_1, o22_1);
            }
            { const double eb = bi[124];
              o22_0 = fma(eb, g0_2, o22_0);
              o22_1 = fma(eb, g1_2, o22_1);
            }
            { const double eb = bi[125];
              o22_0 = fma(eb, g0_5, o22_0);
              o22_1 = fma(eb, g1_5, o22_1);
            }
            { const double eb = bi[126];
              o22_0 = fma(eb, g0_6, o22_0);
              o22_1 = fma(eb, g1_6, o22_1);
            }
            { const double eb = bi[127];
              o22_0 = fma(eb, g0_12, o22_0);
              o22_1 = fma(eb, g1_12, o22_1);
            }
            { const double eb = bi[128];
              o23_0 = fma(eb, g0_0, o23_0);
              o23_1 = fma(eb, g1_0, o23_1);
            }
            { const double eb = bi[129];
              o23_0 = fma(eb, g0_1, o23_0);
              o23_1 = fma(eb, g1_1, o23_1);
            }
            { const double eb = bi[130];
              o23_0 = fma(eb, g0_4, o23_0);
              o23_1 = fma(eb, g1_4, o23_1);
            }
            { const double eb = bi[131];
              o23_0 = fma(eb, g0_2, o23_0);
              o23_1 = fma(eb, g1_2, o23_1);
            }
            { const double eb = bi[132];
              o23_0 = fma(eb, g0_5, o23_0);
              o23_1 = fma(eb, g1_5, o23_1);
            }
            { const double eb = bi[133];
              o23_0 = fma(eb, g0_11, o23_0);
              o23_1 = fma(eb, g1_11, o23_1);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptk1 = PT[(fI + 0) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            jab0 += o0_0 * ptk0 + o0_1 * ptk1;
            jab1 += o1_0 * ptk0 + o1_1 * ptk1;
            jab2 += o2_0 * ptk0 + o2_1 * ptk1;
            jab3 += o3_0 * ptk0 + o3_1 * ptk1;
            jab4 += o4_0 * ptk0 + o4_1 * ptk1;
            jab5 += o5_0 * ptk0 + o5_1 * ptk1;
            jab6 += o6_0 * ptk0 + o6_1 * ptk1;
            jab7 += o7_0 * ptk0 + o7_1 * ptk1;
            jab8 += o8_0 * ptk0 + o8_1 * ptk1;
            jab9 += o9_0 * ptk0 + o9_1 * ptk1;
            jab10 += o10_0 * ptk0 + o10_1 * ptk1;
            jab11 += o11_0 * ptk0 + o11_1 * ptk1;
            jab12 += o12_0 * ptk0 + o12_1 * ptk1;
            jab13 += o13_0 * ptk0 + o13_1 * ptk1;
            jab14 += o14_0 * ptk0 + o14_1 * ptk1;
            jab15 += o15_0 * ptk0 + o15_1 * ptk1;
            jab16 += o16_0 * ptk0 + o16_1 * ptk1;
            jab17 += o17_0 * ptk0 + o17_1 * ptk1;
            jab18 += o18_0 * ptk0 + o18_1 * ptk1;
            jab19 += o19_0 * ptk0 + o19_1 * ptk1;
            jab20 += o20_0 * ptk0 + o20_1 * ptk1;
            jab21 += o21_0 * ptk0 + o21_1 * ptk1;
            jab22 += o22_0 * ptk0 + o22_1 * ptk1;
            jab23 += o23_0 * ptk0 + o23_1 * ptk1;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15 + o16_0 * ptb16 + o17_0 * ptb17 + o18_0 * ptb18 + o19_0 * ptb19 + o20_0 * ptb20 + o21_0 * ptb21 + o22_0 * ptb22 + o23_0 * ptb23));
            atomicAdd(Jacc + (fI + 0) * N + fJ + 1, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17 + o18_1 * ptb18 + o19_1 * ptb19 + o20_1 * ptb20 + o21_1 * ptb21 + o22_1 * ptb22 + o23_1 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o0_1 * Abd0_1 + o1_0 * Abd1_0 + o1_1 * Abd1_1 + o2_0 * Abd2_0 + o2_1 * Abd2_1 + o3_0 * Abd3_0 + o3_1 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o0_1 * Aad0_1 + o4_0 * Aad1_0 + o4_1 * Aad1_1 + o8_0 * Aad2_0 + o8_1 * Aad2_1 + o12_0 * Aad3_0 + o12_1 * Aad3_1 + o16_0 * Aad4_0 + o16_1 * Aad4_1 + o20_0 * Aad5_0 + o20_1 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o1_0 * Abc1_0 + o2_0 * Abc2_0 + o3_0 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o4_0 * Aac1_0 + o8_0 * Aac2_0 + o12_0 * Aac3_0 + o16_0 * Aac4_0 + o20_0 * Aac5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_1 * Abc0_0 + o1_1 * Abc1_0 + o2_1 * Abc2_0 + o3_1 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_1 * Aac0_0 + o4_1 * Aac1_0 + o8_1 * Aac2_0 + o12_1 * Aac3_0 + o16_1 * Aac4_0 + o20_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o1_1 * Aad0_1 + o5_0 * Aad1_0 + o5_1 * Aad1_1 + o9_0 * Aad2_0 + o9_1 * Aad2_1 + o13_0 * Aad3_0 + o13_1 * Aad3_1 + o17_0 * Aad4_0 + o17_1 * Aad4_1 + o21_0 * Aad5_0 + o21_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o5_0 * Aac1_0 + o9_0 * Aac2_0 + o13_0 * Aac3_0 + o17_0 * Aac4_0 + o21_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_1 * Aac0_0 + o5_1 * Aac1_0 + o9_1 * Aac2_0 + o13_1 * Aac3_0 + o17_1 * Aac4_0 + o21_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o2_1 * Aad0_1 + o6_0 * Aad1_0 + o6_1 * Aad1_1 + o10_0 * Aad2_0 + o10_1 * Aad2_1 + o14_0 * Aad3_0 + o14_1 * Aad3_1 + o18_0 * Aad4_0 + o18_1 * Aad4_1 + o22_0 * Aad5_0 + o22_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o6_0 * Aac1_0 + o10_0 * Aac2_0 + o14_0 * Aac3_0 + o18_0 * Aac4_0 + o22_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_1 * Aac0_0 + o6_1 * Aac1_0 + o10_1 * Aac2_0 + o14_1 * Aac3_0 + o18_1 * Aac4_0 + o22_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Aad0_0 + o3_1 * Aad0_1 + o7_0 * Aad1_0 + o7_1 * Aad1_1 + o11_0 * Aad2_0 + o11_1 * Aad2_1 + o15_0 * Aad3_0 + o15_1 * Aad3_1 + o19_0 * Aad4_0 + o19_1 * Aad4_1 + o23_0 * Aad5_0 + o23_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Aac0_0 + o7_0 * Aac1_0 + o11_0 * Aac2_0 + o15_0 * Aac3_0 + o19_0 * Aac4_0 + o23_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_1 * Aac0_0 + o7_1 * Aac1_0 + o11_1 * Aac2_0 + o15_1 * Aac3_0 + o19_1 * Aac4_0 + o23_1 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Abd0_0 + o4_1 * Abd0_1 + o5_0 * Abd1_0 + o5_1 * Abd1_1 + o6_0 * Abd2_0 + o6_1 * Abd2_1 + o7_0 * Abd3_0 + o7_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o5_0 * Abc1_0 + o6_0 * Abc2_0 + o7_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_1 * Abc0_0 + o5_1 * Abc1_0 + o6_1 * Abc2_0 + o7_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Abd0_0 + o8_1 * Abd0_1 + o9_0 * Abd1_0 + o9_1 * Abd1_1 + o10_0 * Abd2_0 + o10_1 * Abd2_1 + o11_0 * Abd3_0 + o11_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Abc0_0 + o9_0 * Abc1_0 + o10_0 * Abc2_0 + o11_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_1 * Abc0_0 + o9_1 * Abc1_0 + o10_1 * Abc2_0 + o11_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Abd0_0 + o12_1 * Abd0_1 + o13_0 * Abd1_0 + o13_1 * Abd1_1 + o14_0 * Abd2_0 + o14_1 * Abd2_1 + o15_0 * Abd3_0 + o15_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o13_0 * Abc1_0 + o14_0 * Abc2_0 + o15_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_1 * Abc0_0 + o13_1 * Abc1_0 + o14_1 * Abc2_0 + o15_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_0 * Abd0_0 + o16_1 * Abd0_1 + o17_0 * Abd1_0 + o17_1 * Abd1_1 + o18_0 * Abd2_0 + o18_1 * Abd2_1 + o19_0 * Abd3_0 + o19_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_0 * Abc0_0 + o17_0 * Abc1_0 + o18_0 * Abc2_0 + o19_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_1 * Abc0_0 + o17_1 * Abc1_0 + o18_1 * Abc2_0 + o19_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_0 * Abd0_0 + o20_1 * Abd0_1 + o21_0 * Abd1_0 + o21_1 * Abd1_1 + o22_0 * Abd2_0 + o22_1 * Abd2_1 + o23_0 * Abd3_0 + o23_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_0 * Abc0_0 + o21_0 * Abc1_0 + o22_0 * Abc2_0 + o23_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_1 * Abc0_0 + o21_1 * Abc1_0 + o22_1 * Abc2_0 + o23_1 * Abc3_0));
          }
        } break;
        case 1: {  // ket functions [2, 3]
          double o0_2 = 0;
          double o0_3 = 0;
          double o1_2 = 0;
          double o1_3 = 0;
          double o2_2 = 0;
          double o2_3 = 0;
          double o3_2 = 0;
          double o3_3 = 0;
          double o4_2 = 0;
          double o4_3 = 0;
          double o5_2 = 0;
          double o5_3 = 0;
          double o6_2 = 0;
          double o6_3 = 0;
          double o7_2 = 0;
          double o7_3 = 0;
          double o8_2 = 0;
          double o8_3 = 0;
          double o9_2 = 0;
          double o9_3 = 0;
          double o10_2 = 0;
          double o10_3 = 0;
          double o11_2 = 0;
          double o11_3 = 0;
          double o12_2 = 0;
          double o12_3 = 0;
          double o13_2 = 0;
          double o13_3 = 0;
          double o14_2 = 0;
          double o14_3 = 0;
          double o15_2 = 0;
          double o15_3 = 0;
          double o16_2 = 0;
          double o16_3 = 0;
          double o17_2 = 0;
          double o17_3 = 0;
          double o18_2 = 0;
          double o18_3 = 0;
          double o19_2 = 0;
          double o19_3 = 0;
          double o20_2 = 0;
          double o20_3 = 0;
          double o21_2 = 0;
          double o21_3 = 0;
          double o22_2 = 0;
          double o22_3 = 0;
          double o23_2 = 0;
          double o23_3 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek2_0 = kj[12 * kS];
              const double ek2_1 = -kj[13 * kS];
              const double ek2_2 = -kj[14 * kS];
              const double ek2_3 = kj[15 * kS];
              const double ek2_4 = kj[16 * kS];
              const double ek2_5 = -kj[17 * kS];
              const double ek3_0 = kj[18 * kS];
              const double ek3_1 = -kj[19 * kS];
              const double ek3_2 = -kj[20 * kS];
              const double ek3_3 = kj[21 * kS];
              const double ek3_4 = kj[22 * kS];
              const double ek3_5 = -kj[23 * kS];
              g2_0 = fma(ek2_0, b0, g2_0);
              g3_0 = fma(ek3_0, b0, g3_0);
              const double r0_0_0_1 = Z * b1;
              g2_1 = fma(ek2_0, r0_0_0_1, g2_1);
              g3_1 = fma(ek3_0, r0_0_0_1, g3_1);
              g3_0 = fma(ek3_1, r0_0_0_1, g3_0);
              const double r0_0_1_0 = Y * b1;
              g2_2 = fma(ek2_0, r0_0_1_0, g2_2);
              g2_0 = fma(ek2_1, r0_0_1_0, g2_0);
              g3_2 = fma(ek3_0, r0_0_1_0, g3_2);
              const double r0_1_0_0 = X * b1;
              g2_3 = fma(ek2_0, r0_1_0_0, g2_3);
              g2_0 = fma(ek2_2, r0_1_0_0, g2_0);
              g3_3 = fma(ek3_0, r0_1_0_0, g3_3);
              g3_0 = fma(ek3_2, r0_1_0_0, g3_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g2_4 = fma(ek2_0, r0_0_0_2, g2_4);
              g3_4 = fma(ek3_0, r0_0_0_2, g3_4);
              g3_1 = fma(ek3_1, r0_0_0_2, g3_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g2_5 = fma(ek2_0, r0_0_1_1, g2_5);
              g2_1 = fma(ek2_1, r0_0_1_1, g2_1);
              g3_5 = fma(ek3_0, r0_0_1_1, g3_5);
              g3_2 = fma(ek3_1, r0_0_1_1, g3_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g2_6 = fma(ek2_0, r0_0_2_0, g2_6);
              g2_2 = fma(ek2_1, r0_0_2_0, g2_2);
              g3_6 = fma(ek3_0, r0_0_2_0, g3_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g2_7 = fma(ek2_0, r0_1_0_1, g2_7);
              g2_1 = fma(ek2_2, r0_1_0_1, g2_1);
              g3_7 = fma(ek3_0, r0_1_0_1, g3_7);
              g3_3 = fma(ek3_1, r0_1_0_1, g3_3);
              g3_1 = fma(ek3_2, r0_1_0_1, g3_1);
              g3_0 = fma(ek3_3, r0_1_0_1, g3_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g2_8 = fma(ek2_0, r0_1_1_0, g2_8);
              g2_3 = fma(ek2_1, r0_1_1_0, g2_3);
              g2_2 = fma(ek2_2, r0_1_1_0, g2_2);
              g2_0 = fma(ek2_3, r0_1_1_0, g2_0);
              g3_8 = fma(ek3_0, r0_1_1_0, g3_8);
              g3_2 = fma(ek3_2, r0_1_1_0, g3_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g2_9 = fma(ek2_0, r0_2_0_0, g2_9);
              g2_3 = fma(ek2_2, r0_2_0_0, g2_3);
              g2_0 = fma(ek2_4, r0_2_0_0, g2_0);
              g3_9 = fma(ek3_0, r0_2_0_0, g3_9);
              g3_3 = fma(ek3_2, r0_2_0_0, g3_3);
              g3_0 = fma(ek3_4, r0_2_0_0, g3_0);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g2_10 = fma(ek2_0, r0_0_0_3, g2_10);
              g3_10 = fma(ek3_0, r0_0_0_3, g3_10);
              g3_4 = fma(ek3_1, r0_0_0_3, g3_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g2_11 = fma(ek2_0, r0_0_1_2, g2_11);
              g2_4 = fma(ek2_1, r0_0_1_2, g2_4);
              g3_11 = fma(ek3_0, r0_0_1_2, g3_11);
              g3_5 = fma(ek3_1, r0_0_1_2, g3_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g2_12 = fma(ek2_0, r0_0_2_1, g2_12);
              g2_5 = fma(ek2_1, r0_0_2_1, g2_5);
              g3_12 = fma(ek3_0, r0_0_2_1, g3_12);
              g3_6 = fma(ek3_1, r0_0_2_1, g3_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g2_13 = fma(ek2_0, r0_0_3_0, g2_13);
              g2_6 = fma(ek2_1, r0_0_3_0, g2_6);
              g3_13 = fma(ek3_0, r0_0_3_0, g3_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g2_14 = fma(ek2_0, r0_1_0_2, g2_14);
              g2_4 = fma(ek2_2, r0_1_0_2, g2_4);
              g3_14 = fma(ek3_0, r0_1_0_2, g3_14);
              g3_7 = fma(ek3_1, r0_1_0_2, g3_7);
              g3_4 = fma(ek3_2, r0_1_0_2, g3_4);
              g3_1 = fma(ek3_3, r0_1_0_2, g3_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g2_15 = fma(ek2_0, r0_1_1_1, g2_15);
              g2_7 = fma(ek2_1, r0_1_1_1, g2_7);
              g2_5 = fma(ek2_2, r0_1_1_1, g2_5);
              g2_1 = fma(ek2_3, r0_1_1_1, g2_1);
              g3_15 = fma(ek3_0, r0_1_1_1, g3_15);
              g3_8 = fma(ek3_1, r0_1_1_1, g3_8);
              g3_5 = fma(ek3_2, r0_1_1_1, g3_5);
              g3_2 = fma(ek3_3, r0_1_1_1, g3_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g2_16 = fma(ek2_0, r0_1_2_0, g2_16);
              g2_8 = fma(ek2_1, r0_1_2_0, g2_8);
              g2_6 = fma(ek2_2, r0_1_2_0, g2_6);
              g2_2 = fma(ek2_3, r0_1_2_0, g2_2);
              g3_16 = fma(ek3_0, r0_1_2_0, g3_16);
              g3_6 = fma(ek3_2, r0_1_2_0, g3_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g2_17 = fma(ek2_0, r0_2_0_1, g2_17);
              g2_7 = fma(ek2_2, r0_2_0_1, g2_7);
              g2_1 = fma(ek2_4, r0_2_0_1, g2_1);
              g3_17 = fma(ek3_0, r0_2_0_1, g3_17);
              g3_9 = fma(ek3_1, r0_2_0_1, g3_9);
              g3_7 = fma(ek3_2, r0_2_0_1, g3_7);
              g3_3 = fma(ek3_3, r0_2_0_1, g3_3);
              g3_1 = fma(ek3_4, r0_2_0_1, g3_1);
              g3_0 = fma(ek3_5, r0_2_0_1, g3_0);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g2_18 = fma(ek2_0, r0_2_1_0, g2_18);
              g2_9 = fma(ek2_1, r0_2_1_0, g2_9);
              g2_8 = fma(ek2_2, r0_2_1_0, g2_8);
              g2_3 = fma(ek2_3, r0_2_1_0, g2_3);
              g2_2 = fma(ek2_4, r0_2_1_0, g2_2);
              g2_0 = fma(ek2_5, r0_2_1_0, g2_0);
              g3_18 = fma(ek3_0, r0_2_1_0, g3_18);
              g3_8 = fma(ek3_2, r0_2_1_0, g3_8);
              g3_2 = fma(ek3_4, r0_2_1_0, g3_2);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g2_19 = fma(ek2_0, r0_3_0_0, g2_19);
              g2_9 = fma(ek2_2, r0_3_0_0, g2_9);
              g2_3 = fma(ek2_4, r0_3_0_0, g2_3);
              g3_19 = fma(ek3_0, r0_3_0_0, g3_19);
              g3_9 = fma(ek3_2, r0_3_0_0, g3_9);
              g3_3 = fma(ek3_4, r0_3_0_0, g3_3);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g3_10 = fma(ek3_1, r0_0_0_4, g3_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g2_10 = fma(ek2_1, r0_0_1_3, g2_10);
              g3_11 = fma(ek3_1, r0_0_1_3, g3_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g2_11 = fma(ek2_1, r0_0_2_2, g2_11);
              g3_12 = fma(ek3_1, r0_0_2_2, g3_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g2_12 = fma(ek2_1, r0_0_3_1, g2_12);
              g3_13 = fma(ek3_1, r0_0_3_1, g3_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g2_13 = fma(ek2_1, r0_0_4_0, g2_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g2_10 = fma(ek2_2, r0_1_0_3, g2_10);
              g3_14 = fma(ek3_1, r0_1_0_3, g3_14);
              g3_10 = fma(ek3_2, r0_1_0_3, g3_10);
              g3_4 = fma(ek3_3, r0_1_0_3, g3_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g2_14 = fma(ek2_1, r0_1_1_2, g2_14);
              g2_11 = fma(ek2_2, r0_1_1_2, g2_11);
              g2_4 = fma(ek2_3, r0_1_1_2, g2_4);
              g3_15 = fma(ek3_1, r0_1_1_2, g3_15);
              g3_11 = fma(ek3_2, r0_1_1_2, g3_11);
              g3_5 = fma(ek3_3, r0_1_1_2, g3_5);
              const double r0_1_2_1 = X * r1_0_2_1;
              g2_15 = fma(ek2_1, r0_1_2_1, g2_15);
              g2_12 = fma(ek2_2, r0_1_2_1, g2_12);
              g2_5 = fma(ek2_3, r0_1_2_1, g2_5);
              g3_16 = fma(ek3_1, r0_1_2_1, g3_16);
              g3_12 = fma(ek3_2, r0_1_2_1, g3_12);
              g3_6 = fma(ek3_3, r0_1_2_1, g3_6);
              const double r0_1_3_0 = X * r1_0_3_0;
              g2_16 = fma(ek2_1, r0_1_3_0, g2_16);
              g2_13 = fma(ek2_2, r0_1_3_0, g2_13);
              g2_6 = fma(ek2_3, r0_1_3_0, g2_6);
              g3_13 = fma(ek3_2, r0_1_3_0, g3_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g2_14 = fma(ek2_2, r0_2_0_2, g2_14);
              g2_4 = fma(ek2_4, r0_2_0_2, g2_4);
              g3_17 = fma(ek3_1, r0_2_0_2, g3_17);
              g3_14 = fma(ek3_2, r0_2_0_2, g3_14);
              g3_7 = fma(ek3_3, r0_2_0_2, g3_7);
              g3_4 = fma(ek3_4, r0_2_0_2, g3_4);
              g3_1 = fma(ek3_5, r0_2_0_2, g3_1);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g2_17 = fma(ek2_1, r0_2_1_1, g2_17);
              g2_15 = fma(ek2_2, r0_2_1_1, g2_15);
              g2_7 = fma(ek2_3, r0_2_1_1, g2_7);
              g2_5 = fma(ek2_4, r0_2_1_1, g2_5);
              g2_1 = fma(ek2_5, r0_2_1_1, g2_1);
              g3_18 = fma(ek3_1, r0_2_1_1, g3_18);
              g3_15 = fma(ek3_2, r0_2_1_1, g3_15);
              g3_8 = fma(ek3_3, r0_2_1_1, g3_8);
              g3_5 = fma(ek3_4, r0_2_1_1, g3_5);
              g3_2 = fma(ek3_5, r0_2_1_1, g3_2);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g2_18 = fma(ek2_1, r0_2_2_0, g2_18);
              g2_16 = fma(ek2_2, r0_2_2_0, g2_16);
              g2_8 = fma(ek2_3, r0_2_2_0, g2_8);
              g2_6 = fma(ek2_4, r0_2_2_0, g2_6);
              g2_2 = fma(ek2_5, r0_2_2_0, g2_2);
              g3_16 = fma(ek3_2, r0_2_2_0, g3_16);
              g3_6 = fma(ek3_4, r0_2_2_0, g3_6);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g2_17 = fma(ek2_2, r0_3_0_1, g2_17);
              g2_7 = fma(ek2_4, r0_3_0_1, g2_7);
              g3_19 = fma(ek3_1, r0_3_0_1, g3_19);
              g3_17 = fma(ek3_2, r0_3_0_1, g3_17);
              g3_9 = fma(ek3_3, r0_3_0_1, g3_9);
              g3_7 = fma(ek3_4, r0_3_0_1, g3_7);
              g3_3 = fma(ek3_5, r0_3_0_1, g3_3);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g2_19 = fma(ek2_1, r0_3_1_0, g2_19);
              g2_18 = fma(ek2_2, r0_3_1_0, g2_18);
              g2_9 = fma(ek2_3, r0_3_1_0, g2_9);
              g2_8 = fma(ek2_4, r0_3_1_0, g2_8);
              g2_3 = fma(ek2_5, r0_3_1_0, g2_3);
              g3_18 = fma(ek3_2, r0_3_1_0, g3_18);
              g3_8 = fma(ek3_4, r0_3_1_0, g3_8);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g2_19 = fma(ek2_2, r0_4_0_0, g2_19);
              g2_9 = fma(ek2_4, r0_4_0_0, g2_9);
              g3_19 = fma(ek3_2, r0_4_0_0, g3_19);
              g3_9 = fma(ek3_4, r0_4_0_0, g3_9);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_1_0_4 = X * r1_0_0_4;
              g3_10 = fma(ek3_3, r0_1_0_4, g3_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g2_10 = fma(ek2_3, r0_1_1_3, g2_10);
              g3_11 = fma(ek3_3, r0_1_1_3, g3_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g2_11 = fma(ek2_3, r0_1_2_2, g2_11);
              g3_12 = fma(ek3_3, r0_1_2_2, g3_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g2_12 = fma(ek2_3, r0_1_3_1, g2_12);
              g3_13 = fma(ek3_3, r0_1_3_1, g3_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g2_13 = fma(ek2_3, r0_1_4_0, g2_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g2_10 = fma(ek2_4, r0_2_0_3, g2_10);
              g3_14 = fma(ek3_3, r0_2_0_3, g3_14);
              g3_10 = fma(ek3_4, r0_2_0_3, g3_10);
              g3_4 = fma(ek3_5, r0_2_0_3, g3_4);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g2_14 = fma(ek2_3, r0_2_1_2, g2_14);
              g2_11 = fma(ek2_4, r0_2_1_2, g2_11);
              g2_4 = fma(ek2_5, r0_2_1_2, g2_4);
              g3_15 = fma(ek3_3, r0_2_1_2, g3_15);
              g3_11 = fma(ek3_4, r0_2_1_2, g3_11);
              g3_5 = fma(ek3_5, r0_2_1_2, g3_5);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g2_15 = fma(ek2_3, r0_2_2_1, g2_15);
              g2_12 = fma(ek2_4, r0_2_2_1, g2_12);
              g2_5 = fma(ek2_5, r0_2_2_1, g2_5);
              g3_16 = fma(ek3_3, r0_2_2_1, g3_16);
              g3_12 = fma(ek3_4, r0_2_2_1, g3_12);
              g3_6 = fma(ek3_5, r0_2_2_1, g3_6);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g2_16 = fma(ek2_3, r0_2_3_0, g2_16);
              g2_13 = fma(ek2_4, r0_2_3_0, g2_13);
              g2_6 = fma(ek2_5, r0_2_3_0, g2_6);
              g3_13 = fma(ek3_4, r0_2_3_0, g3_13);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g2_14 = fma(ek2_4, r0_3_0_2, g2_14);
              g3_17 = fma(ek3_3, r0_3_0_2, g3_17);
              g3_14 = fma(ek3_4, r0_3_0_2, g3_14);
              g3_7 = fma(ek3_5, r0_3_0_2, g3_7);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g2_17 = fma(ek2_3, r0_3_1_1, g2_17);
              g2_15 = fma(ek2_4, r0_3_1_1, g2_15);
              g2_7 = fma(ek2_5, r0_3_1_1, g2_7);
              g3_18 = fma(ek3_3, r0_3_1_1, g3_18);
              g3_15 = fma(ek3_4, r0_3_1_1, g3_15);
              g3_8 = fma(ek3_5, r0_3_1_1, g3_8);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g2_18 = fma(ek2_3, r0_3_2_0, g2_18);
              g2_16 = fma(ek2_4, r0_3_2_0, g2_16);
              g2_8 = fma(ek2_5, r0_3_2_0, g2_8);
              g3_16 = fma(ek3_4, r0_3_2_0, g3_16);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g2_17 = fma(ek2_4, r0_4_0_1, g2_17);
              g3_19 = fma(ek3_3, r0_4_0_1, g3_19);
              g3_17 = fma(ek3_4, r0_4_0_1, g3_17);
              g3_9 = fma(ek3_5, r0_4_0_1, g3_9);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g2_19 = fma(ek2_3, r0_4_1_0, g2_19);
              g2_18 = fma(ek2_4, r0_4_1_0, g2_18);
              g2_9 = fma(ek2_5, r0_4_1_0, g2_9);
              g3_18 = fma(ek3_4, r0_4_1_0, g3_18);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g2_19 = fma(ek2_4, r0_5_0_0, g2_19);
              g3_19 = fma(ek3_4, r0_5_0_0, g3_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g3_10 = fma(ek3_5, r0_2_0_4, g3_10);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g2_10 = fma(ek2_5, r0_2_1_3, g2_10);
              g3_11 = fma(ek3_5, r0_2_1_3, g3_11);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g2_11 = fma(ek2_5, r0_2_2_2, g2_11);
              g3_12 = fma(ek3_5, r0_2_2_2, g3_12);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g2_12 = fma(ek2_5, r0_2_3_1, g2_12);
              g3_13 = fma(ek3_5, r0_2_3_1, g3_13);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g2_13 = fma(ek2_5, r0_2_4_0, g2_13);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g3_14 = fma(ek3_5, r0_3_0_3, g3_14);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g2_14 = fma(ek2_5, r0_3_1_2, g2_14);
              g3_15 = fma(ek3_5, r0_3_1_2, g3_15);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g2_15 = fma(ek2_5, r0_3_2_1, g2_15);
              g3_16 = fma(ek3_5, r0_3_2_1, g3_16);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g2_16 = fma(ek2_5, r0_3_3_0, g2_16);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g3_17 = fma(ek3_5, r0_4_0_2, g3_17);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g2_17 = fma(ek2_5, r0_4_1_1, g2_17);
              g3_18 = fma(ek3_5, r0_4_1_1, g3_18);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g2_18 = fma(ek2_5, r0_4_2_0, g2_18);
              const double r4_1_0_1 = X * r5_0_0_1;
              const double r3_2_0_1 = fma(X, r4_1_0_1, r4_0_0_1);
              const double r2_3_0_1 = fma(X, r3_2_0_1, 2.0 * r3_1_0_1);
              const double r1_4_0_1 = fma(X, r2_3_0_1, 3.0 * r2_2_0_1);
              const double r0_5_0_1 = fma(X, r1_4_0_1, 4.0 * r1_3_0_1);
              g3_19 = fma(ek3_5, r0_5_0_1, g3_19);
              const double r4_1_1_0 = X * r5_0_1_0;
              const double r3_2_1_0 = fma(X, r4_1_1_0, r4_0_1_0);
              const double r2_3_1_0 = fma(X, r3_2_1_0, 2.0 * r3_1_1_0);
              const double r1_4_1_0 = fma(X, r2_3_1_0, 3.0 * r2_2_1_0);
              const double r0_5_1_0 = fma(X, r1_4_1_0, 4.0 * r1_3_1_0);
              g2_19 = fma(ek2_5, r0_5_1_0, g2_19);
            }
            { const double eb = bi[5];
              o0_2 = fma(eb, g2_0, o0_2);
              o0_3 = fma(eb, g3_0, o0_3);
            }
            { const double eb = bi[6];
              o0_2 = fma(eb, g2_3, o0_2);
              o0_3 = fma(eb, g3_3, o0_3);
            }
            { const double eb = bi[7];
              o0_2 = fma(eb, g2_9, o0_2);
              o0_3 = fma(eb, g3_9, o0_3);
            }
            { const double eb = bi[8];
              o1_2 = fma(eb, g2_0, o1_2);
              o1_3 = fma(eb, g3_0, o1_3);
            }
            { const double eb = bi[9];
              o1_2 = fma(eb, g2_3, o1_2);
              o1_3 = fma(eb, g3_3, o1_3);
            }
            { const double eb = bi[10];
              o1_2 = fma(eb, g2_9, o1_2);
              o1_3 = fma(eb, g3_9, o1_3);
            }
            { const double eb = bi[11];
              o1_2 = fma(eb, g2_19, o1_2);
              o1_3 = fma(eb, g3_19, o1_3);
            }
            { const double eb = bi[12];
              o2_2 = fma(eb, g2_0, o2_2);
              o2_3 = fma(eb, g3_0, o2_3);
            }
            { const double eb = bi[13];
              o2_2 = fma(eb, g2_2, o2_2);
              o2_3 = fma(eb, g3_2, o2_3);
            }
            { const double eb = bi[14];
              o2_2 = fma(eb, g2_3, o2_2);
              o2_3 = fma(eb, g3_3, o2_3);
            }
            { const double eb = bi[15];
              o2_2 = fma(eb, g2_8, o2_2);
              o2_3 = fma(eb, g3_8, o2_3);
            }
            { const double eb = bi[16];
              o2_2 = fma(eb, g2_9, o2_2);
              o2_3 = fma(eb, g3_9, o2_3);
            }
            { const double eb = bi[17];
              o2_2 = fma(eb, g2_18, o2_2);
              o2_3 = fma(eb, g3_18, o2_3);
            }
            { const double eb = bi[18];
              o3_2 = fma(eb, g2_0, o3_2);
              o3_3 = fma(eb, g3_0, o3_3);
            }
            { const double eb = bi[19];
              o3_2 = fma(eb, g2_1, o3_2);
              o3_3 = fma(eb, g3_1, o3_3);
            }
            { const double eb = bi[20];
              o3_2 = fma(eb, g2_3, o3_2);
              o3_3 = fma(eb, g3_3, o3_3);
            }
            { const double eb = bi[21];
              o3_2 = fma(eb, g2_7, o3_2);
              o3_3 = fma(eb, g3_7, o3_3);
            }
            { const double eb = bi[22];
              o3_2 = fma(eb, g2_9, o3_2);
              o3_3 = fma(eb, g3_9, o3_3);
            }
            { const double eb = bi[23];
              o3_2 = fma(eb, g2_17, o3_2);
              o3_3 = fma(eb, g3_17, o3_3);
            }
            { const double eb = bi[24];
              o4_2 = fma(eb, g2_0, o4_2);
              o4_3 = fma(eb, g3_0, o4_3);
            }
            { const double eb = bi[25];
              o4_2 = fma(eb, g2_2, o4_2);
              o4_3 = fma(eb, g3_2, o4_3);
            }
            { const double eb = bi[26];
              o4_2 = fma(eb, g2_6, o4_2);
              o4_3 = fma(eb, g3_6, o4_3);
            }
            { const double eb = bi[27];
              o5_2 = fma(eb, g2_0, o5_2);
              o5_3 = fma(eb, g3_0, o5_3);
            }
            { const double eb = bi[28];
              o5_2 = fma(eb, g2_2, o5_2);
              o5_3 = fma(eb, g3_2, o5_3);
            }
            { const double eb = bi[29];
              o5_2 = fma(eb, g2_6, o5_2);
              o5_3 = fma(eb, g3_6, o5_3);
            }
            { const double eb = bi[30];
              o5_2 = fma(eb, g2_3, o5_2);
              o5_3 = fma(eb, g3_3, o5_3);
            }
            { const double eb = bi[31];
              o5_2 = fma(eb, g2_8, o5_2);
              o5_3 = fma(eb, g3_8, o5_3);
            }
            { const double eb = bi[32];
              o5_2 = fma(eb, g2_16, o5_2);
              o5_3 = fma(eb, g3_16, o5_3);
            }
            { const double eb = bi[33];
              o6_2 = fma(eb, g2_0, o6_2);
              o6_3 = fma(eb, g3_0, o6_3);
            }
            { const double eb = bi[34];
              o6_2 = fma(eb, g2_2, o6_2);
              o6_3 = fma(eb, g3_2, o6_3);
            }
            { const double eb = bi[35];
              o6_2 = fma(eb, g2_6, o6_2);
              o6_3 = fma(eb, g3_6, o6_3);
            }
            { const double eb = bi[36];
              o6_2 = fma(eb, g2_13, o6_2);
              o6_3 = fma(eb, g3_13, o6_3);
            }
            { const double eb = bi[37];
              o7_2 = fma(eb, g2_0, o7_2);
              o7_3 = fma(eb, g3_0, o7_3);
            }
            { const double eb = bi[38];
              o7_2 = fma(eb, g2_1, o7_2);
              o7_3 = fma(eb, g3_1, o7_3);
            }
            { const double eb = bi[39];
              o7_2 = fma(eb, g2_2, o7_2);
              o7_3 = fma(eb, g3_2, o7_3);
            }
            { const double eb = bi[40];
              o7_2 = fma(eb, g2_5, o7_2);
              o7_3 = fma(eb, g3_5, o7_3);
            }
            { const double eb = bi[41];
              o7_2 = fma(eb, g2_6, o7_2);
              o7_3 = fma(eb, g3_6, o7_3);
            }
            { const double eb = bi[42];
              o7_2 = fma(eb, g2_12, o7_2);
              o7_3 = fma(eb, g3_12, o7_3);
            }
            { const double eb = bi[43];
              o8_2 = fma(eb, g2_0, o8_2);
              o8_3 = fma(eb, g3_0, o8_3);
            }
            { const double eb = bi[44];
              o8_2 = fma(eb, g2_1, o8_2);
              o8_3 = fma(eb, g3_1, o8_3);
            }
            { const double eb = bi[45];
              o8_2 = fma(eb, g2_4, o8_2);
              o8_3 = fma(eb, g3_4, o8_3);
            }
            { const double eb = bi[46];
              o9_2 = fma(eb, g2_0, o9_2);
              o9_3 = fma(eb, g3_0, o9_3);
            }
            { const double eb = bi[47];
              o9_2 = fma(eb, g2_1, o9_2);
              o9_3 = fma(eb, g3_1, o9_3);
            }
            { const double eb = bi[48];
              o9_2 = fma(eb, g2_4, o9_2);
              o9_3 = fma(eb, g3_4, o9_3);
            }
            { const double eb = bi[49];
              o9_2 = fma(eb, g2_3, o9_2);
              o9_3 = fma(eb, g3_3, o9_3);
            }
            { const double eb = bi[50];
              o9_2 = fma(eb, g2_7, o9_2);
              o9_3 = fma(eb, g3_7, o9_3);
            }
            { const double eb = bi[51];
              o9_2 = fma(eb, g2_14, o9_2);
              o9_3 = fma(eb, g3_14, o9_3);
            }
            { const double eb = bi[52];
              o10_2 = fma(eb, g2_0, o10_2);
              o10_3 = fma(eb, g3_0, o10_3);
            }
            { const double eb = bi[53];
              o10_2 = fma(eb, g2_1, o10_2);
              o10_3 = fma(eb, g3_1, o10_3);
            }
            { const double eb = bi[54];
              o10_2 = fma(eb, g2_4, o10_2);
              o10_3 = fma(eb, g3_4, o10_3);
            }
            { const double eb = bi[55];
              o10_2 = fma(eb, g2_2, o10_2);
              o10_3 = fma(eb, g3_2, o10_3);
            }
            { const double eb = bi[56];
              o10_2 = fma(eb, g2_5, o10_2);
              o10_3 = fma(eb, g3_5, o10_3);
            }
            { const double eb = bi[57];
              o10_2 = fma(eb, g2_11, o10_2);
              o10_3 = fma(eb, g3_11, o10_3);
            }
            { const double eb = bi[58];
              o11_2 = fma(eb, g2_0, o11_2);
              o11_3 = fma(eb, g3_0, o11_3);
            }
            { const double eb = bi[59];
              o11_2 = fma(eb, g2_1, o11_2);
              o11_3 = fma(eb, g3_1, o11_3);
            }
            { const double eb = bi[60];
              o11_2 = fma(eb, g2_4, o11_2);
              o11_3 = fma(eb, g3_4, o11_3);
            }
            { const double eb = bi[61];
              o11_2 = fma(eb, g2_10, o11_2);
              o11_3 = fma(eb, g3_10, o11_3);
            }
            { const double eb = bi[62];
              o12_2 = fma(eb, g2_0, o12_2);
              o12_3 = fma(eb, g3_0, o12_3);
            }
            { const double eb = bi[63];
              o12_2 = fma(eb, g2_2, o12_2);
              o12_3 = fma(eb, g3_2, o12_3);
            }
            { const double eb = bi[64];
              o12_2 = fma(eb, g2_3, o12_2);
              o12_3 = fma(eb, g3_3, o12_3);
            }
            { const double eb = bi[65];
              o12_2 = fma(eb, g2_8, o12_2);
              o12_3 = fma(eb, g3_8, o12_3);
            }
            { const double eb = bi[66];
              o13_2 = fma(eb, g2_0, o13_2);
              o13_3 = fma(eb, g3_0, o13_3);
            }
            { const double eb = bi[67];
              o13_2 = fma(eb, g2_2, o13_2);
              o13_3 = fma(eb, g3_2, o13_3);
            }
            { const double eb = bi[68];
              o13_2 = fma(eb, g2_3, o13_2);
              o13_3 = fma(eb, g3_3, o13_3);
            }
            { const double eb = bi[69];
              o13_2 = fma(eb, g2_8, o13_2);
              o13_3 = fma(eb, g3_8, o13_3);
            }
            { const double eb = bi[70];
              o13_2 = fma(eb, g2_9, o13_2);
              o13_3 = fma(eb, g3_9, o13_3);
            }
            { const double eb = bi[71];
              o13_2 = fma(eb, g2_18, o13_2);
              o13_3 = fma(eb, g3_18, o13_3);
            }
            { const double eb = bi[72];
              o14_2 = fma(eb, g2_0, o14_2);
              o14_3 = fma(eb, g3_0, o14_3);
            }
            { const double eb = bi[73];
              o14_2 = fma(eb, g2_2, o14_2);
              o14_3 = fma(eb, g3_2, o14_3);
            }
            { const double eb = bi[74];
              o14_2 = fma(eb, g2_6, o14_2);
              o14_3 = fma(eb, g3_6, o14_3);
            }
            { const double eb = bi[75];
              o14_2 = fma(eb, g2_3, o14_2);
              o14_3 = fma(eb, g3_3, o14_3);
            }
            { const double eb = bi[76];
              o14_2 = fma(eb, g2_8, o14_2);
              o14_3 = fma(eb, g3_8, o14_3);
            }
            { const double eb = bi[77];
              o14_2 = fma(eb, g2_16, o14_2);
              o14_3 = fma(eb, g3_16, o14_3);
            }
            { const double eb = bi[78];
              o15_2 = fma(eb, g2_0, o15_2);
              o15_3 = fma(eb, g3_0, o15_3);
            }
            { const double eb = bi[79];
              o15_2 = fma(eb, g2_1, o15_2);
              o15_3 = fma(eb, g3_1, o15_3);
            }
            { const double eb = bi[80];
              o15_2 = fma(eb, g2_2, o15_2);
              o15_3 = fma(eb, g3_2, o15_3);
            }
            { const double eb = bi[81];
              o15_2 = fma(eb, g2_5, o15_2);
              o15_3 = fma(eb, g3_5, o15_3);
            }
            { const double eb = bi[82];
              o15_2 = fma(eb, g2_3, o15_2);
              o15_3 = fma(eb, g3_3, o15_3);
            }
            { const double eb = bi[83];
              o15_2 = fma(eb, g2_7, o15_2);
              o15_3 = fma(eb, g3_7, o15_3);
            }
            { const double eb = bi[84];
              o15_2 = fma(eb, g2_8, o15_2);
              o15_3 = fma(eb, g3_8, o15_3);
            }
            { const double eb = bi[85];
              o15_2 = fma(eb, g2_15, o15_2);
              o15_3 = fma(eb, g3_15, o15_3);
            }
            { const double eb = bi[86];
              o16_2 = fma(eb, g2_0, o16_2);
              o16_3 = fma(eb, g3_0, o16_3);
            }
            { const double eb = bi[87];
              o16_2 = fma(eb, g2_1, o16_2);
              o16_3 = fma(eb, g3_1, o16_3);
            }
            { const double eb = bi[88];
              o16_2 = fma(eb, g2_3, o16_2);
              o16_3 = fma(eb, g3_3, o16_3);
            }
            { const double eb = bi[89];
              o16_2 = fma(eb, g2_7, o16_2);
              o16_3 = fma(eb, g3_7, o16_3);
            }
            { const double eb = bi[90];
              o17_2 = fma(eb, g2_0, o17_2);
              o17_3 = fma(eb, g3_0, o17_3);
            }
            { const double eb = bi[91];
              o17_2 = fma(eb, g2_1, o17_2);
              o17_3 = fma(eb, g3_1, o17_3);
            }
            { const double eb = bi[92];
              o17_2 = fma(eb, g2_3, o17_2);
              o17_3 = fma(eb, g3_3, o17_3);
            }
            { const double eb = bi[93];
              o17_2 = fma(eb, g2_7, o17_2);
              o17_3 = fma(eb, g3_7, o17_3);
            }
            { const double eb = bi[94];
              o17_2 = fma(eb, g2_9, o17_2);
              o17_3 = fma(eb, g3_9, o17_3);
            }
            { const double eb = bi[95];
              o17_2 = fma(eb, g2_17, o17_2);
              o17_3 = fma(eb, g3_17, o17_3);
            }
            { const double eb = bi[96];
              o18_2 = fma(eb, g2_0, o18_2);
              o18_3 = fma(eb, g3_0, o18_3);
            }
            { const double eb = bi[97];
              o18_2 = fma(eb, g2_1, o18_2);
              o18_3 = fma(eb, g3_1, o18_3);
            }
            { const double eb = bi[98];
              o18_2 = fma(eb, g2_2, o18_2);
              o18_3 = fma(eb, g3_2, o18_3);
            }
            { const double eb = bi[99];
              o18_2 = fma(eb, g2_5, o18_2);
              o18_3 = fma(eb, g3_5, o18_3);
            }
            { const double eb = bi[100];
              o18_2 = fma(eb, g2_3, o18_2);
              o18_3 = fma(eb, g3_3, o18_3);
            }
            { const double eb = bi[101];
              o18_2 = fma(eb, g2_7, o18_2);
              o18_3 = fma(eb, g3_7, o18_3);
            }
            { const double eb = bi[102];
              o18_2 = fma(eb, g2_8, o18_2);
              o18_3 = fma(eb, g3_8, o18_3);
            }
            { const double eb = bi[103];
              o18_2 = fma(eb, g2_15, o18_2);
              o18_3 = fma(eb, g3_15, o18_3);
            }
            { const double eb = bi[104];
              o19_2 = fma(eb, g2_0, o19_2);
              o19_3 = fma(eb, g3_0, o19_3);
            }
            { const double eb = bi[105];
              o19_2 = fma(eb, g2_1, o19_2);
              o19_3 = fma(eb, g3_1, o19_3);
            }
            { const double eb = bi[106];
              o19_2 = fma(eb, g2_4, o19_2);
              o19_3 = fma(eb, g3_4, o19_3);
            }
            { const double eb = bi[107];
              o19_2 = fma(eb, g2_3, o19_2);
              o19_3 = fma(eb, g3_3, o19_3);
            }
            { const double eb = bi[108];
              o19_2 = fma(eb, g2_7, o19_2);
              o19_3 = fma(eb, g3_7, o19_3);
            }
            { const double eb = bi[109];
              o19_2 = fma(eb, g2_14, o19_2);
              o19_3 = fma(eb, g3_14, o19_3);
            }
            { const double eb = bi[110];
              o20_2 = fma(eb, g2_0, o20_2);
              o20_3 = fma(eb, g3_0, o20_3);
            }
            { const double eb = bi[111];
              o20_2 = fma(eb, g2_1, o20_2);
              o20_3 = fma(eb, g3_1, o20_3);
            }
            { const double eb = bi[112];
              o20_2 = fma(eb, g2_2, o20_2);
              o20_3 = fma(eb, g3_2, o20_3);
            }
            { const double eb = bi[113];
              o20_2 = fma(eb, g2_5, o20_2);
              o20_3 = fma(eb, g3_5, o20_3);
            }
            { const double eb = bi[114];
              o21_2 = fma(eb, g2_0, o21_2);
              o21_3 = fma(eb, g3_0, o21_3);
            }
            { const double eb = bi[115];
              o21_2 = fma(eb, g2_1, o21_2);
              o21_3 = fma(eb, g3_1, o21_3);
            }
            { const double eb = bi[116];
              o21_2 = fma(eb, g2_2, o21_2);
              o21_3 = fma(eb, g3_2, o21_3);
            }
            { const double eb = bi[117];
              o21_2 = fma(eb, g2_5, o21_2);
              o21_3 = fma(eb, g3_5, o21_3);
            }
            { const double eb = bi[118];
              o21_2 = fma(eb, g2_3, o21_2);
              o21_3 = fma(eb, g3_3, o21_3);
            }
            { const double eb = bi[119];
              o21_2 = fma(eb, g2_7, o21_2);
              o21_3 = fma(eb, g3_7, o21_3);
            }
            { const double eb = bi[120];
              o21_2 = fma(eb, g2_8, o21_2);
              o21_3 = fma(eb, g3_8, o21_3);
            }
            { const double eb = bi[121];
              o21_2 = fma(eb, g2_15, o21_2);
              o21_3 = fma(eb, g3_15, o21_3);
            }
            { const double eb = bi[122];
              o22_2 = fma(eb, g2_0, o22_2);
              o22_3 = fma(eb, g3_0, o22_3);
            }
            { const double eb = bi[123];
              o22_2 = fma(eb, g2_1, o22_2);
              o22_3 = fma(eb, g3_1, o22_3);
            }
            { const double eb = bi[124];
              o22_2 = fma(eb, g2_2, o22_2);
              o22_3 = fma(eb, g3_2, o22_3);
            }
            { const double eb = bi[125];
              o22_2 = fma(eb, g2_5, o22_2);
              o22_3 = fma(eb, g3_5, o22_3);
            }
            { const double eb = bi[126];
              o22_2 = fma(eb, g2_6, o22_2);
              o22_3 = fma(eb, g3_6, o22_3);
            }
            { const double eb = bi[127];
              o22_2 = fma(eb, g2_12, o22_2);
              o22_3 = fma(eb, g3_12, o22_3);
            }
            { const double eb = bi[128];
              o23_2 = fma(eb, g2_0, o23_2);
              o23_3 = fma(eb, g3_0, o23_3);
            }
            { const double eb = bi[129];
              o23_2 = fma(eb, g2_1, o23_2);
              o23_3 = fma(eb, g3_1, o23_3);
            }
            { const double eb = bi[130];
              o23_2 = fma(eb, g2_4, o23_2);
              o23_3 = fma(eb, g3_4, o23_3);
            }
            { const double eb = bi[131];
              o23_2 = fma(eb, g2_2, o23_2);
              o23_3 = fma(eb, g3_2, o23_3);
            }
            { const double eb = bi[132];
              o23_2 = fma(eb, g2_5, o23_2);
              o23_3 = fma(eb, g3_5, o23_3);
            }
            { const double eb = bi[133];
              o23_2 = fma(eb, g2_11, o23_2);
              o23_3 = fma(eb, g3_11, o23_3);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 0) * N + fJ + 2];
            const double ptk3 = PT[(fI + 0) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            jab0 += o0_2 * ptk2 + o0_3 * ptk3;
            jab1 += o1_2 * ptk2 + o1_3 * ptk3;
            jab2 += o2_2 * ptk2 + o2_3 * ptk3;
            jab3 += o3_2 * ptk2 + o3_3 * ptk3;
            jab4 += o4_2 * ptk2 + o4_3 * ptk3;
            jab5 += o5_2 * ptk2 + o5_3 * ptk3;
            jab6 += o6_2 * ptk2 + o6_3 * ptk3;
            jab7 += o7_2 * ptk2 + o7_3 * ptk3;
            jab8 += o8_2 * ptk2 + o8_3 * ptk3;
            jab9 += o9_2 * ptk2 + o9_3 * ptk3;
            jab10 += o10_2 * ptk2 + o10_3 * ptk3;
            jab11 += o11_2 * ptk2 + o11_3 * ptk3;
            jab12 += o12_2 * ptk2 + o12_3 * ptk3;
            jab13 += o13_2 * ptk2 + o13_3 * ptk3;
            jab14 += o14_2 * ptk2 + o14_3 * ptk3;
            jab15 += o15_2 * ptk2 + o15_3 * ptk3;
            jab16 += o16_2 * ptk2 + o16_3 * ptk3;
            jab17 += o17_2 * ptk2 + o17_3 * ptk3;
            jab18 += o18_2 * ptk2 + o18_3 * ptk3;
            jab19 += o19_2 * ptk2 + o19_3 * ptk3;
            jab20 += o20_2 * ptk2 + o20_3 * ptk3;
            jab21 += o21_2 * ptk2 + o21_3 * ptk3;
            jab22 += o22_2 * ptk2 + o22_3 * ptk3;
            jab23 += o23_2 * ptk2 + o23_3 * ptk3;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 2, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17 + o18_2 * ptb18 + o19_2 * ptb19 + o20_2 * ptb20 + o21_2 * ptb21 + o22_2 * ptb22 + o23_2 * ptb23));
            atomicAdd(Jacc + (fI + 0) * N + fJ + 3, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5 + o6_3 * ptb6 + o7_3 * ptb7 + o8_3 * ptb8 + o9_3 * ptb9 + o10_3 * ptb10 + o11_3 * ptb11 + o12_3 * ptb12 + o13_3 * ptb13 + o14_3 * ptb14 + o15_3 * ptb15 + o16_3 * ptb16 + o17_3 * ptb17 + o18_3 * ptb18 + o19_3 * ptb19 + o20_3 * ptb20 + o21_3 * ptb21 + o22_3 * ptb22 + o23_3 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_2 * Abd0_2 + o0_3 * Abd0_3 + o1_2 * Abd1_2 + o1_3 * Abd1_3 + o2_2 * Abd2_2 + o2_3 * Abd2_3 + o3_2 * Abd3_2 + o3_3 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_2 * Aad0_2 + o0_3 * Aad0_3 + o4_2 * Aad1_2 + o4_3 * Aad1_3 + o8_2 * Aad2_2 + o8_3 * Aad2_3 + o12_2 * Aad3_2 + o12_3 * Aad3_3 + o16_2 * Aad4_2 + o16_3 * Aad4_3 + o20_2 * Aad5_2 + o20_3 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_2 * Abc0_0 + o1_2 * Abc1_0 + o2_2 * Abc2_0 + o3_2 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_2 * Aac0_0 + o4_2 * Aac1_0 + o8_2 * Aac2_0 + o12_2 * Aac3_0 + o16_2 * Aac4_0 + o20_2 * Aac5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_3 * Abc0_0 + o1_3 * Abc1_0 + o2_3 * Abc2_0 + o3_3 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_3 * Aac0_0 + o4_3 * Aac1_0 + o8_3 * Aac2_0 + o12_3 * Aac3_0 + o16_3 * Aac4_0 + o20_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_2 * Aad0_2 + o1_3 * Aad0_3 + o5_2 * Aad1_2 + o5_3 * Aad1_3 + o9_2 * Aad2_2 + o9_3 * Aad2_3 + o13_2 * Aad3_2 + o13_3 * Aad3_3 + o17_2 * Aad4_2 + o17_3 * Aad4_3 + o21_2 * Aad5_2 + o21_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_2 * Aac0_0 + o5_2 * Aac1_0 + o9_2 * Aac2_0 + o13_2 * Aac3_0 + o17_2 * Aac4_0 + o21_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_3 * Aac0_0 + o5_3 * Aac1_0 + o9_3 * Aac2_0 + o13_3 * Aac3_0 + o17_3 * Aac4_0 + o21_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_2 * Aad0_2 + o2_3 * Aad0_3 + o6_2 * Aad1_2 + o6_3 * Aad1_3 + o10_2 * Aad2_2 + o10_3 * Aad2_3 + o14_2 * Aad3_2 + o14_3 * Aad3_3 + o18_2 * Aad4_2 + o18_3 * Aad4_3 + o22_2 * Aad5_2 + o22_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_2 * Aac0_0 + o6_2 * Aac1_0 + o10_2 * Aac2_0 + o14_2 * Aac3_0 + o18_2 * Aac4_0 + o22_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_3 * Aac0_0 + o6_3 * Aac1_0 + o10_3 * Aac2_0 + o14_3 * Aac3_0 + o18_3 * Aac4_0 + o22_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_2 * Aad0_2 + o3_3 * Aad0_3 + o7_2 * Aad1_2 + o7_3 * Aad1_3 + o11_2 * Aad2_2 + o11_3 * Aad2_3 + o15_2 * Aad3_2 + o15_3 * Aad3_3 + o19_2 * Aad4_2 + o19_3 * Aad4_3 + o23_2 * Aad5_2 + o23_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_2 * Aac0_0 + o7_2 * Aac1_0 + o11_2 * Aac2_0 + o15_2 * Aac3_0 + o19_2 * Aac4_0 + o23_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_3 * Aac0_0 + o7_3 * Aac1_0 + o11_3 * Aac2_0 + o15_3 * Aac3_0 + o19_3 * Aac4_0 + o23_3 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_2 * Abd0_2 + o4_3 * Abd0_3 + o5_2 * Abd1_2 + o5_3 * Abd1_3 + o6_2 * Abd2_2 + o6_3 * Abd2_3 + o7_2 * Abd3_2 + o7_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_2 * Abc0_0 + o5_2 * Abc1_0 + o6_2 * Abc2_0 + o7_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_3 * Abc0_0 + o5_3 * Abc1_0 + o6_3 * Abc2_0 + o7_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_2 * Abd0_2 + o8_3 * Abd0_3 + o9_2 * Abd1_2 + o9_3 * Abd1_3 + o10_2 * Abd2_2 + o10_3 * Abd2_3 + o11_2 * Abd3_2 + o11_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_2 * Abc0_0 + o9_2 * Abc1_0 + o10_2 * Abc2_0 + o11_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_3 * Abc0_0 + o9_3 * Abc1_0 + o10_3 * Abc2_0 + o11_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_2 * Abd0_2 + o12_3 * Abd0_3 + o13_2 * Abd1_2 + o13_3 * Abd1_3 + o14_2 * Abd2_2 + o14_3 * Abd2_3 + o15_2 * Abd3_2 + o15_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_2 * Abc0_0 + o13_2 * Abc1_0 + o14_2 * Abc2_0 + o15_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_3 * Abc0_0 + o13_3 * Abc1_0 + o14_3 * Abc2_0 + o15_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_2 * Abd0_2 + o16_3 * Abd0_3 + o17_2 * Abd1_2 + o17_3 * Abd1_3 + o18_2 * Abd2_2 + o18_3 * Abd2_3 + o19_2 * Abd3_2 + o19_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_2 * Abc0_0 + o17_2 * Abc1_0 + o18_2 * Abc2_0 + o19_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_3 * Abc0_0 + o17_3 * Abc1_0 + o18_3 * Abc2_0 + o19_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_2 * Abd0_2 + o20_3 * Abd0_3 + o21_2 * Abd1_2 + o21_3 * Abd1_3 + o22_2 * Abd2_2 + o22_3 * Abd2_3 + o23_2 * Abd3_2 + o23_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_2 * Abc0_0 + o21_2 * Abc1_0 + o22_2 * Abc2_0 + o23_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_3 * Abc0_0 + o21_3 * Abc1_0 + o22_3 * Abc2_0 + o23_3 * Abc3_0));
          }
        } break;
        case 2: {  // ket functions [4, 5]
          double o0_4 = 0;
          double o0_5 = 0;
          double o1_4 = 0;
          double o1_5 = 0;
          double o2_4 = 0;
          double o2_5 = 0;
          double o3_4 = 0;
          double o3_5 = 0;
          double o4_4 = 0;
          double o4_5 = 0;
          double o5_4 = 0;
          double o5_5 = 0;
          double o6_4 = 0;
          double o6_5 = 0;
          double o7_4 = 0;
          double o7_5 = 0;
          double o8_4 = 0;
          double o8_5 = 0;
          double o9_4 = 0;
          double o9_5 = 0;
          double o10_4 = 0;
          double o10_5 = 0;
          double o11_4 = 0;
          double o11_5 = 0;
          double o12_4 = 0;
          double o12_5 = 0;
          double o13_4 = 0;
          double o13_5 = 0;
          double o14_4 = 0;
          double o14_5 = 0;
          double o15_4 = 0;
          double o15_5 = 0;
          double o16_4 = 0;
          double o16_5 = 0;
          double o17_4 = 0;
          double o17_5 = 0;
          double o18_4 = 0;
          double o18_5 = 0;
          double o19_4 = 0;
          double o19_5 = 0;
          double o20_4 = 0;
          double o20_5 = 0;
          double o21_4 = 0;
          double o21_5 = 0;
          double o22_4 = 0;
          double o22_5 = 0;
          double o23_4 = 0;
          double o23_5 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek4_0 = kj[24 * kS];
              const double ek4_1 = -kj[25 * kS];
              const double ek4_2 = kj[26 * kS];
              const double ek5_0 = kj[27 * kS];
              const double ek5_1 = -kj[28 * kS];
              const double ek5_2 = kj[29 * kS];
              const double ek5_3 = -kj[30 * kS];
              const double ek5_4 = kj[31 * kS];
              const double ek5_5 = -kj[32 * kS];
              g4_0 = fma(ek4_0, b0, g4_0);
              g5_0 = fma(ek5_0, b0, g5_0);
              const double r0_0_0_1 = Z * b1;
              g4_1 = fma(ek4_0, r0_0_0_1, g4_1);
              g5_1 = fma(ek5_0, r0_0_0_1, g5_1);
              const double r0_0_1_0 = Y * b1;
              g4_2 = fma(ek4_0, r0_0_1_0, g4_2);
              g4_0 = fma(ek4_1, r0_0_1_0, g4_0);
              g5_2 = fma(ek5_0, r0_0_1_0, g5_2);
              g5_0 = fma(ek5_1, r0_0_1_0, g5_0);
              const double r0_1_0_0 = X * b1;
              g4_3 = fma(ek4_0, r0_1_0_0, g4_3);
              g5_3 = fma(ek5_0, r0_1_0_0, g5_3);
              g5_0 = fma(ek5_3, r0_1_0_0, g5_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g4_4 = fma(ek4_0, r0_0_0_2, g4_4);
              g5_4 = fma(ek5_0, r0_0_0_2, g5_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g4_5 = fma(ek4_0, r0_0_1_1, g4_5);
              g4_1 = fma(ek4_1, r0_0_1_1, g4_1);
              g5_5 = fma(ek5_0, r0_0_1_1, g5_5);
              g5_1 = fma(ek5_1, r0_0_1_1, g5_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g4_6 = fma(ek4_0, r0_0_2_0, g4_6);
              g4_2 = fma(ek4_1, r0_0_2_0, g4_2);
              g4_0 = fma(ek4_2, r0_0_2_0, g4_0);
              g5_6 = fma(ek5_0, r0_0_2_0, g5_6);
              g5_2 = fma(ek5_1, r0_0_2_0, g5_2);
              g5_0 = fma(ek5_2, r0_0_2_0, g5_0);
              const double r0_1_0_1 = X * r1_0_0_1;
              g4_7 = fma(ek4_0, r0_1_0_1, g4_7);
              g5_7 = fma(ek5_0, r0_1_0_1, g5_7);
              g5_1 = fma(ek5_3, r0_1_0_1, g5_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g4_8 = fma(ek4_0, r0_1_1_0, g4_8);
              g4_3 = fma(ek4_1, r0_1_1_0, g4_3);
              g5_8 = fma(ek5_0, r0_1_1_0, g5_8);
              g5_3 = fma(ek5_1, r0_1_1_0, g5_3);
              g5_2 = fma(ek5_3, r0_1_1_0, g5_2);
              g5_0 = fma(ek5_4, r0_1_1_0, g5_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g4_9 = fma(ek4_0, r0_2_0_0, g4_9);
              g5_9 = fma(ek5_0, r0_2_0_0, g5_9);
              g5_3 = fma(ek5_3, r0_2_0_0, g5_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g4_10 = fma(ek4_0, r0_0_0_3, g4_10);
              g5_10 = fma(ek5_0, r0_0_0_3, g5_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g4_11 = fma(ek4_0, r0_0_1_2, g4_11);
              g4_4 = fma(ek4_1, r0_0_1_2, g4_4);
              g5_11 = fma(ek5_0, r0_0_1_2, g5_11);
              g5_4 = fma(ek5_1, r0_0_1_2, g5_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g4_12 = fma(ek4_0, r0_0_2_1, g4_12);
              g4_5 = fma(ek4_1, r0_0_2_1, g4_5);
              g4_1 = fma(ek4_2, r0_0_2_1, g4_1);
              g5_12 = fma(ek5_0, r0_0_2_1, g5_12);
              g5_5 = fma(ek5_1, r0_0_2_1, g5_5);
              g5_1 = fma(ek5_2, r0_0_2_1, g5_1);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g4_13 = fma(ek4_0, r0_0_3_0, g4_13);
              g4_6 = fma(ek4_1, r0_0_3_0, g4_6);
              g4_2 = fma(ek4_2, r0_0_3_0, g4_2);
              g5_13 = fma(ek5_0, r0_0_3_0, g5_13);
              g5_6 = fma(ek5_1, r0_0_3_0, g5_6);
              g5_2 = fma(ek5_2, r0_0_3_0, g5_2);
              const double r0_1_0_2 = X * r1_0_0_2;
              g4_14 = fma(ek4_0, r0_1_0_2, g4_14);
              g5_14 = fma(ek5_0, r0_1_0_2, g5_14);
              g5_4 = fma(ek5_3, r0_1_0_2, g5_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g4_15 = fma(ek4_0, r0_1_1_1, g4_15);
              g4_7 = fma(ek4_1, r0_1_1_1, g4_7);
              g5_15 = fma(ek5_0, r0_1_1_1, g5_15);
              g5_7 = fma(ek5_1, r0_1_1_1, g5_7);
              g5_5 = fma(ek5_3, r0_1_1_1, g5_5);
              g5_1 = fma(ek5_4, r0_1_1_1, g5_1);
              const double r0_1_2_0 = X * r1_0_2_0;
              g4_16 = fma(ek4_0, r0_1_2_0, g4_16);
              g4_8 = fma(ek4_1, r0_1_2_0, g4_8);
              g4_3 = fma(ek4_2, r0_1_2_0, g4_3);
              g5_16 = fma(ek5_0, r0_1_2_0, g5_16);
              g5_8 = fma(ek5_1, r0_1_2_0, g5_8);
              g5_3 = fma(ek5_2, r0_1_2_0, g5_3);
              g5_6 = fma(ek5_3, r0_1_2_0, g5_6);
              g5_2 = fma(ek5_4, r0_1_2_0, g5_2);
              g5_0 = fma(ek5_5, r0_1_2_0, g5_0);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g4_17 = fma(ek4_0, r0_2_0_1, g4_17);
              g5_17 = fma(ek5_0, r0_2_0_1, g5_17);
              g5_7 = fma(ek5_3, r0_2_0_1, g5_7);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g4_18 = fma(ek4_0, r0_2_1_0, g4_18);
              g4_9 = fma(ek4_1, r0_2_1_0, g4_9);
              g5_18 = fma(ek5_0, r0_2_1_0, g5_18);
              g5_9 = fma(ek5_1, r0_2_1_0, g5_9);
              g5_8 = fma(ek5_3, r0_2_1_0, g5_8);
              g5_3 = fma(ek5_4, r0_2_1_0, g5_3);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g4_19 = fma(ek4_0, r0_3_0_0, g4_19);
              g5_19 = fma(ek5_0, r0_3_0_0, g5_19);
              g5_9 = fma(ek5_3, r0_3_0_0, g5_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g4_10 = fma(ek4_1, r0_0_1_3, g4_10);
              g5_10 = fma(ek5_1, r0_0_1_3, g5_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g4_11 = fma(ek4_1, r0_0_2_2, g4_11);
              g4_4 = fma(ek4_2, r0_0_2_2, g4_4);
              g5_11 = fma(ek5_1, r0_0_2_2, g5_11);
              g5_4 = fma(ek5_2, r0_0_2_2, g5_4);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g4_12 = fma(ek4_1, r0_0_3_1, g4_12);
              g4_5 = fma(ek4_2, r0_0_3_1, g4_5);
              g5_12 = fma(ek5_1, r0_0_3_1, g5_12);
              g5_5 = fma(ek5_2, r0_0_3_1, g5_5);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g4_13 = fma(ek4_1, r0_0_4_0, g4_13);
              g4_6 = fma(ek4_2, r0_0_4_0, g4_6);
              g5_13 = fma(ek5_1, r0_0_4_0, g5_13);
              g5_6 = fma(ek5_2, r0_0_4_0, g5_6);
              const double r0_1_0_3 = X * r1_0_0_3;
              g5_10 = fma(ek5_3, r0_1_0_3, g5_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g4_14 = fma(ek4_1, r0_1_1_2, g4_14);
              g5_14 = fma(ek5_1, r0_1_1_2, g5_14);
              g5_11 = fma(ek5_3, r0_1_1_2, g5_11);
              g5_4 = fma(ek5_4, r0_1_1_2, g5_4);
              const double r0_1_2_1 = X * r1_0_2_1;
              g4_15 = fma(ek4_1, r0_1_2_1, g4_15);
              g4_7 = fma(ek4_2, r0_1_2_1, g4_7);
              g5_15 = fma(ek5_1, r0_1_2_1, g5_15);
              g5_7 = fma(ek5_2, r0_1_2_1, g5_7);
              g5_12 = fma(ek5_3, r0_1_2_1, g5_12);
              g5_5 = fma(ek5_4, r0_1_2_1, g5_5);
              g5_1 = fma(ek5_5, r0_1_2_1, g5_1);
              const double r0_1_3_0 = X * r1_0_3_0;
              g4_16 = fma(ek4_1, r0_1_3_0, g4_16);
              g4_8 = fma(ek4_2, r0_1_3_0, g4_8);
              g5_16 = fma(ek5_1, r0_1_3_0, g5_16);
              g5_8 = fma(ek5_2, r0_1_3_0, g5_8);
              g5_13 = fma(ek5_3, r0_1_3_0, g5_13);
              g5_6 = fma(ek5_4, r0_1_3_0, g5_6);
              g5_2 = fma(ek5_5, r0_1_3_0, g5_2);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g5_14 = fma(ek5_3, r0_2_0_2, g5_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g4_17 = fma(ek4_1, r0_2_1_1, g4_17);
              g5_17 = fma(ek5_1, r0_2_1_1, g5_17);
              g5_15 = fma(ek5_3, r0_2_1_1, g5_15);
              g5_7 = fma(ek5_4, r0_2_1_1, g5_7);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g4_18 = fma(ek4_1, r0_2_2_0, g4_18);
              g4_9 = fma(ek4_2, r0_2_2_0, g4_9);
              g5_18 = fma(ek5_1, r0_2_2_0, g5_18);
              g5_9 = fma(ek5_2, r0_2_2_0, g5_9);
              g5_16 = fma(ek5_3, r0_2_2_0, g5_16);
              g5_8 = fma(ek5_4, r0_2_2_0, g5_8);
              g5_3 = fma(ek5_5, r0_2_2_0, g5_3);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g5_17 = fma(ek5_3, r0_3_0_1, g5_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g4_19 = fma(ek4_1, r0_3_1_0, g4_19);
              g5_19 = fma(ek5_1, r0_3_1_0, g5_19);
              g5_18 = fma(ek5_3, r0_3_1_0, g5_18);
              g5_9 = fma(ek5_4, r0_3_1_0, g5_9);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g5_19 = fma(ek5_3, r0_4_0_0, g5_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g4_10 = fma(ek4_2, r0_0_2_3, g4_10);
              g5_10 = fma(ek5_2, r0_0_2_3, g5_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g4_11 = fma(ek4_2, r0_0_3_2, g4_11);
              g5_11 = fma(ek5_2, r0_0_3_2, g5_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g4_12 = fma(ek4_2, r0_0_4_1, g4_12);
              g5_12 = fma(ek5_2, r0_0_4_1, g5_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g4_13 = fma(ek4_2, r0_0_5_0, g4_13);
              g5_13 = fma(ek5_2, r0_0_5_0, g5_13);
              const double r0_1_1_3 = X * r1_0_1_3;
              g5_10 = fma(ek5_4, r0_1_1_3, g5_10);
              const double r0_1_2_2 = X * r1_0_2_2;
              g4_14 = fma(ek4_2, r0_1_2_2, g4_14);
              g5_14 = fma(ek5_2, r0_1_2_2, g5_14);
              g5_11 = fma(ek5_4, r0_1_2_2, g5_11);
              g5_4 = fma(ek5_5, r0_1_2_2, g5_4);
              const double r0_1_3_1 = X * r1_0_3_1;
              g4_15 = fma(ek4_2, r0_1_3_1, g4_15);
              g5_15 = fma(ek5_2, r0_1_3_1, g5_15);
              g5_12 = fma(ek5_4, r0_1_3_1, g5_12);
              g5_5 = fma(ek5_5, r0_1_3_1, g5_5);
              const double r0_1_4_0 = X * r1_0_4_0;
              g4_16 = fma(ek4_2, r0_1_4_0, g4_16);
              g5_16 = fma(ek5_2, r0_1_4_0, g5_16);
              g5_13 = fma(ek5_4, r0_1_4_0, g5_13);
              g5_6 = fma(ek5_5, r0_1_4_0, g5_6);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g5_14 = fma(ek5_4, r0_2_1_2, g5_14);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g4_17 = fma(ek4_2, r0_2_2_1, g4_17);
              g5_17 = fma(ek5_2, r0_2_2_1, g5_17);
              g5_15 = fma(ek5_4, r0_2_2_1, g5_15);
              g5_7 = fma(ek5_5, r0_2_2_1, g5_7);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g4_18 = fma(ek4_2, r0_2_3_0, g4_18);
              g5_18 = fma(ek5_2, r0_2_3_0, g5_18);
              g5_16 = fma(ek5_4, r0_2_3_0, g5_16);
              g5_8 = fma(ek5_5, r0_2_3_0, g5_8);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g5_17 = fma(ek5_4, r0_3_1_1, g5_17);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g4_19 = fma(ek4_2, r0_3_2_0, g4_19);
              g5_19 = fma(ek5_2, r0_3_2_0, g5_19);
              g5_18 = fma(ek5_4, r0_3_2_0, g5_18);
              g5_9 = fma(ek5_5, r0_3_2_0, g5_9);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g5_19 = fma(ek5_4, r0_4_1_0, g5_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g5_10 = fma(ek5_5, r0_1_2_3, g5_10);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g5_11 = fma(ek5_5, r0_1_3_2, g5_11);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_1_4_1 = X * r1_0_4_1;
              g5_12 = fma(ek5_5, r0_1_4_1, g5_12);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_0_5_0 = fma(Y, r2_0_4_0, 4.0 * r2_0_3_0);
              const double r0_1_5_0 = X * r1_0_5_0;
              g5_13 = fma(ek5_5, r0_1_5_0, g5_13);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g5_14 = fma(ek5_5, r0_2_2_2, g5_14);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g5_15 = fma(ek5_5, r0_2_3_1, g5_15);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g5_16 = fma(ek5_5, r0_2_4_0, g5_16);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g5_17 = fma(ek5_5, r0_3_2_1, g5_17);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g5_18 = fma(ek5_5, r0_3_3_0, g5_18);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g5_19 = fma(ek5_5, r0_4_2_0, g5_19);
            }
            { const double eb = bi[5];
              o0_4 = fma(eb, g4_0, o0_4);
              o0_5 = fma(eb, g5_0, o0_5);
            }
            { const double eb = bi[6];
              o0_4 = fma(eb, g4_3, o0_4);
              o0_5 = fma(eb, g5_3, o0_5);
            }
            { const double eb = bi[7];
              o0_4 = fma(eb, g4_9, o0_4);
              o0_5 = fma(eb, g5_9, o0_5);
            }
            { const double eb = bi[8];
              o1_4 = fma(eb, g4_0, o1_4);
              o1_5 = fma(eb, g5_0, o1_5);
            }
            { const double eb = bi[9];
              o1_4 = fma(eb, g4_3, o1_4);
              o1_5 = fma(eb, g5_3, o1_5);
            }
            { const double eb = bi[10];
              o1_4 = fma(eb, g4_9, o1_4);
              o1_5 = fma(eb, g5_9, o1_5);
            }
            { const double eb = bi[11];
              o1_4 = fma(eb, g4_19, o1_4);
              o1_5 = fma(eb, g5_19, o1_5);
            }
            { const double eb = bi[12];
              o2_4 = fma(eb, g4_0, o2_4);
              o2_5 = fma(eb, g5_0, o2_5);
            }
            { const double eb = bi[13];
              o2_4 = fma(eb, g4_2, o2_4);
              o2_5 = fma(eb, g5_2, o2_5);
            }
            { const double eb = bi[14];
              o2_4 = fma(eb, g4_3, o2_4);
              o2_5 = fma(eb, g5_3, o2_5);
            }
            { const double eb = bi[15];
              o2_4 = fma(eb, g4_8, o2_4);
              o2_5 = fma(eb, g5_8, o2_5);
            }
            { const double eb = bi[16];
              o2_4 = fma(eb, g4_9, o2_4);
              o2_5 = fma(eb, g5_9, o2_5);
            }
            { const double eb = bi[17];
              o2_4 = fma(eb, g4_18, o2_4);
              o2_5 = fma(eb, g5_18, o2_5);
            }
            { const double eb = bi[18];
              o3_4 = fma(eb, g4_0, o3_4);
              o3_5 = fma(eb, g5_0, o3_5);
            }
            { const double eb = bi[19];
              o3_4 = fma(eb, g4_1, o3_4);
              o3_5 = fma(eb, g5_1, o3_5);
            }
            { const double eb = bi[20];
              o3_4 = fma(eb, g4_3, o3_4);
              o3_5 = fma(eb, g5_3, o3_5);
            }
            { const double eb = bi[21];
              o3_4 = fma(eb, g4_7, o3_4);
              o3_5 = fma(eb, g5_7, o3_5);
            }
            { const double eb = bi[22];
              o3_4 = fma(eb, g4_9, o3_4);
              o3_5 = fma(eb, g5_9, o3_5);
            }
            { const double eb = bi[23];
              o3_4 = fma(eb, g4_17, o3_4);
              o3_5 = fma(eb, g5_17, o3_5);
            }
            { const double eb = bi[24];
              o4_4 = fma(eb, g4_0, o4_4);
              o4_5 = fma(eb, g5_0, o4_5);
            }
            { const double eb = bi[25];
              o4_4 = fma(eb, g4_2, o4_4);
              o4_5 = fma(eb, g5_2, o4_5);
            }
            { const double eb = bi[26];
              o4_4 = fma(eb, g4_6, o4_4);
              o4_5 = fma(eb, g5_6, o4_5);
            }
            { const double eb = bi[27];
              o5_4 = fma(eb, g4_0, o5_4);
              o5_5 = fma(eb, g5_0, o5_5);
            }
            { const double eb = bi[28];
              o5_4 = fma(eb, g4_2, o5_4);
              o5_5 = fma(eb, g5_2, o5_5);
            }
            { const double eb = bi[29];
              o5_4 = fma(eb, g4_6, o5_4);
              o5_5 = fma(eb, g5_6, o5_5);
            }
            { const double eb = bi[30];
              o5_4 = fma(eb, g4_3, o5_4);
              o5_5 = fma(eb, g5_3, o5_5);
            }
            { const double eb = bi[31];
              o5_4 = fma(eb, g4_8, o5_4);
              o5_5 = fma(eb, g5_8, o5_5);
            }
            { const double eb = bi[32];
              o5_4 = fma(eb, g4_16, o5_4);
              o5_5 = fma(eb, g5_16, o5_5);
            }
            { const double eb = bi[33];
              o6_4 = fma(eb, g4_0, o6_4);
              o6_5 = fma(eb, g5_0, o6_5);
            }
            { const double eb = bi[34];
              o6_4 = fma(eb, g4_2, o6_4);
              o6_5 = fma(eb, g5_2, o6_5);
            }
            { const double eb = bi[35];
              o6_4 = fma(eb, g4_6, o6_4);
              o6_5 = fma(eb, g5_6, o6_5);
            }
            { const double eb = bi[36];
              o6_4 = fma(eb, g4_13, o6_4);
              o6_5 = fma(eb, g5_13, o6_5);
            }
            { const double eb = bi[37];
              o7_4 = fma(eb, g4_0, o7_4);
              o7_5 = fma(eb, g5_0, o7_5);
            }
            { const double eb = bi[38];
              o7_4 = fma(eb, g4_1, o7_4);
              o7_5 = fma(eb, g5_1, o7_5);
            }
            { const double eb = bi[39];
              o7_4 = fma(eb, g4_2, o7_4);
              o7_5 = fma(eb, g5_2, o7_5);
            }
            { const double eb = bi[40];
              o7_4 = fma(eb, g4_5, o7_4);
              o7_5 = fma(eb, g5_5, o7_5);
            }
            { const double eb = bi[41];
              o7_4 = fma(eb, g4_6, o7_4);
              o7_5 = fma(eb, g5_6, o7_5);
            }
            { const double eb = bi[42];
              o7_4 = fma(eb, g4_12, o7_4);
              o7_5 = fma(eb, g5_12, o7_5);
            }
            { const double eb = bi[43];
              o8_4 = fma(eb, g4_0, o8_4);
              o8_5 = fma(eb, g5_0, o8_5);
            }
            { const double eb = bi[44];
              o8_4 = fma(eb, g4_1, o8_4);
              o8_5 = fma(eb, g5_1, o8_5);
            }
            { const double eb = bi[45];
              o8_4 = fma(eb, g4_4, o8_4);
              o8_5 = fma(eb, g5_4, o8_5);
            }
            { const double eb = bi[46];
              o9_4 = fma(eb, g4_0, o9_4);
              o9_5 = fma(eb, g5_0, o9_5);
            }
            { const double eb = bi[47];
              o9_4 = fma(eb, g4_1, o9_4);
              o9_5 = fma(eb, g5_1, o9_5);
            }
            { const double eb = bi[48];
              o9_4 = fma(eb, g4_4, o9_4);
              o9_5 = fma(eb, g5_4, o9_5);
            }
            { const double eb = bi[49];
              o9_4 = fma(eb, g4_3, o9_4);
              o9_5 = fma(eb, g5_3, o9_5);
            }
            { const double eb = bi[50];
              o9_4 = fma(eb, g4_7, o9_4);
              o9_5 = fma(eb, g5_7, o9_5);
            }
            { const double eb = bi[51];
              o9_4 = fma(eb, g4_14, o9_4);
              o9_5 = fma(eb, g5_14, o9_5);
            }
            { const double eb = bi[52];
              o10_4 = fma(eb, g4_0, o10_4);
              o10_5 = fma(eb, g5_0, o10_5);
            }
            { const double eb = bi[53];
              o10_4 = fma(eb, g4_1, o10_4);
              o10_5 = fma(eb, g5_1, o10_5);
            }
            { const double eb = bi[54];
              o10_4 = fma(eb, g4_4, o10_4);
              o10_5 = fma(eb, g5_4, o10_5);
            }
            { const double eb = bi[55];
              o10_4 = fma(eb, g4_2, o10_4);
              o10_5 = fma(eb, g5_2, o10_5);
            }
            { const double eb = bi[56];
              o10_4 = fma(eb, g4_5, o10_4);
              o10_5 = fma(eb, g5_5, o10_5);
            }
            { const double eb = bi[57];
              o10_4 = fma(eb, g4_11, o10_4);
              o10_5 = fma(eb, g5_11, o10_5);
            }
            { const double eb = bi[58];
              o11_4 = fma(eb, g4_0, o11_4);
              o11_5 = fma(eb, g5_0, o11_5);
            }
            { const double eb = bi[59];
              o11_4 = fma(eb, g4_1, o11_4);
              o11_5 = fma(eb, g5_1, o11_5);
            }
            { const double eb = bi[60];
              o11_4 = fma(eb, g4_4, o11_4);
              o11_5 = fma(eb, g5_4, o11_5);
            }
            { const double eb = bi[61];
              o11_4 = fma(eb, g4_10, o11_4);
              o11_5 = fma(eb, g5_10, o11_5);
            }
            { const double eb = bi[62];
              o12_4 = fma(eb, g4_0, o12_4);
              o12_5 = fma(eb, g5_0, o12_5);
            }
            { const double eb = bi[63];
              o12_4 = fma(eb, g4_2, o12_4);
              o12_5 = fma(eb, g5_2, o12_5);
            }
            { const double eb = bi[64];
              o12_4 = fma(eb, g4_3, o12_4);
              o12_5 = fma(eb, g5_3, o12_5);
            }
            { const double eb = bi[65];
              o12_4 = fma(eb, g4_8, o12_4);
              o12_5 = fma(eb, g5_8, o12_5);
            }
            { const double eb = bi[66];
              o13_4 = fma(eb, g4_0, o13_4);
              o13_5 = fma(eb, g5_0, o13_5);
            }
            { const double eb = bi[67];
              o13_4 = fma(eb, g4_2, o13_4);
              o13_5 = fma(eb, g5_2, o13_5);
            }
            { const double eb = bi[68];
              o13_4 = fma(eb, g4_3, o13_4);
              o13_5 = fma(eb, g5_3, o13_5);
            }
            { const double eb = bi[69];
              o13_4 = fma(eb, g4_8, o13_4);
              o13_5 = fma(eb, g5_8, o13_5);
            }
            { const double eb = bi[70];
              o13_4 = fma(eb, g4_9, o13_4);
              o13_5 = fma(eb, g5_9, o13_5);
            }
            { const double eb = bi[71];
              o13_4 = fma(eb, g4_18, o13_4);
              o13_5 = fma(eb, g5_18, o13_5);
            }
            { const double eb = bi[72];
              o14_4 = fma(eb, g4_0, o14_4);
              o14_5 = fma(eb, g5_0, o14_5);
            }
            { const double eb = bi[73];
              o14_4 = fma(eb, g4_2, o14_4);
              o14_5 = fma(eb, g5_2, o14_5);
            }
            { const double eb = bi[74];
              o14_4 = fma(eb, g4_6, o14_4);
              o14_5 = fma(eb, g5_6, o14_5);
            }
            { const double eb = bi[75];
              o14_4 = fma(eb, g4_3, o14_4);
              o14_5 = fma(eb, g5_3, o14_5);
            }
            { const double eb = bi[76];
              o14_4 = fma(eb, g4_8, o14_4);
              o14_5 = fma(eb, g5_8, o14_5);
            }
            { const double eb = bi[77];
              o14_4 = fma(eb, g4_16, o14_4);
              o14_5 = fma(eb, g5_16, o14_5);
            }
            { const double eb = bi[78];
              o15_4 = fma(eb, g4_0, o15_4);
              o15_5 = fma(eb, g5_0, o15_5);
            }
            { const double eb = bi[79];
              o15_4 = fma(eb, g4_1, o15_4);
              o15_5 = fma(eb, g5_1, o15_5);
            }
            { const double eb = bi[80];
              o15_4 = fma(eb, g4_2, o15_4);
              o15_5 = fma(eb, g5_2, o15_5);
            }
            { const double eb = bi[81];
              o15_4 = fma(eb, g4_5, o15_4);
              o15_5 = fma(eb, g5_5, o15_5);
            }
            { const double eb = bi[82];
              o15_4 = fma(eb, g4_3, o15_4);
              o15_5 = fma(eb, g5_3, o15_5);
            }
            { const double eb = bi[83];
              o15_4 = fma(eb, g4_7, o15_4);
              o15_5 = fma(eb, g5_7, o15_5);
            }
            { const double eb = bi[84];
              o15_4 = fma(eb, g4_8, o15_4);
              o15_5 = fma(eb, g5_8, o15_5);
            }
            { const double eb = bi[85];
              o15_4 = fma(eb, g4_15, o15_4);
              o15_5 = fma(eb, g5_15, o15_5);
            }
            { const double eb = bi[86];
              o16_4 = fma(eb, g4_0, o16_4);
              o16_5 = fma(eb, g5_0, o16_5);
            }
            { const double eb = bi[87];
              o16_4 = fma(eb, g4_1, o16_4);
              o16_5 = fma(eb, g5_1, o16_5);
            }
            { const double eb = bi[88];
              o16_4 = fma(eb, g4_3, o16_4);
              o16_5 = fma(eb, g5_3, o16_5);
            }
            { const double eb = bi[89];
              o16_4 = fma(eb, g4_7, o16_4);
              o16_5 = fma(eb, g5_7, o16_5);
            }
            { const double eb = bi[90];
              o17_4 = fma(eb, g4_0, o17_4);
              o17_5 = fma(eb, g5_0, o17_5);
            }
            { const double eb = bi[91];
              o17_4 = fma(eb, g4_1, o17_4);
              o17_5 = fma(eb, g5_1, o17_5);
            }
            { const double eb = bi[92];
              o17_4 = fma(eb, g4_3, o17_4);
              o17_5 = fma(eb, g5_3, o17_5);
            }
            { const double eb = bi[93];
              o17_4 = fma(eb, g4_7, o17_4);
              o17_5 = fma(eb, g5_7, o17_5);
            }
            { const double eb = bi[94];
              o17_4 = fma(eb, g4_9, o17_4);
              o17_5 = fma(eb, g5_9, o17_5);
            }
            { const double eb = bi[95];
              o17_4 = fma(eb, g4_17, o17_4);
              o17_5 = fma(eb, g5_17, o17_5);
            }
            { const double eb = bi[96];
              o18_4 = fma(eb, g4_0, o18_4);
              o18_5 = fma(eb, g5_0, o18_5);
            }
            { const double eb = bi[97];
              o18_4 = fma(eb, g4_1, o18_4);
              o18_5 = fma(eb, g5_1, o18_5);
            }
            { const double eb = bi[98];
              o18_4 = fma(eb, g4_2, o18_4);
              o18_5 = fma(eb, g5_2, o18_5);
            }
            { const double eb = bi[99];
              o18_4 = fma(eb, g4_5, o18_4);
              o18_5 = fma(eb, g5_5, o18_5);
            }
            { const double eb = bi[100];
              o18_4 = fma(eb, g4_3, o18_4);
              o18_5 = fma(eb, g5_3, o18_5);
            }
            { const double eb = bi[101];
              o18_4 = fma(eb, g4_7, o18_4);
              o18_5 = fma(eb, g5_7, o18_5);
            }
            { const double eb = bi[102];
              o18_4 = fma(eb, g4_8, o18_4);
              o18_5 = fma(eb, g5_8, o18_5);
            }
            { const double eb = bi[103];
              o18_4 = fma(eb, g4_15, o18_4);
              o18_5 = fma(eb, g5_15, o18_5);
            }
            { const double eb = bi[104];
              o19_4 = fma(eb, g4_0, o19_4);
              o19_5 = fma(eb, g5_0, o19_5);
            }
            { const double eb = bi[105];
              o19_4 = fma(eb, g4_1, o19_4);
              o19_5 = fma(eb, g5_1, o19_5);
            }
            { const double eb = bi[106];
              o19_4 = fma(eb, g4_4, o19_4);
              o19_5 = fma(eb, g5_4, o19_5);
            }
            { const double eb = bi[107];
              o19_4 = fma(eb, g4_3, o19_4);
              o19_5 = fma(eb, g5_3, o19_5);
            }
            { const double eb = bi[108];
              o19_4 = fma(eb, g4_7, o19_4);
              o19_5 = fma(eb, g5_7, o19_5);
            }
            { const double eb = bi[109];
              o19_4 = fma(eb, g4_14, o19_4);
              o19_5 = fma(eb, g5_14, o19_5);
            }
            { const double eb = bi[110];
              o20_4 = fma(eb, g4_0, o20_4);
              o20_5 = fma(eb, g5_0, o20_5);
            }
            { const double eb = bi[111];
              o20_4 = fma(eb, g4_1, o20_4);
              o20_5 = fma(eb, g5_1, o20_5);
            }
            { const double eb = bi[112];
              o20_4 = fma(eb, g4_2, o20_4);
              o20_5 = fma(eb, g5_2, o20_5);
            }
            { const double eb = bi[113];
              o20_4 = fma(eb, g4_5, o20_4);
              o20_5 = fma(eb, g5_5, o20_5);
            }
            { const double eb = bi[114];
              o21_4 = fma(eb, g4_0, o21_4);
              o21_5 = fma(eb, g5_0, o21_5);
            }
            { const double eb = bi[115];
              o21_4 = fma(eb, g4_1, o21_4);
              o21_5 = fma(eb, g5_1, o21_5);
            }
            { const double eb = bi[116];
              o21_4 = fma(eb, g4_2, o21_4);
              o21_5 = fma(eb, g5_2, o21_5);
            }
            { const double eb = bi[117];
              o21_4 = fma(eb, g4_5, o21_4);
              o21_5 = fma(eb, g5_5, o21_5);
            }
            { const double eb = bi[118];
              o21_4 = fma(eb, g4_3, o21_4);
              o21_5 = fma(eb, g5_3, o21_5);
            }
            { const double eb = bi[119];
              o21_4 = fma(eb, g4_7, o21_4);
              o21_5 = fma(eb, g5_7, o21_5);
            }
            { const double eb = bi[120];
              o21_4 = fma(eb, g4_8, o21_4);
              o21_5 = fma(eb, g5_8, o21_5);
            }
            { const double eb = bi[121];
              o21_4 = fma(eb, g4_15, o21_4);
              o21_5 = fma(eb, g5_15, o21_5);
            }
            { const double eb = bi[122];
              o22_4 = fma(eb, g4_0, o22_4);
              o22_5 = fma(eb, g5_0, o22_5);
            }
            { const double eb = bi[123];
              o22_4 = fma(eb, g4_1, o22_4);
              o22_5 = fma(eb, g5_1, o22_5);
            }
            { const double eb = bi[124];
              o22_4 = fma(eb, g4_2, o22_4);
              o22_5 = fma(eb, g5_2, o22_5);
            }
            { const double eb = bi[125];
              o22_4 = fma(eb, g4_5, o22_4);
              o22_5 = fma(eb, g5_5, o22_5);
            }
            { const double eb = bi[126];
              o22_4 = fma(eb, g4_6, o22_4);
              o22_5 = fma(eb, g5_6, o22_5);
            }
            { const double eb = bi[127];
              o22_4 = fma(eb, g4_12, o22_4);
              o22_5 = fma(eb, g5_12, o22_5);
            }
            { const double eb = bi[128];
              o23_4 = fma(eb, g4_0, o23_4);
              o23_5 = fma(eb, g5_0, o23_5);
            }
            { const double eb = bi[129];
              o23_4 = fma(eb, g4_1, o23_4);
              o23_5 = fma(eb, g5_1, o23_5);
            }
            { const double eb = bi[130];
              o23_4 = fma(eb, g4_4, o23_4);
              o23_5 = fma(eb, g5_4, o23_5);
            }
            { const double eb = bi[131];
              o23_4 = fma(eb, g4_2, o23_4);
              o23_5 = fma(eb, g5_2, o23_5);
            }
            { const double eb = bi[132];
              o23_4 = fma(eb, g4_5, o23_4);
              o23_5 = fma(eb, g5_5, o23_5);
            }
            { const double eb = bi[133];
              o23_4 = fma(eb, g4_11, o23_4);
              o23_5 = fma(eb, g5_11, o23_5);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk4 = PT[(fI + 1) * N + fJ + 0];
            const double ptk5 = PT[(fI + 1) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc3_1 = PA[(fQ + 3) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            jab0 += o0_4 * ptk4 + o0_5 * ptk5;
            jab1 += o1_4 * ptk4 + o1_5 * ptk5;
            jab2 += o2_4 * ptk4 + o2_5 * ptk5;
            jab3 += o3_4 * ptk4 + o3_5 * ptk5;
            jab4 += o4_4 * ptk4 + o4_5 * ptk5;
            jab5 += o5_4 * ptk4 + o5_5 * ptk5;
            jab6 += o6_4 * ptk4 + o6_5 * ptk5;
            jab7 += o7_4 * ptk4 + o7_5 * ptk5;
            jab8 += o8_4 * ptk4 + o8_5 * ptk5;
            jab9 += o9_4 * ptk4 + o9_5 * ptk5;
            jab10 += o10_4 * ptk4 + o10_5 * ptk5;
            jab11 += o11_4 * ptk4 + o11_5 * ptk5;
            jab12 += o12_4 * ptk4 + o12_5 * ptk5;
            jab13 += o13_4 * ptk4 + o13_5 * ptk5;
            jab14 += o14_4 * ptk4 + o14_5 * ptk5;
            jab15 += o15_4 * ptk4 + o15_5 * ptk5;
            jab16 += o16_4 * ptk4 + o16_5 * ptk5;
            jab17 += o17_4 * ptk4 + o17_5 * ptk5;
            jab18 += o18_4 * ptk4 + o18_5 * ptk5;
            jab19 += o19_4 * ptk4 + o19_5 * ptk5;
            jab20 += o20_4 * ptk4 + o20_5 * ptk5;
            jab21 += o21_4 * ptk4 + o21_5 * ptk5;
            jab22 += o22_4 * ptk4 + o22_5 * ptk5;
            jab23 += o23_4 * ptk4 + o23_5 * ptk5;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_4 * ptb0 + o1_4 * ptb1 + o2_4 * ptb2 + o3_4 * ptb3 + o4_4 * ptb4 + o5_4 * ptb5 + o6_4 * ptb6 + o7_4 * ptb7 + o8_4 * ptb8 + o9_4 * ptb9 + o10_4 * ptb10 + o11_4 * ptb11 + o12_4 * ptb12 + o13_4 * ptb13 + o14_4 * ptb14 + o15_4 * ptb15 + o16_4 * ptb16 + o17_4 * ptb17 + o18_4 * ptb18 + o19_4 * ptb19 + o20_4 * ptb20 + o21_4 * ptb21 + o22_4 * ptb22 + o23_4 * ptb23));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 1, 2.0 * deg * (o0_5 * ptb0 + o1_5 * ptb1 + o2_5 * ptb2 + o3_5 * ptb3 + o4_5 * ptb4 + o5_5 * ptb5 + o6_5 * ptb6 + o7_5 * ptb7 + o8_5 * ptb8 + o9_5 * ptb9 + o10_5 * ptb10 + o11_5 * ptb11 + o12_5 * ptb12 + o13_5 * ptb13 + o14_5 * ptb14 + o15_5 * ptb15 + o16_5 * ptb16 + o17_5 * ptb17 + o18_5 * ptb18 + o19_5 * ptb19 + o20_5 * ptb20 + o21_5 * ptb21 + o22_5 * ptb22 + o23_5 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_4 * Abd0_0 + o0_5 * Abd0_1 + o1_4 * Abd1_0 + o1_5 * Abd1_1 + o2_4 * Abd2_0 + o2_5 * Abd2_1 + o3_4 * Abd3_0 + o3_5 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_4 * Aad0_0 + o0_5 * Aad0_1 + o4_4 * Aad1_0 + o4_5 * Aad1_1 + o8_4 * Aad2_0 + o8_5 * Aad2_1 + o12_4 * Aad3_0 + o12_5 * Aad3_1 + o16_4 * Aad4_0 + o16_5 * Aad4_1 + o20_4 * Aad5_0 + o20_5 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Abc0_1 + o1_4 * Abc1_1 + o2_4 * Abc2_1 + o3_4 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Aac0_1 + o4_4 * Aac1_1 + o8_4 * Aac2_1 + o12_4 * Aac3_1 + o16_4 * Aac4_1 + o20_4 * Aac5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_5 * Abc0_1 + o1_5 * Abc1_1 + o2_5 * Abc2_1 + o3_5 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_5 * Aac0_1 + o4_5 * Aac1_1 + o8_5 * Aac2_1 + o12_5 * Aac3_1 + o16_5 * Aac4_1 + o20_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_4 * Aad0_0 + o1_5 * Aad0_1 + o5_4 * Aad1_0 + o5_5 * Aad1_1 + o9_4 * Aad2_0 + o9_5 * Aad2_1 + o13_4 * Aad3_0 + o13_5 * Aad3_1 + o17_4 * Aad4_0 + o17_5 * Aad4_1 + o21_4 * Aad5_0 + o21_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Aac0_1 + o5_4 * Aac1_1 + o9_4 * Aac2_1 + o13_4 * Aac3_1 + o17_4 * Aac4_1 + o21_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_5 * Aac0_1 + o5_5 * Aac1_1 + o9_5 * Aac2_1 + o13_5 * Aac3_1 + o17_5 * Aac4_1 + o21_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_4 * Aad0_0 + o2_5 * Aad0_1 + o6_4 * Aad1_0 + o6_5 * Aad1_1 + o10_4 * Aad2_0 + o10_5 * Aad2_1 + o14_4 * Aad3_0 + o14_5 * Aad3_1 + o18_4 * Aad4_0 + o18_5 * Aad4_1 + o22_4 * Aad5_0 + o22_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Aac0_1 + o6_4 * Aac1_1 + o10_4 * Aac2_1 + o14_4 * Aac3_1 + o18_4 * Aac4_1 + o22_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_5 * Aac0_1 + o6_5 * Aac1_1 + o10_5 * Aac2_1 + o14_5 * Aac3_1 + o18_5 * Aac4_1 + o22_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_4 * Aad0_0 + o3_5 * Aad0_1 + o7_4 * Aad1_0 + o7_5 * Aad1_1 + o11_4 * Aad2_0 + o11_5 * Aad2_1 + o15_4 * Aad3_0 + o15_5 * Aad3_1 + o19_4 * Aad4_0 + o19_5 * Aad4_1 + o23_4 * Aad5_0 + o23_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Aac0_1 + o7_4 * Aac1_1 + o11_4 * Aac2_1 + o15_4 * Aac3_1 + o19_4 * Aac4_1 + o23_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_5 * Aac0_1 + o7_5 * Aac1_1 + o11_5 * Aac2_1 + o15_5 * Aac3_1 + o19_5 * Aac4_1 + o23_5 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_4 * Abd0_0 + o4_5 * Abd0_1 + o5_4 * Abd1_0 + o5_5 * Abd1_1 + o6_4 * Abd2_0 + o6_5 * Abd2_1 + o7_4 * Abd3_0 + o7_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_4 * Abc0_1 + o5_4 * Abc1_1 + o6_4 * Abc2_1 + o7_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_5 * Abc0_1 + o5_5 * Abc1_1 + o6_5 * Abc2_1 + o7_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_4 * Abd0_0 + o8_5 * Abd0_1 + o9_4 * Abd1_0 + o9_5 * Abd1_1 + o10_4 * Abd2_0 + o10_5 * Abd2_1 + o11_4 * Abd3_0 + o11_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_4 * Abc0_1 + o9_4 * Abc1_1 + o10_4 * Abc2_1 + o11_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_5 * Abc0_1 + o9_5 * Abc1_1 + o10_5 * Abc2_1 + o11_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_4 * Abd0_0 + o12_5 * Abd0_1 + o13_4 * Abd1_0 + o13_5 * Abd1_1 + o14_4 * Abd2_0 + o14_5 * Abd2_1 + o15_4 * Abd3_0 + o15_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_4 * Abc0_1 + o13_4 * Abc1_1 + o14_4 * Abc2_1 + o15_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_5 * Abc0_1 + o13_5 * Abc1_1 + o14_5 * Abc2_1 + o15_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_4 * Abd0_0 + o16_5 * Abd0_1 + o17_4 * Abd1_0 + o17_5 * Abd1_1 + o18_4 * Abd2_0 + o18_5 * Abd2_1 + o19_4 * Abd3_0 + o19_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_4 * Abc0_1 + o17_4 * Abc1_1 + o18_4 * Abc2_1 + o19_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_5 * Abc0_1 + o17_5 * Abc1_1 + o18_5 * Abc2_1 + o19_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_4 * Abd0_0 + o20_5 * Abd0_1 + o21_4 * Abd1_0 + o21_5 * Abd1_1 + o22_4 * Abd2_0 + o22_5 * Abd2_1 + o23_4 * Abd3_0 + o23_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_4 * Abc0_1 + o21_4 * Abc1_1 + o22_4 * Abc2_1 + o23_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_5 * Abc0_1 + o21_5 * Abc1_1 + o22_5 * Abc2_1 + o23_5 * Abc3_1));
          }
        } break;
        case 3: {  // ket functions [6, 7]
          double o0_6 = 0;
          double o0_7 = 0;
          double o1_6 = 0;
          double o1_7 = 0;
          double o2_6 = 0;
          double o2_7 = 0;
          double o3_6 = 0;
          double o3_7 = 0;
          double o4_6 = 0;
          double o4_7 = 0;
          double o5_6 = 0;
          double o5_7 = 0;
          double o6_6 = 0;
          double o6_7 = 0;
          double o7_6 = 0;
          double o7_7 = 0;
          double o8_6 = 0;
          double o8_7 = 0;
          double o9_6 = 0;
          double o9_7 = 0;
          double o10_6 = 0;
          double o10_7 = 0;
          double o11_6 = 0;
          double o11_7 = 0;
          double o12_6 = 0;
          double o12_7 = 0;
          double o13_6 = 0;
          double o13_7 = 0;
          double o14_6 = 0;
          double o14_7 = 0;
          double o15_6 = 0;
          double o15_7 = 0;
          double o16_6 = 0;
          double o16_7 = 0;
          double o17_6 = 0;
          double o17_7 = 0;
          double o18_6 = 0;
          double o18_7 = 0;
          double o19_6 = 0;
          double o19_7 = 0;
          double o20_6 = 0;
          double o20_7 = 0;
          double o21_6 = 0;
          double o21_7 = 0;
          double o22_6 = 0;
          double o22_7 = 0;
          double o23_6 = 0;
          double o23_7 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek6_0 = kj[33 * kS];
              const double ek6_1 = -kj[34 * kS];
              const double ek6_2 = kj[35 * kS];
              const double ek6_3 = -kj[36 * kS];
              const double ek7_0 = kj[37 * kS];
              const double ek7_1 = -kj[38 * kS];
              const double ek7_2 = -kj[39 * kS];
              const double ek7_3 = kj[40 * kS];
              const double ek7_4 = kj[41 * kS];
              const double ek7_5 = -kj[42 * kS];
              g6_0 = fma(ek6_0, b0, g6_0);
              g7_0 = fma(ek7_0, b0, g7_0);
              const double r0_0_0_1 = Z * b1;
              g6_1 = fma(ek6_0, r0_0_0_1, g6_1);
              g7_1 = fma(ek7_0, r0_0_0_1, g7_1);
              g7_0 = fma(ek7_1, r0_0_0_1, g7_0);
              const double r0_0_1_0 = Y * b1;
              g6_2 = fma(ek6_0, r0_0_1_0, g6_2);
              g6_0 = fma(ek6_1, r0_0_1_0, g6_0);
              g7_2 = fma(ek7_0, r0_0_1_0, g7_2);
              g7_0 = fma(ek7_2, r0_0_1_0, g7_0);
              const double r0_1_0_0 = X * b1;
              g6_3 = fma(ek6_0, r0_1_0_0, g6_3);
              g7_3 = fma(ek7_0, r0_1_0_0, g7_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g6_4 = fma(ek6_0, r0_0_0_2, g6_4);
              g7_4 = fma(ek7_0, r0_0_0_2, g7_4);
              g7_1 = fma(ek7_1, r0_0_0_2, g7_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g6_5 = fma(ek6_0, r0_0_1_1, g6_5);
              g6_1 = fma(ek6_1, r0_0_1_1, g6_1);
              g7_5 = fma(ek7_0, r0_0_1_1, g7_5);
              g7_2 = fma(ek7_1, r0_0_1_1, g7_2);
              g7_1 = fma(ek7_2, r0_0_1_1, g7_1);
              g7_0 = fma(ek7_3, r0_0_1_1, g7_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g6_6 = fma(ek6_0, r0_0_2_0, g6_6);
              g6_2 = fma(ek6_1, r0_0_2_0, g6_2);
              g6_0 = fma(ek6_2, r0_0_2_0, g6_0);
              g7_6 = fma(ek7_0, r0_0_2_0, g7_6);
              g7_2 = fma(ek7_2, r0_0_2_0, g7_2);
              g7_0 = fma(ek7_4, r0_0_2_0, g7_0);
              const double r0_1_0_1 = X * r1_0_0_1;
              g6_7 = fma(ek6_0, r0_1_0_1, g6_7);
              g7_7 = fma(ek7_0, r0_1_0_1, g7_7);
              g7_3 = fma(ek7_1, r0_1_0_1, g7_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g6_8 = fma(ek6_0, r0_1_1_0, g6_8);
              g6_3 = fma(ek6_1, r0_1_1_0, g6_3);
              g7_8 = fma(ek7_0, r0_1_1_0, g7_8);
              g7_3 = fma(ek7_2, r0_1_1_0, g7_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g6_9 = fma(ek6_0, r0_2_0_0, g6_9);
              g7_9 = fma(ek7_0, r0_2_0_0, g7_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g6_10 = fma(ek6_0, r0_0_0_3, g6_10);
              g7_10 = fma(ek7_0, r0_0_0_3, g7_10);
              g7_4 = fma(ek7_1, r0_0_0_3, g7_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g6_11 = fma(ek6_0, r0_0_1_2, g6_11);
              g6_4 = fma(ek6_1, r0_0_1_2, g6_4);
              g7_11 = fma(ek7_0, r0_0_1_2, g7_11);
              g7_5 = fma(ek7_1, r0_0_1_2, g7_5);
              g7_4 = fma(ek7_2, r0_0_1_2, g7_4);
              g7_1 = fma(ek7_3, r0_0_1_2, g7_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g6_12 = fma(ek6_0, r0_0_2_1, g6_12);
              g6_5 = fma(ek6_1, r0_0_2_1, g6_5);
              g6_1 = fma(ek6_2, r0_0_2_1, g6_1);
              g7_12 = fma(ek7_0, r0_0_2_1, g7_12);
              g7_6 = fma(ek7_1, r0_0_2_1, g7_6);
              g7_5 = fma(ek7_2, r0_0_2_1, g7_5);
              g7_2 = fma(ek7_3, r0_0_2_1, g7_2);
              g7_1 = fma(ek7_4, r0_0_2_1, g7_1);
              g7_0 = fma(ek7_5, r0_0_2_1, g7_0);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g6_13 = fma(ek6_0, r0_0_3_0, g6_13);
              g6_6 = fma(ek6_1, r0_0_3_0, g6_6);
              g6_2 = fma(ek6_2, r0_0_3_0, g6_2);
              g6_0 = fma(ek6_3, r0_0_3_0, g6_0);
              g7_13 = fma(ek7_0, r0_0_3_0, g7_13);
              g7_6 = fma(ek7_2, r0_0_3_0, g7_6);
              g7_2 = fma(ek7_4, r0_0_3_0, g7_2);
              const double r0_1_0_2 = X * r1_0_0_2;
              g6_14 = fma(ek6_0, r0_1_0_2, g6_14);
              g7_14 = fma(ek7_0, r0_1_0_2, g7_14);
              g7_7 = fma(ek7_1, r0_1_0_2, g7_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g6_15 = fma(ek6_0, r0_1_1_1, g6_15);
              g6_7 = fma(ek6_1, r0_1_1_1, g6_7);
              g7_15 = fma(ek7_0, r0_1_1_1, g7_15);
              g7_8 = fma(ek7_1, r0_1_1_1, g7_8);
              g7_7 = fma(ek7_2, r0_1_1_1, g7_7);
              g7_3 = fma(ek7_3, r0_1_1_1, g7_3);
              const double r0_1_2_0 = X * r1_0_2_0;
              g6_16 = fma(ek6_0, r0_1_2_0, g6_16);
              g6_8 = fma(ek6_1, r0_1_2_0, g6_8);
              g6_3 = fma(ek6_2, r0_1_2_0, g6_3);
              g7_16 = fma(ek7_0, r0_1_2_0, g7_16);
              g7_8 = fma(ek7_2, r0_1_2_0, g7_8);
              g7_3 = fma(ek7_4, r0_1_2_0, g7_3);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g6_17 = fma(ek6_0, r0_2_0_1, g6_17);
              g7_17 = fma(ek7_0, r0_2_0_1, g7_17);
              g7_9 = fma(ek7_1, r0_2_0_1, g7_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g6_18 = fma(ek6_0, r0_2_1_0, g6_18);
              g6_9 = fma(ek6_1, r0_2_1_0, g6_9);
              g7_18 = fma(ek7_0, r0_2_1_0, g7_18);
              g7_9 = fma(ek7_2, r0_2_1_0, g7_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g6_19 = fma(ek6_0, r0_3_0_0, g6_19);
              g7_19 = fma(ek7_0, r0_3_0_0, g7_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g7_10 = fma(ek7_1, r0_0_0_4, g7_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g6_10 = fma(ek6_1, r0_0_1_3, g6_10);
              g7_11 = fma(ek7_1, r0_0_1_3, g7_11);
              g7_10 = fma(ek7_2, r0_0_1_3, g7_10);
              g7_4 = fma(ek7_3, r0_0_1_3, g7_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g6_11 = fma(ek6_1, r0_0_2_2, g6_11);
              g6_4 = fma(ek6_2, r0_0_2_2, g6_4);
              g7_12 = fma(ek7_1, r0_0_2_2, g7_12);
              g7_11 = fma(ek7_2, r0_0_2_2, g7_11);
              g7_5 = fma(ek7_3, r0_0_2_2, g7_5);
              g7_4 = fma(ek7_4, r0_0_2_2, g7_4);
              g7_1 = fma(ek7_5, r0_0_2_2, g7_1);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g6_12 = fma(ek6_1, r0_0_3_1, g6_12);
              g6_5 = fma(ek6_2, r0_0_3_1, g6_5);
              g6_1 = fma(ek6_3, r0_0_3_1, g6_1);
              g7_13 = fma(ek7_1, r0_0_3_1, g7_13);
              g7_12 = fma(ek7_2, r0_0_3_1, g7_12);
              g7_6 = fma(ek7_3, r0_0_3_1, g7_6);
              g7_5 = fma(ek7_4, r0_0_3_1, g7_5);
              g7_2 = fma(ek7_5, r0_0_3_1, g7_2);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g6_13 = fma(ek6_1, r0_0_4_0, g6_13);
              g6_6 = fma(ek6_2, r0_0_4_0, g6_6);
              g6_2 = fma(ek6_3, r0_0_4_0, g6_2);
              g7_13 = fma(ek7_2, r0_0_4_0, g7_13);
              g7_6 = fma(ek7_4, r0_0_4_0, g7_6);
              const double r0_1_0_3 = X * r1_0_0_3;
              g7_14 = fma(ek7_1, r0_1_0_3, g7_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g6_14 = fma(ek6_1, r0_1_1_2, g6_14);
              g7_15 = fma(ek7_1, r0_1_1_2, g7_15);
              g7_14 = fma(ek7_2, r0_1_1_2, g7_14);
              g7_7 = fma(ek7_3, r0_1_1_2, g7_7);
              const double r0_1_2_1 = X * r1_0_2_1;
              g6_15 = fma(ek6_1, r0_1_2_1, g6_15);
              g6_7 = fma(ek6_2, r0_1_2_1, g6_7);
              g7_16 = fma(ek7_1, r0_1_2_1, g7_16);
              g7_15 = fma(ek7_2, r0_1_2_1, g7_15);
              g7_8 = fma(ek7_3, r0_1_2_1, g7_8);
              g7_7 = fma(ek7_4, r0_1_2_1, g7_7);
              g7_3 = fma(ek7_5, r0_1_2_1, g7_3);
              const double r0_1_3_0 = X * r1_0_3_0;
              g6_16 = fma(ek6_1, r0_1_3_0, g6_16);
              g6_8 = fma(ek6_2, r0_1_3_0, g6_8);
              g6_3 = fma(ek6_3, r0_1_3_0, g6_3);
              g7_16 = fma(ek7_2, r0_1_3_0, g7_16);
              g7_8 = fma(ek7_4, r0_1_3_0, g7_8);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g7_17 = fma(ek7_1, r0_2_0_2, g7_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g6_17 = fma(ek6_1, r0_2_1_1, g6_17);
              g7_18 = fma(ek7_1, r0_2_1_1, g7_18);
              g7_17 = fma(ek7_2, r0_2_1_1, g7_17);
              g7_9 = fma(ek7_3, r0_2_1_1, g7_9);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g6_18 = fma(ek6_1, r0_2_2_0, g6_18);
              g6_9 = fma(ek6_2, r0_2_2_0, g6_9);
              g7_18 = fma(ek7_2, r0_2_2_0, g7_18);
              g7_9 = fma(ek7_4, r0_2_2_0, g7_9);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g7_19 = fma(ek7_1, r0_3_0_1, g7_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g6_19 = fma(ek6_1, r0_3_1_0, g6_19);
              g7_19 = fma(ek7_2, r0_3_1_0, g7_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g7_10 = fma(ek7_3, r0_0_1_4, g7_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g6_10 = fma(ek6_2, r0_0_2_3, g6_10);
              g7_11 = fma(ek7_3, r0_0_2_3, g7_11);
              g7_10 = fma(ek7_4, r0_0_2_3, g7_10);
              g7_4 = fma(ek7_5, r0_0_2_3, g7_4);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g6_11 = fma(ek6_2, r0_0_3_2, g6_11);
              g6_4 = fma(ek6_3, r0_0_3_2, g6_4);
              g7_12 = fma(ek7_3, r0_0_3_2, g7_12);
              g7_11 = fma(ek7_4, r0_0_3_2, g7_11);
              g7_5 = fma(ek7_5, r0_0_3_2, g7_5);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g6_12 = fma(ek6_2, r0_0_4_1, g6_12);
              g6_5 = fma(ek6_3, r0_0_4_1, g6_5);
              g7_13 = fma(ek7_3, r0_0_4_1, g7_13);
              g7_12 = fma(ek7_4, r0_0_4_1, g7_12);
              g7_6 = fma(ek7_5, r0_0_4_1, g7_6);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g6_13 = fma(ek6_2, r0_0_5_0, g6_13);
              g6_6 = fma(ek6_3, r0_0_5_0, g6_6);
              g7_13 = fma(ek7_4, r0_0_5_0, g7_13);
              const double r0_1_1_3 = X * r1_0_1_3;
              g7_14 = fma(ek7_3, r0_1_1_3, g7_14);
              const double r0_1_2_2 = X * r1_0_2_2;
              g6_14 = fma(ek6_2, r0_1_2_2, g6_14);
              g7_15 = fma(ek7_3, r0_1_2_2, g7_15);
              g7_14 = fma(ek7_4, r0_1_2_2, g7_14);
              g7_7 = fma(ek7_5, r0_1_2_2, g7_7);
              const double r0_1_3_1 = X * r1_0_3_1;
              g6_15 = fma(ek6_2, r0_1_3_1, g6_15);
              g6_7 = fma(ek6_3, r0_1_3_1, g6_7);
              g7_16 = fma(ek7_3, r0_1_3_1, g7_16);
              g7_15 = fma(ek7_4, r0_1_3_1, g7_15);
              g7_8 = fma(ek7_5, r0_1_3_1, g7_8);
              const double r0_1_4_0 = X * r1_0_4_0;
              g6_16 = fma(ek6_2, r0_1_4_0, g6_16);
              g6_8 = fma(ek6_3, r0_1_4_0, g6_8);
              g7_16 = fma(ek7_4, r0_1_4_0, g7_16);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g7_17 = fma(ek7_3, r0_2_1_2, g7_17);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g6_17 = fma(ek6_2, r0_2_2_1, g6_17);
              g7_18 = fma(ek7_3, r0_2_2_1, g7_18);
              g7_17 = fma(ek7_4, r0_2_2_1, g7_17);
              g7_9 = fma(ek7_5, r0_2_2_1, g7_9);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g6_18 = fma(ek6_2, r0_2_3_0, g6_18);
              g6_9 = fma(ek6_3, r0_2_3_0, g6_9);
              g7_18 = fma(ek7_4, r0_2_3_0, g7_18);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g7_19 = fma(ek7_3, r0_3_1_1, g7_19);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g6_19 = fma(ek6_2, r0_3_2_0, g6_19);
              g7_19 = fma(ek7_4, r0_3_2_0, g7_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_0_2_4 = fma(Y, r1_0_1_4, r1_0_0_4);
              g7_10 = fma(ek7_5, r0_0_2_4, g7_10);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_0_3_3 = fma(Y, r1_0_2_3, 2.0 * r1_0_1_3);
              g6_10 = fma(ek6_3, r0_0_3_3, g6_10);
              g7_11 = fma(ek7_5, r0_0_3_3, g7_11);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_0_4_2 = fma(Y, r1_0_3_2, 3.0 * r1_0_2_2);
              g6_11 = fma(ek6_3, r0_0_4_2, g6_11);
              g7_12 = fma(ek7_5, r0_0_4_2, g7_12);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_0_5_1 = fma(Y, r1_0_4_1, 4.0 * r1_0_3_1);
              g6_12 = fma(ek6_3, r0_0_5_1, g6_12);
              g7_13 = fma(ek7_5, r0_0_5_1, g7_13);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_0_5_0 = fma(Y, r2_0_4_0, 4.0 * r2_0_3_0);
              const double r0_0_6_0 = fma(Y, r1_0_5_0, 5.0 * r1_0_4_0);
              g6_13 = fma(ek6_3, r0_0_6_0, g6_13);
              const double r0_1_2_3 = X * r1_0_2_3;
              g7_14 = fma(ek7_5, r0_1_2_3, g7_14);
              const double r0_1_3_2 = X * r1_0_3_2;
              g6_14 = fma(ek6_3, r0_1_3_2, g6_14);
              g7_15 = fma(ek7_5, r0_1_3_2, g7_15);
              const double r0_1_4_1 = X * r1_0_4_1;
              g6_15 = fma(ek6_3, r0_1_4_1, g6_15);
              g7_16 = fma(ek7_5, r0_1_4_1, g7_16);
              const double r0_1_5_0 = X * r1_0_5_0;
              g6_16 = fma(ek6_3, r0_1_5_0, g6_16);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g7_17 = fma(ek7_5, r0_2_2_2, g7_17);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g6_17 = fma(ek6_3, r0_2_3_1, g6_17);
              g7_18 = fma(ek7_5, r0_2_3_1, g7_18);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g6_18 = fma(ek6_3, r0_2_4_0, g6_18);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g7_19 = fma(ek7_5, r0_3_2_1, g7_19);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g6_19 = fma(ek6_3, r0_3_3_0, g6_19);
            }
            { const double eb = bi[5];
              o0_6 = fma(eb, g6_0, o0_6);
              o0_7 = fma(eb, g7_0, o0_7);
            }
            { const double eb = bi[6];
              o0_6 = fma(eb, g6_3, o0_6);
              o0_7 = fma(eb, g7_3, o0_7);
            }
            { const double eb = bi[7];
              o0_6 = fma(eb, g6_9, o0_6);
              o0_7 = fma(eb, g7_9, o0_7);
            }
            { const double eb = bi[8];
              o1_6 = fma(eb, g6_0, o1_6);
              o1_7 = fma(eb, g7_0, o1_7);
            }
            { const double eb = bi[9];
              o1_6 = fma(eb, g6_3, o1_6);
              o1_7 = fma(eb, g7_3, o1_7);
            }
            { const double eb = bi[10];
              o1_6 = fma(eb, g6_9, o1_6);
              o1_7 = fma(eb, g7_9, o1_7);
            }
            { const double eb = bi[11];
              o1_6 = fma(eb, g6_19, o1_6);
              o1_7 = fma(eb, g7_19, o1_7);
            }
            { const double eb = bi[12];
              o2_6 = fma(eb, g6_0, o2_6);
              o2_7 = fma(eb, g7_0, o2_7);
            }
            { const double eb = bi[13];
              o2_6 = fma(eb, g6_2, o2_6);
              o2_7 = fma(eb, g7_2, o2_7);
            }
            { const double eb = bi[14];
              o2_6 = fma(eb, g6_3, o2_6);
              o2_7 = fma(eb, g7_3, o2_7);
            }
            { const double eb = bi[15];
              o2_6 = fma(eb, g6_8, o2_6);
              o2_7 = fma(eb, g7_8, o2_7);
            }
            { const double eb = bi[16];
              o2_6 = fma(eb, g6_9, o2_6);
              o2_7 = fma(eb, g7_9, o2_7);
            }
            { const double eb = bi[17];
              o2_6 = fma(eb, g6_18, o2_6);
              o2_7 = fma(eb, g7_18, o2_7);
            }
            { const double eb = bi[18];
              o3_6 = fma(eb, g6_0, o3_6);
              o3_7 = fma(eb, g7_0, o3_7);
            }
            { const double eb = bi[19];
              o3_6 = fma(eb, g6_1, o3_6);
              o3_7 = fma(eb, g7_1, o3_7);
            }
            { const double eb = bi[20];
              o3_6 = fma(eb, g6_3, o3_6);
              o3_7 = fma(eb, g7_3, o3_7);
            }
            { const double eb = bi[21];
              o3_6 = fma(eb, g6_7, o3_6);
              o3_7 = fma(eb, g7_7, o3_7);
            }
            { const double eb = bi[22];
              o3_6 = fma(eb, g6_9, o3_6);
              o3_7 = fma(eb, g7_9, o3_7);
            }
            { const double eb = bi[23];
              o3_6 = fma(eb, g6_17, o3_6);
              o3_7 = fma(eb, g7_17, o3_7);
            }
            { const double eb = bi[24];
              o4_6 = fma(eb, g6_0, o4_6);
              o4_7 = fma(eb, g7_0, o4_7);
            }
            { const double eb = bi[25];
              o4_6 = fma(eb, g6_2, o4_6);
              o4_7 = fma(eb, g7_2, o4_7);
            }
            { const double eb = bi[26];
              o4_6 = fma(eb, g6_6, o4_6);
              o4_7 = fma(eb, g7_6, o4_7);
            }
            { const double eb = bi[27];
              o5_6 = fma(eb, g6_0, o5_6);
              o5_7 = fma(eb, g7_0, o5_7);
            }
            { const double eb = bi[28];
              o5_6 = fma(eb, g6_2, o5_6);
              o5_7 = fma(eb, g7_2, o5_7);
            }
            { const double eb = bi[29];
              o5_6 = fma(eb, g6_6, o5_6);
              o5_7 = fma(eb, g7_6, o5_7);
            }
            { const double eb = bi[30];
              o5_6 = fma(eb, g6_3, o5_6);
              o5_7 = fma(eb, g7_3, o5_7);
            }
            { const double eb = bi[31];
              o5_6 = fma(eb, g6_8, o5_6);
              o5_7 = fma(eb, g7_8, o5_7);
            }
            { const double eb = bi[32];
              o5_6 = fma(eb, g6_16, o5_6);
              o5_7 = fma(eb, g7_16, o5_7);
            }
            { const double eb = bi[33];
              o6_6 = fma(eb, g6_0, o6_6);
              o6_7 = fma(eb, g7_0, o6_7);
            }
            { const double eb = bi[34];
              o6_6 = fma(eb, g6_2, o6_6);
              o6_7 = fma(eb, g7_2, o6_7);
            }
            { const double eb = bi[35];
              o6_6 = fma(eb, g6_6, o6_6);
              o6_7 = fma(eb, g7_6, o6_7);
            }
            { const double eb = bi[36];
              o6_6 = fma(eb, g6_13, o6_6);
              o6_7 = fma(eb, g7_13, o6_7);
            }
            { const double eb = bi[37];
              o7_6 = fma(eb, g6_0, o7_6);
              o7_7 = fma(eb, g7_0, o7_7);
            }
            { const double eb = bi[38];
              o7_6 = fma(eb, g6_1, o7_6);
              o7_7 = fma(eb, g7_1, o7_7);
            }
            { const double eb = bi[39];
              o7_6 = fma(eb, g6_2, o7_6);
              o7_7 = fma(eb, g7_2, o7_7);
            }
            { const double eb = bi[40];
              o7_6 = fma(eb, g6_5, o7_6);
              o7_7 = fma(eb, g7_5, o7_7);
            }
            { const double eb = bi[41];
              o7_6 = fma(eb, g6_6, o7_6);
              o7_7 = fma(eb, g7_6, o7_7);
            }
            { const double eb = bi[42];
              o7_6 = fma(eb, g6_12, o7_6);
              o7_7 = fma(eb, g7_12, o7_7);
            }
            { const double eb = bi[43];
              o8_6 = fma(eb, g6_0, o8_6);
              o8_7 = fma(eb, g7_0, o8_7);
            }
            { const double eb = bi[44];
              o8_6 = fma(eb, g6_1, o8_6);
              o8_7 = fma(eb, g7_1, o8_7);
            }
            { const double eb = bi[45];
              o8_6 = fma(eb, g6_4, o8_6);
              o8_7 = fma(eb, g7_4, o8_7);
            }
            { const double eb = bi[46];
              o9_6 = fma(eb, g6_0, o9_6);
              o9_7 = fma(eb, g7_0, o9_7);
            }
            { const double eb = bi[47];
              o9_6 = fma(eb, g6_1, o9_6);
              o9_7 = fma(eb, g7_1, o9_7);
            }
            { const double eb = bi[48];
              o9_6 = fma(eb, g6_4, o9_6);
              o9_7 = fma(eb, g7_4, o9_7);
            }
            { const double eb = bi[49];
              o9_6 = fma(eb, g6_3, o9_6);
              o9_7 = fma(eb, g7_3, o9_7);
            }
            { const double eb = bi[50];
              o9_6 = fma(eb, g6_7, o9_6);
              o9_7 = fma(eb, g7_7, o9_7);
            }
            { const double eb = bi[51];
              o9_6 = fma(eb, g6_14, o9_6);
              o9_7 = fma(eb, g7_14, o9_7);
            }
            { const double eb = bi[52];
              o10_6 = fma(eb, g6_0, o10_6);
              o10_7 = fma(eb, g7_0, o10_7);
            }
            { const double eb = bi[53];
              o10_6 = fma(eb, g6_1, o10_6);
              o10_7 = fma(eb, g7_1, o10_7);
            }
            { const double eb = bi[54];
              o10_6 = fma(eb, g6_4, o10_6);
              o10_7 = fma(eb, g7_4, o10_7);
            }
            { const double eb = bi[55];
              o10_6 = fma(eb, g6_2, o10_6);
              o10_7 = fma(eb, g7_2, o10_7);
            }
            { const double eb = bi[56];
              o10_6 = fma(eb, g6_5, o10_6);
              o10_7 = fma(eb, g7_5, o10_7);
            }
            { const double eb = bi[57];
              o10_6 = fma(eb, g6_11, o10_6);
              o10_7 = fma(eb, g7_11, o10_7);
            }
            { const double eb = bi[58];
              o11_6 = fma(eb, g6_0, o11_6);
              o11_7 = fma(eb, g7_0, o11_7);
            }
            { const double eb = bi[59];
              o11_6 = fma(eb, g6_1, o11_6);
              o11_7 = fma(eb, g7_1, o11_7);
            }
            { const double eb = bi[60];
              o11_6 = fma(eb, g6_4, o11_6);
              o11_7 = fma(eb, g7_4, o11_7);
            }
            { const double eb = bi[61];
              o11_6 = fma(eb, g6_10, o11_6);
              o11_7 = fma(eb, g7_10, o11_7);
            }
            { const double eb = bi[62];
              o12_6 = fma(eb, g6_0, o12_6);
              o12_7 = fma(eb, g7_0, o12_7);
            }
            { const double eb = bi[63];
              o12_6 = fma(eb, g6_2, o12_6);
              o12_7 = fma(eb, g7_2, o12_7);
            }
            { const double eb = bi[64];
              o12_6 = fma(eb, g6_3, o12_6);
              o12_7 = fma(eb, g7_3, o12_7);
            }
            { const double eb = bi[65];
              o12_6 = fma(eb, g6_8, o12_6);
              o12_7 = fma(eb, g7_8, o12_7);
            }
            { const double eb = bi[66];
              o13_6 = fma(eb, g6_0, o13_6);
              o13_7 = fma(eb, g7_0, o13_7);
            }
            { const double eb = bi[67];
              o13_6 = fma(eb, g6_2, o13_6);
              o13_7 = fma(eb, g7_2, o13_7);
            }
            { const double eb = bi[68];
              o13_6 = fma(eb, g6_3, o13_6);
              o13_7 = fma(eb, g7_3, o13_7);
            }
            { const double eb = bi[69];
              o13_6 = fma(eb, g6_8, o13_6);
              o13_7 = fma(eb, g7_8, o13_7);
            }
            { const double eb = bi[70];
              o13_6 = fma(eb, g6_9, o13_6);
              o13_7 = fma(eb, g7_9, o13_7);
            }
            { const double eb = bi[71];
              o13_6 = fma(eb, g6_18, o13_6);
              o13_7 = fma(eb, g7_18, o13_7);
            }
            { const double eb = bi[72];
              o14_6 = fma(eb, g6_0, o14_6);
              o14_7 = fma(eb, g7_0, o14_7);
            }
            { const double eb = bi[73];
              o14_6 = fma(eb, g6_2, o14_6);
              o14_7 = fma(eb, g7_2, o14_7);
            }
            { const double eb = bi[74];
              o14_6 = fma(eb, g6_6, o14_6);
              o14_7 = fma(eb, g7_6, o14_7);
            }
            { const double eb = bi[75];
              o14_6 = fma(eb, g6_3, o14_6);
              o14_7 = fma(eb, g7_3, o14_7);
            }
            { const double eb = bi[76];
              o14_6 = fma(eb, g6_8, o14_6);
              o14_7 = fma(eb, g7_8, o14_7);
            }
            { const double eb = bi[77];
              o14_6 = fma(eb, g6_16, o14_6);
              o14_7 = fma(eb, g7_16, o14_7);
            }
            { const double eb = bi[78];
              o15_6 = fma(eb, g6_0, o15_6);
              o15_7 = fma(eb, g7_0, o15_7);
            }
            { const double eb = bi[79];
              o15_6 = fma(eb, g6_1, o15_6);
              o15_7 = fma(eb, g7_1, o15_7);
            }
            { const double eb = bi[80];
              o15_6 = fma(eb, g6_2, o15_6);
              o15_7 = fma(eb, g7_2, o15_7);
            }
            { const double eb = bi[81];
              o15_6 = fma(eb, g6_5, o15_6);
              o15_7 = fma(eb, g7_5, o15_7);
            }
            { const double eb = bi[82];
              o15_6 = fma(eb, g6_3, o15_6);
              o15_7 = fma(eb, g7_3, o15_7);
            }
            { const double eb = bi[83];
              o15_6 = fma(eb, g6_7, o15_6);
              o15_7 = fma(eb, g7_7, o15_7);
            }
            { const double eb = bi[84];
              o15_6 = fma(eb, g6_8, o15_6);
              o15_7 = fma(eb, g7_8, o15_7);
            }
            { const double eb = bi[85];
              o15_6 = fma(eb, g6_15, o15_6);
              o15_7 = fma(eb, g7_15, o15_7);
            }
            { const double eb = bi[86];
              o16_6 = fma(eb, g6_0, o16_6);
              o16_7 = fma(eb, g7_0, o16_7);
            }
            { const double eb = bi[87];
              o16_6 = fma(eb, g6_1, o16_6);
              o16_7 = fma(eb, g7_1, o16_7);
            }
            { const double eb = bi[88];
              o16_6 = fma(eb, g6_3, o16_6);
              o16_7 = fma(eb, g7_3, o16_7);
            }
            { const double eb = bi[89];
              o16_6 = fma(eb, g6_7, o16_6);
              o16_7 = fma(eb, g7_7, o16_7);
            }
            { const double eb = bi[90];
              o17_6 = fma(eb, g6_0, o17_6);
              o17_7 = fma(eb, g7_0, o17_7);
            }
            { const double eb = bi[91];
              o17_6 = fma(eb, g6_1, o17_6);
              o17_7 = fma(eb, g7_1, o17_7);
            }
            { const double eb = bi[92];
              o17_6 = fma(eb, g6_3, o17_6);
              o17_7 = fma(eb, g7_3, o17_7);
            }
            { const double eb = bi[93];
              o17_6 = fma(eb, g6_7, o17_6);
              o17_7 = fma(eb, g7_7, o17_7);
            }
            { const double eb = bi[94];
              o17_6 = fma(eb, g6_9, o17_6);
              o17_7 = fma(eb, g7_9, o17_7);
            }
            { const double eb = bi[95];
              o17_6 = fma(eb, g6_17, o17_6);
              o17_7 = fma(eb, g7_17, o17_7);
            }
            { const double eb = bi[96];
              o18_6 = fma(eb, g6_0, o18_6);
              o18_7 = fma(eb, g7_0, o18_7);
            }
            { const double eb = bi[97];
              o18_6 = fma(eb, g6_1, o18_6);
              o18_7 = fma(eb, g7_1, o18_7);
            }
            { const double eb = bi[98];
              o18_6 = fma(eb, g6_2, o18_6);
              o18_7 = fma(eb, g7_2, o18_7);
            }
            { const double eb = bi[99];
              o18_6 = fma(eb, g6_5, o18_6);
              o18_7 = fma(eb, g7_5, o18_7);
            }
            { const double eb = bi[100];
              o18_6 = fma(eb, g6_3, o18_6);
              o18_7 = fma(eb, g7_3, o18_7);
            }
            { const double eb = bi[101];
              o18_6 = fma(eb, g6_7, o18_6);
              o18_7 = fma(eb, g7_7, o18_7);
            }
            { const double eb = bi[102];
              o18_6 = fma(eb, g6_8, o18_6);
              o18_7 = fma(eb, g7_8, o18_7);
            }
            { const double eb = bi[103];
              o18_6 = fma(eb, g6_15, o18_6);
              o18_7 = fma(eb, g7_15, o18_7);
            }
            { const double eb = bi[104];
              o19_6 = fma(eb, g6_0, o19_6);
              o19_7 = fma(eb, g7_0, o19_7);
            }
            { const double eb = bi[105];
              o19_6 = fma(eb, g6_1, o19_6);
              o19_7 = fma(eb, g7_1, o19_7);
            }
            { const double eb = bi[106];
              o19_6 = fma(eb, g6_4, o19_6);
              o19_7 = fma(eb, g7_4, o19_7);
            }
            { const double eb = bi[107];
              o19_6 = fma(eb, g6_3, o19_6);
              o19_7 = fma(eb, g7_3, o19_7);
            }
            { const double eb = bi[108];
              o19_6 = fma(eb, g6_7, o19_6);
              o19_7 = fma(eb, g7_7, o19_7);
            }
            { const double eb = bi[109];
              o19_6 = fma(eb, g6_14, o19_6);
              o19_7 = fma(eb, g7_14, o19_7);
            }
            { const double eb = bi[110];
              o20_6 = fma(eb, g6_0, o20_6);
              o20_7 = fma(eb, g7_0, o20_7);
            }
            { const double eb = bi[111];
              o20_6 = fma(eb, g6_1, o20_6);
              o20_7 = fma(eb, g7_1, o20_7);
            }
            { const double eb = bi[112];
              o20_6 = fma(eb, g6_2, o20_6);
              o20_7 = fma(eb, g7_2, o20_7);
            }
            { const double eb = bi[113];
              o20_6 = fma(eb, g6_5, o20_6);
              o20_7 = fma(eb, g7_5, o20_7);
            }
            { const double eb = bi[114];
              o21_6 = fma(eb, g6_0, o21_6);
              o21_7 = fma(eb, g7_0, o21_7);
            }
            { const double eb = bi[115];
              o21_6 = fma(eb, g6_1, o21_6);
              o21_7 = fma(eb, g7_1, o21_7);
            }
            { const double eb = bi[116];
              o21_6 = fma(eb, g6_2, o21_6);
              o21_7 = fma(eb, g7_2, o21_7);
            }
            { const double eb = bi[117];
              o21_6 = fma(eb, g6_5, o21_6);
              o21_7 = fma(eb, g7_5, o21_7);
            }
            { const double eb = bi[118];
              o21_6 = fma(eb, g6_3, o21_6);
              o21_7 = fma(eb, g7_3, o21_7);
            }
            { const double eb = bi[119];
              o21_6 = fma(eb, g6_7, o21_6);
              o21_7 = fma(eb, g7_7, o21_7);
            }
            { const double eb = bi[120];
              o21_6 = fma(eb, g6_8, o21_6);
              o21_7 = fma(eb, g7_8, o21_7);
            }
            { const double eb = bi[121];
              o21_6 = fma(eb, g6_15, o21_6);
              o21_7 = fma(eb, g7_15, o21_7);
            }
            { const double eb = bi[122];
              o22_6 = fma(eb, g6_0, o22_6);
              o22_7 = fma(eb, g7_0, o22_7);
            }
            { const double eb = bi[123];
              o22_6 = fma(eb, g6_1, o22_6);
              o22_7 = fma(eb, g7_1, o22_7);
            }
            { const double eb = bi[124];
              o22_6 = fma(eb, g6_2, o22_6);
              o22_7 = fma(eb, g7_2, o22_7);
            }
            { const double eb = bi[125];
              o22_6 = fma(eb, g6_5, o22_6);
              o22_7 = fma(eb, g7_5, o22_7);
            }
            { const double eb = bi[126];
              o22_6 = fma(eb, g6_6, o22_6);
              o22_7 = fma(eb, g7_6, o22_7);
            }
            { const double eb = bi[127];
              o22_6 = fma(eb, g6_12, o22_6);
              o22_7 = fma(eb, g7_12, o22_7);
            }
            { const double eb = bi[128];
              o23_6 = fma(eb, g6_0, o23_6);
              o23_7 = fma(eb, g7_0, o23_7);
            }
            { const double eb = bi[129];
              o23_6 = fma(eb, g6_1, o23_6);
              o23_7 = fma(eb, g7_1, o23_7);
            }
            { const double eb = bi[130];
              o23_6 = fma(eb, g6_4, o23_6);
              o23_7 = fma(eb, g7_4, o23_7);
            }
            { const double eb = bi[131];
              o23_6 = fma(eb, g6_2, o23_6);
              o23_7 = fma(eb, g7_2, o23_7);
            }
            { const double eb = bi[132];
              o23_6 = fma(eb, g6_5, o23_6);
              o23_7 = fma(eb, g7_5, o23_7);
            }
            { const double eb = bi[133];
              o23_6 = fma(eb, g6_11, o23_6);
              o23_7 = fma(eb, g7_11, o23_7);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk6 = PT[(fI + 1) * N + fJ + 2];
            const double ptk7 = PT[(fI + 1) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc3_1 = PA[(fQ + 3) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            jab0 += o0_6 * ptk6 + o0_7 * ptk7;
            jab1 += o1_6 * ptk6 + o1_7 * ptk7;
            jab2 += o2_6 * ptk6 + o2_7 * ptk7;
            jab3 += o3_6 * ptk6 + o3_7 * ptk7;
            jab4 += o4_6 * ptk6 + o4_7 * ptk7;
            jab5 += o5_6 * ptk6 + o5_7 * ptk7;
            jab6 += o6_6 * ptk6 + o6_7 * ptk7;
            jab7 += o7_6 * ptk6 + o7_7 * ptk7;
            jab8 += o8_6 * ptk6 + o8_7 * ptk7;
            jab9 += o9_6 * ptk6 + o9_7 * ptk7;
            jab10 += o10_6 * ptk6 + o10_7 * ptk7;
            jab11 += o11_6 * ptk6 + o11_7 * ptk7;
            jab12 += o12_6 * ptk6 + o12_7 * ptk7;
            jab13 += o13_6 * ptk6 + o13_7 * ptk7;
            jab14 += o14_6 * ptk6 + o14_7 * ptk7;
            jab15 += o15_6 * ptk6 + o15_7 * ptk7;
            jab16 += o16_6 * ptk6 + o16_7 * ptk7;
            jab17 += o17_6 * ptk6 + o17_7 * ptk7;
            jab18 += o18_6 * ptk6 + o18_7 * ptk7;
            jab19 += o19_6 * ptk6 + o19_7 * ptk7;
            jab20 += o20_6 * ptk6 + o20_7 * ptk7;
            jab21 += o21_6 * ptk6 + o21_7 * ptk7;
            jab22 += o22_6 * ptk6 + o22_7 * ptk7;
            jab23 += o23_6 * ptk6 + o23_7 * ptk7;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 2, 2.0 * deg * (o0_6 * ptb0 + o1_6 * ptb1 + o2_6 * ptb2 + o3_6 * ptb3 + o4_6 * ptb4 + o5_6 * ptb5 + o6_6 * ptb6 + o7_6 * ptb7 + o8_6 * ptb8 + o9_6 * ptb9 + o10_6 * ptb10 + o11_6 * ptb11 + o12_6 * ptb12 + o13_6 * ptb13 + o14_6 * ptb14 + o15_6 * ptb15 + o16_6 * ptb16 + o17_6 * ptb17 + o18_6 * ptb18 + o19_6 * ptb19 + o20_6 * ptb20 + o21_6 * ptb21 + o22_6 * ptb22 + o23_6 * ptb23));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 3, 2.0 * deg * (o0_7 * ptb0 + o1_7 * ptb1 + o2_7 * ptb2 + o3_7 * ptb3 + o4_7 * ptb4 + o5_7 * ptb5 + o6_7 * ptb6 + o7_7 * ptb7 + o8_7 * ptb8 + o9_7 * ptb9 + o10_7 * ptb10 + o11_7 * ptb11 + o12_7 * ptb12 + o13_7 * ptb13 + o14_7 * ptb14 + o15_7 * ptb15 + o16_7 * ptb16 + o17_7 * ptb17 + o18_7 * ptb18 + o19_7 * ptb19 + o20_7 * ptb20 + o21_7 * ptb21 + o22_7 * ptb22 + o23_7 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_6 * Abd0_2 + o0_7 * Abd0_3 + o1_6 * Abd1_2 + o1_7 * Abd1_3 + o2_6 * Abd2_2 + o2_7 * Abd2_3 + o3_6 * Abd3_2 + o3_7 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_6 * Aad0_2 + o0_7 * Aad0_3 + o4_6 * Aad1_2 + o4_7 * Aad1_3 + o8_6 * Aad2_2 + o8_7 * Aad2_3 + o12_6 * Aad3_2 + o12_7 * Aad3_3 + o16_6 * Aad4_2 + o16_7 * Aad4_3 + o20_6 * Aad5_2 + o20_7 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_6 * Abc0_1 + o1_6 * Abc1_1 + o2_6 * Abc2_1 + o3_6 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_6 * Aac0_1 + o4_6 * Aac1_1 + o8_6 * Aac2_1 + o12_6 * Aac3_1 + o16_6 * Aac4_1 + o20_6 * Aac5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_7 * Abc0_1 + o1_7 * Abc1_1 + o2_7 * Abc2_1 + o3_7 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_7 * Aac0_1 + o4_7 * Aac1_1 + o8_7 * Aac2_1 + o12_7 * Aac3_1 + o16_7 * Aac4_1 + o20_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_6 * Aad0_2 + o1_7 * Aad0_3 + o5_6 * Aad1_2 + o5_7 * Aad1_3 + o9_6 * Aad2_2 + o9_7 * Aad2_3 + o13_6 * Aad3_2 + o13_7 * Aad3_3 + o17_6 * Aad4_2 + o17_7 * Aad4_3 + o21_6 * Aad5_2 + o21_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_6 * Aac0_1 + o5_6 * Aac1_1 + o9_6 * Aac2_1 + o13_6 * Aac3_1 + o17_6 * Aac4_1 + o21_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_7 * Aac0_1 + o5_7 * Aac1_1 + o9_7 * Aac2_1 + o13_7 * Aac3_1 + o17_7 * Aac4_1 + o21_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_6 * Aad0_2 + o2_7 * Aad0_3 + o6_6 * Aad1_2 + o6_7 * Aad1_3 + o10_6 * Aad2_2 + o10_7 * Aad2_3 + o14_6 * Aad3_2 + o14_7 * Aad3_3 + o18_6 * Aad4_2 + o18_7 * Aad4_3 + o22_6 * Aad5_2 + o22_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_6 * Aac0_1 + o6_6 * Aac1_1 + o10_6 * Aac2_1 + o14_6 * Aac3_1 + o18_6 * Aac4_1 + o22_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_7 * Aac0_1 + o6_7 * Aac1_1 + o10_7 * Aac2_1 + o14_7 * Aac3_1 + o18_7 * Aac4_1 + o22_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_6 * Aad0_2 + o3_7 * Aad0_3 + o7_6 * Aad1_2 + o7_7 * Aad1_3 + o11_6 * Aad2_2 + o11_7 * Aad2_3 + o15_6 * Aad3_2 + o15_7 * Aad3_3 + o19_6 * Aad4_2 + o19_7 * Aad4_3 + o23_6 * Aad5_2 + o23_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_6 * Aac0_1 + o7_6 * Aac1_1 + o11_6 * Aac2_1 + o15_6 * Aac3_1 + o19_6 * Aac4_1 + o23_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_7 * Aac0_1 + o7_7 * Aac1_1 + o11_7 * Aac2_1 + o15_7 * Aac3_1 + o19_7 * Aac4_1 + o23_7 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_6 * Abd0_2 + o4_7 * Abd0_3 + o5_6 * Abd1_2 + o5_7 * Abd1_3 + o6_6 * Abd2_2 + o6_7 * Abd2_3 + o7_6 * Abd3_2 + o7_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_6 * Abc0_1 + o5_6 * Abc1_1 + o6_6 * Abc2_1 + o7_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_7 * Abc0_1 + o5_7 * Abc1_1 + o6_7 * Abc2_1 + o7_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_6 * Abd0_2 + o8_7 * Abd0_3 + o9_6 * Abd1_2 + o9_7 * Abd1_3 + o10_6 * Abd2_2 + o10_7 * Abd2_3 + o11_6 * Abd3_2 + o11_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_6 * Abc0_1 + o9_6 * Abc1_1 + o10_6 * Abc2_1 + o11_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_7 * Abc0_1 + o9_7 * Abc1_1 + o10_7 * Abc2_1 + o11_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_6 * Abd0_2 + o12_7 * Abd0_3 + o13_6 * Abd1_2 + o13_7 * Abd1_3 + o14_6 * Abd2_2 + o14_7 * Abd2_3 + o15_6 * Abd3_2 + o15_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_6 * Abc0_1 + o13_6 * Abc1_1 + o14_6 * Abc2_1 + o15_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_7 * Abc0_1 + o13_7 * Abc1_1 + o14_7 * Abc2_1 + o15_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_6 * Abd0_2 + o16_7 * Abd0_3 + o17_6 * Abd1_2 + o17_7 * Abd1_3 + o18_6 * Abd2_2 + o18_7 * Abd2_3 + o19_6 * Abd3_2 + o19_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_6 * Abc0_1 + o17_6 * Abc1_1 + o18_6 * Abc2_1 + o19_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_7 * Abc0_1 + o17_7 * Abc1_1 + o18_7 * Abc2_1 + o19_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_6 * Abd0_2 + o20_7 * Abd0_3 + o21_6 * Abd1_2 + o21_7 * Abd1_3 + o22_6 * Abd2_2 + o22_7 * Abd2_3 + o23_6 * Abd3_2 + o23_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_6 * Abc0_1 + o21_6 * Abc1_1 + o22_6 * Abc2_1 + o23_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_7 * Abc0_1 + o21_7 * Abc1_1 + o22_7 * Abc2_1 + o23_7 * Abc3_1));
          }
        } break;
        case 4: {  // ket functions [8, 9]
          double o0_8 = 0;
          double o0_9 = 0;
          double o1_8 = 0;
          double o1_9 = 0;
          double o2_8 = 0;
          double o2_9 = 0;
          double o3_8 = 0;
          double o3_9 = 0;
          double o4_8 = 0;
          double o4_9 = 0;
          double o5_8 = 0;
          double o5_9 = 0;
          double o6_8 = 0;
          double o6_9 = 0;
          double o7_8 = 0;
          double o7_9 = 0;
          double o8_8 = 0;
          double o8_9 = 0;
          double o9_8 = 0;
          double o9_9 = 0;
          double o10_8 = 0;
          double o10_9 = 0;
          double o11_8 = 0;
          double o11_9 = 0;
          double o12_8 = 0;
          double o12_9 = 0;
          double o13_8 = 0;
          double o13_9 = 0;
          double o14_8 = 0;
          double o14_9 = 0;
          double o15_8 = 0;
          double o15_9 = 0;
          double o16_8 = 0;
          double o16_9 = 0;
          double o17_8 = 0;
          double o17_9 = 0;
          double o18_8 = 0;
          double o18_9 = 0;
          double o19_8 = 0;
          double o19_9 = 0;
          double o20_8 = 0;
          double o20_9 = 0;
          double o21_8 = 0;
          double o21_9 = 0;
          double o22_8 = 0;
          double o22_9 = 0;
          double o23_8 = 0;
          double o23_9 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek8_0 = kj[43 * kS];
              const double ek8_1 = -kj[44 * kS];
              const double ek8_2 = kj[45 * kS];
              const double ek9_0 = kj[46 * kS];
              const double ek9_1 = -kj[47 * kS];
              const double ek9_2 = kj[48 * kS];
              const double ek9_3 = -kj[49 * kS];
              const double ek9_4 = kj[50 * kS];
              const double ek9_5 = -kj[51 * kS];
              g8_0 = fma(ek8_0, b0, g8_0);
              g9_0 = fma(ek9_0, b0, g9_0);
              const double r0_0_0_1 = Z * b1;
              g8_1 = fma(ek8_0, r0_0_0_1, g8_1);
              g8_0 = fma(ek8_1, r0_0_0_1, g8_0);
              g9_1 = fma(ek9_0, r0_0_0_1, g9_1);
              g9_0 = fma(ek9_1, r0_0_0_1, g9_0);
              const double r0_0_1_0 = Y * b1;
              g8_2 = fma(ek8_0, r0_0_1_0, g8_2);
              g9_2 = fma(ek9_0, r0_0_1_0, g9_2);
              const double r0_1_0_0 = X * b1;
              g8_3 = fma(ek8_0, r0_1_0_0, g8_3);
              g9_3 = fma(ek9_0, r0_1_0_0, g9_3);
              g9_0 = fma(ek9_3, r0_1_0_0, g9_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g8_4 = fma(ek8_0, r0_0_0_2, g8_4);
              g8_1 = fma(ek8_1, r0_0_0_2, g8_1);
              g8_0 = fma(ek8_2, r0_0_0_2, g8_0);
              g9_4 = fma(ek9_0, r0_0_0_2, g9_4);
              g9_1 = fma(ek9_1, r0_0_0_2, g9_1);
              g9_0 = fma(ek9_2, r0_0_0_2, g9_0);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g8_5 = fma(ek8_0, r0_0_1_1, g8_5);
              g8_2 = fma(ek8_1, r0_0_1_1, g8_2);
              g9_5 = fma(ek9_0, r0_0_1_1, g9_5);
              g9_2 = fma(ek9_1, r0_0_1_1, g9_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g8_6 = fma(ek8_0, r0_0_2_0, g8_6);
              g9_6 = fma(ek9_0, r0_0_2_0, g9_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g8_7 = fma(ek8_0, r0_1_0_1, g8_7);
              g8_3 = fma(ek8_1, r0_1_0_1, g8_3);
              g9_7 = fma(ek9_0, r0_1_0_1, g9_7);
              g9_3 = fma(ek9_1, r0_1_0_1, g9_3);
              g9_1 = fma(ek9_3, r0_1_0_1, g9_1);
              g9_0 = fma(ek9_4, r0_1_0_1, g9_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g8_8 = fma(ek8_0, r0_1_1_0, g8_8);
              g9_8 = fma(ek9_0, r0_1_1_0, g9_8);
              g9_2 = fma(ek9_3, r0_1_1_0, g9_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g8_9 = fma(ek8_0, r0_2_0_0, g8_9);
              g9_9 = fma(ek9_0, r0_2_0_0, g9_9);
              g9_3 = fma(ek9_3, r0_2_0_0, g9_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g8_10 = fma(ek8_0, r0_0_0_3, g8_10);
              g8_4 = fma(ek8_1, r0_0_0_3, g8_4);
              g8_1 = fma(ek8_2, r0_0_0_3, g8_1);
              g9_10 = fma(ek9_0, r0_0_0_3, g9_10);
              g9_4 = fma(ek9_1, r0_0_0_3, g9_4);
              g9_1 = fma(ek9_2, r0_0_0_3, g9_1);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g8_11 = fma(ek8_0, r0_0_1_2, g8_11);
              g8_5 = fma(ek8_1, r0_0_1_2, g8_5);
              g8_2 = fma(ek8_2, r0_0_1_2, g8_2);
              g9_11 = fma(ek9_0, r0_0_1_2, g9_11);
              g9_5 = fma(ek9_1, r0_0_1_2, g9_5);
              g9_2 = fma(ek9_2, r0_0_1_2, g9_2);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g8_12 = fma(ek8_0, r0_0_2_1, g8_12);
              g8_6 = fma(ek8_1, r0_0_2_1, g8_6);
              g9_12 = fma(ek9_0, r0_0_2_1, g9_12);
              g9_6 = fma(ek9_1, r0_0_2_1, g9_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g8_13 = fma(ek8_0, r0_0_3_0, g8_13);
              g9_13 = fma(ek9_0, r0_0_3_0, g9_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g8_14 = fma(ek8_0, r0_1_0_2, g8_14);
              g8_7 = fma(ek8_1, r0_1_0_2, g8_7);
              g8_3 = fma(ek8_2, r0_1_0_2, g8_3);
              g9_14 = fma(ek9_0, r0_1_0_2, g9_14);
              g9_7 = fma(ek9_1, r0_1_0_2, g9_7);
              g9_3 = fma(ek9_2, r0_1_0_2, g9_3);
              g9_4 = fma(ek9_3, r0_1_0_2, g9_4);
              g9_1 = fma(ek9_4, r0_1_0_2, g9_1);
              g9_0 = fma(ek9_5, r0_1_0_2, g9_0);
              const double r0_1_1_1 = X * r1_0_1_1;
              g8_15 = fma(ek8_0, r0_1_1_1, g8_15);
              g8_8 = fma(ek8_1, r0_1_1_1, g8_8);
              g9_15 = fma(ek9_0, r0_1_1_1, g9_15);
              g9_8 = fma(ek9_1, r0_1_1_1, g9_8);
              g9_5 = fma(ek9_3, r0_1_1_1, g9_5);
              g9_2 = fma(ek9_4, r0_1_1_1, g9_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g8_16 = fma(ek8_0, r0_1_2_0, g8_16);
              g9_16 = fma(ek9_0, r0_1_2_0, g9_16);
              g9_6 = fma(ek9_3, r0_1_2_0, g9_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g8_17 = fma(ek8_0, r0_2_0_1, g8_17);
              g8_9 = fma(ek8_1, r0_2_0_1, g8_9);
              g9_17 = fma(ek9_0, r0_2_0_1, g9_17);
              g9_9 = fma(ek9_1, r0_2_0_1, g9_9);
              g9_7 = fma(ek9_3, r0_2_0_1, g9_7);
              g9_3 = fma(ek9_4, r0_2_0_1, g9_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g8_18 = fma(ek8_0, r0_2_1_0, g8_18);
              g9_18 = fma(ek9_0, r0_2_1_0, g9_18);
              g9_8 = fma(ek9_3, r0_2_1_0, g9_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g8_19 = fma(ek8_0, r0_3_0_0, g8_19);
              g9_19 = fma(ek9_0, r0_3_0_0, g9_19);
              g9_9 = fma(ek9_3, r0_3_0_0, g9_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g8_10 = fma(ek8_1, r0_0_0_4, g8_10);
              g8_4 = fma(ek8_2, r0_0_0_4, g8_4);
              g9_10 = fma(ek9_1, r0_0_0_4, g9_10);
              g9_4 = fma(ek9_2, r0_0_0_4, g9_4);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g8_11 = fma(ek8_1, r0_0_1_3, g8_11);
              g8_5 = fma(ek8_2, r0_0_1_3, g8_5);
              g9_11 = fma(ek9_1, r0_0_1_3, g9_11);
              g9_5 = fma(ek9_2, r0_0_1_3, g9_5);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g8_12 = fma(ek8_1, r0_0_2_2, g8_12);
              g8_6 = fma(ek8_2, r0_0_2_2, g8_6);
              g9_12 = fma(ek9_1, r0_0_2_2, g9_12);
              g9_6 = fma(ek9_2, r0_0_2_2, g9_6);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g8_13 = fma(ek8_1, r0_0_3_1, g8_13);
              g9_13 = fma(ek9_1, r0_0_3_1, g9_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g8_14 = fma(ek8_1, r0_1_0_3, g8_14);
              g8_7 = fma(ek8_2, r0_1_0_3, g8_7);
              g9_14 = fma(ek9_1, r0_1_0_3, g9_14);
              g9_7 = fma(ek9_2, r0_1_0_3, g9_7);
              g9_10 = fma(ek9_3, r0_1_0_3, g9_10);
              g9_4 = fma(ek9_4, r0_1_0_3, g9_4);
              g9_1 = fma(ek9_5, r0_1_0_3, g9_1);
              const double r0_1_1_2 = X * r1_0_1_2;
              g8_15 = fma(ek8_1, r0_1_1_2, g8_15);
              g8_8 = fma(ek8_2, r0_1_1_2, g8_8);
              g9_15 = fma(ek9_1, r0_1_1_2, g9_15);
              g9_8 = fma(ek9_2, r0_1_1_2, g9_8);
              g9_11 = fma(ek9_3, r0_1_1_2, g9_11);
              g9_5 = fma(ek9_4, r0_1_1_2, g9_5);
              g9_2 = fma(ek9_5, r0_1_1_2, g9_2);
              const double r0_1_2_1 = X * r1_0_2_1;
              g8_16 = fma(ek8_1, r0_1_2_1, g8_16);
              g9_16 = fma(ek9_1, r0_1_2_1, g9_16);
              g9_12 = fma(ek9_3, r0_1_2_1, g9_12);
              g9_6 = fma(ek9_4, r0_1_2_1, g9_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g9_13 = fma(ek9_3, r0_1_3_0, g9_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g8_17 = fma(ek8_1, r0_2_0_2, g8_17);
              g8_9 = fma(ek8_2, r0_2_0_2, g8_9);
              g9_17 = fma(ek9_1, r0_2_0_2, g9_17);
              g9_9 = fma(ek9_2, r0_2_0_2, g9_9);
              g9_14 = fma(ek9_3, r0_2_0_2, g9_14);
              g9_7 = fma(ek9_4, r0_2_0_2, g9_7);
              g9_3 = fma(ek9_5, r0_2_0_2, g9_3);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g8_18 = fma(ek8_1, r0_2_1_1, g8_18);
              g9_18 = fma(ek9_1, r0_2_1_1, g9_18);
              g9_15 = fma(ek9_3, r0_2_1_1, g9_15);
              g9_8 = fma(ek9_4, r0_2_1_1, g9_8);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g9_16 = fma(ek9_3, r0_2_2_0, g9_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g8_19 = fma(ek8_1, r0_3_0_1, g8_19);
              g9_19 = fma(ek9_1, r0_3_0_1, g9_19);
              g9_17 = fma(ek9_3, r0_3_0_1, g9_17);
              g9_9 = fma(ek9_4, r0_3_0_1, g9_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g9_18 = fma(ek9_3, r0_3_1_0, g9_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g9_19 = fma(ek9_3, r0_4_0_0, g9_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g8_10 = fma(ek8_2, r0_0_0_5, g8_10);
              g9_10 = fma(ek9_2, r0_0_0_5, g9_10);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g8_11 = fma(ek8_2, r0_0_1_4, g8_11);
              g9_11 = fma(ek9_2, r0_0_1_4, g9_11);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g8_12 = fma(ek8_2, r0_0_2_3, g8_12);
              g9_12 = fma(ek9_2, r0_0_2_3, g9_12);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g8_13 = fma(ek8_2, r0_0_3_2, g8_13);
              g9_13 = fma(ek9_2, r0_0_3_2, g9_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g8_14 = fma(ek8_2, r0_1_0_4, g8_14);
              g9_14 = fma(ek9_2, r0_1_0_4, g9_14);
              g9_10 = fma(ek9_4, r0_1_0_4, g9_10);
              g9_4 = fma(ek9_5, r0_1_0_4, g9_4);
              const double r0_1_1_3 = X * r1_0_1_3;
              g8_15 = fma(ek8_2, r0_1_1_3, g8_15);
              g9_15 = fma(ek9_2, r0_1_1_3, g9_15);
              g9_11 = fma(ek9_4, r0_1_1_3, g9_11);
              g9_5 = fma(ek9_5, r0_1_1_3, g9_5);
              const double r0_1_2_2 = X * r1_0_2_2;
              g8_16 = fma(ek8_2, r0_1_2_2, g8_16);
              g9_16 = fma(ek9_2, r0_1_2_2, g9_16);
              g9_12 = fma(ek9_4, r0_1_2_2, g9_12);
              g9_6 = fma(ek9_5, r0_1_2_2, g9_6);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g9_13 = fma(ek9_4, r0_1_3_1, g9_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g8_17 = fma(ek8_2, r0_2_0_3, g8_17);
              g9_17 = fma(ek9_2, r0_2_0_3, g9_17);
              g9_14 = fma(ek9_4, r0_2_0_3, g9_14);
              g9_7 = fma(ek9_5, r0_2_0_3, g9_7);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g8_18 = fma(ek8_2, r0_2_1_2, g8_18);
              g9_18 = fma(ek9_2, r0_2_1_2, g9_18);
              g9_15 = fma(ek9_4, r0_2_1_2, g9_15);
              g9_8 = fma(ek9_5, r0_2_1_2, g9_8);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g9_16 = fma(ek9_4, r0_2_2_1, g9_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g8_19 = fma(ek8_2, r0_3_0_2, g8_19);
              g9_19 = fma(ek9_2, r0_3_0_2, g9_19);
              g9_17 = fma(ek9_4, r0_3_0_2, g9_17);
              g9_9 = fma(ek9_5, r0_3_0_2, g9_9);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g9_18 = fma(ek9_4, r0_3_1_1, g9_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g9_19 = fma(ek9_4, r0_4_0_1, g9_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_1_0_5 = X * r1_0_0_5;
              g9_10 = fma(ek9_5, r0_1_0_5, g9_10);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_1_1_4 = X * r1_0_1_4;
              g9_11 = fma(ek9_5, r0_1_1_4, g9_11);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g9_12 = fma(ek9_5, r0_1_2_3, g9_12);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g9_13 = fma(ek9_5, r0_1_3_2, g9_13);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g9_14 = fma(ek9_5, r0_2_0_4, g9_14);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g9_15 = fma(ek9_5, r0_2_1_3, g9_15);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g9_16 = fma(ek9_5, r0_2_2_2, g9_16);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g9_17 = fma(ek9_5, r0_3_0_3, g9_17);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g9_18 = fma(ek9_5, r0_3_1_2, g9_18);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g9_19 = fma(ek9_5, r0_4_0_2, g9_19);
            }
            { const double eb = bi[5];
              o0_8 = fma(eb, g8_0, o0_8);
              o0_9 = fma(eb, g9_0, o0_9);
            }
            { const double eb = bi[6];
              o0_8 = fma(eb, g8_3, o0_8);
              o0_9 = fma(eb, g9_3, o0_9);
            }
            { const double eb = bi[7];
              o0_8 = fma(eb, g8_9, o0_8);
              o0_9 = fma(eb, g9_9, o0_9);
            }
            { const double eb = bi[8];
              o1_8 = fma(eb, g8_0, o1_8);
              o1_9 = fma(eb, g9_0, o1_9);
            }
            { const double eb = bi[9];
              o1_8 = fma(eb, g8_3, o1_8);
              o1_9 = fma(eb, g9_3, o1_9);
            }
            { const double eb = bi[10];
              o1_8 = fma(eb, g8_9, o1_8);
              o1_9 = fma(eb, g9_9, o1_9);
            }
            { const double eb = bi[11];
              o1_8 = fma(eb, g8_19, o1_8);
              o1_9 = fma(eb, g9_19, o1_9);
            }
            { const double eb = bi[12];
              o2_8 = fma(eb, g8_0, o2_8);
              o2_9 = fma(eb, g9_0, o2_9);
            }
            { const double eb = bi[13];
              o2_8 = fma(eb, g8_2, o2_8);
              o2_9 = fma(eb, g9_2, o2_9);
            }
            { const double eb = bi[14];
              o2_8 = fma(eb, g8_3, o2_8);
              o2_9 = fma(eb, g9_3, o2_9);
            }
            { const double eb = bi[15];
              o2_8 = fma(eb, g8_8, o2_8);
              o2_9 = fma(eb, g9_8, o2_9);
            }
            { const double eb = bi[16];
              o2_8 = fma(eb, g8_9, o2_8);
              o2_9 = fma(eb, g9_9, o2_9);
            }
            { const double eb = bi[17];
              o2_8 = fma(eb, g8_18, o2_8);
              o2_9 = fma(eb, g9_18, o2_9);
            }
            { const double eb = bi[18];
              o3_8 = fma(eb, g8_0, o3_8);
              o3_9 = fma(eb, g9_0, o3_9);
            }
            { const double eb = bi[19];
              o3_8 = fma(eb, g8_1, o3_8);
              o3_9 = fma(eb, g9_1, o3_9);
            }
            { const double eb = bi[20];
              o3_8 = fma(eb, g8_3, o3_8);
              o3_9 = fma(eb, g9_3, o3_9);
            }
            { const double eb = bi[21];
              o3_8 = fma(eb, g8_7, o3_8);
              o3_9 = fma(eb, g9_7, o3_9);
            }
            { const double eb = bi[22];
              o3_8 = fma(eb, g8_9, o3_8);
              o3_9 = fma(eb, g9_9, o3_9);
            }
            { const double eb = bi[23];
              o3_8 = fma(eb, g8_17, o3_8);
              o3_9 = fma(eb, g9_17, o3_9);
            }
            { const double eb = bi[24];
              o4_8 = fma(eb, g8_0, o4_8);
              o4_9 = fma(eb, g9_0, o4_9);
            }
            { const double eb = bi[25];
              o4_8 = fma(eb, g8_2, o4_8);
              o4_9 = fma(eb, g9_2, o4_9);
            }
            { const double eb = bi[26];
              o4_8 = fma(eb, g8_6, o4_8);
              o4_9 = fma(eb, g9_6, o4_9);
            }
            { const double eb = bi[27];
              o5_8 = fma(eb, g8_0, o5_8);
              o5_9 = fma(eb, g9_0, o5_9);
            }
            { const double eb = bi[28];
              o5_8 = fma(eb, g8_2, o5_8);
              o5_9 = fma(eb, g9_2, o5_9);
            }
            { const double eb = bi[29];
              o5_8 = fma(eb, g8_6, o5_8);
              o5_9 = fma(eb, g9_6, o5_9);
            }
            { const double eb = bi[30];
              o5_8 = fma(eb, g8_3, o5_8);
              o5_9 = fma(eb, g9_3, o5_9);
            }
            { const double eb = bi[31];
              o5_8 = fma(eb, g8_8, o5_8);
              o5_9 = fma(eb, g9_8, o5_9);
            }
            { const double eb = bi[32];
              o5_8 = fma(eb, g8_16, o5_8);
              o5_9 = fma(eb, g9_16, o5_9);
            }
            { const double eb = bi[33];
              o6_8 = fma(eb, g8_0, o6_8);
              o6_9 = fma(eb, g9_0, o6_9);
            }
            { const double eb = bi[34];
              o6_8 = fma(eb, g8_2, o6_8);
              o6_9 = fma(eb, g9_2, o6_9);
            }
            { const double eb = bi[35];
              o6_8 = fma(eb, g8_6, o6_8);
              o6_9 = fma(eb, g9_6, o6_9);
            }
            { const double eb = bi[36];
              o6_8 = fma(eb, g8_13, o6_8);
              o6_9 = fma(eb, g9_13, o6_9);
            }
            { const double eb = bi[37];
              o7_8 = fma(eb, g8_0, o7_8);
              o7_9 = fma(eb, g9_0, o7_9);
            }
            { const double eb = bi[38];
              o7_8 = fma(eb, g8_1, o7_8);
              o7_9 = fma(eb, g9_1, o7_9);
            }
            { const double eb = bi[39];
              o7_8 = fma(eb, g8_2, o7_8);
              o7_9 = fma(eb, g9_2, o7_9);
            }
            { const double eb = bi[40];
              o7_8 = fma(eb, g8_5, o7_8);
              o7_9 = fma(eb, g9_5, o7_9);
            }
            { const double eb = bi[41];
              o7_8 = fma(eb, g8_6, o7_8);
              o7_9 = fma(eb, g9_6, o7_9);
            }
            { const double eb = bi[42];
              o7_8 = fma(eb, g8_12, o7_8);
              o7_9 = fma(eb, g9_12, o7_9);
            }
            { const double eb = bi[43];
              o8_8 = fma(eb, g8_0, o8_8);
              o8_9 = fma(eb, g9_0, o8_9);
            }
            { const double eb = bi[44];
              o8_8 = fma(eb, g8_1, o8_8);
              o8_9 = fma(eb, g9_1, o8_9);
            }
            { const double eb = bi[45];
              o8_8 = fma(eb, g8_4, o8_8);
              o8_9 = fma(eb, g9_4, o8_9);
            }
            { const double eb = bi[46];
              o9_8 = fma(eb, g8_0, o9_8);
              o9_9 = fma(eb, g9_0, o9_9);
            }
            { const double eb = bi[47];
              o9_8 = fma(eb, g8_1, o9_8);
              o9_9 = fma(eb, g9_1, o9_9);
            }
            { const double eb = bi[48];
              o9_8 = fma(eb, g8_4, o9_8);
              o9_9 = fma(eb, g9_4, o9_9);
            }
            { const double eb = bi[49];
              o9_8 = fma(eb, g8_3, o9_8);
              o9_9 = fma(eb, g9_3, o9_9);
            }
            { const double eb = bi[50];
              o9_8 = fma(eb, g8_7, o9_8);
              o9_9 = fma(eb, g9_7, o9_9);
            }
            { const double eb = bi[51];
              o9_8 = fma(eb, g8_14, o9_8);
              o9_9 = fma(eb, g9_14, o9_9);
            }
            { const double eb = bi[52];
              o10_8 = fma(eb, g8_0, o10_8);
              o10_9 = fma(eb, g9_0, o10_9);
            }
            { const double eb = bi[53];
              o10_8 = fma(eb, g8_1, o10_8);
              o10_9 = fma(eb, g9_1, o10_9);
            }
            { const double eb = bi[54];
              o10_8 = fma(eb, g8_4, o10_8);
              o10_9 = fma(eb, g9_4, o10_9);
            }
            { const double eb = bi[55];
              o10_8 = fma(eb, g8_2, o10_8);
              o10_9 = fma(eb, g9_2, o10_9);
            }
            { const double eb = bi[56];
              o10_8 = fma(eb, g8_5, o10_8);
              o10_9 = fma(eb, g9_5, o10_9);
            }
            { const double eb = bi[57];
              o10_8 = fma(eb, g8_11, o10_8);
              o10_9 = fma(eb, g9_11, o10_9);
            }
            { const double eb = bi[58];
              o11_8 = fma(eb, g8_0, o11_8);
              o11_9 = fma(eb, g9_0, o11_9);
            }
            { const double eb = bi[59];
              o11_8 = fma(eb, g8_1, o11_8);
              o11_9 = fma(eb, g9_1, o11_9);
            }
            { const double eb = bi[60];
              o11_8 = fma(eb, g8_4, o11_8);
              o11_9 = fma(eb, g9_4, o11_9);
            }
            { const double eb = bi[61];
              o11_8 = fma(eb, g8_10, o11_8);
              o11_9 = fma(eb, g9_10, o11_9);
            }
            { const double eb = bi[62];
              o12_8 = fma(eb, g8_0, o12_8);
              o12_9 = fma(eb, g9_0, o12_9);
            }
            { const double eb = bi[63];
              o12_8 = fma(eb, g8_2, o12_8);
              o12_9 = fma(eb, g9_2, o12_9);
            }
            { const double eb = bi[64];
              o12_8 = fma(eb, g8_3, o12_8);
              o12_9 = fma(eb, g9_3, o12_9);
            }
            { const double eb = bi[65];
              o12_8 = fma(eb, g8_8, o12_8);
              o12_9 = fma(eb, g9_8, o12_9);
            }
            { const double eb = bi[66];
              o13_8 = fma(eb, g8_0, o13_8);
              o13_9 = fma(eb, g9_0, o13_9);
            }
            { const double eb = bi[67];
              o13_8 = fma(eb, g8_2, o13_8);
              o13_9 = fma(eb, g9_2, o13_9);
            }
            { const double eb = bi[68];
              o13_8 = fma(eb, g8_3, o13_8);
              o13_9 = fma(eb, g9_3, o13_9);
            }
            { const double eb = bi[69];
              o13_8 = fma(eb, g8_8, o13_8);
              o13_9 = fma(eb, g9_8, o13_9);
            }
            { const double eb = bi[70];
              o13_8 = fma(eb, g8_9, o13_8);
              o13_9 = fma(eb, g9_9, o13_9);
            }
            { const double eb = bi[71];
              o13_8 = fma(eb, g8_18, o13_8);
              o13_9 = fma(eb, g9_18, o13_9);
            }
            { const double eb = bi[72];
              o14_8 = fma(eb, g8_0, o14_8);
              o14_9 = fma(eb, g9_0, o14_9);
            }
            { const double eb = bi[73];
              o14_8 = fma(eb, g8_2, o14_8);
              o14_9 = fma(eb, g9_2, o14_9);
            }
            { const double eb = bi[74];
              o14_8 = fma(eb, g8_6, o14_8);
              o14_9 = fma(eb, g9_6, o14_9);
            }
            { const double eb = bi[75];
              o14_8 = fma(eb, g8_3, o14_8);
              o14_9 = fma(eb, g9_3, o14_9);
            }
            { const double eb = bi[76];
              o14_8 = fma(eb, g8_8, o14_8);
              o14_9 = fma(eb, g9_8, o14_9);
            }
            { const double eb = bi[77];
              o14_8 = fma(eb, g8_16, o14_8);
              o14_9 = fma(eb, g9_16, o14_9);
            }
            { const double eb = bi[78];
              o15_8 = fma(eb, g8_0, o15_8);
              o15_9 = fma(eb, g9_0, o15_9);
            }
            { const double eb = bi[79];
              o15_8 = fma(eb, g8_1, o15_8);
              o15_9 = fma(eb, g9_1, o15_9);
            }
            { const double eb = bi[80];
              o15_8 = fma(eb, g8_2, o15_8);
              o15_9 = fma(eb, g9_2, o15_9);
            }
            { const double eb = bi[81];
              o15_8 = fma(eb, g8_5, o15_8);
              o15_9 = fma(eb, g9_5, o15_9);
            }
            { const double eb = bi[82];
              o15_8 = fma(eb, g8_3, o15_8);
              o15_9 = fma(eb, g9_3, o15_9);
            }
            { const double eb = bi[83];
              o15_8 = fma(eb, g8_7, o15_8);
              o15_9 = fma(eb, g9_7, o15_9);
            }
            { const double eb = bi[84];
              o15_8 = fma(eb, g8_8, o15_8);
              o15_9 = fma(eb, g9_8, o15_9);
            }
            { const double eb = bi[85];
              o15_8 = fma(eb, g8_15, o15_8);
              o15_9 = fma(eb, g9_15, o15_9);
            }
            { const double eb = bi[86];
              o16_8 = fma(eb, g8_0, o16_8);
              o16_9 = fma(eb, g9_0, o16_9);
            }
            { const double eb = bi[87];
              o16_8 = fma(eb, g8_1, o16_8);
              o16_9 = fma(eb, g9_1, o16_9);
            }
            { const double eb = bi[88];
              o16_8 = fma(eb, g8_3, o16_8);
              o16_9 = fma(eb, g9_3, o16_9);
            }
            { const double eb = bi[89];
              o16_8 = fma(eb, g8_7, o16_8);
              o16_9 = fma(eb, g9_7, o16_9);
            }
            { const double eb = bi[90];
              o17_8 = fma(eb, g8_0, o17_8);
              o17_9 = fma(eb, g9_0, o17_9);
            }
            { const double eb = bi[91];
              o17_8 = fma(eb, g8_1, o17_8);
              o17_9 = fma(eb, g9_1, o17_9);
            }
            { const double eb = bi[92];
              o17_8 = fma(eb, g8_3, o17_8);
              o17_9 = fma(eb, g9_3, o17_9);
            }
            { const double eb = bi[93];
              o17_8 = fma(eb, g8_7, o17_8);
              o17_9 = fma(eb, g9_7, o17_9);
            }
            { const double eb = bi[94];
              o17_8 = fma(eb, g8_9, o17_8);
              o17_9 = fma(eb, g9_9, o17_9);
            }
            { const double eb = bi[95];
              o17_8 = fma(eb, g8_17, o17_8);
              o17_9 = fma(eb, g9_17, o17_9);
            }
            { const double eb = bi[96];
              o18_8 = fma(eb, g8_0, o18_8);
              o18_9 = fma(eb, g9_0, o18_9);
            }
            { const double eb = bi[97];
              o18_8 = fma(eb, g8_1, o18_8);
              o18_9 = fma(eb, g9_1, o18_9);
            }
            { const double eb = bi[98];
              o18_8 = fma(eb, g8_2, o18_8);
              o18_9 = fma(eb, g9_2, o18_9);
            }
            { const double eb = bi[99];
              o18_8 = fma(eb, g8_5, o18_8);
              o18_9 = fma(eb, g9_5, o18_9);
            }
            { const double eb = bi[100];
              o18_8 = fma(eb, g8_3, o18_8);
              o18_9 = fma(eb, g9_3, o18_9);
            }
            { const double eb = bi[101];
              o18_8 = fma(eb, g8_7, o18_8);
              o18_9 = fma(eb, g9_7, o18_9);
            }
            { const double eb = bi[102];
              o18_8 = fma(eb, g8_8, o18_8);
              o18_9 = fma(eb, g9_8, o18_9);
            }
            { const double eb = bi[103];
              o18_8 = fma(eb, g8_15, o18_8);
              o18_9 = fma(eb, g9_15, o18_9);
            }
            { const double eb = bi[104];
              o19_8 = fma(eb, g8_0, o19_8);
              o19_9 = fma(eb, g9_0, o19_9);
            }
            { const double eb = bi[105];
              o19_8 = fma(eb, g8_1, o19_8);
              o19_9 = fma(eb, g9_1, o19_9);
            }
            { const double eb = bi[106];
              o19_8 = fma(eb, g8_4, o19_8);
              o19_9 = fma(eb, g9_4, o19_9);
            }
            { const double eb = bi[107];
              o19_8 = fma(eb, g8_3, o19_8);
              o19_9 = fma(eb, g9_3, o19_9);
            }
            { const double eb = bi[108];
              o19_8 = fma(eb, g8_7, o19_8);
              o19_9 = fma(eb, g9_7, o19_9);
            }
            { const double eb = bi[109];
              o19_8 = fma(eb, g8_14, o19_8);
              o19_9 = fma(eb, g9_14, o19_9);
            }
            { const double eb = bi[110];
              o20_8 = fma(eb, g8_0, o20_8);
              o20_9 = fma(eb, g9_0, o20_9);
            }
            { const double eb = bi[111];
              o20_8 = fma(eb, g8_1, o20_8);
              o20_9 = fma(eb, g9_1, o20_9);
            }
            { const double eb = bi[112];
              o20_8 = fma(eb, g8_2, o20_8);
              o20_9 = fma(eb, g9_2, o20_9);
            }
            { const double eb = bi[113];
              o20_8 = fma(eb, g8_5, o20_8);
              o20_9 = fma(eb, g9_5, o20_9);
            }
            { const double eb = bi[114];
              o21_8 = fma(eb, g8_0, o21_8);
              o21_9 = fma(eb, g9_0, o21_9);
            }
            { const double eb = bi[115];
              o21_8 = fma(eb, g8_1, o21_8);
              o21_9 = fma(eb, g9_1, o21_9);
            }
            { const double eb = bi[116];
              o21_8 = fma(eb, g8_2, o21_8);
              o21_9 = fma(eb, g9_2, o21_9);
            }
            { const double eb = bi[117];
              o21_8 = fma(eb, g8_5, o21_8);
              o21_9 = fma(eb, g9_5, o21_9);
            }
            { const double eb = bi[118];
              o21_8 = fma(eb, g8_3, o21_8);
              o21_9 = fma(eb, g9_3, o21_9);
            }
            { const double eb = bi[119];
              o21_8 = fma(eb, g8_7, o21_8);
              o21_9 = fma(eb, g9_7, o21_9);
            }
            { const double eb = bi[120];
              o21_8 = fma(eb, g8_8, o21_8);
              o21_9 = fma(eb, g9_8, o21_9);
            }
            { const double eb = bi[121];
              o21_8 = fma(eb, g8_15, o21_8);
              o21_9 = fma(eb, g9_15, o21_9);
            }
            { const double eb = bi[122];
              o22_8 = fma(eb, g8_0, o22_8);
              o22_9 = fma(eb, g9_0, o22_9);
            }
            { const double eb = bi[123];
              o22_8 = fma(eb, g8_1, o22_8);
              o22_9 = fma(eb, g9_1, o22_9);
            }
            { const double eb = bi[124];
              o22_8 = fma(eb, g8_2, o22_8);
              o22_9 = fma(eb, g9_2, o22_9);
            }
            { const double eb = bi[125];
              o22_8 = fma(eb, g8_5, o22_8);
              o22_9 = fma(eb, g9_5, o22_9);
            }
            { const double eb = bi[126];
              o22_8 = fma(eb, g8_6, o22_8);
              o22_9 = fma(eb, g9_6, o22_9);
            }
            { const double eb = bi[127];
              o22_8 = fma(eb, g8_12, o22_8);
              o22_9 = fma(eb, g9_12, o22_9);
            }
            { const double eb = bi[128];
              o23_8 = fma(eb, g8_0, o23_8);
              o23_9 = fma(eb, g9_0, o23_9);
            }
            { const double eb = bi[129];
              o23_8 = fma(eb, g8_1, o23_8);
              o23_9 = fma(eb, g9_1, o23_9);
            }
            { const double eb = bi[130];
              o23_8 = fma(eb, g8_4, o23_8);
              o23_9 = fma(eb, g9_4, o23_9);
            }
            { const double eb = bi[131];
              o23_8 = fma(eb, g8_2, o23_8);
              o23_9 = fma(eb, g9_2, o23_9);
            }
            { const double eb = bi[132];
              o23_8 = fma(eb, g8_5, o23_8);
              o23_9 = fma(eb, g9_5, o23_9);
            }
            { const double eb = bi[133];
              o23_8 = fma(eb, g8_11, o23_8);
              o23_9 = fma(eb, g9_11, o23_9);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk8 = PT[(fI + 2) * N + fJ + 0];
            const double ptk9 = PT[(fI + 2) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Abc3_2 = PA[(fQ + 3) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            jab0 += o0_8 * ptk8 + o0_9 * ptk9;
            jab1 += o1_8 * ptk8 + o1_9 * ptk9;
            jab2 += o2_8 * ptk8 + o2_9 * ptk9;
            jab3 += o3_8 * ptk8 + o3_9 * ptk9;
            jab4 += o4_8 * ptk8 + o4_9 * ptk9;
            jab5 += o5_8 * ptk8 + o5_9 * ptk9;
            jab6 += o6_8 * ptk8 + o6_9 * ptk9;
            jab7 += o7_8 * ptk8 + o7_9 * ptk9;
            jab8 += o8_8 * ptk8 + o8_9 * ptk9;
            jab9 += o9_8 * ptk8 + o9_9 * ptk9;
            jab10 += o10_8 * ptk8 + o10_9 * ptk9;
            jab11 += o11_8 * ptk8 + o11_9 * ptk9;
            jab12 += o12_8 * ptk8 + o12_9 * ptk9;
            jab13 += o13_8 * ptk8 + o13_9 * ptk9;
            jab14 += o14_8 * ptk8 + o14_9 * ptk9;
            jab15 += o15_8 * ptk8 + o15_9 * ptk9;
            jab16 += o16_8 * ptk8 + o16_9 * ptk9;
            jab17 += o17_8 * ptk8 + o17_9 * ptk9;
            jab18 += o18_8 * ptk8 + o18_9 * ptk9;
            jab19 += o19_8 * ptk8 + o19_9 * ptk9;
            jab20 += o20_8 * ptk8 + o20_9 * ptk9;
            jab21 += o21_8 * ptk8 + o21_9 * ptk9;
            jab22 += o22_8 * ptk8 + o22_9 * ptk9;
            jab23 += o23_8 * ptk8 + o23_9 * ptk9;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_8 * ptb0 + o1_8 * ptb1 + o2_8 * ptb2 + o3_8 * ptb3 + o4_8 * ptb4 + o5_8 * ptb5 + o6_8 * ptb6 + o7_8 * ptb7 + o8_8 * ptb8 + o9_8 * ptb9 + o10_8 * ptb10 + o11_8 * ptb11 + o12_8 * ptb12 + o13_8 * ptb13 + o14_8 * ptb14 + o15_8 * ptb15 + o16_8 * ptb16 + o17_8 * ptb17 + o18_8 * ptb18 + o19_8 * ptb19 + o20_8 * ptb20 + o21_8 * ptb21 + o22_8 * ptb22 + o23_8 * ptb23));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 1, 2.0 * deg * (o0_9 * ptb0 + o1_9 * ptb1 + o2_9 * ptb2 + o3_9 * ptb3 + o4_9 * ptb4 + o5_9 * ptb5 + o6_9 * ptb6 + o7_9 * ptb7 + o8_9 * ptb8 + o9_9 * ptb9 + o10_9 * ptb10 + o11_9 * ptb11 + o12_9 * ptb12 + o13_9 * ptb13 + o14_9 * ptb14 + o15_9 * ptb15 + o16_9 * ptb16 + o17_9 * ptb17 + o18_9 * ptb18 + o19_9 * ptb19 + o20_9 * ptb20 + o21_9 * ptb21 + o22_9 * ptb22 + o23_9 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_8 * Abd0_0 + o0_9 * Abd0_1 + o1_8 * Abd1_0 + o1_9 * Abd1_1 + o2_8 * Abd2_0 + o2_9 * Abd2_1 + o3_8 * Abd3_0 + o3_9 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_8 * Aad0_0 + o0_9 * Aad0_1 + o4_8 * Aad1_0 + o4_9 * Aad1_1 + o8_8 * Aad2_0 + o8_9 * Aad2_1 + o12_8 * Aad3_0 + o12_9 * Aad3_1 + o16_8 * Aad4_0 + o16_9 * Aad4_1 + o20_8 * Aad5_0 + o20_9 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_8 * Abc0_2 + o1_8 * Abc1_2 + o2_8 * Abc2_2 + o3_8 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_8 * Aac0_2 + o4_8 * Aac1_2 + o8_8 * Aac2_2 + o12_8 * Aac3_2 + o16_8 * Aac4_2 + o20_8 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_9 * Abc0_2 + o1_9 * Abc1_2 + o2_9 * Abc2_2 + o3_9 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_9 * Aac0_2 + o4_9 * Aac1_2 + o8_9 * Aac2_2 + o12_9 * Aac3_2 + o16_9 * Aac4_2 + o20_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_8 * Aad0_0 + o1_9 * Aad0_1 + o5_8 * Aad1_0 + o5_9 * Aad1_1 + o9_8 * Aad2_0 + o9_9 * Aad2_1 + o13_8 * Aad3_0 + o13_9 * Aad3_1 + o17_8 * Aad4_0 + o17_9 * Aad4_1 + o21_8 * Aad5_0 + o21_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_8 * Aac0_2 + o5_8 * Aac1_2 + o9_8 * Aac2_2 + o13_8 * Aac3_2 + o17_8 * Aac4_2 + o21_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_9 * Aac0_2 + o5_9 * Aac1_2 + o9_9 * Aac2_2 + o13_9 * Aac3_2 + o17_9 * Aac4_2 + o21_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_8 * Aad0_0 + o2_9 * Aad0_1 + o6_8 * Aad1_0 + o6_9 * Aad1_1 + o10_8 * Aad2_0 + o10_9 * Aad2_1 + o14_8 * Aad3_0 + o14_9 * Aad3_1 + o18_8 * Aad4_0 + o18_9 * Aad4_1 + o22_8 * Aad5_0 + o22_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_8 * Aac0_2 + o6_8 * Aac1_2 + o10_8 * Aac2_2 + o14_8 * Aac3_2 + o18_8 * Aac4_2 + o22_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_9 * Aac0_2 + o6_9 * Aac1_2 + o10_9 * Aac2_2 + o14_9 * Aac3_2 + o18_9 * Aac4_2 + o22_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_8 * Aad0_0 + o3_9 * Aad0_1 + o7_8 * Aad1_0 + o7_9 * Aad1_1 + o11_8 * Aad2_0 + o11_9 * Aad2_1 + o15_8 * Aad3_0 + o15_9 * Aad3_1 + o19_8 * Aad4_0 + o19_9 * Aad4_1 + o23_8 * Aad5_0 + o23_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_8 * Aac0_2 + o7_8 * Aac1_2 + o11_8 * Aac2_2 + o15_8 * Aac3_2 + o19_8 * Aac4_2 + o23_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_9 * Aac0_2 + o7_9 * Aac1_2 + o11_9 * Aac2_2 + o15_9 * Aac3_2 + o19_9 * Aac4_2 + o23_9 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_8 * Abd0_0 + o4_9 * Abd0_1 + o5_8 * Abd1_0 + o5_9 * Abd1_1 + o6_8 * Abd2_0 + o6_9 * Abd2_1 + o7_8 * Abd3_0 + o7_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_8 * Abc0_2 + o5_8 * Abc1_2 + o6_8 * Abc2_2 + o7_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_9 * Abc0_2 + o5_9 * Abc1_2 + o6_9 * Abc2_2 + o7_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_8 * Abd0_0 + o8_9 * Abd0_1 + o9_8 * Abd1_0 + o9_9 * Abd1_1 + o10_8 * Abd2_0 + o10_9 * Abd2_1 + o11_8 * Abd3_0 + o11_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_8 * Abc0_2 + o9_8 * Abc1_2 + o10_8 * Abc2_2 + o11_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_9 * Abc0_2 + o9_9 * Abc1_2 + o10_9 * Abc2_2 + o11_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_8 * Abd0_0 + o12_9 * Abd0_1 + o13_8 * Abd1_0 + o13_9 * Abd1_1 + o14_8 * Abd2_0 + o14_9 * Abd2_1 + o15_8 * Abd3_0 + o15_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_8 * Abc0_2 + o13_8 * Abc1_2 + o14_8 * Abc2_2 + o15_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_9 * Abc0_2 + o13_9 * Abc1_2 + o14_9 * Abc2_2 + o15_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_8 * Abd0_0 + o16_9 * Abd0_1 + o17_8 * Abd1_0 + o17_9 * Abd1_1 + o18_8 * Abd2_0 + o18_9 * Abd2_1 + o19_8 * Abd3_0 + o19_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_8 * Abc0_2 + o17_8 * Abc1_2 + o18_8 * Abc2_2 + o19_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_9 * Abc0_2 + o17_9 * Abc1_2 + o18_9 * Abc2_2 + o19_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_8 * Abd0_0 + o20_9 * Abd0_1 + o21_8 * Abd1_0 + o21_9 * Abd1_1 + o22_8 * Abd2_0 + o22_9 * Abd2_1 + o23_8 * Abd3_0 + o23_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_8 * Abc0_2 + o21_8 * Abc1_2 + o22_8 * Abc2_2 + o23_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_9 * Abc0_2 + o21_9 * Abc1_2 + o22_9 * Abc2_2 + o23_9 * Abc3_2));
          }
        } break;
        case 5: {  // ket functions [10, 11]
          double o0_10 = 0;
          double o0_11 = 0;
          double o1_10 = 0;
          double o1_11 = 0;
          double o2_10 = 0;
          double o2_11 = 0;
          double o3_10 = 0;
          double o3_11 = 0;
          double o4_10 = 0;
          double o4_11 = 0;
          double o5_10 = 0;
          double o5_11 = 0;
          double o6_10 = 0;
          double o6_11 = 0;
          double o7_10 = 0;
          double o7_11 = 0;
          double o8_10 = 0;
          double o8_11 = 0;
          double o9_10 = 0;
          double o9_11 = 0;
          double o10_10 = 0;
          double o10_11 = 0;
          double o11_10 = 0;
          double o11_11 = 0;
          double o12_10 = 0;
          double o12_11 = 0;
          double o13_10 = 0;
          double o13_11 = 0;
          double o14_10 = 0;
          double o14_11 = 0;
          double o15_10 = 0;
          double o15_11 = 0;
          double o16_10 = 0;
          double o16_11 = 0;
          double o17_10 = 0;
          double o17_11 = 0;
          double o18_10 = 0;
          double o18_11 = 0;
          double o19_10 = 0;
          double o19_11 = 0;
          double o20_10 = 0;
          double o20_11 = 0;
          double o21_10 = 0;
          double o21_11 = 0;
          double o22_10 = 0;
          double o22_11 = 0;
          double o23_10 = 0;
          double o23_11 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek10_0 = kj[52 * kS];
              const double ek10_1 = -kj[53 * kS];
              const double ek10_2 = kj[54 * kS];
              const double ek10_3 = -kj[55 * kS];
              const double ek10_4 = kj[56 * kS];
              const double ek10_5 = -kj[57 * kS];
              const double ek11_0 = kj[58 * kS];
              const double ek11_1 = -kj[59 * kS];
              const double ek11_2 = kj[60 * kS];
              const double ek11_3 = -kj[61 * kS];
              g10_0 = fma(ek10_0, b0, g10_0);
              g11_0 = fma(ek11_0, b0, g11_0);
              const double r0_0_0_1 = Z * b1;
              g10_1 = fma(ek10_0, r0_0_0_1, g10_1);
              g10_0 = fma(ek10_1, r0_0_0_1, g10_0);
              g11_1 = fma(ek11_0, r0_0_0_1, g11_1);
              g11_0 = fma(ek11_1, r0_0_0_1, g11_0);
              const double r0_0_1_0 = Y * b1;
              g10_2 = fma(ek10_0, r0_0_1_0, g10_2);
              g10_0 = fma(ek10_3, r0_0_1_0, g10_0);
              g11_2 = fma(ek11_0, r0_0_1_0, g11_2);
              const double r0_1_0_0 = X * b1;
              g10_3 = fma(ek10_0, r0_1_0_0, g10_3);
              g11_3 = fma(ek11_0, r0_1_0_0, g11_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g10_4 = fma(ek10_0, r0_0_0_2, g10_4);
              g10_1 = fma(ek10_1, r0_0_0_2, g10_1);
              g10_0 = fma(ek10_2, r0_0_0_2, g10_0);
              g11_4 = fma(ek11_0, r0_0_0_2, g11_4);
              g11_1 = fma(ek11_1, r0_0_0_2, g11_1);
              g11_0 = fma(ek11_2, r0_0_0_2, g11_0);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g10_5 = fma(ek10_0, r0_0_1_1, g10_5);
              g10_2 = fma(ek10_1, r0_0_1_1, g10_2);
              g10_1 = fma(ek10_3, r0_0_1_1, g10_1);
              g10_0 = fma(ek10_4, r0_0_1_1, g10_0);
              g11_5 = fma(ek11_0, r0_0_1_1, g11_5);
              g11_2 = fma(ek11_1, r0_0_1_1, g11_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g10_6 = fma(ek10_0, r0_0_2_0, g10_6);
              g10_2 = fma(ek10_3, r0_0_2_0, g10_2);
              g11_6 = fma(ek11_0, r0_0_2_0, g11_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g10_7 = fma(ek10_0, r0_1_0_1, g10_7);
              g10_3 = fma(ek10_1, r0_1_0_1, g10_3);
              g11_7 = fma(ek11_0, r0_1_0_1, g11_7);
              g11_3 = fma(ek11_1, r0_1_0_1, g11_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g10_8 = fma(ek10_0, r0_1_1_0, g10_8);
              g10_3 = fma(ek10_3, r0_1_1_0, g10_3);
              g11_8 = fma(ek11_0, r0_1_1_0, g11_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g10_9 = fma(ek10_0, r0_2_0_0, g10_9);
              g11_9 = fma(ek11_0, r0_2_0_0, g11_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g10_10 = fma(ek10_0, r0_0_0_3, g10_10);
              g10_4 = fma(ek10_1, r0_0_0_3, g10_4);
              g10_1 = fma(ek10_2, r0_0_0_3, g10_1);
              g11_10 = fma(ek11_0, r0_0_0_3, g11_10);
              g11_4 = fma(ek11_1, r0_0_0_3, g11_4);
              g11_1 = fma(ek11_2, r0_0_0_3, g11_1);
              g11_0 = fma(ek11_3, r0_0_0_3, g11_0);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g10_11 = fma(ek10_0, r0_0_1_2, g10_11);
              g10_5 = fma(ek10_1, r0_0_1_2, g10_5);
              g10_2 = fma(ek10_2, r0_0_1_2, g10_2);
              g10_4 = fma(ek10_3, r0_0_1_2, g10_4);
              g10_1 = fma(ek10_4, r0_0_1_2, g10_1);
              g10_0 = fma(ek10_5, r0_0_1_2, g10_0);
              g11_11 = fma(ek11_0, r0_0_1_2, g11_11);
              g11_5 = fma(ek11_1, r0_0_1_2, g11_5);
              g11_2 = fma(ek11_2, r0_0_1_2, g11_2);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g10_12 = fma(ek10_0, r0_0_2_1, g10_12);
              g10_6 = fma(ek10_1, r0_0_2_1, g10_6);
              g10_5 = fma(ek10_3, r0_0_2_1, g10_5);
              g10_2 = fma(ek10_4, r0_0_2_1, g10_2);
              g11_12 = fma(ek11_0, r0_0_2_1, g11_12);
              g11_6 = fma(ek11_1, r0_0_2_1, g11_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g10_13 = fma(ek10_0, r0_0_3_0, g10_13);
              g10_6 = fma(ek10_3, r0_0_3_0, g10_6);
              g11_13 = fma(ek11_0, r0_0_3_0, g11_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g10_14 = fma(ek10_0, r0_1_0_2, g10_14);
              g10_7 = fma(ek10_1, r0_1_0_2, g10_7);
              g10_3 = fma(ek10_2, r0_1_0_2, g10_3);
              g11_14 = fma(ek11_0, r0_1_0_2, g11_14);
              g11_7 = fma(ek11_1, r0_1_0_2, g11_7);
              g11_3 = fma(ek11_2, r0_1_0_2, g11_3);
              const double r0_1_1_1 = X * r1_0_1_1;
              g10_15 = fma(ek10_0, r0_1_1_1, g10_15);
              g10_8 = fma(ek10_1, r0_1_1_1, g10_8);
              g10_7 = fma(ek10_3, r0_1_1_1, g10_7);
              g10_3 = fma(ek10_4, r0_1_1_1, g10_3);
              g11_15 = fma(ek11_0, r0_1_1_1, g11_15);
              g11_8 = fma(ek11_1, r0_1_1_1, g11_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g10_16 = fma(ek10_0, r0_1_2_0, g10_16);
              g10_8 = fma(ek10_3, r0_1_2_0, g10_8);
              g11_16 = fma(ek11_0, r0_1_2_0, g11_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g10_17 = fma(ek10_0, r0_2_0_1, g10_17);
              g10_9 = fma(ek10_1, r0_2_0_1, g10_9);
              g11_17 = fma(ek11_0, r0_2_0_1, g11_17);
              g11_9 = fma(ek11_1, r0_2_0_1, g11_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g10_18 = fma(ek10_0, r0_2_1_0, g10_18);
              g10_9 = fma(ek10_3, r0_2_1_0, g10_9);
              g11_18 = fma(ek11_0, r0_2_1_0, g11_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g10_19 = fma(ek10_0, r0_3_0_0, g10_19);
              g11_19 = fma(ek11_0, r0_3_0_0, g11_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g10_10 = fma(ek10_1, r0_0_0_4, g10_10);
              g10_4 = fma(ek10_2, r0_0_0_4, g10_4);
              g11_10 = fma(ek11_1, r0_0_0_4, g11_10);
              g11_4 = fma(ek11_2, r0_0_0_4, g11_4);
              g11_1 = fma(ek11_3, r0_0_0_4, g11_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g10_11 = fma(ek10_1, r0_0_1_3, g10_11);
              g10_5 = fma(ek10_2, r0_0_1_3, g10_5);
              g10_10 = fma(ek10_3, r0_0_1_3, g10_10);
              g10_4 = fma(ek10_4, r0_0_1_3, g10_4);
              g10_1 = fma(ek10_5, r0_0_1_3, g10_1);
              g11_11 = fma(ek11_1, r0_0_1_3, g11_11);
              g11_5 = fma(ek11_2, r0_0_1_3, g11_5);
              g11_2 = fma(ek11_3, r0_0_1_3, g11_2);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g10_12 = fma(ek10_1, r0_0_2_2, g10_12);
              g10_6 = fma(ek10_2, r0_0_2_2, g10_6);
              g10_11 = fma(ek10_3, r0_0_2_2, g10_11);
              g10_5 = fma(ek10_4, r0_0_2_2, g10_5);
              g10_2 = fma(ek10_5, r0_0_2_2, g10_2);
              g11_12 = fma(ek11_1, r0_0_2_2, g11_12);
              g11_6 = fma(ek11_2, r0_0_2_2, g11_6);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g10_13 = fma(ek10_1, r0_0_3_1, g10_13);
              g10_12 = fma(ek10_3, r0_0_3_1, g10_12);
              g10_6 = fma(ek10_4, r0_0_3_1, g10_6);
              g11_13 = fma(ek11_1, r0_0_3_1, g11_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g10_13 = fma(ek10_3, r0_0_4_0, g10_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g10_14 = fma(ek10_1, r0_1_0_3, g10_14);
              g10_7 = fma(ek10_2, r0_1_0_3, g10_7);
              g11_14 = fma(ek11_1, r0_1_0_3, g11_14);
              g11_7 = fma(ek11_2, r0_1_0_3, g11_7);
              g11_3 = fma(ek11_3, r0_1_0_3, g11_3);
              const double r0_1_1_2 = X * r1_0_1_2;
              g10_15 = fma(ek10_1, r0_1_1_2, g10_15);
              g10_8 = fma(ek10_2, r0_1_1_2, g10_8);
              g10_14 = fma(ek10_3, r0_1_1_2, g10_14);
              g10_7 = fma(ek10_4, r0_1_1_2, g10_7);
              g10_3 = fma(ek10_5, r0_1_1_2, g10_3);
              g11_15 = fma(ek11_1, r0_1_1_2, g11_15);
              g11_8 = fma(ek11_2, r0_1_1_2, g11_8);
              const double r0_1_2_1 = X * r1_0_2_1;
              g10_16 = fma(ek10_1, r0_1_2_1, g10_16);
              g10_15 = fma(ek10_3, r0_1_2_1, g10_15);
              g10_8 = fma(ek10_4, r0_1_2_1, g10_8);
              g11_16 = fma(ek11_1, r0_1_2_1, g11_16);
              const double r0_1_3_0 = X * r1_0_3_0;
              g10_16 = fma(ek10_3, r0_1_3_0, g10_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g10_17 = fma(ek10_1, r0_2_0_2, g10_17);
              g10_9 = fma(ek10_2, r0_2_0_2, g10_9);
              g11_17 = fma(ek11_1, r0_2_0_2, g11_17);
              g11_9 = fma(ek11_2, r0_2_0_2, g11_9);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g10_18 = fma(ek10_1, r0_2_1_1, g10_18);
              g10_17 = fma(ek10_3, r0_2_1_1, g10_17);
              g10_9 = fma(ek10_4, r0_2_1_1, g10_9);
              g11_18 = fma(ek11_1, r0_2_1_1, g11_18);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g10_18 = fma(ek10_3, r0_2_2_0, g10_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g10_19 = fma(ek10_1, r0_3_0_1, g10_19);
              g11_19 = fma(ek11_1, r0_3_0_1, g11_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g10_19 = fma(ek10_3, r0_3_1_0, g10_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g10_10 = fma(ek10_2, r0_0_0_5, g10_10);
              g11_10 = fma(ek11_2, r0_0_0_5, g11_10);
              g11_4 = fma(ek11_3, r0_0_0_5, g11_4);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g10_11 = fma(ek10_2, r0_0_1_4, g10_11);
              g10_10 = fma(ek10_4, r0_0_1_4, g10_10);
              g10_4 = fma(ek10_5, r0_0_1_4, g10_4);
              g11_11 = fma(ek11_2, r0_0_1_4, g11_11);
              g11_5 = fma(ek11_3, r0_0_1_4, g11_5);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g10_12 = fma(ek10_2, r0_0_2_3, g10_12);
              g10_11 = fma(ek10_4, r0_0_2_3, g10_11);
              g10_5 = fma(ek10_5, r0_0_2_3, g10_5);
              g11_12 = fma(ek11_2, r0_0_2_3, g11_12);
              g11_6 = fma(ek11_3, r0_0_2_3, g11_6);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g10_13 = fma(ek10_2, r0_0_3_2, g10_13);
              g10_12 = fma(ek10_4, r0_0_3_2, g10_12);
              g10_6 = fma(ek10_5, r0_0_3_2, g10_6);
              g11_13 = fma(ek11_2, r0_0_3_2, g11_13);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g10_13 = fma(ek10_4, r0_0_4_1, g10_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g10_14 = fma(ek10_2, r0_1_0_4, g10_14);
              g11_14 = fma(ek11_2, r0_1_0_4, g11_14);
              g11_7 = fma(ek11_3, r0_1_0_4, g11_7);
              const double r0_1_1_3 = X * r1_0_1_3;
              g10_15 = fma(ek10_2, r0_1_1_3, g10_15);
              g10_14 = fma(ek10_4, r0_1_1_3, g10_14);
              g10_7 = fma(ek10_5, r0_1_1_3, g10_7);
              g11_15 = fma(ek11_2, r0_1_1_3, g11_15);
              g11_8 = fma(ek11_3, r0_1_1_3, g11_8);
              const double r0_1_2_2 = X * r1_0_2_2;
              g10_16 = fma(ek10_2, r0_1_2_2, g10_16);
              g10_15 = fma(ek10_4, r0_1_2_2, g10_15);
              g10_8 = fma(ek10_5, r0_1_2_2, g10_8);
              g11_16 = fma(ek11_2, r0_1_2_2, g11_16);
              const double r0_1_3_1 = X * r1_0_3_1;
              g10_16 = fma(ek10_4, r0_1_3_1, g10_16);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g10_17 = fma(ek10_2, r0_2_0_3, g10_17);
              g11_17 = fma(ek11_2, r0_2_0_3, g11_17);
              g11_9 = fma(ek11_3, r0_2_0_3, g11_9);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g10_18 = fma(ek10_2, r0_2_1_2, g10_18);
              g10_17 = fma(ek10_4, r0_2_1_2, g10_17);
              g10_9 = fma(ek10_5, r0_2_1_2, g10_9);
              g11_18 = fma(ek11_2, r0_2_1_2, g11_18);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g10_18 = fma(ek10_4, r0_2_2_1, g10_18);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g10_19 = fma(ek10_2, r0_3_0_2, g10_19);
              g11_19 = fma(ek11_2, r0_3_0_2, g11_19);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g10_19 = fma(ek10_4, r0_3_1_1, g10_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_0_0_6 = fma(Z, r1_0_0_5, 5.0 * r1_0_0_4);
              g11_10 = fma(ek11_3, r0_0_0_6, g11_10);
              const double r0_0_1_5 = Y * r1_0_0_5;
              g10_10 = fma(ek10_5, r0_0_1_5, g10_10);
              g11_11 = fma(ek11_3, r0_0_1_5, g11_11);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_0_2_4 = fma(Y, r1_0_1_4, r1_0_0_4);
              g10_11 = fma(ek10_5, r0_0_2_4, g10_11);
              g11_12 = fma(ek11_3, r0_0_2_4, g11_12);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_0_3_3 = fma(Y, r1_0_2_3, 2.0 * r1_0_1_3);
              g10_12 = fma(ek10_5, r0_0_3_3, g10_12);
              g11_13 = fma(ek11_3, r0_0_3_3, g11_13);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_0_4_2 = fma(Y, r1_0_3_2, 3.0 * r1_0_2_2);
              g10_13 = fma(ek10_5, r0_0_4_2, g10_13);
              const double r0_1_0_5 = X * r1_0_0_5;
              g11_14 = fma(ek11_3, r0_1_0_5, g11_14);
              const double r0_1_1_4 = X * r1_0_1_4;
              g10_14 = fma(ek10_5, r0_1_1_4, g10_14);
              g11_15 = fma(ek11_3, r0_1_1_4, g11_15);
              const double r0_1_2_3 = X * r1_0_2_3;
              g10_15 = fma(ek10_5, r0_1_2_3, g10_15);
              g11_16 = fma(ek11_3, r0_1_2_3, g11_16);
              const double r0_1_3_2 = X * r1_0_3_2;
              g10_16 = fma(ek10_5, r0_1_3_2, g10_16);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g11_17 = fma(ek11_3, r0_2_0_4, g11_17);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g10_17 = fma(ek10_5, r0_2_1_3, g10_17);
              g11_18 = fma(ek11_3, r0_2_1_3, g11_18);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g10_18 = fma(ek10_5, r0_2_2_2, g10_18);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g11_19 = fma(ek11_3, r0_3_0_3, g11_19);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g10_19 = fma(ek10_5, r0_3_1_2, g10_19);
            }
            { const double eb = bi[5];
              o0_10 = fma(eb, g10_0, o0_10);
              o0_11 = fma(eb, g11_0, o0_11);
            }
            { const double eb = bi[6];
              o0_10 = fma(eb, g10_3, o0_10);
              o0_11 = fma(eb, g11_3, o0_11);
            }
            { const double eb = bi[7];
              o0_10 = fma(eb, g10_9, o0_10);
              o0_11 = fma(eb, g11_9, o0_11);
            }
            { const double eb = bi[8];
              o1_10 = fma(eb, g10_0, o1_10);
              o1_11 = fma(eb, g11_0, o1_11);
            }
            { const double eb = bi[9];
              o1_10 = fma(eb, g10_3, o1_10);
              o1_11 = fma(eb, g11_3, o1_11);
            }
            { const double eb = bi[10];
              o1_10 = fma(eb, g10_9, o1_10);
              o1_11 = fma(eb, g11_9, o1_11);
            }
            { const double eb = bi[11];
              o1_10 = fma(eb, g10_19, o1_10);
              o1_11 = fma(eb, g11_19, o1_11);
            }
            { const double eb = bi[12];
              o2_10 = fma(eb, g10_0, o2_10);
              o2_11 = fma(eb, g11_0, o2_11);
            }
            { const double eb = bi[13];
              o2_10 = fma(eb, g10_2, o2_10);
              o2_11 = fma(eb, g11_2, o2_11);
            }
            { const double eb = bi[14];
              o2_10 = fma(eb, g10_3, o2_10);
              o2_11 = fma(eb, g11_3, o2_11);
            }
            { const double eb = bi[15];
              o2_10 = fma(eb, g10_8, o2_10);
              o2_11 = fma(eb, g11_8, o2_11);
            }
            { const double eb = bi[16];
              o2_10 = fma(eb, g10_9, o2_10);
              o2_11 = fma(eb, g11_9, o2_11);
            }
            { const double eb = bi[17];
              o2_10 = fma(eb, g10_18, o2_10);
              o2_11 = fma(eb, g11_18, o2_11);
            }
            { const double eb = bi[18];
              o3_10 = fma(eb, g10_0, o3_10);
              o3_11 = fma(eb, g11_0, o3_11);
            }
            { const double eb = bi[19];
              o3_10 = fma(eb, g10_1, o3_10);
              o3_11 = fma(eb, g11_1, o3_11);
            }
            { const double eb = bi[20];
              o3_10 = fma(eb, g10_3, o3_10);
              o3_11 = fma(eb, g11_3, o3_11);
            }
            { const double eb = bi[21];
              o3_10 = fma(eb, g10_7, o3_10);
              o3_11 = fma(eb, g11_7, o3_11);
            }
            { const double eb = bi[22];
              o3_10 = fma(eb, g10_9, o3_10);
              o3_11 = fma(eb, g11_9, o3_11);
            }
            { const double eb = bi[23];
              o3_10 = fma(eb, g10_17, o3_10);
              o3_11 = fma(eb, g11_17, o3_11);
            }
            { const double eb = bi[24];
              o4_10 = fma(eb, g10_0, o4_10);
              o4_11 = fma(eb, g11_0, o4_11);
            }
            { const double eb = bi[25];
              o4_10 = fma(eb, g10_2, o4_10);
              o4_11 = fma(eb, g11_2, o4_11);
            }
            { const double eb = bi[26];
              o4_10 = fma(eb, g10_6, o4_10);
              o4_11 = fma(eb, g11_6, o4_11);
            }
            { const double eb = bi[27];
              o5_10 = fma(eb, g10_0, o5_10);
              o5_11 = fma(eb, g11_0, o5_11);
            }
            { const double eb = bi[28];
              o5_10 = fma(eb, g10_2, o5_10);
              o5_11 = fma(eb, g11_2, o5_11);
            }
            { const double eb = bi[29];
              o5_10 = fma(eb, g10_6, o5_10);
              o5_11 = fma(eb, g11_6, o5_11);
            }
            { const double eb = bi[30];
              o5_10 = fma(eb, g10_3, o5_10);
              o5_11 = fma(eb, g11_3, o5_11);
            }
            { const double eb = bi[31];
              o5_10 = fma(eb, g10_8, o5_10);
              o5_11 = fma(eb, g11_8, o5_11);
            }
            { const double eb = bi[32];
              o5_10 = fma(eb, g10_16, o5_10);
              o5_11 = fma(eb, g11_16, o5_11);
            }
            { const double eb = bi[33];
              o6_10 = fma(eb, g10_0, o6_10);
              o6_11 = fma(eb, g11_0, o6_11);
            }
            { const double eb = bi[34];
              o6_10 = fma(eb, g10_2, o6_10);
              o6_11 = fma(eb, g11_2, o6_11);
            }
            { const double eb = bi[35];
              o6_10 = fma(eb, g10_6, o6_10);
              o6_11 = fma(eb, g11_6, o6_11);
            }
            { const double eb = bi[36];
              o6_10 = fma(eb, g10_13, o6_10);
              o6_11 = fma(eb, g11_13, o6_11);
            }
            { const double eb = bi[37];
              o7_10 = fma(eb, g10_0, o7_10);
              o7_11 = fma(eb, g11_0, o7_11);
            }
            { const double eb = bi[38];
              o7_10 = fma(eb, g10_1, o7_10);
              o7_11 = fma(eb, g11_1, o7_11);
            }
            { const double eb = bi[39];
              o7_10 = fma(eb, g10_2, o7_10);
              o7_11 = fma(eb, g11_2, o7_11);
            }
            { const double eb = bi[40];
              o7_10 = fma(eb, g10_5, o7_10);
              o7_11 = fma(eb, g11_5, o7_11);
            }
            { const double eb = bi[41];
              o7_10 = fma(eb, g10_6, o7_10);
              o7_11 = fma(eb, g11_6, o7_11);
            }
            { const double eb = bi[42];
              o7_10 = fma(eb, g10_12, o7_10);
              o7_11 = fma(eb, g11_12, o7_11);
            }
            { const double eb = bi[43];
              o8_10 = fma(eb, g10_0, o8_10);
              o8_11 = fma(eb, g11_0, o8_11);
            }
            { const double eb = bi[44];
              o8_10 = fma(eb, g10_1, o8_10);
              o8_11 = fma(eb, g11_1, o8_11);
            }
            { const double eb = bi[45];
              o8_10 = fma(eb, g10_4, o8_10);
              o8_11 = fma(eb, g11_4, o8_11);
            }
            { const double eb = bi[46];
              o9_10 = fma(eb, g10_0, o9_10);
              o9_11 = fma(eb, g11_0, o9_11);
            }
            { const double eb = bi[47];
              o9_10 = fma(eb, g10_1, o9_10);
              o9_11 = fma(eb, g11_1, o9_11);
            }
            { const double eb = bi[48];
              o9_10 = fma(eb, g10_4, o9_10);
              o9_11 = fma(eb, g11_4, o9_11);
            }
            { const double eb = bi[49];
              o9_10 = fma(eb, g10_3, o9_10);
              o9_11 = fma(eb, g11_3, o9_11);
            }
            { const double eb = bi[50];
              o9_10 = fma(eb, g10_7, o9_10);
              o9_11 = fma(eb, g11_7, o9_11);
            }
            { const double eb = bi[51];
              o9_10 = fma(eb, g10_14, o9_10);
              o9_11 = fma(eb, g11_14, o9_11);
            }
            { const double eb = bi[52];
              o10_10 = fma(eb, g10_0, o10_10);
              o10_11 = fma(eb, g11_0, o10_11);
            }
            { const double eb = bi[53];
              o10_10 = fma(eb, g10_1, o10_10);
              o10_11 = fma(eb, g11_1, o10_11);
            }
            { const double eb = bi[54];
              o10_10 = fma(eb, g10_4, o10_10);
              o10_11 = fma(eb, g11_4, o10_11);
            }
            { const double eb = bi[55];
              o10_10 = fma(eb, g10_2, o10_10);
              o10_11 = fma(eb, g11_2, o10_11);
            }
            { const double eb = bi[56];
              o10_10 = fma(eb, g10_5, o10_10);
              o10_11 = fma(eb, g11_5, o10_11);
            }
            { const double eb = bi[57];
              o10_10 = fma(eb, g10_11, o10_10);
              o10_11 = fma(eb, g11_11, o10_11);
            }
            { const double eb = bi[58];
              o11_10 = fma(eb, g10_0, o11_10);
              o11_11 = fma(eb, g11_0, o11_11);
            }
            { const double eb = bi[59];
              o11_10 = fma(eb, g10_1, o11_10);
              o11_11 = fma(eb, g11_1, o11_11);
            }
            { const double eb = bi[60];
              o11_10 = fma(eb, g10_4, o11_10);
              o11_11 = fma(eb, g11_4, o11_11);
            }
            { const double eb = bi[61];
              o11_10 = fma(eb, g10_10, o11_10);
              o11_11 = fma(eb, g11_10, o11_11);
            }
            { const double eb = bi[62];
              o12_10 = fma(eb, g10_0, o12_10);
              o12_11 = fma(eb, g11_0, o12_11);
            }
            { const double eb = bi[63];
              o12_10 = fma(eb, g10_2, o12_10);
              o12_11 = fma(eb, g11_2, o12_11);
            }
            { const double eb = bi[64];
              o12_10 = fma(eb, g10_3, o12_10);
              o12_11 = fma(eb, g11_3, o12_11);
            }
            { const double eb = bi[65];
              o12_10 = fma(eb, g10_8, o12_10);
              o12_11 = fma(eb, g11_8, o12_11);
            }
            { const double eb = bi[66];
              o13_10 = fma(eb, g10_0, o13_10);
              o13_11 = fma(eb, g11_0, o13_11);
            }
            { const double eb = bi[67];
              o13_10 = fma(eb, g10_2, o13_10);
              o13_11 = fma(eb, g11_2, o13_11);
            }
            { const double eb = bi[68];
              o13_10 = fma(eb, g10_3, o13_10);
              o13_11 = fma(eb, g11_3, o13_11);
            }
            { const double eb = bi[69];
              o13_10 = fma(eb, g10_8, o13_10);
              o13_11 = fma(eb, g11_8, o13_11);
            }
            { const double eb = bi[70];
              o13_10 = fma(eb, g10_9, o13_10);
              o13_11 = fma(eb, g11_9, o13_11);
            }
            { const double eb = bi[71];
              o13_10 = fma(eb, g10_18, o13_10);
              o13_11 = fma(eb, g11_18, o13_11);
            }
            { const double eb = bi[72];
              o14_10 = fma(eb, g10_0, o14_10);
              o14_11 = fma(eb, g11_0, o14_11);
            }
            { const double eb = bi[73];
              o14_10 = fma(eb, g10_2, o14_10);
              o14_11 = fma(eb, g11_2, o14_11);
            }
            { const double eb = bi[74];
              o14_10 = fma(eb, g10_6, o14_10);
              o14_11 = fma(eb, g11_6, o14_11);
            }
            { const double eb = bi[75];
              o14_10 = fma(eb, g10_3, o14_10);
              o14_11 = fma(eb, g11_3, o14_11);
            }
            { const double eb = bi[76];
              o14_10 = fma(eb, g10_8, o14_10);
              o14_11 = fma(eb, g11_8, o14_11);
            }
            { const double eb = bi[77];
              o14_10 = fma(eb, g10_16, o14_10);
              o14_11 = fma(eb, g11_16, o14_11);
            }
            { const double eb = bi[78];
              o15_10 = fma(eb, g10_0, o15_10);
              o15_11 = fma(eb, g11_0, o15_11);
            }
            { const double eb = bi[79];
              o15_10 = fma(eb, g10_1, o15_10);
              o15_11 = fma(eb, g11_1, o15_11);
            }
            { const double eb = bi[80];
              o15_10 = fma(eb, g10_2, o15_10);
              o15_11 = fma(eb, g11_2, o15_11);
            }
            { const double eb = bi[81];
              o15_10 = fma(eb, g10_5, o15_10);
              o15_11 = fma(eb, g11_5, o15_11);
            }
            { const double eb = bi[82];
              o15_10 = fma(eb, g10_3, o15_10);
              o15_11 = fma(eb, g11_3, o15_11);
            }
            { const double eb = bi[83];
              o15_10 = fma(eb, g10_7, o15_10);
              o15_11 = fma(eb, g11_7, o15_11);
            }
            { const double eb = bi[84];
              o15_10 = fma(eb, g10_8, o15_10);
              o15_11 = fma(eb, g11_8, o15_11);
            }
            { const double eb = bi[85];
              o15_10 = fma(eb, g10_15, o15_10);
              o15_11 = fma(eb, g11_15, o15_11);
            }
            { const double eb = bi[86];
              o16_10 = fma(eb, g10_0, o16_10);
              o16_11 = fma(eb, g11_0, o16_11);
            }
            { const double eb = bi[87];
              o16_10 = fma(eb, g10_1, o16_10);
              o16_11 = fma(eb, g11_1, o16_11);
            }
            { const double eb = bi[88];
              o16_10 = fma(eb, g10_3, o16_10);
              o16_11 = fma(eb, g11_3, o16_11);
            }
            { const double eb = bi[89];
              o16_10 = fma(eb, g10_7, o16_10);
              o16_11 = fma(eb, g11_7, o16_11);
            }
            { const double eb = bi[90];
              o17_10 = fma(eb, g10_0, o17_10);
              o17_11 = fma(eb, g11_0, o17_11);
            }
            { const double eb = bi[91];
              o17_10 = fma(eb, g10_1, o17_10);
              o17_11 = fma(eb, g11_1, o17_11);
            }
            { const double eb = bi[92];
              o17_10 = fma(eb, g10_3, o17_10);
              o17_11 = fma(eb, g11_3, o17_11);
            }
            { const double eb = bi[93];
              o17_10 = fma(eb, g10_7, o17_10);
              o17_11 = fma(eb, g11_7, o17_11);
            }
            { const double eb = bi[94];
              o17_10 = fma(eb, g10_9, o17_10);
              o17_11 = fma(eb, g11_9, o17_11);
            }
            { const double eb = bi[95];
              o17_10 = fma(eb, g10_17, o17_10);
              o17_11 = fma(eb, g11_17, o17_11);
            }
            { const double eb = bi[96];
              o18_10 = fma(eb, g10_0, o18_10);
              o18_11 = fma(eb, g11_0, o18_11);
            }
            { const double eb = bi[97];
              o18_10 = fma(eb, g10_1, o18_10);
              o18_11 = fma(eb, g11_1, o18_11);
            }
            { const double eb = bi[98];
              o18_10 = fma(eb, g10_2, o18_10);
              o18_11 = fma(eb, g11_2, o18_11);
            }
            { const double eb = bi[99];
              o18_10 = fma(eb, g10_5, o18_10);
              o18_11 = fma(eb, g11_5, o18_11);
            }
            { const double eb = bi[100];
              o18_10 = fma(eb, g10_3, o18_10);
              o18_11 = fma(eb, g11_3, o18_11);
            }
            { const double eb = bi[101];
              o18_10 = fma(eb, g10_7, o18_10);
              o18_11 = fma(eb, g11_7, o18_11);
            }
            { const double eb = bi[102];
              o18_10 = fma(eb, g10_8, o18_10);
              o18_11 = fma(eb, g11_8, o18_11);
            }
            { const double eb = bi[103];
              o18_10 = fma(eb, g10_15, o18_10);
              o18_11 = fma(eb, g11_15, o18_11);
            }
            { const double eb = bi[104];
              o19_10 = fma(eb, g10_0, o19_10);
              o19_11 = fma(eb, g11_0, o19_11);
            }
            { const double eb = bi[105];
              o19_10 = fma(eb, g10_1, o19_10);
              o19_11 = fma(eb, g11_1, o19_11);
            }
            { const double eb = bi[106];
              o19_10 = fma(eb, g10_4, o19_10);
              o19_11 = fma(eb, g11_4, o19_11);
            }
            { const double eb = bi[107];
              o19_10 = fma(eb, g10_3, o19_10);
              o19_11 = fma(eb, g11_3, o19_11);
            }
            { const double eb = bi[108];
              o19_10 = fma(eb, g10_7, o19_10);
              o19_11 = fma(eb, g11_7, o19_11);
            }
            { const double eb = bi[109];
              o19_10 = fma(eb, g10_14, o19_10);
              o19_11 = fma(eb, g11_14, o19_11);
            }
            { const double eb = bi[110];
              o20_10 = fma(eb, g10_0, o20_10);
              o20_11 = fma(eb, g11_0, o20_11);
            }
            { const double eb = bi[111];
              o20_10 = fma(eb, g10_1, o20_10);
              o20_11 = fma(eb, g11_1, o20_11);
            }
            { const double eb = bi[112];
              o20_10 = fma(eb, g10_2, o20_10);
              o20_11 = fma(eb, g11_2, o20_11);
            }
            { const double eb = bi[113];
              o20_10 = fma(eb, g10_5, o20_10);
              o20_11 = fma(eb, g11_5, o20_11);
            }
            { const double eb = bi[114];
              o21_10 = fma(eb, g10_0, o21_10);
              o21_11 = fma(eb, g11_0, o21_11);
            }
            { const double eb = bi[115];
              o21_10 = fma(eb, g10_1, o21_10);
              o21_11 = fma(eb, g11_1, o21_11);
            }
            { const double eb = bi[116];
              o21_10 = fma(eb, g10_2, o21_10);
              o21_11 = fma(eb, g11_2, o21_11);
            }
            { const double eb = bi[117];
              o21_10 = fma(eb, g10_5, o21_10);
              o21_11 = fma(eb, g11_5, o21_11);
            }
            { const double eb = bi[118];
              o21_10 = fma(eb, g10_3, o21_10);
              o21_11 = fma(eb, g11_3, o21_11);
            }
            { const double eb = bi[119];
              o21_10 = fma(eb, g10_7, o21_10);
              o21_11 = fma(eb, g11_7, o21_11);
            }
            { const double eb = bi[120];
              o21_10 = fma(eb, g10_8, o21_10);
              o21_11 = fma(eb, g11_8, o21_11);
            }
            { const double eb = bi[121];
              o21_10 = fma(eb, g10_15, o21_10);
              o21_11 = fma(eb, g11_15, o21_11);
            }
            { const double eb = bi[122];
              o22_10 = fma(eb, g10_0, o22_10);
              o22_11 = fma(eb, g11_0, o22_11);
            }
            { const double eb = bi[123];
              o22_10 = fma(eb, g10_1, o22_10);
              o22_11 = fma(eb, g11_1, o22_11);
            }
            { const double eb = bi[124];
              o22_10 = fma(eb, g10_2, o22_10);
              o22_11 = fma(eb, g11_2, o22_11);
            }
            { const double eb = bi[125];
              o22_10 = fma(eb, g10_5, o22_10);
              o22_11 = fma(eb, g11_5, o22_11);
            }
            { const double eb = bi[126];
              o22_10 = fma(eb, g10_6, o22_10);
              o22_11 = fma(eb, g11_6, o22_11);
            }
            { const double eb = bi[127];
              o22_10 = fma(eb, g10_12, o22_10);
              o22_11 = fma(eb, g11_12, o22_11);
            }
            { const double eb = bi[128];
              o23_10 = fma(eb, g10_0, o23_10);
              o23_11 = fma(eb, g11_0, o23_11);
            }
            { const double eb = bi[129];
              o23_10 = fma(eb, g10_1, o23_10);
              o23_11 = fma(eb, g11_1, o23_11);
            }
            { const double eb = bi[130];
              o23_10 = fma(eb, g10_4, o23_10);
              o23_11 = fma(eb, g11_4, o23_11);
            }
            { const double eb = bi[131];
              o23_10 = fma(eb, g10_2, o23_10);
              o23_11 = fma(eb, g11_2, o23_11);
            }
            { const double eb = bi[132];
              o23_10 = fma(eb, g10_5, o23_10);
              o23_11 = fma(eb, g11_5, o23_11);
            }
            { const double eb = bi[133];
              o23_10 = fma(eb, g10_11, o23_10);
              o23_11 = fma(eb, g11_11, o23_11);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk10 = PT[(fI + 2) * N + fJ + 2];
            const double ptk11 = PT[(fI + 2) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Abc3_2 = PA[(fQ + 3) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            jab0 += o0_10 * ptk10 + o0_11 * ptk11;
            jab1 += o1_10 * ptk10 + o1_11 * ptk11;
            jab2 += o2_10 * ptk10 + o2_11 * ptk11;
            jab3 += o3_10 * ptk10 + o3_11 * ptk11;
            jab4 += o4_10 * ptk10 + o4_11 * ptk11;
            jab5 += o5_10 * ptk10 + o5_11 * ptk11;
            jab6 += o6_10 * ptk10 + o6_11 * ptk11;
            jab7 += o7_10 * ptk10 + o7_11 * ptk11;
            jab8 += o8_10 * ptk10 + o8_11 * ptk11;
            jab9 += o9_10 * ptk10 + o9_11 * ptk11;
            jab10 += o10_10 * ptk10 + o10_11 * ptk11;
            jab11 += o11_10 * ptk10 + o11_11 * ptk11;
            jab12 += o12_10 * ptk10 + o12_11 * ptk11;
            jab13 += o13_10 * ptk10 + o13_11 * ptk11;
            jab14 += o14_10 * ptk10 + o14_11 * ptk11;
            jab15 += o15_10 * ptk10 + o15_11 * ptk11;
            jab16 += o16_10 * ptk10 + o16_11 * ptk11;
            jab17 += o17_10 * ptk10 + o17_11 * ptk11;
            jab18 += o18_10 * ptk10 + o18_11 * ptk11;
            jab19 += o19_10 * ptk10 + o19_11 * ptk11;
            jab20 += o20_10 * ptk10 + o20_11 * ptk11;
            jab21 += o21_10 * ptk10 + o21_11 * ptk11;
            jab22 += o22_10 * ptk10 + o22_11 * ptk11;
            jab23 += o23_10 * ptk10 + o23_11 * ptk11;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 2, 2.0 * deg * (o0_10 * ptb0 + o1_10 * ptb1 + o2_10 * ptb2 + o3_10 * ptb3 + o4_10 * ptb4 + o5_10 * ptb5 + o6_10 * ptb6 + o7_10 * ptb7 + o8_10 * ptb8 + o9_10 * ptb9 + o10_10 * ptb10 + o11_10 * ptb11 + o12_10 * ptb12 + o13_10 * ptb13 + o14_10 * ptb14 + o15_10 * ptb15 + o16_10 * ptb16 + o17_10 * ptb17 + o18_10 * ptb18 + o19_10 * ptb19 + o20_10 * ptb20 + o21_10 * ptb21 + o22_10 * ptb22 + o23_10 * ptb23));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 3, 2.0 * deg * (o0_11 * ptb0 + o1_11 * ptb1 + o2_11 * ptb2 + o3_11 * ptb3 + o4_11 * ptb4 + o5_11 * ptb5 + o6_11 * ptb6 + o7_11 * ptb7 + o8_11 * ptb8 + o9_11 * ptb9 + o10_11 * ptb10 + o11_11 * ptb11 + o12_11 * ptb12 + o13_11 * ptb13 + o14_11 * ptb14 + o15_11 * ptb15 + o16_11 * ptb16 + o17_11 * ptb17 + o18_11 * ptb18 + o19_11 * ptb19 + o20_11 * ptb20 + o21_11 * ptb21 + o22_11 * ptb22 + o23_11 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_10 * Abd0_2 + o0_11 * Abd0_3 + o1_10 * Abd1_2 + o1_11 * Abd1_3 + o2_10 * Abd2_2 + o2_11 * Abd2_3 + o3_10 * Abd3_2 + o3_11 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_10 * Aad0_2 + o0_11 * Aad0_3 + o4_10 * Aad1_2 + o4_11 * Aad1_3 + o8_10 * Aad2_2 + o8_11 * Aad2_3 + o12_10 * Aad3_2 + o12_11 * Aad3_3 + o16_10 * Aad4_2 + o16_11 * Aad4_3 + o20_10 * Aad5_2 + o20_11 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_10 * Abc0_2 + o1_10 * Abc1_2 + o2_10 * Abc2_2 + o3_10 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_10 * Aac0_2 + o4_10 * Aac1_2 + o8_10 * Aac2_2 + o12_10 * Aac3_2 + o16_10 * Aac4_2 + o20_10 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_11 * Abc0_2 + o1_11 * Abc1_2 + o2_11 * Abc2_2 + o3_11 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_11 * Aac0_2 + o4_11 * Aac1_2 + o8_11 * Aac2_2 + o12_11 * Aac3_2 + o16_11 * Aac4_2 + o20_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_10 * Aad0_2 + o1_11 * Aad0_3 + o5_10 * Aad1_2 + o5_11 * Aad1_3 + o9_10 * Aad2_2 + o9_11 * Aad2_3 + o13_10 * Aad3_2 + o13_11 * Aad3_3 + o17_10 * Aad4_2 + o17_11 * Aad4_3 + o21_10 * Aad5_2 + o21_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_10 * Aac0_2 + o5_10 * Aac1_2 + o9_10 * Aac2_2 + o13_10 * Aac3_2 + o17_10 * Aac4_2 + o21_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_11 * Aac0_2 + o5_11 * Aac1_2 + o9_11 * Aac2_2 + o13_11 * Aac3_2 + o17_11 * Aac4_2 + o21_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_10 * Aad0_2 + o2_11 * Aad0_3 + o6_10 * Aad1_2 + o6_11 * Aad1_3 + o10_10 * Aad2_2 + o10_11 * Aad2_3 + o14_10 * Aad3_2 + o14_11 * Aad3_3 + o18_10 * Aad4_2 + o18_11 * Aad4_3 + o22_10 * Aad5_2 + o22_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_10 * Aac0_2 + o6_10 * Aac1_2 + o10_10 * Aac2_2 + o14_10 * Aac3_2 + o18_10 * Aac4_2 + o22_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_11 * Aac0_2 + o6_11 * Aac1_2 + o10_11 * Aac2_2 + o14_11 * Aac3_2 + o18_11 * Aac4_2 + o22_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_10 * Aad0_2 + o3_11 * Aad0_3 + o7_10 * Aad1_2 + o7_11 * Aad1_3 + o11_10 * Aad2_2 + o11_11 * Aad2_3 + o15_10 * Aad3_2 + o15_11 * Aad3_3 + o19_10 * Aad4_2 + o19_11 * Aad4_3 + o23_10 * Aad5_2 + o23_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_10 * Aac0_2 + o7_10 * Aac1_2 + o11_10 * Aac2_2 + o15_10 * Aac3_2 + o19_10 * Aac4_2 + o23_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_11 * Aac0_2 + o7_11 * Aac1_2 + o11_11 * Aac2_2 + o15_11 * Aac3_2 + o19_11 * Aac4_2 + o23_11 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_10 * Abd0_2 + o4_11 * Abd0_3 + o5_10 * Abd1_2 + o5_11 * Abd1_3 + o6_10 * Abd2_2 + o6_11 * Abd2_3 + o7_10 * Abd3_2 + o7_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_10 * Abc0_2 + o5_10 * Abc1_2 + o6_10 * Abc2_2 + o7_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_11 * Abc0_2 + o5_11 * Abc1_2 + o6_11 * Abc2_2 + o7_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_10 * Abd0_2 + o8_11 * Abd0_3 + o9_10 * Abd1_2 + o9_11 * Abd1_3 + o10_10 * Abd2_2 + o10_11 * Abd2_3 + o11_10 * Abd3_2 + o11_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_10 * Abc0_2 + o9_10 * Abc1_2 + o10_10 * Abc2_2 + o11_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_11 * Abc0_2 + o9_11 * Abc1_2 + o10_11 * Abc2_2 + o11_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_10 * Abd0_2 + o12_11 * Abd0_3 + o13_10 * Abd1_2 + o13_11 * Abd1_3 + o14_10 * Abd2_2 + o14_11 * Abd2_3 + o15_10 * Abd3_2 + o15_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_10 * Abc0_2 + o13_10 * Abc1_2 + o14_10 * Abc2_2 + o15_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_11 * Abc0_2 + o13_11 * Abc1_2 + o14_11 * Abc2_2 + o15_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_10 * Abd0_2 + o16_11 * Abd0_3 + o17_10 * Abd1_2 + o17_11 * Abd1_3 + o18_10 * Abd2_2 + o18_11 * Abd2_3 + o19_10 * Abd3_2 + o19_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_10 * Abc0_2 + o17_10 * Abc1_2 + o18_10 * Abc2_2 + o19_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_11 * Abc0_2 + o17_11 * Abc1_2 + o18_11 * Abc2_2 + o19_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_10 * Abd0_2 + o20_11 * Abd0_3 + o21_10 * Abd1_2 + o21_11 * Abd1_3 + o22_10 * Abd2_2 + o22_11 * Abd2_3 + o23_10 * Abd3_2 + o23_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_10 * Abc0_2 + o21_10 * Abc1_2 + o22_10 * Abc2_2 + o23_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_11 * Abc0_2 + o21_11 * Abc1_2 + o22_11 * Abc2_2 + o23_11 * Abc3_2));
          }
        } break;
        case 6: {  // ket functions [12, 13]
          double o0_12 = 0;
          double o0_13 = 0;
          double o1_12 = 0;
          double o1_13 = 0;
          double o2_12 = 0;
          double o2_13 = 0;
          double o3_12 = 0;
          double o3_13 = 0;
          double o4_12 = 0;
          double o4_13 = 0;
          double o5_12 = 0;
          double o5_13 = 0;
          double o6_12 = 0;
          double o6_13 = 0;
          double o7_12 = 0;
          double o7_13 = 0;
          double o8_12 = 0;
          double o8_13 = 0;
          double o9_12 = 0;
          double o9_13 = 0;
          double o10_12 = 0;
          double o10_13 = 0;
          double o11_12 = 0;
          double o11_13 = 0;
          double o12_12 = 0;
          double o12_13 = 0;
          double o13_12 = 0;
          double o13_13 = 0;
          double o14_12 = 0;
          double o14_13 = 0;
          double o15_12 = 0;
          double o15_13 = 0;
          double o16_12 = 0;
          double o16_13 = 0;
          double o17_12 = 0;
          double o17_13 = 0;
          double o18_12 = 0;
          double o18_13 = 0;
          double o19_12 = 0;
          double o19_13 = 0;
          double o20_12 = 0;
          double o20_13 = 0;
          double o21_12 = 0;
          double o21_13 = 0;
          double o22_12 = 0;
          double o22_13 = 0;
          double o23_12 = 0;
          double o23_13 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g12_0 = 0;
            double g12_1 = 0;
            double g12_2 = 0;
            double g12_3 = 0;
            double g12_4 = 0;
            double g12_5 = 0;
            double g12_6 = 0;
            double g12_7 = 0;
            double g12_8 = 0;
            double g12_9 = 0;
            double g12_10 = 0;
            double g12_11 = 0;
            double g12_12 = 0;
            double g12_13 = 0;
            double g12_14 = 0;
            double g12_15 = 0;
            double g12_16 = 0;
            double g12_17 = 0;
            double g12_18 = 0;
            double g12_19 = 0;
            double g13_0 = 0;
            double g13_1 = 0;
            double g13_2 = 0;
            double g13_3 = 0;
            double g13_4 = 0;
            double g13_5 = 0;
            double g13_6 = 0;
            double g13_7 = 0;
            double g13_8 = 0;
            double g13_9 = 0;
            double g13_10 = 0;
            double g13_11 = 0;
            double g13_12 = 0;
            double g13_13 = 0;
            double g13_14 = 0;
            double g13_15 = 0;
            double g13_16 = 0;
            double g13_17 = 0;
            double g13_18 = 0;
            double g13_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek12_0 = kj[62 * kS];
              const double ek12_1 = -kj[63 * kS];
              const double ek12_2 = -kj[64 * kS];
              const double ek12_3 = kj[65 * kS];
              const double ek13_0 = kj[66 * kS];
              const double ek13_1 = -kj[67 * kS];
              const double ek13_2 = -kj[68 * kS];
              const double ek13_3 = kj[69 * kS];
              const double ek13_4 = kj[70 * kS];
              const double ek13_5 = -kj[71 * kS];
              g12_0 = fma(ek12_0, b0, g12_0);
              g13_0 = fma(ek13_0, b0, g13_0);
              const double r0_0_0_1 = Z * b1;
              g12_1 = fma(ek12_0, r0_0_0_1, g12_1);
              g13_1 = fma(ek13_0, r0_0_0_1, g13_1);
              const double r0_0_1_0 = Y * b1;
              g12_2 = fma(ek12_0, r0_0_1_0, g12_2);
              g12_0 = fma(ek12_1, r0_0_1_0, g12_0);
              g13_2 = fma(ek13_0, r0_0_1_0, g13_2);
              g13_0 = fma(ek13_1, r0_0_1_0, g13_0);
              const double r0_1_0_0 = X * b1;
              g12_3 = fma(ek12_0, r0_1_0_0, g12_3);
              g12_0 = fma(ek12_2, r0_1_0_0, g12_0);
              g13_3 = fma(ek13_0, r0_1_0_0, g13_3);
              g13_0 = fma(ek13_2, r0_1_0_0, g13_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g12_4 = fma(ek12_0, r0_0_0_2, g12_4);
              g13_4 = fma(ek13_0, r0_0_0_2, g13_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g12_5 = fma(ek12_0, r0_0_1_1, g12_5);
              g12_1 = fma(ek12_1, r0_0_1_1, g12_1);
              g13_5 = fma(ek13_0, r0_0_1_1, g13_5);
              g13_1 = fma(ek13_1, r0_0_1_1, g13_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g12_6 = fma(ek12_0, r0_0_2_0, g12_6);
              g12_2 = fma(ek12_1, r0_0_2_0, g12_2);
              g13_6 = fma(ek13_0, r0_0_2_0, g13_6);
              g13_2 = fma(ek13_1, r0_0_2_0, g13_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g12_7 = fma(ek12_0, r0_1_0_1, g12_7);
              g12_1 = fma(ek12_2, r0_1_0_1, g12_1);
              g13_7 = fma(ek13_0, r0_1_0_1, g13_7);
              g13_1 = fma(ek13_2, r0_1_0_1, g13_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g12_8 = fma(ek12_0, r0_1_1_0, g12_8);
              g12_3 = fma(ek12_1, r0_1_1_0, g12_3);
              g12_2 = fma(ek12_2, r0_1_1_0, g12_2);
              g12_0 = fma(ek12_3, r0_1_1_0, g12_0);
              g13_8 = fma(ek13_0, r0_1_1_0, g13_8);
              g13_3 = fma(ek13_1, r0_1_1_0, g13_3);
              g13_2 = fma(ek13_2, r0_1_1_0, g13_2);
              g13_0 = fma(ek13_3, r0_1_1_0, g13_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g12_9 = fma(ek12_0, r0_2_0_0, g12_9);
              g12_3 = fma(ek12_2, r0_2_0_0, g12_3);
              g13_9 = fma(ek13_0, r0_2_0_0, g13_9);
              g13_3 = fma(ek13_2, r0_2_0_0, g13_3);
              g13_0 = fma(ek13_4, r0_2_0_0, g13_0);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g12_10 = fma(ek12_0, r0_0_0_3, g12_10);
              g13_10 = fma(ek13_0, r0_0_0_3, g13_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g12_11 = fma(ek12_0, r0_0_1_2, g12_11);
              g12_4 = fma(ek12_1, r0_0_1_2, g12_4);
              g13_11 = fma(ek13_0, r0_0_1_2, g13_11);
              g13_4 = fma(ek13_1, r0_0_1_2, g13_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g12_12 = fma(ek12_0, r0_0_2_1, g12_12);
              g12_5 = fma(ek12_1, r0_0_2_1, g12_5);
              g13_12 = fma(ek13_0, r0_0_2_1, g13_12);
              g13_5 = fma(ek13_1, r0_0_2_1, g13_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g12_13 = fma(ek12_0, r0_0_3_0, g12_13);
              g12_6 = fma(ek12_1, r0_0_3_0, g12_6);
              g13_13 = fma(ek13_0, r0_0_3_0, g13_13);
              g13_6 = fma(ek13_1, r0_0_3_0, g13_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g12_14 = fma(ek12_0, r0_1_0_2, g12_14);
              g12_4 = fma(ek12_2, r0_1_0_2, g12_4);
              g13_14 = fma(ek13_0, r0_1_0_2, g13_14);
              g13_4 = fma(ek13_2, r0_1_0_2, g13_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g12_15 = fma(ek12_0, r0_1_1_1, g12_15);
              g12_7 = fma(ek12_1, r0_1_1_1, g12_7);
              g12_5 = fma(ek12_2, r0_1_1_1, g12_5);
              g12_1 = fma(ek12_3, r0_1_1_1, g12_1);
              g13_15 = fma(ek13_0, r0_1_1_1, g13_15);
              g13_7 = fma(ek13_1, r0_1_1_1, g13_7);
              g13_5 = fma(ek13_2, r0_1_1_1, g13_5);
              g13_1 = fma(ek13_3, r0_1_1_1, g13_1);
              const double r0_1_2_0 = X * r1_0_2_0;
              g12_16 = fma(ek12_0, r0_1_2_0, g12_16);
              g12_8 = fma(ek12_1, r0_1_2_0, g12_8);
              g12_6 = fma(ek12_2, r0_1_2_0, g12_6);
              g12_2 = fma(ek12_3, r0_1_2_0, g12_2);
              g13_16 = fma(ek13_0, r0_1_2_0, g13_16);
              g13_8 = fma(ek13_1, r0_1_2_0, g13_8);
              g13_6 = fma(ek13_2, r0_1_2_0, g13_6);
              g13_2 = fma(ek13_3, r0_1_2_0, g13_2);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g12_17 = fma(ek12_0, r0_2_0_1, g12_17);
              g12_7 = fma(ek12_2, r0_2_0_1, g12_7);
              g13_17 = fma(ek13_0, r0_2_0_1, g13_17);
              g13_7 = fma(ek13_2, r0_2_0_1, g13_7);
              g13_1 = fma(ek13_4, r0_2_0_1, g13_1);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g12_18 = fma(ek12_0, r0_2_1_0, g12_18);
              g12_9 = fma(ek12_1, r0_2_1_0, g12_9);
              g12_8 = fma(ek12_2, r0_2_1_0, g12_8);
              g12_3 = fma(ek12_3, r0_2_1_0, g12_3);
              g13_18 = fma(ek13_0, r0_2_1_0, g13_18);
              g13_9 = fma(ek13_1, r0_2_1_0, g13_9);
              g13_8 = fma(ek13_2, r0_2_1_0, g13_8);
              g13_3 = fma(ek13_3, r0_2_1_0, g13_3);
              g13_2 = fma(ek13_4, r0_2_1_0, g13_2);
              g13_0 = fma(ek13_5, r0_2_1_0, g13_0);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g12_19 = fma(ek12_0, r0_3_0_0, g12_19);
              g12_9 = fma(ek12_2, r0_3_0_0, g12_9);
              g13_19 = fma(ek13_0, r0_3_0_0, g13_19);
              g13_9 = fma(ek13_2, r0_3_0_0, g13_9);
              g13_3 = fma(ek13_4, r0_3_0_0, g13_3);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g12_10 = fma(ek12_1, r0_0_1_3, g12_10);
              g13_10 = fma(ek13_1, r0_0_1_3, g13_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g12_11 = fma(ek12_1, r0_0_2_2, g12_11);
              g13_11 = fma(ek13_1, r0_0_2_2, g13_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g12_12 = fma(ek12_1, r0_0_3_1, g12_12);
              g13_12 = fma(ek13_1, r0_0_3_1, g13_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g12_13 = fma(ek12_1, r0_0_4_0, g12_13);
              g13_13 = fma(ek13_1, r0_0_4_0, g13_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g12_10 = fma(ek12_2, r0_1_0_3, g12_10);
              g13_10 = fma(ek13_2, r0_1_0_3, g13_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g12_14 = fma(ek12_1, r0_1_1_2, g12_14);
              g12_11 = fma(ek12_2, r0_1_1_2, g12_11);
              g12_4 = fma(ek12_3, r0_1_1_2, g12_4);
              g13_14 = fma(ek13_1, r0_1_1_2, g13_14);
              g13_11 = fma(ek13_2, r0_1_1_2, g13_11);
              g13_4 = fma(ek13_3, r0_1_1_2, g13_4);
              const double r0_1_2_1 = X * r1_0_2_1;
              g12_15 = fma(ek12_1, r0_1_2_1, g12_15);
              g12_12 = fma(ek12_2, r0_1_2_1, g12_12);
              g12_5 = fma(ek12_3, r0_1_2_1, g12_5);
              g13_15 = fma(ek13_1, r0_1_2_1, g13_15);
              g13_12 = fma(ek13_2, r0_1_2_1, g13_12);
              g13_5 = fma(ek13_3, r0_1_2_1, g13_5);
              const double r0_1_3_0 = X * r1_0_3_0;
              g12_16 = fma(ek12_1, r0_1_3_0, g12_16);
              g12_13 = fma(ek12_2, r0_1_3_0, g12_13);
              g12_6 = fma(ek12_3, r0_1_3_0, g12_6);
              g13_16 = fma(ek13_1, r0_1_3_0, g13_16);
              g13_13 = fma(ek13_2, r0_1_3_0, g13_13);
              g13_6 = fma(ek13_3, r0_1_3_0, g13_6);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g12_14 = fma(ek12_2, r0_2_0_2, g12_14);
              g13_14 = fma(ek13_2, r0_2_0_2, g13_14);
              g13_4 = fma(ek13_4, r0_2_0_2, g13_4);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g12_17 = fma(ek12_1, r0_2_1_1, g12_17);
              g12_15 = fma(ek12_2, r0_2_1_1, g12_15);
              g12_7 = fma(ek12_3, r0_2_1_1, g12_7);
              g13_17 = fma(ek13_1, r0_2_1_1, g13_17);
              g13_15 = fma(ek13_2, r0_2_1_1, g13_15);
              g13_7 = fma(ek13_3, r0_2_1_1, g13_7);
              g13_5 = fma(ek13_4, r0_2_1_1, g13_5);
              g13_1 = fma(ek13_5, r0_2_1_1, g13_1);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g12_18 = fma(ek12_1, r0_2_2_0, g12_18);
              g12_16 = fma(ek12_2, r0_2_2_0, g12_16);
              g12_8 = fma(ek12_3, r0_2_2_0, g12_8);
              g13_18 = fma(ek13_1, r0_2_2_0, g13_18);
              g13_16 = fma(ek13_2, r0_2_2_0, g13_16);
              g13_8 = fma(ek13_3, r0_2_2_0, g13_8);
              g13_6 = fma(ek13_4, r0_2_2_0, g13_6);
              g13_2 = fma(ek13_5, r0_2_2_0, g13_2);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g12_17 = fma(ek12_2, r0_3_0_1, g12_17);
              g13_17 = fma(ek13_2, r0_3_0_1, g13_17);
              g13_7 = fma(ek13_4, r0_3_0_1, g13_7);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g12_19 = fma(ek12_1, r0_3_1_0, g12_19);
              g12_18 = fma(ek12_2, r0_3_1_0, g12_18);
              g12_9 = fma(ek12_3, r0_3_1_0, g12_9);
              g13_19 = fma(ek13_1, r0_3_1_0, g13_19);
              g13_18 = fma(ek13_2, r0_3_1_0, g13_18);
              g13_9 = fma(ek13_3, r0_3_1_0, g13_9);
              g13_8 = fma(ek13_4, r0_3_1_0, g13_8);
              g13_3 = fma(ek13_5, r0_3_1_0, g13_3);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g12_19 = fma(ek12_2, r0_4_0_0, g12_19);
              g13_19 = fma(ek13_2, r0_4_0_0, g13_19);
              g13_9 = fma(ek13_4, r0_4_0_0, g13_9);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g12_10 = fma(ek12_3, r0_1_1_3, g12_10);
              g13_10 = fma(ek13_3, r0_1_1_3, g13_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g12_11 = fma(ek12_3, r0_1_2_2, g12_11);
              g13_11 = fma(ek13_3, r0_1_2_2, g13_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g12_12 = fma(ek12_3, r0_1_3_1, g12_12);
              g13_12 = fma(ek13_3, r0_1_3_1, g13_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g12_13 = fma(ek12_3, r0_1_4_0, g12_13);
              g13_13 = fma(ek13_3, r0_1_4_0, g13_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g13_10 = fma(ek13_4, r0_2_0_3, g13_10);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g12_14 = fma(ek12_3, r0_2_1_2, g12_14);
              g13_14 = fma(ek13_3, r0_2_1_2, g13_14);
              g13_11 = fma(ek13_4, r0_2_1_2, g13_11);
              g13_4 = fma(ek13_5, r0_2_1_2, g13_4);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g12_15 = fma(ek12_3, r0_2_2_1, g12_15);
              g13_15 = fma(ek13_3, r0_2_2_1, g13_15);
              g13_12 = fma(ek13_4, r0_2_2_1, g13_12);
              g13_5 = fma(ek13_5, r0_2_2_1, g13_5);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g12_16 = fma(ek12_3, r0_2_3_0, g12_16);
              g13_16 = fma(ek13_3, r0_2_3_0, g13_16);
              g13_13 = fma(ek13_4, r0_2_3_0, g13_13);
              g13_6 = fma(ek13_5, r0_2_3_0, g13_6);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g13_14 = fma(ek13_4, r0_3_0_2, g13_14);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g12_17 = fma(ek12_3, r0_3_1_1, g12_17);
              g13_17 = fma(ek13_3, r0_3_1_1, g13_17);
              g13_15 = fma(ek13_4, r0_3_1_1, g13_15);
              g13_7 = fma(ek13_5, r0_3_1_1, g13_7);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g12_18 = fma(ek12_3, r0_3_2_0, g12_18);
              g13_18 = fma(ek13_3, r0_3_2_0, g13_18);
              g13_16 = fma(ek13_4, r0_3_2_0, g13_16);
              g13_8 = fma(ek13_5, r0_3_2_0, g13_8);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g13_17 = fma(ek13_4, r0_4_0_1, g13_17);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g12_19 = fma(ek12_3, r0_4_1_0, g12_19);
              g13_19 = fma(ek13_3, r0_4_1_0, g13_19);
              g13_18 = fma(ek13_4, r0_4_1_0, g13_18);
              g13_9 = fma(ek13_5, r0_4_1_0, g13_9);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g13_19 = fma(ek13_4, r0_5_0_0, g13_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g13_10 = fma(ek13_5, r0_2_1_3, g13_10);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g13_11 = fma(ek13_5, r0_2_2_2, g13_11);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g13_12 = fma(ek13_5, r0_2_3_1, g13_12);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g13_13 = fma(ek13_5, r0_2_4_0, g13_13);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g13_14 = fma(ek13_5, r0_3_1_2, g13_14);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g13_15 = fma(ek13_5, r0_3_2_1, g13_15);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g13_16 = fma(ek13_5, r0_3_3_0, g13_16);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g13_17 = fma(ek13_5, r0_4_1_1, g13_17);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g13_18 = fma(ek13_5, r0_4_2_0, g13_18);
              const double r4_1_1_0 = X * r5_0_1_0;
              const double r3_2_1_0 = fma(X, r4_1_1_0, r4_0_1_0);
              const double r2_3_1_0 = fma(X, r3_2_1_0, 2.0 * r3_1_1_0);
              const double r1_4_1_0 = fma(X, r2_3_1_0, 3.0 * r2_2_1_0);
              const double r0_5_1_0 = fma(X, r1_4_1_0, 4.0 * r1_3_1_0);
              g13_19 = fma(ek13_5, r0_5_1_0, g13_19);
            }
            { const double eb = bi[5];
              o0_12 = fma(eb, g12_0, o0_12);
              o0_13 = fma(eb, g13_0, o0_13);
            }
            { const double eb = bi[6];
              o0_12 = fma(eb, g12_3, o0_12);
              o0_13 = fma(eb, g13_3, o0_13);
            }
            { const double eb = bi[7];
              o0_12 = fma(eb, g12_9, o0_12);
              o0_13 = fma(eb, g13_9, o0_13);
            }
            { const double eb = bi[8];
              o1_12 = fma(eb, g12_0, o1_12);
              o1_13 = fma(eb, g13_0, o1_13);
            }
            { const double eb = bi[9];
              o1_12 = fma(eb, g12_3, o1_12);
              o1_13 = fma(eb, g13_3, o1_13);
            }
            { const double eb = bi[10];
              o1_12 = fma(eb, g12_9, o1_12);
              o1_13 = fma(eb, g13_9, o1_13);
            }
            { const double eb = bi[11];
              o1_12 = fma(eb, g12_19, o1_12);
              o1_13 = fma(eb, g13_19, o1_13);
            }
            { const double eb = bi[12];
              o2_12 = fma(eb, g12_0, o2_12);
              o2_13 = fma(eb, g13_0, o2_13);
            }
            { const double eb = bi[13];
              o2_12 = fma(eb, g12_2, o2_12);
              o2_13 = fma(eb, g13_2, o2_13);
            }
            { const double eb = bi[14];
              o2_12 = fma(eb, g12_3, o2_12);
              o2_13 = fma(eb, g13_3, o2_13);
            }
            { const double eb = bi[15];
              o2_12 = fma(eb, g12_8, o2_12);
              o2_13 = fma(eb, g13_8, o2_13);
            }
            { const double eb = bi[16];
              o2_12 = fma(eb, g12_9, o2_12);
              o2_13 = fma(eb, g13_9, o2_13);
            }
            { const double eb = bi[17];
              o2_12 = fma(eb, g12_18, o2_12);
              o2_13 = fma(eb, g13_18, o2_13);
            }
            { const double eb = bi[18];
              o3_12 = fma(eb, g12_0, o3_12);
              o3_13 = fma(eb, g13_0, o3_13);
            }
            { const double eb = bi[19];
              o3_12 = fma(eb, g12_1, o3_12);
              o3_13 = fma(eb, g13_1, o3_13);
            }
            { const double eb = bi[20];
              o3_12 = fma(eb, g12_3, o3_12);
              o3_13 = fma(eb, g13_3, o3_13);
            }
            { const double eb = bi[21];
              o3_12 = fma(eb, g12_7, o3_12);
              o3_13 = fma(eb, g13_7, o3_13);
            }
            { const double eb = bi[22];
              o3_12 = fma(eb, g12_9, o3_12);
              o3_13 = fma(eb, g13_9, o3_13);
            }
            { const double eb = bi[23];
              o3_12 = fma(eb, g12_17, o3_12);
              o3_13 = fma(eb, g13_17, o3_13);
            }
            { const double eb = bi[24];
              o4_12 = fma(eb, g12_0, o4_12);
              o4_13 = fma(eb, g13_0, o4_13);
            }
            { const double eb = bi[25];
              o4_12 = fma(eb, g12_2, o4_12);
              o4_13 = fma(eb, g13_2, o4_13);
            }
            { const double eb = bi[26];
              o4_12 = fma(eb, g12_6, o4_12);
              o4_13 = fma(eb, g13_6, o4_13);
            }
            { const double eb = bi[27];
              o5_12 = fma(eb, g12_0, o5_12);
              o5_13 = fma(eb, g13_0, o5_13);
            }
            { const double eb = bi[28];
              o5_12 = fma(eb, g12_2, o5_12);
              o5_13 = fma(eb, g13_2, o5_13);
            }
            { const double eb = bi[29];
              o5_12 = fma(eb, g12_6, o5_12);
              o5_13 = fma(eb, g13_6, o5_13);
            }
            { const double eb = bi[30];
              o5_12 = fma(eb, g12_3, o5_12);
              o5_13 = fma(eb, g13_3, o5_13);
            }
            { const double eb = bi[31];
              o5_12 = fma(eb, g12_8, o5_12);
              o5_13 = fma(eb, g13_8, o5_13);
            }
            { const double eb = bi[32];
              o5_12 = fma(eb, g12_16, o5_12);
              o5_13 = fma(eb, g13_16, o5_13);
            }
            { const double eb = bi[33];
              o6_12 = fma(eb, g12_0, o6_12);
              o6_13 = fma(eb, g13_0, o6_13);
            }
            { const double eb = bi[34];
              o6_12 = fma(eb, g12_2, o6_12);
              o6_13 = fma(eb, g13_2, o6_13);
            }
            { const double eb = bi[35];
              o6_12 = fma(eb, g12_6, o6_12);
              o6_13 = fma(eb, g13_6, o6_13);
            }
            { const double eb = bi[36];
              o6_12 = fma(eb, g12_13, o6_12);
              o6_13 = fma(eb, g13_13, o6_13);
            }
            { const double eb = bi[37];
              o7_12 = fma(eb, g12_0, o7_12);
              o7_13 = fma(eb, g13_0, o7_13);
            }
            { const double eb = bi[38];
              o7_12 = fma(eb, g12_1, o7_12);
              o7_13 = fma(eb, g13_1, o7_13);
            }
            { const double eb = bi[39];
              o7_12 = fma(eb, g12_2, o7_12);
              o7_13 = fma(eb, g13_2, o7_13);
            }
            { const double eb = bi[40];
              o7_12 = fma(eb, g12_5, o7_12);
              o7_13 = fma(eb, g13_5, o7_13);
            }
            { const double eb = bi[41];
              o7_12 = fma(eb, g12_6, o7_12);
              o7_13 = fma(eb, g13_6, o7_13);
            }
            { const double eb = bi[42];
              o7_12 = fma(eb, g12_12, o7_12);
              o7_13 = fma(eb, g13_12, o7_13);
            }
            { const double eb = bi[43];
              o8_12 = fma(eb, g12_0, o8_12);
              o8_13 = fma(eb, g13_0, o8_13);
            }
            { const double eb = bi[44];
              o8_12 = fma(eb, g12_1, o8_12);
              o8_13 = fma(eb, g13_1, o8_13);
            }
            { const double eb = bi[45];
              o8_12 = fma(eb, g12_4, o8_12);
              o8_13 = fma(eb, g13_4, o8_13);
            }
            { const double eb = bi[46];
              o9_12 = fma(eb, g12_0, o9_12);
              o9_13 = fma(eb, g13_0, o9_13);
            }
            { const double eb = bi[47];
              o9_12 = fma(eb, g12_1, o9_12);
              o9_13 = fma(eb, g13_1, o9_13);
            }
            { const double eb = bi[48];
              o9_12 = fma(eb, g12_4, o9_12);
              o9_13 = fma(eb, g13_4, o9_13);
            }
            { const double eb = bi[49];
              o9_12 = fma(eb, g12_3, o9_12);
              o9_13 = fma(eb, g13_3, o9_13);
            }
            { const double eb = bi[50];
              o9_12 = fma(eb, g12_7, o9_12);
              o9_13 = fma(eb, g13_7, o9_13);
            }
            { const double eb = bi[51];
              o9_12 = fma(eb, g12_14, o9_12);
              o9_13 = fma(eb, g13_14, o9_13);
            }
            { const double eb = bi[52];
              o10_12 = fma(eb, g12_0, o10_12);
              o10_13 = fma(eb, g13_0, o10_13);
            }
            { const double eb = bi[53];
              o10_12 = fma(eb, g12_1, o10_12);
              o10_13 = fma(eb, g13_1, o10_13);
            }
            { const double eb = bi[54];
              o10_12 = fma(eb, g12_4, o10_12);
              o10_13 = fma(eb, g13_4, o10_13);
            }
            { const double eb = bi[55];
              o10_12 = fma(eb, g12_2, o10_12);
              o10_13 = fma(eb, g13_2, o10_13);
            }
            { const double eb = bi[56];
              o10_12 = fma(eb, g12_5, o10_12);
              o10_13 = fma(eb, g13_5, o10_13);
            }
            { const double eb = bi[57];
              o10_12 = fma(eb, g12_11, o10_12);
              o10_13 = fma(eb, g13_11, o10_13);
            }
            { const double eb = bi[58];
              o11_12 = fma(eb, g12_0, o11_12);
              o11_13 = fma(eb, g13_0, o11_13);
            }
            { const double eb = bi[59];
              o11_12 = fma(eb, g12_1, o11_12);
              o11_13 = fma(eb, g13_1, o11_13);
            }
            { const double eb = bi[60];
              o11_12 = fma(eb, g12_4, o11_12);
              o11_13 = fma(eb, g13_4, o11_13);
            }
            { const double eb = bi[61];
              o11_12 = fma(eb, g12_10, o11_12);
              o11_13 = fma(eb, g13_10, o11_13);
            }
            { const double eb = bi[62];
              o12_12 = fma(eb, g12_0, o12_12);
              o12_13 = fma(eb, g13_0, o12_13);
            }
            { const double eb = bi[63];
              o12_12 = fma(eb, g12_2, o12_12);
              o12_13 = fma(eb, g13_2, o12_13);
            }
            { const double eb = bi[64];
              o12_12 = fma(eb, g12_3, o12_12);
              o12_13 = fma(eb, g13_3, o12_13);
            }
            { const double eb = bi[65];
              o12_12 = fma(eb, g12_8, o12_12);
              o12_13 = fma(eb, g13_8, o12_13);
            }
            { const double eb = bi[66];
              o13_12 = fma(eb, g12_0, o13_12);
              o13_13 = fma(eb, g13_0, o13_13);
            }
            { const double eb = bi[67];
              o13_12 = fma(eb, g12_2, o13_12);
              o13_13 = fma(eb, g13_2, o13_13);
            }
            { const double eb = bi[68];
              o13_12 = fma(eb, g12_3, o13_12);
              o13_13 = fma(eb, g13_3, o13_13);
            }
            { const double eb = bi[69];
              o13_12 = fma(eb, g12_8, o13_12);
              o13_13 = fma(eb, g13_8, o13_13);
            }
            { const double eb = bi[70];
              o13_12 = fma(eb, g12_9, o13_12);
              o13_13 = fma(eb, g13_9, o13_13);
            }
            { const double eb = bi[71];
              o13_12 = fma(eb, g12_18, o13_12);
              o13_13 = fma(eb, g13_18, o13_13);
            }
            { const double eb = bi[72];
              o14_12 = fma(eb, g12_0, o14_12);
              o14_13 = fma(eb, g13_0, o14_13);
            }
            { const double eb = bi[73];
              o14_12 = fma(eb, g12_2, o14_12);
              o14_13 = fma(eb, g13_2, o14_13);
            }
            { const double eb = bi[74];
              o14_12 = fma(eb, g12_6, o14_12);
              o14_13 = fma(eb, g13_6, o14_13);
            }
            { const double eb = bi[75];
              o14_12 = fma(eb, g12_3, o14_12);
              o14_13 = fma(eb, g13_3, o14_13);
            }
            { const double eb = bi[76];
              o14_12 = fma(eb, g12_8, o14_12);
              o14_13 = fma(eb, g13_8, o14_13);
            }
            { const double eb = bi[77];
              o14_12 = fma(eb, g12_16, o14_12);
              o14_13 = fma(eb, g13_16, o14_13);
            }
            { const double eb = bi[78];
              o15_12 = fma(eb, g12_0, o15_12);
              o15_13 = fma(eb, g13_0, o15_13);
            }
            { const double eb = bi[79];
              o15_12 = fma(eb, g12_1, o15_12);
              o15_13 = fma(eb, g13_1, o15_13);
            }
            { const double eb = bi[80];
              o15_12 = fma(eb, g12_2, o15_12);
              o15_13 = fma(eb, g13_2, o15_13);
            }
            { const double eb = bi[81];
              o15_12 = fma(eb, g12_5, o15_12);
              o15_13 = fma(eb, g13_5, o15_13);
            }
            { const double eb = bi[82];
              o15_12 = fma(eb, g12_3, o15_12);
              o15_13 = fma(eb, g13_3, o15_13);
            }
            { const double eb = bi[83];
              o15_12 = fma(eb, g12_7, o15_12);
              o15_13 = fma(eb, g13_7, o15_13);
            }
            { const double eb = bi[84];
              o15_12 = fma(eb, g12_8, o15_12);
              o15_13 = fma(eb, g13_8, o15_13);
            }
            { const double eb = bi[85];
              o15_12 = fma(eb, g12_15, o15_12);
              o15_13 = fma(eb, g13_15, o15_13);
            }
            { const double eb = bi[86];
              o16_12 = fma(eb, g12_0, o16_12);
              o16_13 = fma(eb, g13_0, o16_13);
            }
            { const double eb = bi[87];
              o16_12 = fma(eb, g12_1, o16_12);
              o16_13 = fma(eb, g13_1, o16_13);
            }
            { const double eb = bi[88];
              o16_12 = fma(eb, g12_3, o16_12);
              o16_13 = fma(eb, g13_3, o16_13);
            }
            { const double eb = bi[89];
              o16_12 = fma(eb, g12_7, o16_12);
              o16_13 = fma(eb, g13_7, o16_13);
            }
            { const double eb = bi[90];
              o17_12 = fma(eb, g12_0, o17_12);
              o17_13 = fma(eb, g13_0, o17_13);
            }
            { const double eb = bi[91];
              o17_12 = fma(eb, g12_1, o17_12);
              o17_13 = fma(eb, g13_1, o17_13);
            }
            { const double eb = bi[92];
              o17_12 = fma(eb, g12_3, o17_12);
              o17_13 = fma(eb, g13_3, o17_13);
            }
            { const double eb = bi[93];
              o17_12 = fma(eb, g12_7, o17_12);
              o17_13 = fma(eb, g13_7, o17_13);
            }
            { const double eb = bi[94];
              o17_12 = fma(eb, g12_9, o17_12);
              o17_13 = fma(eb, g13_9, o17_13);
            }
            { const double eb = bi[95];
              o17_12 = fma(eb, g12_17, o17_12);
              o17_13 = fma(eb, g13_17, o17_13);
            }
            { const double eb = bi[96];
              o18_12 = fma(eb, g12_0, o18_12);
              o18_13 = fma(eb, g13_0, o18_13);
            }
            { const double eb = bi[97];
              o18_12 = fma(eb, g12_1, o18_12);
              o18_13 = fma(eb, g13_1, o18_13);
            }
            { const double eb = bi[98];
              o18_12 = fma(eb, g12_2, o18_12);
              o18_13 = fma(eb, g13_2, o18_13);
            }
            { const double eb = bi[99];
              o18_12 = fma(eb, g12_5, o18_12);
              o18_13 = fma(eb, g13_5, o18_13);
            }
            { const double eb = bi[100];
              o18_12 = fma(eb, g12_3, o18_12);
              o18_13 = fma(eb, g13_3, o18_13);
            }
            { const double eb = bi[101];
              o18_12 = fma(eb, g12_7, o18_12);
              o18_13 = fma(eb, g13_7, o18_13);
            }
            { const double eb = bi[102];
              o18_12 = fma(eb, g12_8, o18_12);
              o18_13 = fma(eb, g13_8, o18_13);
            }
            { const double eb = bi[103];
              o18_12 = fma(eb, g12_15, o18_12);
              o18_13 = fma(eb, g13_15, o18_13);
            }
            { const double eb = bi[104];
              o19_12 = fma(eb, g12_0, o19_12);
              o19_13 = fma(eb, g13_0, o19_13);
            }
            { const double eb = bi[105];
              o19_12 = fma(eb, g12_1, o19_12);
              o19_13 = fma(eb, g13_1, o19_13);
            }
            { const double eb = bi[106];
              o19_12 = fma(eb, g12_4, o19_12);
              o19_13 = fma(eb, g13_4, o19_13);
            }
            { const double eb = bi[107];
              o19_12 = fma(eb, g12_3, o19_12);
              o19_13 = fma(eb, g13_3, o19_13);
            }
            { const double eb = bi[108];
              o19_12 = fma(eb, g12_7, o19_12);
              o19_13 = fma(eb, g13_7, o19_13);
            }
            { const double eb = bi[109];
              o19_12 = fma(eb, g12_14, o19_12);
              o19_13 = fma(eb, g13_14, o19_13);
            }
            { const double eb = bi[110];
              o20_12 = fma(eb, g12_0, o20_12);
              o20_13 = fma(eb, g13_0, o20_13);
            }
            { const double eb = bi[111];
              o20_12 = fma(eb, g12_1, o20_12);
              o20_13 = fma(eb, g13_1, o20_13);
            }
            { const double eb = bi[112];
              o20_12 = fma(eb, g12_2, o20_12);
              o20_13 = fma(eb, g13_2, o20_13);
            }
            { const double eb = bi[113];
              o20_12 = fma(eb, g12_5, o20_12);
              o20_13 = fma(eb, g13_5, o20_13);
            }
            { const double eb = bi[114];
              o21_12 = fma(eb, g12_0, o21_12);
              o21_13 = fma(eb, g13_0, o21_13);
            }
            { const double eb = bi[115];
              o21_12 = fma(eb, g12_1, o21_12);
              o21_13 = fma(eb, g13_1, o21_13);
            }
            { const double eb = bi[116];
              o21_12 = fma(eb, g12_2, o21_12);
              o21_13 = fma(eb, g13_2, o21_13);
            }
            { const double eb = bi[117];
              o21_12 = fma(eb, g12_5, o21_12);
              o21_13 = fma(eb, g13_5, o21_13);
            }
            { const double eb = bi[118];
              o21_12 = fma(eb, g12_3, o21_12);
              o21_13 = fma(eb, g13_3, o21_13);
            }
            { const double eb = bi[119];
              o21_12 = fma(eb, g12_7, o21_12);
              o21_13 = fma(eb, g13_7, o21_13);
            }
            { const double eb = bi[120];
              o21_12 = fma(eb, g12_8, o21_12);
              o21_13 = fma(eb, g13_8, o21_13);
            }
            { const double eb = bi[121];
              o21_12 = fma(eb, g12_15, o21_12);
              o21_13 = fma(eb, g13_15, o21_13);
            }
            { const double eb = bi[122];
              o22_12 = fma(eb, g12_0, o22_12);
              o22_13 = fma(eb, g13_0, o22_13);
            }
            { const double eb = bi[123];
              o22_12 = fma(eb, g12_1, o22_12);
              o22_13 = fma(eb, g13_1, o22_13);
            }
            { const double eb = bi[124];
              o22_12 = fma(eb, g12_2, o22_12);
              o22_13 = fma(eb, g13_2, o22_13);
            }
            { const double eb = bi[125];
              o22_12 = fma(eb, g12_5, o22_12);
              o22_13 = fma(eb, g13_5, o22_13);
            }
            { const double eb = bi[126];
              o22_12 = fma(eb, g12_6, o22_12);
              o22_13 = fma(eb, g13_6, o22_13);
            }
            { const double eb = bi[127];
              o22_12 = fma(eb, g12_12, o22_12);
              o22_13 = fma(eb, g13_12, o22_13);
            }
            { const double eb = bi[128];
              o23_12 = fma(eb, g12_0, o23_12);
              o23_13 = fma(eb, g13_0, o23_13);
            }
            { const double eb = bi[129];
              o23_12 = fma(eb, g12_1, o23_12);
              o23_13 = fma(eb, g13_1, o23_13);
            }
            { const double eb = bi[130];
              o23_12 = fma(eb, g12_4, o23_12);
              o23_13 = fma(eb, g13_4, o23_13);
            }
            { const double eb = bi[131];
              o23_12 = fma(eb, g12_2, o23_12);
              o23_13 = fma(eb, g13_2, o23_13);
            }
            { const double eb = bi[132];
              o23_12 = fma(eb, g12_5, o23_12);
              o23_13 = fma(eb, g13_5, o23_13);
            }
            { const double eb = bi[133];
              o23_12 = fma(eb, g12_11, o23_12);
              o23_13 = fma(eb, g13_11, o23_13);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk12 = PT[(fI + 3) * N + fJ + 0];
            const double ptk13 = PT[(fI + 3) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_3 = PA[(fQ + 0) * N + fI + 3];
            const double Abc1_3 = PA[(fQ + 1) * N + fI + 3];
            const double Abc2_3 = PA[(fQ + 2) * N + fI + 3];
            const double Abc3_3 = PA[(fQ + 3) * N + fI + 3];
            const double Aac0_3 = PA[(fP + 0) * N + fI + 3];
            const double Aac1_3 = PA[(fP + 1) * N + fI + 3];
            const double Aac2_3 = PA[(fP + 2) * N + fI + 3];
            const double Aac3_3 = PA[(fP + 3) * N + fI + 3];
            const double Aac4_3 = PA[(fP + 4) * N + fI + 3];
            const double Aac5_3 = PA[(fP + 5) * N + fI + 3];
            jab0 += o0_12 * ptk12 + o0_13 * ptk13;
            jab1 += o1_12 * ptk12 + o1_13 * ptk13;
            jab2 += o2_12 * ptk12 + o2_13 * ptk13;
            jab3 += o3_12 * ptk12 + o3_13 * ptk13;
            jab4 += o4_12 * ptk12 + o4_13 * ptk13;
            jab5 += o5_12 * ptk12 + o5_13 * ptk13;
            jab6 += o6_12 * ptk12 + o6_13 * ptk13;
            jab7 += o7_12 * ptk12 + o7_13 * ptk13;
            jab8 += o8_12 * ptk12 + o8_13 * ptk13;
            jab9 += o9_12 * ptk12 + o9_13 * ptk13;
            jab10 += o10_12 * ptk12 + o10_13 * ptk13;
            jab11 += o11_12 * ptk12 + o11_13 * ptk13;
            jab12 += o12_12 * ptk12 + o12_13 * ptk13;
            jab13 += o13_12 * ptk12 + o13_13 * ptk13;
            jab14 += o14_12 * ptk12 + o14_13 * ptk13;
            jab15 += o15_12 * ptk12 + o15_13 * ptk13;
            jab16 += o16_12 * ptk12 + o16_13 * ptk13;
            jab17 += o17_12 * ptk12 + o17_13 * ptk13;
            jab18 += o18_12 * ptk12 + o18_13 * ptk13;
            jab19 += o19_12 * ptk12 + o19_13 * ptk13;
            jab20 += o20_12 * ptk12 + o20_13 * ptk13;
            jab21 += o21_12 * ptk12 + o21_13 * ptk13;
            jab22 += o22_12 * ptk12 + o22_13 * ptk13;
            jab23 += o23_12 * ptk12 + o23_13 * ptk13;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 0, 2.0 * deg * (o0_12 * ptb0 + o1_12 * ptb1 + o2_12 * ptb2 + o3_12 * ptb3 + o4_12 * ptb4 + o5_12 * ptb5 + o6_12 * ptb6 + o7_12 * ptb7 + o8_12 * ptb8 + o9_12 * ptb9 + o10_12 * ptb10 + o11_12 * ptb11 + o12_12 * ptb12 + o13_12 * ptb13 + o14_12 * ptb14 + o15_12 * ptb15 + o16_12 * ptb16 + o17_12 * ptb17 + o18_12 * ptb18 + o19_12 * ptb19 + o20_12 * ptb20 + o21_12 * ptb21 + o22_12 * ptb22 + o23_12 * ptb23));
            atomicAdd(Jacc + (fI + 3) * N + fJ + 1, 2.0 * deg * (o0_13 * ptb0 + o1_13 * ptb1 + o2_13 * ptb2 + o3_13 * ptb3 + o4_13 * ptb4 + o5_13 * ptb5 + o6_13 * ptb6 + o7_13 * ptb7 + o8_13 * ptb8 + o9_13 * ptb9 + o10_13 * ptb10 + o11_13 * ptb11 + o12_13 * ptb12 + o13_13 * ptb13 + o14_13 * ptb14 + o15_13 * ptb15 + o16_13 * ptb16 + o17_13 * ptb17 + o18_13 * ptb18 + o19_13 * ptb19 + o20_13 * ptb20 + o21_13 * ptb21 + o22_13 * ptb22 + o23_13 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_12 * Abd0_0 + o0_13 * Abd0_1 + o1_12 * Abd1_0 + o1_13 * Abd1_1 + o2_12 * Abd2_0 + o2_13 * Abd2_1 + o3_12 * Abd3_0 + o3_13 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_12 * Aad0_0 + o0_13 * Aad0_1 + o4_12 * Aad1_0 + o4_13 * Aad1_1 + o8_12 * Aad2_0 + o8_13 * Aad2_1 + o12_12 * Aad3_0 + o12_13 * Aad3_1 + o16_12 * Aad4_0 + o16_13 * Aad4_1 + o20_12 * Aad5_0 + o20_13 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_12 * Abc0_3 + o1_12 * Abc1_3 + o2_12 * Abc2_3 + o3_12 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_12 * Aac0_3 + o4_12 * Aac1_3 + o8_12 * Aac2_3 + o12_12 * Aac3_3 + o16_12 * Aac4_3 + o20_12 * Aac5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_13 * Abc0_3 + o1_13 * Abc1_3 + o2_13 * Abc2_3 + o3_13 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_13 * Aac0_3 + o4_13 * Aac1_3 + o8_13 * Aac2_3 + o12_13 * Aac3_3 + o16_13 * Aac4_3 + o20_13 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_12 * Aad0_0 + o1_13 * Aad0_1 + o5_12 * Aad1_0 + o5_13 * Aad1_1 + o9_12 * Aad2_0 + o9_13 * Aad2_1 + o13_12 * Aad3_0 + o13_13 * Aad3_1 + o17_12 * Aad4_0 + o17_13 * Aad4_1 + o21_12 * Aad5_0 + o21_13 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_12 * Aac0_3 + o5_12 * Aac1_3 + o9_12 * Aac2_3 + o13_12 * Aac3_3 + o17_12 * Aac4_3 + o21_12 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_13 * Aac0_3 + o5_13 * Aac1_3 + o9_13 * Aac2_3 + o13_13 * Aac3_3 + o17_13 * Aac4_3 + o21_13 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_12 * Aad0_0 + o2_13 * Aad0_1 + o6_12 * Aad1_0 + o6_13 * Aad1_1 + o10_12 * Aad2_0 + o10_13 * Aad2_1 + o14_12 * Aad3_0 + o14_13 * Aad3_1 + o18_12 * Aad4_0 + o18_13 * Aad4_1 + o22_12 * Aad5_0 + o22_13 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_12 * Aac0_3 + o6_12 * Aac1_3 + o10_12 * Aac2_3 + o14_12 * Aac3_3 + o18_12 * Aac4_3 + o22_12 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_13 * Aac0_3 + o6_13 * Aac1_3 + o10_13 * Aac2_3 + o14_13 * Aac3_3 + o18_13 * Aac4_3 + o22_13 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_12 * Aad0_0 + o3_13 * Aad0_1 + o7_12 * Aad1_0 + o7_13 * Aad1_1 + o11_12 * Aad2_0 + o11_13 * Aad2_1 + o15_12 * Aad3_0 + o15_13 * Aad3_1 + o19_12 * Aad4_0 + o19_13 * Aad4_1 + o23_12 * Aad5_0 + o23_13 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_12 * Aac0_3 + o7_12 * Aac1_3 + o11_12 * Aac2_3 + o15_12 * Aac3_3 + o19_12 * Aac4_3 + o23_12 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_13 * Aac0_3 + o7_13 * Aac1_3 + o11_13 * Aac2_3 + o15_13 * Aac3_3 + o19_13 * Aac4_3 + o23_13 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_12 * Abd0_0 + o4_13 * Abd0_1 + o5_12 * Abd1_0 + o5_13 * Abd1_1 + o6_12 * Abd2_0 + o6_13 * Abd2_1 + o7_12 * Abd3_0 + o7_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_12 * Abc0_3 + o5_12 * Abc1_3 + o6_12 * Abc2_3 + o7_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_13 * Abc0_3 + o5_13 * Abc1_3 + o6_13 * Abc2_3 + o7_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_12 * Abd0_0 + o8_13 * Abd0_1 + o9_12 * Abd1_0 + o9_13 * Abd1_1 + o10_12 * Abd2_0 + o10_13 * Abd2_1 + o11_12 * Abd3_0 + o11_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_12 * Abc0_3 + o9_12 * Abc1_3 + o10_12 * Abc2_3 + o11_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_13 * Abc0_3 + o9_13 * Abc1_3 + o10_13 * Abc2_3 + o11_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_12 * Abd0_0 + o12_13 * Abd0_1 + o13_12 * Abd1_0 + o13_13 * Abd1_1 + o14_12 * Abd2_0 + o14_13 * Abd2_1 + o15_12 * Abd3_0 + o15_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_12 * Abc0_3 + o13_12 * Abc1_3 + o14_12 * Abc2_3 + o15_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_13 * Abc0_3 + o13_13 * Abc1_3 + o14_13 * Abc2_3 + o15_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o16_12 * Abd0_0 + o16_13 * Abd0_1 + o17_12 * Abd1_0 + o17_13 * Abd1_1 + o18_12 * Abd2_0 + o18_13 * Abd2_1 + o19_12 * Abd3_0 + o19_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_12 * Abc0_3 + o17_12 * Abc1_3 + o18_12 * Abc2_3 + o19_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_13 * Abc0_3 + o17_13 * Abc1_3 + o18_13 * Abc2_3 + o19_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o20_12 * Abd0_0 + o20_13 * Abd0_1 + o21_12 * Abd1_0 + o21_13 * Abd1_1 + o22_12 * Abd2_0 + o22_13 * Abd2_1 + o23_12 * Abd3_0 + o23_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_12 * Abc0_3 + o21_12 * Abc1_3 + o22_12 * Abc2_3 + o23_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_13 * Abc0_3 + o21_13 * Abc1_3 + o22_13 * Abc2_3 + o23_13 * Abc3_3));
          }
        } break;
        case 7: {  // ket functions [14, 15]
          double o0_14 = 0;
          double o0_15 = 0;
          double o1_14 = 0;
          double o1_15 = 0;
          double o2_14 = 0;
          double o2_15 = 0;
          double o3_14 = 0;
          double o3_15 = 0;
          double o4_14 = 0;
          double o4_15 = 0;
          double o5_14 = 0;
          double o5_15 = 0;
          double o6_14 = 0;
          double o6_15 = 0;
          double o7_14 = 0;
          double o7_15 = 0;
          double o8_14 = 0;
          double o8_15 = 0;
          double o9_14 = 0;
          double o9_15 = 0;
          double o10_14 = 0;
          double o10_15 = 0;
          double o11_14 = 0;
          double o11_15 = 0;
          double o12_14 = 0;
          double o12_15 = 0;
          double o13_14 = 0;
          double o13_15 = 0;
          double o14_14 = 0;
          double o14_15 = 0;
          double o15_14 = 0;
          double o15_15 = 0;
          double o16_14 = 0;
          double o16_15 = 0;
          double o17_14 = 0;
          double o17_15 = 0;
          double o18_14 = 0;
          double o18_15 = 0;
          double o19_14 = 0;
          double o19_15 = 0;
          double o20_14 = 0;
          double o20_15 = 0;
          double o21_14 = 0;
          double o21_15 = 0;
          double o22_14 = 0;
          double o22_15 = 0;
          double o23_14 = 0;
          double o23_15 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g14_0 = 0;
            double g14_1 = 0;
            double g14_2 = 0;
            double g14_3 = 0;
            double g14_4 = 0;
            double g14_5 = 0;
            double g14_6 = 0;
            double g14_7 = 0;
            double g14_8 = 0;
            double g14_9 = 0;
            double g14_10 = 0;
            double g14_11 = 0;
            double g14_12 = 0;
            double g14_13 = 0;
            double g14_14 = 0;
            double g14_15 = 0;
            double g14_16 = 0;
            double g14_17 = 0;
            double g14_18 = 0;
            double g14_19 = 0;
            double g15_0 = 0;
            double g15_1 = 0;
            double g15_2 = 0;
            double g15_3 = 0;
            double g15_4 = 0;
            double g15_5 = 0;
            double g15_6 = 0;
            double g15_7 = 0;
            double g15_8 = 0;
            double g15_9 = 0;
            double g15_10 = 0;
            double g15_11 = 0;
            double g15_12 = 0;
            double g15_13 = 0;
            double g15_14 = 0;
            double g15_15 = 0;
            double g15_16 = 0;
            double g15_17 = 0;
            double g15_18 = 0;
            double g15_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek14_0 = kj[72 * kS];
              const double ek14_1 = -kj[73 * kS];
              const double ek14_2 = kj[74 * kS];
              const double ek14_3 = -kj[75 * kS];
              const double ek14_4 = kj[76 * kS];
              const double ek14_5 = -kj[77 * kS];
              const double ek15_0 = kj[78 * kS];
              const double ek15_1 = -kj[79 * kS];
              const double ek15_2 = -kj[80 * kS];
              const double ek15_3 = kj[81 * kS];
              const double ek15_4 = -kj[82 * kS];
              const double ek15_5 = kj[83 * kS];
              const double ek15_6 = kj[84 * kS];
              const double ek15_7 = -kj[85 * kS];
              g14_0 = fma(ek14_0, b0, g14_0);
              g15_0 = fma(ek15_0, b0, g15_0);
              const double r0_0_0_1 = Z * b1;
              g14_1 = fma(ek14_0, r0_0_0_1, g14_1);
              g15_1 = fma(ek15_0, r0_0_0_1, g15_1);
              g15_0 = fma(ek15_1, r0_0_0_1, g15_0);
              const double r0_0_1_0 = Y * b1;
              g14_2 = fma(ek14_0, r0_0_1_0, g14_2);
              g14_0 = fma(ek14_1, r0_0_1_0, g14_0);
              g15_2 = fma(ek15_0, r0_0_1_0, g15_2);
              g15_0 = fma(ek15_2, r0_0_1_0, g15_0);
              const double r0_1_0_0 = X * b1;
              g14_3 = fma(ek14_0, r0_1_0_0, g14_3);
              g14_0 = fma(ek14_3, r0_1_0_0, g14_0);
              g15_3 = fma(ek15_0, r0_1_0_0, g15_3);
              g15_0 = fma(ek15_4, r0_1_0_0, g15_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g14_4 = fma(ek14_0, r0_0_0_2, g14_4);
              g15_4 = fma(ek15_0, r0_0_0_2, g15_4);
              g15_1 = fma(ek15_1, r0_0_0_2, g15_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g14_5 = fma(ek14_0, r0_0_1_1, g14_5);
              g14_1 = fma(ek14_1, r0_0_1_1, g14_1);
              g15_5 = fma(ek15_0, r0_0_1_1, g15_5);
              g15_2 = fma(ek15_1, r0_0_1_1, g15_2);
              g15_1 = fma(ek15_2, r0_0_1_1, g15_1);
              g15_0 = fma(ek15_3, r0_0_1_1, g15_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g14_6 = fma(ek14_0, r0_0_2_0, g14_6);
              g14_2 = fma(ek14_1, r0_0_2_0, g14_2);
              g14_0 = fma(ek14_2, r0_0_2_0, g14_0);
              g15_6 = fma(ek15_0, r0_0_2_0, g15_6);
              g15_2 = fma(ek15_2, r0_0_2_0, g15_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g14_7 = fma(ek14_0, r0_1_0_1, g14_7);
              g14_1 = fma(ek14_3, r0_1_0_1, g14_1);
              g15_7 = fma(ek15_0, r0_1_0_1, g15_7);
              g15_3 = fma(ek15_1, r0_1_0_1, g15_3);
              g15_1 = fma(ek15_4, r0_1_0_1, g15_1);
              g15_0 = fma(ek15_5, r0_1_0_1, g15_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g14_8 = fma(ek14_0, r0_1_1_0, g14_8);
              g14_3 = fma(ek14_1, r0_1_1_0, g14_3);
              g14_2 = fma(ek14_3, r0_1_1_0, g14_2);
              g14_0 = fma(ek14_4, r0_1_1_0, g14_0);
              g15_8 = fma(ek15_0, r0_1_1_0, g15_8);
              g15_3 = fma(ek15_2, r0_1_1_0, g15_3);
              g15_2 = fma(ek15_4, r0_1_1_0, g15_2);
              g15_0 = fma(ek15_6, r0_1_1_0, g15_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g14_9 = fma(ek14_0, r0_2_0_0, g14_9);
              g14_3 = fma(ek14_3, r0_2_0_0, g14_3);
              g15_9 = fma(ek15_0, r0_2_0_0, g15_9);
              g15_3 = fma(ek15_4, r0_2_0_0, g15_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g14_10 = fma(ek14_0, r0_0_0_3, g14_10);
              g15_10 = fma(ek15_0, r0_0_0_3, g15_10);
              g15_4 = fma(ek15_1, r0_0_0_3, g15_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g14_11 = fma(ek14_0, r0_0_1_2, g14_11);
              g14_4 = fma(ek14_1, r0_0_1_2, g14_4);
              g15_11 = fma(ek15_0, r0_0_1_2, g15_11);
              g15_5 = fma(ek15_1, r0_0_1_2, g15_5);
              g15_4 = fma(ek15_2, r0_0_1_2, g15_4);
              g15_1 = fma(ek15_3, r0_0_1_2, g15_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g14_12 = fma(ek14_0, r0_0_2_1, g14_12);
              g14_5 = fma(ek14_1, r0_0_2_1, g14_5);
              g14_1 = fma(ek14_2, r0_0_2_1, g14_1);
              g15_12 = fma(ek15_0, r0_0_2_1, g15_12);
              g15_6 = fma(ek15_1, r0_0_2_1, g15_6);
              g15_5 = fma(ek15_2, r0_0_2_1, g15_5);
              g15_2 = fma(ek15_3, r0_0_2_1, g15_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g14_13 = fma(ek14_0, r0_0_3_0, g14_13);
              g14_6 = fma(ek14_1, r0_0_3_0, g14_6);
              g14_2 = fma(ek14_2, r0_0_3_0, g14_2);
              g15_13 = fma(ek15_0, r0_0_3_0, g15_13);
              g15_6 = fma(ek15_2, r0_0_3_0, g15_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g14_14 = fma(ek14_0, r0_1_0_2, g14_14);
              g14_4 = fma(ek14_3, r0_1_0_2, g14_4);
              g15_14 = fma(ek15_0, r0_1_0_2, g15_14);
              g15_7 = fma(ek15_1, r0_1_0_2, g15_7);
              g15_4 = fma(ek15_4, r0_1_0_2, g15_4);
              g15_1 = fma(ek15_5, r0_1_0_2, g15_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g14_15 = fma(ek14_0, r0_1_1_1, g14_15);
              g14_7 = fma(ek14_1, r0_1_1_1, g14_7);
              g14_5 = fma(ek14_3, r0_1_1_1, g14_5);
              g14_1 = fma(ek14_4, r0_1_1_1, g14_1);
              g15_15 = fma(ek15_0, r0_1_1_1, g15_15);
              g15_8 = fma(ek15_1, r0_1_1_1, g15_8);
              g15_7 = fma(ek15_2, r0_1_1_1, g15_7);
              g15_3 = fma(ek15_3, r0_1_1_1, g15_3);
              g15_5 = fma(ek15_4, r0_1_1_1, g15_5);
              g15_2 = fma(ek15_5, r0_1_1_1, g15_2);
              g15_1 = fma(ek15_6, r0_1_1_1, g15_1);
              g15_0 = fma(ek15_7, r0_1_1_1, g15_0);
              const double r0_1_2_0 = X * r1_0_2_0;
              g14_16 = fma(ek14_0, r0_1_2_0, g14_16);
              g14_8 = fma(ek14_1, r0_1_2_0, g14_8);
              g14_3 = fma(ek14_2, r0_1_2_0, g14_3);
              g14_6 = fma(ek14_3, r0_1_2_0, g14_6);
              g14_2 = fma(ek14_4, r0_1_2_0, g14_2);
              g14_0 = fma(ek14_5, r0_1_2_0, g14_0);
              g15_16 = fma(ek15_0, r0_1_2_0, g15_16);
              g15_8 = fma(ek15_2, r0_1_2_0, g15_8);
              g15_6 = fma(ek15_4, r0_1_2_0, g15_6);
              g15_2 = fma(ek15_6, r0_1_2_0, g15_2);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g14_17 = fma(ek14_0, r0_2_0_1, g14_17);
              g14_7 = fma(ek14_3, r0_2_0_1, g14_7);
              g15_17 = fma(ek15_0, r0_2_0_1, g15_17);
              g15_9 = fma(ek15_1, r0_2_0_1, g15_9);
              g15_7 = fma(ek15_4, r0_2_0_1, g15_7);
              g15_3 = fma(ek15_5, r0_2_0_1, g15_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g14_18 = fma(ek14_0, r0_2_1_0, g14_18);
              g14_9 = fma(ek14_1, r0_2_1_0, g14_9);
              g14_8 = fma(ek14_3, r0_2_1_0, g14_8);
              g14_3 = fma(ek14_4, r0_2_1_0, g14_3);
              g15_18 = fma(ek15_0, r0_2_1_0, g15_18);
              g15_9 = fma(ek15_2, r0_2_1_0, g15_9);
              g15_8 = fma(ek15_4, r0_2_1_0, g15_8);
              g15_3 = fma(ek15_6, r0_2_1_0, g15_3);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g14_19 = fma(ek14_0, r0_3_0_0, g14_19);
              g14_9 = fma(ek14_3, r0_3_0_0, g14_9);
              g15_19 = fma(ek15_0, r0_3_0_0, g15_19);
              g15_9 = fma(ek15_4, r0_3_0_0, g15_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g15_10 = fma(ek15_1, r0_0_0_4, g15_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g14_10 = fma(ek14_1, r0_0_1_3, g14_10);
              g15_11 = fma(ek15_1, r0_0_1_3, g15_11);
              g15_10 = fma(ek15_2, r0_0_1_3, g15_10);
              g15_4 = fma(ek15_3, r0_0_1_3, g15_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g14_11 = fma(ek14_1, r0_0_2_2, g14_11);
              g14_4 = fma(ek14_2, r0_0_2_2, g14_4);
              g15_12 = fma(ek15_1, r0_0_2_2, g15_12);
              g15_11 = fma(ek15_2, r0_0_2_2, g15_11);
              g15_5 = fma(ek15_3, r0_0_2_2, g15_5);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g14_12 = fma(ek14_1, r0_0_3_1, g14_12);
              g14_5 = fma(ek14_2, r0_0_3_1, g14_5);
              g15_13 = fma(ek15_1, r0_0_3_1, g15_13);
              g15_12 = fma(ek15_2, r0_0_3_1, g15_12);
              g15_6 = fma(ek15_3, r0_0_3_1, g15_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g14_13 = fma(ek14_1, r0_0_4_0, g14_13);
              g14_6 = fma(ek14_2, r0_0_4_0, g14_6);
              g15_13 = fma(ek15_2, r0_0_4_0, g15_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g14_10 = fma(ek14_3, r0_1_0_3, g14_10);
              g15_14 = fma(ek15_1, r0_1_0_3, g15_14);
              g15_10 = fma(ek15_4, r0_1_0_3, g15_10);
              g15_4 = fma(ek15_5, r0_1_0_3, g15_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g14_14 = fma(ek14_1, r0_1_1_2, g14_14);
              g14_11 = fma(ek14_3, r0_1_1_2, g14_11);
              g14_4 = fma(ek14_4, r0_1_1_2, g14_4);
              g15_15 = fma(ek15_1, r0_1_1_2, g15_15);
              g15_14 = fma(ek15_2, r0_1_1_2, g15_14);
              g15_7 = fma(ek15_3, r0_1_1_2, g15_7);
              g15_11 = fma(ek15_4, r0_1_1_2, g15_11);
              g15_5 = fma(ek15_5, r0_1_1_2, g15_5);
              g15_4 = fma(ek15_6, r0_1_1_2, g15_4);
              g15_1 = fma(ek15_7, r0_1_1_2, g15_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g14_15 = fma(ek14_1, r0_1_2_1, g14_15);
              g14_7 = fma(ek14_2, r0_1_2_1, g14_7);
              g14_12 = fma(ek14_3, r0_1_2_1, g14_12);
              g14_5 = fma(ek14_4, r0_1_2_1, g14_5);
              g14_1 = fma(ek14_5, r0_1_2_1, g14_1);
              g15_16 = fma(ek15_1, r0_1_2_1, g15_16);
              g15_15 = fma(ek15_2, r0_1_2_1, g15_15);
              g15_8 = fma(ek15_3, r0_1_2_1, g15_8);
              g15_12 = fma(ek15_4, r0_1_2_1, g15_12);
              g15_6 = fma(ek15_5, r0_1_2_1, g15_6);
              g15_5 = fma(ek15_6, r0_1_2_1, g15_5);
              g15_2 = fma(ek15_7, r0_1_2_1, g15_2);
              const double r0_1_3_0 = X * r1_0_3_0;
              g14_16 = fma(ek14_1, r0_1_3_0, g14_16);
              g14_8 = fma(ek14_2, r0_1_3_0, g14_8);
              g14_13 = fma(ek14_3, r0_1_3_0, g14_13);
              g14_6 = fma(ek14_4, r0_1_3_0, g14_6);
              g14_2 = fma(ek14_5, r0_1_3_0, g14_2);
              g15_16 = fma(ek15_2, r0_1_3_0, g15_16);
              g15_13 = fma(ek15_4, r0_1_3_0, g15_13);
              g15_6 = fma(ek15_6, r0_1_3_0, g15_6);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g14_14 = fma(ek14_3, r0_2_0_2, g14_14);
              g15_17 = fma(ek15_1, r0_2_0_2, g15_17);
              g15_14 = fma(ek15_4, r0_2_0_2, g15_14);
              g15_7 = fma(ek15_5, r0_2_0_2, g15_7);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g14_17 = fma(ek14_1, r0_2_1_1, g14_17);
              g14_15 = fma(ek14_3, r0_2_1_1, g14_15);
              g14_7 = fma(ek14_4, r0_2_1_1, g14_7);
              g15_18 = fma(ek15_1, r0_2_1_1, g15_18);
              g15_17 = fma(ek15_2, r0_2_1_1, g15_17);
              g15_9 = fma(ek15_3, r0_2_1_1, g15_9);
              g15_15 = fma(ek15_4, r0_2_1_1, g15_15);
              g15_8 = fma(ek15_5, r0_2_1_1, g15_8);
              g15_7 = fma(ek15_6, r0_2_1_1, g15_7);
              g15_3 = fma(ek15_7, r0_2_1_1, g15_3);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g14_18 = fma(ek14_1, r0_2_2_0, g14_18);
              g14_9 = fma(ek14_2, r0_2_2_0, g14_9);
              g14_16 = fma(ek14_3, r0_2_2_0, g14_16);
              g14_8 = fma(ek14_4, r0_2_2_0, g14_8);
              g14_3 = fma(ek14_5, r0_2_2_0, g14_3);
              g15_18 = fma(ek15_2, r0_2_2_0, g15_18);
              g15_16 = fma(ek15_4, r0_2_2_0, g15_16);
              g15_8 = fma(ek15_6, r0_2_2_0, g15_8);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g14_17 = fma(ek14_3, r0_3_0_1, g14_17);
              g15_19 = fma(ek15_1, r0_3_0_1, g15_19);
              g15_17 = fma(ek15_4, r0_3_0_1, g15_17);
              g15_9 = fma(ek15_5, r0_3_0_1, g15_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g14_19 = fma(ek14_1, r0_3_1_0, g14_19);
              g14_18 = fma(ek14_3, r0_3_1_0, g14_18);
              g14_9 = fma(ek14_4, r0_3_1_0, g14_9);
              g15_19 = fma(ek15_2, r0_3_1_0, g15_19);
              g15_18 = fma(ek15_4, r0_3_1_0, g15_18);
              g15_9 = fma(ek15_6, r0_3_1_0, g15_9);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g14_19 = fma(ek14_3, r0_4_0_0, g14_19);
              g15_19 = fma(ek15_4, r0_4_0_0, g15_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g15_10 = fma(ek15_3, r0_0_1_4, g15_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g14_10 = fma(ek14_2, r0_0_2_3, g14_10);
              g15_11 = fma(ek15_3, r0_0_2_3, g15_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g14_11 = fma(ek14_2, r0_0_3_2, g14_11);
              g15_12 = fma(ek15_3, r0_0_3_2, g15_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g14_12 = fma(ek14_2, r0_0_4_1, g14_12);
              g15_13 = fma(ek15_3, r0_0_4_1, g15_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g14_13 = fma(ek14_2, r0_0_5_0, g14_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g15_10 = fma(ek15_5, r0_1_0_4, g15_10);
              const double r0_1_1_3 = X * r1_0_1_3;
              g14_10 = fma(ek14_4, r0_1_1_3, g14_10);
              g15_14 = fma(ek15_3, r0_1_1_3, g15_14);
              g15_11 = fma(ek15_5, r0_1_1_3, g15_11);
              g15_10 = fma(ek15_6, r0_1_1_3, g15_10);
              g15_4 = fma(ek15_7, r0_1_1_3, g15_4);
              const double r0_1_2_2 = X * r1_0_2_2;
              g14_14 = fma(ek14_2, r0_1_2_2, g14_14);
              g14_11 = fma(ek14_4, r0_1_2_2, g14_11);
              g14_4 = fma(ek14_5, r0_1_2_2, g14_4);
              g15_15 = fma(ek15_3, r0_1_2_2, g15_15);
              g15_12 = fma(ek15_5, r0_1_2_2, g15_12);
              g15_11 = fma(ek15_6, r0_1_2_2, g15_11);
              g15_5 = fma(ek15_7, r0_1_2_2, g15_5);
              const double r0_1_3_1 = X * r1_0_3_1;
              g14_15 = fma(ek14_2, r0_1_3_1, g14_15);
              g14_12 = fma(ek14_4, r0_1_3_1, g14_12);
              g14_5 = fma(ek14_5, r0_1_3_1, g14_5);
              g15_16 = fma(ek15_3, r0_1_3_1, g15_16);
              g15_13 = fma(ek15_5, r0_1_3_1, g15_13);
              g15_12 = fma(ek15_6, r0_1_3_1, g15_12);
              g15_6 = fma(ek15_7, r0_1_3_1, g15_6);
              const double r0_1_4_0 = X * r1_0_4_0;
              g14_16 = fma(ek14_2, r0_1_4_0, g14_16);
              g14_13 = fma(ek14_4, r0_1_4_0, g14_13);
              g14_6 = fma(ek14_5, r0_1_4_0, g14_6);
              g15_13 = fma(ek15_6, r0_1_4_0, g15_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g15_14 = fma(ek15_5, r0_2_0_3, g15_14);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g14_14 = fma(ek14_4, r0_2_1_2, g14_14);
              g15_17 = fma(ek15_3, r0_2_1_2, g15_17);
              g15_15 = fma(ek15_5, r0_2_1_2, g15_15);
              g15_14 = fma(ek15_6, r0_2_1_2, g15_14);
              g15_7 = fma(ek15_7, r0_2_1_2, g15_7);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g14_17 = fma(ek14_2, r0_2_2_1, g14_17);
              g14_15 = fma(ek14_4, r0_2_2_1, g14_15);
              g14_7 = fma(ek14_5, r0_2_2_1, g14_7);
              g15_18 = fma(ek15_3, r0_2_2_1, g15_18);
              g15_16 = fma(ek15_5, r0_2_2_1, g15_16);
              g15_15 = fma(ek15_6, r0_2_2_1, g15_15);
              g15_8 = fma(ek15_7, r0_2_2_1, g15_8);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g14_18 = fma(ek14_2, r0_2_3_0, g14_18);
              g14_16 = fma(ek14_4, r0_2_3_0, g14_16);
              g14_8 = fma(ek14_5, r0_2_3_0, g14_8);
              g15_16 = fma(ek15_6, r0_2_3_0, g15_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g15_17 = fma(ek15_5, r0_3_0_2, g15_17);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g14_17 = fma(ek14_4, r0_3_1_1, g14_17);
              g15_19 = fma(ek15_3, r0_3_1_1, g15_19);
              g15_18 = fma(ek15_5, r0_3_1_1, g15_18);
              g15_17 = fma(ek15_6, r0_3_1_1, g15_17);
              g15_9 = fma(ek15_7, r0_3_1_1, g15_9);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g14_19 = fma(ek14_2, r0_3_2_0, g14_19);
              g14_18 = fma(ek14_4, r0_3_2_0, g14_18);
              g14_9 = fma(ek14_5, r0_3_2_0, g14_9);
              g15_18 = fma(ek15_6, r0_3_2_0, g15_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g15_19 = fma(ek15_5, r0_4_0_1, g15_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g14_19 = fma(ek14_4, r0_4_1_0, g14_19);
              g15_19 = fma(ek15_6, r0_4_1_0, g15_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_1_1_4 = X * r1_0_1_4;
              g15_10 = fma(ek15_7, r0_1_1_4, g15_10);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g14_10 = fma(ek14_5, r0_1_2_3, g14_10);
              g15_11 = fma(ek15_7, r0_1_2_3, g15_11);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g14_11 = fma(ek14_5, r0_1_3_2, g14_11);
              g15_12 = fma(ek15_7, r0_1_3_2, g15_12);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_1_4_1 = X * r1_0_4_1;
              g14_12 = fma(ek14_5, r0_1_4_1, g14_12);
              g15_13 = fma(ek15_7, r0_1_4_1, g15_13);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_0_5_0 = fma(Y, r2_0_4_0, 4.0 * r2_0_3_0);
              const double r0_1_5_0 = X * r1_0_5_0;
              g14_13 = fma(ek14_5, r0_1_5_0, g14_13);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g15_14 = fma(ek15_7, r0_2_1_3, g15_14);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g14_14 = fma(ek14_5, r0_2_2_2, g14_14);
              g15_15 = fma(ek15_7, r0_2_2_2, g15_15);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g14_15 = fma(ek14_5, r0_2_3_1, g14_15);
              g15_16 = fma(ek15_7, r0_2_3_1, g15_16);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g14_16 = fma(ek14_5, r0_2_4_0, g14_16);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g15_17 = fma(ek15_7, r0_3_1_2, g15_17);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g14_17 = fma(ek14_5, r0_3_2_1, g14_17);
              g15_18 = fma(ek15_7, r0_3_2_1, g15_18);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g14_18 = fma(ek14_5, r0_3_3_0, g14_18);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g15_19 = fma(ek15_7, r0_4_1_1, g15_19);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g14_19 = fma(ek14_5, r0_4_2_0, g14_19);
            }
            { const double eb = bi[5];
              o0_14 = fma(eb, g14_0, o0_14);
              o0_15 = fma(eb, g15_0, o0_15);
            }
            { const double eb = bi[6];
              o0_14 = fma(eb, g14_3, o0_14);
              o0_15 = fma(eb, g15_3, o0_15);
            }
            { const double eb = bi[7];
              o0_14 = fma(eb, g14_9, o0_14);
              o0_15 = fma(eb, g15_9, o0_15);
            }
            { const double eb = bi[8];
              o1_14 = fma(eb, g14_0, o1_14);
              o1_15 = fma(eb, g15_0, o1_15);
            }
            { const double eb = bi[9];
              o1_14 = fma(eb, g14_3, o1_14);
              o1_15 = fma(eb, g15_3, o1_15);
            }
            { const double eb = bi[10];
              o1_14 = fma(eb, g14_9, o1_14);
              o1_15 = fma(eb, g15_9, o1_15);
            }
            { const double eb = bi[11];
              o1_14 = fma(eb, g14_19, o1_14);
              o1_15 = fma(eb, g15_19, o1_15);
            }
            { const double eb = bi[12];
              o2_14 = fma(eb, g14_0, o2_14);
              o2_15 = fma(eb, g15_0, o2_15);
            }
            { const double eb = bi[13];
              o2_14 = fma(eb, g14_2, o2_14);
              o2_15 = fma(eb, g15_2, o2_15);
            }
            { const double eb = bi[14];
              o2_14 = fma(eb, g14_3, o2_14);
              o2_15 = fma(eb, g15_3, o2_15);
            }
            { const double eb = bi[15];
              o2_14 = fma(eb, g14_8, o2_14);
              o2_15 = fma(eb, g15_8, o2_15);
            }
            { const double eb = bi[16];
              o2_14 = fma(eb, g14_9, o2_14);
              o2_15 = fma(eb, g15_9, o2_15);
            }
            { const double eb = bi[17];
              o2_14 = fma(eb, g14_18, o2_14);
              o2_15 = fma(eb, g15_18, o2_15);
            }
            { const double eb = bi[18];
              o3_14 = fma(eb, g14_0, o3_14);
              o3_15 = fma(eb, g15_0, o3_15);
            }
            { const double eb = bi[19];
              o3_14 = fma(eb, g14_1, o3_14);
              o3_15 = fma(eb, g15_1, o3_15);
            }
            { const double eb = bi[20];
              o3_14 = fma(eb, g14_3, o3_14);
              o3_15 = fma(eb, g15_3, o3_15);
            }
            { const double eb = bi[21];
              o3_14 = fma(eb, g14_7, o3_14);
              o3_15 = fma(eb, g15_7, o3_15);
            }
            { const double eb = bi[22];
              o3_14 = fma(eb, g14_9, o3_14);
              o3_15 = fma(eb, g15_9, o3_15);
            }
            { const double eb = bi[23];
              o3_14 = fma(eb, g14_17, o3_14);
              o3_15 = fma(eb, g15_17, o3_15);
            }
            { const double eb = bi[24];
              o4_14 = fma(eb, g14_0, o4_14);
              o4_15 = fma(eb, g15_0, o4_15);
            }
            { const double eb = bi[25];
              o4_14 = fma(eb, g14_2, o4_14);
              o4_15 = fma(eb, g15_2, o4_15);
            }
            { const double eb = bi[26];
              o4_14 = fma(eb, g14_6, o4_14);
              o4_15 = fma(eb, g15_6, o4_15);
            }
            { const double eb = bi[27];
              o5_14 = fma(eb, g14_0, o5_14);
              o5_15 = fma(eb, g15_0, o5_15);
            }
            { const double eb = bi[28];
              o5_14 = fma(eb, g14_2, o5_14);
              o5_15 = fma(eb, g15_2, o5_15);
            }
            { const double eb = bi[29];
              o5_14 = fma(eb, g14_6, o5_14);
              o5_15 = fma(eb, g15_6, o5_15);
            }
            { const double eb = bi[30];
              o5_14 = fma(eb, g14_3, o5_14);
              o5_15 = fma(eb, g15_3, o5_15);
            }
            { const double eb = bi[31];
              o5_14 = fma(eb, g14_8, o5_14);
              o5_15 = fma(eb, g15_8, o5_15);
            }
            { const double eb = bi[32];
              o5_14 = fma(eb, g14_16, o5_14);
              o5_15 = fma(eb, g15_16, o5_15);
            }
            { const double eb = bi[33];
              o6_14 = fma(eb, g14_0, o6_14);
              o6_15 = fma(eb, g15_0, o6_15);
            }
            { const double eb = bi[34];
              o6_14 = fma(eb, g14_2, o6_14);
              o6_15 = fma(eb, g15_2, o6_15);
            }
            { const double eb = bi[35];
              o6_14 = fma(eb, g14_6, o6_14);
              o6_15 = fma(eb, g15_6, o6_15);
            }
            { const double eb = bi[36];
              o6_14 = fma(eb, g14_13, o6_14);
              o6_15 = fma(eb, g15_13, o6_15);
            }
            { const double eb = bi[37];
              o7_14 = fma(eb, g14_0, o7_14);
              o7_15 = fma(eb, g15_0, o7_15);
            }
            { const double eb = bi[38];
              o7_14 = fma(eb, g14_1, o7_14);
              o7_15 = fma(eb, g15_1, o7_15);
            }
            { const double eb = bi[39];
              o7_14 = fma(eb, g14_2, o7_14);
              o7_15 = fma(eb, g15_2, o7_15);
            }
            { const double eb = bi[40];
              o7_14 = fma(eb, g14_5, o7_14);
              o7_15 = fma(eb, g15_5, o7_15);
            }
            { const double eb = bi[41];
              o7_14 = fma(eb, g14_6, o7_14);
              o7_15 = fma(eb, g15_6, o7_15);
            }
            { const double eb = bi[42];
              o7_14 = fma(eb, g14_12, o7_14);
              o7_15 = fma(eb, g15_12, o7_15);
            }
            { const double eb = bi[43];
              o8_14 = fma(eb, g14_0, o8_14);
              o8_15 = fma(eb, g15_0, o8_15);
            }
            { const double eb = bi[44];
              o8_14 = fma(eb, g14_1, o8_14);
              o8_15 = fma(eb, g15_1, o8_15);
            }
            { const double eb = bi[45];
              o8_14 = fma(eb, g14_4, o8_14);
              o8_15 = fma(eb, g15_4, o8_15);
            }
            { const double eb = bi[46];
              o9_14 = fma(eb, g14_0, o9_14);
              o9_15 = fma(eb, g15_0, o9_15);
            }
            { const double eb = bi[47];
              o9_14 = fma(eb, g14_1, o9_14);
              o9_15 = fma(eb, g15_1, o9_15);
            }
            { const double eb = bi[48];
              o9_14 = fma(eb, g14_4, o9_14);
              o9_15 = fma(eb, g15_4, o9_15);
            }
            { const double eb = bi[49];
              o9_14 = fma(eb, g14_3, o9_14);
              o9_15 = fma(eb, g15_3, o9_15);
            }
            { const double eb = bi[50];
              o9_14 = fma(eb, g14_7, o9_14);
              o9_15 = fma(eb, g15_7, o9_15);
            }
            { const double eb = bi[51];
              o9_14 = fma(eb, g14_14, o9_14);
              o9_15 = fma(eb, g15_14, o9_15);
            }
            { const double eb = bi[52];
              o10_14 = fma(eb, g14_0, o10_14);
              o10_15 = fma(eb, g15_0, o10_15);
            }
            { const double eb = bi[53];
              o10_14 = fma(eb, g14_1, o10_14);
              o10_15 = fma(eb, g15_1, o10_15);
            }
            { const double eb = bi[54];
              o10_14 = fma(eb, g14_4, o10_14);
              o10_15 = fma(eb, g15_4, o10_15);
            }
            { const double eb = bi[55];
              o10_14 = fma(eb, g14_2, o10_14);
              o10_15 = fma(eb, g15_2, o10_15);
            }
            { const double eb = bi[56];
              o10_14 = fma(eb, g14_5, o10_14);
              o10_15 = fma(eb, g15_5, o10_15);
            }
            { const double eb = bi[57];
              o10_14 = fma(eb, g14_11, o10_14);
              o10_15 = fma(eb, g15_11, o10_15);
            }
            { const double eb = bi[58];
              o11_14 = fma(eb, g14_0, o11_14);
              o11_15 = fma(eb, g15_0, o11_15);
            }
            { const double eb = bi[59];
              o11_14 = fma(eb, g14_1, o11_14);
              o11_15 = fma(eb, g15_1, o11_15);
            }
            { const double eb = bi[60];
              o11_14 = fma(eb, g14_4, o11_14);
              o11_15 = fma(eb, g15_4, o11_15);
            }
            { const double eb = bi[61];
              o11_14 = fma(eb, g14_10, o11_14);
              o11_15 = fma(eb, g15_10, o11_15);
            }
            { const double eb = bi[62];
              o12_14 = fma(eb, g14_0, o12_14);
              o12_15 = fma(eb, g15_0, o12_15);
            }
            { const double eb = bi[63];
              o12_14 = fma(eb, g14_2, o12_14);
              o12_15 = fma(eb, g15_2, o12_15);
            }
            { const double eb = bi[64];
              o12_14 = fma(eb, g14_3, o12_14);
              o12_15 = fma(eb, g15_3, o12_15);
            }
            { const double eb = bi[65];
              o12_14 = fma(eb, g14_8, o12_14);
              o12_15 = fma(eb, g15_8, o12_15);
            }
            { const double eb = bi[66];
              o13_14 = fma(eb, g14_0, o13_14);
              o13_15 = fma(eb, g15_0, o13_15);
            }
            { const double eb = bi[67];
              o13_14 = fma(eb, g14_2, o13_14);
              o13_15 = fma(eb, g15_2, o13_15);
            }
            { const double eb = bi[68];
              o13_14 = fma(eb, g14_3, o13_14);
              o13_15 = fma(eb, g15_3, o13_15);
            }
            { const double eb = bi[69];
              o13_14 = fma(eb, g14_8, o13_14);
              o13_15 = fma(eb, g15_8, o13_15);
            }
            { const double eb = bi[70];
              o13_14 = fma(eb, g14_9, o13_14);
              o13_15 = fma(eb, g15_9, o13_15);
            }
            { const double eb = bi[71];
              o13_14 = fma(eb, g14_18, o13_14);
              o13_15 = fma(eb, g15_18, o13_15);
            }
            { const double eb = bi[72];
              o14_14 = fma(eb, g14_0, o14_14);
              o14_15 = fma(eb, g15_0, o14_15);
            }
            { const double eb = bi[73];
              o14_14 = fma(eb, g14_2, o14_14);
              o14_15 = fma(eb, g15_2, o14_15);
            }
            { const double eb = bi[74];
              o14_14 = fma(eb, g14_6, o14_14);
              o14_15 = fma(eb, g15_6, o14_15);
            }
            { const double eb = bi[75];
              o14_14 = fma(eb, g14_3, o14_14);
              o14_15 = fma(eb, g15_3, o14_15);
            }
            { const double eb = bi[76];
              o14_14 = fma(eb, g14_8, o14_14);
              o14_15 = fma(eb, g15_8, o14_15);
            }
            { const double eb = bi[77];
              o14_14 = fma(eb, g14_16, o14_14);
              o14_15 = fma(eb, g15_16, o14_15);
            }
            { const double eb = bi[78];
              o15_14 = fma(eb, g14_0, o15_14);
              o15_15 = fma(eb, g15_0, o15_15);
            }
            { const double eb = bi[79];
              o15_14 = fma(eb, g14_1, o15_14);
              o15_15 = fma(eb, g15_1, o15_15);
            }
            { const double eb = bi[80];
              o15_14 = fma(eb, g14_2, o15_14);
              o15_15 = fma(eb, g15_2, o15_15);
            }
            { const double eb = bi[81];
              o15_14 = fma(eb, g14_5, o15_14);
              o15_15 = fma(eb, g15_5, o15_15);
            }
            { const double eb = bi[82];
              o15_14 = fma(eb, g14_3, o15_14);
              o15_15 = fma(eb, g15_3, o15_15);
            }
            { const double eb = bi[83];
              o15_14 = fma(eb, g14_7, o15_14);
              o15_15 = fma(eb, g15_7, o15_15);
            }
            { const double eb = bi[84];
              o15_14 = fma(eb, g14_8, o15_14);
              o15_15 = fma(eb, g15_8, o15_15);
            }
            { const double eb = bi[85];
              o15_14 = fma(eb, g14_15, o15_14);
              o15_15 = fma(eb, g15_15, o15_15);
            }
            { const double eb = bi[86];
              o16_14 = fma(eb, g14_0, o16_14);
              o16_15 = fma(eb, g15_0, o16_15);
            }
            { const double eb = bi[87];
              o16_14 = fma(eb, g14_1, o16_14);
              o16_15 = fma(eb, g15_1, o16_15);
            }
            { const double eb = bi[88];
              o16_14 = fma(eb, g14_3, o16_14);
              o16_15 = fma(eb, g15_3, o16_15);
            }
            { const double eb = bi[89];
              o16_14 = fma(eb, g14_7, o16_14);
              o16_15 = fma(eb, g15_7, o16_15);
            }
            { const double eb = bi[90];
              o17_14 = fma(eb, g14_0, o17_14);
              o17_15 = fma(eb, g15_0, o17_15);
            }
            { const double eb = bi[91];
              o17_14 = fma(eb, g14_1, o17_14);
              o17_15 = fma(eb, g15_1, o17_15);
            }
            { const double eb = bi[92];
              o17_14 = fma(eb, g14_3, o17_14);
              o17_15 = fma(eb, g15_3, o17_15);
            }
            { const double eb = bi[93];
              o17_14 = fma(eb, g14_7, o17_14);
              o17_15 = fma(eb, g15_7, o17_15);
            }
            { const double eb = bi[94];
              o17_14 = fma(eb, g14_9, o17_14);
              o17_15 = fma(eb, g15_9, o17_15);
            }
            { const double eb = bi[95];
              o17_14 = fma(eb, g14_17, o17_14);
              o17_15 = fma(eb, g15_17, o17_15);
            }
            { const double eb = bi[96];
              o18_14 = fma(eb, g14_0, o18_14);
              o18_15 = fma(eb, g15_0, o18_15);
            }
            { const double eb = bi[97];
              o18_14 = fma(eb, g14_1, o18_14);
              o18_15 = fma(eb, g15_1, o18_15);
            }
            { const double eb = bi[98];
              o18_14 = fma(eb, g14_2, o18_14);
              o18_15 = fma(eb, g15_2, o18_15);
            }
            { const double eb = bi[99];
              o18_14 = fma(eb, g14_5, o18_14);
              o18_15 = fma(eb, g15_5, o18_15);
            }
            { const double eb = bi[100];
              o18_14 = fma(eb, g14_3, o18_14);
              o18_15 = fma(eb, g15_3, o18_15);
            }
            { const double eb = bi[101];
              o18_14 = fma(eb, g14_7, o18_14);
              o18_15 = fma(eb, g15_7, o18_15);
            }
            { const double eb = bi[102];
              o18_14 = fma(eb, g14_8, o18_14);
              o18_15 = fma(eb, g15_8, o18_15);
            }
            { const double eb = bi[103];
              o18_14 = fma(eb, g14_15, o18_14);
              o18_15 = fma(eb, g15_15, o18_15);
            }
            { const double eb = bi[104];
              o19_14 = fma(eb, g14_0, o19_14);
              o19_15 = fma(eb, g15_0, o19_15);
            }
            { const double eb = bi[105];
              o19_14 = fma(eb, g14_1, o19_14);
              o19_15 = fma(eb, g15_1, o19_15);
            }
            { const double eb = bi[106];
              o19_14 = fma(eb, g14_4, o19_14);
              o19_15 = fma(eb, g15_4, o19_15);
            }
            { const double eb = bi[107];
              o19_14 = fma(eb, g14_3, o19_14);
              o19_15 = fma(eb, g15_3, o19_15);
            }
            { const double eb = bi[108];
              o19_14 = fma(eb, g14_7, o19_14);
              o19_15 = fma(eb, g15_7, o19_15);
            }
            { const double eb = bi[109];
              o19_14 = fma(eb, g14_14, o19_14);
              o19_15 = fma(eb, g15_14, o19_15);
            }
            { const double eb = bi[110];
              o20_14 = fma(eb, g14_0, o20_14);
              o20_15 = fma(eb, g15_0, o20_15);
            }
            { const double eb = bi[111];
              o20_14 = fma(eb, g14_1, o20_14);
              o20_15 = fma(eb, g15_1, o20_15);
            }
            { const double eb = bi[112];
              o20_14 = fma(eb, g14_2, o20_14);
              o20_15 = fma(eb, g15_2, o20_15);
            }
            { const double eb = bi[113];
              o20_14 = fma(eb, g14_5, o20_14);
              o20_15 = fma(eb, g15_5, o20_15);
            }
            { const double eb = bi[114];
              o21_14 = fma(eb, g14_0, o21_14);
              o21_15 = fma(eb, g15_0, o21_15);
            }
            { const double eb = bi[115];
              o21_14 = fma(eb, g14_1, o21_14);
              o21_15 = fma(eb, g15_1, o21_15);
            }
            { const double eb = bi[116];
              o21_14 = fma(eb, g14_2, o21_14);
              o21_15 = fma(eb, g15_2, o21_15);
            }
            { const double eb = bi[117];
              o21_14 = fma(eb, g14_5, o21_14);
              o21_15 = fma(eb, g15_5, o21_15);
            }
            { const double eb = bi[118];
              o21_14 = fma(eb, g14_3, o21_14);
              o21_15 = fma(eb, g15_3, o21_15);
            }
            { const double eb = bi[119];
              o21_14 = fma(eb, g14_7, o21_14);
              o21_15 = fma(eb, g15_7, o21_15);
            }
            { const double eb = bi[120];
              o21_14 = fma(eb, g14_8, o21_14);
              o21_15 = fma(eb, g15_8, o21_15);
            }
            { const double eb = bi[121];
              o21_14 = fma(eb, g14_15, o21_14);
              o21_15 = fma(eb, g15_15, o21_15);
            }
            { const double eb = bi[122];
              o22_14 = fma(eb, g14_0, o22_14);
              o22_15 = fma(eb, g15_0, o22_15);
            }
            { const double eb = bi[123];
              o22_14 = fma(eb, g14_1, o22_14);
              o22_15 = fma(eb, g15_1, o22_15);
            }
            { const double eb = bi[124];
              o22_14 = fma(eb, g14_2, o22_14);
              o22_15 = fma(eb, g15_2, o22_15);
            }
            { const double eb = bi[125];
              o22_14 = fma(eb, g14_5, o22_14);
              o22_15 = fma(eb, g15_5, o22_15);
            }
            { const double eb = bi[126];
              o22_14 = fma(eb, g14_6, o22_14);
              o22_15 = fma(eb, g15_6, o22_15);
            }
            { const double eb = bi[127];
              o22_14 = fma(eb, g14_12, o22_14);
              o22_15 = fma(eb, g15_12, o22_15);
            }
            { const double eb = bi[128];
              o23_14 = fma(eb, g14_0, o23_14);
              o23_15 = fma(eb, g15_0, o23_15);
            }
            { const double eb = bi[129];
              o23_14 = fma(eb, g14_1, o23_14);
              o23_15 = fma(eb, g15_1, o23_15);
            }
            { const double eb = bi[130];
              o23_14 = fma(eb, g14_4, o23_14);
              o23_15 = fma(eb, g15_4, o23_15);
            }
            { const double eb = bi[131];
              o23_14 = fma(eb, g14_2, o23_14);
              o23_15 = fma(eb, g15_2, o23_15);
            }
            { const double eb = bi[132];
              o23_14 = fma(eb, g14_5, o23_14);
              o23_15 = fma(eb, g15_5, o23_15);
            }
            { const double eb = bi[133];
              o23_14 = fma(eb, g14_11, o23_14);
              o23_15 = fma(eb, g15_11, o23_15);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk14 = PT[(fI + 3) * N + fJ + 2];
            const double ptk15 = PT[(fI + 3) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_3 = PA[(fQ + 0) * N + fI + 3];
            const double Abc1_3 = PA[(fQ + 1) * N + fI + 3];
            const double Abc2_3 = PA[(fQ + 2) * N + fI + 3];
            const double Abc3_3 = PA[(fQ + 3) * N + fI + 3];
            const double Aac0_3 = PA[(fP + 0) * N + fI + 3];
            const double Aac1_3 = PA[(fP + 1) * N + fI + 3];
            const double Aac2_3 = PA[(fP + 2) * N + fI + 3];
            const double Aac3_3 = PA[(fP + 3) * N + fI + 3];
            const double Aac4_3 = PA[(fP + 4) * N + fI + 3];
            const double Aac5_3 = PA[(fP + 5) * N + fI + 3];
            jab0 += o0_14 * ptk14 + o0_15 * ptk15;
            jab1 += o1_14 * ptk14 + o1_15 * ptk15;
            jab2 += o2_14 * ptk14 + o2_15 * ptk15;
            jab3 += o3_14 * ptk14 + o3_15 * ptk15;
            jab4 += o4_14 * ptk14 + o4_15 * ptk15;
            jab5 += o5_14 * ptk14 + o5_15 * ptk15;
            jab6 += o6_14 * ptk14 + o6_15 * ptk15;
            jab7 += o7_14 * ptk14 + o7_15 * ptk15;
            jab8 += o8_14 * ptk14 + o8_15 * ptk15;
            jab9 += o9_14 * ptk14 + o9_15 * ptk15;
            jab10 += o10_14 * ptk14 + o10_15 * ptk15;
            jab11 += o11_14 * ptk14 + o11_15 * ptk15;
            jab12 += o12_14 * ptk14 + o12_15 * ptk15;
            jab13 += o13_14 * ptk14 + o13_15 * ptk15;
            jab14 += o14_14 * ptk14 + o14_15 * ptk15;
            jab15 += o15_14 * ptk14 + o15_15 * ptk15;
            jab16 += o16_14 * ptk14 + o16_15 * ptk15;
            jab17 += o17_14 * ptk14 + o17_15 * ptk15;
            jab18 += o18_14 * ptk14 + o18_15 * ptk15;
            jab19 += o19_14 * ptk14 + o19_15 * ptk15;
            jab20 += o20_14 * ptk14 + o20_15 * ptk15;
            jab21 += o21_14 * ptk14 + o21_15 * ptk15;
            jab22 += o22_14 * ptk14 + o22_15 * ptk15;
            jab23 += o23_14 * ptk14 + o23_15 * ptk15;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 2, 2.0 * deg * (o0_14 * ptb0 + o1_14 * ptb1 + o2_14 * ptb2 + o3_14 * ptb3 + o4_14 * ptb4 + o5_14 * ptb5 + o6_14 * ptb6 + o7_14 * ptb7 + o8_14 * ptb8 + o9_14 * ptb9 + o10_14 * ptb10 + o11_14 * ptb11 + o12_14 * ptb12 + o13_14 * ptb13 + o14_14 * ptb14 + o15_14 * ptb15 + o16_14 * ptb16 + o17_14 * ptb17 + o18_14 * ptb18 + o19_14 * ptb19 + o20_14 * ptb20 + o21_14 * ptb21 + o22_14 * ptb22 + o23_14 * ptb23));
            atomicAdd(Jacc + (fI + 3) * N + fJ + 3, 2.0 * deg * (o0_15 * ptb0 + o1_15 * ptb1 + o2_15 * ptb2 + o3_15 * ptb3 + o4_15 * ptb4 + o5_15 * ptb5 + o6_15 * ptb6 + o7_15 * ptb7 + o8_15 * ptb8 + o9_15 * ptb9 + o10_15 * ptb10 + o11_15 * ptb11 + o12_15 * ptb12 + o13_15 * ptb13 + o14_15 * ptb14 + o15_15 * ptb15 + o16_15 * ptb16 + o17_15 * ptb17 + o18_15 * ptb18 + o19_15 * ptb19 + o20_15 * ptb20 + o21_15 * ptb21 + o22_15 * ptb22 + o23_15 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_14 * Abd0_2 + o0_15 * Abd0_3 + o1_14 * Abd1_2 + o1_15 * Abd1_3 + o2_14 * Abd2_2 + o2_15 * Abd2_3 + o3_14 * Abd3_2 + o3_15 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_14 * Aad0_2 + o0_15 * Aad0_3 + o4_14 * Aad1_2 + o4_15 * Aad1_3 + o8_14 * Aad2_2 + o8_15 * Aad2_3 + o12_14 * Aad3_2 + o12_15 * Aad3_3 + o16_14 * Aad4_2 + o16_15 * Aad4_3 + o20_14 * Aad5_2 + o20_15 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_14 * Abc0_3 + o1_14 * Abc1_3 + o2_14 * Abc2_3 + o3_14 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_14 * Aac0_3 + o4_14 * Aac1_3 + o8_14 * Aac2_3 + o12_14 * Aac3_3 + o16_14 * Aac4_3 + o20_14 * Aac5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_15 * Abc0_3 + o1_15 * Abc1_3 + o2_15 * Abc2_3 + o3_15 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_15 * Aac0_3 + o4_15 * Aac1_3 + o8_15 * Aac2_3 + o12_15 * Aac3_3 + o16_15 * Aac4_3 + o20_15 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_14 * Aad0_2 + o1_15 * Aad0_3 + o5_14 * Aad1_2 + o5_15 * Aad1_3 + o9_14 * Aad2_2 + o9_15 * Aad2_3 + o13_14 * Aad3_2 + o13_15 * Aad3_3 + o17_14 * Aad4_2 + o17_15 * Aad4_3 + o21_14 * Aad5_2 + o21_15 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_14 * Aac0_3 + o5_14 * Aac1_3 + o9_14 * Aac2_3 + o13_14 * Aac3_3 + o17_14 * Aac4_3 + o21_14 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_15 * Aac0_3 + o5_15 * Aac1_3 + o9_15 * Aac2_3 + o13_15 * Aac3_3 + o17_15 * Aac4_3 + o21_15 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_14 * Aad0_2 + o2_15 * Aad0_3 + o6_14 * Aad1_2 + o6_15 * Aad1_3 + o10_14 * Aad2_2 + o10_15 * Aad2_3 + o14_14 * Aad3_2 + o14_15 * Aad3_3 + o18_14 * Aad4_2 + o18_15 * Aad4_3 + o22_14 * Aad5_2 + o22_15 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_14 * Aac0_3 + o6_14 * Aac1_3 + o10_14 * Aac2_3 + o14_14 * Aac3_3 + o18_14 * Aac4_3 + o22_14 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_15 * Aac0_3 + o6_15 * Aac1_3 + o10_15 * Aac2_3 + o14_15 * Aac3_3 + o18_15 * Aac4_3 + o22_15 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_14 * Aad0_2 + o3_15 * Aad0_3 + o7_14 * Aad1_2 + o7_15 * Aad1_3 + o11_14 * Aad2_2 + o11_15 * Aad2_3 + o15_14 * Aad3_2 + o15_15 * Aad3_3 + o19_14 * Aad4_2 + o19_15 * Aad4_3 + o23_14 * Aad5_2 + o23_15 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_14 * Aac0_3 + o7_14 * Aac1_3 + o11_14 * Aac2_3 + o15_14 * Aac3_3 + o19_14 * Aac4_3 + o23_14 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_15 * Aac0_3 + o7_15 * Aac1_3 + o11_15 * Aac2_3 + o15_15 * Aac3_3 + o19_15 * Aac4_3 + o23_15 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_14 * Abd0_2 + o4_15 * Abd0_3 + o5_14 * Abd1_2 + o5_15 * Abd1_3 + o6_14 * Abd2_2 + o6_15 * Abd2_3 + o7_14 * Abd3_2 + o7_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_14 * Abc0_3 + o5_14 * Abc1_3 + o6_14 * Abc2_3 + o7_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_15 * Abc0_3 + o5_15 * Abc1_3 + o6_15 * Abc2_3 + o7_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_14 * Abd0_2 + o8_15 * Abd0_3 + o9_14 * Abd1_2 + o9_15 * Abd1_3 + o10_14 * Abd2_2 + o10_15 * Abd2_3 + o11_14 * Abd3_2 + o11_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_14 * Abc0_3 + o9_14 * Abc1_3 + o10_14 * Abc2_3 + o11_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_15 * Abc0_3 + o9_15 * Abc1_3 + o10_15 * Abc2_3 + o11_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_14 * Abd0_2 + o12_15 * Abd0_3 + o13_14 * Abd1_2 + o13_15 * Abd1_3 + o14_14 * Abd2_2 + o14_15 * Abd2_3 + o15_14 * Abd3_2 + o15_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_14 * Abc0_3 + o13_14 * Abc1_3 + o14_14 * Abc2_3 + o15_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_15 * Abc0_3 + o13_15 * Abc1_3 + o14_15 * Abc2_3 + o15_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o16_14 * Abd0_2 + o16_15 * Abd0_3 + o17_14 * Abd1_2 + o17_15 * Abd1_3 + o18_14 * Abd2_2 + o18_15 * Abd2_3 + o19_14 * Abd3_2 + o19_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_14 * Abc0_3 + o17_14 * Abc1_3 + o18_14 * Abc2_3 + o19_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_15 * Abc0_3 + o17_15 * Abc1_3 + o18_15 * Abc2_3 + o19_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o20_14 * Abd0_2 + o20_15 * Abd0_3 + o21_14 * Abd1_2 + o21_15 * Abd1_3 + o22_14 * Abd2_2 + o22_15 * Abd2_3 + o23_14 * Abd3_2 + o23_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_14 * Abc0_3 + o21_14 * Abc1_3 + o22_14 * Abc2_3 + o23_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_15 * Abc0_3 + o21_15 * Abc1_3 + o22_15 * Abc2_3 + o23_15 * Abc3_3));
          }
        } break;
        case 8: {  // ket functions [16, 17]
          double o0_16 = 0;
          double o0_17 = 0;
          double o1_16 = 0;
          double o1_17 = 0;
          double o2_16 = 0;
          double o2_17 = 0;
          double o3_16 = 0;
          double o3_17 = 0;
          double o4_16 = 0;
          double o4_17 = 0;
          double o5_16 = 0;
          double o5_17 = 0;
          double o6_16 = 0;
          double o6_17 = 0;
          double o7_16 = 0;
          double o7_17 = 0;
          double o8_16 = 0;
          double o8_17 = 0;
          double o9_16 = 0;
          double o9_17 = 0;
          double o10_16 = 0;
          double o10_17 = 0;
          double o11_16 = 0;
          double o11_17 = 0;
          double o12_16 = 0;
          double o12_17 = 0;
          double o13_16 = 0;
          double o13_17 = 0;
          double o14_16 = 0;
          double o14_17 = 0;
          double o15_16 = 0;
          double o15_17 = 0;
          double o16_16 = 0;
          double o16_17 = 0;
          double o17_16 = 0;
          double o17_17 = 0;
          double o18_16 = 0;
          double o18_17 = 0;
          double o19_16 = 0;
          double o19_17 = 0;
          double o20_16 = 0;
          double o20_17 = 0;
          double o21_16 = 0;
          double o21_17 = 0;
          double o22_16 = 0;
          double o22_17 = 0;
          double o23_16 = 0;
          double o23_17 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g16_0 = 0;
            double g16_1 = 0;
            double g16_2 = 0;
            double g16_3 = 0;
            double g16_4 = 0;
            double g16_5 = 0;
            double g16_6 = 0;
            double g16_7 = 0;
            double g16_8 = 0;
            double g16_9 = 0;
            double g16_10 = 0;
            double g16_11 = 0;
            double g16_12 = 0;
            double g16_13 = 0;
            double g16_14 = 0;
            double g16_15 = 0;
            double g16_16 = 0;
            double g16_17 = 0;
            double g16_18 = 0;
            double g16_19 = 0;
            double g17_0 = 0;
            double g17_1 = 0;
            double g17_2 = 0;
            double g17_3 = 0;
            double g17_4 = 0;
            double g17_5 = 0;
            double g17_6 = 0;
            double g17_7 = 0;
            double g17_8 = 0;
            double g17_9 = 0;
            double g17_10 = 0;
            double g17_11 = 0;
            double g17_12 = 0;
            double g17_13 = 0;
            double g17_14 = 0;
            double g17_15 = 0;
            double g17_16 = 0;
            double g17_17 = 0;
            double g17_18 = 0;
            double g17_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek16_0 = kj[86 * kS];
              const double ek16_1 = -kj[87 * kS];
              const double ek16_2 = -kj[88 * kS];
              const double ek16_3 = kj[89 * kS];
              const double ek17_0 = kj[90 * kS];
              const double ek17_1 = -kj[91 * kS];
              const double ek17_2 = -kj[92 * kS];
              const double ek17_3 = kj[93 * kS];
              const double ek17_4 = kj[94 * kS];
              const double ek17_5 = -kj[95 * kS];
              g16_0 = fma(ek16_0, b0, g16_0);
              g17_0 = fma(ek17_0, b0, g17_0);
              const double r0_0_0_1 = Z * b1;
              g16_1 = fma(ek16_0, r0_0_0_1, g16_1);
              g16_0 = fma(ek16_1, r0_0_0_1, g16_0);
              g17_1 = fma(ek17_0, r0_0_0_1, g17_1);
              g17_0 = fma(ek17_1, r0_0_0_1, g17_0);
              const double r0_0_1_0 = Y * b1;
              g16_2 = fma(ek16_0, r0_0_1_0, g16_2);
              g17_2 = fma(ek17_0, r0_0_1_0, g17_2);
              const double r0_1_0_0 = X * b1;
              g16_3 = fma(ek16_0, r0_1_0_0, g16_3);
              g16_0 = fma(ek16_2, r0_1_0_0, g16_0);
              g17_3 = fma(ek17_0, r0_1_0_0, g17_3);
              g17_0 = fma(ek17_2, r0_1_0_0, g17_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g16_4 = fma(ek16_0, r0_0_0_2, g16_4);
              g16_1 = fma(ek16_1, r0_0_0_2, g16_1);
              g17_4 = fma(ek17_0, r0_0_0_2, g17_4);
              g17_1 = fma(ek17_1, r0_0_0_2, g17_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g16_5 = fma(ek16_0, r0_0_1_1, g16_5);
              g16_2 = fma(ek16_1, r0_0_1_1, g16_2);
              g17_5 = fma(ek17_0, r0_0_1_1, g17_5);
              g17_2 = fma(ek17_1, r0_0_1_1, g17_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g16_6 = fma(ek16_0, r0_0_2_0, g16_6);
              g17_6 = fma(ek17_0, r0_0_2_0, g17_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g16_7 = fma(ek16_0, r0_1_0_1, g16_7);
              g16_3 = fma(ek16_1, r0_1_0_1, g16_3);
              g16_1 = fma(ek16_2, r0_1_0_1, g16_1);
              g16_0 = fma(ek16_3, r0_1_0_1, g16_0);
              g17_7 = fma(ek17_0, r0_1_0_1, g17_7);
              g17_3 = fma(ek17_1, r0_1_0_1, g17_3);
              g17_1 = fma(ek17_2, r0_1_0_1, g17_1);
              g17_0 = fma(ek17_3, r0_1_0_1, g17_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g16_8 = fma(ek16_0, r0_1_1_0, g16_8);
              g16_2 = fma(ek16_2, r0_1_1_0, g16_2);
              g17_8 = fma(ek17_0, r0_1_1_0, g17_8);
              g17_2 = fma(ek17_2, r0_1_1_0, g17_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g16_9 = fma(ek16_0, r0_2_0_0, g16_9);
              g16_3 = fma(ek16_2, r0_2_0_0, g16_3);
              g17_9 = fma(ek17_0, r0_2_0_0, g17_9);
              g17_3 = fma(ek17_2, r0_2_0_0, g17_3);
              g17_0 = fma(ek17_4, r0_2_0_0, g17_0);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g16_10 = fma(ek16_0, r0_0_0_3, g16_10);
              g16_4 = fma(ek16_1, r0_0_0_3, g16_4);
              g17_10 = fma(ek17_0, r0_0_0_3, g17_10);
              g17_4 = fma(ek17_1, r0_0_0_3, g17_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g16_11 = fma(ek16_0, r0_0_1_2, g16_11);
              g16_5 = fma(ek16_1, r0_0_1_2, g16_5);
              g17_11 = fma(ek17_0, r0_0_1_2, g17_11);
              g17_5 = fma(ek17_1, r0_0_1_2, g17_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g16_12 = fma(ek16_0, r0_0_2_1, g16_12);
              g16_6 = fma(ek16_1, r0_0_2_1, g16_6);
              g17_12 = fma(ek17_0, r0_0_2_1, g17_12);
              g17_6 = fma(ek17_1, r0_0_2_1, g17_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g16_13 = fma(ek16_0, r0_0_3_0, g16_13);
              g17_13 = fma(ek17_0, r0_0_3_0, g17_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g16_14 = fma(ek16_0, r0_1_0_2, g16_14);
              g16_7 = fma(ek16_1, r0_1_0_2, g16_7);
              g16_4 = fma(ek16_2, r0_1_0_2, g16_4);
              g16_1 = fma(ek16_3, r0_1_0_2, g16_1);
              g17_14 = fma(ek17_0, r0_1_0_2, g17_14);
              g17_7 = fma(ek17_1, r0_1_0_2, g17_7);
              g17_4 = fma(ek17_2, r0_1_0_2, g17_4);
              g17_1 = fma(ek17_3, r0_1_0_2, g17_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g16_15 = fma(ek16_0, r0_1_1_1, g16_15);
              g16_8 = fma(ek16_1, r0_1_1_1, g16_8);
              g16_5 = fma(ek16_2, r0_1_1_1, g16_5);
              g16_2 = fma(ek16_3, r0_1_1_1, g16_2);
              g17_15 = fma(ek17_0, r0_1_1_1, g17_15);
              g17_8 = fma(ek17_1, r0_1_1_1, g17_8);
              g17_5 = fma(ek17_2, r0_1_1_1, g17_5);
              g17_2 = fma(ek17_3, r0_1_1_1, g17_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g16_16 = fma(ek16_0, r0_1_2_0, g16_16);
              g16_6 = fma(ek16_2, r0_1_2_0, g16_6);
              g17_16 = fma(ek17_0, r0_1_2_0, g17_16);
              g17_6 = fma(ek17_2, r0_1_2_0, g17_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g16_17 = fma(ek16_0, r0_2_0_1, g16_17);
              g16_9 = fma(ek16_1, r0_2_0_1, g16_9);
              g16_7 = fma(ek16_2, r0_2_0_1, g16_7);
              g16_3 = fma(ek16_3, r0_2_0_1, g16_3);
              g17_17 = fma(ek17_0, r0_2_0_1, g17_17);
              g17_9 = fma(ek17_1, r0_2_0_1, g17_9);
              g17_7 = fma(ek17_2, r0_2_0_1, g17_7);
              g17_3 = fma(ek17_3, r0_2_0_1, g17_3);
              g17_1 = fma(ek17_4, r0_2_0_1, g17_1);
              g17_0 = fma(ek17_5, r0_2_0_1, g17_0);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g16_18 = fma(ek16_0, r0_2_1_0, g16_18);
              g16_8 = fma(ek16_2, r0_2_1_0, g16_8);
              g17_18 = fma(ek17_0, r0_2_1_0, g17_18);
              g17_8 = fma(ek17_2, r0_2_1_0, g17_8);
              g17_2 = fma(ek17_4, r0_2_1_0, g17_2);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g16_19 = fma(ek16_0, r0_3_0_0, g16_19);
              g16_9 = fma(ek16_2, r0_3_0_0, g16_9);
              g17_19 = fma(ek17_0, r0_3_0_0, g17_19);
              g17_9 = fma(ek17_2, r0_3_0_0, g17_9);
              g17_3 = fma(ek17_4, r0_3_0_0, g17_3);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g16_10 = fma(ek16_1, r0_0_0_4, g16_10);
              g17_10 = fma(ek17_1, r0_0_0_4, g17_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g16_11 = fma(ek16_1, r0_0_1_3, g16_11);
              g17_11 = fma(ek17_1, r0_0_1_3, g17_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g16_12 = fma(ek16_1, r0_0_2_2, g16_12);
              g17_12 = fma(ek17_1, r0_0_2_2, g17_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g16_13 = fma(ek16_1, r0_0_3_1, g16_13);
              g17_13 = fma(ek17_1, r0_0_3_1, g17_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g16_14 = fma(ek16_1, r0_1_0_3, g16_14);
              g16_10 = fma(ek16_2, r0_1_0_3, g16_10);
              g16_4 = fma(ek16_3, r0_1_0_3, g16_4);
              g17_14 = fma(ek17_1, r0_1_0_3, g17_14);
              g17_10 = fma(ek17_2, r0_1_0_3, g17_10);
              g17_4 = fma(ek17_3, r0_1_0_3, g17_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g16_15 = fma(ek16_1, r0_1_1_2, g16_15);
              g16_11 = fma(ek16_2, r0_1_1_2, g16_11);
              g16_5 = fma(ek16_3, r0_1_1_2, g16_5);
              g17_15 = fma(ek17_1, r0_1_1_2, g17_15);
              g17_11 = fma(ek17_2, r0_1_1_2, g17_11);
              g17_5 = fma(ek17_3, r0_1_1_2, g17_5);
              const double r0_1_2_1 = X * r1_0_2_1;
              g16_16 = fma(ek16_1, r0_1_2_1, g16_16);
              g16_12 = fma(ek16_2, r0_1_2_1, g16_12);
              g16_6 = fma(ek16_3, r0_1_2_1, g16_6);
              g17_16 = fma(ek17_1, r0_1_2_1, g17_16);
              g17_12 = fma(ek17_2, r0_1_2_1, g17_12);
              g17_6 = fma(ek17_3, r0_1_2_1, g17_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g16_13 = fma(ek16_2, r0_1_3_0, g16_13);
              g17_13 = fma(ek17_2, r0_1_3_0, g17_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g16_17 = fma(ek16_1, r0_2_0_2, g16_17);
              g16_14 = fma(ek16_2, r0_2_0_2, g16_14);
              g16_7 = fma(ek16_3, r0_2_0_2, g16_7);
              g17_17 = fma(ek17_1, r0_2_0_2, g17_17);
              g17_14 = fma(ek17_2, r0_2_0_2, g17_14);
              g17_7 = fma(ek17_3, r0_2_0_2, g17_7);
              g17_4 = fma(ek17_4, r0_2_0_2, g17_4);
              g17_1 = fma(ek17_5, r0_2_0_2, g17_1);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g16_18 = fma(ek16_1, r0_2_1_1, g16_18);
              g16_15 = fma(ek16_2, r0_2_1_1, g16_15);
              g16_8 = fma(ek16_3, r0_2_1_1, g16_8);
              g17_18 = fma(ek17_1, r0_2_1_1, g17_18);
              g17_15 = fma(ek17_2, r0_2_1_1, g17_15);
              g17_8 = fma(ek17_3, r0_2_1_1, g17_8);
              g17_5 = fma(ek17_4, r0_2_1_1, g17_5);
              g17_2 = fma(ek17_5, r0_2_1_1, g17_2);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g16_16 = fma(ek16_2, r0_2_2_0, g16_16);
              g17_16 = fma(ek17_2, r0_2_2_0, g17_16);
              g17_6 = fma(ek17_4, r0_2_2_0, g17_6);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g16_19 = fma(ek16_1, r0_3_0_1, g16_19);
              g16_17 = fma(ek16_2, r0_3_0_1, g16_17);
              g16_9 = fma(ek16_3, r0_3_0_1, g16_9);
              g17_19 = fma(ek17_1, r0_3_0_1, g17_19);
              g17_17 = fma(ek17_2, r0_3_0_1, g17_17);
              g17_9 = fma(ek17_3, r0_3_0_1, g17_9);
              g17_7 = fma(ek17_4, r0_3_0_1, g17_7);
              g17_3 = fma(ek17_5, r0_3_0_1, g17_3);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g16_18 = fma(ek16_2, r0_3_1_0, g16_18);
              g17_18 = fma(ek17_2, r0_3_1_0, g17_18);
              g17_8 = fma(ek17_4, r0_3_1_0, g17_8);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g16_19 = fma(ek16_2, r0_4_0_0, g16_19);
              g17_19 = fma(ek17_2, r0_4_0_0, g17_19);
              g17_9 = fma(ek17_4, r0_4_0_0, g17_9);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_1_0_4 = X * r1_0_0_4;
              g16_10 = fma(ek16_3, r0_1_0_4, g16_10);
              g17_10 = fma(ek17_3, r0_1_0_4, g17_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g16_11 = fma(ek16_3, r0_1_1_3, g16_11);
              g17_11 = fma(ek17_3, r0_1_1_3, g17_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g16_12 = fma(ek16_3, r0_1_2_2, g16_12);
              g17_12 = fma(ek17_3, r0_1_2_2, g17_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g16_13 = fma(ek16_3, r0_1_3_1, g16_13);
              g17_13 = fma(ek17_3, r0_1_3_1, g17_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g16_14 = fma(ek16_3, r0_2_0_3, g16_14);
              g17_14 = fma(ek17_3, r0_2_0_3, g17_14);
              g17_10 = fma(ek17_4, r0_2_0_3, g17_10);
              g17_4 = fma(ek17_5, r0_2_0_3, g17_4);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g16_15 = fma(ek16_3, r0_2_1_2, g16_15);
              g17_15 = fma(ek17_3, r0_2_1_2, g17_15);
              g17_11 = fma(ek17_4, r0_2_1_2, g17_11);
              g17_5 = fma(ek17_5, r0_2_1_2, g17_5);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g16_16 = fma(ek16_3, r0_2_2_1, g16_16);
              g17_16 = fma(ek17_3, r0_2_2_1, g17_16);
              g17_12 = fma(ek17_4, r0_2_2_1, g17_12);
              g17_6 = fma(ek17_5, r0_2_2_1, g17_6);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g17_13 = fma(ek17_4, r0_2_3_0, g17_13);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g16_17 = fma(ek16_3, r0_3_0_2, g16_17);
              g17_17 = fma(ek17_3, r0_3_0_2, g17_17);
              g17_14 = fma(ek17_4, r0_3_0_2, g17_14);
              g17_7 = fma(ek17_5, r0_3_0_2, g17_7);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g16_18 = fma(ek16_3, r0_3_1_1, g16_18);
              g17_18 = fma(ek17_3, r0_3_1_1, g17_18);
              g17_15 = fma(ek17_4, r0_3_1_1, g17_15);
              g17_8 = fma(ek17_5, r0_3_1_1, g17_8);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g17_16 = fma(ek17_4, r0_3_2_0, g17_16);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g16_19 = fma(ek16_3, r0_4_0_1, g16_19);
              g17_19 = fma(ek17_3, r0_4_0_1, g17_19);
              g17_17 = fma(ek17_4, r0_4_0_1, g17_17);
              g17_9 = fma(ek17_5, r0_4_0_1, g17_9);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g17_18 = fma(ek17_4, r0_4_1_0, g17_18);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g17_19 = fma(ek17_4, r0_5_0_0, g17_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g17_10 = fma(ek17_5, r0_2_0_4, g17_10);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g17_11 = fma(ek17_5, r0_2_1_3, g17_11);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g17_12 = fma(ek17_5, r0_2_2_2, g17_12);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g17_13 = fma(ek17_5, r0_2_3_1, g17_13);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g17_14 = fma(ek17_5, r0_3_0_3, g17_14);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g17_15 = fma(ek17_5, r0_3_1_2, g17_15);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g17_16 = fma(ek17_5, r0_3_2_1, g17_16);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g17_17 = fma(ek17_5, r0_4_0_2, g17_17);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g17_18 = fma(ek17_5, r0_4_1_1, g17_18);
              const double r4_1_0_1 = X * r5_0_0_1;
              const double r3_2_0_1 = fma(X, r4_1_0_1, r4_0_0_1);
              const double r2_3_0_1 = fma(X, r3_2_0_1, 2.0 * r3_1_0_1);
              const double r1_4_0_1 = fma(X, r2_3_0_1, 3.0 * r2_2_0_1);
              const double r0_5_0_1 = fma(X, r1_4_0_1, 4.0 * r1_3_0_1);
              g17_19 = fma(ek17_5, r0_5_0_1, g17_19);
            }
            { const double eb = bi[5];
              o0_16 = fma(eb, g16_0, o0_16);
              o0_17 = fma(eb, g17_0, o0_17);
            }
            { const double eb = bi[6];
              o0_16 = fma(eb, g16_3, o0_16);
              o0_17 = fma(eb, g17_3, o0_17);
            }
            { const double eb = bi[7];
              o0_16 = fma(eb, g16_9, o0_16);
              o0_17 = fma(eb, g17_9, o0_17);
            }
            { const double eb = bi[8];
              o1_16 = fma(eb, g16_0, o1_16);
              o1_17 = fma(eb, g17_0, o1_17);
            }
            { const double eb = bi[9];
              o1_16 = fma(eb, g16_3, o1_16);
              o1_17 = fma(eb, g17_3, o1_17);
            }
            { const double eb = bi[10];
              o1_16 = fma(eb, g16_9, o1_16);
              o1_17 = fma(eb, g17_9, o1_17);
            }
            { const double eb = bi[11];
              o1_16 = fma(eb, g16_19, o1_16);
              o1_17 = fma(eb, g17_19, o1_17);
            }
            { const double eb = bi[12];
              o2_16 = fma(eb, g16_0, o2_16);
              o2_17 = fma(eb, g17_0, o2_17);
            }
            { const double eb = bi[13];
              o2_16 = fma(eb, g16_2, o2_16);
              o2_17 = fma(eb, g17_2, o2_17);
            }
            { const double eb = bi[14];
              o2_16 = fma(eb, g16_3, o2_16);
              o2_17 = fma(eb, g17_3, o2_17);
            }
            { const double eb = bi[15];
              o2_16 = fma(eb, g16_8, o2_16);
              o2_17 = fma(eb, g17_8, o2_17);
            }
            { const double eb = bi[16];
              o2_16 = fma(eb, g16_9, o2_16);
              o2_17 = fma(eb, g17_9, o2_17);
            }
            { const double eb = bi[17];
              o2_16 = fma(eb, g16_18, o2_16);
              o2_17 = fma(eb, g17_18, o2_17);
            }
            { const double eb = bi[18];
              o3_16 = fma(eb, g16_0, o3_16);
              o3_17 = fma(eb, g17_0, o3_17);
            }
            { const double eb = bi[19];
              o3_16 = fma(eb, g16_1, o3_16);
              o3_17 = fma(eb, g17_1, o3_17);
            }
            { const double eb = bi[20];
              o3_16 = fma(eb, g16_3, o3_16);
              o3_17 = fma(eb, g17_3, o3_17);
            }
            { const double eb = bi[21];
              o3_16 = fma(eb, g16_7, o3_16);
              o3_17 = fma(eb, g17_7, o3_17);
            }
            { const double eb = bi[22];
              o3_16 = fma(eb, g16_9, o3_16);
              o3_17 = fma(eb, g17_9, o3_17);
            }
            { const double eb = bi[23];
              o3_16 = fma(eb, g16_17, o3_16);
              o3_17 = fma(eb, g17_17, o3_17);
            }
            { const double eb = bi[24];
              o4_16 = fma(eb, g16_0, o4_16);
              o4_17 = fma(eb, g17_0, o4_17);
            }
            { const double eb = bi[25];
              o4_16 = fma(eb, g16_2, o4_16);
              o4_17 = fma(eb, g17_2, o4_17);
            }
            { const double eb = bi[26];
              o4_16 = fma(eb, g16_6, o4_16);
              o4_17 = fma(eb, g17_6, o4_17);
            }
            { const double eb = bi[27];
              o5_16 = fma(eb, g16_0, o5_16);
              o5_17 = fma(eb, g17_0, o5_17);
            }
            { const double eb = bi[28];
              o5_16 = fma(eb, g16_2, o5_16);
              o5_17 = fma(eb, g17_2, o5_17);
            }
            { const double eb = bi[29];
              o5_16 = fma(eb, g16_6, o5_16);
              o5_17 = fma(eb, g17_6, o5_17);
            }
            { const double eb = bi[30];
              o5_16 = fma(eb, g16_3, o5_16);
              o5_17 = fma(eb, g17_3, o5_17);
            }
            { const double eb = bi[31];
              o5_16 = fma(eb, g16_8, o5_16);
              o5_17 = fma(eb, g17_8, o5_17);
            }
            { const double eb = bi[32];
              o5_16 = fma(eb, g16_16, o5_16);
              o5_17 = fma(eb, g17_16, o5_17);
            }
            { const double eb = bi[33];
              o6_16 = fma(eb, g16_0, o6_16);
              o6_17 = fma(eb, g17_0, o6_17);
            }
            { const double eb = bi[34];
              o6_16 = fma(eb, g16_2, o6_16);
              o6_17 = fma(eb, g17_2, o6_17);
            }
            { const double eb = bi[35];
              o6_16 = fma(eb, g16_6, o6_16);
              o6_17 = fma(eb, g17_6, o6_17);
            }
            { const double eb = bi[36];
              o6_16 = fma(eb, g16_13, o6_16);
              o6_17 = fma(eb, g17_13, o6_17);
            }
            { const double eb = bi[37];
              o7_16 = fma(eb, g16_0, o7_16);
              o7_17 = fma(eb, g17_0, o7_17);
            }
            { const double eb = bi[38];
              o7_16 = fma(eb, g16_1, o7_16);
              o7_17 = fma(eb, g17_1, o7_17);
            }
            { const double eb = bi[39];
              o7_16 = fma(eb, g16_2, o7_16);
              o7_17 = fma(eb, g17_2, o7_17);
            }
            { const double eb = bi[40];
              o7_16 = fma(eb, g16_5, o7_16);
              o7_17 = fma(eb, g17_5, o7_17);
            }
            { const double eb = bi[41];
              o7_16 = fma(eb, g16_6, o7_16);
              o7_17 = fma(eb, g17_6, o7_17);
            }
            { const double eb = bi[42];
              o7_16 = fma(eb, g16_12, o7_16);
              o7_17 = fma(eb, g17_12, o7_17);
            }
            { const double eb = bi[43];
              o8_16 = fma(eb, g16_0, o8_16);
              o8_17 = fma(eb, g17_0, o8_17);
            }
            { const double eb = bi[44];
              o8_16 = fma(eb, g16_1, o8_16);
              o8_17 = fma(eb, g17_1, o8_17);
            }
            { const double eb = bi[45];
              o8_16 = fma(eb, g16_4, o8_16);
              o8_17 = fma(eb, g17_4, o8_17);
            }
            { const double eb = bi[46];
              o9_16 = fma(eb, g16_0, o9_16);
              o9_17 = fma(eb, g17_0, o9_17);
            }
            { const double eb = bi[47];
              o9_16 = fma(eb, g16_1, o9_16);
              o9_17 = fma(eb, g17_1, o9_17);
            }
            { const double eb = bi[48];
              o9_16 = fma(eb, g16_4, o9_16);
              o9_17 = fma(eb, g17_4, o9_17);
            }
            { const double eb = bi[49];
              o9_16 = fma(eb, g16_3, o9_16);
              o9_17 = fma(eb, g17_3, o9_17);
            }
            { const double eb = bi[50];
              o9_16 = fma(eb, g16_7, o9_16);
              o9_17 = fma(eb, g17_7, o9_17);
            }
            { const double eb = bi[51];
              o9_16 = fma(eb, g16_14, o9_16);
              o9_17 = fma(eb, g17_14, o9_17);
            }
            { const double eb = bi[52];
              o10_16 = fma(eb, g16_0, o10_16);
              o10_17 = fma(eb, g17_0, o10_17);
            }
            { const double eb = bi[53];
              o10_16 = fma(eb, g16_1, o10_16);
              o10_17 = fma(eb, g17_1, o10_17);
            }
            { const double eb = bi[54];
              o10_16 = fma(eb, g16_4, o10_16);
              o10_17 = fma(eb, g17_4, o10_17);
            }
            { const double eb = bi[55];
              o10_16 = fma(eb, g16_2, o10_16);
              o10_17 = fma(eb, g17_2, o10_17);
            }
            { const double eb = bi[56];
              o10_16 = fma(eb, g16_5, o10_16);
              o10_17 = fma(eb, g17_5, o10_17);
            }
            { const double eb = bi[57];
              o10_16 = fma(eb, g16_11, o10_16);
              o10_17 = fma(eb, g17_11, o10_17);
            }
            { const double eb = bi[58];
              o11_16 = fma(eb, g16_0, o11_16);
              o11_17 = fma(eb, g17_0, o11_17);
            }
            { const double eb = bi[59];
              o11_16 = fma(eb, g16_1, o11_16);
              o11_17 = fma(eb, g17_1, o11_17);
            }
            { const double eb = bi[60];
              o11_16 = fma(eb, g16_4, o11_16);
              o11_17 = fma(eb, g17_4, o11_17);
            }
            { const double eb = bi[61];
              o11_16 = fma(eb, g16_10, o11_16);
              o11_17 = fma(eb, g17_10, o11_17);
            }
            { const double eb = bi[62];
              o12_16 = fma(eb, g16_0, o12_16);
              o12_17 = fma(eb, g17_0, o12_17);
            }
            { const double eb = bi[63];
              o12_16 = fma(eb, g16_2, o12_16);
              o12_17 = fma(eb, g17_2, o12_17);
            }
            { const double eb = bi[64];
              o12_16 = fma(eb, g16_3, o12_16);
              o12_17 = fma(eb, g17_3, o12_17);
            }
            { const double eb = bi[65];
              o12_16 = fma(eb, g16_8, o12_16);
              o12_17 = fma(eb, g17_8, o12_17);
            }
            { const double eb = bi[66];
              o13_16 = fma(eb, g16_0, o13_16);
              o13_17 = fma(eb, g17_0, o13_17);
            }
            { const double eb = bi[67];
              o13_16 = fma(eb, g16_2, o13_16);
              o13_17 = fma(eb, g17_2, o13_17);
            }
            { const double eb = bi[68];
              o13_16 = fma(eb, g16_3, o13_16);
              o13_17 = fma(eb, g17_3, o13_17);
            }
            { const double eb = bi[69];
              o13_16 = fma(eb, g16_8, o13_16);
              o13_17 = fma(eb, g17_8, o13_17);
            }
            { const double eb = bi[70];
              o13_16 = fma(eb, g16_9, o13_16);
              o13_17 = fma(eb, g17_9, o13_17);
            }
            { const double eb = bi[71];
              o13_16 = fma(eb, g16_18, o13_16);
              o13_17 = fma(eb, g17_18, o13_17);
            }
            { const double eb = bi[72];
              o14_16 = fma(eb, g16_0, o14_16);
              o14_17 = fma(eb, g17_0, o14_17);
            }
            { const double eb = bi[73];
              o14_16 = fma(eb, g16_2, o14_16);
              o14_17 = fma(eb, g17_2, o14_17);
            }
            { const double eb = bi[74];
              o14_16 = fma(eb, g16_6, o14_16);
              o14_17 = fma(eb, g17_6, o14_17);
            }
            { const double eb = bi[75];
              o14_16 = fma(eb, g16_3, o14_16);
              o14_17 = fma(eb, g17_3, o14_17);
            }
            { const double eb = bi[76];
              o14_16 = fma(eb, g16_8, o14_16);
              o14_17 = fma(eb, g17_8, o14_17);
            }
            { const double eb = bi[77];
              o14_16 = fma(eb, g16_16, o14_16);
              o14_17 = fma(eb, g17_16, o14_17);
            }
            { const double eb = bi[78];
              o15_16 = fma(eb, g16_0, o15_16);
              o15_17 = fma(eb, g17_0, o15_17);
            }
            { const double eb = bi[79];
              o15_16 = fma(eb, g16_1, o15_16);
              o15_17 = fma(eb, g17_1, o15_17);
            }
            { const double eb = bi[80];
              o15_16 = fma(eb, g16_2, o15_16);
              o15_17 = fma(eb, g17_2, o15_17);
            }
            { const double eb = bi[81];
              o15_16 = fma(eb, g16_5, o15_16);
              o15_17 = fma(eb, g17_5, o15_17);
            }
            { const double eb = bi[82];
              o15_16 = fma(eb, g16_3, o15_16);
              o15_17 = fma(eb, g17_3, o15_17);
            }
            { const double eb = bi[83];
              o15_16 = fma(eb, g16_7, o15_16);
              o15_17 = fma(eb, g17_7, o15_17);
            }
            { const double eb = bi[84];
              o15_16 = fma(eb, g16_8, o15_16);
              o15_17 = fma(eb, g17_8, o15_17);
            }
            { const double eb = bi[85];
              o15_16 = fma(eb, g16_15, o15_16);
              o15_17 = fma(eb, g17_15, o15_17);
            }
            { const double eb = bi[86];
              o16_16 = fma(eb, g16_0, o16_16);
              o16_17 = fma(eb, g17_0, o16_17);
            }
            { const double eb = bi[87];
              o16_16 = fma(eb, g16_1, o16_16);
              o16_17 = fma(eb, g17_1, o16_17);
            }
            { const double eb = bi[88];
              o16_16 = fma(eb, g16_3, o16_16);
              o16_17 = fma(eb, g17_3, o16_17);
            }
            { const double eb = bi[89];
              o16_16 = fma(eb, g16_7, o16_16);
              o16_17 = fma(eb, g17_7, o16_17);
            }
            { const double eb = bi[90];
              o17_16 = fma(eb, g16_0, o17_16);
              o17_17 = fma(eb, g17_0, o17_17);
            }
            { const double eb = bi[91];
              o17_16 = fma(eb, g16_1, o17_16);
              o17_17 = fma(eb, g17_1, o17_17);
            }
            { const double eb = bi[92];
              o17_16 = fma(eb, g16_3, o17_16);
              o17_17 = fma(eb, g17_3, o17_17);
            }
            { const double eb = bi[93];
              o17_16 = fma(eb, g16_7, o17_16);
              o17_17 = fma(eb, g17_7, o17_17);
            }
            { const double eb = bi[94];
              o17_16 = fma(eb, g16_9, o17_16);
              o17_17 = fma(eb, g17_9, o17_17);
            }
            { const double eb = bi[95];
              o17_16 = fma(eb, g16_17, o17_16);
              o17_17 = fma(eb, g17_17, o17_17);
            }
            { const double eb = bi[96];
              o18_16 = fma(eb, g16_0, o18_16);
              o18_17 = fma(eb, g17_0, o18_17);
            }
            { const double eb = bi[97];
              o18_16 = fma(eb, g16_1, o18_16);
              o18_17 = fma(eb, g17_1, o18_17);
            }
            { const double eb = bi[98];
              o18_16 = fma(eb, g16_2, o18_16);
              o18_17 = fma(eb, g17_2, o18_17);
            }
            { const double eb = bi[99];
              o18_16 = fma(eb, g16_5, o18_16);
              o18_17 = fma(eb, g17_5, o18_17);
            }
            { const double eb = bi[100];
              o18_16 = fma(eb, g16_3, o18_16);
              o18_17 = fma(eb, g17_3, o18_17);
            }
            { const double eb = bi[101];
              o18_16 = fma(eb, g16_7, o18_16);
              o18_17 = fma(eb, g17_7, o18_17);
            }
            { const double eb = bi[102];
              o18_16 = fma(eb, g16_8, o18_16);
              o18_17 = fma(eb, g17_8, o18_17);
            }
            { const double eb = bi[103];
              o18_16 = fma(eb, g16_15, o18_16);
              o18_17 = fma(eb, g17_15, o18_17);
            }
            { const double eb = bi[104];
              o19_16 = fma(eb, g16_0, o19_16);
              o19_17 = fma(eb, g17_0, o19_17);
            }
            { const double eb = bi[105];
              o19_16 = fma(eb, g16_1, o19_16);
              o19_17 = fma(eb, g17_1, o19_17);
            }
            { const double eb = bi[106];
              o19_16 = fma(eb, g16_4, o19_16);
              o19_17 = fma(eb, g17_4, o19_17);
            }
            { const double eb = bi[107];
              o19_16 = fma(eb, g16_3, o19_16);
              o19_17 = fma(eb, g17_3, o19_17);
            }
            { const double eb = bi[108];
              o19_16 = fma(eb, g16_7, o19_16);
              o19_17 = fma(eb, g17_7, o19_17);
            }
            { const double eb = bi[109];
              o19_16 = fma(eb, g16_14, o19_16);
              o19_17 = fma(eb, g17_14, o19_17);
            }
            { const double eb = bi[110];
              o20_16 = fma(eb, g16_0, o20_16);
              o20_17 = fma(eb, g17_0, o20_17);
            }
            { const double eb = bi[111];
              o20_16 = fma(eb, g16_1, o20_16);
              o20_17 = fma(eb, g17_1, o20_17);
            }
            { const double eb = bi[112];
              o20_16 = fma(eb, g16_2, o20_16);
              o20_17 = fma(eb, g17_2, o20_17);
            }
            { const double eb = bi[113];
              o20_16 = fma(eb, g16_5, o20_16);
              o20_17 = fma(eb, g17_5, o20_17);
            }
            { const double eb = bi[114];
              o21_16 = fma(eb, g16_0, o21_16);
              o21_17 = fma(eb, g17_0, o21_17);
            }
            { const double eb = bi[115];
              o21_16 = fma(eb, g16_1, o21_16);
              o21_17 = fma(eb, g17_1, o21_17);
            }
            { const double eb = bi[116];
              o21_16 = fma(eb, g16_2, o21_16);
              o21_17 = fma(eb, g17_2, o21_17);
            }
            { const double eb = bi[117];
              o21_16 = fma(eb, g16_5, o21_16);
              o21_17 = fma(eb, g17_5, o21_17);
            }
            { const double eb = bi[118];
              o21_16 = fma(eb, g16_3, o21_16);
              o21_17 = fma(eb, g17_3, o21_17);
            }
            { const double eb = bi[119];
              o21_16 = fma(eb, g16_7, o21_16);
              o21_17 = fma(eb, g17_7, o21_17);
            }
            { const double eb = bi[120];
              o21_16 = fma(eb, g16_8, o21_16);
              o21_17 = fma(eb, g17_8, o21_17);
            }
            { const double eb = bi[121];
              o21_16 = fma(eb, g16_15, o21_16);
              o21_17 = fma(eb, g17_15, o21_17);
            }
            { const double eb = bi[122];
              o22_16 = fma(eb, g16_0, o22_16);
              o22_17 = fma(eb, g17_0, o22_17);
            }
            { const double eb = bi[123];
              o22_16 = fma(eb, g16_1, o22_16);
              o22_17 = fma(eb, g17_1, o22_17);
            }
            { const double eb = bi[124];
              o22_16 = fma(eb, g16_2, o22_16);
              o22_17 = fma(eb, g17_2, o22_17);
            }
            { const double eb = bi[125];
              o22_16 = fma(eb, g16_5, o22_16);
              o22_17 = fma(eb, g17_5, o22_17);
            }
            { const double eb = bi[126];
              o22_16 = fma(eb, g16_6, o22_16);
              o22_17 = fma(eb, g17_6, o22_17);
            }
            { const double eb = bi[127];
              o22_16 = fma(eb, g16_12, o22_16);
              o22_17 = fma(eb, g17_12, o22_17);
            }
            { const double eb = bi[128];
              o23_16 = fma(eb, g16_0, o23_16);
              o23_17 = fma(eb, g17_0, o23_17);
            }
            { const double eb = bi[129];
              o23_16 = fma(eb, g16_1, o23_16);
              o23_17 = fma(eb, g17_1, o23_17);
            }
            { const double eb = bi[130];
              o23_16 = fma(eb, g16_4, o23_16);
              o23_17 = fma(eb, g17_4, o23_17);
            }
            { const double eb = bi[131];
              o23_16 = fma(eb, g16_2, o23_16);
              o23_17 = fma(eb, g17_2, o23_17);
            }
            { const double eb = bi[132];
              o23_16 = fma(eb, g16_5, o23_16);
              o23_17 = fma(eb, g17_5, o23_17);
            }
            { const double eb = bi[133];
              o23_16 = fma(eb, g16_11, o23_16);
              o23_17 = fma(eb, g17_11, o23_17);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk16 = PT[(fI + 4) * N + fJ + 0];
            const double ptk17 = PT[(fI + 4) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_4 = PA[(fQ + 0) * N + fI + 4];
            const double Abc1_4 = PA[(fQ + 1) * N + fI + 4];
            const double Abc2_4 = PA[(fQ + 2) * N + fI + 4];
            const double Abc3_4 = PA[(fQ + 3) * N + fI + 4];
            const double Aac0_4 = PA[(fP + 0) * N + fI + 4];
            const double Aac1_4 = PA[(fP + 1) * N + fI + 4];
            const double Aac2_4 = PA[(fP + 2) * N + fI + 4];
            const double Aac3_4 = PA[(fP + 3) * N + fI + 4];
            const double Aac4_4 = PA[(fP + 4) * N + fI + 4];
            const double Aac5_4 = PA[(fP + 5) * N + fI + 4];
            jab0 += o0_16 * ptk16 + o0_17 * ptk17;
            jab1 += o1_16 * ptk16 + o1_17 * ptk17;
            jab2 += o2_16 * ptk16 + o2_17 * ptk17;
            jab3 += o3_16 * ptk16 + o3_17 * ptk17;
            jab4 += o4_16 * ptk16 + o4_17 * ptk17;
            jab5 += o5_16 * ptk16 + o5_17 * ptk17;
            jab6 += o6_16 * ptk16 + o6_17 * ptk17;
            jab7 += o7_16 * ptk16 + o7_17 * ptk17;
            jab8 += o8_16 * ptk16 + o8_17 * ptk17;
            jab9 += o9_16 * ptk16 + o9_17 * ptk17;
            jab10 += o10_16 * ptk16 + o10_17 * ptk17;
            jab11 += o11_16 * ptk16 + o11_17 * ptk17;
            jab12 += o12_16 * ptk16 + o12_17 * ptk17;
            jab13 += o13_16 * ptk16 + o13_17 * ptk17;
            jab14 += o14_16 * ptk16 + o14_17 * ptk17;
            jab15 += o15_16 * ptk16 + o15_17 * ptk17;
            jab16 += o16_16 * ptk16 + o16_17 * ptk17;
            jab17 += o17_16 * ptk16 + o17_17 * ptk17;
            jab18 += o18_16 * ptk16 + o18_17 * ptk17;
            jab19 += o19_16 * ptk16 + o19_17 * ptk17;
            jab20 += o20_16 * ptk16 + o20_17 * ptk17;
            jab21 += o21_16 * ptk16 + o21_17 * ptk17;
            jab22 += o22_16 * ptk16 + o22_17 * ptk17;
            jab23 += o23_16 * ptk16 + o23_17 * ptk17;
            atomicAdd(Jacc + (fI + 4) * N + fJ + 0, 2.0 * deg * (o0_16 * ptb0 + o1_16 * ptb1 + o2_16 * ptb2 + o3_16 * ptb3 + o4_16 * ptb4 + o5_16 * ptb5 + o6_16 * ptb6 + o7_16 * ptb7 + o8_16 * ptb8 + o9_16 * ptb9 + o10_16 * ptb10 + o11_16 * ptb11 + o12_16 * ptb12 + o13_16 * ptb13 + o14_16 * ptb14 + o15_16 * ptb15 + o16_16 * ptb16 + o17_16 * ptb17 + o18_16 * ptb18 + o19_16 * ptb19 + o20_16 * ptb20 + o21_16 * ptb21 + o22_16 * ptb22 + o23_16 * ptb23));
            atomicAdd(Jacc + (fI + 4) * N + fJ + 1, 2.0 * deg * (o0_17 * ptb0 + o1_17 * ptb1 + o2_17 * ptb2 + o3_17 * ptb3 + o4_17 * ptb4 + o5_17 * ptb5 + o6_17 * ptb6 + o7_17 * ptb7 + o8_17 * ptb8 + o9_17 * ptb9 + o10_17 * ptb10 + o11_17 * ptb11 + o12_17 * ptb12 + o13_17 * ptb13 + o14_17 * ptb14 + o15_17 * ptb15 + o16_17 * ptb16 + o17_17 * ptb17 + o18_17 * ptb18 + o19_17 * ptb19 + o20_17 * ptb20 + o21_17 * ptb21 + o22_17 * ptb22 + o23_17 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 4, deg * (o0_16 * Abd0_0 + o0_17 * Abd0_1 + o1_16 * Abd1_0 + o1_17 * Abd1_1 + o2_16 * Abd2_0 + o2_17 * Abd2_1 + o3_16 * Abd3_0 + o3_17 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 4, deg * (o0_16 * Aad0_0 + o0_17 * Aad0_1 + o4_16 * Aad1_0 + o4_17 * Aad1_1 + o8_16 * Aad2_0 + o8_17 * Aad2_1 + o12_16 * Aad3_0 + o12_17 * Aad3_1 + o16_16 * Aad4_0 + o16_17 * Aad4_1 + o20_16 * Aad5_0 + o20_17 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_16 * Abc0_4 + o1_16 * Abc1_4 + o2_16 * Abc2_4 + o3_16 * Abc3_4));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_16 * Aac0_4 + o4_16 * Aac1_4 + o8_16 * Aac2_4 + o12_16 * Aac3_4 + o16_16 * Aac4_4 + o20_16 * Aac5_4));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_17 * Abc0_4 + o1_17 * Abc1_4 + o2_17 * Abc2_4 + o3_17 * Abc3_4));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_17 * Aac0_4 + o4_17 * Aac1_4 + o8_17 * Aac2_4 + o12_17 * Aac3_4 + o16_17 * Aac4_4 + o20_17 * Aac5_4));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 4, deg * (o1_16 * Aad0_0 + o1_17 * Aad0_1 + o5_16 * Aad1_0 + o5_17 * Aad1_1 + o9_16 * Aad2_0 + o9_17 * Aad2_1 + o13_16 * Aad3_0 + o13_17 * Aad3_1 + o17_16 * Aad4_0 + o17_17 * Aad4_1 + o21_16 * Aad5_0 + o21_17 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_16 * Aac0_4 + o5_16 * Aac1_4 + o9_16 * Aac2_4 + o13_16 * Aac3_4 + o17_16 * Aac4_4 + o21_16 * Aac5_4));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_17 * Aac0_4 + o5_17 * Aac1_4 + o9_17 * Aac2_4 + o13_17 * Aac3_4 + o17_17 * Aac4_4 + o21_17 * Aac5_4));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 4, deg * (o2_16 * Aad0_0 + o2_17 * Aad0_1 + o6_16 * Aad1_0 + o6_17 * Aad1_1 + o10_16 * Aad2_0 + o10_17 * Aad2_1 + o14_16 * Aad3_0 + o14_17 * Aad3_1 + o18_16 * Aad4_0 + o18_17 * Aad4_1 + o22_16 * Aad5_0 + o22_17 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_16 * Aac0_4 + o6_16 * Aac1_4 + o10_16 * Aac2_4 + o14_16 * Aac3_4 + o18_16 * Aac4_4 + o22_16 * Aac5_4));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_17 * Aac0_4 + o6_17 * Aac1_4 + o10_17 * Aac2_4 + o14_17 * Aac3_4 + o18_17 * Aac4_4 + o22_17 * Aac5_4));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 4, deg * (o3_16 * Aad0_0 + o3_17 * Aad0_1 + o7_16 * Aad1_0 + o7_17 * Aad1_1 + o11_16 * Aad2_0 + o11_17 * Aad2_1 + o15_16 * Aad3_0 + o15_17 * Aad3_1 + o19_16 * Aad4_0 + o19_17 * Aad4_1 + o23_16 * Aad5_0 + o23_17 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_16 * Aac0_4 + o7_16 * Aac1_4 + o11_16 * Aac2_4 + o15_16 * Aac3_4 + o19_16 * Aac4_4 + o23_16 * Aac5_4));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_17 * Aac0_4 + o7_17 * Aac1_4 + o11_17 * Aac2_4 + o15_17 * Aac3_4 + o19_17 * Aac4_4 + o23_17 * Aac5_4));
            atomicAdd(KAacc + (fP + 1) * N + fI + 4, deg * (o4_16 * Abd0_0 + o4_17 * Abd0_1 + o5_16 * Abd1_0 + o5_17 * Abd1_1 + o6_16 * Abd2_0 + o6_17 * Abd2_1 + o7_16 * Abd3_0 + o7_17 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_16 * Abc0_4 + o5_16 * Abc1_4 + o6_16 * Abc2_4 + o7_16 * Abc3_4));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_17 * Abc0_4 + o5_17 * Abc1_4 + o6_17 * Abc2_4 + o7_17 * Abc3_4));
            atomicAdd(KAacc + (fP + 2) * N + fI + 4, deg * (o8_16 * Abd0_0 + o8_17 * Abd0_1 + o9_16 * Abd1_0 + o9_17 * Abd1_1 + o10_16 * Abd2_0 + o10_17 * Abd2_1 + o11_16 * Abd3_0 + o11_17 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_16 * Abc0_4 + o9_16 * Abc1_4 + o10_16 * Abc2_4 + o11_16 * Abc3_4));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_17 * Abc0_4 + o9_17 * Abc1_4 + o10_17 * Abc2_4 + o11_17 * Abc3_4));
            atomicAdd(KAacc + (fP + 3) * N + fI + 4, deg * (o12_16 * Abd0_0 + o12_17 * Abd0_1 + o13_16 * Abd1_0 + o13_17 * Abd1_1 + o14_16 * Abd2_0 + o14_17 * Abd2_1 + o15_16 * Abd3_0 + o15_17 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_16 * Abc0_4 + o13_16 * Abc1_4 + o14_16 * Abc2_4 + o15_16 * Abc3_4));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_17 * Abc0_4 + o13_17 * Abc1_4 + o14_17 * Abc2_4 + o15_17 * Abc3_4));
            atomicAdd(KAacc + (fP + 4) * N + fI + 4, deg * (o16_16 * Abd0_0 + o16_17 * Abd0_1 + o17_16 * Abd1_0 + o17_17 * Abd1_1 + o18_16 * Abd2_0 + o18_17 * Abd2_1 + o19_16 * Abd3_0 + o19_17 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_16 * Abc0_4 + o17_16 * Abc1_4 + o18_16 * Abc2_4 + o19_16 * Abc3_4));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_17 * Abc0_4 + o17_17 * Abc1_4 + o18_17 * Abc2_4 + o19_17 * Abc3_4));
            atomicAdd(KAacc + (fP + 5) * N + fI + 4, deg * (o20_16 * Abd0_0 + o20_17 * Abd0_1 + o21_16 * Abd1_0 + o21_17 * Abd1_1 + o22_16 * Abd2_0 + o22_17 * Abd2_1 + o23_16 * Abd3_0 + o23_17 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_16 * Abc0_4 + o21_16 * Abc1_4 + o22_16 * Abc2_4 + o23_16 * Abc3_4));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_17 * Abc0_4 + o21_17 * Abc1_4 + o22_17 * Abc2_4 + o23_17 * Abc3_4));
          }
        } break;
        case 9: {  // ket functions [18, 19]
          double o0_18 = 0;
          double o0_19 = 0;
          double o1_18 = 0;
          double o1_19 = 0;
          double o2_18 = 0;
          double o2_19 = 0;
          double o3_18 = 0;
          double o3_19 = 0;
          double o4_18 = 0;
          double o4_19 = 0;
          double o5_18 = 0;
          double o5_19 = 0;
          double o6_18 = 0;
          double o6_19 = 0;
          double o7_18 = 0;
          double o7_19 = 0;
          double o8_18 = 0;
          double o8_19 = 0;
          double o9_18 = 0;
          double o9_19 = 0;
          double o10_18 = 0;
          double o10_19 = 0;
          double o11_18 = 0;
          double o11_19 = 0;
          double o12_18 = 0;
          double o12_19 = 0;
          double o13_18 = 0;
          double o13_19 = 0;
          double o14_18 = 0;
          double o14_19 = 0;
          double o15_18 = 0;
          double o15_19 = 0;
          double o16_18 = 0;
          double o16_19 = 0;
          double o17_18 = 0;
          double o17_19 = 0;
          double o18_18 = 0;
          double o18_19 = 0;
          double o19_18 = 0;
          double o19_19 = 0;
          double o20_18 = 0;
          double o20_19 = 0;
          double o21_18 = 0;
          double o21_19 = 0;
          double o22_18 = 0;
          double o22_19 = 0;
          double o23_18 = 0;
          double o23_19 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g18_0 = 0;
            double g18_1 = 0;
            double g18_2 = 0;
            double g18_3 = 0;
            double g18_4 = 0;
            double g18_5 = 0;
            double g18_6 = 0;
            double g18_7 = 0;
            double g18_8 = 0;
            double g18_9 = 0;
            double g18_10 = 0;
            double g18_11 = 0;
            double g18_12 = 0;
            double g18_13 = 0;
            double g18_14 = 0;
            double g18_15 = 0;
            double g18_16 = 0;
            double g18_17 = 0;
            double g18_18 = 0;
            double g18_19 = 0;
            double g19_0 = 0;
            double g19_1 = 0;
            double g19_2 = 0;
            double g19_3 = 0;
            double g19_4 = 0;
            double g19_5 = 0;
            double g19_6 = 0;
            double g19_7 = 0;
            double g19_8 = 0;
            double g19_9 = 0;
            double g19_10 = 0;
            double g19_11 = 0;
            double g19_12 = 0;
            double g19_13 = 0;
            double g19_14 = 0;
            double g19_15 = 0;
            double g19_16 = 0;
            double g19_17 = 0;
            double g19_18 = 0;
            double g19_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek18_0 = kj[96 * kS];
              const double ek18_1 = -kj[97 * kS];
              const double ek18_2 = -kj[98 * kS];
              const double ek18_3 = kj[99 * kS];
              const double ek18_4 = -kj[100 * kS];
              const double ek18_5 = kj[101 * kS];
              const double ek18_6 = kj[102 * kS];
              const double ek18_7 = -kj[103 * kS];
              const double ek19_0 = kj[104 * kS];
              const double ek19_1 = -kj[105 * kS];
              const double ek19_2 = kj[106 * kS];
              const double ek19_3 = -kj[107 * kS];
              const double ek19_4 = kj[108 * kS];
              const double ek19_5 = -kj[109 * kS];
              g18_0 = fma(ek18_0, b0, g18_0);
              g19_0 = fma(ek19_0, b0, g19_0);
              const double r0_0_0_1 = Z * b1;
              g18_1 = fma(ek18_0, r0_0_0_1, g18_1);
              g18_0 = fma(ek18_1, r0_0_0_1, g18_0);
              g19_1 = fma(ek19_0, r0_0_0_1, g19_1);
              g19_0 = fma(ek19_1, r0_0_0_1, g19_0);
              const double r0_0_1_0 = Y * b1;
              g18_2 = fma(ek18_0, r0_0_1_0, g18_2);
              g18_0 = fma(ek18_2, r0_0_1_0, g18_0);
              g19_2 = fma(ek19_0, r0_0_1_0, g19_2);
              const double r0_1_0_0 = X * b1;
              g18_3 = fma(ek18_0, r0_1_0_0, g18_3);
              g18_0 = fma(ek18_4, r0_1_0_0, g18_0);
              g19_3 = fma(ek19_0, r0_1_0_0, g19_3);
              g19_0 = fma(ek19_3, r0_1_0_0, g19_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g18_4 = fma(ek18_0, r0_0_0_2, g18_4);
              g18_1 = fma(ek18_1, r0_0_0_2, g18_1);
              g19_4 = fma(ek19_0, r0_0_0_2, g19_4);
              g19_1 = fma(ek19_1, r0_0_0_2, g19_1);
              g19_0 = fma(ek19_2, r0_0_0_2, g19_0);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g18_5 = fma(ek18_0, r0_0_1_1, g18_5);
              g18_2 = fma(ek18_1, r0_0_1_1, g18_2);
              g18_1 = fma(ek18_2, r0_0_1_1, g18_1);
              g18_0 = fma(ek18_3, r0_0_1_1, g18_0);
              g19_5 = fma(ek19_0, r0_0_1_1, g19_5);
              g19_2 = fma(ek19_1, r0_0_1_1, g19_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g18_6 = fma(ek18_0, r0_0_2_0, g18_6);
              g18_2 = fma(ek18_2, r0_0_2_0, g18_2);
              g19_6 = fma(ek19_0, r0_0_2_0, g19_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g18_7 = fma(ek18_0, r0_1_0_1, g18_7);
              g18_3 = fma(ek18_1, r0_1_0_1, g18_3);
              g18_1 = fma(ek18_4, r0_1_0_1, g18_1);
              g18_0 = fma(ek18_5, r0_1_0_1, g18_0);
              g19_7 = fma(ek19_0, r0_1_0_1, g19_7);
              g19_3 = fma(ek19_1, r0_1_0_1, g19_3);
              g19_1 = fma(ek19_3, r0_1_0_1, g19_1);
              g19_0 = fma(ek19_4, r0_1_0_1, g19_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g18_8 = fma(ek18_0, r0_1_1_0, g18_8);
              g18_3 = fma(ek18_2, r0_1_1_0, g18_3);
              g18_2 = fma(ek18_4, r0_1_1_0, g18_2);
              g18_0 = fma(ek18_6, r0_1_1_0, g18_0);
              g19_8 = fma(ek19_0, r0_1_1_0, g19_8);
              g19_2 = fma(ek19_3, r0_1_1_0, g19_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g18_9 = fma(ek18_0, r0_2_0_0, g18_9);
              g18_3 = fma(ek18_4, r0_2_0_0, g18_3);
              g19_9 = fma(ek19_0, r0_2_0_0, g19_9);
              g19_3 = fma(ek19_3, r0_2_0_0, g19_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g18_10 = fma(ek18_0, r0_0_0_3, g18_10);
              g18_4 = fma(ek18_1, r0_0_0_3, g18_4);
              g19_10 = fma(ek19_0, r0_0_0_3, g19_10);
              g19_4 = fma(ek19_1, r0_0_0_3, g19_4);
              g19_1 = fma(ek19_2, r0_0_0_3, g19_1);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g18_11 = fma(ek18_0, r0_0_1_2, g18_11);
              g18_5 = fma(ek18_1, r0_0_1_2, g18_5);
              g18_4 = fma(ek18_2, r0_0_1_2, g18_4);
              g18_1 = fma(ek18_3, r0_0_1_2, g18_1);
              g19_11 = fma(ek19_0, r0_0_1_2, g19_11);
              g19_5 = fma(ek19_1, r0_0_1_2, g19_5);
              g19_2 = fma(ek19_2, r0_0_1_2, g19_2);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g18_12 = fma(ek18_0, r0_0_2_1, g18_12);
              g18_6 = fma(ek18_1, r0_0_2_1, g18_6);
              g18_5 = fma(ek18_2, r0_0_2_1, g18_5);
              g18_2 = fma(ek18_3, r0_0_2_1, g18_2);
              g19_12 = fma(ek19_0, r0_0_2_1, g19_12);
              g19_6 = fma(ek19_1, r0_0_2_1, g19_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g18_13 = fma(ek18_0, r0_0_3_0, g18_13);
              g18_6 = fma(ek18_2, r0_0_3_0, g18_6);
              g19_13 = fma(ek19_0, r0_0_3_0, g19_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g18_14 = fma(ek18_0, r0_1_0_2, g18_14);
              g18_7 = fma(ek18_1, r0_1_0_2, g18_7);
              g18_4 = fma(ek18_4, r0_1_0_2, g18_4);
              g18_1 = fma(ek18_5, r0_1_0_2, g18_1);
              g19_14 = fma(ek19_0, r0_1_0_2, g19_14);
              g19_7 = fma(ek19_1, r0_1_0_2, g19_7);
              g19_3 = fma(ek19_2, r0_1_0_2, g19_3);
              g19_4 = fma(ek19_3, r0_1_0_2, g19_4);
              g19_1 = fma(ek19_4, r0_1_0_2, g19_1);
              g19_0 = fma(ek19_5, r0_1_0_2, g19_0);
              const double r0_1_1_1 = X * r1_0_1_1;
              g18_15 = fma(ek18_0, r0_1_1_1, g18_15);
              g18_8 = fma(ek18_1, r0_1_1_1, g18_8);
              g18_7 = fma(ek18_2, r0_1_1_1, g18_7);
              g18_3 = fma(ek18_3, r0_1_1_1, g18_3);
              g18_5 = fma(ek18_4, r0_1_1_1, g18_5);
              g18_2 = fma(ek18_5, r0_1_1_1, g18_2);
              g18_1 = fma(ek18_6, r0_1_1_1, g18_1);
              g18_0 = fma(ek18_7, r0_1_1_1, g18_0);
              g19_15 = fma(ek19_0, r0_1_1_1, g19_15);
              g19_8 = fma(ek19_1, r0_1_1_1, g19_8);
              g19_5 = fma(ek19_3, r0_1_1_1, g19_5);
              g19_2 = fma(ek19_4, r0_1_1_1, g19_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g18_16 = fma(ek18_0, r0_1_2_0, g18_16);
              g18_8 = fma(ek18_2, r0_1_2_0, g18_8);
              g18_6 = fma(ek18_4, r0_1_2_0, g18_6);
              g18_2 = fma(ek18_6, r0_1_2_0, g18_2);
              g19_16 = fma(ek19_0, r0_1_2_0, g19_16);
              g19_6 = fma(ek19_3, r0_1_2_0, g19_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g18_17 = fma(ek18_0, r0_2_0_1, g18_17);
              g18_9 = fma(ek18_1, r0_2_0_1, g18_9);
              g18_7 = fma(ek18_4, r0_2_0_1, g18_7);
              g18_3 = fma(ek18_5, r0_2_0_1, g18_3);
              g19_17 = fma(ek19_0, r0_2_0_1, g19_17);
              g19_9 = fma(ek19_1, r0_2_0_1, g19_9);
              g19_7 = fma(ek19_3, r0_2_0_1, g19_7);
              g19_3 = fma(ek19_4, r0_2_0_1, g19_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g18_18 = fma(ek18_0, r0_2_1_0, g18_18);
              g18_9 = fma(ek18_2, r0_2_1_0, g18_9);
              g18_8 = fma(ek18_4, r0_2_1_0, g18_8);
              g18_3 = fma(ek18_6, r0_2_1_0, g18_3);
              g19_18 = fma(ek19_0, r0_2_1_0, g19_18);
              g19_8 = fma(ek19_3, r0_2_1_0, g19_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g18_19 = fma(ek18_0, r0_3_0_0, g18_19);
              g18_9 = fma(ek18_4, r0_3_0_0, g18_9);
              g19_19 = fma(ek19_0, r0_3_0_0, g19_19);
              g19_9 = fma(ek19_3, r0_3_0_0, g19_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g18_10 = fma(ek18_1, r0_0_0_4, g18_10);
              g19_10 = fma(ek19_1, r0_0_0_4, g19_10);
              g19_4 = fma(ek19_2, r0_0_0_4, g19_4);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g18_11 = fma(ek18_1, r0_0_1_3, g18_11);
              g18_10 = fma(ek18_2, r0_0_1_3, g18_10);
              g18_4 = fma(ek18_3, r0_0_1_3, g18_4);
              g19_11 = fma(ek19_1, r0_0_1_3, g19_11);
              g19_5 = fma(ek19_2, r0_0_1_3, g19_5);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g18_12 = fma(ek18_1, r0_0_2_2, g18_12);
              g18_11 = fma(ek18_2, r0_0_2_2, g18_11);
              g18_5 = fma(ek18_3, r0_0_2_2, g18_5);
              g19_12 = fma(ek19_1, r0_0_2_2, g19_12);
              g19_6 = fma(ek19_2, r0_0_2_2, g19_6);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g18_13 = fma(ek18_1, r0_0_3_1, g18_13);
              g18_12 = fma(ek18_2, r0_0_3_1, g18_12);
              g18_6 = fma(ek18_3, r0_0_3_1, g18_6);
              g19_13 = fma(ek19_1, r0_0_3_1, g19_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g18_13 = fma(ek18_2, r0_0_4_0, g18_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g18_14 = fma(ek18_1, r0_1_0_3, g18_14);
              g18_10 = fma(ek18_4, r0_1_0_3, g18_10);
              g18_4 = fma(ek18_5, r0_1_0_3, g18_4);
              g19_14 = fma(ek19_1, r0_1_0_3, g19_14);
              g19_7 = fma(ek19_2, r0_1_0_3, g19_7);
              g19_10 = fma(ek19_3, r0_1_0_3, g19_10);
              g19_4 = fma(ek19_4, r0_1_0_3, g19_4);
              g19_1 = fma(ek19_5, r0_1_0_3, g19_1);
              const double r0_1_1_2 = X * r1_0_1_2;
              g18_15 = fma(ek18_1, r0_1_1_2, g18_15);
              g18_14 = fma(ek18_2, r0_1_1_2, g18_14);
              g18_7 = fma(ek18_3, r0_1_1_2, g18_7);
              g18_11 = fma(ek18_4, r0_1_1_2, g18_11);
              g18_5 = fma(ek18_5, r0_1_1_2, g18_5);
              g18_4 = fma(ek18_6, r0_1_1_2, g18_4);
              g18_1 = fma(ek18_7, r0_1_1_2, g18_1);
              g19_15 = fma(ek19_1, r0_1_1_2, g19_15);
              g19_8 = fma(ek19_2, r0_1_1_2, g19_8);
              g19_11 = fma(ek19_3, r0_1_1_2, g19_11);
              g19_5 = fma(ek19_4, r0_1_1_2, g19_5);
              g19_2 = fma(ek19_5, r0_1_1_2, g19_2);
              const double r0_1_2_1 = X * r1_0_2_1;
              g18_16 = fma(ek18_1, r0_1_2_1, g18_16);
              g18_15 = fma(ek18_2, r0_1_2_1, g18_15);
              g18_8 = fma(ek18_3, r0_1_2_1, g18_8);
              g18_12 = fma(ek18_4, r0_1_2_1, g18_12);
              g18_6 = fma(ek18_5, r0_1_2_1, g18_6);
              g18_5 = fma(ek18_6, r0_1_2_1, g18_5);
              g18_2 = fma(ek18_7, r0_1_2_1, g18_2);
              g19_16 = fma(ek19_1, r0_1_2_1, g19_16);
              g19_12 = fma(ek19_3, r0_1_2_1, g19_12);
              g19_6 = fma(ek19_4, r0_1_2_1, g19_6);
              const double r0_1_3_0 = X * r1_0_3_0;
              g18_16 = fma(ek18_2, r0_1_3_0, g18_16);
              g18_13 = fma(ek18_4, r0_1_3_0, g18_13);
              g18_6 = fma(ek18_6, r0_1_3_0, g18_6);
              g19_13 = fma(ek19_3, r0_1_3_0, g19_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g18_17 = fma(ek18_1, r0_2_0_2, g18_17);
              g18_14 = fma(ek18_4, r0_2_0_2, g18_14);
              g18_7 = fma(ek18_5, r0_2_0_2, g18_7);
              g19_17 = fma(ek19_1, r0_2_0_2, g19_17);
              g19_9 = fma(ek19_2, r0_2_0_2, g19_9);
              g19_14 = fma(ek19_3, r0_2_0_2, g19_14);
              g19_7 = fma(ek19_4, r0_2_0_2, g19_7);
              g19_3 = fma(ek19_5, r0_2_0_2, g19_3);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g18_18 = fma(ek18_1, r0_2_1_1, g18_18);
              g18_17 = fma(ek18_2, r0_2_1_1, g18_17);
              g18_9 = fma(ek18_3, r0_2_1_1, g18_9);
              g18_15 = fma(ek18_4, r0_2_1_1, g18_15);
              g18_8 = fma(ek18_5, r0_2_1_1, g18_8);
              g18_7 = fma(ek18_6, r0_2_1_1, g18_7);
              g18_3 = fma(ek18_7, r0_2_1_1, g18_3);
              g19_18 = fma(ek19_1, r0_2_1_1, g19_18);
              g19_15 = fma(ek19_3, r0_2_1_1, g19_15);
              g19_8 = fma(ek19_4, r0_2_1_1, g19_8);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g18_18 = fma(ek18_2, r0_2_2_0, g18_18);
              g18_16 = fma(ek18_4, r0_2_2_0, g18_16);
              g18_8 = fma(ek18_6, r0_2_2_0, g18_8);
              g19_16 = fma(ek19_3, r0_2_2_0, g19_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g18_19 = fma(ek18_1, r0_3_0_1, g18_19);
              g18_17 = fma(ek18_4, r0_3_0_1, g18_17);
              g18_9 = fma(ek18_5, r0_3_0_1, g18_9);
              g19_19 = fma(ek19_1, r0_3_0_1, g19_19);
              g19_17 = fma(ek19_3, r0_3_0_1, g19_17);
              g19_9 = fma(ek19_4, r0_3_0_1, g19_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g18_19 = fma(ek18_2, r0_3_1_0, g18_19);
              g18_18 = fma(ek18_4, r0_3_1_0, g18_18);
              g18_9 = fma(ek18_6, r0_3_1_0, g18_9);
              g19_18 = fma(ek19_3, r0_3_1_0, g19_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g18_19 = fma(ek18_4, r0_4_0_0, g18_19);
              g19_19 = fma(ek19_3, r0_4_0_0, g19_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g19_10 = fma(ek19_2, r0_0_0_5, g19_10);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g18_10 = fma(ek18_3, r0_0_1_4, g18_10);
              g19_11 = fma(ek19_2, r0_0_1_4, g19_11);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g18_11 = fma(ek18_3, r0_0_2_3, g18_11);
              g19_12 = fma(ek19_2, r0_0_2_3, g19_12);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g18_12 = fma(ek18_3, r0_0_3_2, g18_12);
              g19_13 = fma(ek19_2, r0_0_3_2, g19_13);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g18_13 = fma(ek18_3, r0_0_4_1, g18_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g18_10 = fma(ek18_5, r0_1_0_4, g18_10);
              g19_14 = fma(ek19_2, r0_1_0_4, g19_14);
              g19_10 = fma(ek19_4, r0_1_0_4, g19_10);
              g19_4 = fma(ek19_5, r0_1_0_4, g19_4);
              const double r0_1_1_3 = X * r1_0_1_3;
              g18_14 = fma(ek18_3, r0_1_1_3, g18_14);
              g18_11 = fma(ek18_5, r0_1_1_3, g18_11);
              g18_10 = fma(ek18_6, r0_1_1_3, g18_10);
              g18_4 = fma(ek18_7, r0_1_1_3, g18_4);
              g19_15 = fma(ek19_2, r0_1_1_3, g19_15);
              g19_11 = fma(ek19_4, r0_1_1_3, g19_11);
              g19_5 = fma(ek19_5, r0_1_1_3, g19_5);
              const double r0_1_2_2 = X * r1_0_2_2;
              g18_15 = fma(ek18_3, r0_1_2_2, g18_15);
              g18_12 = fma(ek18_5, r0_1_2_2, g18_12);
              g18_11 = fma(ek18_6, r0_1_2_2, g18_11);
              g18_5 = fma(ek18_7, r0_1_2_2, g18_5);
              g19_16 = fma(ek19_2, r0_1_2_2, g19_16);
              g19_12 = fma(ek19_4, r0_1_2_2, g19_12);
              g19_6 = fma(ek19_5, r0_1_2_2, g19_6);
              const double r0_1_3_1 = X * r1_0_3_1;
              g18_16 = fma(ek18_3, r0_1_3_1, g18_16);
              g18_13 = fma(ek18_5, r0_1_3_1, g18_13);
              g18_12 = fma(ek18_6, r0_1_3_1, g18_12);
              g18_6 = fma(ek18_7, r0_1_3_1, g18_6);
              g19_13 = fma(ek19_4, r0_1_3_1, g19_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g18_13 = fma(ek18_6, r0_1_4_0, g18_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g18_14 = fma(ek18_5, r0_2_0_3, g18_14);
              g19_17 = fma(ek19_2, r0_2_0_3, g19_17);
              g19_14 = fma(ek19_4, r0_2_0_3, g19_14);
              g19_7 = fma(ek19_5, r0_2_0_3, g19_7);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g18_17 = fma(ek18_3, r0_2_1_2, g18_17);
              g18_15 = fma(ek18_5, r0_2_1_2, g18_15);
              g18_14 = fma(ek18_6, r0_2_1_2, g18_14);
              g18_7 = fma(ek18_7, r0_2_1_2, g18_7);
              g19_18 = fma(ek19_2, r0_2_1_2, g19_18);
              g19_15 = fma(ek19_4, r0_2_1_2, g19_15);
              g19_8 = fma(ek19_5, r0_2_1_2, g19_8);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g18_18 = fma(ek18_3, r0_2_2_1, g18_18);
              g18_16 = fma(ek18_5, r0_2_2_1, g18_16);
              g18_15 = fma(ek18_6, r0_2_2_1, g18_15);
              g18_8 = fma(ek18_7, r0_2_2_1, g18_8);
              g19_16 = fma(ek19_4, r0_2_2_1, g19_16);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g18_16 = fma(ek18_6, r0_2_3_0, g18_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g18_17 = fma(ek18_5, r0_3_0_2, g18_17);
              g19_19 = fma(ek19_2, r0_3_0_2, g19_19);
              g19_17 = fma(ek19_4, r0_3_0_2, g19_17);
              g19_9 = fma(ek19_5, r0_3_0_2, g19_9);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g18_19 = fma(ek18_3, r0_3_1_1, g18_19);
              g18_18 = fma(ek18_5, r0_3_1_1, g18_18);
              g18_17 = fma(ek18_6, r0_3_1_1, g18_17);
              g18_9 = fma(ek18_7, r0_3_1_1, g18_9);
              g19_18 = fma(ek19_4, r0_3_1_1, g19_18);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g18_18 = fma(ek18_6, r0_3_2_0, g18_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g18_19 = fma(ek18_5, r0_4_0_1, g18_19);
              g19_19 = fma(ek19_4, r0_4_0_1, g19_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g18_19 = fma(ek18_6, r0_4_1_0, g18_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_1_0_5 = X * r1_0_0_5;
              g19_10 = fma(ek19_5, r0_1_0_5, g19_10);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_1_1_4 = X * r1_0_1_4;
              g18_10 = fma(ek18_7, r0_1_1_4, g18_10);
              g19_11 = fma(ek19_5, r0_1_1_4, g19_11);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g18_11 = fma(ek18_7, r0_1_2_3, g18_11);
              g19_12 = fma(ek19_5, r0_1_2_3, g19_12);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g18_12 = fma(ek18_7, r0_1_3_2, g18_12);
              g19_13 = fma(ek19_5, r0_1_3_2, g19_13);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_1_4_1 = X * r1_0_4_1;
              g18_13 = fma(ek18_7, r0_1_4_1, g18_13);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g19_14 = fma(ek19_5, r0_2_0_4, g19_14);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g18_14 = fma(ek18_7, r0_2_1_3, g18_14);
              g19_15 = fma(ek19_5, r0_2_1_3, g19_15);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g18_15 = fma(ek18_7, r0_2_2_2, g18_15);
              g19_16 = fma(ek19_5, r0_2_2_2, g19_16);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g18_16 = fma(ek18_7, r0_2_3_1, g18_16);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g19_17 = fma(ek19_5, r0_3_0_3, g19_17);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g18_17 = fma(ek18_7, r0_3_1_2, g18_17);
              g19_18 = fma(ek19_5, r0_3_1_2, g19_18);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g18_18 = fma(ek18_7, r0_3_2_1, g18_18);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g19_19 = fma(ek19_5, r0_4_0_2, g19_19);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g18_19 = fma(ek18_7, r0_4_1_1, g18_19);
            }
            { const double eb = bi[5];
              o0_18 = fma(eb, g18_0, o0_18);
              o0_19 = fma(eb, g19_0, o0_19);
            }
            { const double eb = bi[6];
              o0_18 = fma(eb, g18_3, o0_18);
              o0_19 = fma(eb, g19_3, o0_19);
            }
            { const double eb = bi[7];
              o0_18 = fma(eb, g18_9, o0_18);
              o0_19 = fma(eb, g19_9, o0_19);
            }
            { const double eb = bi[8];
              o1_18 = fma(eb, g18_0, o1_18);
              o1_19 = fma(eb, g19_0, o1_19);
            }
            { const double eb = bi[9];
              o1_18 = fma(eb, g18_3, o1_18);
              o1_19 = fma(eb, g19_3, o1_19);
            }
            { const double eb = bi[10];
              o1_18 = fma(eb, g18_9, o1_18);
              o1_19 = fma(eb, g19_9, o1_19);
            }
            { const double eb = bi[11];
              o1_18 = fma(eb, g18_19, o1_18);
              o1_19 = fma(eb, g19_19, o1_19);
            }
            { const double eb = bi[12];
              o2_18 = fma(eb, g18_0, o2_18);
              o2_19 = fma(eb, g19_0, o2_19);
            }
            { const double eb = bi[13];
              o2_18 = fma(eb, g18_2, o2_18);
              o2_19 = fma(eb, g19_2, o2_19);
            }
            { const double eb = bi[14];
              o2_18 = fma(eb, g18_3, o2_18);
              o2_19 = fma(eb, g19_3, o2_19);
            }
            { const double eb = bi[15];
              o2_18 = fma(eb, g18_8, o2_18);
              o2_19 = fma(eb, g19_8, o2_19);
            }
            { const double eb = bi[16];
              o2_18 = fma(eb, g18_9, o2_18);
              o2_19 = fma(eb, g19_9, o2_19);
            }
            { const double eb = bi[17];
              o2_18 = fma(eb, g18_18, o2_18);
              o2_19 = fma(eb, g19_18, o2_19);
            }
            { const double eb = bi[18];
              o3_18 = fma(eb, g18_0, o3_18);
              o3_19 = fma(eb, g19_0, o3_19);
            }
            { const double eb = bi[19];
              o3_18 = fma(eb, g18_1, o3_18);
              o3_19 = fma(eb, g19_1, o3_19);
            }
            { const double eb = bi[20];
              o3_18 = fma(eb, g18_3, o3_18);
              o3_19 = fma(eb, g19_3, o3_19);
            }
            { const double eb = bi[21];
              o3_18 = fma(eb, g18_7, o3_18);
              o3_19 = fma(eb, g19_7, o3_19);
            }
            { const double eb = bi[22];
              o3_18 = fma(eb, g18_9, o3_18);
              o3_19 = fma(eb, g19_9, o3_19);
            }
            { const double eb = bi[23];
              o3_18 = fma(eb, g18_17, o3_18);
              o3_19 = fma(eb, g19_17, o3_19);
            }
            { const double eb = bi[24];
              o4_18 = fma(eb, g18_0, o4_18);
              o4_19 = fma(eb, g19_0, o4_19);
            }
            { const double eb = bi[25];
              o4_18 = fma(eb, g18_2, o4_18);
              o4_19 = fma(eb, g19_2, o4_19);
            }
            { const double eb = bi[26];
              o4_18 = fma(eb, g18_6, o4_18);
              o4_19 = fma(eb, g19_6, o4_19);
            }
            { const double eb = bi[27];
              o5_18 = fma(eb, g18_0, o5_18);
              o5_19 = fma(eb, g19_0, o5_19);
            }
            { const double eb = bi[28];
              o5_18 = fma(eb, g18_2, o5_18);
              o5_19 = fma(eb, g19_2, o5_19);
            }
            { const double eb = bi[29];
              o5_18 = fma(eb, g18_6, o5_18);
              o5_19 = fma(eb, g19_6, o5_19);
            }
            { const double eb = bi[30];
              o5_18 = fma(eb, g18_3, o5_18);
              o5_19 = fma(eb, g19_3, o5_19);
            }
            { const double eb = bi[31];
              o5_18 = fma(eb, g18_8, o5_18);
              o5_19 = fma(eb, g19_8, o5_19);
            }
            { const double eb = bi[32];
              o5_18 = fma(eb, g18_16, o5_18);
              o5_19 = fma(eb, g19_16, o5_19);
            }
            { const double eb = bi[33];
              o6_18 = fma(eb, g18_0, o6_18);
              o6_19 = fma(eb, g19_0, o6_19);
            }
            { const double eb = bi[34];
              o6_18 = fma(eb, g18_2, o6_18);
              o6_19 = fma(eb, g19_2, o6_19);
            }
            { const double eb = bi[35];
              o6_18 = fma(eb, g18_6, o6_18);
              o6_19 = fma(eb, g19_6, o6_19);
            }
            { const double eb = bi[36];
              o6_18 = fma(eb, g18_13, o6_18);
              o6_19 = fma(eb, g19_13, o6_19);
            }
            { const double eb = bi[37];
              o7_18 = fma(eb, g18_0, o7_18);
              o7_19 = fma(eb, g19_0, o7_19);
            }
            { const double eb = bi[38];
              o7_18 = fma(eb, g18_1, o7_18);
              o7_19 = fma(eb, g19_1, o7_19);
            }
            { const double eb = bi[39];
              o7_18 = fma(eb, g18_2, o7_18);
              o7_19 = fma(eb, g19_2, o7_19);
            }
            { const double eb = bi[40];
              o7_18 = fma(eb, g18_5, o7_18);
              o7_19 = fma(eb, g19_5, o7_19);
            }
            { const double eb = bi[41];
              o7_18 = fma(eb, g18_6, o7_18);
              o7_19 = fma(eb, g19_6, o7_19);
            }
            { const double eb = bi[42];
              o7_18 = fma(eb, g18_12, o7_18);
              o7_19 = fma(eb, g19_12, o7_19);
            }
            { const double eb = bi[43];
              o8_18 = fma(eb, g18_0, o8_18);
              o8_19 = fma(eb, g19_0, o8_19);
            }
            { const double eb = bi[44];
              o8_18 = fma(eb, g18_1, o8_18);
              o8_19 = fma(eb, g19_1, o8_19);
            }
            { const double eb = bi[45];
              o8_18 = fma(eb, g18_4, o8_18);
              o8_19 = fma(eb, g19_4, o8_19);
            }
            { const double eb = bi[46];
              o9_18 = fma(eb, g18_0, o9_18);
              o9_19 = fma(eb, g19_0, o9_19);
            }
            { const double eb = bi[47];
              o9_18 = fma(eb, g18_1, o9_18);
              o9_19 = fma(eb, g19_1, o9_19);
            }
            { const double eb = bi[48];
              o9_18 = fma(eb, g18_4, o9_18);
              o9_19 = fma(eb, g19_4, o9_19);
            }
            { const double eb = bi[49];
              o9_18 = fma(eb, g18_3, o9_18);
              o9_19 = fma(eb, g19_3, o9_19);
            }
            { const double eb = bi[50];
              o9_18 = fma(eb, g18_7, o9_18);
              o9_19 = fma(eb, g19_7, o9_19);
            }
            { const double eb = bi[51];
              o9_18 = fma(eb, g18_14, o9_18);
              o9_19 = fma(eb, g19_14, o9_19);
            }
            { const double eb = bi[52];
              o10_18 = fma(eb, g18_0, o10_18);
              o10_19 = fma(eb, g19_0, o10_19);
            }
            { const double eb = bi[53];
              o10_18 = fma(eb, g18_1, o10_18);
              o10_19 = fma(eb, g19_1, o10_19);
            }
            { const double eb = bi[54];
              o10_18 = fma(eb, g18_4, o10_18);
              o10_19 = fma(eb, g19_4, o10_19);
            }
            { const double eb = bi[55];
              o10_18 = fma(eb, g18_2, o10_18);
              o10_19 = fma(eb, g19_2, o10_19);
            }
            { const double eb = bi[56];
              o10_18 = fma(eb, g18_5, o10_18);
              o10_19 = fma(eb, g19_5, o10_19);
            }
            { const double eb = bi[57];
              o10_18 = fma(eb, g18_11, o10_18);
              o10_19 = fma(eb, g19_11, o10_19);
            }
            { const double eb = bi[58];
              o11_18 = fma(eb, g18_0, o11_18);
              o11_19 = fma(eb, g19_0, o11_19);
            }
            { const double eb = bi[59];
              o11_18 = fma(eb, g18_1, o11_18);
              o11_19 = fma(eb, g19_1, o11_19);
            }
            { const double eb = bi[60];
              o11_18 = fma(eb, g18_4, o11_18);
              o11_19 = fma(eb, g19_4, o11_19);
            }
            { const double eb = bi[61];
              o11_18 = fma(eb, g18_10, o11_18);
              o11_19 = fma(eb, g19_10, o11_19);
            }
            { const double eb = bi[62];
              o12_18 = fma(eb, g18_0, o12_18);
              o12_19 = fma(eb, g19_0, o12_19);
            }
            { const double eb = bi[63];
              o12_18 = fma(eb, g18_2, o12_18);
              o12_19 = fma(eb, g19_2, o12_19);
            }
            { const double eb = bi[64];
              o12_18 = fma(eb, g18_3, o12_18);
              o12_19 = fma(eb, g19_3, o12_19);
            }
            { const double eb = bi[65];
              o12_18 = fma(eb, g18_8, o12_18);
              o12_19 = fma(eb, g19_8, o12_19);
            }
            { const double eb = bi[66];
              o13_18 = fma(eb, g18_0, o13_18);
              o13_19 = fma(eb, g19_0, o13_19);
            }
            { const double eb = bi[67];
              o13_18 = fma(eb, g18_2, o13_18);
              o13_19 = fma(eb, g19_2, o13_19);
            }
            { const double eb = bi[68];
              o13_18 = fma(eb, g18_3, o13_18);
              o13_19 = fma(eb, g19_3, o13_19);
            }
            { const double eb = bi[69];
              o13_18 = fma(eb, g18_8, o13_18);
              o13_19 = fma(eb, g19_8, o13_19);
            }
            { const double eb = bi[70];
              o13_18 = fma(eb, g18_9, o13_18);
              o13_19 = fma(eb, g19_9, o13_19);
            }
            { const double eb = bi[71];
              o13_18 = fma(eb, g18_18, o13_18);
              o13_19 = fma(eb, g19_18, o13_19);
            }
            { const double eb = bi[72];
              o14_18 = fma(eb, g18_0, o14_18);
              o14_19 = fma(eb, g19_0, o14_19);
            }
            { const double eb = bi[73];
              o14_18 = fma(eb, g18_2, o14_18);
              o14_19 = fma(eb, g19_2, o14_19);
            }
            { const double eb = bi[74];
              o14_18 = fma(eb, g18_6, o14_18);
              o14_19 = fma(eb, g19_6, o14_19);
            }
            { const double eb = bi[75];
              o14_18 = fma(eb, g18_3, o14_18);
              o14_19 = fma(eb, g19_3, o14_19);
            }
            { const double eb = bi[76];
              o14_18 = fma(eb, g18_8, o14_18);
              o14_19 = fma(eb, g19_8, o14_19);
            }
            { const double eb = bi[77];
              o14_18 = fma(eb, g18_16, o14_18);
              o14_19 = fma(eb, g19_16, o14_19);
            }
            { const double eb = bi[78];
              o15_18 = fma(eb, g18_0, o15_18);
              o15_19 = fma(eb, g19_0, o15_19);
            }
            { const double eb = bi[79];
              o15_18 = fma(eb, g18_1, o15_18);
              o15_19 = fma(eb, g19_1, o15_19);
            }
            { const double eb = bi[80];
              o15_18 = fma(eb, g18_2, o15_18);
              o15_19 = fma(eb, g19_2, o15_19);
            }
            { const double eb = bi[81];
              o15_18 = fma(eb, g18_5, o15_18);
              o15_19 = fma(eb, g19_5, o15_19);
            }
            { const double eb = bi[82];
              o15_18 = fma(eb, g18_3, o15_18);
              o15_19 = fma(eb, g19_3, o15_19);
            }
            { const double eb = bi[83];
              o15_18 = fma(eb, g18_7, o15_18);
              o15_19 = fma(eb, g19_7, o15_19);
            }
            { const double eb = bi[84];
              o15_18 = fma(eb, g18_8, o15_18);
              o15_19 = fma(eb, g19_8, o15_19);
            }
            { const double eb = bi[85];
              o15_18 = fma(eb, g18_15, o15_18);
              o15_19 = fma(eb, g19_15, o15_19);
            }
            { const double eb = bi[86];
              o16_18 = fma(eb, g18_0, o16_18);
              o16_19 = fma(eb, g19_0, o16_19);
            }
            { const double eb = bi[87];
              o16_18 = fma(eb, g18_1, o16_18);
              o16_19 = fma(eb, g19_1, o16_19);
            }
            { const double eb = bi[88];
              o16_18 = fma(eb, g18_3, o16_18);
              o16_19 = fma(eb, g19_3, o16_19);
            }
            { const double eb = bi[89];
              o16_18 = fma(eb, g18_7, o16_18);
              o16_19 = fma(eb, g19_7, o16_19);
            }
            { const double eb = bi[90];
              o17_18 = fma(eb, g18_0, o17_18);
              o17_19 = fma(eb, g19_0, o17_19);
            }
            { const double eb = bi[91];
              o17_18 = fma(eb, g18_1, o17_18);
              o17_19 = fma(eb, g19_1, o17_19);
            }
            { const double eb = bi[92];
              o17_18 = fma(eb, g18_3, o17_18);
              o17_19 = fma(eb, g19_3, o17_19);
            }
            { const double eb = bi[93];
              o17_18 = fma(eb, g18_7, o17_18);
              o17_19 = fma(eb, g19_7, o17_19);
            }
            { const double eb = bi[94];
              o17_18 = fma(eb, g18_9, o17_18);
              o17_19 = fma(eb, g19_9, o17_19);
            }
            { const double eb = bi[95];
              o17_18 = fma(eb, g18_17, o17_18);
              o17_19 = fma(eb, g19_17, o17_19);
            }
            { const double eb = bi[96];
              o18_18 = fma(eb, g18_0, o18_18);
              o18_19 = fma(eb, g19_0, o18_19);
            }
            { const double eb = bi[97];
              o18_18 = fma(eb, g18_1, o18_18);
              o18_19 = fma(eb, g19_1, o18_19);
            }
            { const double eb = bi[98];
              o18_18 = fma(eb, g18_2, o18_18);
              o18_19 = fma(eb, g19_2, o18_19);
            }
            { const double eb = bi[99];
              o18_18 = fma(eb, g18_5, o18_18);
              o18_19 = fma(eb, g19_5, o18_19);
            }
            { const double eb = bi[100];
              o18_18 = fma(eb, g18_3, o18_18);
              o18_19 = fma(eb, g19_3, o18_19);
            }
            { const double eb = bi[101];
              o18_18 = fma(eb, g18_7, o18_18);
              o18_19 = fma(eb, g19_7, o18_19);
            }
            { const double eb = bi[102];
              o18_18 = fma(eb, g18_8, o18_18);
              o18_19 = fma(eb, g19_8, o18_19);
            }
            { const double eb = bi[103];
              o18_18 = fma(eb, g18_15, o18_18);
              o18_19 = fma(eb, g19_15, o18_19);
            }
            { const double eb = bi[104];
              o19_18 = fma(eb, g18_0, o19_18);
              o19_19 = fma(eb, g19_0, o19_19);
            }
            { const double eb = bi[105];
              o19_18 = fma(eb, g18_1, o19_18);
              o19_19 = fma(eb, g19_1, o19_19);
            }
            { const double eb = bi[106];
              o19_18 = fma(eb, g18_4, o19_18);
              o19_19 = fma(eb, g19_4, o19_19);
            }
            { const double eb = bi[107];
              o19_18 = fma(eb, g18_3, o19_18);
              o19_19 = fma(eb, g19_3, o19_19);
            }
            { const double eb = bi[108];
              o19_18 = fma(eb, g18_7, o19_18);
              o19_19 = fma(eb, g19_7, o19_19);
            }
            { const double eb = bi[109];
              o19_18 = fma(eb, g18_14, o19_18);
              o19_19 = fma(eb, g19_14, o19_19);
            }
            { const double eb = bi[110];
              o20_18 = fma(eb, g18_0, o20_18);
              o20_19 = fma(eb, g19_0, o20_19);
            }
            { const double eb = bi[111];
              o20_18 = fma(eb, g18_1, o20_18);
              o20_19 = fma(eb, g19_1, o20_19);
            }
            { const double eb = bi[112];
              o20_18 = fma(eb, g18_2, o20_18);
              o20_19 = fma(eb, g19_2, o20_19);
            }
            { const double eb = bi[113];
              o20_18 = fma(eb, g18_5, o20_18);
              o20_19 = fma(eb, g19_5, o20_19);
            }
            { const double eb = bi[114];
              o21_18 = fma(eb, g18_0, o21_18);
              o21_19 = fma(eb, g19_0, o21_19);
            }
            { const double eb = bi[115];
              o21_18 = fma(eb, g18_1, o21_18);
              o21_19 = fma(eb, g19_1, o21_19);
            }
            { const double eb = bi[116];
              o21_18 = fma(eb, g18_2, o21_18);
              o21_19 = fma(eb, g19_2, o21_19);
            }
            { const double eb = bi[117];
              o21_18 = fma(eb, g18_5, o21_18);
              o21_19 = fma(eb, g19_5, o21_19);
            }
            { const double eb = bi[118];
              o21_18 = fma(eb, g18_3, o21_18);
              o21_19 = fma(eb, g19_3, o21_19);
            }
            { const double eb = bi[119];
              o21_18 = fma(eb, g18_7, o21_18);
              o21_19 = fma(eb, g19_7, o21_19);
            }
            { const double eb = bi[120];
              o21_18 = fma(eb, g18_8, o21_18);
              o21_19 = fma(eb, g19_8, o21_19);
            }
            { const double eb = bi[121];
              o21_18 = fma(eb, g18_15, o21_18);
              o21_19 = fma(eb, g19_15, o21_19);
            }
            { const double eb = bi[122];
              o22_18 = fma(eb, g18_0, o22_18);
              o22_19 = fma(eb, g19_0, o22_19);
            }
            { const double eb = bi[123];
              o22_18 = fma(eb, g18_1, o22_18);
              o22_19 = fma(eb, g19_1, o22_19);
            }
            { const double eb = bi[124];
              o22_18 = fma(eb, g18_2, o22_18);
              o22_19 = fma(eb, g19_2, o22_19);
            }
            { const double eb = bi[125];
              o22_18 = fma(eb, g18_5, o22_18);
              o22_19 = fma(eb, g19_5, o22_19);
            }
            { const double eb = bi[126];
              o22_18 = fma(eb, g18_6, o22_18);
              o22_19 = fma(eb, g19_6, o22_19);
            }
            { const double eb = bi[127];
              o22_18 = fma(eb, g18_12, o22_18);
              o22_19 = fma(eb, g19_12, o22_19);
            }
            { const double eb = bi[128];
              o23_18 = fma(eb, g18_0, o23_18);
              o23_19 = fma(eb, g19_0, o23_19);
            }
            { const double eb = bi[129];
              o23_18 = fma(eb, g18_1, o23_18);
              o23_19 = fma(eb, g19_1, o23_19);
            }
            { const double eb = bi[130];
              o23_18 = fma(eb, g18_4, o23_18);
              o23_19 = fma(eb, g19_4, o23_19);
            }
            { const double eb = bi[131];
              o23_18 = fma(eb, g18_2, o23_18);
              o23_19 = fma(eb, g19_2, o23_19);
            }
            { const double eb = bi[132];
              o23_18 = fma(eb, g18_5, o23_18);
              o23_19 = fma(eb, g19_5, o23_19);
            }
            { const double eb = bi[133];
              o23_18 = fma(eb, g18_11, o23_18);
              o23_19 = fma(eb, g19_11, o23_19);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk18 = PT[(fI + 4) * N + fJ + 2];
            const double ptk19 = PT[(fI + 4) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_4 = PA[(fQ + 0) * N + fI + 4];
            const double Abc1_4 = PA[(fQ + 1) * N + fI + 4];
            const double Abc2_4 = PA[(fQ + 2) * N + fI + 4];
            const double Abc3_4 = PA[(fQ + 3) * N + fI + 4];
            const double Aac0_4 = PA[(fP + 0) * N + fI + 4];
            const double Aac1_4 = PA[(fP + 1) * N + fI + 4];
            const double Aac2_4 = PA[(fP + 2) * N + fI + 4];
            const double Aac3_4 = PA[(fP + 3) * N + fI + 4];
            const double Aac4_4 = PA[(fP + 4) * N + fI + 4];
            const double Aac5_4 = PA[(fP + 5) * N + fI + 4];
            jab0 += o0_18 * ptk18 + o0_19 * ptk19;
            jab1 += o1_18 * ptk18 + o1_19 * ptk19;
            jab2 += o2_18 * ptk18 + o2_19 * ptk19;
            jab3 += o3_18 * ptk18 + o3_19 * ptk19;
            jab4 += o4_18 * ptk18 + o4_19 * ptk19;
            jab5 += o5_18 * ptk18 + o5_19 * ptk19;
            jab6 += o6_18 * ptk18 + o6_19 * ptk19;
            jab7 += o7_18 * ptk18 + o7_19 * ptk19;
            jab8 += o8_18 * ptk18 + o8_19 * ptk19;
            jab9 += o9_18 * ptk18 + o9_19 * ptk19;
            jab10 += o10_18 * ptk18 + o10_19 * ptk19;
            jab11 += o11_18 * ptk18 + o11_19 * ptk19;
            jab12 += o12_18 * ptk18 + o12_19 * ptk19;
            jab13 += o13_18 * ptk18 + o13_19 * ptk19;
            jab14 += o14_18 * ptk18 + o14_19 * ptk19;
            jab15 += o15_18 * ptk18 + o15_19 * ptk19;
            jab16 += o16_18 * ptk18 + o16_19 * ptk19;
            jab17 += o17_18 * ptk18 + o17_19 * ptk19;
            jab18 += o18_18 * ptk18 + o18_19 * ptk19;
            jab19 += o19_18 * ptk18 + o19_19 * ptk19;
            jab20 += o20_18 * ptk18 + o20_19 * ptk19;
            jab21 += o21_18 * ptk18 + o21_19 * ptk19;
            jab22 += o22_18 * ptk18 + o22_19 * ptk19;
            jab23 += o23_18 * ptk18 + o23_19 * ptk19;
            atomicAdd(Jacc + (fI + 4) * N + fJ + 2, 2.0 * deg * (o0_18 * ptb0 + o1_18 * ptb1 + o2_18 * ptb2 + o3_18 * ptb3 + o4_18 * ptb4 + o5_18 * ptb5 + o6_18 * ptb6 + o7_18 * ptb7 + o8_18 * ptb8 + o9_18 * ptb9 + o10_18 * ptb10 + o11_18 * ptb11 + o12_18 * ptb12 + o13_18 * ptb13 + o14_18 * ptb14 + o15_18 * ptb15 + o16_18 * ptb16 + o17_18 * ptb17 + o18_18 * ptb18 + o19_18 * ptb19 + o20_18 * ptb20 + o21_18 * ptb21 + o22_18 * ptb22 + o23_18 * ptb23));
            atomicAdd(Jacc + (fI + 4) * N + fJ + 3, 2.0 * deg * (o0_19 * ptb0 + o1_19 * ptb1 + o2_19 * ptb2 + o3_19 * ptb3 + o4_19 * ptb4 + o5_19 * ptb5 + o6_19 * ptb6 + o7_19 * ptb7 + o8_19 * ptb8 + o9_19 * ptb9 + o10_19 * ptb10 + o11_19 * ptb11 + o12_19 * ptb12 + o13_19 * ptb13 + o14_19 * ptb14 + o15_19 * ptb15 + o16_19 * ptb16 + o17_19 * ptb17 + o18_19 * ptb18 + o19_19 * ptb19 + o20_19 * ptb20 + o21_19 * ptb21 + o22_19 * ptb22 + o23_19 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 4, deg * (o0_18 * Abd0_2 + o0_19 * Abd0_3 + o1_18 * Abd1_2 + o1_19 * Abd1_3 + o2_18 * Abd2_2 + o2_19 * Abd2_3 + o3_18 * Abd3_2 + o3_19 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 4, deg * (o0_18 * Aad0_2 + o0_19 * Aad0_3 + o4_18 * Aad1_2 + o4_19 * Aad1_3 + o8_18 * Aad2_2 + o8_19 * Aad2_3 + o12_18 * Aad3_2 + o12_19 * Aad3_3 + o16_18 * Aad4_2 + o16_19 * Aad4_3 + o20_18 * Aad5_2 + o20_19 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_18 * Abc0_4 + o1_18 * Abc1_4 + o2_18 * Abc2_4 + o3_18 * Abc3_4));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_18 * Aac0_4 + o4_18 * Aac1_4 + o8_18 * Aac2_4 + o12_18 * Aac3_4 + o16_18 * Aac4_4 + o20_18 * Aac5_4));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_19 * Abc0_4 + o1_19 * Abc1_4 + o2_19 * Abc2_4 + o3_19 * Abc3_4));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_19 * Aac0_4 + o4_19 * Aac1_4 + o8_19 * Aac2_4 + o12_19 * Aac3_4 + o16_19 * Aac4_4 + o20_19 * Aac5_4));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 4, deg * (o1_18 * Aad0_2 + o1_19 * Aad0_3 + o5_18 * Aad1_2 + o5_19 * Aad1_3 + o9_18 * Aad2_2 + o9_19 * Aad2_3 + o13_18 * Aad3_2 + o13_19 * Aad3_3 + o17_18 * Aad4_2 + o17_19 * Aad4_3 + o21_18 * Aad5_2 + o21_19 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_18 * Aac0_4 + o5_18 * Aac1_4 + o9_18 * Aac2_4 + o13_18 * Aac3_4 + o17_18 * Aac4_4 + o21_18 * Aac5_4));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_19 * Aac0_4 + o5_19 * Aac1_4 + o9_19 * Aac2_4 + o13_19 * Aac3_4 + o17_19 * Aac4_4 + o21_19 * Aac5_4));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 4, deg * (o2_18 * Aad0_2 + o2_19 * Aad0_3 + o6_18 * Aad1_2 + o6_19 * Aad1_3 + o10_18 * Aad2_2 + o10_19 * Aad2_3 + o14_18 * Aad3_2 + o14_19 * Aad3_3 + o18_18 * Aad4_2 + o18_19 * Aad4_3 + o22_18 * Aad5_2 + o22_19 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_18 * Aac0_4 + o6_18 * Aac1_4 + o10_18 * Aac2_4 + o14_18 * Aac3_4 + o18_18 * Aac4_4 + o22_18 * Aac5_4));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_19 * Aac0_4 + o6_19 * Aac1_4 + o10_19 * Aac2_4 + o14_19 * Aac3_4 + o18_19 * Aac4_4 + o22_19 * Aac5_4));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 4, deg * (o3_18 * Aad0_2 + o3_19 * Aad0_3 + o7_18 * Aad1_2 + o7_19 * Aad1_3 + o11_18 * Aad2_2 + o11_19 * Aad2_3 + o15_18 * Aad3_2 + o15_19 * Aad3_3 + o19_18 * Aad4_2 + o19_19 * Aad4_3 + o23_18 * Aad5_2 + o23_19 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_18 * Aac0_4 + o7_18 * Aac1_4 + o11_18 * Aac2_4 + o15_18 * Aac3_4 + o19_18 * Aac4_4 + o23_18 * Aac5_4));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_19 * Aac0_4 + o7_19 * Aac1_4 + o11_19 * Aac2_4 + o15_19 * Aac3_4 + o19_19 * Aac4_4 + o23_19 * Aac5_4));
            atomicAdd(KAacc + (fP + 1) * N + fI + 4, deg * (o4_18 * Abd0_2 + o4_19 * Abd0_3 + o5_18 * Abd1_2 + o5_19 * Abd1_3 + o6_18 * Abd2_2 + o6_19 * Abd2_3 + o7_18 * Abd3_2 + o7_19 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_18 * Abc0_4 + o5_18 * Abc1_4 + o6_18 * Abc2_4 + o7_18 * Abc3_4));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_19 * Abc0_4 + o5_19 * Abc1_4 + o6_19 * Abc2_4 + o7_19 * Abc3_4));
            atomicAdd(KAacc + (fP + 2) * N + fI + 4, deg * (o8_18 * Abd0_2 + o8_19 * Abd0_3 + o9_18 * Abd1_2 + o9_19 * Abd1_3 + o10_18 * Abd2_2 + o10_19 * Abd2_3 + o11_18 * Abd3_2 + o11_19 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_18 * Abc0_4 + o9_18 * Abc1_4 + o10_18 * Abc2_4 + o11_18 * Abc3_4));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_19 * Abc0_4 + o9_19 * Abc1_4 + o10_19 * Abc2_4 + o11_19 * Abc3_4));
            atomicAdd(KAacc + (fP + 3) * N + fI + 4, deg * (o12_18 * Abd0_2 + o12_19 * Abd0_3 + o13_18 * Abd1_2 + o13_19 * Abd1_3 + o14_18 * Abd2_2 + o14_19 * Abd2_3 + o15_18 * Abd3_2 + o15_19 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_18 * Abc0_4 + o13_18 * Abc1_4 + o14_18 * Abc2_4 + o15_18 * Abc3_4));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_19 * Abc0_4 + o13_19 * Abc1_4 + o14_19 * Abc2_4 + o15_19 * Abc3_4));
            atomicAdd(KAacc + (fP + 4) * N + fI + 4, deg * (o16_18 * Abd0_2 + o16_19 * Abd0_3 + o17_18 * Abd1_2 + o17_19 * Abd1_3 + o18_18 * Abd2_2 + o18_19 * Abd2_3 + o19_18 * Abd3_2 + o19_19 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_18 * Abc0_4 + o17_18 * Abc1_4 + o18_18 * Abc2_4 + o19_18 * Abc3_4));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_19 * Abc0_4 + o17_19 * Abc1_4 + o18_19 * Abc2_4 + o19_19 * Abc3_4));
            atomicAdd(KAacc + (fP + 5) * N + fI + 4, deg * (o20_18 * Abd0_2 + o20_19 * Abd0_3 + o21_18 * Abd1_2 + o21_19 * Abd1_3 + o22_18 * Abd2_2 + o22_19 * Abd2_3 + o23_18 * Abd3_2 + o23_19 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_18 * Abc0_4 + o21_18 * Abc1_4 + o22_18 * Abc2_4 + o23_18 * Abc3_4));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_19 * Abc0_4 + o21_19 * Abc1_4 + o22_19 * Abc2_4 + o23_19 * Abc3_4));
          }
        } break;
        case 10: {  // ket functions [20, 21]
          double o0_20 = 0;
          double o0_21 = 0;
          double o1_20 = 0;
          double o1_21 = 0;
          double o2_20 = 0;
          double o2_21 = 0;
          double o3_20 = 0;
          double o3_21 = 0;
          double o4_20 = 0;
          double o4_21 = 0;
          double o5_20 = 0;
          double o5_21 = 0;
          double o6_20 = 0;
          double o6_21 = 0;
          double o7_20 = 0;
          double o7_21 = 0;
          double o8_20 = 0;
          double o8_21 = 0;
          double o9_20 = 0;
          double o9_21 = 0;
          double o10_20 = 0;
          double o10_21 = 0;
          double o11_20 = 0;
          double o11_21 = 0;
          double o12_20 = 0;
          double o12_21 = 0;
          double o13_20 = 0;
          double o13_21 = 0;
          double o14_20 = 0;
          double o14_21 = 0;
          double o15_20 = 0;
          double o15_21 = 0;
          double o16_20 = 0;
          double o16_21 = 0;
          double o17_20 = 0;
          double o17_21 = 0;
          double o18_20 = 0;
          double o18_21 = 0;
          double o19_20 = 0;
          double o19_21 = 0;
          double o20_20 = 0;
          double o20_21 = 0;
          double o21_20 = 0;
          double o21_21 = 0;
          double o22_20 = 0;
          double o22_21 = 0;
          double o23_20 = 0;
          double o23_21 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g20_0 = 0;
            double g20_1 = 0;
            double g20_2 = 0;
            double g20_3 = 0;
            double g20_4 = 0;
            double g20_5 = 0;
            double g20_6 = 0;
            double g20_7 = 0;
            double g20_8 = 0;
            double g20_9 = 0;
            double g20_10 = 0;
            double g20_11 = 0;
            double g20_12 = 0;
            double g20_13 = 0;
            double g20_14 = 0;
            double g20_15 = 0;
            double g20_16 = 0;
            double g20_17 = 0;
            double g20_18 = 0;
            double g20_19 = 0;
            double g21_0 = 0;
            double g21_1 = 0;
            double g21_2 = 0;
            double g21_3 = 0;
            double g21_4 = 0;
            double g21_5 = 0;
            double g21_6 = 0;
            double g21_7 = 0;
            double g21_8 = 0;
            double g21_9 = 0;
            double g21_10 = 0;
            double g21_11 = 0;
            double g21_12 = 0;
            double g21_13 = 0;
            double g21_14 = 0;
            double g21_15 = 0;
            double g21_16 = 0;
            double g21_17 = 0;
            double g21_18 = 0;
            double g21_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek20_0 = kj[110 * kS];
              const double ek20_1 = -kj[111 * kS];
              const double ek20_2 = -kj[112 * kS];
              const double ek20_3 = kj[113 * kS];
              const double ek21_0 = kj[114 * kS];
              const double ek21_1 = -kj[115 * kS];
              const double ek21_2 = -kj[116 * kS];
              const double ek21_3 = kj[117 * kS];
              const double ek21_4 = -kj[118 * kS];
              const double ek21_5 = kj[119 * kS];
              const double ek21_6 = kj[120 * kS];
              const double ek21_7 = -kj[121 * kS];
              g20_0 = fma(ek20_0, b0, g20_0);
              g21_0 = fma(ek21_0, b0, g21_0);
              const double r0_0_0_1 = Z * b1;
              g20_1 = fma(ek20_0, r0_0_0_1, g20_1);
              g20_0 = fma(ek20_1, r0_0_0_1, g20_0);
              g21_1 = fma(ek21_0, r0_0_0_1, g21_1);
              g21_0 = fma(ek21_1, r0_0_0_1, g21_0);
              const double r0_0_1_0 = Y * b1;
              g20_2 = fma(ek20_0, r0_0_1_0, g20_2);
              g20_0 = fma(ek20_2, r0_0_1_0, g20_0);
              g21_2 = fma(ek21_0, r0_0_1_0, g21_2);
              g21_0 = fma(ek21_2, r0_0_1_0, g21_0);
              const double r0_1_0_0 = X * b1;
              g20_3 = fma(ek20_0, r0_1_0_0, g20_3);
              g21_3 = fma(ek21_0, r0_1_0_0, g21_3);
              g21_0 = fma(ek21_4, r0_1_0_0, g21_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g20_4 = fma(ek20_0, r0_0_0_2, g20_4);
              g20_1 = fma(ek20_1, r0_0_0_2, g20_1);
              g21_4 = fma(ek21_0, r0_0_0_2, g21_4);
              g21_1 = fma(ek21_1, r0_0_0_2, g21_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g20_5 = fma(ek20_0, r0_0_1_1, g20_5);
              g20_2 = fma(ek20_1, r0_0_1_1, g20_2);
              g20_1 = fma(ek20_2, r0_0_1_1, g20_1);
              g20_0 = fma(ek20_3, r0_0_1_1, g20_0);
              g21_5 = fma(ek21_0, r0_0_1_1, g21_5);
              g21_2 = fma(ek21_1, r0_0_1_1, g21_2);
              g21_1 = fma(ek21_2, r0_0_1_1, g21_1);
              g21_0 = fma(ek21_3, r0_0_1_1, g21_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g20_6 = fma(ek20_0, r0_0_2_0, g20_6);
              g20_2 = fma(ek20_2, r0_0_2_0, g20_2);
              g21_6 = fma(ek21_0, r0_0_2_0, g21_6);
              g21_2 = fma(ek21_2, r0_0_2_0, g21_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g20_7 = fma(ek20_0, r0_1_0_1, g20_7);
              g20_3 = fma(ek20_1, r0_1_0_1, g20_3);
              g21_7 = fma(ek21_0, r0_1_0_1, g21_7);
              g21_3 = fma(ek21_1, r0_1_0_1, g21_3);
              g21_1 = fma(ek21_4, r0_1_0_1, g21_1);
              g21_0 = fma(ek21_5, r0_1_0_1, g21_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g20_8 = fma(ek20_0, r0_1_1_0, g20_8);
              g20_3 = fma(ek20_2, r0_1_1_0, g20_3);
              g21_8 = fma(ek21_0, r0_1_1_0, g21_8);
              g21_3 = fma(ek21_2, r0_1_1_0, g21_3);
              g21_2 = fma(ek21_4, r0_1_1_0, g21_2);
              g21_0 = fma(ek21_6, r0_1_1_0, g21_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g20_9 = fma(ek20_0, r0_2_0_0, g20_9);
              g21_9 = fma(ek21_0, r0_2_0_0, g21_9);
              g21_3 = fma(ek21_4, r0_2_0_0, g21_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g20_10 = fma(ek20_0, r0_0_0_3, g20_10);
              g20_4 = fma(ek20_1, r0_0_0_3, g20_4);
              g21_10 = fma(ek21_0, r0_0_0_3, g21_10);
              g21_4 = fma(ek21_1, r0_0_0_3, g21_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g20_11 = fma(ek20_0, r0_0_1_2, g20_11);
              g20_5 = fma(ek20_1, r0_0_1_2, g20_5);
              g20_4 = fma(ek20_2, r0_0_1_2, g20_4);
              g20_1 = fma(ek20_3, r0_0_1_2, g20_1);
              g21_11 = fma(ek21_0, r0_0_1_2, g21_11);
              g21_5 = fma(ek21_1, r0_0_1_2, g21_5);
              g21_4 = fma(ek21_2, r0_0_1_2, g21_4);
              g21_1 = fma(ek21_3, r0_0_1_2, g21_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g20_12 = fma(ek20_0, r0_0_2_1, g20_12);
              g20_6 = fma(ek20_1, r0_0_2_1, g20_6);
              g20_5 = fma(ek20_2, r0_0_2_1, g20_5);
              g20_2 = fma(ek20_3, r0_0_2_1, g20_2);
              g21_12 = fma(ek21_0, r0_0_2_1, g21_12);
              g21_6 = fma(ek21_1, r0_0_2_1, g21_6);
              g21_5 = fma(ek21_2, r0_0_2_1, g21_5);
              g21_2 = fma(ek21_3, r0_0_2_1, g21_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g20_13 = fma(ek20_0, r0_0_3_0, g20_13);
              g20_6 = fma(ek20_2, r0_0_3_0, g20_6);
              g21_13 = fma(ek21_0, r0_0_3_0, g21_13);
              g21_6 = fma(ek21_2, r0_0_3_0, g21_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g20_14 = fma(ek20_0, r0_1_0_2, g20_14);
              g20_7 = fma(ek20_1, r0_1_0_2, g20_7);
              g21_14 = fma(ek21_0, r0_1_0_2, g21_14);
              g21_7 = fma(ek21_1, r0_1_0_2, g21_7);
              g21_4 = fma(ek21_4, r0_1_0_2, g21_4);
              g21_1 = fma(ek21_5, r0_1_0_2, g21_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g20_15 = fma(ek20_0, r0_1_1_1, g20_15);
              g20_8 = fma(ek20_1, r0_1_1_1, g20_8);
              g20_7 = fma(ek20_2, r0_1_1_1, g20_7);
              g20_3 = fma(ek20_3, r0_1_1_1, g20_3);
              g21_15 = fma(ek21_0, r0_1_1_1, g21_15);
              g21_8 = fma(ek21_1, r0_1_1_1, g21_8);
              g21_7 = fma(ek21_2, r0_1_1_1, g21_7);
              g21_3 = fma(ek21_3, r0_1_1_1, g21_3);
              g21_5 = fma(ek21_4, r0_1_1_1, g21_5);
              g21_2 = fma(ek21_5, r0_1_1_1, g21_2);
              g21_1 = fma(ek21_6, r0_1_1_1, g21_1);
              g21_0 = fma(ek21_7, r0_1_1_1, g21_0);
              const double r0_1_2_0 = X * r1_0_2_0;
              g20_16 = fma(ek20_0, r0_1_2_0, g20_16);
              g20_8 = fma(ek20_2, r0_1_2_0, g20_8);
              g21_16 = fma(ek21_0, r0_1_2_0, g21_16);
              g21_8 = fma(ek21_2, r0_1_2_0, g21_8);
              g21_6 = fma(ek21_4, r0_1_2_0, g21_6);
              g21_2 = fma(ek21_6, r0_1_2_0, g21_2);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g20_17 = fma(ek20_0, r0_2_0_1, g20_17);
              g20_9 = fma(ek20_1, r0_2_0_1, g20_9);
              g21_17 = fma(ek21_0, r0_2_0_1, g21_17);
              g21_9 = fma(ek21_1, r0_2_0_1, g21_9);
              g21_7 = fma(ek21_4, r0_2_0_1, g21_7);
              g21_3 = fma(ek21_5, r0_2_0_1, g21_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g20_18 = fma(ek20_0, r0_2_1_0, g20_18);
              g20_9 = fma(ek20_2, r0_2_1_0, g20_9);
              g21_18 = fma(ek21_0, r0_2_1_0, g21_18);
              g21_9 = fma(ek21_2, r0_2_1_0, g21_9);
              g21_8 = fma(ek21_4, r0_2_1_0, g21_8);
              g21_3 = fma(ek21_6, r0_2_1_0, g21_3);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g20_19 = fma(ek20_0, r0_3_0_0, g20_19);
              g21_19 = fma(ek21_0, r0_3_0_0, g21_19);
              g21_9 = fma(ek21_4, r0_3_0_0, g21_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g20_10 = fma(ek20_1, r0_0_0_4, g20_10);
              g21_10 = fma(ek21_1, r0_0_0_4, g21_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g20_11 = fma(ek20_1, r0_0_1_3, g20_11);
              g20_10 = fma(ek20_2, r0_0_1_3, g20_10);
              g20_4 = fma(ek20_3, r0_0_1_3, g20_4);
              g21_11 = fma(ek21_1, r0_0_1_3, g21_11);
              g21_10 = fma(ek21_2, r0_0_1_3, g21_10);
              g21_4 = fma(ek21_3, r0_0_1_3, g21_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g20_12 = fma(ek20_1, r0_0_2_2, g20_12);
              g20_11 = fma(ek20_2, r0_0_2_2, g20_11);
              g20_5 = fma(ek20_3, r0_0_2_2, g20_5);
              g21_12 = fma(ek21_1, r0_0_2_2, g21_12);
              g21_11 = fma(ek21_2, r0_0_2_2, g21_11);
              g21_5 = fma(ek21_3, r0_0_2_2, g21_5);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g20_13 = fma(ek20_1, r0_0_3_1, g20_13);
              g20_12 = fma(ek20_2, r0_0_3_1, g20_12);
              g20_6 = fma(ek20_3, r0_0_3_1, g20_6);
              g21_13 = fma(ek21_1, r0_0_3_1, g21_13);
              g21_12 = fma(ek21_2, r0_0_3_1, g21_12);
              g21_6 = fma(ek21_3, r0_0_3_1, g21_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g20_13 = fma(ek20_2, r0_0_4_0, g20_13);
              g21_13 = fma(ek21_2, r0_0_4_0, g21_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g20_14 = fma(ek20_1, r0_1_0_3, g20_14);
              g21_14 = fma(ek21_1, r0_1_0_3, g21_14);
              g21_10 = fma(ek21_4, r0_1_0_3, g21_10);
              g21_4 = fma(ek21_5, r0_1_0_3, g21_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g20_15 = fma(ek20_1, r0_1_1_2, g20_15);
              g20_14 = fma(ek20_2, r0_1_1_2, g20_14);
              g20_7 = fma(ek20_3, r0_1_1_2, g20_7);
              g21_15 = fma(ek21_1, r0_1_1_2, g21_15);
              g21_14 = fma(ek21_2, r0_1_1_2, g21_14);
              g21_7 = fma(ek21_3, r0_1_1_2, g21_7);
              g21_11 = fma(ek21_4, r0_1_1_2, g21_11);
              g21_5 = fma(ek21_5, r0_1_1_2, g21_5);
              g21_4 = fma(ek21_6, r0_1_1_2, g21_4);
              g21_1 = fma(ek21_7, r0_1_1_2, g21_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g20_16 = fma(ek20_1, r0_1_2_1, g20_16);
              g20_15 = fma(ek20_2, r0_1_2_1, g20_15);
              g20_8 = fma(ek20_3, r0_1_2_1, g20_8);
              g21_16 = fma(ek21_1, r0_1_2_1, g21_16);
              g21_15 = fma(ek21_2, r0_1_2_1, g21_15);
              g21_8 = fma(ek21_3, r0_1_2_1, g21_8);
              g21_12 = fma(ek21_4, r0_1_2_1, g21_12);
              g21_6 = fma(ek21_5, r0_1_2_1, g21_6);
              g21_5 = fma(ek21_6, r0_1_2_1, g21_5);
              g21_2 = fma(ek21_7, r0_1_2_1, g21_2);
              const double r0_1_3_0 = X * r1_0_3_0;
              g20_16 = fma(ek20_2, r0_1_3_0, g20_16);
              g21_16 = fma(ek21_2, r0_1_3_0, g21_16);
              g21_13 = fma(ek21_4, r0_1_3_0, g21_13);
              g21_6 = fma(ek21_6, r0_1_3_0, g21_6);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g20_17 = fma(ek20_1, r0_2_0_2, g20_17);
              g21_17 = fma(ek21_1, r0_2_0_2, g21_17);
              g21_14 = fma(ek21_4, r0_2_0_2, g21_14);
              g21_7 = fma(ek21_5, r0_2_0_2, g21_7);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g20_18 = fma(ek20_1, r0_2_1_1, g20_18);
              g20_17 = fma(ek20_2, r0_2_1_1, g20_17);
              g20_9 = fma(ek20_3, r0_2_1_1, g20_9);
              g21_18 = fma(ek21_1, r0_2_1_1, g21_18);
              g21_17 = fma(ek21_2, r0_2_1_1, g21_17);
              g21_9 = fma(ek21_3, r0_2_1_1, g21_9);
              g21_15 = fma(ek21_4, r0_2_1_1, g21_15);
              g21_8 = fma(ek21_5, r0_2_1_1, g21_8);
              g21_7 = fma(ek21_6, r0_2_1_1, g21_7);
              g21_3 = fma(ek21_7, r0_2_1_1, g21_3);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g20_18 = fma(ek20_2, r0_2_2_0, g20_18);
              g21_18 = fma(ek21_2, r0_2_2_0, g21_18);
              g21_16 = fma(ek21_4, r0_2_2_0, g21_16);
              g21_8 = fma(ek21_6, r0_2_2_0, g21_8);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g20_19 = fma(ek20_1, r0_3_0_1, g20_19);
              g21_19 = fma(ek21_1, r0_3_0_1, g21_19);
              g21_17 = fma(ek21_4, r0_3_0_1, g21_17);
              g21_9 = fma(ek21_5, r0_3_0_1, g21_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g20_19 = fma(ek20_2, r0_3_1_0, g20_19);
              g21_19 = fma(ek21_2, r0_3_1_0, g21_19);
              g21_18 = fma(ek21_4, r0_3_1_0, g21_18);
              g21_9 = fma(ek21_6, r0_3_1_0, g21_9);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g21_19 = fma(ek21_4, r0_4_0_0, g21_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g20_10 = fma(ek20_3, r0_0_1_4, g20_10);
              g21_10 = fma(ek21_3, r0_0_1_4, g21_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g20_11 = fma(ek20_3, r0_0_2_3, g20_11);
              g21_11 = fma(ek21_3, r0_0_2_3, g21_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g20_12 = fma(ek20_3, r0_0_3_2, g20_12);
              g21_12 = fma(ek21_3, r0_0_3_2, g21_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g20_13 = fma(ek20_3, r0_0_4_1, g20_13);
              g21_13 = fma(ek21_3, r0_0_4_1, g21_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g21_10 = fma(ek21_5, r0_1_0_4, g21_10);
              const double r0_1_1_3 = X * r1_0_1_3;
              g20_14 = fma(ek20_3, r0_1_1_3, g20_14);
              g21_14 = fma(ek21_3, r0_1_1_3, g21_14);
              g21_11 = fma(ek21_5, r0_1_1_3, g21_11);
              g21_10 = fma(ek21_6, r0_1_1_3, g21_10);
              g21_4 = fma(ek21_7, r0_1_1_3, g21_4);
              const double r0_1_2_2 = X * r1_0_2_2;
              g20_15 = fma(ek20_3, r0_1_2_2, g20_15);
              g21_15 = fma(ek21_3, r0_1_2_2, g21_15);
              g21_12 = fma(ek21_5, r0_1_2_2, g21_12);
              g21_11 = fma(ek21_6, r0_1_2_2, g21_11);
              g21_5 = fma(ek21_7, r0_1_2_2, g21_5);
              const double r0_1_3_1 = X * r1_0_3_1;
              g20_16 = fma(ek20_3, r0_1_3_1, g20_16);
              g21_16 = fma(ek21_3, r0_1_3_1, g21_16);
              g21_13 = fma(ek21_5, r0_1_3_1, g21_13);
              g21_12 = fma(ek21_6, r0_1_3_1, g21_12);
              g21_6 = fma(ek21_7, r0_1_3_1, g21_6);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g21_13 = fma(ek21_6, r0_1_4_0, g21_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g21_14 = fma(ek21_5, r0_2_0_3, g21_14);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g20_17 = fma(ek20_3, r0_2_1_2, g20_17);
              g21_17 = fma(ek21_3, r0_2_1_2, g21_17);
              g21_15 = fma(ek21_5, r0_2_1_2, g21_15);
              g21_14 = fma(ek21_6, r0_2_1_2, g21_14);
              g21_7 = fma(ek21_7, r0_2_1_2, g21_7);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g20_18 = fma(ek20_3, r0_2_2_1, g20_18);
              g21_18 = fma(ek21_3, r0_2_2_1, g21_18);
              g21_16 = fma(ek21_5, r0_2_2_1, g21_16);
              g21_15 = fma(ek21_6, r0_2_2_1, g21_15);
              g21_8 = fma(ek21_7, r0_2_2_1, g21_8);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g21_16 = fma(ek21_6, r0_2_3_0, g21_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g21_17 = fma(ek21_5, r0_3_0_2, g21_17);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g20_19 = fma(ek20_3, r0_3_1_1, g20_19);
              g21_19 = fma(ek21_3, r0_3_1_1, g21_19);
              g21_18 = fma(ek21_5, r0_3_1_1, g21_18);
              g21_17 = fma(ek21_6, r0_3_1_1, g21_17);
              g21_9 = fma(ek21_7, r0_3_1_1, g21_9);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g21_18 = fma(ek21_6, r0_3_2_0, g21_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g21_19 = fma(ek21_5, r0_4_0_1, g21_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g21_19 = fma(ek21_6, r0_4_1_0, g21_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_1_1_4 = X * r1_0_1_4;
              g21_10 = fma(ek21_7, r0_1_1_4, g21_10);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g21_11 = fma(ek21_7, r0_1_2_3, g21_11);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g21_12 = fma(ek21_7, r0_1_3_2, g21_12);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_1_4_1 = X * r1_0_4_1;
              g21_13 = fma(ek21_7, r0_1_4_1, g21_13);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g21_14 = fma(ek21_7, r0_2_1_3, g21_14);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g21_15 = fma(ek21_7, r0_2_2_2, g21_15);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g21_16 = fma(ek21_7, r0_2_3_1, g21_16);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g21_17 = fma(ek21_7, r0_3_1_2, g21_17);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g21_18 = fma(ek21_7, r0_3_2_1, g21_18);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g21_19 = fma(ek21_7, r0_4_1_1, g21_19);
            }
            { const double eb = bi[5];
              o0_20 = fma(eb, g20_0, o0_20);
              o0_21 = fma(eb, g21_0, o0_21);
            }
            { const double eb = bi[6];
              o0_20 = fma(eb, g20_3, o0_20);
              o0_21 = fma(eb, g21_3, o0_21);
            }
            { const double eb = bi[7];
              o0_20 = fma(eb, g20_9, o0_20);
              o0_21 = fma(eb, g21_9, o0_21);
            }
            { const double eb = bi[8];
              o1_20 = fma(eb, g20_0, o1_20);
              o1_21 = fma(eb, g21_0, o1_21);
            }
            { const double eb = bi[9];
              o1_20 = fma(eb, g20_3, o1_20);
              o1_21 = fma(eb, g21_3, o1_21);
            }
            { const double eb = bi[10];
              o1_20 = fma(eb, g20_9, o1_20);
              o1_21 = fma(eb, g21_9, o1_21);
            }
            { const double eb = bi[11];
              o1_20 = fma(eb, g20_19, o1_20);
              o1_21 = fma(eb, g21_19, o1_21);
            }
            { const double eb = bi[12];
              o2_20 = fma(eb, g20_0, o2_20);
              o2_21 = fma(eb, g21_0, o2_21);
            }
            { const double eb = bi[13];
              o2_20 = fma(eb, g20_2, o2_20);
              o2_21 = fma(eb, g21_2, o2_21);
            }
            { const double eb = bi[14];
              o2_20 = fma(eb, g20_3, o2_20);
              o2_21 = fma(eb, g21_3, o2_21);
            }
            { const double eb = bi[15];
              o2_20 = fma(eb, g20_8, o2_20);
              o2_21 = fma(eb, g21_8, o2_21);
            }
            { const double eb = bi[16];
              o2_20 = fma(eb, g20_9, o2_20);
              o2_21 = fma(eb, g21_9, o2_21);
            }
            { const double eb = bi[17];
              o2_20 = fma(eb, g20_18, o2_20);
              o2_21 = fma(eb, g21_18, o2_21);
            }
            { const double eb = bi[18];
              o3_20 = fma(eb, g20_0, o3_20);
              o3_21 = fma(eb, g21_0, o3_21);
            }
            { const double eb = bi[19];
              o3_20 = fma(eb, g20_1, o3_20);
              o3_21 = fma(eb, g21_1, o3_21);
            }
            { const double eb = bi[20];
              o3_20 = fma(eb, g20_3, o3_20);
              o3_21 = fma(eb, g21_3, o3_21);
            }
            { const double eb = bi[21];
              o3_20 = fma(eb, g20_7, o3_20);
              o3_21 = fma(eb, g21_7, o3_21);
            }
            { const double eb = bi[22];
              o3_20 = fma(eb, g20_9, o3_20);
              o3_21 = fma(eb, g21_9, o3_21);
            }
            { const double eb = bi[23];
              o3_20 = fma(eb, g20_17, o3_20);
              o3_21 = fma(eb, g21_17, o3_21);
            }
            { const double eb = bi[24];
              o4_20 = fma(eb, g20_0, o4_20);
              o4_21 = fma(eb, g21_0, o4_21);
            }
            { const double eb = bi[25];
              o4_20 = fma(eb, g20_2, o4_20);
              o4_21 = fma(eb, g21_2, o4_21);
            }
            { const double eb = bi[26];
              o4_20 = fma(eb, g20_6, o4_20);
              o4_21 = fma(eb, g21_6, o4_21);
            }
            { const double eb = bi[27];
              o5_20 = fma(eb, g20_0, o5_20);
              o5_21 = fma(eb, g21_0, o5_21);
            }
            { const double eb = bi[28];
              o5_20 = fma(eb, g20_2, o5_20);
              o5_21 = fma(eb, g21_2, o5_21);
            }
            { const double eb = bi[29];
              o5_20 = fma(eb, g20_6, o5_20);
              o5_21 = fma(eb, g21_6, o5_21);
            }
            { const double eb = bi[30];
              o5_20 = fma(eb, g20_3, o5_20);
              o5_21 = fma(eb, g21_3, o5_21);
            }
            { const double eb = bi[31];
              o5_20 = fma(eb, g20_8, o5_20);
              o5_21 = fma(eb, g21_8, o5_21);
            }
            { const double eb = bi[32];
              o5_20 = fma(eb, g20_16, o5_20);
              o5_21 = fma(eb, g21_16, o5_21);
            }
            { const double eb = bi[33];
              o6_20 = fma(eb, g20_0, o6_20);
              o6_21 = fma(eb, g21_0, o6_21);
            }
            { const double eb = bi[34];
              o6_20 = fma(eb, g20_2, o6_20);
              o6_21 = fma(eb, g21_2, o6_21);
            }
            { const double eb = bi[35];
              o6_20 = fma(eb, g20_6, o6_20);
              o6_21 = fma(eb, g21_6, o6_21);
            }
            { const double eb = bi[36];
              o6_20 = fma(eb, g20_13, o6_20);
              o6_21 = fma(eb, g21_13, o6_21);
            }
            { const double eb = bi[37];
              o7_20 = fma(eb, g20_0, o7_20);
              o7_21 = fma(eb, g21_0, o7_21);
            }
            { const double eb = bi[38];
              o7_20 = fma(eb, g20_1, o7_20);
              o7_21 = fma(eb, g21_1, o7_21);
            }
            { const double eb = bi[39];
              o7_20 = fma(eb, g20_2, o7_20);
              o7_21 = fma(eb, g21_2, o7_21);
            }
            { const double eb = bi[40];
              o7_20 = fma(eb, g20_5, o7_20);
              o7_21 = fma(eb, g21_5, o7_21);
            }
            { const double eb = bi[41];
              o7_20 = fma(eb, g20_6, o7_20);
              o7_21 = fma(eb, g21_6, o7_21);
            }
            { const double eb = bi[42];
              o7_20 = fma(eb, g20_12, o7_20);
              o7_21 = fma(eb, g21_12, o7_21);
            }
            { const double eb = bi[43];
              o8_20 = fma(eb, g20_0, o8_20);
              o8_21 = fma(eb, g21_0, o8_21);
            }
            { const double eb = bi[44];
              o8_20 = fma(eb, g20_1, o8_20);
              o8_21 = fma(eb, g21_1, o8_21);
            }
            { const double eb = bi[45];
              o8_20 = fma(eb, g20_4, o8_20);
              o8_21 = fma(eb, g21_4, o8_21);
            }
            { const double eb = bi[46];
              o9_20 = fma(eb, g20_0, o9_20);
              o9_21 = fma(eb, g21_0, o9_21);
            }
            { const double eb = bi[47];
              o9_20 = fma(eb, g20_1, o9_20);
              o9_21 = fma(eb, g21_1, o9_21);
            }
            { const double eb = bi[48];
              o9_20 = fma(eb, g20_4, o9_20);
              o9_21 = fma(eb, g21_4, o9_21);
            }
            { const double eb = bi[49];
              o9_20 = fma(eb, g20_3, o9_20);
              o9_21 = fma(eb, g21_3, o9_21);
            }
            { const double eb = bi[50];
              o9_20 = fma(eb, g20_7, o9_20);
              o9_21 = fma(eb, g21_7, o9_21);
            }
            { const double eb = bi[51];
              o9_20 = fma(eb, g20_14, o9_20);
              o9_21 = fma(eb, g21_14, o9_21);
            }
            { const double eb = bi[52];
              o10_20 = fma(eb, g20_0, o10_20);
              o10_21 = fma(eb, g21_0, o10_21);
            }
            { const double eb = bi[53];
              o10_20 = fma(eb, g20_1, o10_20);
              o10_21 = fma(eb, g21_1, o10_21);
            }
            { const double eb = bi[54];
              o10_20 = fma(eb, g20_4, o10_20);
              o10_21 = fma(eb, g21_4, o10_21);
            }
            { const double eb = bi[55];
              o10_20 = fma(eb, g20_2, o10_20);
              o10_21 = fma(eb, g21_2, o10_21);
            }
            { const double eb = bi[56];
              o10_20 = fma(eb, g20_5, o10_20);
              o10_21 = fma(eb, g21_5, o10_21);
            }
            { const double eb = bi[57];
              o10_20 = fma(eb, g20_11, o10_20);
              o10_21 = fma(eb, g21_11, o10_21);
            }
            { const double eb = bi[58];
              o11_20 = fma(eb, g20_0, o11_20);
              o11_21 = fma(eb, g21_0, o11_21);
            }
            { const double eb = bi[59];
              o11_20 = fma(eb, g20_1, o11_20);
              o11_21 = fma(eb, g21_1, o11_21);
            }
            { const double eb = bi[60];
              o11_20 = fma(eb, g20_4, o11_20);
              o11_21 = fma(eb, g21_4, o11_21);
            }
            { const double eb = bi[61];
              o11_20 = fma(eb, g20_10, o11_20);
              o11_21 = fma(eb, g21_10, o11_21);
            }
            { const double eb = bi[62];
              o12_20 = fma(eb, g20_0, o12_20);
              o12_21 = fma(eb, g21_0, o12_21);
            }
            { const double eb = bi[63];
              o12_20 = fma(eb, g20_2, o12_20);
              o12_21 = fma(eb, g21_2, o12_21);
            }
            { const double eb = bi[64];
              o12_20 = fma(eb, g20_3, o12_20);
              o12_21 = fma(eb, g21_3, o12_21);
            }
            { const double eb = bi[65];
              o12_20 = fma(eb, g20_8, o12_20);
              o12_21 = fma(eb, g21_8, o12_21);
            }
            { const double eb = bi[66];
              o13_20 = fma(eb, g20_0, o13_20);
              o13_21 = fma(eb, g21_0, o13_21);
            }
            { const double eb = bi[67];
              o13_20 = fma(eb, g20_2, o13_20);
              o13_21 = fma(eb, g21_2, o13_21);
            }
            { const double eb = bi[68];
              o13_20 = fma(eb, g20_3, o13_20);
              o13_21 = fma(eb, g21_3, o13_21);
            }
            { const double eb = bi[69];
              o13_20 = fma(eb, g20_8, o13_20);
              o13_21 = fma(eb, g21_8, o13_21);
            }
            { const double eb = bi[70];
              o13_20 = fma(eb, g20_9, o13_20);
              o13_21 = fma(eb, g21_9, o13_21);
            }
            { const double eb = bi[71];
              o13_20 = fma(eb, g20_18, o13_20);
              o13_21 = fma(eb, g21_18, o13_21);
            }
            { const double eb = bi[72];
              o14_20 = fma(eb, g20_0, o14_20);
              o14_21 = fma(eb, g21_0, o14_21);
            }
            { const double eb = bi[73];
              o14_20 = fma(eb, g20_2, o14_20);
              o14_21 = fma(eb, g21_2, o14_21);
            }
            { const double eb = bi[74];
              o14_20 = fma(eb, g20_6, o14_20);
              o14_21 = fma(eb, g21_6, o14_21);
            }
            { const double eb = bi[75];
              o14_20 = fma(eb, g20_3, o14_20);
              o14_21 = fma(eb, g21_3, o14_21);
            }
            { const double eb = bi[76];
              o14_20 = fma(eb, g20_8, o14_20);
              o14_21 = fma(eb, g21_8, o14_21);
            }
            { const double eb = bi[77];
              o14_20 = fma(eb, g20_16, o14_20);
              o14_21 = fma(eb, g21_16, o14_21);
            }
            { const double eb = bi[78];
              o15_20 = fma(eb, g20_0, o15_20);
              o15_21 = fma(eb, g21_0, o15_21);
            }
            { const double eb = bi[79];
              o15_20 = fma(eb, g20_1, o15_20);
              o15_21 = fma(eb, g21_1, o15_21);
            }
            { const double eb = bi[80];
              o15_20 = fma(eb, g20_2, o15_20);
              o15_21 = fma(eb, g21_2, o15_21);
            }
            { const double eb = bi[81];
              o15_20 = fma(eb, g20_5, o15_20);
              o15_21 = fma(eb, g21_5, o15_21);
            }
            { const double eb = bi[82];
              o15_20 = fma(eb, g20_3, o15_20);
              o15_21 = fma(eb, g21_3, o15_21);
            }
            { const double eb = bi[83];
              o15_20 = fma(eb, g20_7, o15_20);
              o15_21 = fma(eb, g21_7, o15_21);
            }
            { const double eb = bi[84];
              o15_20 = fma(eb, g20_8, o15_20);
              o15_21 = fma(eb, g21_8, o15_21);
            }
            { const double eb = bi[85];
              o15_20 = fma(eb, g20_15, o15_20);
              o15_21 = fma(eb, g21_15, o15_21);
            }
            { const double eb = bi[86];
              o16_20 = fma(eb, g20_0, o16_20);
              o16_21 = fma(eb, g21_0, o16_21);
            }
            { const double eb = bi[87];
              o16_20 = fma(eb, g20_1, o16_20);
              o16_21 = fma(eb, g21_1, o16_21);
            }
            { const double eb = bi[88];
              o16_20 = fma(eb, g20_3, o16_20);
              o16_21 = fma(eb, g21_3, o16_21);
            }
            { const double eb = bi[89];
              o16_20 = fma(eb, g20_7, o16_20);
              o16_21 = fma(eb, g21_7, o16_21);
            }
            { const double eb = bi[90];
              o17_20 = fma(eb, g20_0, o17_20);
              o17_21 = fma(eb, g21_0, o17_21);
            }
            { const double eb = bi[91];
              o17_20 = fma(eb, g20_1, o17_20);
              o17_21 = fma(eb, g21_1, o17_21);
            }
            { const double eb = bi[92];
              o17_20 = fma(eb, g20_3, o17_20);
              o17_21 = fma(eb, g21_3, o17_21);
            }
            { const double eb = bi[93];
              o17_20 = fma(eb, g20_7, o17_20);
              o17_21 = fma(eb, g21_7, o17_21);
            }
            { const double eb = bi[94];
              o17_20 = fma(eb, g20_9, o17_20);
              o17_21 = fma(eb, g21_9, o17_21);
            }
            { const double eb = bi[95];
              o17_20 = fma(eb, g20_17, o17_20);
              o17_21 = fma(eb, g21_17, o17_21);
            }
            { const double eb = bi[96];
              o18_20 = fma(eb, g20_0, o18_20);
              o18_21 = fma(eb, g21_0, o18_21);
            }
            { const double eb = bi[97];
              o18_20 = fma(eb, g20_1, o18_20);
              o18_21 = fma(eb, g21_1, o18_21);
            }
            { const double eb = bi[98];
              o18_20 = fma(eb, g20_2, o18_20);
              o18_21 = fma(eb, g21_2, o18_21);
            }
            { const double eb = bi[99];
              o18_20 = fma(eb, g20_5, o18_20);
              o18_21 = fma(eb, g21_5, o18_21);
            }
            { const double eb = bi[100];
              o18_20 = fma(eb, g20_3, o18_20);
              o18_21 = fma(eb, g21_3, o18_21);
            }
            { const double eb = bi[101];
              o18_20 = fma(eb, g20_7, o18_20);
              o18_21 = fma(eb, g21_7, o18_21);
            }
            { const double eb = bi[102];
              o18_20 = fma(eb, g20_8, o18_20);
              o18_21 = fma(eb, g21_8, o18_21);
            }
            { const double eb = bi[103];
              o18_20 = fma(eb, g20_15, o18_20);
              o18_21 = fma(eb, g21_15, o18_21);
            }
            { const double eb = bi[104];
              o19_20 = fma(eb, g20_0, o19_20);
              o19_21 = fma(eb, g21_0, o19_21);
            }
            { const double eb = bi[105];
              o19_20 = fma(eb, g20_1, o19_20);
              o19_21 = fma(eb, g21_1, o19_21);
            }
            { const double eb = bi[106];
              o19_20 = fma(eb, g20_4, o19_20);
              o19_21 = fma(eb, g21_4, o19_21);
            }
            { const double eb = bi[107];
              o19_20 = fma(eb, g20_3, o19_20);
              o19_21 = fma(eb, g21_3, o19_21);
            }
            { const double eb = bi[108];
              o19_20 = fma(eb, g20_7, o19_20);
              o19_21 = fma(eb, g21_7, o19_21);
            }
            { const double eb = bi[109];
              o19_20 = fma(eb, g20_14, o19_20);
              o19_21 = fma(eb, g21_14, o19_21);
            }
            { const double eb = bi[110];
              o20_20 = fma(eb, g20_0, o20_20);
              o20_21 = fma(eb, g21_0, o20_21);
            }
            { const double eb = bi[111];
              o20_20 = fma(eb, g20_1, o20_20);
              o20_21 = fma(eb, g21_1, o20_21);
            }
            { const double eb = bi[112];
              o20_20 = fma(eb, g20_2, o20_20);
              o20_21 = fma(eb, g21_2, o20_21);
            }
            { const double eb = bi[113];
              o20_20 = fma(eb, g20_5, o20_20);
              o20_21 = fma(eb, g21_5, o20_21);
            }
            { const double eb = bi[114];
              o21_20 = fma(eb, g20_0, o21_20);
              o21_21 = fma(eb, g21_0, o21_21);
            }
            { const double eb = bi[115];
              o21_20 = fma(eb, g20_1, o21_20);
              o21_21 = fma(eb, g21_1, o21_21);
            }
            { const double eb = bi[116];
              o21_20 = fma(eb, g20_2, o21_20);
              o21_21 = fma(eb, g21_2, o21_21);
            }
            { const double eb = bi[117];
              o21_20 = fma(eb, g20_5, o21_20);
              o21_21 = fma(eb, g21_5, o21_21);
            }
            { const double eb = bi[118];
              o21_20 = fma(eb, g20_3, o21_20);
              o21_21 = fma(eb, g21_3, o21_21);
            }
            { const double eb = bi[119];
              o21_20 = fma(eb, g20_7, o21_20);
              o21_21 = fma(eb, g21_7, o21_21);
            }
            { const double eb = bi[120];
              o21_20 = fma(eb, g20_8, o21_20);
              o21_21 = fma(eb, g21_8, o21_21);
            }
            { const double eb = bi[121];
              o21_20 = fma(eb, g20_15, o21_20);
              o21_21 = fma(eb, g21_15, o21_21);
            }
            { const double eb = bi[122];
              o22_20 = fma(eb, g20_0, o22_20);
              o22_21 = fma(eb, g21_0, o22_21);
            }
            { const double eb = bi[123];
              o22_20 = fma(eb, g20_1, o22_20);
              o22_21 = fma(eb, g21_1, o22_21);
            }
            { const double eb = bi[124];
              o22_20 = fma(eb, g20_2, o22_20);
              o22_21 = fma(eb, g21_2, o22_21);
            }
            { const double eb = bi[125];
              o22_20 = fma(eb, g20_5, o22_20);
              o22_21 = fma(eb, g21_5, o22_21);
            }
            { const double eb = bi[126];
              o22_20 = fma(eb, g20_6, o22_20);
              o22_21 = fma(eb, g21_6, o22_21);
            }
            { const double eb = bi[127];
              o22_20 = fma(eb, g20_12, o22_20);
              o22_21 = fma(eb, g21_12, o22_21);
            }
            { const double eb = bi[128];
              o23_20 = fma(eb, g20_0, o23_20);
              o23_21 = fma(eb, g21_0, o23_21);
            }
            { const double eb = bi[129];
              o23_20 = fma(eb, g20_1, o23_20);
              o23_21 = fma(eb, g21_1, o23_21);
            }
            { const double eb = bi[130];
              o23_20 = fma(eb, g20_4, o23_20);
              o23_21 = fma(eb, g21_4, o23_21);
            }
            { const double eb = bi[131];
              o23_20 = fma(eb, g20_2, o23_20);
              o23_21 = fma(eb, g21_2, o23_21);
            }
            { const double eb = bi[132];
              o23_20 = fma(eb, g20_5, o23_20);
              o23_21 = fma(eb, g21_5, o23_21);
            }
            { const double eb = bi[133];
              o23_20 = fma(eb, g20_11, o23_20);
              o23_21 = fma(eb, g21_11, o23_21);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk20 = PT[(fI + 5) * N + fJ + 0];
            const double ptk21 = PT[(fI + 5) * N + fJ + 1];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Aad5_1 = PA[(fP + 5) * N + fJ + 1];
            const double Abc0_5 = PA[(fQ + 0) * N + fI + 5];
            const double Abc1_5 = PA[(fQ + 1) * N + fI + 5];
            const double Abc2_5 = PA[(fQ + 2) * N + fI + 5];
            const double Abc3_5 = PA[(fQ + 3) * N + fI + 5];
            const double Aac0_5 = PA[(fP + 0) * N + fI + 5];
            const double Aac1_5 = PA[(fP + 1) * N + fI + 5];
            const double Aac2_5 = PA[(fP + 2) * N + fI + 5];
            const double Aac3_5 = PA[(fP + 3) * N + fI + 5];
            const double Aac4_5 = PA[(fP + 4) * N + fI + 5];
            const double Aac5_5 = PA[(fP + 5) * N + fI + 5];
            jab0 += o0_20 * ptk20 + o0_21 * ptk21;
            jab1 += o1_20 * ptk20 + o1_21 * ptk21;
            jab2 += o2_20 * ptk20 + o2_21 * ptk21;
            jab3 += o3_20 * ptk20 + o3_21 * ptk21;
            jab4 += o4_20 * ptk20 + o4_21 * ptk21;
            jab5 += o5_20 * ptk20 + o5_21 * ptk21;
            jab6 += o6_20 * ptk20 + o6_21 * ptk21;
            jab7 += o7_20 * ptk20 + o7_21 * ptk21;
            jab8 += o8_20 * ptk20 + o8_21 * ptk21;
            jab9 += o9_20 * ptk20 + o9_21 * ptk21;
            jab10 += o10_20 * ptk20 + o10_21 * ptk21;
            jab11 += o11_20 * ptk20 + o11_21 * ptk21;
            jab12 += o12_20 * ptk20 + o12_21 * ptk21;
            jab13 += o13_20 * ptk20 + o13_21 * ptk21;
            jab14 += o14_20 * ptk20 + o14_21 * ptk21;
            jab15 += o15_20 * ptk20 + o15_21 * ptk21;
            jab16 += o16_20 * ptk20 + o16_21 * ptk21;
            jab17 += o17_20 * ptk20 + o17_21 * ptk21;
            jab18 += o18_20 * ptk20 + o18_21 * ptk21;
            jab19 += o19_20 * ptk20 + o19_21 * ptk21;
            jab20 += o20_20 * ptk20 + o20_21 * ptk21;
            jab21 += o21_20 * ptk20 + o21_21 * ptk21;
            jab22 += o22_20 * ptk20 + o22_21 * ptk21;
            jab23 += o23_20 * ptk20 + o23_21 * ptk21;
            atomicAdd(Jacc + (fI + 5) * N + fJ + 0, 2.0 * deg * (o0_20 * ptb0 + o1_20 * ptb1 + o2_20 * ptb2 + o3_20 * ptb3 + o4_20 * ptb4 + o5_20 * ptb5 + o6_20 * ptb6 + o7_20 * ptb7 + o8_20 * ptb8 + o9_20 * ptb9 + o10_20 * ptb10 + o11_20 * ptb11 + o12_20 * ptb12 + o13_20 * ptb13 + o14_20 * ptb14 + o15_20 * ptb15 + o16_20 * ptb16 + o17_20 * ptb17 + o18_20 * ptb18 + o19_20 * ptb19 + o20_20 * ptb20 + o21_20 * ptb21 + o22_20 * ptb22 + o23_20 * ptb23));
            atomicAdd(Jacc + (fI + 5) * N + fJ + 1, 2.0 * deg * (o0_21 * ptb0 + o1_21 * ptb1 + o2_21 * ptb2 + o3_21 * ptb3 + o4_21 * ptb4 + o5_21 * ptb5 + o6_21 * ptb6 + o7_21 * ptb7 + o8_21 * ptb8 + o9_21 * ptb9 + o10_21 * ptb10 + o11_21 * ptb11 + o12_21 * ptb12 + o13_21 * ptb13 + o14_21 * ptb14 + o15_21 * ptb15 + o16_21 * ptb16 + o17_21 * ptb17 + o18_21 * ptb18 + o19_21 * ptb19 + o20_21 * ptb20 + o21_21 * ptb21 + o22_21 * ptb22 + o23_21 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 5, deg * (o0_20 * Abd0_0 + o0_21 * Abd0_1 + o1_20 * Abd1_0 + o1_21 * Abd1_1 + o2_20 * Abd2_0 + o2_21 * Abd2_1 + o3_20 * Abd3_0 + o3_21 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 5, deg * (o0_20 * Aad0_0 + o0_21 * Aad0_1 + o4_20 * Aad1_0 + o4_21 * Aad1_1 + o8_20 * Aad2_0 + o8_21 * Aad2_1 + o12_20 * Aad3_0 + o12_21 * Aad3_1 + o16_20 * Aad4_0 + o16_21 * Aad4_1 + o20_20 * Aad5_0 + o20_21 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_20 * Abc0_5 + o1_20 * Abc1_5 + o2_20 * Abc2_5 + o3_20 * Abc3_5));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_20 * Aac0_5 + o4_20 * Aac1_5 + o8_20 * Aac2_5 + o12_20 * Aac3_5 + o16_20 * Aac4_5 + o20_20 * Aac5_5));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_21 * Abc0_5 + o1_21 * Abc1_5 + o2_21 * Abc2_5 + o3_21 * Abc3_5));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_21 * Aac0_5 + o4_21 * Aac1_5 + o8_21 * Aac2_5 + o12_21 * Aac3_5 + o16_21 * Aac4_5 + o20_21 * Aac5_5));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 5, deg * (o1_20 * Aad0_0 + o1_21 * Aad0_1 + o5_20 * Aad1_0 + o5_21 * Aad1_1 + o9_20 * Aad2_0 + o9_21 * Aad2_1 + o13_20 * Aad3_0 + o13_21 * Aad3_1 + o17_20 * Aad4_0 + o17_21 * Aad4_1 + o21_20 * Aad5_0 + o21_21 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_20 * Aac0_5 + o5_20 * Aac1_5 + o9_20 * Aac2_5 + o13_20 * Aac3_5 + o17_20 * Aac4_5 + o21_20 * Aac5_5));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_21 * Aac0_5 + o5_21 * Aac1_5 + o9_21 * Aac2_5 + o13_21 * Aac3_5 + o17_21 * Aac4_5 + o21_21 * Aac5_5));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 5, deg * (o2_20 * Aad0_0 + o2_21 * Aad0_1 + o6_20 * Aad1_0 + o6_21 * Aad1_1 + o10_20 * Aad2_0 + o10_21 * Aad2_1 + o14_20 * Aad3_0 + o14_21 * Aad3_1 + o18_20 * Aad4_0 + o18_21 * Aad4_1 + o22_20 * Aad5_0 + o22_21 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_20 * Aac0_5 + o6_20 * Aac1_5 + o10_20 * Aac2_5 + o14_20 * Aac3_5 + o18_20 * Aac4_5 + o22_20 * Aac5_5));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_21 * Aac0_5 + o6_21 * Aac1_5 + o10_21 * Aac2_5 + o14_21 * Aac3_5 + o18_21 * Aac4_5 + o22_21 * Aac5_5));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 5, deg * (o3_20 * Aad0_0 + o3_21 * Aad0_1 + o7_20 * Aad1_0 + o7_21 * Aad1_1 + o11_20 * Aad2_0 + o11_21 * Aad2_1 + o15_20 * Aad3_0 + o15_21 * Aad3_1 + o19_20 * Aad4_0 + o19_21 * Aad4_1 + o23_20 * Aad5_0 + o23_21 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_20 * Aac0_5 + o7_20 * Aac1_5 + o11_20 * Aac2_5 + o15_20 * Aac3_5 + o19_20 * Aac4_5 + o23_20 * Aac5_5));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_21 * Aac0_5 + o7_21 * Aac1_5 + o11_21 * Aac2_5 + o15_21 * Aac3_5 + o19_21 * Aac4_5 + o23_21 * Aac5_5));
            atomicAdd(KAacc + (fP + 1) * N + fI + 5, deg * (o4_20 * Abd0_0 + o4_21 * Abd0_1 + o5_20 * Abd1_0 + o5_21 * Abd1_1 + o6_20 * Abd2_0 + o6_21 * Abd2_1 + o7_20 * Abd3_0 + o7_21 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_20 * Abc0_5 + o5_20 * Abc1_5 + o6_20 * Abc2_5 + o7_20 * Abc3_5));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_21 * Abc0_5 + o5_21 * Abc1_5 + o6_21 * Abc2_5 + o7_21 * Abc3_5));
            atomicAdd(KAacc + (fP + 2) * N + fI + 5, deg * (o8_20 * Abd0_0 + o8_21 * Abd0_1 + o9_20 * Abd1_0 + o9_21 * Abd1_1 + o10_20 * Abd2_0 + o10_21 * Abd2_1 + o11_20 * Abd3_0 + o11_21 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_20 * Abc0_5 + o9_20 * Abc1_5 + o10_20 * Abc2_5 + o11_20 * Abc3_5));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_21 * Abc0_5 + o9_21 * Abc1_5 + o10_21 * Abc2_5 + o11_21 * Abc3_5));
            atomicAdd(KAacc + (fP + 3) * N + fI + 5, deg * (o12_20 * Abd0_0 + o12_21 * Abd0_1 + o13_20 * Abd1_0 + o13_21 * Abd1_1 + o14_20 * Abd2_0 + o14_21 * Abd2_1 + o15_20 * Abd3_0 + o15_21 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_20 * Abc0_5 + o13_20 * Abc1_5 + o14_20 * Abc2_5 + o15_20 * Abc3_5));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_21 * Abc0_5 + o13_21 * Abc1_5 + o14_21 * Abc2_5 + o15_21 * Abc3_5));
            atomicAdd(KAacc + (fP + 4) * N + fI + 5, deg * (o16_20 * Abd0_0 + o16_21 * Abd0_1 + o17_20 * Abd1_0 + o17_21 * Abd1_1 + o18_20 * Abd2_0 + o18_21 * Abd2_1 + o19_20 * Abd3_0 + o19_21 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_20 * Abc0_5 + o17_20 * Abc1_5 + o18_20 * Abc2_5 + o19_20 * Abc3_5));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_21 * Abc0_5 + o17_21 * Abc1_5 + o18_21 * Abc2_5 + o19_21 * Abc3_5));
            atomicAdd(KAacc + (fP + 5) * N + fI + 5, deg * (o20_20 * Abd0_0 + o20_21 * Abd0_1 + o21_20 * Abd1_0 + o21_21 * Abd1_1 + o22_20 * Abd2_0 + o22_21 * Abd2_1 + o23_20 * Abd3_0 + o23_21 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_20 * Abc0_5 + o21_20 * Abc1_5 + o22_20 * Abc2_5 + o23_20 * Abc3_5));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_21 * Abc0_5 + o21_21 * Abc1_5 + o22_21 * Abc2_5 + o23_21 * Abc3_5));
          }
        } break;
        case 11: {  // ket functions [22, 23]
          double o0_22 = 0;
          double o0_23 = 0;
          double o1_22 = 0;
          double o1_23 = 0;
          double o2_22 = 0;
          double o2_23 = 0;
          double o3_22 = 0;
          double o3_23 = 0;
          double o4_22 = 0;
          double o4_23 = 0;
          double o5_22 = 0;
          double o5_23 = 0;
          double o6_22 = 0;
          double o6_23 = 0;
          double o7_22 = 0;
          double o7_23 = 0;
          double o8_22 = 0;
          double o8_23 = 0;
          double o9_22 = 0;
          double o9_23 = 0;
          double o10_22 = 0;
          double o10_23 = 0;
          double o11_22 = 0;
          double o11_23 = 0;
          double o12_22 = 0;
          double o12_23 = 0;
          double o13_22 = 0;
          double o13_23 = 0;
          double o14_22 = 0;
          double o14_23 = 0;
          double o15_22 = 0;
          double o15_23 = 0;
          double o16_22 = 0;
          double o16_23 = 0;
          double o17_22 = 0;
          double o17_23 = 0;
          double o18_22 = 0;
          double o18_23 = 0;
          double o19_22 = 0;
          double o19_23 = 0;
          double o20_22 = 0;
          double o20_23 = 0;
          double o21_22 = 0;
          double o21_23 = 0;
          double o22_22 = 0;
          double o22_23 = 0;
          double o23_22 = 0;
          double o23_23 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g22_0 = 0;
            double g22_1 = 0;
            double g22_2 = 0;
            double g22_3 = 0;
            double g22_4 = 0;
            double g22_5 = 0;
            double g22_6 = 0;
            double g22_7 = 0;
            double g22_8 = 0;
            double g22_9 = 0;
            double g22_10 = 0;
            double g22_11 = 0;
            double g22_12 = 0;
            double g22_13 = 0;
            double g22_14 = 0;
            double g22_15 = 0;
            double g22_16 = 0;
            double g22_17 = 0;
            double g22_18 = 0;
            double g22_19 = 0;
            double g23_0 = 0;
            double g23_1 = 0;
            double g23_2 = 0;
            double g23_3 = 0;
            double g23_4 = 0;
            double g23_5 = 0;
            double g23_6 = 0;
            double g23_7 = 0;
            double g23_8 = 0;
            double g23_9 = 0;
            double g23_10 = 0;
            double g23_11 = 0;
            double g23_12 = 0;
            double g23_13 = 0;
            double g23_14 = 0;
            double g23_15 = 0;
            double g23_16 = 0;
            double g23_17 = 0;
            double g23_18 = 0;
            double g23_19 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 134 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[7];
              sqb::boys<6>(T, a.boys_tab, F);
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
              w *= m2a;
              const double b6 = w * F[6];
              const double ek22_0 = kj[122 * kS];
              const double ek22_1 = -kj[123 * kS];
              const double ek22_2 = -kj[124 * kS];
              const double ek22_3 = kj[125 * kS];
              const double ek22_4 = kj[126 * kS];
              const double ek22_5 = -kj[127 * kS];
              const double ek23_0 = kj[128 * kS];
              const double ek23_1 = -kj[129 * kS];
              const double ek23_2 = kj[130 * kS];
              const double ek23_3 = -kj[131 * kS];
              const double ek23_4 = kj[132 * kS];
              const double ek23_5 = -kj[133 * kS];
              g22_0 = fma(ek22_0, b0, g22_0);
              g23_0 = fma(ek23_0, b0, g23_0);
              const double r0_0_0_1 = Z * b1;
              g22_1 = fma(ek22_0, r0_0_0_1, g22_1);
              g22_0 = fma(ek22_1, r0_0_0_1, g22_0);
              g23_1 = fma(ek23_0, r0_0_0_1, g23_1);
              g23_0 = fma(ek23_1, r0_0_0_1, g23_0);
              const double r0_0_1_0 = Y * b1;
              g22_2 = fma(ek22_0, r0_0_1_0, g22_2);
              g22_0 = fma(ek22_2, r0_0_1_0, g22_0);
              g23_2 = fma(ek23_0, r0_0_1_0, g23_2);
              g23_0 = fma(ek23_3, r0_0_1_0, g23_0);
              const double r0_1_0_0 = X * b1;
              g22_3 = fma(ek22_0, r0_1_0_0, g22_3);
              g23_3 = fma(ek23_0, r0_1_0_0, g23_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g22_4 = fma(ek22_0, r0_0_0_2, g22_4);
              g22_1 = fma(ek22_1, r0_0_0_2, g22_1);
              g23_4 = fma(ek23_0, r0_0_0_2, g23_4);
              g23_1 = fma(ek23_1, r0_0_0_2, g23_1);
              g23_0 = fma(ek23_2, r0_0_0_2, g23_0);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g22_5 = fma(ek22_0, r0_0_1_1, g22_5);
              g22_2 = fma(ek22_1, r0_0_1_1, g22_2);
              g22_1 = fma(ek22_2, r0_0_1_1, g22_1);
              g22_0 = fma(ek22_3, r0_0_1_1, g22_0);
              g23_5 = fma(ek23_0, r0_0_1_1, g23_5);
              g23_2 = fma(ek23_1, r0_0_1_1, g23_2);
              g23_1 = fma(ek23_3, r0_0_1_1, g23_1);
              g23_0 = fma(ek23_4, r0_0_1_1, g23_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g22_6 = fma(ek22_0, r0_0_2_0, g22_6);
              g22_2 = fma(ek22_2, r0_0_2_0, g22_2);
              g22_0 = fma(ek22_4, r0_0_2_0, g22_0);
              g23_6 = fma(ek23_0, r0_0_2_0, g23_6);
              g23_2 = fma(ek23_3, r0_0_2_0, g23_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g22_7 = fma(ek22_0, r0_1_0_1, g22_7);
              g22_3 = fma(ek22_1, r0_1_0_1, g22_3);
              g23_7 = fma(ek23_0, r0_1_0_1, g23_7);
              g23_3 = fma(ek23_1, r0_1_0_1, g23_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g22_8 = fma(ek22_0, r0_1_1_0, g22_8);
              g22_3 = fma(ek22_2, r0_1_1_0, g22_3);
              g23_8 = fma(ek23_0, r0_1_1_0, g23_8);
              g23_3 = fma(ek23_3, r0_1_1_0, g23_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g22_9 = fma(ek22_0, r0_2_0_0, g22_9);
              g23_9 = fma(ek23_0, r0_2_0_0, g23_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g22_10 = fma(ek22_0, r0_0_0_3, g22_10);
              g22_4 = fma(ek22_1, r0_0_0_3, g22_4);
              g23_10 = fma(ek23_0, r0_0_0_3, g23_10);
              g23_4 = fma(ek23_1, r0_0_0_3, g23_4);
              g23_1 = fma(ek23_2, r0_0_0_3, g23_1);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g22_11 = fma(ek22_0, r0_0_1_2, g22_11);
              g22_5 = fma(ek22_1, r0_0_1_2, g22_5);
              g22_4 = fma(ek22_2, r0_0_1_2, g22_4);
              g22_1 = fma(ek22_3, r0_0_1_2, g22_1);
              g23_11 = fma(ek23_0, r0_0_1_2, g23_11);
              g23_5 = fma(ek23_1, r0_0_1_2, g23_5);
              g23_2 = fma(ek23_2, r0_0_1_2, g23_2);
              g23_4 = fma(ek23_3, r0_0_1_2, g23_4);
              g23_1 = fma(ek23_4, r0_0_1_2, g23_1);
              g23_0 = fma(ek23_5, r0_0_1_2, g23_0);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g22_12 = fma(ek22_0, r0_0_2_1, g22_12);
              g22_6 = fma(ek22_1, r0_0_2_1, g22_6);
              g22_5 = fma(ek22_2, r0_0_2_1, g22_5);
              g22_2 = fma(ek22_3, r0_0_2_1, g22_2);
              g22_1 = fma(ek22_4, r0_0_2_1, g22_1);
              g22_0 = fma(ek22_5, r0_0_2_1, g22_0);
              g23_12 = fma(ek23_0, r0_0_2_1, g23_12);
              g23_6 = fma(ek23_1, r0_0_2_1, g23_6);
              g23_5 = fma(ek23_3, r0_0_2_1, g23_5);
              g23_2 = fma(ek23_4, r0_0_2_1, g23_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g22_13 = fma(ek22_0, r0_0_3_0, g22_13);
              g22_6 = fma(ek22_2, r0_0_3_0, g22_6);
              g22_2 = fma(ek22_4, r0_0_3_0, g22_2);
              g23_13 = fma(ek23_0, r0_0_3_0, g23_13);
              g23_6 = fma(ek23_3, r0_0_3_0, g23_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g22_14 = fma(ek22_0, r0_1_0_2, g22_14);
              g22_7 = fma(ek22_1, r0_1_0_2, g22_7);
              g23_14 = fma(ek23_0, r0_1_0_2, g23_14);
              g23_7 = fma(ek23_1, r0_1_0_2, g23_7);
              g23_3 = fma(ek23_2, r0_1_0_2, g23_3);
              const double r0_1_1_1 = X * r1_0_1_1;
              g22_15 = fma(ek22_0, r0_1_1_1, g22_15);
              g22_8 = fma(ek22_1, r0_1_1_1, g22_8);
              g22_7 = fma(ek22_2, r0_1_1_1, g22_7);
              g22_3 = fma(ek22_3, r0_1_1_1, g22_3);
              g23_15 = fma(ek23_0, r0_1_1_1, g23_15);
              g23_8 = fma(ek23_1, r0_1_1_1, g23_8);
              g23_7 = fma(ek23_3, r0_1_1_1, g23_7);
              g23_3 = fma(ek23_4, r0_1_1_1, g23_3);
              const double r0_1_2_0 = X * r1_0_2_0;
              g22_16 = fma(ek22_0, r0_1_2_0, g22_16);
              g22_8 = fma(ek22_2, r0_1_2_0, g22_8);
              g22_3 = fma(ek22_4, r0_1_2_0, g22_3);
              g23_16 = fma(ek23_0, r0_1_2_0, g23_16);
              g23_8 = fma(ek23_3, r0_1_2_0, g23_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g22_17 = fma(ek22_0, r0_2_0_1, g22_17);
              g22_9 = fma(ek22_1, r0_2_0_1, g22_9);
              g23_17 = fma(ek23_0, r0_2_0_1, g23_17);
              g23_9 = fma(ek23_1, r0_2_0_1, g23_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g22_18 = fma(ek22_0, r0_2_1_0, g22_18);
              g22_9 = fma(ek22_2, r0_2_1_0, g22_9);
              g23_18 = fma(ek23_0, r0_2_1_0, g23_18);
              g23_9 = fma(ek23_3, r0_2_1_0, g23_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g22_19 = fma(ek22_0, r0_3_0_0, g22_19);
              g23_19 = fma(ek23_0, r0_3_0_0, g23_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g22_10 = fma(ek22_1, r0_0_0_4, g22_10);
              g23_10 = fma(ek23_1, r0_0_0_4, g23_10);
              g23_4 = fma(ek23_2, r0_0_0_4, g23_4);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g22_11 = fma(ek22_1, r0_0_1_3, g22_11);
              g22_10 = fma(ek22_2, r0_0_1_3, g22_10);
              g22_4 = fma(ek22_3, r0_0_1_3, g22_4);
              g23_11 = fma(ek23_1, r0_0_1_3, g23_11);
              g23_5 = fma(ek23_2, r0_0_1_3, g23_5);
              g23_10 = fma(ek23_3, r0_0_1_3, g23_10);
              g23_4 = fma(ek23_4, r0_0_1_3, g23_4);
              g23_1 = fma(ek23_5, r0_0_1_3, g23_1);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g22_12 = fma(ek22_1, r0_0_2_2, g22_12);
              g22_11 = fma(ek22_2, r0_0_2_2, g22_11);
              g22_5 = fma(ek22_3, r0_0_2_2, g22_5);
              g22_4 = fma(ek22_4, r0_0_2_2, g22_4);
              g22_1 = fma(ek22_5, r0_0_2_2, g22_1);
              g23_12 = fma(ek23_1, r0_0_2_2, g23_12);
              g23_6 = fma(ek23_2, r0_0_2_2, g23_6);
              g23_11 = fma(ek23_3, r0_0_2_2, g23_11);
              g23_5 = fma(ek23_4, r0_0_2_2, g23_5);
              g23_2 = fma(ek23_5, r0_0_2_2, g23_2);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g22_13 = fma(ek22_1, r0_0_3_1, g22_13);
              g22_12 = fma(ek22_2, r0_0_3_1, g22_12);
              g22_6 = fma(ek22_3, r0_0_3_1, g22_6);
              g22_5 = fma(ek22_4, r0_0_3_1, g22_5);
              g22_2 = fma(ek22_5, r0_0_3_1, g22_2);
              g23_13 = fma(ek23_1, r0_0_3_1, g23_13);
              g23_12 = fma(ek23_3, r0_0_3_1, g23_12);
              g23_6 = fma(ek23_4, r0_0_3_1, g23_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g22_13 = fma(ek22_2, r0_0_4_0, g22_13);
              g22_6 = fma(ek22_4, r0_0_4_0, g22_6);
              g23_13 = fma(ek23_3, r0_0_4_0, g23_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g22_14 = fma(ek22_1, r0_1_0_3, g22_14);
              g23_14 = fma(ek23_1, r0_1_0_3, g23_14);
              g23_7 = fma(ek23_2, r0_1_0_3, g23_7);
              const double r0_1_1_2 = X * r1_0_1_2;
              g22_15 = fma(ek22_1, r0_1_1_2, g22_15);
              g22_14 = fma(ek22_2, r0_1_1_2, g22_14);
              g22_7 = fma(ek22_3, r0_1_1_2, g22_7);
              g23_15 = fma(ek23_1, r0_1_1_2, g23_15);
              g23_8 = fma(ek23_2, r0_1_1_2, g23_8);
              g23_14 = fma(ek23_3, r0_1_1_2, g23_14);
              g23_7 = fma(ek23_4, r0_1_1_2, g23_7);
              g23_3 = fma(ek23_5, r0_1_1_2, g23_3);
              const double r0_1_2_1 = X * r1_0_2_1;
              g22_16 = fma(ek22_1, r0_1_2_1, g22_16);
              g22_15 = fma(ek22_2, r0_1_2_1, g22_15);
              g22_8 = fma(ek22_3, r0_1_2_1, g22_8);
              g22_7 = fma(ek22_4, r0_1_2_1, g22_7);
              g22_3 = fma(ek22_5, r0_1_2_1, g22_3);
              g23_16 = fma(ek23_1, r0_1_2_1, g23_16);
              g23_15 = fma(ek23_3, r0_1_2_1, g23_15);
              g23_8 = fma(ek23_4, r0_1_2_1, g23_8);
              const double r0_1_3_0 = X * r1_0_3_0;
              g22_16 = fma(ek22_2, r0_1_3_0, g22_16);
              g22_8 = fma(ek22_4, r0_1_3_0, g22_8);
              g23_16 = fma(ek23_3, r0_1_3_0, g23_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g22_17 = fma(ek22_1, r0_2_0_2, g22_17);
              g23_17 = fma(ek23_1, r0_2_0_2, g23_17);
              g23_9 = fma(ek23_2, r0_2_0_2, g23_9);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g22_18 = fma(ek22_1, r0_2_1_1, g22_18);
              g22_17 = fma(ek22_2, r0_2_1_1, g22_17);
              g22_9 = fma(ek22_3, r0_2_1_1, g22_9);
              g23_18 = fma(ek23_1, r0_2_1_1, g23_18);
              g23_17 = fma(ek23_3, r0_2_1_1, g23_17);
              g23_9 = fma(ek23_4, r0_2_1_1, g23_9);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g22_18 = fma(ek22_2, r0_2_2_0, g22_18);
              g22_9 = fma(ek22_4, r0_2_2_0, g22_9);
              g23_18 = fma(ek23_3, r0_2_2_0, g23_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g22_19 = fma(ek22_1, r0_3_0_1, g22_19);
              g23_19 = fma(ek23_1, r0_3_0_1, g23_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g22_19 = fma(ek22_2, r0_3_1_0, g22_19);
              g23_19 = fma(ek23_3, r0_3_1_0, g23_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g23_10 = fma(ek23_2, r0_0_0_5, g23_10);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g22_10 = fma(ek22_3, r0_0_1_4, g22_10);
              g23_11 = fma(ek23_2, r0_0_1_4, g23_11);
              g23_10 = fma(ek23_4, r0_0_1_4, g23_10);
              g23_4 = fma(ek23_5, r0_0_1_4, g23_4);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g22_11 = fma(ek22_3, r0_0_2_3, g22_11);
              g22_10 = fma(ek22_4, r0_0_2_3, g22_10);
              g22_4 = fma(ek22_5, r0_0_2_3, g22_4);
              g23_12 = fma(ek23_2, r0_0_2_3, g23_12);
              g23_11 = fma(ek23_4, r0_0_2_3, g23_11);
              g23_5 = fma(ek23_5, r0_0_2_3, g23_5);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g22_12 = fma(ek22_3, r0_0_3_2, g22_12);
              g22_11 = fma(ek22_4, r0_0_3_2, g22_11);
              g22_5 = fma(ek22_5, r0_0_3_2, g22_5);
              g23_13 = fma(ek23_2, r0_0_3_2, g23_13);
              g23_12 = fma(ek23_4, r0_0_3_2, g23_12);
              g23_6 = fma(ek23_5, r0_0_3_2, g23_6);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g22_13 = fma(ek22_3, r0_0_4_1, g22_13);
              g22_12 = fma(ek22_4, r0_0_4_1, g22_12);
              g22_6 = fma(ek22_5, r0_0_4_1, g22_6);
              g23_13 = fma(ek23_4, r0_0_4_1, g23_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g22_13 = fma(ek22_4, r0_0_5_0, g22_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g23_14 = fma(ek23_2, r0_1_0_4, g23_14);
              const double r0_1_1_3 = X * r1_0_1_3;
              g22_14 = fma(ek22_3, r0_1_1_3, g22_14);
              g23_15 = fma(ek23_2, r0_1_1_3, g23_15);
              g23_14 = fma(ek23_4, r0_1_1_3, g23_14);
              g23_7 = fma(ek23_5, r0_1_1_3, g23_7);
              const double r0_1_2_2 = X * r1_0_2_2;
              g22_15 = fma(ek22_3, r0_1_2_2, g22_15);
              g22_14 = fma(ek22_4, r0_1_2_2, g22_14);
              g22_7 = fma(ek22_5, r0_1_2_2, g22_7);
              g23_16 = fma(ek23_2, r0_1_2_2, g23_16);
              g23_15 = fma(ek23_4, r0_1_2_2, g23_15);
              g23_8 = fma(ek23_5, r0_1_2_2, g23_8);
              const double r0_1_3_1 = X * r1_0_3_1;
              g22_16 = fma(ek22_3, r0_1_3_1, g22_16);
              g22_15 = fma(ek22_4, r0_1_3_1, g22_15);
              g22_8 = fma(ek22_5, r0_1_3_1, g22_8);
              g23_16 = fma(ek23_4, r0_1_3_1, g23_16);
              const double r0_1_4_0 = X * r1_0_4_0;
              g22_16 = fma(ek22_4, r0_1_4_0, g22_16);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g23_17 = fma(ek23_2, r0_2_0_3, g23_17);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g22_17 = fma(ek22_3, r0_2_1_2, g22_17);
              g23_18 = fma(ek23_2, r0_2_1_2, g23_18);
              g23_17 = fma(ek23_4, r0_2_1_2, g23_17);
              g23_9 = fma(ek23_5, r0_2_1_2, g23_9);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g22_18 = fma(ek22_3, r0_2_2_1, g22_18);
              g22_17 = fma(ek22_4, r0_2_2_1, g22_17);
              g22_9 = fma(ek22_5, r0_2_2_1, g22_9);
              g23_18 = fma(ek23_4, r0_2_2_1, g23_18);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g22_18 = fma(ek22_4, r0_2_3_0, g22_18);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g23_19 = fma(ek23_2, r0_3_0_2, g23_19);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g22_19 = fma(ek22_3, r0_3_1_1, g22_19);
              g23_19 = fma(ek23_4, r0_3_1_1, g23_19);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g22_19 = fma(ek22_4, r0_3_2_0, g22_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_0_1_5 = Y * r1_0_0_5;
              g23_10 = fma(ek23_5, r0_0_1_5, g23_10);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_0_2_4 = fma(Y, r1_0_1_4, r1_0_0_4);
              g22_10 = fma(ek22_5, r0_0_2_4, g22_10);
              g23_11 = fma(ek23_5, r0_0_2_4, g23_11);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_0_3_3 = fma(Y, r1_0_2_3, 2.0 * r1_0_1_3);
              g22_11 = fma(ek22_5, r0_0_3_3, g22_11);
              g23_12 = fma(ek23_5, r0_0_3_3, g23_12);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_0_4_2 = fma(Y, r1_0_3_2, 3.0 * r1_0_2_2);
              g22_12 = fma(ek22_5, r0_0_4_2, g22_12);
              g23_13 = fma(ek23_5, r0_0_4_2, g23_13);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_0_5_1 = fma(Y, r1_0_4_1, 4.0 * r1_0_3_1);
              g22_13 = fma(ek22_5, r0_0_5_1, g22_13);
              const double r0_1_1_4 = X * r1_0_1_4;
              g23_14 = fma(ek23_5, r0_1_1_4, g23_14);
              const double r0_1_2_3 = X * r1_0_2_3;
              g22_14 = fma(ek22_5, r0_1_2_3, g22_14);
              g23_15 = fma(ek23_5, r0_1_2_3, g23_15);
              const double r0_1_3_2 = X * r1_0_3_2;
              g22_15 = fma(ek22_5, r0_1_3_2, g22_15);
              g23_16 = fma(ek23_5, r0_1_3_2, g23_16);
              const double r0_1_4_1 = X * r1_0_4_1;
              g22_16 = fma(ek22_5, r0_1_4_1, g22_16);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g23_17 = fma(ek23_5, r0_2_1_3, g23_17);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g22_17 = fma(ek22_5, r0_2_2_2, g22_17);
              g23_18 = fma(ek23_5, r0_2_2_2, g23_18);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g22_18 = fma(ek22_5, r0_2_3_1, g22_18);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g23_19 = fma(ek23_5, r0_3_1_2, g23_19);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g22_19 = fma(ek22_5, r0_3_2_1, g22_19);
            }
            { const double eb = bi[5];
              o0_22 = fma(eb, g22_0, o0_22);
              o0_23 = fma(eb, g23_0, o0_23);
            }
            { const double eb = bi[6];
              o0_22 = fma(eb, g22_3, o0_22);
              o0_23 = fma(eb, g23_3, o0_23);
            }
            { const double eb = bi[7];
              o0_22 = fma(eb, g22_9, o0_22);
              o0_23 = fma(eb, g23_9, o0_23);
            }
            { const double eb = bi[8];
              o1_22 = fma(eb, g22_0, o1_22);
              o1_23 = fma(eb, g23_0, o1_23);
            }
            { const double eb = bi[9];
              o1_22 = fma(eb, g22_3, o1_22);
              o1_23 = fma(eb, g23_3, o1_23);
            }
            { const double eb = bi[10];
              o1_22 = fma(eb, g22_9, o1_22);
              o1_23 = fma(eb, g23_9, o1_23);
            }
            { const double eb = bi[11];
              o1_22 = fma(eb, g22_19, o1_22);
              o1_23 = fma(eb, g23_19, o1_23);
            }
            { const double eb = bi[12];
              o2_22 = fma(eb, g22_0, o2_22);
              o2_23 = fma(eb, g23_0, o2_23);
            }
            { const double eb = bi[13];
              o2_22 = fma(eb, g22_2, o2_22);
              o2_23 = fma(eb, g23_2, o2_23);
            }
            { const double eb = bi[14];
              o2_22 = fma(eb, g22_3, o2_22);
              o2_23 = fma(eb, g23_3, o2_23);
            }
            { const double eb = bi[15];
              o2_22 = fma(eb, g22_8, o2_22);
              o2_23 = fma(eb, g23_8, o2_23);
            }
            { const double eb = bi[16];
              o2_22 = fma(eb, g22_9, o2_22);
              o2_23 = fma(eb, g23_9, o2_23);
            }
            { const double eb = bi[17];
              o2_22 = fma(eb, g22_18, o2_22);
              o2_23 = fma(eb, g23_18, o2_23);
            }
            { const double eb = bi[18];
              o3_22 = fma(eb, g22_0, o3_22);
              o3_23 = fma(eb, g23_0, o3_23);
            }
            { const double eb = bi[19];
              o3_22 = fma(eb, g22_1, o3_22);
              o3_23 = fma(eb, g23_1, o3_23);
            }
            { const double eb = bi[20];
              o3_22 = fma(eb, g22_3, o3_22);
              o3_23 = fma(eb, g23_3, o3_23);
            }
            { const double eb = bi[21];
              o3_22 = fma(eb, g22_7, o3_22);
              o3_23 = fma(eb, g23_7, o3_23);
            }
            { const double eb = bi[22];
              o3_22 = fma(eb, g22_9, o3_22);
              o3_23 = fma(eb, g23_9, o3_23);
            }
            { const double eb = bi[23];
              o3_22 = fma(eb, g22_17, o3_22);
              o3_23 = fma(eb, g23_17, o3_23);
            }
            { const double eb = bi[24];
              o4_22 = fma(eb, g22_0, o4_22);
              o4_23 = fma(eb, g23_0, o4_23);
            }
            { const double eb = bi[25];
              o4_22 = fma(eb, g22_2, o4_22);
              o4_23 = fma(eb, g23_2, o4_23);
            }
            { const double eb = bi[26];
              o4_22 = fma(eb, g22_6, o4_22);
              o4_23 = fma(eb, g23_6, o4_23);
            }
            { const double eb = bi[27];
              o5_22 = fma(eb, g22_0, o5_22);
              o5_23 = fma(eb, g23_0, o5_23);
            }
            { const double eb = bi[28];
              o5_22 = fma(eb, g22_2, o5_22);
              o5_23 = fma(eb, g23_2, o5_23);
            }
            { const double eb = bi[29];
              o5_22 = fma(eb, g22_6, o5_22);
              o5_23 = fma(eb, g23_6, o5_23);
            }
            { const double eb = bi[30];
              o5_22 = fma(eb, g22_3, o5_22);
              o5_23 = fma(eb, g23_3, o5_23);
            }
            { const double eb = bi[31];
              o5_22 = fma(eb, g22_8, o5_22);
              o5_23 = fma(eb, g23_8, o5_23);
            }
            { const double eb = bi[32];
              o5_22 = fma(eb, g22_16, o5_22);
              o5_23 = fma(eb, g23_16, o5_23);
            }
            { const double eb = bi[33];
              o6_22 = fma(eb, g22_0, o6_22);
              o6_23 = fma(eb, g23_0, o6_23);
            }
            { const double eb = bi[34];
              o6_22 = fma(eb, g22_2, o6_22);
              o6_23 = fma(eb, g23_2, o6_23);
            }
            { const double eb = bi[35];
              o6_22 = fma(eb, g22_6, o6_22);
              o6_23 = fma(eb, g23_6, o6_23);
            }
            { const double eb = bi[36];
              o6_22 = fma(eb, g22_13, o6_22);
              o6_23 = fma(eb, g23_13, o6_23);
            }
            { const double eb = bi[37];
              o7_22 = fma(eb, g22_0, o7_22);
              o7_23 = fma(eb, g23_0, o7_23);
            }
            { const double eb = bi[38];
              o7_22 = fma(eb, g22_1, o7_22);
              o7_23 = fma(eb, g23_1, o7_23);
            }
            { const double eb = bi[39];
              o7_22 = fma(eb, g22_2, o7_22);
              o7_23 = fma(eb, g23_2, o7_23);
            }
            { const double eb = bi[40];
              o7_22 = fma(eb, g22_5, o7_22);
              o7_23 = fma(eb, g23_5, o7_23);
            }
            { const double eb = bi[41];
              o7_22 = fma(eb, g22_6, o7_22);
              o7_23 = fma(eb, g23_6, o7_23);
            }
            { const double eb = bi[42];
              o7_22 = fma(eb, g22_12, o7_22);
              o7_23 = fma(eb, g23_12, o7_23);
            }
            { const double eb = bi[43];
              o8_22 = fma(eb, g22_0, o8_22);
              o8_23 = fma(eb, g23_0, o8_23);
            }
            { const double eb = bi[44];
              o8_22 = fma(eb, g22_1, o8_22);
              o8_23 = fma(eb, g23_1, o8_23);
            }
            { const double eb = bi[45];
              o8_22 = fma(eb, g22_4, o8_22);
              o8_23 = fma(eb, g23_4, o8_23);
            }
            { const double eb = bi[46];
              o9_22 = fma(eb, g22_0, o9_22);
              o9_23 = fma(eb, g23_0, o9_23);
            }
            { const double eb = bi[47];
              o9_22 = fma(eb, g22_1, o9_22);
              o9_23 = fma(eb, g23_1, o9_23);
            }
            { const double eb = bi[48];
              o9_22 = fma(eb, g22_4, o9_22);
              o9_23 = fma(eb, g23_4, o9_23);
            }
            { const double eb = bi[49];
              o9_22 = fma(eb, g22_3, o9_22);
              o9_23 = fma(eb, g23_3, o9_23);
            }
            { const double eb = bi[50];
              o9_22 = fma(eb, g22_7, o9_22);
              o9_23 = fma(eb, g23_7, o9_23);
            }
            { const double eb = bi[51];
              o9_22 = fma(eb, g22_14, o9_22);
              o9_23 = fma(eb, g23_14, o9_23);
            }
            { const double eb = bi[52];
              o10_22 = fma(eb, g22_0, o10_22);
              o10_23 = fma(eb, g23_0, o10_23);
            }
            { const double eb = bi[53];
              o10_22 = fma(eb, g22_1, o10_22);
              o10_23 = fma(eb, g23_1, o10_23);
            }
            { const double eb = bi[54];
              o10_22 = fma(eb, g22_4, o10_22);
              o10_23 = fma(eb, g23_4, o10_23);
            }
            { const double eb = bi[55];
              o10_22 = fma(eb, g22_2, o10_22);
              o10_23 = fma(eb, g23_2, o10_23);
            }
            { const double eb = bi[56];
              o10_22 = fma(eb, g22_5, o10_22);
              o10_23 = fma(eb, g23_5, o10_23);
            }
            { const double eb = bi[57];
              o10_22 = fma(eb, g22_11, o10_22);
              o10_23 = fma(eb, g23_11, o10_23);
            }
            { const double eb = bi[58];
              o11_22 = fma(eb, g22_0, o11_22);
              o11_23 = fma(eb, g23_0, o11_23);
            }
            { const double eb = bi[59];
              o11_22 = fma(eb, g22_1, o11_22);
              o11_23 = fma(eb, g23_1, o11_23);
            }
            { const double eb = bi[60];
              o11_22 = fma(eb, g22_4, o11_22);
              o11_23 = fma(eb, g23_4, o11_23);
            }
            { const double eb = bi[61];
              o11_22 = fma(eb, g22_10, o11_22);
              o11_23 = fma(eb, g23_10, o11_23);
            }
            { const double eb = bi[62];
              o12_22 = fma(eb, g22_0, o12_22);
              o12_23 = fma(eb, g23_0, o12_23);
            }
            { const double eb = bi[63];
              o12_22 = fma(eb, g22_2, o12_22);
              o12_23 = fma(eb, g23_2, o12_23);
            }
            { const double eb = bi[64];
              o12_22 = fma(eb, g22_3, o12_22);
              o12_23 = fma(eb, g23_3, o12_23);
            }
            { const double eb = bi[65];
              o12_22 = fma(eb, g22_8, o12_22);
              o12_23 = fma(eb, g23_8, o12_23);
            }
            { const double eb = bi[66];
              o13_22 = fma(eb, g22_0, o13_22);
              o13_23 = fma(eb, g23_0, o13_23);
            }
            { const double eb = bi[67];
              o13_22 = fma(eb, g22_2, o13_22);
              o13_23 = fma(eb, g23_2, o13_23);
            }
            { const double eb = bi[68];
              o13_22 = fma(eb, g22_3, o13_22);
              o13_23 = fma(eb, g23_3, o13_23);
            }
            { const double eb = bi[69];
              o13_22 = fma(eb, g22_8, o13_22);
              o13_23 = fma(eb, g23_8, o13_23);
            }
            { const double eb = bi[70];
              o13_22 = fma(eb, g22_9, o13_22);
              o13_23 = fma(eb, g23_9, o13_23);
            }
            { const double eb = bi[71];
              o13_22 = fma(eb, g22_18, o13_22);
              o13_23 = fma(eb, g23_18, o13_23);
            }
            { const double eb = bi[72];
              o14_22 = fma(eb, g22_0, o14_22);
              o14_23 = fma(eb, g23_0, o14_23);
            }
            { const double eb = bi[73];
              o14_22 = fma(eb, g22_2, o14_22);
              o14_23 = fma(eb, g23_2, o14_23);
            }
            { const double eb = bi[74];
              o14_22 = fma(eb, g22_6, o14_22);
              o14_23 = fma(eb, g23_6, o14_23);
            }
            { const double eb = bi[75];
              o14_22 = fma(eb, g22_3, o14_22);
              o14_23 = fma(eb, g23_3, o14_23);
            }
            { const double eb = bi[76];
              o14_22 = fma(eb, g22_8, o14_22);
              o14_23 = fma(eb, g23_8, o14_23);
            }
            { const double eb = bi[77];
              o14_22 = fma(eb, g22_16, o14_22);
              o14_23 = fma(eb, g23_16, o14_23);
            }
            { const double eb = bi[78];
              o15_22 = fma(eb, g22_0, o15_22);
              o15_23 = fma(eb, g23_0, o15_23);
            }
            { const double eb = bi[79];
              o15_22 = fma(eb, g22_1, o15_22);
              o15_23 = fma(eb, g23_1, o15_23);
            }
            { const double eb = bi[80];
              o15_22 = fma(eb, g22_2, o15_22);
              o15_23 = fma(eb, g23_2, o15_23);
            }
            { const double eb = bi[81];
              o15_22 = fma(eb, g22_5, o15_22);
              o15_23 = fma(eb, g23_5, o15_23);
            }
            { const double eb = bi[82];
              o15_22 = fma(eb, g22_3, o15_22);
              o15_23 = fma(eb, g23_3, o15_23);
            }
            { const double eb = bi[83];
              o15_22 = fma(eb, g22_7, o15_22);
              o15_23 = fma(eb, g23_7, o15_23);
            }
            { const double eb = bi[84];
              o15_22 = fma(eb, g22_8, o15_22);
              o15_23 = fma(eb, g23_8, o15_23);
            }
            { const double eb = bi[85];
              o15_22 = fma(eb, g22_15, o15_22);
              o15_23 = fma(eb, g23_15, o15_23);
            }
            { const double eb = bi[86];
              o16_22 = fma(eb, g22_0, o16_22);
              o16_23 = fma(eb, g23_0, o16_23);
            }
            { const double eb = bi[87];
              o16_22 = fma(eb, g22_1, o16_22);
              o16_23 = fma(eb, g23_1, o16_23);
            }
            { const double eb = bi[88];
              o16_22 = fma(eb, g22_3, o16_22);
              o16_23 = fma(eb, g23_3, o16_23);
            }
            { const double eb = bi[89];
              o16_22 = fma(eb, g22_7, o16_22);
              o16_23 = fma(eb, g23_7, o16_23);
            }
            { const double eb = bi[90];
              o17_22 = fma(eb, g22_0, o17_22);
              o17_23 = fma(eb, g23_0, o17_23);
            }
            { const double eb = bi[91];
              o17_22 = fma(eb, g22_1, o17_22);
              o17_23 = fma(eb, g23_1, o17_23);
            }
            { const double eb = bi[92];
              o17_22 = fma(eb, g22_3, o17_22);
              o17_23 = fma(eb, g23_3, o17_23);
            }
            { const double eb = bi[93];
              o17_22 = fma(eb, g22_7, o17_22);
              o17_23 = fma(eb, g23_7, o17_23);
            }
            { const double eb = bi[94];
              o17_22 = fma(eb, g22_9, o17_22);
              o17_23 = fma(eb, g23_9, o17_23);
            }
            { const double eb = bi[95];
              o17_22 = fma(eb, g22_17, o17_22);
              o17_23 = fma(eb, g23_17, o17_23);
            }
            { const double eb = bi[96];
              o18_22 = fma(eb, g22_0, o18_22);
              o18_23 = fma(eb, g23_0, o18_23);
            }
            { const double eb = bi[97];
              o18_22 = fma(eb, g22_1, o18_22);
              o18_23 = fma(eb, g23_1, o18_23);
            }
            { const double eb = bi[98];
              o18_22 = fma(eb, g22_2, o18_22);
              o18_23 = fma(eb, g23_2, o18_23);
            }
            { const double eb = bi[99];
              o18_22 = fma(eb, g22_5, o18_22);
              o18_23 = fma(eb, g23_5, o18_23);
            }
            { const double eb = bi[100];
              o18_22 = fma(eb, g22_3, o18_22);
              o18_23 = fma(eb, g23_3, o18_23);
            }
            { const double eb = bi[101];
              o18_22 = fma(eb, g22_7, o18_22);
              o18_23 = fma(eb, g23_7, o18_23);
            }
            { const double eb = bi[102];
              o18_22 = fma(eb, g22_8, o18_22);
              o18_23 = fma(eb, g23_8, o18_23);
            }
            { const double eb = bi[103];
              o18_22 = fma(eb, g22_15, o18_22);
              o18_23 = fma(eb, g23_15, o18_23);
            }
            { const double eb = bi[104];
              o19_22 = fma(eb, g22_0, o19_22);
              o19_23 = fma(eb, g23_0, o19_23);
            }
            { const double eb = bi[105];
              o19_22 = fma(eb, g22_1, o19_22);
              o19_23 = fma(eb, g23_1, o19_23);
            }
            { const double eb = bi[106];
              o19_22 = fma(eb, g22_4, o19_22);
              o19_23 = fma(eb, g23_4, o19_23);
            }
            { const double eb = bi[107];
              o19_22 = fma(eb, g22_3, o19_22);
              o19_23 = fma(eb, g23_3, o19_23);
            }
            { const double eb = bi[108];
              o19_22 = fma(eb, g22_7, o19_22);
              o19_23 = fma(eb, g23_7, o19_23);
            }
            { const double eb = bi[109];
              o19_22 = fma(eb, g22_14, o19_22);
              o19_23 = fma(eb, g23_14, o19_23);
            }
            { const double eb = bi[110];
              o20_22 = fma(eb, g22_0, o20_22);
              o20_23 = fma(eb, g23_0, o20_23);
            }
            { const double eb = bi[111];
              o20_22 = fma(eb, g22_1, o20_22);
              o20_23 = fma(eb, g23_1, o20_23);
            }
            { const double eb = bi[112];
              o20_22 = fma(eb, g22_2, o20_22);
              o20_23 = fma(eb, g23_2, o20_23);
            }
            { const double eb = bi[113];
              o20_22 = fma(eb, g22_5, o20_22);
              o20_23 = fma(eb, g23_5, o20_23);
            }
            { const double eb = bi[114];
              o21_22 = fma(eb, g22_0, o21_22);
              o21_23 = fma(eb, g23_0, o21_23);
            }
            { const double eb = bi[115];
              o21_22 = fma(eb, g22_1, o21_22);
              o21_23 = fma(eb, g23_1, o21_23);
            }
            { const double eb = bi[116];
              o21_22 = fma(eb, g22_2, o21_22);
              o21_23 = fma(eb, g23_2, o21_23);
            }
            { const double eb = bi[117];
              o21_22 = fma(eb, g22_5, o21_22);
              o21_23 = fma(eb, g23_5, o21_23);
            }
            { const double eb = bi[118];
              o21_22 = fma(eb, g22_3, o21_22);
              o21_23 = fma(eb, g23_3, o21_23);
            }
            { const double eb = bi[119];
              o21_22 = fma(eb, g22_7, o21_22);
              o21_23 = fma(eb, g23_7, o21_23);
            }
            { const double eb = bi[120];
              o21_22 = fma(eb, g22_8, o21_22);
              o21_23 = fma(eb, g23_8, o21_23);
            }
            { const double eb = bi[121];
              o21_22 = fma(eb, g22_15, o21_22);
              o21_23 = fma(eb, g23_15, o21_23);
            }
            { const double eb = bi[122];
              o22_22 = fma(eb, g22_0, o22_22);
              o22_23 = fma(eb, g23_0, o22_23);
            }
            { const double eb = bi[123];
              o22_22 = fma(eb, g22_1, o22_22);
              o22_23 = fma(eb, g23_1, o22_23);
            }
            { const double eb = bi[124];
              o22_22 = fma(eb, g22_2, o22_22);
              o22_23 = fma(eb, g23_2, o22_23);
            }
            { const double eb = bi[125];
              o22_22 = fma(eb, g22_5, o22_22);
              o22_23 = fma(eb, g23_5, o22_23);
            }
            { const double eb = bi[126];
              o22_22 = fma(eb, g22_6, o22_22);
              o22_23 = fma(eb, g23_6, o22_23);
            }
            { const double eb = bi[127];
              o22_22 = fma(eb, g22_12, o22_22);
              o22_23 = fma(eb, g23_12, o22_23);
            }
            { const double eb = bi[128];
              o23_22 = fma(eb, g22_0, o23_22);
              o23_23 = fma(eb, g23_0, o23_23);
            }
            { const double eb = bi[129];
              o23_22 = fma(eb, g22_1, o23_22);
              o23_23 = fma(eb, g23_1, o23_23);
            }
            { const double eb = bi[130];
              o23_22 = fma(eb, g22_4, o23_22);
              o23_23 = fma(eb, g23_4, o23_23);
            }
            { const double eb = bi[131];
              o23_22 = fma(eb, g22_2, o23_22);
              o23_23 = fma(eb, g23_2, o23_23);
            }
            { const double eb = bi[132];
              o23_22 = fma(eb, g22_5, o23_22);
              o23_23 = fma(eb, g23_5, o23_23);
            }
            { const double eb = bi[133];
              o23_22 = fma(eb, g22_11, o23_22);
              o23_23 = fma(eb, g23_11, o23_23);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk22 = PT[(fI + 5) * N + fJ + 2];
            const double ptk23 = PT[(fI + 5) * N + fJ + 3];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 1) * N + fQ + 0];
            const double ptb5 = PT[(fP + 1) * N + fQ + 1];
            const double ptb6 = PT[(fP + 1) * N + fQ + 2];
            const double ptb7 = PT[(fP + 1) * N + fQ + 3];
            const double ptb8 = PT[(fP + 2) * N + fQ + 0];
            const double ptb9 = PT[(fP + 2) * N + fQ + 1];
            const double ptb10 = PT[(fP + 2) * N + fQ + 2];
            const double ptb11 = PT[(fP + 2) * N + fQ + 3];
            const double ptb12 = PT[(fP + 3) * N + fQ + 0];
            const double ptb13 = PT[(fP + 3) * N + fQ + 1];
            const double ptb14 = PT[(fP + 3) * N + fQ + 2];
            const double ptb15 = PT[(fP + 3) * N + fQ + 3];
            const double ptb16 = PT[(fP + 4) * N + fQ + 0];
            const double ptb17 = PT[(fP + 4) * N + fQ + 1];
            const double ptb18 = PT[(fP + 4) * N + fQ + 2];
            const double ptb19 = PT[(fP + 4) * N + fQ + 3];
            const double ptb20 = PT[(fP + 5) * N + fQ + 0];
            const double ptb21 = PT[(fP + 5) * N + fQ + 1];
            const double ptb22 = PT[(fP + 5) * N + fQ + 2];
            const double ptb23 = PT[(fP + 5) * N + fQ + 3];
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
            const double Aad5_3 = PA[(fP + 5) * N + fJ + 3];
            const double Abc0_5 = PA[(fQ + 0) * N + fI + 5];
            const double Abc1_5 = PA[(fQ + 1) * N + fI + 5];
            const double Abc2_5 = PA[(fQ + 2) * N + fI + 5];
            const double Abc3_5 = PA[(fQ + 3) * N + fI + 5];
            const double Aac0_5 = PA[(fP + 0) * N + fI + 5];
            const double Aac1_5 = PA[(fP + 1) * N + fI + 5];
            const double Aac2_5 = PA[(fP + 2) * N + fI + 5];
            const double Aac3_5 = PA[(fP + 3) * N + fI + 5];
            const double Aac4_5 = PA[(fP + 4) * N + fI + 5];
            const double Aac5_5 = PA[(fP + 5) * N + fI + 5];
            jab0 += o0_22 * ptk22 + o0_23 * ptk23;
            jab1 += o1_22 * ptk22 + o1_23 * ptk23;
            jab2 += o2_22 * ptk22 + o2_23 * ptk23;
            jab3 += o3_22 * ptk22 + o3_23 * ptk23;
            jab4 += o4_22 * ptk22 + o4_23 * ptk23;
            jab5 += o5_22 * ptk22 + o5_23 * ptk23;
            jab6 += o6_22 * ptk22 + o6_23 * ptk23;
            jab7 += o7_22 * ptk22 + o7_23 * ptk23;
            jab8 += o8_22 * ptk22 + o8_23 * ptk23;
            jab9 += o9_22 * ptk22 + o9_23 * ptk23;
            jab10 += o10_22 * ptk22 + o10_23 * ptk23;
            jab11 += o11_22 * ptk22 + o11_23 * ptk23;
            jab12 += o12_22 * ptk22 + o12_23 * ptk23;
            jab13 += o13_22 * ptk22 + o13_23 * ptk23;
            jab14 += o14_22 * ptk22 + o14_23 * ptk23;
            jab15 += o15_22 * ptk22 + o15_23 * ptk23;
            jab16 += o16_22 * ptk22 + o16_23 * ptk23;
            jab17 += o17_22 * ptk22 + o17_23 * ptk23;
            jab18 += o18_22 * ptk22 + o18_23 * ptk23;
            jab19 += o19_22 * ptk22 + o19_23 * ptk23;
            jab20 += o20_22 * ptk22 + o20_23 * ptk23;
            jab21 += o21_22 * ptk22 + o21_23 * ptk23;
            jab22 += o22_22 * ptk22 + o22_23 * ptk23;
            jab23 += o23_22 * ptk22 + o23_23 * ptk23;
            atomicAdd(Jacc + (fI + 5) * N + fJ + 2, 2.0 * deg * (o0_22 * ptb0 + o1_22 * ptb1 + o2_22 * ptb2 + o3_22 * ptb3 + o4_22 * ptb4 + o5_22 * ptb5 + o6_22 * ptb6 + o7_22 * ptb7 + o8_22 * ptb8 + o9_22 * ptb9 + o10_22 * ptb10 + o11_22 * ptb11 + o12_22 * ptb12 + o13_22 * ptb13 + o14_22 * ptb14 + o15_22 * ptb15 + o16_22 * ptb16 + o17_22 * ptb17 + o18_22 * ptb18 + o19_22 * ptb19 + o20_22 * ptb20 + o21_22 * ptb21 + o22_22 * ptb22 + o23_22 * ptb23));
            atomicAdd(Jacc + (fI + 5) * N + fJ + 3, 2.0 * deg * (o0_23 * ptb0 + o1_23 * ptb1 + o2_23 * ptb2 + o3_23 * ptb3 + o4_23 * ptb4 + o5_23 * ptb5 + o6_23 * ptb6 + o7_23 * ptb7 + o8_23 * ptb8 + o9_23 * ptb9 + o10_23 * ptb10 + o11_23 * ptb11 + o12_23 * ptb12 + o13_23 * ptb13 + o14_23 * ptb14 + o15_23 * ptb15 + o16_23 * ptb16 + o17_23 * ptb17 + o18_23 * ptb18 + o19_23 * ptb19 + o20_23 * ptb20 + o21_23 * ptb21 + o22_23 * ptb22 + o23_23 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 5, deg * (o0_22 * Abd0_2 + o0_23 * Abd0_3 + o1_22 * Abd1_2 + o1_23 * Abd1_3 + o2_22 * Abd2_2 + o2_23 * Abd2_3 + o3_22 * Abd3_2 + o3_23 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 5, deg * (o0_22 * Aad0_2 + o0_23 * Aad0_3 + o4_22 * Aad1_2 + o4_23 * Aad1_3 + o8_22 * Aad2_2 + o8_23 * Aad2_3 + o12_22 * Aad3_2 + o12_23 * Aad3_3 + o16_22 * Aad4_2 + o16_23 * Aad4_3 + o20_22 * Aad5_2 + o20_23 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_22 * Abc0_5 + o1_22 * Abc1_5 + o2_22 * Abc2_5 + o3_22 * Abc3_5));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_22 * Aac0_5 + o4_22 * Aac1_5 + o8_22 * Aac2_5 + o12_22 * Aac3_5 + o16_22 * Aac4_5 + o20_22 * Aac5_5));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_23 * Abc0_5 + o1_23 * Abc1_5 + o2_23 * Abc2_5 + o3_23 * Abc3_5));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_23 * Aac0_5 + o4_23 * Aac1_5 + o8_23 * Aac2_5 + o12_23 * Aac3_5 + o16_23 * Aac4_5 + o20_23 * Aac5_5));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 5, deg * (o1_22 * Aad0_2 + o1_23 * Aad0_3 + o5_22 * Aad1_2 + o5_23 * Aad1_3 + o9_22 * Aad2_2 + o9_23 * Aad2_3 + o13_22 * Aad3_2 + o13_23 * Aad3_3 + o17_22 * Aad4_2 + o17_23 * Aad4_3 + o21_22 * Aad5_2 + o21_23 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_22 * Aac0_5 + o5_22 * Aac1_5 + o9_22 * Aac2_5 + o13_22 * Aac3_5 + o17_22 * Aac4_5 + o21_22 * Aac5_5));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_23 * Aac0_5 + o5_23 * Aac1_5 + o9_23 * Aac2_5 + o13_23 * Aac3_5 + o17_23 * Aac4_5 + o21_23 * Aac5_5));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 5, deg * (o2_22 * Aad0_2 + o2_23 * Aad0_3 + o6_22 * Aad1_2 + o6_23 * Aad1_3 + o10_22 * Aad2_2 + o10_23 * Aad2_3 + o14_22 * Aad3_2 + o14_23 * Aad3_3 + o18_22 * Aad4_2 + o18_23 * Aad4_3 + o22_22 * Aad5_2 + o22_23 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_22 * Aac0_5 + o6_22 * Aac1_5 + o10_22 * Aac2_5 + o14_22 * Aac3_5 + o18_22 * Aac4_5 + o22_22 * Aac5_5));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_23 * Aac0_5 + o6_23 * Aac1_5 + o10_23 * Aac2_5 + o14_23 * Aac3_5 + o18_23 * Aac4_5 + o22_23 * Aac5_5));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 5, deg * (o3_22 * Aad0_2 + o3_23 * Aad0_3 + o7_22 * Aad1_2 + o7_23 * Aad1_3 + o11_22 * Aad2_2 + o11_23 * Aad2_3 + o15_22 * Aad3_2 + o15_23 * Aad3_3 + o19_22 * Aad4_2 + o19_23 * Aad4_3 + o23_22 * Aad5_2 + o23_23 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_22 * Aac0_5 + o7_22 * Aac1_5 + o11_22 * Aac2_5 + o15_22 * Aac3_5 + o19_22 * Aac4_5 + o23_22 * Aac5_5));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_23 * Aac0_5 + o7_23 * Aac1_5 + o11_23 * Aac2_5 + o15_23 * Aac3_5 + o19_23 * Aac4_5 + o23_23 * Aac5_5));
            atomicAdd(KAacc + (fP + 1) * N + fI + 5, deg * (o4_22 * Abd0_2 + o4_23 * Abd0_3 + o5_22 * Abd1_2 + o5_23 * Abd1_3 + o6_22 * Abd2_2 + o6_23 * Abd2_3 + o7_22 * Abd3_2 + o7_23 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_22 * Abc0_5 + o5_22 * Abc1_5 + o6_22 * Abc2_5 + o7_22 * Abc3_5));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_23 * Abc0_5 + o5_23 * Abc1_5 + o6_23 * Abc2_5 + o7_23 * Abc3_5));
            atomicAdd(KAacc + (fP + 2) * N + fI + 5, deg * (o8_22 * Abd0_2 + o8_23 * Abd0_3 + o9_22 * Abd1_2 + o9_23 * Abd1_3 + o10_22 * Abd2_2 + o10_23 * Abd2_3 + o11_22 * Abd3_2 + o11_23 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_22 * Abc0_5 + o9_22 * Abc1_5 + o10_22 * Abc2_5 + o11_22 * Abc3_5));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_23 * Abc0_5 + o9_23 * Abc1_5 + o10_23 * Abc2_5 + o11_23 * Abc3_5));
            atomicAdd(KAacc + (fP + 3) * N + fI + 5, deg * (o12_22 * Abd0_2 + o12_23 * Abd0_3 + o13_22 * Abd1_2 + o13_23 * Abd1_3 + o14_22 * Abd2_2 + o14_23 * Abd2_3 + o15_22 * Abd3_2 + o15_23 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_22 * Abc0_5 + o13_22 * Abc1_5 + o14_22 * Abc2_5 + o15_22 * Abc3_5));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_23 * Abc0_5 + o13_23 * Abc1_5 + o14_23 * Abc2_5 + o15_23 * Abc3_5));
            atomicAdd(KAacc + (fP + 4) * N + fI + 5, deg * (o16_22 * Abd0_2 + o16_23 * Abd0_3 + o17_22 * Abd1_2 + o17_23 * Abd1_3 + o18_22 * Abd2_2 + o18_23 * Abd2_3 + o19_22 * Abd3_2 + o19_23 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_22 * Abc0_5 + o17_22 * Abc1_5 + o18_22 * Abc2_5 + o19_22 * Abc3_5));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_23 * Abc0_5 + o17_23 * Abc1_5 + o18_23 * Abc2_5 + o19_23 * Abc3_5));
            atomicAdd(KAacc + (fP + 5) * N + fI + 5, deg * (o20_22 * Abd0_2 + o20_23 * Abd0_3 + o21_22 * Abd1_2 + o21_23 * Abd1_3 + o22_22 * Abd2_2 + o22_23 * Abd2_3 + o23_22 * Abd3_2 + o23_23 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_22 * Abc0_5 + o21_22 * Abc1_5 + o22_22 * Abc2_5 + o23_22 * Abc3_5));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_23 * Abc0_5 + o21_23 * Abc1_5 + o22_23 * Abc2_5 + o23_23 * Abc3_5));
          }
        } break;
        }
      }
      {
        const double s2 = 2.0 * deg;
        double v[32] = {s2 * jab0, s2 * jab1, s2 * jab2, s2 * jab3, s2 * jab4, s2 * jab5, s2 * jab6, s2 * jab7, s2 * jab8, s2 * jab9, s2 * jab10, s2 * jab11, s2 * jab12, s2 * jab13, s2 * jab14, s2 * jab15, s2 * jab16, s2 * jab17, s2 * jab18, s2 * jab19, s2 * jab20, s2 * jab21, s2 * jab22, s2 * jab23, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const double s = sqb::warp_sum_scatter<32>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 24 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 4) * N + bp.fQ + ab % 4, s);
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
