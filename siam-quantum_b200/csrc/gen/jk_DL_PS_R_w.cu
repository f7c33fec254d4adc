// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DL_PS_R_w(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
              const double* __restrict__ kj = kprim + (long long)j * 11 * kS;
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
              const double ek1_0 = kj[7 * kS];
              const double ek1_1 = -kj[8 * kS];
              g0_0 = fma(ek0_0, b0, g0_0);
              g1_0 = fma(ek1_0, b0, g1_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              g1_1 = fma(ek1_0, r0_0_0_1, g1_1);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              g1_2 = fma(ek1_0, r0_0_1_0, g1_2);
              g1_0 = fma(ek1_1, r0_0_1_0, g1_0);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fma(ek0_1, r0_1_0_0, g0_0);
              g1_3 = fma(ek1_0, r0_1_0_0, g1_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g0_4 = fma(ek0_0, r0_0_0_2, g0_4);
              g1_4 = fma(ek1_0, r0_0_0_2, g1_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fma(ek0_0, r0_0_1_1, g0_5);
              g1_5 = fma(ek1_0, r0_0_1_1, g1_5);
              g1_1 = fma(ek1_1, r0_0_1_1, g1_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g0_6 = fma(ek0_0, r0_0_2_0, g0_6);
              g1_6 = fma(ek1_0, r0_0_2_0, g1_6);
              g1_2 = fma(ek1_1, r0_0_2_0, g1_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fma(ek0_0, r0_1_0_1, g0_7);
              g0_1 = fma(ek0_1, r0_1_0_1, g0_1);
              g1_7 = fma(ek1_0, r0_1_0_1, g1_7);
              const double r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fma(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fma(ek0_1, r0_1_1_0, g0_2);
              g1_8 = fma(ek1_0, r0_1_1_0, g1_8);
              g1_3 = fma(ek1_1, r0_1_1_0, g1_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g0_9 = fma(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fma(ek0_1, r0_2_0_0, g0_3);
              g1_9 = fma(ek1_0, r0_2_0_0, g1_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g0_10 = fma(ek0_0, r0_0_0_3, g0_10);
              g1_10 = fma(ek1_0, r0_0_0_3, g1_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g0_11 = fma(ek0_0, r0_0_1_2, g0_11);
              g1_11 = fma(ek1_0, r0_0_1_2, g1_11);
              g1_4 = fma(ek1_1, r0_0_1_2, g1_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g0_12 = fma(ek0_0, r0_0_2_1, g0_12);
              g1_12 = fma(ek1_0, r0_0_2_1, g1_12);
              g1_5 = fma(ek1_1, r0_0_2_1, g1_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g0_13 = fma(ek0_0, r0_0_3_0, g0_13);
              g1_13 = fma(ek1_0, r0_0_3_0, g1_13);
              g1_6 = fma(ek1_1, r0_0_3_0, g1_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g0_14 = fma(ek0_0, r0_1_0_2, g0_14);
              g0_4 = fma(ek0_1, r0_1_0_2, g0_4);
              g1_14 = fma(ek1_0, r0_1_0_2, g1_14);
              const double r0_1_1_1 = X * r1_0_1_1;
              g0_15 = fma(ek0_0, r0_1_1_1, g0_15);
              g0_5 = fma(ek0_1, r0_1_1_1, g0_5);
              g1_15 = fma(ek1_0, r0_1_1_1, g1_15);
              g1_7 = fma(ek1_1, r0_1_1_1, g1_7);
              const double r0_1_2_0 = X * r1_0_2_0;
              g0_16 = fma(ek0_0, r0_1_2_0, g0_16);
              g0_6 = fma(ek0_1, r0_1_2_0, g0_6);
              g1_16 = fma(ek1_0, r0_1_2_0, g1_16);
              g1_8 = fma(ek1_1, r0_1_2_0, g1_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g0_17 = fma(ek0_0, r0_2_0_1, g0_17);
              g0_7 = fma(ek0_1, r0_2_0_1, g0_7);
              g1_17 = fma(ek1_0, r0_2_0_1, g1_17);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fma(ek0_0, r0_2_1_0, g0_18);
              g0_8 = fma(ek0_1, r0_2_1_0, g0_8);
              g1_18 = fma(ek1_0, r0_2_1_0, g1_18);
              g1_9 = fma(ek1_1, r0_2_1_0, g1_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_19 = fma(ek0_0, r0_3_0_0, g0_19);
              g0_9 = fma(ek0_1, r0_3_0_0, g0_9);
              g1_19 = fma(ek1_0, r0_3_0_0, g1_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g1_10 = fma(ek1_1, r0_0_1_3, g1_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g1_11 = fma(ek1_1, r0_0_2_2, g1_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g1_12 = fma(ek1_1, r0_0_3_1, g1_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g1_13 = fma(ek1_1, r0_0_4_0, g1_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g0_10 = fma(ek0_1, r0_1_0_3, g0_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g0_11 = fma(ek0_1, r0_1_1_2, g0_11);
              g1_14 = fma(ek1_1, r0_1_1_2, g1_14);
              const double r0_1_2_1 = X * r1_0_2_1;
              g0_12 = fma(ek0_1, r0_1_2_1, g0_12);
              g1_15 = fma(ek1_1, r0_1_2_1, g1_15);
              const double r0_1_3_0 = X * r1_0_3_0;
              g0_13 = fma(ek0_1, r0_1_3_0, g0_13);
              g1_16 = fma(ek1_1, r0_1_3_0, g1_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g0_14 = fma(ek0_1, r0_2_0_2, g0_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g0_15 = fma(ek0_1, r0_2_1_1, g0_15);
              g1_17 = fma(ek1_1, r0_2_1_1, g1_17);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g0_16 = fma(ek0_1, r0_2_2_0, g0_16);
              g1_18 = fma(ek1_1, r0_2_2_0, g1_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g0_17 = fma(ek0_1, r0_3_0_1, g0_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g0_18 = fma(ek0_1, r0_3_1_0, g0_18);
              g1_19 = fma(ek1_1, r0_3_1_0, g1_19);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g0_19 = fma(ek0_1, r0_4_0_0, g0_19);
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
            const double ptk1 = PT[(fI + 1) * N + fJ + 0];
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
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
            const double Abc3_1 = PA[(fQ + 3) * N + fI + 1];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
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
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17 + o18_1 * ptb18 + o19_1 * ptb19 + o20_1 * ptb20 + o21_1 * ptb21 + o22_1 * ptb22 + o23_1 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0 + o3_0 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o4_0 * Aad1_0 + o8_0 * Aad2_0 + o12_0 * Aad3_0 + o16_0 * Aad4_0 + o20_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o0_1 * Abc0_1 + o1_0 * Abc1_0 + o1_1 * Abc1_1 + o2_0 * Abc2_0 + o2_1 * Abc2_1 + o3_0 * Abc3_0 + o3_1 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o0_1 * Aac0_1 + o4_0 * Aac1_0 + o4_1 * Aac1_1 + o8_0 * Aac2_0 + o8_1 * Aac2_1 + o12_0 * Aac3_0 + o12_1 * Aac3_1 + o16_0 * Aac4_0 + o16_1 * Aac4_1 + o20_0 * Aac5_0 + o20_1 * Aac5_1));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Abd0_0 + o1_1 * Abd1_0 + o2_1 * Abd2_0 + o3_1 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Aad0_0 + o4_1 * Aad1_0 + o8_1 * Aad2_0 + o12_1 * Aad3_0 + o16_1 * Aad4_0 + o20_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o5_0 * Aad1_0 + o9_0 * Aad2_0 + o13_0 * Aad3_0 + o17_0 * Aad4_0 + o21_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o1_1 * Aac0_1 + o5_0 * Aac1_0 + o5_1 * Aac1_1 + o9_0 * Aac2_0 + o9_1 * Aac2_1 + o13_0 * Aac3_0 + o13_1 * Aac3_1 + o17_0 * Aac4_0 + o17_1 * Aac4_1 + o21_0 * Aac5_0 + o21_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_1 * Aad0_0 + o5_1 * Aad1_0 + o9_1 * Aad2_0 + o13_1 * Aad3_0 + o17_1 * Aad4_0 + o21_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o6_0 * Aad1_0 + o10_0 * Aad2_0 + o14_0 * Aad3_0 + o18_0 * Aad4_0 + o22_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o2_1 * Aac0_1 + o6_0 * Aac1_0 + o6_1 * Aac1_1 + o10_0 * Aac2_0 + o10_1 * Aac2_1 + o14_0 * Aac3_0 + o14_1 * Aac3_1 + o18_0 * Aac4_0 + o18_1 * Aac4_1 + o22_0 * Aac5_0 + o22_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_1 * Aad0_0 + o6_1 * Aad1_0 + o10_1 * Aad2_0 + o14_1 * Aad3_0 + o18_1 * Aad4_0 + o22_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Aad0_0 + o7_0 * Aad1_0 + o11_0 * Aad2_0 + o15_0 * Aad3_0 + o19_0 * Aad4_0 + o23_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Aac0_0 + o3_1 * Aac0_1 + o7_0 * Aac1_0 + o7_1 * Aac1_1 + o11_0 * Aac2_0 + o11_1 * Aac2_1 + o15_0 * Aac3_0 + o15_1 * Aac3_1 + o19_0 * Aac4_0 + o19_1 * Aac4_1 + o23_0 * Aac5_0 + o23_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_1 * Aad0_0 + o7_1 * Aad1_0 + o11_1 * Aad2_0 + o15_1 * Aad3_0 + o19_1 * Aad4_0 + o23_1 * Aad5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Abd0_0 + o5_0 * Abd1_0 + o6_0 * Abd2_0 + o7_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o4_1 * Abc0_1 + o5_0 * Abc1_0 + o5_1 * Abc1_1 + o6_0 * Abc2_0 + o6_1 * Abc2_1 + o7_0 * Abc3_0 + o7_1 * Abc3_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_1 * Abd0_0 + o5_1 * Abd1_0 + o6_1 * Abd2_0 + o7_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Abd0_0 + o9_0 * Abd1_0 + o10_0 * Abd2_0 + o11_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Abc0_0 + o8_1 * Abc0_1 + o9_0 * Abc1_0 + o9_1 * Abc1_1 + o10_0 * Abc2_0 + o10_1 * Abc2_1 + o11_0 * Abc3_0 + o11_1 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_1 * Abd0_0 + o9_1 * Abd1_0 + o10_1 * Abd2_0 + o11_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0 + o15_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o12_1 * Abc0_1 + o13_0 * Abc1_0 + o13_1 * Abc1_1 + o14_0 * Abc2_0 + o14_1 * Abc2_1 + o15_0 * Abc3_0 + o15_1 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_1 * Abd0_0 + o13_1 * Abd1_0 + o14_1 * Abd2_0 + o15_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_0 * Abd0_0 + o17_0 * Abd1_0 + o18_0 * Abd2_0 + o19_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_0 * Abc0_0 + o16_1 * Abc0_1 + o17_0 * Abc1_0 + o17_1 * Abc1_1 + o18_0 * Abc2_0 + o18_1 * Abc2_1 + o19_0 * Abc3_0 + o19_1 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_1 * Abd0_0 + o17_1 * Abd1_0 + o18_1 * Abd2_0 + o19_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_0 * Abd0_0 + o21_0 * Abd1_0 + o22_0 * Abd2_0 + o23_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_0 * Abc0_0 + o20_1 * Abc0_1 + o21_0 * Abc1_0 + o21_1 * Abc1_1 + o22_0 * Abc2_0 + o22_1 * Abc2_1 + o23_0 * Abc3_0 + o23_1 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_1 * Abd0_0 + o21_1 * Abd1_0 + o22_1 * Abd2_0 + o23_1 * Abd3_0));
          }
        } break;
        case 1: {  // ket functions [2]
          double o0_2 = 0;
          double o1_2 = 0;
          double o2_2 = 0;
          double o3_2 = 0;
          double o4_2 = 0;
          double o5_2 = 0;
          double o6_2 = 0;
          double o7_2 = 0;
          double o8_2 = 0;
          double o9_2 = 0;
          double o10_2 = 0;
          double o11_2 = 0;
          double o12_2 = 0;
          double o13_2 = 0;
          double o14_2 = 0;
          double o15_2 = 0;
          double o16_2 = 0;
          double o17_2 = 0;
          double o18_2 = 0;
          double o19_2 = 0;
          double o20_2 = 0;
          double o21_2 = 0;
          double o22_2 = 0;
          double o23_2 = 0;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 11 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
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
              const double ek2_0 = kj[9 * kS];
              const double ek2_1 = -kj[10 * kS];
              g2_0 = fma(ek2_0, b0, g2_0);
              const double r0_0_0_1 = Z * b1;
              g2_1 = fma(ek2_0, r0_0_0_1, g2_1);
              g2_0 = fma(ek2_1, r0_0_0_1, g2_0);
              const double r0_0_1_0 = Y * b1;
              g2_2 = fma(ek2_0, r0_0_1_0, g2_2);
              const double r0_1_0_0 = X * b1;
              g2_3 = fma(ek2_0, r0_1_0_0, g2_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g2_4 = fma(ek2_0, r0_0_0_2, g2_4);
              g2_1 = fma(ek2_1, r0_0_0_2, g2_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g2_5 = fma(ek2_0, r0_0_1_1, g2_5);
              g2_2 = fma(ek2_1, r0_0_1_1, g2_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g2_6 = fma(ek2_0, r0_0_2_0, g2_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g2_7 = fma(ek2_0, r0_1_0_1, g2_7);
              g2_3 = fma(ek2_1, r0_1_0_1, g2_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g2_8 = fma(ek2_0, r0_1_1_0, g2_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g2_9 = fma(ek2_0, r0_2_0_0, g2_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g2_10 = fma(ek2_0, r0_0_0_3, g2_10);
              g2_4 = fma(ek2_1, r0_0_0_3, g2_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g2_11 = fma(ek2_0, r0_0_1_2, g2_11);
              g2_5 = fma(ek2_1, r0_0_1_2, g2_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g2_12 = fma(ek2_0, r0_0_2_1, g2_12);
              g2_6 = fma(ek2_1, r0_0_2_1, g2_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g2_13 = fma(ek2_0, r0_0_3_0, g2_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g2_14 = fma(ek2_0, r0_1_0_2, g2_14);
              g2_7 = fma(ek2_1, r0_1_0_2, g2_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g2_15 = fma(ek2_0, r0_1_1_1, g2_15);
              g2_8 = fma(ek2_1, r0_1_1_1, g2_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g2_16 = fma(ek2_0, r0_1_2_0, g2_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g2_17 = fma(ek2_0, r0_2_0_1, g2_17);
              g2_9 = fma(ek2_1, r0_2_0_1, g2_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g2_18 = fma(ek2_0, r0_2_1_0, g2_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g2_19 = fma(ek2_0, r0_3_0_0, g2_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g2_10 = fma(ek2_1, r0_0_0_4, g2_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g2_11 = fma(ek2_1, r0_0_1_3, g2_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g2_12 = fma(ek2_1, r0_0_2_2, g2_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g2_13 = fma(ek2_1, r0_0_3_1, g2_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g2_14 = fma(ek2_1, r0_1_0_3, g2_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g2_15 = fma(ek2_1, r0_1_1_2, g2_15);
              const double r0_1_2_1 = X * r1_0_2_1;
              g2_16 = fma(ek2_1, r0_1_2_1, g2_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g2_17 = fma(ek2_1, r0_2_0_2, g2_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g2_18 = fma(ek2_1, r0_2_1_1, g2_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g2_19 = fma(ek2_1, r0_3_0_1, g2_19);
            }
            { const double eb = bi[5];
              o0_2 = fma(eb, g2_0, o0_2);
            }
            { const double eb = bi[6];
              o0_2 = fma(eb, g2_3, o0_2);
            }
            { const double eb = bi[7];
              o0_2 = fma(eb, g2_9, o0_2);
            }
            { const double eb = bi[8];
              o1_2 = fma(eb, g2_0, o1_2);
            }
            { const double eb = bi[9];
              o1_2 = fma(eb, g2_3, o1_2);
            }
            { const double eb = bi[10];
              o1_2 = fma(eb, g2_9, o1_2);
            }
            { const double eb = bi[11];
              o1_2 = fma(eb, g2_19, o1_2);
            }
            { const double eb = bi[12];
              o2_2 = fma(eb, g2_0, o2_2);
            }
            { const double eb = bi[13];
              o2_2 = fma(eb, g2_2, o2_2);
            }
            { const double eb = bi[14];
              o2_2 = fma(eb, g2_3, o2_2);
            }
            { const double eb = bi[15];
              o2_2 = fma(eb, g2_8, o2_2);
            }
            { const double eb = bi[16];
              o2_2 = fma(eb, g2_9, o2_2);
            }
            { const double eb = bi[17];
              o2_2 = fma(eb, g2_18, o2_2);
            }
            { const double eb = bi[18];
              o3_2 = fma(eb, g2_0, o3_2);
            }
            { const double eb = bi[19];
              o3_2 = fma(eb, g2_1, o3_2);
            }
            { const double eb = bi[20];
              o3_2 = fma(eb, g2_3, o3_2);
            }
            { const double eb = bi[21];
              o3_2 = fma(eb, g2_7, o3_2);
            }
            { const double eb = bi[22];
              o3_2 = fma(eb, g2_9, o3_2);
            }
            { const double eb = bi[23];
              o3_2 = fma(eb, g2_17, o3_2);
            }
            { const double eb = bi[24];
              o4_2 = fma(eb, g2_0, o4_2);
            }
            { const double eb = bi[25];
              o4_2 = fma(eb, g2_2, o4_2);
            }
            { const double eb = bi[26];
              o4_2 = fma(eb, g2_6, o4_2);
            }
            { const double eb = bi[27];
              o5_2 = fma(eb, g2_0, o5_2);
            }
            { const double eb = bi[28];
              o5_2 = fma(eb, g2_2, o5_2);
            }
            { const double eb = bi[29];
              o5_2 = fma(eb, g2_6, o5_2);
            }
            { const double eb = bi[30];
              o5_2 = fma(eb, g2_3, o5_2);
            }
            { const double eb = bi[31];
              o5_2 = fma(eb, g2_8, o5_2);
            }
            { const double eb = bi[32];
              o5_2 = fma(eb, g2_16, o5_2);
            }
            { const double eb = bi[33];
              o6_2 = fma(eb, g2_0, o6_2);
            }
            { const double eb = bi[34];
              o6_2 = fma(eb, g2_2, o6_2);
            }
            { const double eb = bi[35];
              o6_2 = fma(eb, g2_6, o6_2);
            }
            { const double eb = bi[36];
              o6_2 = fma(eb, g2_13, o6_2);
            }
            { const double eb = bi[37];
              o7_2 = fma(eb, g2_0, o7_2);
            }
            { const double eb = bi[38];
              o7_2 = fma(eb, g2_1, o7_2);
            }
            { const double eb = bi[39];
              o7_2 = fma(eb, g2_2, o7_2);
            }
            { const double eb = bi[40];
              o7_2 = fma(eb, g2_5, o7_2);
            }
            { const double eb = bi[41];
              o7_2 = fma(eb, g2_6, o7_2);
            }
            { const double eb = bi[42];
              o7_2 = fma(eb, g2_12, o7_2);
            }
            { const double eb = bi[43];
              o8_2 = fma(eb, g2_0, o8_2);
            }
            { const double eb = bi[44];
              o8_2 = fma(eb, g2_1, o8_2);
            }
            { const double eb = bi[45];
              o8_2 = fma(eb, g2_4, o8_2);
            }
            { const double eb = bi[46];
              o9_2 = fma(eb, g2_0, o9_2);
            }
            { const double eb = bi[47];
              o9_2 = fma(eb, g2_1, o9_2);
            }
            { const double eb = bi[48];
              o9_2 = fma(eb, g2_4, o9_2);
            }
            { const double eb = bi[49];
              o9_2 = fma(eb, g2_3, o9_2);
            }
            { const double eb = bi[50];
              o9_2 = fma(eb, g2_7, o9_2);
            }
            { const double eb = bi[51];
              o9_2 = fma(eb, g2_14, o9_2);
            }
            { const double eb = bi[52];
              o10_2 = fma(eb, g2_0, o10_2);
            }
            { const double eb = bi[53];
              o10_2 = fma(eb, g2_1, o10_2);
            }
            { const double eb = bi[54];
              o10_2 = fma(eb, g2_4, o10_2);
            }
            { const double eb = bi[55];
              o10_2 = fma(eb, g2_2, o10_2);
            }
            { const double eb = bi[56];
              o10_2 = fma(eb, g2_5, o10_2);
            }
            { const double eb = bi[57];
              o10_2 = fma(eb, g2_11, o10_2);
            }
            { const double eb = bi[58];
              o11_2 = fma(eb, g2_0, o11_2);
            }
            { const double eb = bi[59];
              o11_2 = fma(eb, g2_1, o11_2);
            }
            { const double eb = bi[60];
              o11_2 = fma(eb, g2_4, o11_2);
            }
            { const double eb = bi[61];
              o11_2 = fma(eb, g2_10, o11_2);
            }
            { const double eb = bi[62];
              o12_2 = fma(eb, g2_0, o12_2);
            }
            { const double eb = bi[63];
              o12_2 = fma(eb, g2_2, o12_2);
            }
            { const double eb = bi[64];
              o12_2 = fma(eb, g2_3, o12_2);
            }
            { const double eb = bi[65];
              o12_2 = fma(eb, g2_8, o12_2);
            }
            { const double eb = bi[66];
              o13_2 = fma(eb, g2_0, o13_2);
            }
            { const double eb = bi[67];
              o13_2 = fma(eb, g2_2, o13_2);
            }
            { const double eb = bi[68];
              o13_2 = fma(eb, g2_3, o13_2);
            }
            { const double eb = bi[69];
              o13_2 = fma(eb, g2_8, o13_2);
            }
            { const double eb = bi[70];
              o13_2 = fma(eb, g2_9, o13_2);
            }
            { const double eb = bi[71];
              o13_2 = fma(eb, g2_18, o13_2);
            }
            { const double eb = bi[72];
              o14_2 = fma(eb, g2_0, o14_2);
            }
            { const double eb = bi[73];
              o14_2 = fma(eb, g2_2, o14_2);
            }
            { const double eb = bi[74];
              o14_2 = fma(eb, g2_6, o14_2);
            }
            { const double eb = bi[75];
              o14_2 = fma(eb, g2_3, o14_2);
            }
            { const double eb = bi[76];
              o14_2 = fma(eb, g2_8, o14_2);
            }
            { const double eb = bi[77];
              o14_2 = fma(eb, g2_16, o14_2);
            }
            { const double eb = bi[78];
              o15_2 = fma(eb, g2_0, o15_2);
            }
            { const double eb = bi[79];
              o15_2 = fma(eb, g2_1, o15_2);
            }
            { const double eb = bi[80];
              o15_2 = fma(eb, g2_2, o15_2);
            }
            { const double eb = bi[81];
              o15_2 = fma(eb, g2_5, o15_2);
            }
            { const double eb = bi[82];
              o15_2 = fma(eb, g2_3, o15_2);
            }
            { const double eb = bi[83];
              o15_2 = fma(eb, g2_7, o15_2);
            }
            { const double eb = bi[84];
              o15_2 = fma(eb, g2_8, o15_2);
            }
            { const double eb = bi[85];
              o15_2 = fma(eb, g2_15, o15_2);
            }
            { const double eb = bi[86];
              o16_2 = fma(eb, g2_0, o16_2);
            }
            { const double eb = bi[87];
              o16_2 = fma(eb, g2_1, o16_2);
            }
            { const double eb = bi[88];
              o16_2 = fma(eb, g2_3, o16_2);
            }
            { const double eb = bi[89];
              o16_2 = fma(eb, g2_7, o16_2);
            }
            { const double eb = bi[90];
              o17_2 = fma(eb, g2_0, o17_2);
            }
            { const double eb = bi[91];
              o17_2 = fma(eb, g2_1, o17_2);
            }
            { const double eb = bi[92];
              o17_2 = fma(eb, g2_3, o17_2);
            }
            { const double eb = bi[93];
              o17_2 = fma(eb, g2_7, o17_2);
            }
            { const double eb = bi[94];
              o17_2 = fma(eb, g2_9, o17_2);
            }
            { const double eb = bi[95];
              o17_2 = fma(eb, g2_17, o17_2);
            }
            { const double eb = bi[96];
              o18_2 = fma(eb, g2_0, o18_2);
            }
            { const double eb = bi[97];
              o18_2 = fma(eb, g2_1, o18_2);
            }
            { const double eb = bi[98];
              o18_2 = fma(eb, g2_2, o18_2);
            }
            { const double eb = bi[99];
              o18_2 = fma(eb, g2_5, o18_2);
            }
            { const double eb = bi[100];
              o18_2 = fma(eb, g2_3, o18_2);
            }
            { const double eb = bi[101];
              o18_2 = fma(eb, g2_7, o18_2);
            }
            { const double eb = bi[102];
              o18_2 = fma(eb, g2_8, o18_2);
            }
            { const double eb = bi[103];
              o18_2 = fma(eb, g2_15, o18_2);
            }
            { const double eb = bi[104];
              o19_2 = fma(eb, g2_0, o19_2);
            }
            { const double eb = bi[105];
              o19_2 = fma(eb, g2_1, o19_2);
            }
            { const double eb = bi[106];
              o19_2 = fma(eb, g2_4, o19_2);
            }
            { const double eb = bi[107];
              o19_2 = fma(eb, g2_3, o19_2);
            }
            { const double eb = bi[108];
              o19_2 = fma(eb, g2_7, o19_2);
            }
            { const double eb = bi[109];
              o19_2 = fma(eb, g2_14, o19_2);
            }
            { const double eb = bi[110];
              o20_2 = fma(eb, g2_0, o20_2);
            }
            { const double eb = bi[111];
              o20_2 = fma(eb, g2_1, o20_2);
            }
            { const double eb = bi[112];
              o20_2 = fma(eb, g2_2, o20_2);
            }
            { const double eb = bi[113];
              o20_2 = fma(eb, g2_5, o20_2);
            }
            { const double eb = bi[114];
              o21_2 = fma(eb, g2_0, o21_2);
            }
            { const double eb = bi[115];
              o21_2 = fma(eb, g2_1, o21_2);
            }
            { const double eb = bi[116];
              o21_2 = fma(eb, g2_2, o21_2);
            }
            { const double eb = bi[117];
              o21_2 = fma(eb, g2_5, o21_2);
            }
            { const double eb = bi[118];
              o21_2 = fma(eb, g2_3, o21_2);
            }
            { const double eb = bi[119];
              o21_2 = fma(eb, g2_7, o21_2);
            }
            { const double eb = bi[120];
              o21_2 = fma(eb, g2_8, o21_2);
            }
            { const double eb = bi[121];
              o21_2 = fma(eb, g2_15, o21_2);
            }
            { const double eb = bi[122];
              o22_2 = fma(eb, g2_0, o22_2);
            }
            { const double eb = bi[123];
              o22_2 = fma(eb, g2_1, o22_2);
            }
            { const double eb = bi[124];
              o22_2 = fma(eb, g2_2, o22_2);
            }
            { const double eb = bi[125];
              o22_2 = fma(eb, g2_5, o22_2);
            }
            { const double eb = bi[126];
              o22_2 = fma(eb, g2_6, o22_2);
            }
            { const double eb = bi[127];
              o22_2 = fma(eb, g2_12, o22_2);
            }
            { const double eb = bi[128];
              o23_2 = fma(eb, g2_0, o23_2);
            }
            { const double eb = bi[129];
              o23_2 = fma(eb, g2_1, o23_2);
            }
            { const double eb = bi[130];
              o23_2 = fma(eb, g2_4, o23_2);
            }
            { const double eb = bi[131];
              o23_2 = fma(eb, g2_2, o23_2);
            }
            { const double eb = bi[132];
              o23_2 = fma(eb, g2_5, o23_2);
            }
            { const double eb = bi[133];
              o23_2 = fma(eb, g2_11, o23_2);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 2) * N + fJ + 0];
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
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
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
            jab0 += o0_2 * ptk2;
            jab1 += o1_2 * ptk2;
            jab2 += o2_2 * ptk2;
            jab3 += o3_2 * ptk2;
            jab4 += o4_2 * ptk2;
            jab5 += o5_2 * ptk2;
            jab6 += o6_2 * ptk2;
            jab7 += o7_2 * ptk2;
            jab8 += o8_2 * ptk2;
            jab9 += o9_2 * ptk2;
            jab10 += o10_2 * ptk2;
            jab11 += o11_2 * ptk2;
            jab12 += o12_2 * ptk2;
            jab13 += o13_2 * ptk2;
            jab14 += o14_2 * ptk2;
            jab15 += o15_2 * ptk2;
            jab16 += o16_2 * ptk2;
            jab17 += o17_2 * ptk2;
            jab18 += o18_2 * ptk2;
            jab19 += o19_2 * ptk2;
            jab20 += o20_2 * ptk2;
            jab21 += o21_2 * ptk2;
            jab22 += o22_2 * ptk2;
            jab23 += o23_2 * ptk2;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17 + o18_2 * ptb18 + o19_2 * ptb19 + o20_2 * ptb20 + o21_2 * ptb21 + o22_2 * ptb22 + o23_2 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Abd0_0 + o1_2 * Abd1_0 + o2_2 * Abd2_0 + o3_2 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Aad0_0 + o4_2 * Aad1_0 + o8_2 * Aad2_0 + o12_2 * Aad3_0 + o16_2 * Aad4_0 + o20_2 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_2 * Abc0_2 + o1_2 * Abc1_2 + o2_2 * Abc2_2 + o3_2 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_2 * Aac0_2 + o4_2 * Aac1_2 + o8_2 * Aac2_2 + o12_2 * Aac3_2 + o16_2 * Aac4_2 + o20_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_2 * Aad0_0 + o5_2 * Aad1_0 + o9_2 * Aad2_0 + o13_2 * Aad3_0 + o17_2 * Aad4_0 + o21_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_2 * Aac0_2 + o5_2 * Aac1_2 + o9_2 * Aac2_2 + o13_2 * Aac3_2 + o17_2 * Aac4_2 + o21_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_2 * Aad0_0 + o6_2 * Aad1_0 + o10_2 * Aad2_0 + o14_2 * Aad3_0 + o18_2 * Aad4_0 + o22_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_2 * Aac0_2 + o6_2 * Aac1_2 + o10_2 * Aac2_2 + o14_2 * Aac3_2 + o18_2 * Aac4_2 + o22_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_2 * Aad0_0 + o7_2 * Aad1_0 + o11_2 * Aad2_0 + o15_2 * Aad3_0 + o19_2 * Aad4_0 + o23_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_2 * Aac0_2 + o7_2 * Aac1_2 + o11_2 * Aac2_2 + o15_2 * Aac3_2 + o19_2 * Aac4_2 + o23_2 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_2 * Abd0_0 + o5_2 * Abd1_0 + o6_2 * Abd2_0 + o7_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_2 * Abc0_2 + o5_2 * Abc1_2 + o6_2 * Abc2_2 + o7_2 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_2 * Abd0_0 + o9_2 * Abd1_0 + o10_2 * Abd2_0 + o11_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_2 * Abc0_2 + o9_2 * Abc1_2 + o10_2 * Abc2_2 + o11_2 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_2 * Abd0_0 + o13_2 * Abd1_0 + o14_2 * Abd2_0 + o15_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_2 * Abc0_2 + o13_2 * Abc1_2 + o14_2 * Abc2_2 + o15_2 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_2 * Abd0_0 + o17_2 * Abd1_0 + o18_2 * Abd2_0 + o19_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_2 * Abc0_2 + o17_2 * Abc1_2 + o18_2 * Abc2_2 + o19_2 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_2 * Abd0_0 + o21_2 * Abd1_0 + o22_2 * Abd2_0 + o23_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_2 * Abc0_2 + o21_2 * Abc1_2 + o22_2 * Abc2_2 + o23_2 * Abc3_2));
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
