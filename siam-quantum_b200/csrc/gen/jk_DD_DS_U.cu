// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DD_DS_U(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 341; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];
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
      bool mpq = false;                            // multipole mode: the quartet takes monopole values
      int erx = -1, erexp = sqb::ERR_UNKNOWN;      // its error-bank slot and stored exponent
      if (ok) {
        kp = a.ket_pairs[it.k0 + kl];
        const double r = bp.schwarz * kp.schwarz;
        ok = !(r < mr.cut_outer) && !(r < mr.cut_fixed);
        if (ok && a.erbank) { erx = a.er_items[qi_] + kl; erexp = a.erbank[erx]; }
        const bool mpc = erexp != sqb::ERR_UNKNOWN && r < a.mp_rmax;   // substitution candidate
        if (ok && (r < mr.dscreen_rmax || mpc)) {
          const bool bf = (bp.P > kp.P) || (bp.P == kp.P && bp.Q >= kp.Q);
          const int P = bf ? bp.P : kp.P, Q = bf ? bp.Q : kp.Q, I = bf ? kp.P : bp.P, J = bf ? kp.Q : bp.Q;
          const double* PM = a.PM + mr.pmoff; const int ns = mr.ns;
          const double mp = PM[P * ns + Q] + PM[I * ns + J] + PM[P * ns + I] + PM[P * ns + J] + PM[Q * ns + I] + PM[Q * ns + J];
          if (r < mr.dscreen_rmax) ok = !(r * mp < mr.cut_fixed);
          if (ok && mpc) mpq = a.pow15[erexp - sqb::ERR_MIN] * mp < mr.cut_fixed;
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
      double jab24 = 0.0;
      double jab25 = 0.0;
      double jab26 = 0.0;
      double jab27 = 0.0;
      double jab28 = 0.0;
      double jab29 = 0.0;
      double jab30 = 0.0;
      double jab31 = 0.0;
      double jab32 = 0.0;
      double jab33 = 0.0;
      double jab34 = 0.0;
      double jab35 = 0.0;
      unsigned long long nprimq = 0, nflush = 0;
      if (ok) {
        const double* __restrict__ kprim = a.ket_prims + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = mpq ? 0 : bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
        const double* __restrict__ PB = a.PB + mr.moff;
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // ket functions [0]
          double o0_0 = 0;
          double o1_0 = 0;
          double o2_0 = 0;
          double o3_0 = 0;
          double o4_0 = 0;
          double o5_0 = 0;
          double o6_0 = 0;
          double o7_0 = 0;
          double o8_0 = 0;
          double o9_0 = 0;
          double o10_0 = 0;
          double o11_0 = 0;
          double o12_0 = 0;
          double o13_0 = 0;
          double o14_0 = 0;
          double o15_0 = 0;
          double o16_0 = 0;
          double o17_0 = 0;
          double o18_0 = 0;
          double o19_0 = 0;
          double o20_0 = 0;
          double o21_0 = 0;
          double o22_0 = 0;
          double o23_0 = 0;
          double o24_0 = 0;
          double o25_0 = 0;
          double o26_0 = 0;
          double o27_0 = 0;
          double o28_0 = 0;
          double o29_0 = 0;
          double o30_0 = 0;
          double o31_0 = 0;
          double o32_0 = 0;
          double o33_0 = 0;
          double o34_0 = 0;
          double o35_0 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 341;
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
            double g0_20 = 0;
            double g0_21 = 0;
            double g0_22 = 0;
            double g0_23 = 0;
            double g0_24 = 0;
            double g0_25 = 0;
            double g0_26 = 0;
            double g0_27 = 0;
            double g0_28 = 0;
            double g0_29 = 0;
            double g0_30 = 0;
            double g0_31 = 0;
            double g0_32 = 0;
            double g0_33 = 0;
            double g0_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 26 * kS;
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
              g0_0 = fma(ek0_0, b0, g0_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fma(ek0_1, r0_1_0_0, g0_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g0_4 = fma(ek0_0, r0_0_0_2, g0_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fma(ek0_0, r0_0_1_1, g0_5);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g0_6 = fma(ek0_0, r0_0_2_0, g0_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fma(ek0_0, r0_1_0_1, g0_7);
              g0_1 = fma(ek0_1, r0_1_0_1, g0_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fma(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fma(ek0_1, r0_1_1_0, g0_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g0_9 = fma(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fma(ek0_1, r0_2_0_0, g0_3);
              g0_0 = fma(ek0_2, r0_2_0_0, g0_0);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g0_10 = fma(ek0_0, r0_0_0_3, g0_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g0_11 = fma(ek0_0, r0_0_1_2, g0_11);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g0_12 = fma(ek0_0, r0_0_2_1, g0_12);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g0_13 = fma(ek0_0, r0_0_3_0, g0_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g0_14 = fma(ek0_0, r0_1_0_2, g0_14);
              g0_4 = fma(ek0_1, r0_1_0_2, g0_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g0_15 = fma(ek0_0, r0_1_1_1, g0_15);
              g0_5 = fma(ek0_1, r0_1_1_1, g0_5);
              const double r0_1_2_0 = X * r1_0_2_0;
              g0_16 = fma(ek0_0, r0_1_2_0, g0_16);
              g0_6 = fma(ek0_1, r0_1_2_0, g0_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g0_17 = fma(ek0_0, r0_2_0_1, g0_17);
              g0_7 = fma(ek0_1, r0_2_0_1, g0_7);
              g0_1 = fma(ek0_2, r0_2_0_1, g0_1);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fma(ek0_0, r0_2_1_0, g0_18);
              g0_8 = fma(ek0_1, r0_2_1_0, g0_8);
              g0_2 = fma(ek0_2, r0_2_1_0, g0_2);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_19 = fma(ek0_0, r0_3_0_0, g0_19);
              g0_9 = fma(ek0_1, r0_3_0_0, g0_9);
              g0_3 = fma(ek0_2, r0_3_0_0, g0_3);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g0_20 = fma(ek0_0, r0_0_0_4, g0_20);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g0_21 = fma(ek0_0, r0_0_1_3, g0_21);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g0_22 = fma(ek0_0, r0_0_2_2, g0_22);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g0_23 = fma(ek0_0, r0_0_3_1, g0_23);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g0_24 = fma(ek0_0, r0_0_4_0, g0_24);
              const double r0_1_0_3 = X * r1_0_0_3;
              g0_25 = fma(ek0_0, r0_1_0_3, g0_25);
              g0_10 = fma(ek0_1, r0_1_0_3, g0_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g0_26 = fma(ek0_0, r0_1_1_2, g0_26);
              g0_11 = fma(ek0_1, r0_1_1_2, g0_11);
              const double r0_1_2_1 = X * r1_0_2_1;
              g0_27 = fma(ek0_0, r0_1_2_1, g0_27);
              g0_12 = fma(ek0_1, r0_1_2_1, g0_12);
              const double r0_1_3_0 = X * r1_0_3_0;
              g0_28 = fma(ek0_0, r0_1_3_0, g0_28);
              g0_13 = fma(ek0_1, r0_1_3_0, g0_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g0_29 = fma(ek0_0, r0_2_0_2, g0_29);
              g0_14 = fma(ek0_1, r0_2_0_2, g0_14);
              g0_4 = fma(ek0_2, r0_2_0_2, g0_4);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g0_30 = fma(ek0_0, r0_2_1_1, g0_30);
              g0_15 = fma(ek0_1, r0_2_1_1, g0_15);
              g0_5 = fma(ek0_2, r0_2_1_1, g0_5);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g0_31 = fma(ek0_0, r0_2_2_0, g0_31);
              g0_16 = fma(ek0_1, r0_2_2_0, g0_16);
              g0_6 = fma(ek0_2, r0_2_2_0, g0_6);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g0_32 = fma(ek0_0, r0_3_0_1, g0_32);
              g0_17 = fma(ek0_1, r0_3_0_1, g0_17);
              g0_7 = fma(ek0_2, r0_3_0_1, g0_7);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g0_33 = fma(ek0_0, r0_3_1_0, g0_33);
              g0_18 = fma(ek0_1, r0_3_1_0, g0_18);
              g0_8 = fma(ek0_2, r0_3_1_0, g0_8);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g0_34 = fma(ek0_0, r0_4_0_0, g0_34);
              g0_19 = fma(ek0_1, r0_4_0_0, g0_19);
              g0_9 = fma(ek0_2, r0_4_0_0, g0_9);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_1_0_4 = X * r1_0_0_4;
              g0_20 = fma(ek0_1, r0_1_0_4, g0_20);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g0_21 = fma(ek0_1, r0_1_1_3, g0_21);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g0_22 = fma(ek0_1, r0_1_2_2, g0_22);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g0_23 = fma(ek0_1, r0_1_3_1, g0_23);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g0_24 = fma(ek0_1, r0_1_4_0, g0_24);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g0_25 = fma(ek0_1, r0_2_0_3, g0_25);
              g0_10 = fma(ek0_2, r0_2_0_3, g0_10);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g0_26 = fma(ek0_1, r0_2_1_2, g0_26);
              g0_11 = fma(ek0_2, r0_2_1_2, g0_11);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g0_27 = fma(ek0_1, r0_2_2_1, g0_27);
              g0_12 = fma(ek0_2, r0_2_2_1, g0_12);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g0_28 = fma(ek0_1, r0_2_3_0, g0_28);
              g0_13 = fma(ek0_2, r0_2_3_0, g0_13);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g0_29 = fma(ek0_1, r0_3_0_2, g0_29);
              g0_14 = fma(ek0_2, r0_3_0_2, g0_14);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g0_30 = fma(ek0_1, r0_3_1_1, g0_30);
              g0_15 = fma(ek0_2, r0_3_1_1, g0_15);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g0_31 = fma(ek0_1, r0_3_2_0, g0_31);
              g0_16 = fma(ek0_2, r0_3_2_0, g0_16);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g0_32 = fma(ek0_1, r0_4_0_1, g0_32);
              g0_17 = fma(ek0_2, r0_4_0_1, g0_17);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g0_33 = fma(ek0_1, r0_4_1_0, g0_33);
              g0_18 = fma(ek0_2, r0_4_1_0, g0_18);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g0_34 = fma(ek0_1, r0_5_0_0, g0_34);
              g0_19 = fma(ek0_2, r0_5_0_0, g0_19);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g0_20 = fma(ek0_2, r0_2_0_4, g0_20);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g0_21 = fma(ek0_2, r0_2_1_3, g0_21);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g0_22 = fma(ek0_2, r0_2_2_2, g0_22);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g0_23 = fma(ek0_2, r0_2_3_1, g0_23);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g0_24 = fma(ek0_2, r0_2_4_0, g0_24);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g0_25 = fma(ek0_2, r0_3_0_3, g0_25);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g0_26 = fma(ek0_2, r0_3_1_2, g0_26);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g0_27 = fma(ek0_2, r0_3_2_1, g0_27);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g0_28 = fma(ek0_2, r0_3_3_0, g0_28);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g0_29 = fma(ek0_2, r0_4_0_2, g0_29);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g0_30 = fma(ek0_2, r0_4_1_1, g0_30);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g0_31 = fma(ek0_2, r0_4_2_0, g0_31);
              const double r4_1_0_1 = X * r5_0_0_1;
              const double r3_2_0_1 = fma(X, r4_1_0_1, r4_0_0_1);
              const double r2_3_0_1 = fma(X, r3_2_0_1, 2.0 * r3_1_0_1);
              const double r1_4_0_1 = fma(X, r2_3_0_1, 3.0 * r2_2_0_1);
              const double r0_5_0_1 = fma(X, r1_4_0_1, 4.0 * r1_3_0_1);
              g0_32 = fma(ek0_2, r0_5_0_1, g0_32);
              const double r4_1_1_0 = X * r5_0_1_0;
              const double r3_2_1_0 = fma(X, r4_1_1_0, r4_0_1_0);
              const double r2_3_1_0 = fma(X, r3_2_1_0, 2.0 * r3_1_1_0);
              const double r1_4_1_0 = fma(X, r2_3_1_0, 3.0 * r2_2_1_0);
              const double r0_5_1_0 = fma(X, r1_4_1_0, 4.0 * r1_3_1_0);
              g0_33 = fma(ek0_2, r0_5_1_0, g0_33);
              const double r5_1_0_0 = X * b6;
              const double r4_2_0_0 = fma(X, r5_1_0_0, b5);
              const double r3_3_0_0 = fma(X, r4_2_0_0, 2.0 * r4_1_0_0);
              const double r2_4_0_0 = fma(X, r3_3_0_0, 3.0 * r3_2_0_0);
              const double r1_5_0_0 = fma(X, r2_4_0_0, 4.0 * r2_3_0_0);
              const double r0_6_0_0 = fma(X, r1_5_0_0, 5.0 * r1_4_0_0);
              g0_34 = fma(ek0_2, r0_6_0_0, g0_34);
            }
            { const double eb = bi[5];
              o0_0 = fma(eb, g0_0, o0_0);
            }
            { const double eb = bi[6];
              o0_0 = fma(eb, g0_3, o0_0);
            }
            { const double eb = bi[7];
              o0_0 = fma(eb, g0_9, o0_0);
            }
            { const double eb = bi[8];
              o0_0 = fma(eb, g0_19, o0_0);
            }
            { const double eb = bi[9];
              o0_0 = fma(eb, g0_34, o0_0);
            }
            { const double eb = bi[10];
              o1_0 = fma(eb, g0_0, o1_0);
            }
            { const double eb = bi[11];
              o1_0 = fma(eb, g0_2, o1_0);
            }
            { const double eb = bi[12];
              o1_0 = fma(eb, g0_6, o1_0);
            }
            { const double eb = bi[13];
              o1_0 = fma(eb, g0_3, o1_0);
            }
            { const double eb = bi[14];
              o1_0 = fma(eb, g0_8, o1_0);
            }
            { const double eb = bi[15];
              o1_0 = fma(eb, g0_16, o1_0);
            }
            { const double eb = bi[16];
              o1_0 = fma(eb, g0_9, o1_0);
            }
            { const double eb = bi[17];
              o1_0 = fma(eb, g0_18, o1_0);
            }
            { const double eb = bi[18];
              o1_0 = fma(eb, g0_31, o1_0);
            }
            { const double eb = bi[19];
              o2_0 = fma(eb, g0_0, o2_0);
            }
            { const double eb = bi[20];
              o2_0 = fma(eb, g0_1, o2_0);
            }
            { const double eb = bi[21];
              o2_0 = fma(eb, g0_4, o2_0);
            }
            { const double eb = bi[22];
              o2_0 = fma(eb, g0_3, o2_0);
            }
            { const double eb = bi[23];
              o2_0 = fma(eb, g0_7, o2_0);
            }
            { const double eb = bi[24];
              o2_0 = fma(eb, g0_14, o2_0);
            }
            { const double eb = bi[25];
              o2_0 = fma(eb, g0_9, o2_0);
            }
            { const double eb = bi[26];
              o2_0 = fma(eb, g0_17, o2_0);
            }
            { const double eb = bi[27];
              o2_0 = fma(eb, g0_29, o2_0);
            }
            { const double eb = bi[28];
              o3_0 = fma(eb, g0_0, o3_0);
            }
            { const double eb = bi[29];
              o3_0 = fma(eb, g0_2, o3_0);
            }
            { const double eb = bi[30];
              o3_0 = fma(eb, g0_3, o3_0);
            }
            { const double eb = bi[31];
              o3_0 = fma(eb, g0_8, o3_0);
            }
            { const double eb = bi[32];
              o3_0 = fma(eb, g0_9, o3_0);
            }
            { const double eb = bi[33];
              o3_0 = fma(eb, g0_18, o3_0);
            }
            { const double eb = bi[34];
              o3_0 = fma(eb, g0_19, o3_0);
            }
            { const double eb = bi[35];
              o3_0 = fma(eb, g0_33, o3_0);
            }
            { const double eb = bi[36];
              o4_0 = fma(eb, g0_0, o4_0);
            }
            { const double eb = bi[37];
              o4_0 = fma(eb, g0_1, o4_0);
            }
            { const double eb = bi[38];
              o4_0 = fma(eb, g0_3, o4_0);
            }
            { const double eb = bi[39];
              o4_0 = fma(eb, g0_7, o4_0);
            }
            { const double eb = bi[40];
              o4_0 = fma(eb, g0_9, o4_0);
            }
            { const double eb = bi[41];
              o4_0 = fma(eb, g0_17, o4_0);
            }
            { const double eb = bi[42];
              o4_0 = fma(eb, g0_19, o4_0);
            }
            { const double eb = bi[43];
              o4_0 = fma(eb, g0_32, o4_0);
            }
            { const double eb = bi[44];
              o5_0 = fma(eb, g0_0, o5_0);
            }
            { const double eb = bi[45];
              o5_0 = fma(eb, g0_1, o5_0);
            }
            { const double eb = bi[46];
              o5_0 = fma(eb, g0_2, o5_0);
            }
            { const double eb = bi[47];
              o5_0 = fma(eb, g0_5, o5_0);
            }
            { const double eb = bi[48];
              o5_0 = fma(eb, g0_3, o5_0);
            }
            { const double eb = bi[49];
              o5_0 = fma(eb, g0_7, o5_0);
            }
            { const double eb = bi[50];
              o5_0 = fma(eb, g0_8, o5_0);
            }
            { const double eb = bi[51];
              o5_0 = fma(eb, g0_15, o5_0);
            }
            { const double eb = bi[52];
              o5_0 = fma(eb, g0_9, o5_0);
            }
            { const double eb = bi[53];
              o5_0 = fma(eb, g0_17, o5_0);
            }
            { const double eb = bi[54];
              o5_0 = fma(eb, g0_18, o5_0);
            }
            { const double eb = bi[55];
              o5_0 = fma(eb, g0_30, o5_0);
            }
            { const double eb = bi[56];
              o6_0 = fma(eb, g0_0, o6_0);
            }
            { const double eb = bi[57];
              o6_0 = fma(eb, g0_2, o6_0);
            }
            { const double eb = bi[58];
              o6_0 = fma(eb, g0_6, o6_0);
            }
            { const double eb = bi[59];
              o6_0 = fma(eb, g0_3, o6_0);
            }
            { const double eb = bi[60];
              o6_0 = fma(eb, g0_8, o6_0);
            }
            { const double eb = bi[61];
              o6_0 = fma(eb, g0_16, o6_0);
            }
            { const double eb = bi[62];
              o6_0 = fma(eb, g0_9, o6_0);
            }
            { const double eb = bi[63];
              o6_0 = fma(eb, g0_18, o6_0);
            }
            { const double eb = bi[64];
              o6_0 = fma(eb, g0_31, o6_0);
            }
            { const double eb = bi[65];
              o7_0 = fma(eb, g0_0, o7_0);
            }
            { const double eb = bi[66];
              o7_0 = fma(eb, g0_2, o7_0);
            }
            { const double eb = bi[67];
              o7_0 = fma(eb, g0_6, o7_0);
            }
            { const double eb = bi[68];
              o7_0 = fma(eb, g0_13, o7_0);
            }
            { const double eb = bi[69];
              o7_0 = fma(eb, g0_24, o7_0);
            }
            { const double eb = bi[70];
              o8_0 = fma(eb, g0_0, o8_0);
            }
            { const double eb = bi[71];
              o8_0 = fma(eb, g0_1, o8_0);
            }
            { const double eb = bi[72];
              o8_0 = fma(eb, g0_4, o8_0);
            }
            { const double eb = bi[73];
              o8_0 = fma(eb, g0_2, o8_0);
            }
            { const double eb = bi[74];
              o8_0 = fma(eb, g0_5, o8_0);
            }
            { const double eb = bi[75];
              o8_0 = fma(eb, g0_11, o8_0);
            }
            { const double eb = bi[76];
              o8_0 = fma(eb, g0_6, o8_0);
            }
            { const double eb = bi[77];
              o8_0 = fma(eb, g0_12, o8_0);
            }
            { const double eb = bi[78];
              o8_0 = fma(eb, g0_22, o8_0);
            }
            { const double eb = bi[79];
              o9_0 = fma(eb, g0_0, o9_0);
            }
            { const double eb = bi[80];
              o9_0 = fma(eb, g0_2, o9_0);
            }
            { const double eb = bi[81];
              o9_0 = fma(eb, g0_6, o9_0);
            }
            { const double eb = bi[82];
              o9_0 = fma(eb, g0_13, o9_0);
            }
            { const double eb = bi[83];
              o9_0 = fma(eb, g0_3, o9_0);
            }
            { const double eb = bi[84];
              o9_0 = fma(eb, g0_8, o9_0);
            }
            { const double eb = bi[85];
              o9_0 = fma(eb, g0_16, o9_0);
            }
            { const double eb = bi[86];
              o9_0 = fma(eb, g0_28, o9_0);
            }
            { const double eb = bi[87];
              o10_0 = fma(eb, g0_0, o10_0);
            }
            { const double eb = bi[88];
              o10_0 = fma(eb, g0_1, o10_0);
            }
            { const double eb = bi[89];
              o10_0 = fma(eb, g0_2, o10_0);
            }
            { const double eb = bi[90];
              o10_0 = fma(eb, g0_5, o10_0);
            }
            { const double eb = bi[91];
              o10_0 = fma(eb, g0_6, o10_0);
            }
            { const double eb = bi[92];
              o10_0 = fma(eb, g0_12, o10_0);
            }
            { const double eb = bi[93];
              o10_0 = fma(eb, g0_3, o10_0);
            }
            { const double eb = bi[94];
              o10_0 = fma(eb, g0_7, o10_0);
            }
            { const double eb = bi[95];
              o10_0 = fma(eb, g0_8, o10_0);
            }
            { const double eb = bi[96];
              o10_0 = fma(eb, g0_15, o10_0);
            }
            { const double eb = bi[97];
              o10_0 = fma(eb, g0_16, o10_0);
            }
            { const double eb = bi[98];
              o10_0 = fma(eb, g0_27, o10_0);
            }
            { const double eb = bi[99];
              o11_0 = fma(eb, g0_0, o11_0);
            }
            { const double eb = bi[100];
              o11_0 = fma(eb, g0_1, o11_0);
            }
            { const double eb = bi[101];
              o11_0 = fma(eb, g0_2, o11_0);
            }
            { const double eb = bi[102];
              o11_0 = fma(eb, g0_5, o11_0);
            }
            { const double eb = bi[103];
              o11_0 = fma(eb, g0_6, o11_0);
            }
            { const double eb = bi[104];
              o11_0 = fma(eb, g0_12, o11_0);
            }
            { const double eb = bi[105];
              o11_0 = fma(eb, g0_13, o11_0);
            }
            { const double eb = bi[106];
              o11_0 = fma(eb, g0_23, o11_0);
            }
            { const double eb = bi[107];
              o12_0 = fma(eb, g0_0, o12_0);
            }
            { const double eb = bi[108];
              o12_0 = fma(eb, g0_1, o12_0);
            }
            { const double eb = bi[109];
              o12_0 = fma(eb, g0_4, o12_0);
            }
            { const double eb = bi[110];
              o12_0 = fma(eb, g0_3, o12_0);
            }
            { const double eb = bi[111];
              o12_0 = fma(eb, g0_7, o12_0);
            }
            { const double eb = bi[112];
              o12_0 = fma(eb, g0_14, o12_0);
            }
            { const double eb = bi[113];
              o12_0 = fma(eb, g0_9, o12_0);
            }
            { const double eb = bi[114];
              o12_0 = fma(eb, g0_17, o12_0);
            }
            { const double eb = bi[115];
              o12_0 = fma(eb, g0_29, o12_0);
            }
            { const double eb = bi[116];
              o13_0 = fma(eb, g0_0, o13_0);
            }
            { const double eb = bi[117];
              o13_0 = fma(eb, g0_1, o13_0);
            }
            { const double eb = bi[118];
              o13_0 = fma(eb, g0_4, o13_0);
            }
            { const double eb = bi[119];
              o13_0 = fma(eb, g0_2, o13_0);
            }
            { const double eb = bi[120];
              o13_0 = fma(eb, g0_5, o13_0);
            }
            { const double eb = bi[121];
              o13_0 = fma(eb, g0_11, o13_0);
            }
            { const double eb = bi[122];
              o13_0 = fma(eb, g0_6, o13_0);
            }
            { const double eb = bi[123];
              o13_0 = fma(eb, g0_12, o13_0);
            }
            { const double eb = bi[124];
              o13_0 = fma(eb, g0_22, o13_0);
            }
            { const double eb = bi[125];
              o14_0 = fma(eb, g0_0, o14_0);
            }
            { const double eb = bi[126];
              o14_0 = fma(eb, g0_1, o14_0);
            }
            { const double eb = bi[127];
              o14_0 = fma(eb, g0_4, o14_0);
            }
            { const double eb = bi[128];
              o14_0 = fma(eb, g0_10, o14_0);
            }
            { const double eb = bi[129];
              o14_0 = fma(eb, g0_20, o14_0);
            }
            { const double eb = bi[130];
              o15_0 = fma(eb, g0_0, o15_0);
            }
            { const double eb = bi[131];
              o15_0 = fma(eb, g0_1, o15_0);
            }
            { const double eb = bi[132];
              o15_0 = fma(eb, g0_4, o15_0);
            }
            { const double eb = bi[133];
              o15_0 = fma(eb, g0_2, o15_0);
            }
            { const double eb = bi[134];
              o15_0 = fma(eb, g0_5, o15_0);
            }
            { const double eb = bi[135];
              o15_0 = fma(eb, g0_11, o15_0);
            }
            { const double eb = bi[136];
              o15_0 = fma(eb, g0_3, o15_0);
            }
            { const double eb = bi[137];
              o15_0 = fma(eb, g0_7, o15_0);
            }
            { const double eb = bi[138];
              o15_0 = fma(eb, g0_14, o15_0);
            }
            { const double eb = bi[139];
              o15_0 = fma(eb, g0_8, o15_0);
            }
            { const double eb = bi[140];
              o15_0 = fma(eb, g0_15, o15_0);
            }
            { const double eb = bi[141];
              o15_0 = fma(eb, g0_26, o15_0);
            }
            { const double eb = bi[142];
              o16_0 = fma(eb, g0_0, o16_0);
            }
            { const double eb = bi[143];
              o16_0 = fma(eb, g0_1, o16_0);
            }
            { const double eb = bi[144];
              o16_0 = fma(eb, g0_4, o16_0);
            }
            { const double eb = bi[145];
              o16_0 = fma(eb, g0_10, o16_0);
            }
            { const double eb = bi[146];
              o16_0 = fma(eb, g0_3, o16_0);
            }
            { const double eb = bi[147];
              o16_0 = fma(eb, g0_7, o16_0);
            }
            { const double eb = bi[148];
              o16_0 = fma(eb, g0_14, o16_0);
            }
            { const double eb = bi[149];
              o16_0 = fma(eb, g0_25, o16_0);
            }
            { const double eb = bi[150];
              o17_0 = fma(eb, g0_0, o17_0);
            }
            { const double eb = bi[151];
              o17_0 = fma(eb, g0_1, o17_0);
            }
            { const double eb = bi[152];
              o17_0 = fma(eb, g0_4, o17_0);
            }
            { const double eb = bi[153];
              o17_0 = fma(eb, g0_10, o17_0);
            }
            { const double eb = bi[154];
              o17_0 = fma(eb, g0_2, o17_0);
            }
            { const double eb = bi[155];
              o17_0 = fma(eb, g0_5, o17_0);
            }
            { const double eb = bi[156];
              o17_0 = fma(eb, g0_11, o17_0);
            }
            { const double eb = bi[157];
              o17_0 = fma(eb, g0_21, o17_0);
            }
            { const double eb = bi[158];
              o18_0 = fma(eb, g0_0, o18_0);
            }
            { const double eb = bi[159];
              o18_0 = fma(eb, g0_2, o18_0);
            }
            { const double eb = bi[160];
              o18_0 = fma(eb, g0_3, o18_0);
            }
            { const double eb = bi[161];
              o18_0 = fma(eb, g0_8, o18_0);
            }
            { const double eb = bi[162];
              o18_0 = fma(eb, g0_9, o18_0);
            }
            { const double eb = bi[163];
              o18_0 = fma(eb, g0_18, o18_0);
            }
            { const double eb = bi[164];
              o18_0 = fma(eb, g0_19, o18_0);
            }
            { const double eb = bi[165];
              o18_0 = fma(eb, g0_33, o18_0);
            }
            { const double eb = bi[166];
              o19_0 = fma(eb, g0_0, o19_0);
            }
            { const double eb = bi[167];
              o19_0 = fma(eb, g0_2, o19_0);
            }
            { const double eb = bi[168];
              o19_0 = fma(eb, g0_6, o19_0);
            }
            { const double eb = bi[169];
              o19_0 = fma(eb, g0_13, o19_0);
            }
            { const double eb = bi[170];
              o19_0 = fma(eb, g0_3, o19_0);
            }
            { const double eb = bi[171];
              o19_0 = fma(eb, g0_8, o19_0);
            }
            { const double eb = bi[172];
              o19_0 = fma(eb, g0_16, o19_0);
            }
            { const double eb = bi[173];
              o19_0 = fma(eb, g0_28, o19_0);
            }
            { const double eb = bi[174];
              o20_0 = fma(eb, g0_0, o20_0);
            }
            { const double eb = bi[175];
              o20_0 = fma(eb, g0_1, o20_0);
            }
            { const double eb = bi[176];
              o20_0 = fma(eb, g0_4, o20_0);
            }
            { const double eb = bi[177];
              o20_0 = fma(eb, g0_2, o20_0);
            }
            { const double eb = bi[178];
              o20_0 = fma(eb, g0_5, o20_0);
            }
            { const double eb = bi[179];
              o20_0 = fma(eb, g0_11, o20_0);
            }
            { const double eb = bi[180];
              o20_0 = fma(eb, g0_3, o20_0);
            }
            { const double eb = bi[181];
              o20_0 = fma(eb, g0_7, o20_0);
            }
            { const double eb = bi[182];
              o20_0 = fma(eb, g0_14, o20_0);
            }
            { const double eb = bi[183];
              o20_0 = fma(eb, g0_8, o20_0);
            }
            { const double eb = bi[184];
              o20_0 = fma(eb, g0_15, o20_0);
            }
            { const double eb = bi[185];
              o20_0 = fma(eb, g0_26, o20_0);
            }
            { const double eb = bi[186];
              o21_0 = fma(eb, g0_0, o21_0);
            }
            { const double eb = bi[187];
              o21_0 = fma(eb, g0_2, o21_0);
            }
            { const double eb = bi[188];
              o21_0 = fma(eb, g0_6, o21_0);
            }
            { const double eb = bi[189];
              o21_0 = fma(eb, g0_3, o21_0);
            }
            { const double eb = bi[190];
              o21_0 = fma(eb, g0_8, o21_0);
            }
            { const double eb = bi[191];
              o21_0 = fma(eb, g0_16, o21_0);
            }
            { const double eb = bi[192];
              o21_0 = fma(eb, g0_9, o21_0);
            }
            { const double eb = bi[193];
              o21_0 = fma(eb, g0_18, o21_0);
            }
            { const double eb = bi[194];
              o21_0 = fma(eb, g0_31, o21_0);
            }
            { const double eb = bi[195];
              o22_0 = fma(eb, g0_0, o22_0);
            }
            { const double eb = bi[196];
              o22_0 = fma(eb, g0_1, o22_0);
            }
            { const double eb = bi[197];
              o22_0 = fma(eb, g0_2, o22_0);
            }
            { const double eb = bi[198];
              o22_0 = fma(eb, g0_5, o22_0);
            }
            { const double eb = bi[199];
              o22_0 = fma(eb, g0_3, o22_0);
            }
            { const double eb = bi[200];
              o22_0 = fma(eb, g0_7, o22_0);
            }
            { const double eb = bi[201];
              o22_0 = fma(eb, g0_8, o22_0);
            }
            { const double eb = bi[202];
              o22_0 = fma(eb, g0_15, o22_0);
            }
            { const double eb = bi[203];
              o22_0 = fma(eb, g0_9, o22_0);
            }
            { const double eb = bi[204];
              o22_0 = fma(eb, g0_17, o22_0);
            }
            { const double eb = bi[205];
              o22_0 = fma(eb, g0_18, o22_0);
            }
            { const double eb = bi[206];
              o22_0 = fma(eb, g0_30, o22_0);
            }
            { const double eb = bi[207];
              o23_0 = fma(eb, g0_0, o23_0);
            }
            { const double eb = bi[208];
              o23_0 = fma(eb, g0_1, o23_0);
            }
            { const double eb = bi[209];
              o23_0 = fma(eb, g0_2, o23_0);
            }
            { const double eb = bi[210];
              o23_0 = fma(eb, g0_5, o23_0);
            }
            { const double eb = bi[211];
              o23_0 = fma(eb, g0_6, o23_0);
            }
            { const double eb = bi[212];
              o23_0 = fma(eb, g0_12, o23_0);
            }
            { const double eb = bi[213];
              o23_0 = fma(eb, g0_3, o23_0);
            }
            { const double eb = bi[214];
              o23_0 = fma(eb, g0_7, o23_0);
            }
            { const double eb = bi[215];
              o23_0 = fma(eb, g0_8, o23_0);
            }
            { const double eb = bi[216];
              o23_0 = fma(eb, g0_15, o23_0);
            }
            { const double eb = bi[217];
              o23_0 = fma(eb, g0_16, o23_0);
            }
            { const double eb = bi[218];
              o23_0 = fma(eb, g0_27, o23_0);
            }
            { const double eb = bi[219];
              o24_0 = fma(eb, g0_0, o24_0);
            }
            { const double eb = bi[220];
              o24_0 = fma(eb, g0_1, o24_0);
            }
            { const double eb = bi[221];
              o24_0 = fma(eb, g0_3, o24_0);
            }
            { const double eb = bi[222];
              o24_0 = fma(eb, g0_7, o24_0);
            }
            { const double eb = bi[223];
              o24_0 = fma(eb, g0_9, o24_0);
            }
            { const double eb = bi[224];
              o24_0 = fma(eb, g0_17, o24_0);
            }
            { const double eb = bi[225];
              o24_0 = fma(eb, g0_19, o24_0);
            }
            { const double eb = bi[226];
              o24_0 = fma(eb, g0_32, o24_0);
            }
            { const double eb = bi[227];
              o25_0 = fma(eb, g0_0, o25_0);
            }
            { const double eb = bi[228];
              o25_0 = fma(eb, g0_1, o25_0);
            }
            { const double eb = bi[229];
              o25_0 = fma(eb, g0_2, o25_0);
            }
            { const double eb = bi[230];
              o25_0 = fma(eb, g0_5, o25_0);
            }
            { const double eb = bi[231];
              o25_0 = fma(eb, g0_6, o25_0);
            }
            { const double eb = bi[232];
              o25_0 = fma(eb, g0_12, o25_0);
            }
            { const double eb = bi[233];
              o25_0 = fma(eb, g0_3, o25_0);
            }
            { const double eb = bi[234];
              o25_0 = fma(eb, g0_7, o25_0);
            }
            { const double eb = bi[235];
              o25_0 = fma(eb, g0_8, o25_0);
            }
            { const double eb = bi[236];
              o25_0 = fma(eb, g0_15, o25_0);
            }
            { const double eb = bi[237];
              o25_0 = fma(eb, g0_16, o25_0);
            }
            { const double eb = bi[238];
              o25_0 = fma(eb, g0_27, o25_0);
            }
            { const double eb = bi[239];
              o26_0 = fma(eb, g0_0, o26_0);
            }
            { const double eb = bi[240];
              o26_0 = fma(eb, g0_1, o26_0);
            }
            { const double eb = bi[241];
              o26_0 = fma(eb, g0_4, o26_0);
            }
            { const double eb = bi[242];
              o26_0 = fma(eb, g0_10, o26_0);
            }
            { const double eb = bi[243];
              o26_0 = fma(eb, g0_3, o26_0);
            }
            { const double eb = bi[244];
              o26_0 = fma(eb, g0_7, o26_0);
            }
            { const double eb = bi[245];
              o26_0 = fma(eb, g0_14, o26_0);
            }
            { const double eb = bi[246];
              o26_0 = fma(eb, g0_25, o26_0);
            }
            { const double eb = bi[247];
              o27_0 = fma(eb, g0_0, o27_0);
            }
            { const double eb = bi[248];
              o27_0 = fma(eb, g0_1, o27_0);
            }
            { const double eb = bi[249];
              o27_0 = fma(eb, g0_2, o27_0);
            }
            { const double eb = bi[250];
              o27_0 = fma(eb, g0_5, o27_0);
            }
            { const double eb = bi[251];
              o27_0 = fma(eb, g0_3, o27_0);
            }
            { const double eb = bi[252];
              o27_0 = fma(eb, g0_7, o27_0);
            }
            { const double eb = bi[253];
              o27_0 = fma(eb, g0_8, o27_0);
            }
            { const double eb = bi[254];
              o27_0 = fma(eb, g0_15, o27_0);
            }
            { const double eb = bi[255];
              o27_0 = fma(eb, g0_9, o27_0);
            }
            { const double eb = bi[256];
              o27_0 = fma(eb, g0_17, o27_0);
            }
            { const double eb = bi[257];
              o27_0 = fma(eb, g0_18, o27_0);
            }
            { const double eb = bi[258];
              o27_0 = fma(eb, g0_30, o27_0);
            }
            { const double eb = bi[259];
              o28_0 = fma(eb, g0_0, o28_0);
            }
            { const double eb = bi[260];
              o28_0 = fma(eb, g0_1, o28_0);
            }
            { const double eb = bi[261];
              o28_0 = fma(eb, g0_4, o28_0);
            }
            { const double eb = bi[262];
              o28_0 = fma(eb, g0_3, o28_0);
            }
            { const double eb = bi[263];
              o28_0 = fma(eb, g0_7, o28_0);
            }
            { const double eb = bi[264];
              o28_0 = fma(eb, g0_14, o28_0);
            }
            { const double eb = bi[265];
              o28_0 = fma(eb, g0_9, o28_0);
            }
            { const double eb = bi[266];
              o28_0 = fma(eb, g0_17, o28_0);
            }
            { const double eb = bi[267];
              o28_0 = fma(eb, g0_29, o28_0);
            }
            { const double eb = bi[268];
              o29_0 = fma(eb, g0_0, o29_0);
            }
            { const double eb = bi[269];
              o29_0 = fma(eb, g0_1, o29_0);
            }
            { const double eb = bi[270];
              o29_0 = fma(eb, g0_4, o29_0);
            }
            { const double eb = bi[271];
              o29_0 = fma(eb, g0_2, o29_0);
            }
            { const double eb = bi[272];
              o29_0 = fma(eb, g0_5, o29_0);
            }
            { const double eb = bi[273];
              o29_0 = fma(eb, g0_11, o29_0);
            }
            { const double eb = bi[274];
              o29_0 = fma(eb, g0_3, o29_0);
            }
            { const double eb = bi[275];
              o29_0 = fma(eb, g0_7, o29_0);
            }
            { const double eb = bi[276];
              o29_0 = fma(eb, g0_14, o29_0);
            }
            { const double eb = bi[277];
              o29_0 = fma(eb, g0_8, o29_0);
            }
            { const double eb = bi[278];
              o29_0 = fma(eb, g0_15, o29_0);
            }
            { const double eb = bi[279];
              o29_0 = fma(eb, g0_26, o29_0);
            }
            { const double eb = bi[280];
              o30_0 = fma(eb, g0_0, o30_0);
            }
            { const double eb = bi[281];
              o30_0 = fma(eb, g0_1, o30_0);
            }
            { const double eb = bi[282];
              o30_0 = fma(eb, g0_2, o30_0);
            }
            { const double eb = bi[283];
              o30_0 = fma(eb, g0_5, o30_0);
            }
            { const double eb = bi[284];
              o30_0 = fma(eb, g0_3, o30_0);
            }
            { const double eb = bi[285];
              o30_0 = fma(eb, g0_7, o30_0);
            }
            { const double eb = bi[286];
              o30_0 = fma(eb, g0_8, o30_0);
            }
            { const double eb = bi[287];
              o30_0 = fma(eb, g0_15, o30_0);
            }
            { const double eb = bi[288];
              o30_0 = fma(eb, g0_9, o30_0);
            }
            { const double eb = bi[289];
              o30_0 = fma(eb, g0_17, o30_0);
            }
            { const double eb = bi[290];
              o30_0 = fma(eb, g0_18, o30_0);
            }
            { const double eb = bi[291];
              o30_0 = fma(eb, g0_30, o30_0);
            }
            { const double eb = bi[292];
              o31_0 = fma(eb, g0_0, o31_0);
            }
            { const double eb = bi[293];
              o31_0 = fma(eb, g0_1, o31_0);
            }
            { const double eb = bi[294];
              o31_0 = fma(eb, g0_2, o31_0);
            }
            { const double eb = bi[295];
              o31_0 = fma(eb, g0_5, o31_0);
            }
            { const double eb = bi[296];
              o31_0 = fma(eb, g0_6, o31_0);
            }
            { const double eb = bi[297];
              o31_0 = fma(eb, g0_12, o31_0);
            }
            { const double eb = bi[298];
              o31_0 = fma(eb, g0_13, o31_0);
            }
            { const double eb = bi[299];
              o31_0 = fma(eb, g0_23, o31_0);
            }
            { const double eb = bi[300];
              o32_0 = fma(eb, g0_0, o32_0);
            }
            { const double eb = bi[301];
              o32_0 = fma(eb, g0_1, o32_0);
            }
            { const double eb = bi[302];
              o32_0 = fma(eb, g0_4, o32_0);
            }
            { const double eb = bi[303];
              o32_0 = fma(eb, g0_10, o32_0);
            }
            { const double eb = bi[304];
              o32_0 = fma(eb, g0_2, o32_0);
            }
            { const double eb = bi[305];
              o32_0 = fma(eb, g0_5, o32_0);
            }
            { const double eb = bi[306];
              o32_0 = fma(eb, g0_11, o32_0);
            }
            { const double eb = bi[307];
              o32_0 = fma(eb, g0_21, o32_0);
            }
            { const double eb = bi[308];
              o33_0 = fma(eb, g0_0, o33_0);
            }
            { const double eb = bi[309];
              o33_0 = fma(eb, g0_1, o33_0);
            }
            { const double eb = bi[310];
              o33_0 = fma(eb, g0_2, o33_0);
            }
            { const double eb = bi[311];
              o33_0 = fma(eb, g0_5, o33_0);
            }
            { const double eb = bi[312];
              o33_0 = fma(eb, g0_6, o33_0);
            }
            { const double eb = bi[313];
              o33_0 = fma(eb, g0_12, o33_0);
            }
            { const double eb = bi[314];
              o33_0 = fma(eb, g0_3, o33_0);
            }
            { const double eb = bi[315];
              o33_0 = fma(eb, g0_7, o33_0);
            }
            { const double eb = bi[316];
              o33_0 = fma(eb, g0_8, o33_0);
            }
            { const double eb = bi[317];
              o33_0 = fma(eb, g0_15, o33_0);
            }
            { const double eb = bi[318];
              o33_0 = fma(eb, g0_16, o33_0);
            }
            { const double eb = bi[319];
              o33_0 = fma(eb, g0_27, o33_0);
            }
            { const double eb = bi[320];
              o34_0 = fma(eb, g0_0, o34_0);
            }
            { const double eb = bi[321];
              o34_0 = fma(eb, g0_1, o34_0);
            }
            { const double eb = bi[322];
              o34_0 = fma(eb, g0_4, o34_0);
            }
            { const double eb = bi[323];
              o34_0 = fma(eb, g0_2, o34_0);
            }
            { const double eb = bi[324];
              o34_0 = fma(eb, g0_5, o34_0);
            }
            { const double eb = bi[325];
              o34_0 = fma(eb, g0_11, o34_0);
            }
            { const double eb = bi[326];
              o34_0 = fma(eb, g0_3, o34_0);
            }
            { const double eb = bi[327];
              o34_0 = fma(eb, g0_7, o34_0);
            }
            { const double eb = bi[328];
              o34_0 = fma(eb, g0_14, o34_0);
            }
            { const double eb = bi[329];
              o34_0 = fma(eb, g0_8, o34_0);
            }
            { const double eb = bi[330];
              o34_0 = fma(eb, g0_15, o34_0);
            }
            { const double eb = bi[331];
              o34_0 = fma(eb, g0_26, o34_0);
            }
            { const double eb = bi[332];
              o35_0 = fma(eb, g0_0, o35_0);
            }
            { const double eb = bi[333];
              o35_0 = fma(eb, g0_1, o35_0);
            }
            { const double eb = bi[334];
              o35_0 = fma(eb, g0_4, o35_0);
            }
            { const double eb = bi[335];
              o35_0 = fma(eb, g0_2, o35_0);
            }
            { const double eb = bi[336];
              o35_0 = fma(eb, g0_5, o35_0);
            }
            { const double eb = bi[337];
              o35_0 = fma(eb, g0_11, o35_0);
            }
            { const double eb = bi[338];
              o35_0 = fma(eb, g0_6, o35_0);
            }
            { const double eb = bi[339];
              o35_0 = fma(eb, g0_12, o35_0);
            }
            { const double eb = bi[340];
              o35_0 = fma(eb, g0_22, o35_0);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0);
            o1_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 0);
            o2_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 0);
            o3_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 0);
            o4_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 0, fJ + 0);
            o5_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 0, fJ + 0);
            o6_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0);
            o7_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 0);
            o8_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 0);
            o9_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 0);
            o10_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 0, fJ + 0);
            o11_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 0, fJ + 0);
            o12_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0);
            o13_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 0);
            o14_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 0);
            o15_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 0);
            o16_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 0, fJ + 0);
            o17_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 0, fJ + 0);
            o18_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0);
            o19_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 0);
            o20_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 0);
            o21_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 0);
            o22_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 0, fJ + 0);
            o23_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 0, fJ + 0);
            o24_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0);
            o25_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 0);
            o26_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 0);
            o27_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 0);
            o28_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 0, fJ + 0);
            o29_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 0, fJ + 0);
            o30_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0);
            o31_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 0);
            o32_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 0);
            o33_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 0);
            o34_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 0, fJ + 0);
            o35_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 0, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o1_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o2_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o3_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o4_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o5_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o6_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o7_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o8_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o9_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o10_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o11_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o12_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o13_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o14_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o15_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o16_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o17_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o18_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o19_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o20_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o21_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o22_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o23_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o24_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o25_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o26_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o27_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o28_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o29_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o30_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o31_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o32_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o33_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o34_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o35_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 0, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 0) * N + fQ + 4];
            const double ptb5 = PT[(fP + 0) * N + fQ + 5];
            const double ptb6 = PT[(fP + 1) * N + fQ + 0];
            const double ptb7 = PT[(fP + 1) * N + fQ + 1];
            const double ptb8 = PT[(fP + 1) * N + fQ + 2];
            const double ptb9 = PT[(fP + 1) * N + fQ + 3];
            const double ptb10 = PT[(fP + 1) * N + fQ + 4];
            const double ptb11 = PT[(fP + 1) * N + fQ + 5];
            const double ptb12 = PT[(fP + 2) * N + fQ + 0];
            const double ptb13 = PT[(fP + 2) * N + fQ + 1];
            const double ptb14 = PT[(fP + 2) * N + fQ + 2];
            const double ptb15 = PT[(fP + 2) * N + fQ + 3];
            const double ptb16 = PT[(fP + 2) * N + fQ + 4];
            const double ptb17 = PT[(fP + 2) * N + fQ + 5];
            const double ptb18 = PT[(fP + 3) * N + fQ + 0];
            const double ptb19 = PT[(fP + 3) * N + fQ + 1];
            const double ptb20 = PT[(fP + 3) * N + fQ + 2];
            const double ptb21 = PT[(fP + 3) * N + fQ + 3];
            const double ptb22 = PT[(fP + 3) * N + fQ + 4];
            const double ptb23 = PT[(fP + 3) * N + fQ + 5];
            const double ptb24 = PT[(fP + 4) * N + fQ + 0];
            const double ptb25 = PT[(fP + 4) * N + fQ + 1];
            const double ptb26 = PT[(fP + 4) * N + fQ + 2];
            const double ptb27 = PT[(fP + 4) * N + fQ + 3];
            const double ptb28 = PT[(fP + 4) * N + fQ + 4];
            const double ptb29 = PT[(fP + 4) * N + fQ + 5];
            const double ptb30 = PT[(fP + 5) * N + fQ + 0];
            const double ptb31 = PT[(fP + 5) * N + fQ + 1];
            const double ptb32 = PT[(fP + 5) * N + fQ + 2];
            const double ptb33 = PT[(fP + 5) * N + fQ + 3];
            const double ptb34 = PT[(fP + 5) * N + fQ + 4];
            const double ptb35 = PT[(fP + 5) * N + fQ + 5];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd4_0 = PA[(fQ + 4) * N + fJ + 0];
            const double Abd5_0 = PA[(fQ + 5) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
            const double Abc4_0 = PA[(fQ + 4) * N + fI + 0];
            const double Abc5_0 = PA[(fQ + 5) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bbd4_0 = PB[(fQ + 4) * N + fJ + 0];
            const double Bbd5_0 = PB[(fQ + 5) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc1_0 = PB[(fQ + 1) * N + fI + 0];
            const double Bbc2_0 = PB[(fQ + 2) * N + fI + 0];
            const double Bbc3_0 = PB[(fQ + 3) * N + fI + 0];
            const double Bbc4_0 = PB[(fQ + 4) * N + fI + 0];
            const double Bbc5_0 = PB[(fQ + 5) * N + fI + 0];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            const double Bac1_0 = PB[(fP + 1) * N + fI + 0];
            const double Bac2_0 = PB[(fP + 2) * N + fI + 0];
            const double Bac3_0 = PB[(fP + 3) * N + fI + 0];
            const double Bac4_0 = PB[(fP + 4) * N + fI + 0];
            const double Bac5_0 = PB[(fP + 5) * N + fI + 0];
            jab0 += o0_0 * ptk0;
            jab1 += o1_0 * ptk0;
            jab2 += o2_0 * ptk0;
            jab3 += o3_0 * ptk0;
            jab4 += o4_0 * ptk0;
            jab5 += o5_0 * ptk0;
            jab6 += o6_0 * ptk0;
            jab7 += o7_0 * ptk0;
            jab8 += o8_0 * ptk0;
            jab9 += o9_0 * ptk0;
            jab10 += o10_0 * ptk0;
            jab11 += o11_0 * ptk0;
            jab12 += o12_0 * ptk0;
            jab13 += o13_0 * ptk0;
            jab14 += o14_0 * ptk0;
            jab15 += o15_0 * ptk0;
            jab16 += o16_0 * ptk0;
            jab17 += o17_0 * ptk0;
            jab18 += o18_0 * ptk0;
            jab19 += o19_0 * ptk0;
            jab20 += o20_0 * ptk0;
            jab21 += o21_0 * ptk0;
            jab22 += o22_0 * ptk0;
            jab23 += o23_0 * ptk0;
            jab24 += o24_0 * ptk0;
            jab25 += o25_0 * ptk0;
            jab26 += o26_0 * ptk0;
            jab27 += o27_0 * ptk0;
            jab28 += o28_0 * ptk0;
            jab29 += o29_0 * ptk0;
            jab30 += o30_0 * ptk0;
            jab31 += o31_0 * ptk0;
            jab32 += o32_0 * ptk0;
            jab33 += o33_0 * ptk0;
            jab34 += o34_0 * ptk0;
            jab35 += o35_0 * ptk0;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15 + o16_0 * ptb16 + o17_0 * ptb17 + o18_0 * ptb18 + o19_0 * ptb19 + o20_0 * ptb20 + o21_0 * ptb21 + o22_0 * ptb22 + o23_0 * ptb23 + o24_0 * ptb24 + o25_0 * ptb25 + o26_0 * ptb26 + o27_0 * ptb27 + o28_0 * ptb28 + o29_0 * ptb29 + o30_0 * ptb30 + o31_0 * ptb31 + o32_0 * ptb32 + o33_0 * ptb33 + o34_0 * ptb34 + o35_0 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0 + o3_0 * Abd3_0 + o4_0 * Abd4_0 + o5_0 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o6_0 * Aad1_0 + o12_0 * Aad2_0 + o18_0 * Aad3_0 + o24_0 * Aad4_0 + o30_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o1_0 * Abc1_0 + o2_0 * Abc2_0 + o3_0 * Abc3_0 + o4_0 * Abc4_0 + o5_0 * Abc5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o6_0 * Aac1_0 + o12_0 * Aac2_0 + o18_0 * Aac3_0 + o24_0 * Aac4_0 + o30_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o7_0 * Aad1_0 + o13_0 * Aad2_0 + o19_0 * Aad3_0 + o25_0 * Aad4_0 + o31_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o7_0 * Aac1_0 + o13_0 * Aac2_0 + o19_0 * Aac3_0 + o25_0 * Aac4_0 + o31_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o8_0 * Aad1_0 + o14_0 * Aad2_0 + o20_0 * Aad3_0 + o26_0 * Aad4_0 + o32_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o8_0 * Aac1_0 + o14_0 * Aac2_0 + o20_0 * Aac3_0 + o26_0 * Aac4_0 + o32_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Aad0_0 + o9_0 * Aad1_0 + o15_0 * Aad2_0 + o21_0 * Aad3_0 + o27_0 * Aad4_0 + o33_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Aac0_0 + o9_0 * Aac1_0 + o15_0 * Aac2_0 + o21_0 * Aac3_0 + o27_0 * Aac4_0 + o33_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 0, deg * (o4_0 * Aad0_0 + o10_0 * Aad1_0 + o16_0 * Aad2_0 + o22_0 * Aad3_0 + o28_0 * Aad4_0 + o34_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_0 * Aac0_0 + o10_0 * Aac1_0 + o16_0 * Aac2_0 + o22_0 * Aac3_0 + o28_0 * Aac4_0 + o34_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 0, deg * (o5_0 * Aad0_0 + o11_0 * Aad1_0 + o17_0 * Aad2_0 + o23_0 * Aad3_0 + o29_0 * Aad4_0 + o35_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_0 * Aac0_0 + o11_0 * Aac1_0 + o17_0 * Aac2_0 + o23_0 * Aac3_0 + o29_0 * Aac4_0 + o35_0 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o6_0 * Abd0_0 + o7_0 * Abd1_0 + o8_0 * Abd2_0 + o9_0 * Abd3_0 + o10_0 * Abd4_0 + o11_0 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_0 * Abc0_0 + o7_0 * Abc1_0 + o8_0 * Abc2_0 + o9_0 * Abc3_0 + o10_0 * Abc4_0 + o11_0 * Abc5_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0 + o15_0 * Abd3_0 + o16_0 * Abd4_0 + o17_0 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o13_0 * Abc1_0 + o14_0 * Abc2_0 + o15_0 * Abc3_0 + o16_0 * Abc4_0 + o17_0 * Abc5_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o18_0 * Abd0_0 + o19_0 * Abd1_0 + o20_0 * Abd2_0 + o21_0 * Abd3_0 + o22_0 * Abd4_0 + o23_0 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_0 * Abc0_0 + o19_0 * Abc1_0 + o20_0 * Abc2_0 + o21_0 * Abc3_0 + o22_0 * Abc4_0 + o23_0 * Abc5_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o24_0 * Abd0_0 + o25_0 * Abd1_0 + o26_0 * Abd2_0 + o27_0 * Abd3_0 + o28_0 * Abd4_0 + o29_0 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_0 * Abc0_0 + o25_0 * Abc1_0 + o26_0 * Abc2_0 + o27_0 * Abc3_0 + o28_0 * Abc4_0 + o29_0 * Abc5_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o30_0 * Abd0_0 + o31_0 * Abd1_0 + o32_0 * Abd2_0 + o33_0 * Abd3_0 + o34_0 * Abd4_0 + o35_0 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_0 * Abc0_0 + o31_0 * Abc1_0 + o32_0 * Abc2_0 + o33_0 * Abc3_0 + o34_0 * Abc4_0 + o35_0 * Abc5_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Bbd0_0 + o1_0 * Bbd1_0 + o2_0 * Bbd2_0 + o3_0 * Bbd3_0 + o4_0 * Bbd4_0 + o5_0 * Bbd5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Bad0_0 + o6_0 * Bad1_0 + o12_0 * Bad2_0 + o18_0 * Bad3_0 + o24_0 * Bad4_0 + o30_0 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Bbc0_0 + o1_0 * Bbc1_0 + o2_0 * Bbc2_0 + o3_0 * Bbc3_0 + o4_0 * Bbc4_0 + o5_0 * Bbc5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Bac0_0 + o6_0 * Bac1_0 + o12_0 * Bac2_0 + o18_0 * Bac3_0 + o24_0 * Bac4_0 + o30_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Bad0_0 + o7_0 * Bad1_0 + o13_0 * Bad2_0 + o19_0 * Bad3_0 + o25_0 * Bad4_0 + o31_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Bac0_0 + o7_0 * Bac1_0 + o13_0 * Bac2_0 + o19_0 * Bac3_0 + o25_0 * Bac4_0 + o31_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Bad0_0 + o8_0 * Bad1_0 + o14_0 * Bad2_0 + o20_0 * Bad3_0 + o26_0 * Bad4_0 + o32_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Bac0_0 + o8_0 * Bac1_0 + o14_0 * Bac2_0 + o20_0 * Bac3_0 + o26_0 * Bac4_0 + o32_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Bad0_0 + o9_0 * Bad1_0 + o15_0 * Bad2_0 + o21_0 * Bad3_0 + o27_0 * Bad4_0 + o33_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Bac0_0 + o9_0 * Bac1_0 + o15_0 * Bac2_0 + o21_0 * Bac3_0 + o27_0 * Bac4_0 + o33_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fI + 0, deg * (o4_0 * Bad0_0 + o10_0 * Bad1_0 + o16_0 * Bad2_0 + o22_0 * Bad3_0 + o28_0 * Bad4_0 + o34_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fJ + 0, deg * (o4_0 * Bac0_0 + o10_0 * Bac1_0 + o16_0 * Bac2_0 + o22_0 * Bac3_0 + o28_0 * Bac4_0 + o34_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fI + 0, deg * (o5_0 * Bad0_0 + o11_0 * Bad1_0 + o17_0 * Bad2_0 + o23_0 * Bad3_0 + o29_0 * Bad4_0 + o35_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fJ + 0, deg * (o5_0 * Bac0_0 + o11_0 * Bac1_0 + o17_0 * Bac2_0 + o23_0 * Bac3_0 + o29_0 * Bac4_0 + o35_0 * Bac5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o6_0 * Bbd0_0 + o7_0 * Bbd1_0 + o8_0 * Bbd2_0 + o9_0 * Bbd3_0 + o10_0 * Bbd4_0 + o11_0 * Bbd5_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o6_0 * Bbc0_0 + o7_0 * Bbc1_0 + o8_0 * Bbc2_0 + o9_0 * Bbc3_0 + o10_0 * Bbc4_0 + o11_0 * Bbc5_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o12_0 * Bbd0_0 + o13_0 * Bbd1_0 + o14_0 * Bbd2_0 + o15_0 * Bbd3_0 + o16_0 * Bbd4_0 + o17_0 * Bbd5_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o12_0 * Bbc0_0 + o13_0 * Bbc1_0 + o14_0 * Bbc2_0 + o15_0 * Bbc3_0 + o16_0 * Bbc4_0 + o17_0 * Bbc5_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o18_0 * Bbd0_0 + o19_0 * Bbd1_0 + o20_0 * Bbd2_0 + o21_0 * Bbd3_0 + o22_0 * Bbd4_0 + o23_0 * Bbd5_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o18_0 * Bbc0_0 + o19_0 * Bbc1_0 + o20_0 * Bbc2_0 + o21_0 * Bbc3_0 + o22_0 * Bbc4_0 + o23_0 * Bbc5_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o24_0 * Bbd0_0 + o25_0 * Bbd1_0 + o26_0 * Bbd2_0 + o27_0 * Bbd3_0 + o28_0 * Bbd4_0 + o29_0 * Bbd5_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o24_0 * Bbc0_0 + o25_0 * Bbc1_0 + o26_0 * Bbc2_0 + o27_0 * Bbc3_0 + o28_0 * Bbc4_0 + o29_0 * Bbc5_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o30_0 * Bbd0_0 + o31_0 * Bbd1_0 + o32_0 * Bbd2_0 + o33_0 * Bbd3_0 + o34_0 * Bbd4_0 + o35_0 * Bbd5_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o30_0 * Bbc0_0 + o31_0 * Bbc1_0 + o32_0 * Bbc2_0 + o33_0 * Bbc3_0 + o34_0 * Bbc4_0 + o35_0 * Bbc5_0));
          }
        } break;
        case 1: {  // ket functions [1]
          double o0_1 = 0;
          double o1_1 = 0;
          double o2_1 = 0;
          double o3_1 = 0;
          double o4_1 = 0;
          double o5_1 = 0;
          double o6_1 = 0;
          double o7_1 = 0;
          double o8_1 = 0;
          double o9_1 = 0;
          double o10_1 = 0;
          double o11_1 = 0;
          double o12_1 = 0;
          double o13_1 = 0;
          double o14_1 = 0;
          double o15_1 = 0;
          double o16_1 = 0;
          double o17_1 = 0;
          double o18_1 = 0;
          double o19_1 = 0;
          double o20_1 = 0;
          double o21_1 = 0;
          double o22_1 = 0;
          double o23_1 = 0;
          double o24_1 = 0;
          double o25_1 = 0;
          double o26_1 = 0;
          double o27_1 = 0;
          double o28_1 = 0;
          double o29_1 = 0;
          double o30_1 = 0;
          double o31_1 = 0;
          double o32_1 = 0;
          double o33_1 = 0;
          double o34_1 = 0;
          double o35_1 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 341;
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
            double g1_20 = 0;
            double g1_21 = 0;
            double g1_22 = 0;
            double g1_23 = 0;
            double g1_24 = 0;
            double g1_25 = 0;
            double g1_26 = 0;
            double g1_27 = 0;
            double g1_28 = 0;
            double g1_29 = 0;
            double g1_30 = 0;
            double g1_31 = 0;
            double g1_32 = 0;
            double g1_33 = 0;
            double g1_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 26 * kS;
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
              const double ek1_0 = kj[8 * kS];
              const double ek1_1 = -kj[9 * kS];
              const double ek1_2 = kj[10 * kS];
              g1_0 = fma(ek1_0, b0, g1_0);
              const double r0_0_0_1 = Z * b1;
              g1_1 = fma(ek1_0, r0_0_0_1, g1_1);
              const double r0_0_1_0 = Y * b1;
              g1_2 = fma(ek1_0, r0_0_1_0, g1_2);
              g1_0 = fma(ek1_1, r0_0_1_0, g1_0);
              const double r0_1_0_0 = X * b1;
              g1_3 = fma(ek1_0, r0_1_0_0, g1_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g1_4 = fma(ek1_0, r0_0_0_2, g1_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g1_5 = fma(ek1_0, r0_0_1_1, g1_5);
              g1_1 = fma(ek1_1, r0_0_1_1, g1_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g1_6 = fma(ek1_0, r0_0_2_0, g1_6);
              g1_2 = fma(ek1_1, r0_0_2_0, g1_2);
              g1_0 = fma(ek1_2, r0_0_2_0, g1_0);
              const double r0_1_0_1 = X * r1_0_0_1;
              g1_7 = fma(ek1_0, r0_1_0_1, g1_7);
              const double r0_1_1_0 = X * r1_0_1_0;
              g1_8 = fma(ek1_0, r0_1_1_0, g1_8);
              g1_3 = fma(ek1_1, r0_1_1_0, g1_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g1_9 = fma(ek1_0, r0_2_0_0, g1_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g1_10 = fma(ek1_0, r0_0_0_3, g1_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g1_11 = fma(ek1_0, r0_0_1_2, g1_11);
              g1_4 = fma(ek1_1, r0_0_1_2, g1_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g1_12 = fma(ek1_0, r0_0_2_1, g1_12);
              g1_5 = fma(ek1_1, r0_0_2_1, g1_5);
              g1_1 = fma(ek1_2, r0_0_2_1, g1_1);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g1_13 = fma(ek1_0, r0_0_3_0, g1_13);
              g1_6 = fma(ek1_1, r0_0_3_0, g1_6);
              g1_2 = fma(ek1_2, r0_0_3_0, g1_2);
              const double r0_1_0_2 = X * r1_0_0_2;
              g1_14 = fma(ek1_0, r0_1_0_2, g1_14);
              const double r0_1_1_1 = X * r1_0_1_1;
              g1_15 = fma(ek1_0, r0_1_1_1, g1_15);
              g1_7 = fma(ek1_1, r0_1_1_1, g1_7);
              const double r0_1_2_0 = X * r1_0_2_0;
              g1_16 = fma(ek1_0, r0_1_2_0, g1_16);
              g1_8 = fma(ek1_1, r0_1_2_0, g1_8);
              g1_3 = fma(ek1_2, r0_1_2_0, g1_3);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g1_17 = fma(ek1_0, r0_2_0_1, g1_17);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g1_18 = fma(ek1_0, r0_2_1_0, g1_18);
              g1_9 = fma(ek1_1, r0_2_1_0, g1_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g1_19 = fma(ek1_0, r0_3_0_0, g1_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g1_20 = fma(ek1_0, r0_0_0_4, g1_20);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g1_21 = fma(ek1_0, r0_0_1_3, g1_21);
              g1_10 = fma(ek1_1, r0_0_1_3, g1_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g1_22 = fma(ek1_0, r0_0_2_2, g1_22);
              g1_11 = fma(ek1_1, r0_0_2_2, g1_11);
              g1_4 = fma(ek1_2, r0_0_2_2, g1_4);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g1_23 = fma(ek1_0, r0_0_3_1, g1_23);
              g1_12 = fma(ek1_1, r0_0_3_1, g1_12);
              g1_5 = fma(ek1_2, r0_0_3_1, g1_5);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g1_24 = fma(ek1_0, r0_0_4_0, g1_24);
              g1_13 = fma(ek1_1, r0_0_4_0, g1_13);
              g1_6 = fma(ek1_2, r0_0_4_0, g1_6);
              const double r0_1_0_3 = X * r1_0_0_3;
              g1_25 = fma(ek1_0, r0_1_0_3, g1_25);
              const double r0_1_1_2 = X * r1_0_1_2;
              g1_26 = fma(ek1_0, r0_1_1_2, g1_26);
              g1_14 = fma(ek1_1, r0_1_1_2, g1_14);
              const double r0_1_2_1 = X * r1_0_2_1;
              g1_27 = fma(ek1_0, r0_1_2_1, g1_27);
              g1_15 = fma(ek1_1, r0_1_2_1, g1_15);
              g1_7 = fma(ek1_2, r0_1_2_1, g1_7);
              const double r0_1_3_0 = X * r1_0_3_0;
              g1_28 = fma(ek1_0, r0_1_3_0, g1_28);
              g1_16 = fma(ek1_1, r0_1_3_0, g1_16);
              g1_8 = fma(ek1_2, r0_1_3_0, g1_8);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g1_29 = fma(ek1_0, r0_2_0_2, g1_29);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g1_30 = fma(ek1_0, r0_2_1_1, g1_30);
              g1_17 = fma(ek1_1, r0_2_1_1, g1_17);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g1_31 = fma(ek1_0, r0_2_2_0, g1_31);
              g1_18 = fma(ek1_1, r0_2_2_0, g1_18);
              g1_9 = fma(ek1_2, r0_2_2_0, g1_9);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g1_32 = fma(ek1_0, r0_3_0_1, g1_32);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g1_33 = fma(ek1_0, r0_3_1_0, g1_33);
              g1_19 = fma(ek1_1, r0_3_1_0, g1_19);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g1_34 = fma(ek1_0, r0_4_0_0, g1_34);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g1_20 = fma(ek1_1, r0_0_1_4, g1_20);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g1_21 = fma(ek1_1, r0_0_2_3, g1_21);
              g1_10 = fma(ek1_2, r0_0_2_3, g1_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g1_22 = fma(ek1_1, r0_0_3_2, g1_22);
              g1_11 = fma(ek1_2, r0_0_3_2, g1_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g1_23 = fma(ek1_1, r0_0_4_1, g1_23);
              g1_12 = fma(ek1_2, r0_0_4_1, g1_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g1_24 = fma(ek1_1, r0_0_5_0, g1_24);
              g1_13 = fma(ek1_2, r0_0_5_0, g1_13);
              const double r0_1_1_3 = X * r1_0_1_3;
              g1_25 = fma(ek1_1, r0_1_1_3, g1_25);
              const double r0_1_2_2 = X * r1_0_2_2;
              g1_26 = fma(ek1_1, r0_1_2_2, g1_26);
              g1_14 = fma(ek1_2, r0_1_2_2, g1_14);
              const double r0_1_3_1 = X * r1_0_3_1;
              g1_27 = fma(ek1_1, r0_1_3_1, g1_27);
              g1_15 = fma(ek1_2, r0_1_3_1, g1_15);
              const double r0_1_4_0 = X * r1_0_4_0;
              g1_28 = fma(ek1_1, r0_1_4_0, g1_28);
              g1_16 = fma(ek1_2, r0_1_4_0, g1_16);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g1_29 = fma(ek1_1, r0_2_1_2, g1_29);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g1_30 = fma(ek1_1, r0_2_2_1, g1_30);
              g1_17 = fma(ek1_2, r0_2_2_1, g1_17);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g1_31 = fma(ek1_1, r0_2_3_0, g1_31);
              g1_18 = fma(ek1_2, r0_2_3_0, g1_18);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g1_32 = fma(ek1_1, r0_3_1_1, g1_32);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g1_33 = fma(ek1_1, r0_3_2_0, g1_33);
              g1_19 = fma(ek1_2, r0_3_2_0, g1_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g1_34 = fma(ek1_1, r0_4_1_0, g1_34);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_0_2_4 = fma(Y, r1_0_1_4, r1_0_0_4);
              g1_20 = fma(ek1_2, r0_0_2_4, g1_20);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_0_3_3 = fma(Y, r1_0_2_3, 2.0 * r1_0_1_3);
              g1_21 = fma(ek1_2, r0_0_3_3, g1_21);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_0_4_2 = fma(Y, r1_0_3_2, 3.0 * r1_0_2_2);
              g1_22 = fma(ek1_2, r0_0_4_2, g1_22);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_0_5_1 = fma(Y, r1_0_4_1, 4.0 * r1_0_3_1);
              g1_23 = fma(ek1_2, r0_0_5_1, g1_23);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_0_5_0 = fma(Y, r2_0_4_0, 4.0 * r2_0_3_0);
              const double r0_0_6_0 = fma(Y, r1_0_5_0, 5.0 * r1_0_4_0);
              g1_24 = fma(ek1_2, r0_0_6_0, g1_24);
              const double r0_1_2_3 = X * r1_0_2_3;
              g1_25 = fma(ek1_2, r0_1_2_3, g1_25);
              const double r0_1_3_2 = X * r1_0_3_2;
              g1_26 = fma(ek1_2, r0_1_3_2, g1_26);
              const double r0_1_4_1 = X * r1_0_4_1;
              g1_27 = fma(ek1_2, r0_1_4_1, g1_27);
              const double r0_1_5_0 = X * r1_0_5_0;
              g1_28 = fma(ek1_2, r0_1_5_0, g1_28);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g1_29 = fma(ek1_2, r0_2_2_2, g1_29);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g1_30 = fma(ek1_2, r0_2_3_1, g1_30);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g1_31 = fma(ek1_2, r0_2_4_0, g1_31);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g1_32 = fma(ek1_2, r0_3_2_1, g1_32);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g1_33 = fma(ek1_2, r0_3_3_0, g1_33);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g1_34 = fma(ek1_2, r0_4_2_0, g1_34);
            }
            { const double eb = bi[5];
              o0_1 = fma(eb, g1_0, o0_1);
            }
            { const double eb = bi[6];
              o0_1 = fma(eb, g1_3, o0_1);
            }
            { const double eb = bi[7];
              o0_1 = fma(eb, g1_9, o0_1);
            }
            { const double eb = bi[8];
              o0_1 = fma(eb, g1_19, o0_1);
            }
            { const double eb = bi[9];
              o0_1 = fma(eb, g1_34, o0_1);
            }
            { const double eb = bi[10];
              o1_1 = fma(eb, g1_0, o1_1);
            }
            { const double eb = bi[11];
              o1_1 = fma(eb, g1_2, o1_1);
            }
            { const double eb = bi[12];
              o1_1 = fma(eb, g1_6, o1_1);
            }
            { const double eb = bi[13];
              o1_1 = fma(eb, g1_3, o1_1);
            }
            { const double eb = bi[14];
              o1_1 = fma(eb, g1_8, o1_1);
            }
            { const double eb = bi[15];
              o1_1 = fma(eb, g1_16, o1_1);
            }
            { const double eb = bi[16];
              o1_1 = fma(eb, g1_9, o1_1);
            }
            { const double eb = bi[17];
              o1_1 = fma(eb, g1_18, o1_1);
            }
            { const double eb = bi[18];
              o1_1 = fma(eb, g1_31, o1_1);
            }
            { const double eb = bi[19];
              o2_1 = fma(eb, g1_0, o2_1);
            }
            { const double eb = bi[20];
              o2_1 = fma(eb, g1_1, o2_1);
            }
            { const double eb = bi[21];
              o2_1 = fma(eb, g1_4, o2_1);
            }
            { const double eb = bi[22];
              o2_1 = fma(eb, g1_3, o2_1);
            }
            { const double eb = bi[23];
              o2_1 = fma(eb, g1_7, o2_1);
            }
            { const double eb = bi[24];
              o2_1 = fma(eb, g1_14, o2_1);
            }
            { const double eb = bi[25];
              o2_1 = fma(eb, g1_9, o2_1);
            }
            { const double eb = bi[26];
              o2_1 = fma(eb, g1_17, o2_1);
            }
            { const double eb = bi[27];
              o2_1 = fma(eb, g1_29, o2_1);
            }
            { const double eb = bi[28];
              o3_1 = fma(eb, g1_0, o3_1);
            }
            { const double eb = bi[29];
              o3_1 = fma(eb, g1_2, o3_1);
            }
            { const double eb = bi[30];
              o3_1 = fma(eb, g1_3, o3_1);
            }
            { const double eb = bi[31];
              o3_1 = fma(eb, g1_8, o3_1);
            }
            { const double eb = bi[32];
              o3_1 = fma(eb, g1_9, o3_1);
            }
            { const double eb = bi[33];
              o3_1 = fma(eb, g1_18, o3_1);
            }
            { const double eb = bi[34];
              o3_1 = fma(eb, g1_19, o3_1);
            }
            { const double eb = bi[35];
              o3_1 = fma(eb, g1_33, o3_1);
            }
            { const double eb = bi[36];
              o4_1 = fma(eb, g1_0, o4_1);
            }
            { const double eb = bi[37];
              o4_1 = fma(eb, g1_1, o4_1);
            }
            { const double eb = bi[38];
              o4_1 = fma(eb, g1_3, o4_1);
            }
            { const double eb = bi[39];
              o4_1 = fma(eb, g1_7, o4_1);
            }
            { const double eb = bi[40];
              o4_1 = fma(eb, g1_9, o4_1);
            }
            { const double eb = bi[41];
              o4_1 = fma(eb, g1_17, o4_1);
            }
            { const double eb = bi[42];
              o4_1 = fma(eb, g1_19, o4_1);
            }
            { const double eb = bi[43];
              o4_1 = fma(eb, g1_32, o4_1);
            }
            { const double eb = bi[44];
              o5_1 = fma(eb, g1_0, o5_1);
            }
            { const double eb = bi[45];
              o5_1 = fma(eb, g1_1, o5_1);
            }
            { const double eb = bi[46];
              o5_1 = fma(eb, g1_2, o5_1);
            }
            { const double eb = bi[47];
              o5_1 = fma(eb, g1_5, o5_1);
            }
            { const double eb = bi[48];
              o5_1 = fma(eb, g1_3, o5_1);
            }
            { const double eb = bi[49];
              o5_1 = fma(eb, g1_7, o5_1);
            }
            { const double eb = bi[50];
              o5_1 = fma(eb, g1_8, o5_1);
            }
            { const double eb = bi[51];
              o5_1 = fma(eb, g1_15, o5_1);
            }
            { const double eb = bi[52];
              o5_1 = fma(eb, g1_9, o5_1);
            }
            { const double eb = bi[53];
              o5_1 = fma(eb, g1_17, o5_1);
            }
            { const double eb = bi[54];
              o5_1 = fma(eb, g1_18, o5_1);
            }
            { const double eb = bi[55];
              o5_1 = fma(eb, g1_30, o5_1);
            }
            { const double eb = bi[56];
              o6_1 = fma(eb, g1_0, o6_1);
            }
            { const double eb = bi[57];
              o6_1 = fma(eb, g1_2, o6_1);
            }
            { const double eb = bi[58];
              o6_1 = fma(eb, g1_6, o6_1);
            }
            { const double eb = bi[59];
              o6_1 = fma(eb, g1_3, o6_1);
            }
            { const double eb = bi[60];
              o6_1 = fma(eb, g1_8, o6_1);
            }
            { const double eb = bi[61];
              o6_1 = fma(eb, g1_16, o6_1);
            }
            { const double eb = bi[62];
              o6_1 = fma(eb, g1_9, o6_1);
            }
            { const double eb = bi[63];
              o6_1 = fma(eb, g1_18, o6_1);
            }
            { const double eb = bi[64];
              o6_1 = fma(eb, g1_31, o6_1);
            }
            { const double eb = bi[65];
              o7_1 = fma(eb, g1_0, o7_1);
            }
            { const double eb = bi[66];
              o7_1 = fma(eb, g1_2, o7_1);
            }
            { const double eb = bi[67];
              o7_1 = fma(eb, g1_6, o7_1);
            }
            { const double eb = bi[68];
              o7_1 = fma(eb, g1_13, o7_1);
            }
            { const double eb = bi[69];
              o7_1 = fma(eb, g1_24, o7_1);
            }
            { const double eb = bi[70];
              o8_1 = fma(eb, g1_0, o8_1);
            }
            { const double eb = bi[71];
              o8_1 = fma(eb, g1_1, o8_1);
            }
            { const double eb = bi[72];
              o8_1 = fma(eb, g1_4, o8_1);
            }
            { const double eb = bi[73];
              o8_1 = fma(eb, g1_2, o8_1);
            }
            { const double eb = bi[74];
              o8_1 = fma(eb, g1_5, o8_1);
            }
            { const double eb = bi[75];
              o8_1 = fma(eb, g1_11, o8_1);
            }
            { const double eb = bi[76];
              o8_1 = fma(eb, g1_6, o8_1);
            }
            { const double eb = bi[77];
              o8_1 = fma(eb, g1_12, o8_1);
            }
            { const double eb = bi[78];
              o8_1 = fma(eb, g1_22, o8_1);
            }
            { const double eb = bi[79];
              o9_1 = fma(eb, g1_0, o9_1);
            }
            { const double eb = bi[80];
              o9_1 = fma(eb, g1_2, o9_1);
            }
            { const double eb = bi[81];
              o9_1 = fma(eb, g1_6, o9_1);
            }
            { const double eb = bi[82];
              o9_1 = fma(eb, g1_13, o9_1);
            }
            { const double eb = bi[83];
              o9_1 = fma(eb, g1_3, o9_1);
            }
            { const double eb = bi[84];
              o9_1 = fma(eb, g1_8, o9_1);
            }
            { const double eb = bi[85];
              o9_1 = fma(eb, g1_16, o9_1);
            }
            { const double eb = bi[86];
              o9_1 = fma(eb, g1_28, o9_1);
            }
            { const double eb = bi[87];
              o10_1 = fma(eb, g1_0, o10_1);
            }
            { const double eb = bi[88];
              o10_1 = fma(eb, g1_1, o10_1);
            }
            { const double eb = bi[89];
              o10_1 = fma(eb, g1_2, o10_1);
            }
            { const double eb = bi[90];
              o10_1 = fma(eb, g1_5, o10_1);
            }
            { const double eb = bi[91];
              o10_1 = fma(eb, g1_6, o10_1);
            }
            { const double eb = bi[92];
              o10_1 = fma(eb, g1_12, o10_1);
            }
            { const double eb = bi[93];
              o10_1 = fma(eb, g1_3, o10_1);
            }
            { const double eb = bi[94];
              o10_1 = fma(eb, g1_7, o10_1);
            }
            { const double eb = bi[95];
              o10_1 = fma(eb, g1_8, o10_1);
            }
            { const double eb = bi[96];
              o10_1 = fma(eb, g1_15, o10_1);
            }
            { const double eb = bi[97];
              o10_1 = fma(eb, g1_16, o10_1);
            }
            { const double eb = bi[98];
              o10_1 = fma(eb, g1_27, o10_1);
            }
            { const double eb = bi[99];
              o11_1 = fma(eb, g1_0, o11_1);
            }
            { const double eb = bi[100];
              o11_1 = fma(eb, g1_1, o11_1);
            }
            { const double eb = bi[101];
              o11_1 = fma(eb, g1_2, o11_1);
            }
            { const double eb = bi[102];
              o11_1 = fma(eb, g1_5, o11_1);
            }
            { const double eb = bi[103];
              o11_1 = fma(eb, g1_6, o11_1);
            }
            { const double eb = bi[104];
              o11_1 = fma(eb, g1_12, o11_1);
            }
            { const double eb = bi[105];
              o11_1 = fma(eb, g1_13, o11_1);
            }
            { const double eb = bi[106];
              o11_1 = fma(eb, g1_23, o11_1);
            }
            { const double eb = bi[107];
              o12_1 = fma(eb, g1_0, o12_1);
            }
            { const double eb = bi[108];
              o12_1 = fma(eb, g1_1, o12_1);
            }
            { const double eb = bi[109];
              o12_1 = fma(eb, g1_4, o12_1);
            }
            { const double eb = bi[110];
              o12_1 = fma(eb, g1_3, o12_1);
            }
            { const double eb = bi[111];
              o12_1 = fma(eb, g1_7, o12_1);
            }
            { const double eb = bi[112];
              o12_1 = fma(eb, g1_14, o12_1);
            }
            { const double eb = bi[113];
              o12_1 = fma(eb, g1_9, o12_1);
            }
            { const double eb = bi[114];
              o12_1 = fma(eb, g1_17, o12_1);
            }
            { const double eb = bi[115];
              o12_1 = fma(eb, g1_29, o12_1);
            }
            { const double eb = bi[116];
              o13_1 = fma(eb, g1_0, o13_1);
            }
            { const double eb = bi[117];
              o13_1 = fma(eb, g1_1, o13_1);
            }
            { const double eb = bi[118];
              o13_1 = fma(eb, g1_4, o13_1);
            }
            { const double eb = bi[119];
              o13_1 = fma(eb, g1_2, o13_1);
            }
            { const double eb = bi[120];
              o13_1 = fma(eb, g1_5, o13_1);
            }
            { const double eb = bi[121];
              o13_1 = fma(eb, g1_11, o13_1);
            }
            { const double eb = bi[122];
              o13_1 = fma(eb, g1_6, o13_1);
            }
            { const double eb = bi[123];
              o13_1 = fma(eb, g1_12, o13_1);
            }
            { const double eb = bi[124];
              o13_1 = fma(eb, g1_22, o13_1);
            }
            { const double eb = bi[125];
              o14_1 = fma(eb, g1_0, o14_1);
            }
            { const double eb = bi[126];
              o14_1 = fma(eb, g1_1, o14_1);
            }
            { const double eb = bi[127];
              o14_1 = fma(eb, g1_4, o14_1);
            }
            { const double eb = bi[128];
              o14_1 = fma(eb, g1_10, o14_1);
            }
            { const double eb = bi[129];
              o14_1 = fma(eb, g1_20, o14_1);
            }
            { const double eb = bi[130];
              o15_1 = fma(eb, g1_0, o15_1);
            }
            { const double eb = bi[131];
              o15_1 = fma(eb, g1_1, o15_1);
            }
            { const double eb = bi[132];
              o15_1 = fma(eb, g1_4, o15_1);
            }
            { const double eb = bi[133];
              o15_1 = fma(eb, g1_2, o15_1);
            }
            { const double eb = bi[134];
              o15_1 = fma(eb, g1_5, o15_1);
            }
            { const double eb = bi[135];
              o15_1 = fma(eb, g1_11, o15_1);
            }
            { const double eb = bi[136];
              o15_1 = fma(eb, g1_3, o15_1);
            }
            { const double eb = bi[137];
              o15_1 = fma(eb, g1_7, o15_1);
            }
            { const double eb = bi[138];
              o15_1 = fma(eb, g1_14, o15_1);
            }
            { const double eb = bi[139];
              o15_1 = fma(eb, g1_8, o15_1);
            }
            { const double eb = bi[140];
              o15_1 = fma(eb, g1_15, o15_1);
            }
            { const double eb = bi[141];
              o15_1 = fma(eb, g1_26, o15_1);
            }
            { const double eb = bi[142];
              o16_1 = fma(eb, g1_0, o16_1);
            }
            { const double eb = bi[143];
              o16_1 = fma(eb, g1_1, o16_1);
            }
            { const double eb = bi[144];
              o16_1 = fma(eb, g1_4, o16_1);
            }
            { const double eb = bi[145];
              o16_1 = fma(eb, g1_10, o16_1);
            }
            { const double eb = bi[146];
              o16_1 = fma(eb, g1_3, o16_1);
            }
            { const double eb = bi[147];
              o16_1 = fma(eb, g1_7, o16_1);
            }
            { const double eb = bi[148];
              o16_1 = fma(eb, g1_14, o16_1);
            }
            { const double eb = bi[149];
              o16_1 = fma(eb, g1_25, o16_1);
            }
            { const double eb = bi[150];
              o17_1 = fma(eb, g1_0, o17_1);
            }
            { const double eb = bi[151];
              o17_1 = fma(eb, g1_1, o17_1);
            }
            { const double eb = bi[152];
              o17_1 = fma(eb, g1_4, o17_1);
            }
            { const double eb = bi[153];
              o17_1 = fma(eb, g1_10, o17_1);
            }
            { const double eb = bi[154];
              o17_1 = fma(eb, g1_2, o17_1);
            }
            { const double eb = bi[155];
              o17_1 = fma(eb, g1_5, o17_1);
            }
            { const double eb = bi[156];
              o17_1 = fma(eb, g1_11, o17_1);
            }
            { const double eb = bi[157];
              o17_1 = fma(eb, g1_21, o17_1);
            }
            { const double eb = bi[158];
              o18_1 = fma(eb, g1_0, o18_1);
            }
            { const double eb = bi[159];
              o18_1 = fma(eb, g1_2, o18_1);
            }
            { const double eb = bi[160];
              o18_1 = fma(eb, g1_3, o18_1);
            }
            { const double eb = bi[161];
              o18_1 = fma(eb, g1_8, o18_1);
            }
            { const double eb = bi[162];
              o18_1 = fma(eb, g1_9, o18_1);
            }
            { const double eb = bi[163];
              o18_1 = fma(eb, g1_18, o18_1);
            }
            { const double eb = bi[164];
              o18_1 = fma(eb, g1_19, o18_1);
            }
            { const double eb = bi[165];
              o18_1 = fma(eb, g1_33, o18_1);
            }
            { const double eb = bi[166];
              o19_1 = fma(eb, g1_0, o19_1);
            }
            { const double eb = bi[167];
              o19_1 = fma(eb, g1_2, o19_1);
            }
            { const double eb = bi[168];
              o19_1 = fma(eb, g1_6, o19_1);
            }
            { const double eb = bi[169];
              o19_1 = fma(eb, g1_13, o19_1);
            }
            { const double eb = bi[170];
              o19_1 = fma(eb, g1_3, o19_1);
            }
            { const double eb = bi[171];
              o19_1 = fma(eb, g1_8, o19_1);
            }
            { const double eb = bi[172];
              o19_1 = fma(eb, g1_16, o19_1);
            }
            { const double eb = bi[173];
              o19_1 = fma(eb, g1_28, o19_1);
            }
            { const double eb = bi[174];
              o20_1 = fma(eb, g1_0, o20_1);
            }
            { const double eb = bi[175];
              o20_1 = fma(eb, g1_1, o20_1);
            }
            { const double eb = bi[176];
              o20_1 = fma(eb, g1_4, o20_1);
            }
            { const double eb = bi[177];
              o20_1 = fma(eb, g1_2, o20_1);
            }
            { const double eb = bi[178];
              o20_1 = fma(eb, g1_5, o20_1);
            }
            { const double eb = bi[179];
              o20_1 = fma(eb, g1_11, o20_1);
            }
            { const double eb = bi[180];
              o20_1 = fma(eb, g1_3, o20_1);
            }
            { const double eb = bi[181];
              o20_1 = fma(eb, g1_7, o20_1);
            }
            { const double eb = bi[182];
              o20_1 = fma(eb, g1_14, o20_1);
            }
            { const double eb = bi[183];
              o20_1 = fma(eb, g1_8, o20_1);
            }
            { const double eb = bi[184];
              o20_1 = fma(eb, g1_15, o20_1);
            }
            { const double eb = bi[185];
              o20_1 = fma(eb, g1_26, o20_1);
            }
            { const double eb = bi[186];
              o21_1 = fma(eb, g1_0, o21_1);
            }
            { const double eb = bi[187];
              o21_1 = fma(eb, g1_2, o21_1);
            }
            { const double eb = bi[188];
              o21_1 = fma(eb, g1_6, o21_1);
            }
            { const double eb = bi[189];
              o21_1 = fma(eb, g1_3, o21_1);
            }
            { const double eb = bi[190];
              o21_1 = fma(eb, g1_8, o21_1);
            }
            { const double eb = bi[191];
              o21_1 = fma(eb, g1_16, o21_1);
            }
            { const double eb = bi[192];
              o21_1 = fma(eb, g1_9, o21_1);
            }
            { const double eb = bi[193];
              o21_1 = fma(eb, g1_18, o21_1);
            }
            { const double eb = bi[194];
              o21_1 = fma(eb, g1_31, o21_1);
            }
            { const double eb = bi[195];
              o22_1 = fma(eb, g1_0, o22_1);
            }
            { const double eb = bi[196];
              o22_1 = fma(eb, g1_1, o22_1);
            }
            { const double eb = bi[197];
              o22_1 = fma(eb, g1_2, o22_1);
            }
            { const double eb = bi[198];
              o22_1 = fma(eb, g1_5, o22_1);
            }
            { const double eb = bi[199];
              o22_1 = fma(eb, g1_3, o22_1);
            }
            { const double eb = bi[200];
              o22_1 = fma(eb, g1_7, o22_1);
            }
            { const double eb = bi[201];
              o22_1 = fma(eb, g1_8, o22_1);
            }
            { const double eb = bi[202];
              o22_1 = fma(eb, g1_15, o22_1);
            }
            { const double eb = bi[203];
              o22_1 = fma(eb, g1_9, o22_1);
            }
            { const double eb = bi[204];
              o22_1 = fma(eb, g1_17, o22_1);
            }
            { const double eb = bi[205];
              o22_1 = fma(eb, g1_18, o22_1);
            }
            { const double eb = bi[206];
              o22_1 = fma(eb, g1_30, o22_1);
            }
            { const double eb = bi[207];
              o23_1 = fma(eb, g1_0, o23_1);
            }
            { const double eb = bi[208];
              o23_1 = fma(eb, g1_1, o23_1);
            }
            { const double eb = bi[209];
              o23_1 = fma(eb, g1_2, o23_1);
            }
            { const double eb = bi[210];
              o23_1 = fma(eb, g1_5, o23_1);
            }
            { const double eb = bi[211];
              o23_1 = fma(eb, g1_6, o23_1);
            }
            { const double eb = bi[212];
              o23_1 = fma(eb, g1_12, o23_1);
            }
            { const double eb = bi[213];
              o23_1 = fma(eb, g1_3, o23_1);
            }
            { const double eb = bi[214];
              o23_1 = fma(eb, g1_7, o23_1);
            }
            { const double eb = bi[215];
              o23_1 = fma(eb, g1_8, o23_1);
            }
            { const double eb = bi[216];
              o23_1 = fma(eb, g1_15, o23_1);
            }
            { const double eb = bi[217];
              o23_1 = fma(eb, g1_16, o23_1);
            }
            { const double eb = bi[218];
              o23_1 = fma(eb, g1_27, o23_1);
            }
            { const double eb = bi[219];
              o24_1 = fma(eb, g1_0, o24_1);
            }
            { const double eb = bi[220];
              o24_1 = fma(eb, g1_1, o24_1);
            }
            { const double eb = bi[221];
              o24_1 = fma(eb, g1_3, o24_1);
            }
            { const double eb = bi[222];
              o24_1 = fma(eb, g1_7, o24_1);
            }
            { const double eb = bi[223];
              o24_1 = fma(eb, g1_9, o24_1);
            }
            { const double eb = bi[224];
              o24_1 = fma(eb, g1_17, o24_1);
            }
            { const double eb = bi[225];
              o24_1 = fma(eb, g1_19, o24_1);
            }
            { const double eb = bi[226];
              o24_1 = fma(eb, g1_32, o24_1);
            }
            { const double eb = bi[227];
              o25_1 = fma(eb, g1_0, o25_1);
            }
            { const double eb = bi[228];
              o25_1 = fma(eb, g1_1, o25_1);
            }
            { const double eb = bi[229];
              o25_1 = fma(eb, g1_2, o25_1);
            }
            { const double eb = bi[230];
              o25_1 = fma(eb, g1_5, o25_1);
            }
            { const double eb = bi[231];
              o25_1 = fma(eb, g1_6, o25_1);
            }
            { const double eb = bi[232];
              o25_1 = fma(eb, g1_12, o25_1);
            }
            { const double eb = bi[233];
              o25_1 = fma(eb, g1_3, o25_1);
            }
            { const double eb = bi[234];
              o25_1 = fma(eb, g1_7, o25_1);
            }
            { const double eb = bi[235];
              o25_1 = fma(eb, g1_8, o25_1);
            }
            { const double eb = bi[236];
              o25_1 = fma(eb, g1_15, o25_1);
            }
            { const double eb = bi[237];
              o25_1 = fma(eb, g1_16, o25_1);
            }
            { const double eb = bi[238];
              o25_1 = fma(eb, g1_27, o25_1);
            }
            { const double eb = bi[239];
              o26_1 = fma(eb, g1_0, o26_1);
            }
            { const double eb = bi[240];
              o26_1 = fma(eb, g1_1, o26_1);
            }
            { const double eb = bi[241];
              o26_1 = fma(eb, g1_4, o26_1);
            }
            { const double eb = bi[242];
              o26_1 = fma(eb, g1_10, o26_1);
            }
            { const double eb = bi[243];
              o26_1 = fma(eb, g1_3, o26_1);
            }
            { const double eb = bi[244];
              o26_1 = fma(eb, g1_7, o26_1);
            }
            { const double eb = bi[245];
              o26_1 = fma(eb, g1_14, o26_1);
            }
            { const double eb = bi[246];
              o26_1 = fma(eb, g1_25, o26_1);
            }
            { const double eb = bi[247];
              o27_1 = fma(eb, g1_0, o27_1);
            }
            { const double eb = bi[248];
              o27_1 = fma(eb, g1_1, o27_1);
            }
            { const double eb = bi[249];
              o27_1 = fma(eb, g1_2, o27_1);
            }
            { const double eb = bi[250];
              o27_1 = fma(eb, g1_5, o27_1);
            }
            { const double eb = bi[251];
              o27_1 = fma(eb, g1_3, o27_1);
            }
            { const double eb = bi[252];
              o27_1 = fma(eb, g1_7, o27_1);
            }
            { const double eb = bi[253];
              o27_1 = fma(eb, g1_8, o27_1);
            }
            { const double eb = bi[254];
              o27_1 = fma(eb, g1_15, o27_1);
            }
            { const double eb = bi[255];
              o27_1 = fma(eb, g1_9, o27_1);
            }
            { const double eb = bi[256];
              o27_1 = fma(eb, g1_17, o27_1);
            }
            { const double eb = bi[257];
              o27_1 = fma(eb, g1_18, o27_1);
            }
            { const double eb = bi[258];
              o27_1 = fma(eb, g1_30, o27_1);
            }
            { const double eb = bi[259];
              o28_1 = fma(eb, g1_0, o28_1);
            }
            { const double eb = bi[260];
              o28_1 = fma(eb, g1_1, o28_1);
            }
            { const double eb = bi[261];
              o28_1 = fma(eb, g1_4, o28_1);
            }
            { const double eb = bi[262];
              o28_1 = fma(eb, g1_3, o28_1);
            }
            { const double eb = bi[263];
              o28_1 = fma(eb, g1_7, o28_1);
            }
            { const double eb = bi[264];
              o28_1 = fma(eb, g1_14, o28_1);
            }
            { const double eb = bi[265];
              o28_1 = fma(eb, g1_9, o28_1);
            }
            { const double eb = bi[266];
              o28_1 = fma(eb, g1_17, o28_1);
            }
            { const double eb = bi[267];
              o28_1 = fma(eb, g1_29, o28_1);
            }
            { const double eb = bi[268];
              o29_1 = fma(eb, g1_0, o29_1);
            }
            { const double eb = bi[269];
              o29_1 = fma(eb, g1_1, o29_1);
            }
            { const double eb = bi[270];
              o29_1 = fma(eb, g1_4, o29_1);
            }
            { const double eb = bi[271];
              o29_1 = fma(eb, g1_2, o29_1);
            }
            { const double eb = bi[272];
              o29_1 = fma(eb, g1_5, o29_1);
            }
            { const double eb = bi[273];
              o29_1 = fma(eb, g1_11, o29_1);
            }
            { const double eb = bi[274];
              o29_1 = fma(eb, g1_3, o29_1);
            }
            { const double eb = bi[275];
              o29_1 = fma(eb, g1_7, o29_1);
            }
            { const double eb = bi[276];
              o29_1 = fma(eb, g1_14, o29_1);
            }
            { const double eb = bi[277];
              o29_1 = fma(eb, g1_8, o29_1);
            }
            { const double eb = bi[278];
              o29_1 = fma(eb, g1_15, o29_1);
            }
            { const double eb = bi[279];
              o29_1 = fma(eb, g1_26, o29_1);
            }
            { const double eb = bi[280];
              o30_1 = fma(eb, g1_0, o30_1);
            }
            { const double eb = bi[281];
              o30_1 = fma(eb, g1_1, o30_1);
            }
            { const double eb = bi[282];
              o30_1 = fma(eb, g1_2, o30_1);
            }
            { const double eb = bi[283];
              o30_1 = fma(eb, g1_5, o30_1);
            }
            { const double eb = bi[284];
              o30_1 = fma(eb, g1_3, o30_1);
            }
            { const double eb = bi[285];
              o30_1 = fma(eb, g1_7, o30_1);
            }
            { const double eb = bi[286];
              o30_1 = fma(eb, g1_8, o30_1);
            }
            { const double eb = bi[287];
              o30_1 = fma(eb, g1_15, o30_1);
            }
            { const double eb = bi[288];
              o30_1 = fma(eb, g1_9, o30_1);
            }
            { const double eb = bi[289];
              o30_1 = fma(eb, g1_17, o30_1);
            }
            { const double eb = bi[290];
              o30_1 = fma(eb, g1_18, o30_1);
            }
            { const double eb = bi[291];
              o30_1 = fma(eb, g1_30, o30_1);
            }
            { const double eb = bi[292];
              o31_1 = fma(eb, g1_0, o31_1);
            }
            { const double eb = bi[293];
              o31_1 = fma(eb, g1_1, o31_1);
            }
            { const double eb = bi[294];
              o31_1 = fma(eb, g1_2, o31_1);
            }
            { const double eb = bi[295];
              o31_1 = fma(eb, g1_5, o31_1);
            }
            { const double eb = bi[296];
              o31_1 = fma(eb, g1_6, o31_1);
            }
            { const double eb = bi[297];
              o31_1 = fma(eb, g1_12, o31_1);
            }
            { const double eb = bi[298];
              o31_1 = fma(eb, g1_13, o31_1);
            }
            { const double eb = bi[299];
              o31_1 = fma(eb, g1_23, o31_1);
            }
            { const double eb = bi[300];
              o32_1 = fma(eb, g1_0, o32_1);
            }
            { const double eb = bi[301];
              o32_1 = fma(eb, g1_1, o32_1);
            }
            { const double eb = bi[302];
              o32_1 = fma(eb, g1_4, o32_1);
            }
            { const double eb = bi[303];
              o32_1 = fma(eb, g1_10, o32_1);
            }
            { const double eb = bi[304];
              o32_1 = fma(eb, g1_2, o32_1);
            }
            { const double eb = bi[305];
              o32_1 = fma(eb, g1_5, o32_1);
            }
            { const double eb = bi[306];
              o32_1 = fma(eb, g1_11, o32_1);
            }
            { const double eb = bi[307];
              o32_1 = fma(eb, g1_21, o32_1);
            }
            { const double eb = bi[308];
              o33_1 = fma(eb, g1_0, o33_1);
            }
            { const double eb = bi[309];
              o33_1 = fma(eb, g1_1, o33_1);
            }
            { const double eb = bi[310];
              o33_1 = fma(eb, g1_2, o33_1);
            }
            { const double eb = bi[311];
              o33_1 = fma(eb, g1_5, o33_1);
            }
            { const double eb = bi[312];
              o33_1 = fma(eb, g1_6, o33_1);
            }
            { const double eb = bi[313];
              o33_1 = fma(eb, g1_12, o33_1);
            }
            { const double eb = bi[314];
              o33_1 = fma(eb, g1_3, o33_1);
            }
            { const double eb = bi[315];
              o33_1 = fma(eb, g1_7, o33_1);
            }
            { const double eb = bi[316];
              o33_1 = fma(eb, g1_8, o33_1);
            }
            { const double eb = bi[317];
              o33_1 = fma(eb, g1_15, o33_1);
            }
            { const double eb = bi[318];
              o33_1 = fma(eb, g1_16, o33_1);
            }
            { const double eb = bi[319];
              o33_1 = fma(eb, g1_27, o33_1);
            }
            { const double eb = bi[320];
              o34_1 = fma(eb, g1_0, o34_1);
            }
            { const double eb = bi[321];
              o34_1 = fma(eb, g1_1, o34_1);
            }
            { const double eb = bi[322];
              o34_1 = fma(eb, g1_4, o34_1);
            }
            { const double eb = bi[323];
              o34_1 = fma(eb, g1_2, o34_1);
            }
            { const double eb = bi[324];
              o34_1 = fma(eb, g1_5, o34_1);
            }
            { const double eb = bi[325];
              o34_1 = fma(eb, g1_11, o34_1);
            }
            { const double eb = bi[326];
              o34_1 = fma(eb, g1_3, o34_1);
            }
            { const double eb = bi[327];
              o34_1 = fma(eb, g1_7, o34_1);
            }
            { const double eb = bi[328];
              o34_1 = fma(eb, g1_14, o34_1);
            }
            { const double eb = bi[329];
              o34_1 = fma(eb, g1_8, o34_1);
            }
            { const double eb = bi[330];
              o34_1 = fma(eb, g1_15, o34_1);
            }
            { const double eb = bi[331];
              o34_1 = fma(eb, g1_26, o34_1);
            }
            { const double eb = bi[332];
              o35_1 = fma(eb, g1_0, o35_1);
            }
            { const double eb = bi[333];
              o35_1 = fma(eb, g1_1, o35_1);
            }
            { const double eb = bi[334];
              o35_1 = fma(eb, g1_4, o35_1);
            }
            { const double eb = bi[335];
              o35_1 = fma(eb, g1_2, o35_1);
            }
            { const double eb = bi[336];
              o35_1 = fma(eb, g1_5, o35_1);
            }
            { const double eb = bi[337];
              o35_1 = fma(eb, g1_11, o35_1);
            }
            { const double eb = bi[338];
              o35_1 = fma(eb, g1_6, o35_1);
            }
            { const double eb = bi[339];
              o35_1 = fma(eb, g1_12, o35_1);
            }
            { const double eb = bi[340];
              o35_1 = fma(eb, g1_22, o35_1);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0);
            o1_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 0);
            o2_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 0);
            o3_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 0);
            o4_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 1, fJ + 0);
            o5_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 1, fJ + 0);
            o6_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0);
            o7_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 0);
            o8_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 0);
            o9_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 0);
            o10_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 1, fJ + 0);
            o11_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 1, fJ + 0);
            o12_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0);
            o13_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 0);
            o14_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 0);
            o15_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 0);
            o16_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 1, fJ + 0);
            o17_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 1, fJ + 0);
            o18_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0);
            o19_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 0);
            o20_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 0);
            o21_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 0);
            o22_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 1, fJ + 0);
            o23_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 1, fJ + 0);
            o24_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0);
            o25_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 0);
            o26_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 0);
            o27_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 0);
            o28_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 1, fJ + 0);
            o29_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 1, fJ + 0);
            o30_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0);
            o31_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 0);
            o32_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 0);
            o33_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 0);
            o34_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 1, fJ + 0);
            o35_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 1, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o1_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o2_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o3_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o4_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o5_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o6_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o7_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o8_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o9_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o10_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o11_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o12_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o13_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o14_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o15_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o16_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o17_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o18_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o19_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o20_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o21_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o22_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o23_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o24_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o25_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o26_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o27_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o28_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o29_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o30_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o31_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o32_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o33_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o34_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o35_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 1, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk1 = PT[(fI + 1) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 0) * N + fQ + 4];
            const double ptb5 = PT[(fP + 0) * N + fQ + 5];
            const double ptb6 = PT[(fP + 1) * N + fQ + 0];
            const double ptb7 = PT[(fP + 1) * N + fQ + 1];
            const double ptb8 = PT[(fP + 1) * N + fQ + 2];
            const double ptb9 = PT[(fP + 1) * N + fQ + 3];
            const double ptb10 = PT[(fP + 1) * N + fQ + 4];
            const double ptb11 = PT[(fP + 1) * N + fQ + 5];
            const double ptb12 = PT[(fP + 2) * N + fQ + 0];
            const double ptb13 = PT[(fP + 2) * N + fQ + 1];
            const double ptb14 = PT[(fP + 2) * N + fQ + 2];
            const double ptb15 = PT[(fP + 2) * N + fQ + 3];
            const double ptb16 = PT[(fP + 2) * N + fQ + 4];
            const double ptb17 = PT[(fP + 2) * N + fQ + 5];
            const double ptb18 = PT[(fP + 3) * N + fQ + 0];
            const double ptb19 = PT[(fP + 3) * N + fQ + 1];
            const double ptb20 = PT[(fP + 3) * N + fQ + 2];
            const double ptb21 = PT[(fP + 3) * N + fQ + 3];
            const double ptb22 = PT[(fP + 3) * N + fQ + 4];
            const double ptb23 = PT[(fP + 3) * N + fQ + 5];
            const double ptb24 = PT[(fP + 4) * N + fQ + 0];
            const double ptb25 = PT[(fP + 4) * N + fQ + 1];
            const double ptb26 = PT[(fP + 4) * N + fQ + 2];
            const double ptb27 = PT[(fP + 4) * N + fQ + 3];
            const double ptb28 = PT[(fP + 4) * N + fQ + 4];
            const double ptb29 = PT[(fP + 4) * N + fQ + 5];
            const double ptb30 = PT[(fP + 5) * N + fQ + 0];
            const double ptb31 = PT[(fP + 5) * N + fQ + 1];
            const double ptb32 = PT[(fP + 5) * N + fQ + 2];
            const double ptb33 = PT[(fP + 5) * N + fQ + 3];
            const double ptb34 = PT[(fP + 5) * N + fQ + 4];
            const double ptb35 = PT[(fP + 5) * N + fQ + 5];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd4_0 = PA[(fQ + 4) * N + fJ + 0];
            const double Abd5_0 = PA[(fQ + 5) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc3_1 = PA[(fQ + 3) * N + fI + 1];
            const double Abc4_1 = PA[(fQ + 4) * N + fI + 1];
            const double Abc5_1 = PA[(fQ + 5) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bbd4_0 = PB[(fQ + 4) * N + fJ + 0];
            const double Bbd5_0 = PB[(fQ + 5) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_1 = PB[(fQ + 0) * N + fI + 1];
            const double Bbc1_1 = PB[(fQ + 1) * N + fI + 1];
            const double Bbc2_1 = PB[(fQ + 2) * N + fI + 1];
            const double Bbc3_1 = PB[(fQ + 3) * N + fI + 1];
            const double Bbc4_1 = PB[(fQ + 4) * N + fI + 1];
            const double Bbc5_1 = PB[(fQ + 5) * N + fI + 1];
            const double Bac0_1 = PB[(fP + 0) * N + fI + 1];
            const double Bac1_1 = PB[(fP + 1) * N + fI + 1];
            const double Bac2_1 = PB[(fP + 2) * N + fI + 1];
            const double Bac3_1 = PB[(fP + 3) * N + fI + 1];
            const double Bac4_1 = PB[(fP + 4) * N + fI + 1];
            const double Bac5_1 = PB[(fP + 5) * N + fI + 1];
            jab0 += o0_1 * ptk1;
            jab1 += o1_1 * ptk1;
            jab2 += o2_1 * ptk1;
            jab3 += o3_1 * ptk1;
            jab4 += o4_1 * ptk1;
            jab5 += o5_1 * ptk1;
            jab6 += o6_1 * ptk1;
            jab7 += o7_1 * ptk1;
            jab8 += o8_1 * ptk1;
            jab9 += o9_1 * ptk1;
            jab10 += o10_1 * ptk1;
            jab11 += o11_1 * ptk1;
            jab12 += o12_1 * ptk1;
            jab13 += o13_1 * ptk1;
            jab14 += o14_1 * ptk1;
            jab15 += o15_1 * ptk1;
            jab16 += o16_1 * ptk1;
            jab17 += o17_1 * ptk1;
            jab18 += o18_1 * ptk1;
            jab19 += o19_1 * ptk1;
            jab20 += o20_1 * ptk1;
            jab21 += o21_1 * ptk1;
            jab22 += o22_1 * ptk1;
            jab23 += o23_1 * ptk1;
            jab24 += o24_1 * ptk1;
            jab25 += o25_1 * ptk1;
            jab26 += o26_1 * ptk1;
            jab27 += o27_1 * ptk1;
            jab28 += o28_1 * ptk1;
            jab29 += o29_1 * ptk1;
            jab30 += o30_1 * ptk1;
            jab31 += o31_1 * ptk1;
            jab32 += o32_1 * ptk1;
            jab33 += o33_1 * ptk1;
            jab34 += o34_1 * ptk1;
            jab35 += o35_1 * ptk1;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17 + o18_1 * ptb18 + o19_1 * ptb19 + o20_1 * ptb20 + o21_1 * ptb21 + o22_1 * ptb22 + o23_1 * ptb23 + o24_1 * ptb24 + o25_1 * ptb25 + o26_1 * ptb26 + o27_1 * ptb27 + o28_1 * ptb28 + o29_1 * ptb29 + o30_1 * ptb30 + o31_1 * ptb31 + o32_1 * ptb32 + o33_1 * ptb33 + o34_1 * ptb34 + o35_1 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Abd0_0 + o1_1 * Abd1_0 + o2_1 * Abd2_0 + o3_1 * Abd3_0 + o4_1 * Abd4_0 + o5_1 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Aad0_0 + o6_1 * Aad1_0 + o12_1 * Aad2_0 + o18_1 * Aad3_0 + o24_1 * Aad4_0 + o30_1 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_1 * Abc0_1 + o1_1 * Abc1_1 + o2_1 * Abc2_1 + o3_1 * Abc3_1 + o4_1 * Abc4_1 + o5_1 * Abc5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_1 * Aac0_1 + o6_1 * Aac1_1 + o12_1 * Aac2_1 + o18_1 * Aac3_1 + o24_1 * Aac4_1 + o30_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_1 * Aad0_0 + o7_1 * Aad1_0 + o13_1 * Aad2_0 + o19_1 * Aad3_0 + o25_1 * Aad4_0 + o31_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_1 * Aac0_1 + o7_1 * Aac1_1 + o13_1 * Aac2_1 + o19_1 * Aac3_1 + o25_1 * Aac4_1 + o31_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_1 * Aad0_0 + o8_1 * Aad1_0 + o14_1 * Aad2_0 + o20_1 * Aad3_0 + o26_1 * Aad4_0 + o32_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_1 * Aac0_1 + o8_1 * Aac1_1 + o14_1 * Aac2_1 + o20_1 * Aac3_1 + o26_1 * Aac4_1 + o32_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_1 * Aad0_0 + o9_1 * Aad1_0 + o15_1 * Aad2_0 + o21_1 * Aad3_0 + o27_1 * Aad4_0 + o33_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_1 * Aac0_1 + o9_1 * Aac1_1 + o15_1 * Aac2_1 + o21_1 * Aac3_1 + o27_1 * Aac4_1 + o33_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 1, deg * (o4_1 * Aad0_0 + o10_1 * Aad1_0 + o16_1 * Aad2_0 + o22_1 * Aad3_0 + o28_1 * Aad4_0 + o34_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_1 * Aac0_1 + o10_1 * Aac1_1 + o16_1 * Aac2_1 + o22_1 * Aac3_1 + o28_1 * Aac4_1 + o34_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 1, deg * (o5_1 * Aad0_0 + o11_1 * Aad1_0 + o17_1 * Aad2_0 + o23_1 * Aad3_0 + o29_1 * Aad4_0 + o35_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_1 * Aac0_1 + o11_1 * Aac1_1 + o17_1 * Aac2_1 + o23_1 * Aac3_1 + o29_1 * Aac4_1 + o35_1 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o6_1 * Abd0_0 + o7_1 * Abd1_0 + o8_1 * Abd2_0 + o9_1 * Abd3_0 + o10_1 * Abd4_0 + o11_1 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_1 * Abc0_1 + o7_1 * Abc1_1 + o8_1 * Abc2_1 + o9_1 * Abc3_1 + o10_1 * Abc4_1 + o11_1 * Abc5_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o12_1 * Abd0_0 + o13_1 * Abd1_0 + o14_1 * Abd2_0 + o15_1 * Abd3_0 + o16_1 * Abd4_0 + o17_1 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_1 * Abc0_1 + o13_1 * Abc1_1 + o14_1 * Abc2_1 + o15_1 * Abc3_1 + o16_1 * Abc4_1 + o17_1 * Abc5_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o18_1 * Abd0_0 + o19_1 * Abd1_0 + o20_1 * Abd2_0 + o21_1 * Abd3_0 + o22_1 * Abd4_0 + o23_1 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_1 * Abc0_1 + o19_1 * Abc1_1 + o20_1 * Abc2_1 + o21_1 * Abc3_1 + o22_1 * Abc4_1 + o23_1 * Abc5_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o24_1 * Abd0_0 + o25_1 * Abd1_0 + o26_1 * Abd2_0 + o27_1 * Abd3_0 + o28_1 * Abd4_0 + o29_1 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_1 * Abc0_1 + o25_1 * Abc1_1 + o26_1 * Abc2_1 + o27_1 * Abc3_1 + o28_1 * Abc4_1 + o29_1 * Abc5_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o30_1 * Abd0_0 + o31_1 * Abd1_0 + o32_1 * Abd2_0 + o33_1 * Abd3_0 + o34_1 * Abd4_0 + o35_1 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_1 * Abc0_1 + o31_1 * Abc1_1 + o32_1 * Abc2_1 + o33_1 * Abc3_1 + o34_1 * Abc4_1 + o35_1 * Abc5_1));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Bbd0_0 + o1_1 * Bbd1_0 + o2_1 * Bbd2_0 + o3_1 * Bbd3_0 + o4_1 * Bbd4_0 + o5_1 * Bbd5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Bad0_0 + o6_1 * Bad1_0 + o12_1 * Bad2_0 + o18_1 * Bad3_0 + o24_1 * Bad4_0 + o30_1 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_1 * Bbc0_1 + o1_1 * Bbc1_1 + o2_1 * Bbc2_1 + o3_1 * Bbc3_1 + o4_1 * Bbc4_1 + o5_1 * Bbc5_1));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_1 * Bac0_1 + o6_1 * Bac1_1 + o12_1 * Bac2_1 + o18_1 * Bac3_1 + o24_1 * Bac4_1 + o30_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 1, deg * (o1_1 * Bad0_0 + o7_1 * Bad1_0 + o13_1 * Bad2_0 + o19_1 * Bad3_0 + o25_1 * Bad4_0 + o31_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_1 * Bac0_1 + o7_1 * Bac1_1 + o13_1 * Bac2_1 + o19_1 * Bac3_1 + o25_1 * Bac4_1 + o31_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 1, deg * (o2_1 * Bad0_0 + o8_1 * Bad1_0 + o14_1 * Bad2_0 + o20_1 * Bad3_0 + o26_1 * Bad4_0 + o32_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_1 * Bac0_1 + o8_1 * Bac1_1 + o14_1 * Bac2_1 + o20_1 * Bac3_1 + o26_1 * Bac4_1 + o32_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 1, deg * (o3_1 * Bad0_0 + o9_1 * Bad1_0 + o15_1 * Bad2_0 + o21_1 * Bad3_0 + o27_1 * Bad4_0 + o33_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_1 * Bac0_1 + o9_1 * Bac1_1 + o15_1 * Bac2_1 + o21_1 * Bac3_1 + o27_1 * Bac4_1 + o33_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 4) * N + fI + 1, deg * (o4_1 * Bad0_0 + o10_1 * Bad1_0 + o16_1 * Bad2_0 + o22_1 * Bad3_0 + o28_1 * Bad4_0 + o34_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fJ + 0, deg * (o4_1 * Bac0_1 + o10_1 * Bac1_1 + o16_1 * Bac2_1 + o22_1 * Bac3_1 + o28_1 * Bac4_1 + o34_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 5) * N + fI + 1, deg * (o5_1 * Bad0_0 + o11_1 * Bad1_0 + o17_1 * Bad2_0 + o23_1 * Bad3_0 + o29_1 * Bad4_0 + o35_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fJ + 0, deg * (o5_1 * Bac0_1 + o11_1 * Bac1_1 + o17_1 * Bac2_1 + o23_1 * Bac3_1 + o29_1 * Bac4_1 + o35_1 * Bac5_1));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o6_1 * Bbd0_0 + o7_1 * Bbd1_0 + o8_1 * Bbd2_0 + o9_1 * Bbd3_0 + o10_1 * Bbd4_0 + o11_1 * Bbd5_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o6_1 * Bbc0_1 + o7_1 * Bbc1_1 + o8_1 * Bbc2_1 + o9_1 * Bbc3_1 + o10_1 * Bbc4_1 + o11_1 * Bbc5_1));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o12_1 * Bbd0_0 + o13_1 * Bbd1_0 + o14_1 * Bbd2_0 + o15_1 * Bbd3_0 + o16_1 * Bbd4_0 + o17_1 * Bbd5_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o12_1 * Bbc0_1 + o13_1 * Bbc1_1 + o14_1 * Bbc2_1 + o15_1 * Bbc3_1 + o16_1 * Bbc4_1 + o17_1 * Bbc5_1));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o18_1 * Bbd0_0 + o19_1 * Bbd1_0 + o20_1 * Bbd2_0 + o21_1 * Bbd3_0 + o22_1 * Bbd4_0 + o23_1 * Bbd5_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o18_1 * Bbc0_1 + o19_1 * Bbc1_1 + o20_1 * Bbc2_1 + o21_1 * Bbc3_1 + o22_1 * Bbc4_1 + o23_1 * Bbc5_1));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o24_1 * Bbd0_0 + o25_1 * Bbd1_0 + o26_1 * Bbd2_0 + o27_1 * Bbd3_0 + o28_1 * Bbd4_0 + o29_1 * Bbd5_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o24_1 * Bbc0_1 + o25_1 * Bbc1_1 + o26_1 * Bbc2_1 + o27_1 * Bbc3_1 + o28_1 * Bbc4_1 + o29_1 * Bbc5_1));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o30_1 * Bbd0_0 + o31_1 * Bbd1_0 + o32_1 * Bbd2_0 + o33_1 * Bbd3_0 + o34_1 * Bbd4_0 + o35_1 * Bbd5_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o30_1 * Bbc0_1 + o31_1 * Bbc1_1 + o32_1 * Bbc2_1 + o33_1 * Bbc3_1 + o34_1 * Bbc4_1 + o35_1 * Bbc5_1));
          }
        } break;
        case 2: {  // ket functions [2]
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
          double o24_2 = 0;
          double o25_2 = 0;
          double o26_2 = 0;
          double o27_2 = 0;
          double o28_2 = 0;
          double o29_2 = 0;
          double o30_2 = 0;
          double o31_2 = 0;
          double o32_2 = 0;
          double o33_2 = 0;
          double o34_2 = 0;
          double o35_2 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 341;
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
            double g2_20 = 0;
            double g2_21 = 0;
            double g2_22 = 0;
            double g2_23 = 0;
            double g2_24 = 0;
            double g2_25 = 0;
            double g2_26 = 0;
            double g2_27 = 0;
            double g2_28 = 0;
            double g2_29 = 0;
            double g2_30 = 0;
            double g2_31 = 0;
            double g2_32 = 0;
            double g2_33 = 0;
            double g2_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 26 * kS;
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
              const double ek2_0 = kj[11 * kS];
              const double ek2_1 = -kj[12 * kS];
              const double ek2_2 = kj[13 * kS];
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
              g2_0 = fma(ek2_2, r0_0_0_2, g2_0);
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
              g2_1 = fma(ek2_2, r0_0_0_3, g2_1);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g2_11 = fma(ek2_0, r0_0_1_2, g2_11);
              g2_5 = fma(ek2_1, r0_0_1_2, g2_5);
              g2_2 = fma(ek2_2, r0_0_1_2, g2_2);
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
              g2_3 = fma(ek2_2, r0_1_0_2, g2_3);
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
              g2_20 = fma(ek2_0, r0_0_0_4, g2_20);
              g2_10 = fma(ek2_1, r0_0_0_4, g2_10);
              g2_4 = fma(ek2_2, r0_0_0_4, g2_4);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g2_21 = fma(ek2_0, r0_0_1_3, g2_21);
              g2_11 = fma(ek2_1, r0_0_1_3, g2_11);
              g2_5 = fma(ek2_2, r0_0_1_3, g2_5);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g2_22 = fma(ek2_0, r0_0_2_2, g2_22);
              g2_12 = fma(ek2_1, r0_0_2_2, g2_12);
              g2_6 = fma(ek2_2, r0_0_2_2, g2_6);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g2_23 = fma(ek2_0, r0_0_3_1, g2_23);
              g2_13 = fma(ek2_1, r0_0_3_1, g2_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g2_24 = fma(ek2_0, r0_0_4_0, g2_24);
              const double r0_1_0_3 = X * r1_0_0_3;
              g2_25 = fma(ek2_0, r0_1_0_3, g2_25);
              g2_14 = fma(ek2_1, r0_1_0_3, g2_14);
              g2_7 = fma(ek2_2, r0_1_0_3, g2_7);
              const double r0_1_1_2 = X * r1_0_1_2;
              g2_26 = fma(ek2_0, r0_1_1_2, g2_26);
              g2_15 = fma(ek2_1, r0_1_1_2, g2_15);
              g2_8 = fma(ek2_2, r0_1_1_2, g2_8);
              const double r0_1_2_1 = X * r1_0_2_1;
              g2_27 = fma(ek2_0, r0_1_2_1, g2_27);
              g2_16 = fma(ek2_1, r0_1_2_1, g2_16);
              const double r0_1_3_0 = X * r1_0_3_0;
              g2_28 = fma(ek2_0, r0_1_3_0, g2_28);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g2_29 = fma(ek2_0, r0_2_0_2, g2_29);
              g2_17 = fma(ek2_1, r0_2_0_2, g2_17);
              g2_9 = fma(ek2_2, r0_2_0_2, g2_9);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g2_30 = fma(ek2_0, r0_2_1_1, g2_30);
              g2_18 = fma(ek2_1, r0_2_1_1, g2_18);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g2_31 = fma(ek2_0, r0_2_2_0, g2_31);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g2_32 = fma(ek2_0, r0_3_0_1, g2_32);
              g2_19 = fma(ek2_1, r0_3_0_1, g2_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g2_33 = fma(ek2_0, r0_3_1_0, g2_33);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g2_34 = fma(ek2_0, r0_4_0_0, g2_34);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g2_20 = fma(ek2_1, r0_0_0_5, g2_20);
              g2_10 = fma(ek2_2, r0_0_0_5, g2_10);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g2_21 = fma(ek2_1, r0_0_1_4, g2_21);
              g2_11 = fma(ek2_2, r0_0_1_4, g2_11);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g2_22 = fma(ek2_1, r0_0_2_3, g2_22);
              g2_12 = fma(ek2_2, r0_0_2_3, g2_12);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g2_23 = fma(ek2_1, r0_0_3_2, g2_23);
              g2_13 = fma(ek2_2, r0_0_3_2, g2_13);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g2_24 = fma(ek2_1, r0_0_4_1, g2_24);
              const double r0_1_0_4 = X * r1_0_0_4;
              g2_25 = fma(ek2_1, r0_1_0_4, g2_25);
              g2_14 = fma(ek2_2, r0_1_0_4, g2_14);
              const double r0_1_1_3 = X * r1_0_1_3;
              g2_26 = fma(ek2_1, r0_1_1_3, g2_26);
              g2_15 = fma(ek2_2, r0_1_1_3, g2_15);
              const double r0_1_2_2 = X * r1_0_2_2;
              g2_27 = fma(ek2_1, r0_1_2_2, g2_27);
              g2_16 = fma(ek2_2, r0_1_2_2, g2_16);
              const double r0_1_3_1 = X * r1_0_3_1;
              g2_28 = fma(ek2_1, r0_1_3_1, g2_28);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g2_29 = fma(ek2_1, r0_2_0_3, g2_29);
              g2_17 = fma(ek2_2, r0_2_0_3, g2_17);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g2_30 = fma(ek2_1, r0_2_1_2, g2_30);
              g2_18 = fma(ek2_2, r0_2_1_2, g2_18);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g2_31 = fma(ek2_1, r0_2_2_1, g2_31);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g2_32 = fma(ek2_1, r0_3_0_2, g2_32);
              g2_19 = fma(ek2_2, r0_3_0_2, g2_19);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g2_33 = fma(ek2_1, r0_3_1_1, g2_33);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g2_34 = fma(ek2_1, r0_4_0_1, g2_34);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_0_0_6 = fma(Z, r1_0_0_5, 5.0 * r1_0_0_4);
              g2_20 = fma(ek2_2, r0_0_0_6, g2_20);
              const double r0_0_1_5 = Y * r1_0_0_5;
              g2_21 = fma(ek2_2, r0_0_1_5, g2_21);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_0_2_4 = fma(Y, r1_0_1_4, r1_0_0_4);
              g2_22 = fma(ek2_2, r0_0_2_4, g2_22);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_0_3_3 = fma(Y, r1_0_2_3, 2.0 * r1_0_1_3);
              g2_23 = fma(ek2_2, r0_0_3_3, g2_23);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_0_4_2 = fma(Y, r1_0_3_2, 3.0 * r1_0_2_2);
              g2_24 = fma(ek2_2, r0_0_4_2, g2_24);
              const double r0_1_0_5 = X * r1_0_0_5;
              g2_25 = fma(ek2_2, r0_1_0_5, g2_25);
              const double r0_1_1_4 = X * r1_0_1_4;
              g2_26 = fma(ek2_2, r0_1_1_4, g2_26);
              const double r0_1_2_3 = X * r1_0_2_3;
              g2_27 = fma(ek2_2, r0_1_2_3, g2_27);
              const double r0_1_3_2 = X * r1_0_3_2;
              g2_28 = fma(ek2_2, r0_1_3_2, g2_28);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g2_29 = fma(ek2_2, r0_2_0_4, g2_29);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g2_30 = fma(ek2_2, r0_2_1_3, g2_30);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g2_31 = fma(ek2_2, r0_2_2_2, g2_31);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g2_32 = fma(ek2_2, r0_3_0_3, g2_32);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g2_33 = fma(ek2_2, r0_3_1_2, g2_33);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g2_34 = fma(ek2_2, r0_4_0_2, g2_34);
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
              o0_2 = fma(eb, g2_19, o0_2);
            }
            { const double eb = bi[9];
              o0_2 = fma(eb, g2_34, o0_2);
            }
            { const double eb = bi[10];
              o1_2 = fma(eb, g2_0, o1_2);
            }
            { const double eb = bi[11];
              o1_2 = fma(eb, g2_2, o1_2);
            }
            { const double eb = bi[12];
              o1_2 = fma(eb, g2_6, o1_2);
            }
            { const double eb = bi[13];
              o1_2 = fma(eb, g2_3, o1_2);
            }
            { const double eb = bi[14];
              o1_2 = fma(eb, g2_8, o1_2);
            }
            { const double eb = bi[15];
              o1_2 = fma(eb, g2_16, o1_2);
            }
            { const double eb = bi[16];
              o1_2 = fma(eb, g2_9, o1_2);
            }
            { const double eb = bi[17];
              o1_2 = fma(eb, g2_18, o1_2);
            }
            { const double eb = bi[18];
              o1_2 = fma(eb, g2_31, o1_2);
            }
            { const double eb = bi[19];
              o2_2 = fma(eb, g2_0, o2_2);
            }
            { const double eb = bi[20];
              o2_2 = fma(eb, g2_1, o2_2);
            }
            { const double eb = bi[21];
              o2_2 = fma(eb, g2_4, o2_2);
            }
            { const double eb = bi[22];
              o2_2 = fma(eb, g2_3, o2_2);
            }
            { const double eb = bi[23];
              o2_2 = fma(eb, g2_7, o2_2);
            }
            { const double eb = bi[24];
              o2_2 = fma(eb, g2_14, o2_2);
            }
            { const double eb = bi[25];
              o2_2 = fma(eb, g2_9, o2_2);
            }
            { const double eb = bi[26];
              o2_2 = fma(eb, g2_17, o2_2);
            }
            { const double eb = bi[27];
              o2_2 = fma(eb, g2_29, o2_2);
            }
            { const double eb = bi[28];
              o3_2 = fma(eb, g2_0, o3_2);
            }
            { const double eb = bi[29];
              o3_2 = fma(eb, g2_2, o3_2);
            }
            { const double eb = bi[30];
              o3_2 = fma(eb, g2_3, o3_2);
            }
            { const double eb = bi[31];
              o3_2 = fma(eb, g2_8, o3_2);
            }
            { const double eb = bi[32];
              o3_2 = fma(eb, g2_9, o3_2);
            }
            { const double eb = bi[33];
              o3_2 = fma(eb, g2_18, o3_2);
            }
            { const double eb = bi[34];
              o3_2 = fma(eb, g2_19, o3_2);
            }
            { const double eb = bi[35];
              o3_2 = fma(eb, g2_33, o3_2);
            }
            { const double eb = bi[36];
              o4_2 = fma(eb, g2_0, o4_2);
            }
            { const double eb = bi[37];
              o4_2 = fma(eb, g2_1, o4_2);
            }
            { const double eb = bi[38];
              o4_2 = fma(eb, g2_3, o4_2);
            }
            { const double eb = bi[39];
              o4_2 = fma(eb, g2_7, o4_2);
            }
            { const double eb = bi[40];
              o4_2 = fma(eb, g2_9, o4_2);
            }
            { const double eb = bi[41];
              o4_2 = fma(eb, g2_17, o4_2);
            }
            { const double eb = bi[42];
              o4_2 = fma(eb, g2_19, o4_2);
            }
            { const double eb = bi[43];
              o4_2 = fma(eb, g2_32, o4_2);
            }
            { const double eb = bi[44];
              o5_2 = fma(eb, g2_0, o5_2);
            }
            { const double eb = bi[45];
              o5_2 = fma(eb, g2_1, o5_2);
            }
            { const double eb = bi[46];
              o5_2 = fma(eb, g2_2, o5_2);
            }
            { const double eb = bi[47];
              o5_2 = fma(eb, g2_5, o5_2);
            }
            { const double eb = bi[48];
              o5_2 = fma(eb, g2_3, o5_2);
            }
            { const double eb = bi[49];
              o5_2 = fma(eb, g2_7, o5_2);
            }
            { const double eb = bi[50];
              o5_2 = fma(eb, g2_8, o5_2);
            }
            { const double eb = bi[51];
              o5_2 = fma(eb, g2_15, o5_2);
            }
            { const double eb = bi[52];
              o5_2 = fma(eb, g2_9, o5_2);
            }
            { const double eb = bi[53];
              o5_2 = fma(eb, g2_17, o5_2);
            }
            { const double eb = bi[54];
              o5_2 = fma(eb, g2_18, o5_2);
            }
            { const double eb = bi[55];
              o5_2 = fma(eb, g2_30, o5_2);
            }
            { const double eb = bi[56];
              o6_2 = fma(eb, g2_0, o6_2);
            }
            { const double eb = bi[57];
              o6_2 = fma(eb, g2_2, o6_2);
            }
            { const double eb = bi[58];
              o6_2 = fma(eb, g2_6, o6_2);
            }
            { const double eb = bi[59];
              o6_2 = fma(eb, g2_3, o6_2);
            }
            { const double eb = bi[60];
              o6_2 = fma(eb, g2_8, o6_2);
            }
            { const double eb = bi[61];
              o6_2 = fma(eb, g2_16, o6_2);
            }
            { const double eb = bi[62];
              o6_2 = fma(eb, g2_9, o6_2);
            }
            { const double eb = bi[63];
              o6_2 = fma(eb, g2_18, o6_2);
            }
            { const double eb = bi[64];
              o6_2 = fma(eb, g2_31, o6_2);
            }
            { const double eb = bi[65];
              o7_2 = fma(eb, g2_0, o7_2);
            }
            { const double eb = bi[66];
              o7_2 = fma(eb, g2_2, o7_2);
            }
            { const double eb = bi[67];
              o7_2 = fma(eb, g2_6, o7_2);
            }
            { const double eb = bi[68];
              o7_2 = fma(eb, g2_13, o7_2);
            }
            { const double eb = bi[69];
              o7_2 = fma(eb, g2_24, o7_2);
            }
            { const double eb = bi[70];
              o8_2 = fma(eb, g2_0, o8_2);
            }
            { const double eb = bi[71];
              o8_2 = fma(eb, g2_1, o8_2);
            }
            { const double eb = bi[72];
              o8_2 = fma(eb, g2_4, o8_2);
            }
            { const double eb = bi[73];
              o8_2 = fma(eb, g2_2, o8_2);
            }
            { const double eb = bi[74];
              o8_2 = fma(eb, g2_5, o8_2);
            }
            { const double eb = bi[75];
              o8_2 = fma(eb, g2_11, o8_2);
            }
            { const double eb = bi[76];
              o8_2 = fma(eb, g2_6, o8_2);
            }
            { const double eb = bi[77];
              o8_2 = fma(eb, g2_12, o8_2);
            }
            { const double eb = bi[78];
              o8_2 = fma(eb, g2_22, o8_2);
            }
            { const double eb = bi[79];
              o9_2 = fma(eb, g2_0, o9_2);
            }
            { const double eb = bi[80];
              o9_2 = fma(eb, g2_2, o9_2);
            }
            { const double eb = bi[81];
              o9_2 = fma(eb, g2_6, o9_2);
            }
            { const double eb = bi[82];
              o9_2 = fma(eb, g2_13, o9_2);
            }
            { const double eb = bi[83];
              o9_2 = fma(eb, g2_3, o9_2);
            }
            { const double eb = bi[84];
              o9_2 = fma(eb, g2_8, o9_2);
            }
            { const double eb = bi[85];
              o9_2 = fma(eb, g2_16, o9_2);
            }
            { const double eb = bi[86];
              o9_2 = fma(eb, g2_28, o9_2);
            }
            { const double eb = bi[87];
              o10_2 = fma(eb, g2_0, o10_2);
            }
            { const double eb = bi[88];
              o10_2 = fma(eb, g2_1, o10_2);
            }
            { const double eb = bi[89];
              o10_2 = fma(eb, g2_2, o10_2);
            }
            { const double eb = bi[90];
              o10_2 = fma(eb, g2_5, o10_2);
            }
            { const double eb = bi[91];
              o10_2 = fma(eb, g2_6, o10_2);
            }
            { const double eb = bi[92];
              o10_2 = fma(eb, g2_12, o10_2);
            }
            { const double eb = bi[93];
              o10_2 = fma(eb, g2_3, o10_2);
            }
            { const double eb = bi[94];
              o10_2 = fma(eb, g2_7, o10_2);
            }
            { const double eb = bi[95];
              o10_2 = fma(eb, g2_8, o10_2);
            }
            { const double eb = bi[96];
              o10_2 = fma(eb, g2_15, o10_2);
            }
            { const double eb = bi[97];
              o10_2 = fma(eb, g2_16, o10_2);
            }
            { const double eb = bi[98];
              o10_2 = fma(eb, g2_27, o10_2);
            }
            { const double eb = bi[99];
              o11_2 = fma(eb, g2_0, o11_2);
            }
            { const double eb = bi[100];
              o11_2 = fma(eb, g2_1, o11_2);
            }
            { const double eb = bi[101];
              o11_2 = fma(eb, g2_2, o11_2);
            }
            { const double eb = bi[102];
              o11_2 = fma(eb, g2_5, o11_2);
            }
            { const double eb = bi[103];
              o11_2 = fma(eb, g2_6, o11_2);
            }
            { const double eb = bi[104];
              o11_2 = fma(eb, g2_12, o11_2);
            }
            { const double eb = bi[105];
              o11_2 = fma(eb, g2_13, o11_2);
            }
            { const double eb = bi[106];
              o11_2 = fma(eb, g2_23, o11_2);
            }
            { const double eb = bi[107];
              o12_2 = fma(eb, g2_0, o12_2);
            }
            { const double eb = bi[108];
              o12_2 = fma(eb, g2_1, o12_2);
            }
            { const double eb = bi[109];
              o12_2 = fma(eb, g2_4, o12_2);
            }
            { const double eb = bi[110];
              o12_2 = fma(eb, g2_3, o12_2);
            }
            { const double eb = bi[111];
              o12_2 = fma(eb, g2_7, o12_2);
            }
            { const double eb = bi[112];
              o12_2 = fma(eb, g2_14, o12_2);
            }
            { const double eb = bi[113];
              o12_2 = fma(eb, g2_9, o12_2);
            }
            { const double eb = bi[114];
              o12_2 = fma(eb, g2_17, o12_2);
            }
            { const double eb = bi[115];
              o12_2 = fma(eb, g2_29, o12_2);
            }
            { const double eb = bi[116];
              o13_2 = fma(eb, g2_0, o13_2);
            }
            { const double eb = bi[117];
              o13_2 = fma(eb, g2_1, o13_2);
            }
            { const double eb = bi[118];
              o13_2 = fma(eb, g2_4, o13_2);
            }
            { const double eb = bi[119];
              o13_2 = fma(eb, g2_2, o13_2);
            }
            { const double eb = bi[120];
              o13_2 = fma(eb, g2_5, o13_2);
            }
            { const double eb = bi[121];
              o13_2 = fma(eb, g2_11, o13_2);
            }
            { const double eb = bi[122];
              o13_2 = fma(eb, g2_6, o13_2);
            }
            { const double eb = bi[123];
              o13_2 = fma(eb, g2_12, o13_2);
            }
            { const double eb = bi[124];
              o13_2 = fma(eb, g2_22, o13_2);
            }
            { const double eb = bi[125];
              o14_2 = fma(eb, g2_0, o14_2);
            }
            { const double eb = bi[126];
              o14_2 = fma(eb, g2_1, o14_2);
            }
            { const double eb = bi[127];
              o14_2 = fma(eb, g2_4, o14_2);
            }
            { const double eb = bi[128];
              o14_2 = fma(eb, g2_10, o14_2);
            }
            { const double eb = bi[129];
              o14_2 = fma(eb, g2_20, o14_2);
            }
            { const double eb = bi[130];
              o15_2 = fma(eb, g2_0, o15_2);
            }
            { const double eb = bi[131];
              o15_2 = fma(eb, g2_1, o15_2);
            }
            { const double eb = bi[132];
              o15_2 = fma(eb, g2_4, o15_2);
            }
            { const double eb = bi[133];
              o15_2 = fma(eb, g2_2, o15_2);
            }
            { const double eb = bi[134];
              o15_2 = fma(eb, g2_5, o15_2);
            }
            { const double eb = bi[135];
              o15_2 = fma(eb, g2_11, o15_2);
            }
            { const double eb = bi[136];
              o15_2 = fma(eb, g2_3, o15_2);
            }
            { const double eb = bi[137];
              o15_2 = fma(eb, g2_7, o15_2);
            }
            { const double eb = bi[138];
              o15_2 = fma(eb, g2_14, o15_2);
            }
            { const double eb = bi[139];
              o15_2 = fma(eb, g2_8, o15_2);
            }
            { const double eb = bi[140];
              o15_2 = fma(eb, g2_15, o15_2);
            }
            { const double eb = bi[141];
              o15_2 = fma(eb, g2_26, o15_2);
            }
            { const double eb = bi[142];
              o16_2 = fma(eb, g2_0, o16_2);
            }
            { const double eb = bi[143];
              o16_2 = fma(eb, g2_1, o16_2);
            }
            { const double eb = bi[144];
              o16_2 = fma(eb, g2_4, o16_2);
            }
            { const double eb = bi[145];
              o16_2 = fma(eb, g2_10, o16_2);
            }
            { const double eb = bi[146];
              o16_2 = fma(eb, g2_3, o16_2);
            }
            { const double eb = bi[147];
              o16_2 = fma(eb, g2_7, o16_2);
            }
            { const double eb = bi[148];
              o16_2 = fma(eb, g2_14, o16_2);
            }
            { const double eb = bi[149];
              o16_2 = fma(eb, g2_25, o16_2);
            }
            { const double eb = bi[150];
              o17_2 = fma(eb, g2_0, o17_2);
            }
            { const double eb = bi[151];
              o17_2 = fma(eb, g2_1, o17_2);
            }
            { const double eb = bi[152];
              o17_2 = fma(eb, g2_4, o17_2);
            }
            { const double eb = bi[153];
              o17_2 = fma(eb, g2_10, o17_2);
            }
            { const double eb = bi[154];
              o17_2 = fma(eb, g2_2, o17_2);
            }
            { const double eb = bi[155];
              o17_2 = fma(eb, g2_5, o17_2);
            }
            { const double eb = bi[156];
              o17_2 = fma(eb, g2_11, o17_2);
            }
            { const double eb = bi[157];
              o17_2 = fma(eb, g2_21, o17_2);
            }
            { const double eb = bi[158];
              o18_2 = fma(eb, g2_0, o18_2);
            }
            { const double eb = bi[159];
              o18_2 = fma(eb, g2_2, o18_2);
            }
            { const double eb = bi[160];
              o18_2 = fma(eb, g2_3, o18_2);
            }
            { const double eb = bi[161];
              o18_2 = fma(eb, g2_8, o18_2);
            }
            { const double eb = bi[162];
              o18_2 = fma(eb, g2_9, o18_2);
            }
            { const double eb = bi[163];
              o18_2 = fma(eb, g2_18, o18_2);
            }
            { const double eb = bi[164];
              o18_2 = fma(eb, g2_19, o18_2);
            }
            { const double eb = bi[165];
              o18_2 = fma(eb, g2_33, o18_2);
            }
            { const double eb = bi[166];
              o19_2 = fma(eb, g2_0, o19_2);
            }
            { const double eb = bi[167];
              o19_2 = fma(eb, g2_2, o19_2);
            }
            { const double eb = bi[168];
              o19_2 = fma(eb, g2_6, o19_2);
            }
            { const double eb = bi[169];
              o19_2 = fma(eb, g2_13, o19_2);
            }
            { const double eb = bi[170];
              o19_2 = fma(eb, g2_3, o19_2);
            }
            { const double eb = bi[171];
              o19_2 = fma(eb, g2_8, o19_2);
            }
            { const double eb = bi[172];
              o19_2 = fma(eb, g2_16, o19_2);
            }
            { const double eb = bi[173];
              o19_2 = fma(eb, g2_28, o19_2);
            }
            { const double eb = bi[174];
              o20_2 = fma(eb, g2_0, o20_2);
            }
            { const double eb = bi[175];
              o20_2 = fma(eb, g2_1, o20_2);
            }
            { const double eb = bi[176];
              o20_2 = fma(eb, g2_4, o20_2);
            }
            { const double eb = bi[177];
              o20_2 = fma(eb, g2_2, o20_2);
            }
            { const double eb = bi[178];
              o20_2 = fma(eb, g2_5, o20_2);
            }
            { const double eb = bi[179];
              o20_2 = fma(eb, g2_11, o20_2);
            }
            { const double eb = bi[180];
              o20_2 = fma(eb, g2_3, o20_2);
            }
            { const double eb = bi[181];
              o20_2 = fma(eb, g2_7, o20_2);
            }
            { const double eb = bi[182];
              o20_2 = fma(eb, g2_14, o20_2);
            }
            { const double eb = bi[183];
              o20_2 = fma(eb, g2_8, o20_2);
            }
            { const double eb = bi[184];
              o20_2 = fma(eb, g2_15, o20_2);
            }
            { const double eb = bi[185];
              o20_2 = fma(eb, g2_26, o20_2);
            }
            { const double eb = bi[186];
              o21_2 = fma(eb, g2_0, o21_2);
            }
            { const double eb = bi[187];
              o21_2 = fma(eb, g2_2, o21_2);
            }
            { const double eb = bi[188];
              o21_2 = fma(eb, g2_6, o21_2);
            }
            { const double eb = bi[189];
              o21_2 = fma(eb, g2_3, o21_2);
            }
            { const double eb = bi[190];
              o21_2 = fma(eb, g2_8, o21_2);
            }
            { const double eb = bi[191];
              o21_2 = fma(eb, g2_16, o21_2);
            }
            { const double eb = bi[192];
              o21_2 = fma(eb, g2_9, o21_2);
            }
            { const double eb = bi[193];
              o21_2 = fma(eb, g2_18, o21_2);
            }
            { const double eb = bi[194];
              o21_2 = fma(eb, g2_31, o21_2);
            }
            { const double eb = bi[195];
              o22_2 = fma(eb, g2_0, o22_2);
            }
            { const double eb = bi[196];
              o22_2 = fma(eb, g2_1, o22_2);
            }
            { const double eb = bi[197];
              o22_2 = fma(eb, g2_2, o22_2);
            }
            { const double eb = bi[198];
              o22_2 = fma(eb, g2_5, o22_2);
            }
            { const double eb = bi[199];
              o22_2 = fma(eb, g2_3, o22_2);
            }
            { const double eb = bi[200];
              o22_2 = fma(eb, g2_7, o22_2);
            }
            { const double eb = bi[201];
              o22_2 = fma(eb, g2_8, o22_2);
            }
            { const double eb = bi[202];
              o22_2 = fma(eb, g2_15, o22_2);
            }
            { const double eb = bi[203];
              o22_2 = fma(eb, g2_9, o22_2);
            }
            { const double eb = bi[204];
              o22_2 = fma(eb, g2_17, o22_2);
            }
            { const double eb = bi[205];
              o22_2 = fma(eb, g2_18, o22_2);
            }
            { const double eb = bi[206];
              o22_2 = fma(eb, g2_30, o22_2);
            }
            { const double eb = bi[207];
              o23_2 = fma(eb, g2_0, o23_2);
            }
            { const double eb = bi[208];
              o23_2 = fma(eb, g2_1, o23_2);
            }
            { const double eb = bi[209];
              o23_2 = fma(eb, g2_2, o23_2);
            }
            { const double eb = bi[210];
              o23_2 = fma(eb, g2_5, o23_2);
            }
            { const double eb = bi[211];
              o23_2 = fma(eb, g2_6, o23_2);
            }
            { const double eb = bi[212];
              o23_2 = fma(eb, g2_12, o23_2);
            }
            { const double eb = bi[213];
              o23_2 = fma(eb, g2_3, o23_2);
            }
            { const double eb = bi[214];
              o23_2 = fma(eb, g2_7, o23_2);
            }
            { const double eb = bi[215];
              o23_2 = fma(eb, g2_8, o23_2);
            }
            { const double eb = bi[216];
              o23_2 = fma(eb, g2_15, o23_2);
            }
            { const double eb = bi[217];
              o23_2 = fma(eb, g2_16, o23_2);
            }
            { const double eb = bi[218];
              o23_2 = fma(eb, g2_27, o23_2);
            }
            { const double eb = bi[219];
              o24_2 = fma(eb, g2_0, o24_2);
            }
            { const double eb = bi[220];
              o24_2 = fma(eb, g2_1, o24_2);
            }
            { const double eb = bi[221];
              o24_2 = fma(eb, g2_3, o24_2);
            }
            { const double eb = bi[222];
              o24_2 = fma(eb, g2_7, o24_2);
            }
            { const double eb = bi[223];
              o24_2 = fma(eb, g2_9, o24_2);
            }
            { const double eb = bi[224];
              o24_2 = fma(eb, g2_17, o24_2);
            }
            { const double eb = bi[225];
              o24_2 = fma(eb, g2_19, o24_2);
            }
            { const double eb = bi[226];
              o24_2 = fma(eb, g2_32, o24_2);
            }
            { const double eb = bi[227];
              o25_2 = fma(eb, g2_0, o25_2);
            }
            { const double eb = bi[228];
              o25_2 = fma(eb, g2_1, o25_2);
            }
            { const double eb = bi[229];
              o25_2 = fma(eb, g2_2, o25_2);
            }
            { const double eb = bi[230];
              o25_2 = fma(eb, g2_5, o25_2);
            }
            { const double eb = bi[231];
              o25_2 = fma(eb, g2_6, o25_2);
            }
            { const double eb = bi[232];
              o25_2 = fma(eb, g2_12, o25_2);
            }
            { const double eb = bi[233];
              o25_2 = fma(eb, g2_3, o25_2);
            }
            { const double eb = bi[234];
              o25_2 = fma(eb, g2_7, o25_2);
            }
            { const double eb = bi[235];
              o25_2 = fma(eb, g2_8, o25_2);
            }
            { const double eb = bi[236];
              o25_2 = fma(eb, g2_15, o25_2);
            }
            { const double eb = bi[237];
              o25_2 = fma(eb, g2_16, o25_2);
            }
            { const double eb = bi[238];
              o25_2 = fma(eb, g2_27, o25_2);
            }
            { const double eb = bi[239];
              o26_2 = fma(eb, g2_0, o26_2);
            }
            { const double eb = bi[240];
              o26_2 = fma(eb, g2_1, o26_2);
            }
            { const double eb = bi[241];
              o26_2 = fma(eb, g2_4, o26_2);
            }
            { const double eb = bi[242];
              o26_2 = fma(eb, g2_10, o26_2);
            }
            { const double eb = bi[243];
              o26_2 = fma(eb, g2_3, o26_2);
            }
            { const double eb = bi[244];
              o26_2 = fma(eb, g2_7, o26_2);
            }
            { const double eb = bi[245];
              o26_2 = fma(eb, g2_14, o26_2);
            }
            { const double eb = bi[246];
              o26_2 = fma(eb, g2_25, o26_2);
            }
            { const double eb = bi[247];
              o27_2 = fma(eb, g2_0, o27_2);
            }
            { const double eb = bi[248];
              o27_2 = fma(eb, g2_1, o27_2);
            }
            { const double eb = bi[249];
              o27_2 = fma(eb, g2_2, o27_2);
            }
            { const double eb = bi[250];
              o27_2 = fma(eb, g2_5, o27_2);
            }
            { const double eb = bi[251];
              o27_2 = fma(eb, g2_3, o27_2);
            }
            { const double eb = bi[252];
              o27_2 = fma(eb, g2_7, o27_2);
            }
            { const double eb = bi[253];
              o27_2 = fma(eb, g2_8, o27_2);
            }
            { const double eb = bi[254];
              o27_2 = fma(eb, g2_15, o27_2);
            }
            { const double eb = bi[255];
              o27_2 = fma(eb, g2_9, o27_2);
            }
            { const double eb = bi[256];
              o27_2 = fma(eb, g2_17, o27_2);
            }
            { const double eb = bi[257];
              o27_2 = fma(eb, g2_18, o27_2);
            }
            { const double eb = bi[258];
              o27_2 = fma(eb, g2_30, o27_2);
            }
            { const double eb = bi[259];
              o28_2 = fma(eb, g2_0, o28_2);
            }
            { const double eb = bi[260];
              o28_2 = fma(eb, g2_1, o28_2);
            }
            { const double eb = bi[261];
              o28_2 = fma(eb, g2_4, o28_2);
            }
            { const double eb = bi[262];
              o28_2 = fma(eb, g2_3, o28_2);
            }
            { const double eb = bi[263];
              o28_2 = fma(eb, g2_7, o28_2);
            }
            { const double eb = bi[264];
              o28_2 = fma(eb, g2_14, o28_2);
            }
            { const double eb = bi[265];
              o28_2 = fma(eb, g2_9, o28_2);
            }
            { const double eb = bi[266];
              o28_2 = fma(eb, g2_17, o28_2);
            }
            { const double eb = bi[267];
              o28_2 = fma(eb, g2_29, o28_2);
            }
            { const double eb = bi[268];
              o29_2 = fma(eb, g2_0, o29_2);
            }
            { const double eb = bi[269];
              o29_2 = fma(eb, g2_1, o29_2);
            }
            { const double eb = bi[270];
              o29_2 = fma(eb, g2_4, o29_2);
            }
            { const double eb = bi[271];
              o29_2 = fma(eb, g2_2, o29_2);
            }
            { const double eb = bi[272];
              o29_2 = fma(eb, g2_5, o29_2);
            }
            { const double eb = bi[273];
              o29_2 = fma(eb, g2_11, o29_2);
            }
            { const double eb = bi[274];
              o29_2 = fma(eb, g2_3, o29_2);
            }
            { const double eb = bi[275];
              o29_2 = fma(eb, g2_7, o29_2);
            }
            { const double eb = bi[276];
              o29_2 = fma(eb, g2_14, o29_2);
            }
            { const double eb = bi[277];
              o29_2 = fma(eb, g2_8, o29_2);
            }
            { const double eb = bi[278];
              o29_2 = fma(eb, g2_15, o29_2);
            }
            { const double eb = bi[279];
              o29_2 = fma(eb, g2_26, o29_2);
            }
            { const double eb = bi[280];
              o30_2 = fma(eb, g2_0, o30_2);
            }
            { const double eb = bi[281];
              o30_2 = fma(eb, g2_1, o30_2);
            }
            { const double eb = bi[282];
              o30_2 = fma(eb, g2_2, o30_2);
            }
            { const double eb = bi[283];
              o30_2 = fma(eb, g2_5, o30_2);
            }
            { const double eb = bi[284];
              o30_2 = fma(eb, g2_3, o30_2);
            }
            { const double eb = bi[285];
              o30_2 = fma(eb, g2_7, o30_2);
            }
            { const double eb = bi[286];
              o30_2 = fma(eb, g2_8, o30_2);
            }
            { const double eb = bi[287];
              o30_2 = fma(eb, g2_15, o30_2);
            }
            { const double eb = bi[288];
              o30_2 = fma(eb, g2_9, o30_2);
            }
            { const double eb = bi[289];
              o30_2 = fma(eb, g2_17, o30_2);
            }
            { const double eb = bi[290];
              o30_2 = fma(eb, g2_18, o30_2);
            }
            { const double eb = bi[291];
              o30_2 = fma(eb, g2_30, o30_2);
            }
            { const double eb = bi[292];
              o31_2 = fma(eb, g2_0, o31_2);
            }
            { const double eb = bi[293];
              o31_2 = fma(eb, g2_1, o31_2);
            }
            { const double eb = bi[294];
              o31_2 = fma(eb, g2_2, o31_2);
            }
            { const double eb = bi[295];
              o31_2 = fma(eb, g2_5, o31_2);
            }
            { const double eb = bi[296];
              o31_2 = fma(eb, g2_6, o31_2);
            }
            { const double eb = bi[297];
              o31_2 = fma(eb, g2_12, o31_2);
            }
            { const double eb = bi[298];
              o31_2 = fma(eb, g2_13, o31_2);
            }
            { const double eb = bi[299];
              o31_2 = fma(eb, g2_23, o31_2);
            }
            { const double eb = bi[300];
              o32_2 = fma(eb, g2_0, o32_2);
            }
            { const double eb = bi[301];
              o32_2 = fma(eb, g2_1, o32_2);
            }
            { const double eb = bi[302];
              o32_2 = fma(eb, g2_4, o32_2);
            }
            { const double eb = bi[303];
              o32_2 = fma(eb, g2_10, o32_2);
            }
            { const double eb = bi[304];
              o32_2 = fma(eb, g2_2, o32_2);
            }
            { const double eb = bi[305];
              o32_2 = fma(eb, g2_5, o32_2);
            }
            { const double eb = bi[306];
              o32_2 = fma(eb, g2_11, o32_2);
            }
            { const double eb = bi[307];
              o32_2 = fma(eb, g2_21, o32_2);
            }
            { const double eb = bi[308];
              o33_2 = fma(eb, g2_0, o33_2);
            }
            { const double eb = bi[309];
              o33_2 = fma(eb, g2_1, o33_2);
            }
            { const double eb = bi[310];
              o33_2 = fma(eb, g2_2, o33_2);
            }
            { const double eb = bi[311];
              o33_2 = fma(eb, g2_5, o33_2);
            }
            { const double eb = bi[312];
              o33_2 = fma(eb, g2_6, o33_2);
            }
            { const double eb = bi[313];
              o33_2 = fma(eb, g2_12, o33_2);
            }
            { const double eb = bi[314];
              o33_2 = fma(eb, g2_3, o33_2);
            }
            { const double eb = bi[315];
              o33_2 = fma(eb, g2_7, o33_2);
            }
            { const double eb = bi[316];
              o33_2 = fma(eb, g2_8, o33_2);
            }
            { const double eb = bi[317];
              o33_2 = fma(eb, g2_15, o33_2);
            }
            { const double eb = bi[318];
              o33_2 = fma(eb, g2_16, o33_2);
            }
            { const double eb = bi[319];
              o33_2 = fma(eb, g2_27, o33_2);
            }
            { const double eb = bi[320];
              o34_2 = fma(eb, g2_0, o34_2);
            }
            { const double eb = bi[321];
              o34_2 = fma(eb, g2_1, o34_2);
            }
            { const double eb = bi[322];
              o34_2 = fma(eb, g2_4, o34_2);
            }
            { const double eb = bi[323];
              o34_2 = fma(eb, g2_2, o34_2);
            }
            { const double eb = bi[324];
              o34_2 = fma(eb, g2_5, o34_2);
            }
            { const double eb = bi[325];
              o34_2 = fma(eb, g2_11, o34_2);
            }
            { const double eb = bi[326];
              o34_2 = fma(eb, g2_3, o34_2);
            }
            { const double eb = bi[327];
              o34_2 = fma(eb, g2_7, o34_2);
            }
            { const double eb = bi[328];
              o34_2 = fma(eb, g2_14, o34_2);
            }
            { const double eb = bi[329];
              o34_2 = fma(eb, g2_8, o34_2);
            }
            { const double eb = bi[330];
              o34_2 = fma(eb, g2_15, o34_2);
            }
            { const double eb = bi[331];
              o34_2 = fma(eb, g2_26, o34_2);
            }
            { const double eb = bi[332];
              o35_2 = fma(eb, g2_0, o35_2);
            }
            { const double eb = bi[333];
              o35_2 = fma(eb, g2_1, o35_2);
            }
            { const double eb = bi[334];
              o35_2 = fma(eb, g2_4, o35_2);
            }
            { const double eb = bi[335];
              o35_2 = fma(eb, g2_2, o35_2);
            }
            { const double eb = bi[336];
              o35_2 = fma(eb, g2_5, o35_2);
            }
            { const double eb = bi[337];
              o35_2 = fma(eb, g2_11, o35_2);
            }
            { const double eb = bi[338];
              o35_2 = fma(eb, g2_6, o35_2);
            }
            { const double eb = bi[339];
              o35_2 = fma(eb, g2_12, o35_2);
            }
            { const double eb = bi[340];
              o35_2 = fma(eb, g2_22, o35_2);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0);
            o1_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 0);
            o2_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 0);
            o3_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 0);
            o4_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 2, fJ + 0);
            o5_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 2, fJ + 0);
            o6_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0);
            o7_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 0);
            o8_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 0);
            o9_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 0);
            o10_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 2, fJ + 0);
            o11_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 2, fJ + 0);
            o12_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0);
            o13_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 0);
            o14_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 0);
            o15_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 0);
            o16_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 2, fJ + 0);
            o17_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 2, fJ + 0);
            o18_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0);
            o19_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 0);
            o20_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 0);
            o21_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 0);
            o22_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 2, fJ + 0);
            o23_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 2, fJ + 0);
            o24_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0);
            o25_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 0);
            o26_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 0);
            o27_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 0);
            o28_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 2, fJ + 0);
            o29_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 2, fJ + 0);
            o30_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0);
            o31_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 0);
            o32_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 0);
            o33_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 0);
            o34_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 2, fJ + 0);
            o35_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 2, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o1_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o2_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o3_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o4_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o5_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o6_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o7_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o8_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o9_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o10_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o11_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o12_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o13_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o14_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o15_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o16_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o17_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o18_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o19_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o20_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o21_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o22_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o23_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o24_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o25_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o26_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o27_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o28_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o29_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o30_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o31_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o32_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o33_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o34_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o35_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 2, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 2) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 0) * N + fQ + 4];
            const double ptb5 = PT[(fP + 0) * N + fQ + 5];
            const double ptb6 = PT[(fP + 1) * N + fQ + 0];
            const double ptb7 = PT[(fP + 1) * N + fQ + 1];
            const double ptb8 = PT[(fP + 1) * N + fQ + 2];
            const double ptb9 = PT[(fP + 1) * N + fQ + 3];
            const double ptb10 = PT[(fP + 1) * N + fQ + 4];
            const double ptb11 = PT[(fP + 1) * N + fQ + 5];
            const double ptb12 = PT[(fP + 2) * N + fQ + 0];
            const double ptb13 = PT[(fP + 2) * N + fQ + 1];
            const double ptb14 = PT[(fP + 2) * N + fQ + 2];
            const double ptb15 = PT[(fP + 2) * N + fQ + 3];
            const double ptb16 = PT[(fP + 2) * N + fQ + 4];
            const double ptb17 = PT[(fP + 2) * N + fQ + 5];
            const double ptb18 = PT[(fP + 3) * N + fQ + 0];
            const double ptb19 = PT[(fP + 3) * N + fQ + 1];
            const double ptb20 = PT[(fP + 3) * N + fQ + 2];
            const double ptb21 = PT[(fP + 3) * N + fQ + 3];
            const double ptb22 = PT[(fP + 3) * N + fQ + 4];
            const double ptb23 = PT[(fP + 3) * N + fQ + 5];
            const double ptb24 = PT[(fP + 4) * N + fQ + 0];
            const double ptb25 = PT[(fP + 4) * N + fQ + 1];
            const double ptb26 = PT[(fP + 4) * N + fQ + 2];
            const double ptb27 = PT[(fP + 4) * N + fQ + 3];
            const double ptb28 = PT[(fP + 4) * N + fQ + 4];
            const double ptb29 = PT[(fP + 4) * N + fQ + 5];
            const double ptb30 = PT[(fP + 5) * N + fQ + 0];
            const double ptb31 = PT[(fP + 5) * N + fQ + 1];
            const double ptb32 = PT[(fP + 5) * N + fQ + 2];
            const double ptb33 = PT[(fP + 5) * N + fQ + 3];
            const double ptb34 = PT[(fP + 5) * N + fQ + 4];
            const double ptb35 = PT[(fP + 5) * N + fQ + 5];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd4_0 = PA[(fQ + 4) * N + fJ + 0];
            const double Abd5_0 = PA[(fQ + 5) * N + fJ + 0];
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
            const double Abc4_2 = PA[(fQ + 4) * N + fI + 2];
            const double Abc5_2 = PA[(fQ + 5) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bbd4_0 = PB[(fQ + 4) * N + fJ + 0];
            const double Bbd5_0 = PB[(fQ + 5) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_2 = PB[(fQ + 0) * N + fI + 2];
            const double Bbc1_2 = PB[(fQ + 1) * N + fI + 2];
            const double Bbc2_2 = PB[(fQ + 2) * N + fI + 2];
            const double Bbc3_2 = PB[(fQ + 3) * N + fI + 2];
            const double Bbc4_2 = PB[(fQ + 4) * N + fI + 2];
            const double Bbc5_2 = PB[(fQ + 5) * N + fI + 2];
            const double Bac0_2 = PB[(fP + 0) * N + fI + 2];
            const double Bac1_2 = PB[(fP + 1) * N + fI + 2];
            const double Bac2_2 = PB[(fP + 2) * N + fI + 2];
            const double Bac3_2 = PB[(fP + 3) * N + fI + 2];
            const double Bac4_2 = PB[(fP + 4) * N + fI + 2];
            const double Bac5_2 = PB[(fP + 5) * N + fI + 2];
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
            jab24 += o24_2 * ptk2;
            jab25 += o25_2 * ptk2;
            jab26 += o26_2 * ptk2;
            jab27 += o27_2 * ptk2;
            jab28 += o28_2 * ptk2;
            jab29 += o29_2 * ptk2;
            jab30 += o30_2 * ptk2;
            jab31 += o31_2 * ptk2;
            jab32 += o32_2 * ptk2;
            jab33 += o33_2 * ptk2;
            jab34 += o34_2 * ptk2;
            jab35 += o35_2 * ptk2;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17 + o18_2 * ptb18 + o19_2 * ptb19 + o20_2 * ptb20 + o21_2 * ptb21 + o22_2 * ptb22 + o23_2 * ptb23 + o24_2 * ptb24 + o25_2 * ptb25 + o26_2 * ptb26 + o27_2 * ptb27 + o28_2 * ptb28 + o29_2 * ptb29 + o30_2 * ptb30 + o31_2 * ptb31 + o32_2 * ptb32 + o33_2 * ptb33 + o34_2 * ptb34 + o35_2 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Abd0_0 + o1_2 * Abd1_0 + o2_2 * Abd2_0 + o3_2 * Abd3_0 + o4_2 * Abd4_0 + o5_2 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Aad0_0 + o6_2 * Aad1_0 + o12_2 * Aad2_0 + o18_2 * Aad3_0 + o24_2 * Aad4_0 + o30_2 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_2 * Abc0_2 + o1_2 * Abc1_2 + o2_2 * Abc2_2 + o3_2 * Abc3_2 + o4_2 * Abc4_2 + o5_2 * Abc5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_2 * Aac0_2 + o6_2 * Aac1_2 + o12_2 * Aac2_2 + o18_2 * Aac3_2 + o24_2 * Aac4_2 + o30_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_2 * Aad0_0 + o7_2 * Aad1_0 + o13_2 * Aad2_0 + o19_2 * Aad3_0 + o25_2 * Aad4_0 + o31_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_2 * Aac0_2 + o7_2 * Aac1_2 + o13_2 * Aac2_2 + o19_2 * Aac3_2 + o25_2 * Aac4_2 + o31_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_2 * Aad0_0 + o8_2 * Aad1_0 + o14_2 * Aad2_0 + o20_2 * Aad3_0 + o26_2 * Aad4_0 + o32_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_2 * Aac0_2 + o8_2 * Aac1_2 + o14_2 * Aac2_2 + o20_2 * Aac3_2 + o26_2 * Aac4_2 + o32_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_2 * Aad0_0 + o9_2 * Aad1_0 + o15_2 * Aad2_0 + o21_2 * Aad3_0 + o27_2 * Aad4_0 + o33_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_2 * Aac0_2 + o9_2 * Aac1_2 + o15_2 * Aac2_2 + o21_2 * Aac3_2 + o27_2 * Aac4_2 + o33_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 2, deg * (o4_2 * Aad0_0 + o10_2 * Aad1_0 + o16_2 * Aad2_0 + o22_2 * Aad3_0 + o28_2 * Aad4_0 + o34_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_2 * Aac0_2 + o10_2 * Aac1_2 + o16_2 * Aac2_2 + o22_2 * Aac3_2 + o28_2 * Aac4_2 + o34_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 2, deg * (o5_2 * Aad0_0 + o11_2 * Aad1_0 + o17_2 * Aad2_0 + o23_2 * Aad3_0 + o29_2 * Aad4_0 + o35_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_2 * Aac0_2 + o11_2 * Aac1_2 + o17_2 * Aac2_2 + o23_2 * Aac3_2 + o29_2 * Aac4_2 + o35_2 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o6_2 * Abd0_0 + o7_2 * Abd1_0 + o8_2 * Abd2_0 + o9_2 * Abd3_0 + o10_2 * Abd4_0 + o11_2 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_2 * Abc0_2 + o7_2 * Abc1_2 + o8_2 * Abc2_2 + o9_2 * Abc3_2 + o10_2 * Abc4_2 + o11_2 * Abc5_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o12_2 * Abd0_0 + o13_2 * Abd1_0 + o14_2 * Abd2_0 + o15_2 * Abd3_0 + o16_2 * Abd4_0 + o17_2 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_2 * Abc0_2 + o13_2 * Abc1_2 + o14_2 * Abc2_2 + o15_2 * Abc3_2 + o16_2 * Abc4_2 + o17_2 * Abc5_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o18_2 * Abd0_0 + o19_2 * Abd1_0 + o20_2 * Abd2_0 + o21_2 * Abd3_0 + o22_2 * Abd4_0 + o23_2 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_2 * Abc0_2 + o19_2 * Abc1_2 + o20_2 * Abc2_2 + o21_2 * Abc3_2 + o22_2 * Abc4_2 + o23_2 * Abc5_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o24_2 * Abd0_0 + o25_2 * Abd1_0 + o26_2 * Abd2_0 + o27_2 * Abd3_0 + o28_2 * Abd4_0 + o29_2 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_2 * Abc0_2 + o25_2 * Abc1_2 + o26_2 * Abc2_2 + o27_2 * Abc3_2 + o28_2 * Abc4_2 + o29_2 * Abc5_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o30_2 * Abd0_0 + o31_2 * Abd1_0 + o32_2 * Abd2_0 + o33_2 * Abd3_0 + o34_2 * Abd4_0 + o35_2 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_2 * Abc0_2 + o31_2 * Abc1_2 + o32_2 * Abc2_2 + o33_2 * Abc3_2 + o34_2 * Abc4_2 + o35_2 * Abc5_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Bbd0_0 + o1_2 * Bbd1_0 + o2_2 * Bbd2_0 + o3_2 * Bbd3_0 + o4_2 * Bbd4_0 + o5_2 * Bbd5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Bad0_0 + o6_2 * Bad1_0 + o12_2 * Bad2_0 + o18_2 * Bad3_0 + o24_2 * Bad4_0 + o30_2 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_2 * Bbc0_2 + o1_2 * Bbc1_2 + o2_2 * Bbc2_2 + o3_2 * Bbc3_2 + o4_2 * Bbc4_2 + o5_2 * Bbc5_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_2 * Bac0_2 + o6_2 * Bac1_2 + o12_2 * Bac2_2 + o18_2 * Bac3_2 + o24_2 * Bac4_2 + o30_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 2, deg * (o1_2 * Bad0_0 + o7_2 * Bad1_0 + o13_2 * Bad2_0 + o19_2 * Bad3_0 + o25_2 * Bad4_0 + o31_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_2 * Bac0_2 + o7_2 * Bac1_2 + o13_2 * Bac2_2 + o19_2 * Bac3_2 + o25_2 * Bac4_2 + o31_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 2, deg * (o2_2 * Bad0_0 + o8_2 * Bad1_0 + o14_2 * Bad2_0 + o20_2 * Bad3_0 + o26_2 * Bad4_0 + o32_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_2 * Bac0_2 + o8_2 * Bac1_2 + o14_2 * Bac2_2 + o20_2 * Bac3_2 + o26_2 * Bac4_2 + o32_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 2, deg * (o3_2 * Bad0_0 + o9_2 * Bad1_0 + o15_2 * Bad2_0 + o21_2 * Bad3_0 + o27_2 * Bad4_0 + o33_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_2 * Bac0_2 + o9_2 * Bac1_2 + o15_2 * Bac2_2 + o21_2 * Bac3_2 + o27_2 * Bac4_2 + o33_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 4) * N + fI + 2, deg * (o4_2 * Bad0_0 + o10_2 * Bad1_0 + o16_2 * Bad2_0 + o22_2 * Bad3_0 + o28_2 * Bad4_0 + o34_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fJ + 0, deg * (o4_2 * Bac0_2 + o10_2 * Bac1_2 + o16_2 * Bac2_2 + o22_2 * Bac3_2 + o28_2 * Bac4_2 + o34_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 5) * N + fI + 2, deg * (o5_2 * Bad0_0 + o11_2 * Bad1_0 + o17_2 * Bad2_0 + o23_2 * Bad3_0 + o29_2 * Bad4_0 + o35_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fJ + 0, deg * (o5_2 * Bac0_2 + o11_2 * Bac1_2 + o17_2 * Bac2_2 + o23_2 * Bac3_2 + o29_2 * Bac4_2 + o35_2 * Bac5_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o6_2 * Bbd0_0 + o7_2 * Bbd1_0 + o8_2 * Bbd2_0 + o9_2 * Bbd3_0 + o10_2 * Bbd4_0 + o11_2 * Bbd5_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o6_2 * Bbc0_2 + o7_2 * Bbc1_2 + o8_2 * Bbc2_2 + o9_2 * Bbc3_2 + o10_2 * Bbc4_2 + o11_2 * Bbc5_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o12_2 * Bbd0_0 + o13_2 * Bbd1_0 + o14_2 * Bbd2_0 + o15_2 * Bbd3_0 + o16_2 * Bbd4_0 + o17_2 * Bbd5_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o12_2 * Bbc0_2 + o13_2 * Bbc1_2 + o14_2 * Bbc2_2 + o15_2 * Bbc3_2 + o16_2 * Bbc4_2 + o17_2 * Bbc5_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o18_2 * Bbd0_0 + o19_2 * Bbd1_0 + o20_2 * Bbd2_0 + o21_2 * Bbd3_0 + o22_2 * Bbd4_0 + o23_2 * Bbd5_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o18_2 * Bbc0_2 + o19_2 * Bbc1_2 + o20_2 * Bbc2_2 + o21_2 * Bbc3_2 + o22_2 * Bbc4_2 + o23_2 * Bbc5_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o24_2 * Bbd0_0 + o25_2 * Bbd1_0 + o26_2 * Bbd2_0 + o27_2 * Bbd3_0 + o28_2 * Bbd4_0 + o29_2 * Bbd5_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o24_2 * Bbc0_2 + o25_2 * Bbc1_2 + o26_2 * Bbc2_2 + o27_2 * Bbc3_2 + o28_2 * Bbc4_2 + o29_2 * Bbc5_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o30_2 * Bbd0_0 + o31_2 * Bbd1_0 + o32_2 * Bbd2_0 + o33_2 * Bbd3_0 + o34_2 * Bbd4_0 + o35_2 * Bbd5_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o30_2 * Bbc0_2 + o31_2 * Bbc1_2 + o32_2 * Bbc2_2 + o33_2 * Bbc3_2 + o34_2 * Bbc4_2 + o35_2 * Bbc5_2));
          }
        } break;
        case 3: {  // ket functions [3]
          double o0_3 = 0;
          double o1_3 = 0;
          double o2_3 = 0;
          double o3_3 = 0;
          double o4_3 = 0;
          double o5_3 = 0;
          double o6_3 = 0;
          double o7_3 = 0;
          double o8_3 = 0;
          double o9_3 = 0;
          double o10_3 = 0;
          double o11_3 = 0;
          double o12_3 = 0;
          double o13_3 = 0;
          double o14_3 = 0;
          double o15_3 = 0;
          double o16_3 = 0;
          double o17_3 = 0;
          double o18_3 = 0;
          double o19_3 = 0;
          double o20_3 = 0;
          double o21_3 = 0;
          double o22_3 = 0;
          double o23_3 = 0;
          double o24_3 = 0;
          double o25_3 = 0;
          double o26_3 = 0;
          double o27_3 = 0;
          double o28_3 = 0;
          double o29_3 = 0;
          double o30_3 = 0;
          double o31_3 = 0;
          double o32_3 = 0;
          double o33_3 = 0;
          double o34_3 = 0;
          double o35_3 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 341;
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
            double g3_20 = 0;
            double g3_21 = 0;
            double g3_22 = 0;
            double g3_23 = 0;
            double g3_24 = 0;
            double g3_25 = 0;
            double g3_26 = 0;
            double g3_27 = 0;
            double g3_28 = 0;
            double g3_29 = 0;
            double g3_30 = 0;
            double g3_31 = 0;
            double g3_32 = 0;
            double g3_33 = 0;
            double g3_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 26 * kS;
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
              const double ek3_0 = kj[14 * kS];
              const double ek3_1 = -kj[15 * kS];
              const double ek3_2 = -kj[16 * kS];
              const double ek3_3 = kj[17 * kS];
              g3_0 = fma(ek3_0, b0, g3_0);
              const double r0_0_0_1 = Z * b1;
              g3_1 = fma(ek3_0, r0_0_0_1, g3_1);
              const double r0_0_1_0 = Y * b1;
              g3_2 = fma(ek3_0, r0_0_1_0, g3_2);
              g3_0 = fma(ek3_1, r0_0_1_0, g3_0);
              const double r0_1_0_0 = X * b1;
              g3_3 = fma(ek3_0, r0_1_0_0, g3_3);
              g3_0 = fma(ek3_2, r0_1_0_0, g3_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g3_4 = fma(ek3_0, r0_0_0_2, g3_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g3_5 = fma(ek3_0, r0_0_1_1, g3_5);
              g3_1 = fma(ek3_1, r0_0_1_1, g3_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g3_6 = fma(ek3_0, r0_0_2_0, g3_6);
              g3_2 = fma(ek3_1, r0_0_2_0, g3_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g3_7 = fma(ek3_0, r0_1_0_1, g3_7);
              g3_1 = fma(ek3_2, r0_1_0_1, g3_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g3_8 = fma(ek3_0, r0_1_1_0, g3_8);
              g3_3 = fma(ek3_1, r0_1_1_0, g3_3);
              g3_2 = fma(ek3_2, r0_1_1_0, g3_2);
              g3_0 = fma(ek3_3, r0_1_1_0, g3_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g3_9 = fma(ek3_0, r0_2_0_0, g3_9);
              g3_3 = fma(ek3_2, r0_2_0_0, g3_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g3_10 = fma(ek3_0, r0_0_0_3, g3_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g3_11 = fma(ek3_0, r0_0_1_2, g3_11);
              g3_4 = fma(ek3_1, r0_0_1_2, g3_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g3_12 = fma(ek3_0, r0_0_2_1, g3_12);
              g3_5 = fma(ek3_1, r0_0_2_1, g3_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g3_13 = fma(ek3_0, r0_0_3_0, g3_13);
              g3_6 = fma(ek3_1, r0_0_3_0, g3_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g3_14 = fma(ek3_0, r0_1_0_2, g3_14);
              g3_4 = fma(ek3_2, r0_1_0_2, g3_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g3_15 = fma(ek3_0, r0_1_1_1, g3_15);
              g3_7 = fma(ek3_1, r0_1_1_1, g3_7);
              g3_5 = fma(ek3_2, r0_1_1_1, g3_5);
              g3_1 = fma(ek3_3, r0_1_1_1, g3_1);
              const double r0_1_2_0 = X * r1_0_2_0;
              g3_16 = fma(ek3_0, r0_1_2_0, g3_16);
              g3_8 = fma(ek3_1, r0_1_2_0, g3_8);
              g3_6 = fma(ek3_2, r0_1_2_0, g3_6);
              g3_2 = fma(ek3_3, r0_1_2_0, g3_2);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g3_17 = fma(ek3_0, r0_2_0_1, g3_17);
              g3_7 = fma(ek3_2, r0_2_0_1, g3_7);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g3_18 = fma(ek3_0, r0_2_1_0, g3_18);
              g3_9 = fma(ek3_1, r0_2_1_0, g3_9);
              g3_8 = fma(ek3_2, r0_2_1_0, g3_8);
              g3_3 = fma(ek3_3, r0_2_1_0, g3_3);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g3_19 = fma(ek3_0, r0_3_0_0, g3_19);
              g3_9 = fma(ek3_2, r0_3_0_0, g3_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g3_20 = fma(ek3_0, r0_0_0_4, g3_20);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g3_21 = fma(ek3_0, r0_0_1_3, g3_21);
              g3_10 = fma(ek3_1, r0_0_1_3, g3_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g3_22 = fma(ek3_0, r0_0_2_2, g3_22);
              g3_11 = fma(ek3_1, r0_0_2_2, g3_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g3_23 = fma(ek3_0, r0_0_3_1, g3_23);
              g3_12 = fma(ek3_1, r0_0_3_1, g3_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g3_24 = fma(ek3_0, r0_0_4_0, g3_24);
              g3_13 = fma(ek3_1, r0_0_4_0, g3_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g3_25 = fma(ek3_0, r0_1_0_3, g3_25);
              g3_10 = fma(ek3_2, r0_1_0_3, g3_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g3_26 = fma(ek3_0, r0_1_1_2, g3_26);
              g3_14 = fma(ek3_1, r0_1_1_2, g3_14);
              g3_11 = fma(ek3_2, r0_1_1_2, g3_11);
              g3_4 = fma(ek3_3, r0_1_1_2, g3_4);
              const double r0_1_2_1 = X * r1_0_2_1;
              g3_27 = fma(ek3_0, r0_1_2_1, g3_27);
              g3_15 = fma(ek3_1, r0_1_2_1, g3_15);
              g3_12 = fma(ek3_2, r0_1_2_1, g3_12);
              g3_5 = fma(ek3_3, r0_1_2_1, g3_5);
              const double r0_1_3_0 = X * r1_0_3_0;
              g3_28 = fma(ek3_0, r0_1_3_0, g3_28);
              g3_16 = fma(ek3_1, r0_1_3_0, g3_16);
              g3_13 = fma(ek3_2, r0_1_3_0, g3_13);
              g3_6 = fma(ek3_3, r0_1_3_0, g3_6);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g3_29 = fma(ek3_0, r0_2_0_2, g3_29);
              g3_14 = fma(ek3_2, r0_2_0_2, g3_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g3_30 = fma(ek3_0, r0_2_1_1, g3_30);
              g3_17 = fma(ek3_1, r0_2_1_1, g3_17);
              g3_15 = fma(ek3_2, r0_2_1_1, g3_15);
              g3_7 = fma(ek3_3, r0_2_1_1, g3_7);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g3_31 = fma(ek3_0, r0_2_2_0, g3_31);
              g3_18 = fma(ek3_1, r0_2_2_0, g3_18);
              g3_16 = fma(ek3_2, r0_2_2_0, g3_16);
              g3_8 = fma(ek3_3, r0_2_2_0, g3_8);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g3_32 = fma(ek3_0, r0_3_0_1, g3_32);
              g3_17 = fma(ek3_2, r0_3_0_1, g3_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g3_33 = fma(ek3_0, r0_3_1_0, g3_33);
              g3_19 = fma(ek3_1, r0_3_1_0, g3_19);
              g3_18 = fma(ek3_2, r0_3_1_0, g3_18);
              g3_9 = fma(ek3_3, r0_3_1_0, g3_9);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g3_34 = fma(ek3_0, r0_4_0_0, g3_34);
              g3_19 = fma(ek3_2, r0_4_0_0, g3_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g3_20 = fma(ek3_1, r0_0_1_4, g3_20);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g3_21 = fma(ek3_1, r0_0_2_3, g3_21);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g3_22 = fma(ek3_1, r0_0_3_2, g3_22);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g3_23 = fma(ek3_1, r0_0_4_1, g3_23);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g3_24 = fma(ek3_1, r0_0_5_0, g3_24);
              const double r0_1_0_4 = X * r1_0_0_4;
              g3_20 = fma(ek3_2, r0_1_0_4, g3_20);
              const double r0_1_1_3 = X * r1_0_1_3;
              g3_25 = fma(ek3_1, r0_1_1_3, g3_25);
              g3_21 = fma(ek3_2, r0_1_1_3, g3_21);
              g3_10 = fma(ek3_3, r0_1_1_3, g3_10);
              const double r0_1_2_2 = X * r1_0_2_2;
              g3_26 = fma(ek3_1, r0_1_2_2, g3_26);
              g3_22 = fma(ek3_2, r0_1_2_2, g3_22);
              g3_11 = fma(ek3_3, r0_1_2_2, g3_11);
              const double r0_1_3_1 = X * r1_0_3_1;
              g3_27 = fma(ek3_1, r0_1_3_1, g3_27);
              g3_23 = fma(ek3_2, r0_1_3_1, g3_23);
              g3_12 = fma(ek3_3, r0_1_3_1, g3_12);
              const double r0_1_4_0 = X * r1_0_4_0;
              g3_28 = fma(ek3_1, r0_1_4_0, g3_28);
              g3_24 = fma(ek3_2, r0_1_4_0, g3_24);
              g3_13 = fma(ek3_3, r0_1_4_0, g3_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g3_25 = fma(ek3_2, r0_2_0_3, g3_25);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g3_29 = fma(ek3_1, r0_2_1_2, g3_29);
              g3_26 = fma(ek3_2, r0_2_1_2, g3_26);
              g3_14 = fma(ek3_3, r0_2_1_2, g3_14);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g3_30 = fma(ek3_1, r0_2_2_1, g3_30);
              g3_27 = fma(ek3_2, r0_2_2_1, g3_27);
              g3_15 = fma(ek3_3, r0_2_2_1, g3_15);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g3_31 = fma(ek3_1, r0_2_3_0, g3_31);
              g3_28 = fma(ek3_2, r0_2_3_0, g3_28);
              g3_16 = fma(ek3_3, r0_2_3_0, g3_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g3_29 = fma(ek3_2, r0_3_0_2, g3_29);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g3_32 = fma(ek3_1, r0_3_1_1, g3_32);
              g3_30 = fma(ek3_2, r0_3_1_1, g3_30);
              g3_17 = fma(ek3_3, r0_3_1_1, g3_17);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g3_33 = fma(ek3_1, r0_3_2_0, g3_33);
              g3_31 = fma(ek3_2, r0_3_2_0, g3_31);
              g3_18 = fma(ek3_3, r0_3_2_0, g3_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g3_32 = fma(ek3_2, r0_4_0_1, g3_32);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g3_34 = fma(ek3_1, r0_4_1_0, g3_34);
              g3_33 = fma(ek3_2, r0_4_1_0, g3_33);
              g3_19 = fma(ek3_3, r0_4_1_0, g3_19);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g3_34 = fma(ek3_2, r0_5_0_0, g3_34);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_1_1_4 = X * r1_0_1_4;
              g3_20 = fma(ek3_3, r0_1_1_4, g3_20);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g3_21 = fma(ek3_3, r0_1_2_3, g3_21);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g3_22 = fma(ek3_3, r0_1_3_2, g3_22);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_1_4_1 = X * r1_0_4_1;
              g3_23 = fma(ek3_3, r0_1_4_1, g3_23);
              const double r5_0_1_0 = Y * b6;
              const double r4_0_2_0 = fma(Y, r5_0_1_0, b5);
              const double r3_0_3_0 = fma(Y, r4_0_2_0, 2.0 * r4_0_1_0);
              const double r2_0_4_0 = fma(Y, r3_0_3_0, 3.0 * r3_0_2_0);
              const double r1_0_5_0 = fma(Y, r2_0_4_0, 4.0 * r2_0_3_0);
              const double r0_1_5_0 = X * r1_0_5_0;
              g3_24 = fma(ek3_3, r0_1_5_0, g3_24);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g3_25 = fma(ek3_3, r0_2_1_3, g3_25);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g3_26 = fma(ek3_3, r0_2_2_2, g3_26);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g3_27 = fma(ek3_3, r0_2_3_1, g3_27);
              const double r1_1_4_0 = X * r2_0_4_0;
              const double r0_2_4_0 = fma(X, r1_1_4_0, r1_0_4_0);
              g3_28 = fma(ek3_3, r0_2_4_0, g3_28);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g3_29 = fma(ek3_3, r0_3_1_2, g3_29);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g3_30 = fma(ek3_3, r0_3_2_1, g3_30);
              const double r2_1_3_0 = X * r3_0_3_0;
              const double r1_2_3_0 = fma(X, r2_1_3_0, r2_0_3_0);
              const double r0_3_3_0 = fma(X, r1_2_3_0, 2.0 * r1_1_3_0);
              g3_31 = fma(ek3_3, r0_3_3_0, g3_31);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g3_32 = fma(ek3_3, r0_4_1_1, g3_32);
              const double r3_1_2_0 = X * r4_0_2_0;
              const double r2_2_2_0 = fma(X, r3_1_2_0, r3_0_2_0);
              const double r1_3_2_0 = fma(X, r2_2_2_0, 2.0 * r2_1_2_0);
              const double r0_4_2_0 = fma(X, r1_3_2_0, 3.0 * r1_2_2_0);
              g3_33 = fma(ek3_3, r0_4_2_0, g3_33);
              const double r4_1_1_0 = X * r5_0_1_0;
              const double r3_2_1_0 = fma(X, r4_1_1_0, r4_0_1_0);
              const double r2_3_1_0 = fma(X, r3_2_1_0, 2.0 * r3_1_1_0);
              const double r1_4_1_0 = fma(X, r2_3_1_0, 3.0 * r2_2_1_0);
              const double r0_5_1_0 = fma(X, r1_4_1_0, 4.0 * r1_3_1_0);
              g3_34 = fma(ek3_3, r0_5_1_0, g3_34);
            }
            { const double eb = bi[5];
              o0_3 = fma(eb, g3_0, o0_3);
            }
            { const double eb = bi[6];
              o0_3 = fma(eb, g3_3, o0_3);
            }
            { const double eb = bi[7];
              o0_3 = fma(eb, g3_9, o0_3);
            }
            { const double eb = bi[8];
              o0_3 = fma(eb, g3_19, o0_3);
            }
            { const double eb = bi[9];
              o0_3 = fma(eb, g3_34, o0_3);
            }
            { const double eb = bi[10];
              o1_3 = fma(eb, g3_0, o1_3);
            }
            { const double eb = bi[11];
              o1_3 = fma(eb, g3_2, o1_3);
            }
            { const double eb = bi[12];
              o1_3 = fma(eb, g3_6, o1_3);
            }
            { const double eb = bi[13];
              o1_3 = fma(eb, g3_3, o1_3);
            }
            { const double eb = bi[14];
              o1_3 = fma(eb, g3_8, o1_3);
            }
            { const double eb = bi[15];
              o1_3 = fma(eb, g3_16, o1_3);
            }
            { const double eb = bi[16];
              o1_3 = fma(eb, g3_9, o1_3);
            }
            { const double eb = bi[17];
              o1_3 = fma(eb, g3_18, o1_3);
            }
            { const double eb = bi[18];
              o1_3 = fma(eb, g3_31, o1_3);
            }
            { const double eb = bi[19];
              o2_3 = fma(eb, g3_0, o2_3);
            }
            { const double eb = bi[20];
              o2_3 = fma(eb, g3_1, o2_3);
            }
            { const double eb = bi[21];
              o2_3 = fma(eb, g3_4, o2_3);
            }
            { const double eb = bi[22];
              o2_3 = fma(eb, g3_3, o2_3);
            }
            { const double eb = bi[23];
              o2_3 = fma(eb, g3_7, o2_3);
            }
            { const double eb = bi[24];
              o2_3 = fma(eb, g3_14, o2_3);
            }
            { const double eb = bi[25];
              o2_3 = fma(eb, g3_9, o2_3);
            }
            { const double eb = bi[26];
              o2_3 = fma(eb, g3_17, o2_3);
            }
            { const double eb = bi[27];
              o2_3 = fma(eb, g3_29, o2_3);
            }
            { const double eb = bi[28];
              o3_3 = fma(eb, g3_0, o3_3);
            }
            { const double eb = bi[29];
              o3_3 = fma(eb, g3_2, o3_3);
            }
            { const double eb = bi[30];
              o3_3 = fma(eb, g3_3, o3_3);
            }
            { const double eb = bi[31];
              o3_3 = fma(eb, g3_8, o3_3);
            }
            { const double eb = bi[32];
              o3_3 = fma(eb, g3_9, o3_3);
            }
            { const double eb = bi[33];
              o3_3 = fma(eb, g3_18, o3_3);
            }
            { const double eb = bi[34];
              o3_3 = fma(eb, g3_19, o3_3);
            }
            { const double eb = bi[35];
              o3_3 = fma(eb, g3_33, o3_3);
            }
            { const double eb = bi[36];
              o4_3 = fma(eb, g3_0, o4_3);
            }
            { const double eb = bi[37];
              o4_3 = fma(eb, g3_1, o4_3);
            }
            { const double eb = bi[38];
              o4_3 = fma(eb, g3_3, o4_3);
            }
            { const double eb = bi[39];
              o4_3 = fma(eb, g3_7, o4_3);
            }
            { const double eb = bi[40];
              o4_3 = fma(eb, g3_9, o4_3);
            }
            { const double eb = bi[41];
              o4_3 = fma(eb, g3_17, o4_3);
            }
            { const double eb = bi[42];
              o4_3 = fma(eb, g3_19, o4_3);
            }
            { const double eb = bi[43];
              o4_3 = fma(eb, g3_32, o4_3);
            }
            { const double eb = bi[44];
              o5_3 = fma(eb, g3_0, o5_3);
            }
            { const double eb = bi[45];
              o5_3 = fma(eb, g3_1, o5_3);
            }
            { const double eb = bi[46];
              o5_3 = fma(eb, g3_2, o5_3);
            }
            { const double eb = bi[47];
              o5_3 = fma(eb, g3_5, o5_3);
            }
            { const double eb = bi[48];
              o5_3 = fma(eb, g3_3, o5_3);
            }
            { const double eb = bi[49];
              o5_3 = fma(eb, g3_7, o5_3);
            }
            { const double eb = bi[50];
              o5_3 = fma(eb, g3_8, o5_3);
            }
            { const double eb = bi[51];
              o5_3 = fma(eb, g3_15, o5_3);
            }
            { const double eb = bi[52];
              o5_3 = fma(eb, g3_9, o5_3);
            }
            { const double eb = bi[53];
              o5_3 = fma(eb, g3_17, o5_3);
            }
            { const double eb = bi[54];
              o5_3 = fma(eb, g3_18, o5_3);
            }
            { const double eb = bi[55];
              o5_3 = fma(eb, g3_30, o5_3);
            }
            { const double eb = bi[56];
              o6_3 = fma(eb, g3_0, o6_3);
            }
            { const double eb = bi[57];
              o6_3 = fma(eb, g3_2, o6_3);
            }
            { const double eb = bi[58];
              o6_3 = fma(eb, g3_6, o6_3);
            }
            { const double eb = bi[59];
              o6_3 = fma(eb, g3_3, o6_3);
            }
            { const double eb = bi[60];
              o6_3 = fma(eb, g3_8, o6_3);
            }
            { const double eb = bi[61];
              o6_3 = fma(eb, g3_16, o6_3);
            }
            { const double eb = bi[62];
              o6_3 = fma(eb, g3_9, o6_3);
            }
            { const double eb = bi[63];
              o6_3 = fma(eb, g3_18, o6_3);
            }
            { const double eb = bi[64];
              o6_3 = fma(eb, g3_31, o6_3);
            }
            { const double eb = bi[65];
              o7_3 = fma(eb, g3_0, o7_3);
            }
            { const double eb = bi[66];
              o7_3 = fma(eb, g3_2, o7_3);
            }
            { const double eb = bi[67];
              o7_3 = fma(eb, g3_6, o7_3);
            }
            { const double eb = bi[68];
              o7_3 = fma(eb, g3_13, o7_3);
            }
            { const double eb = bi[69];
              o7_3 = fma(eb, g3_24, o7_3);
            }
            { const double eb = bi[70];
              o8_3 = fma(eb, g3_0, o8_3);
            }
            { const double eb = bi[71];
              o8_3 = fma(eb, g3_1, o8_3);
            }
            { const double eb = bi[72];
              o8_3 = fma(eb, g3_4, o8_3);
            }
            { const double eb = bi[73];
              o8_3 = fma(eb, g3_2, o8_3);
            }
            { const double eb = bi[74];
              o8_3 = fma(eb, g3_5, o8_3);
            }
            { const double eb = bi[75];
              o8_3 = fma(eb, g3_11, o8_3);
            }
            { const double eb = bi[76];
              o8_3 = fma(eb, g3_6, o8_3);
            }
            { const double eb = bi[77];
              o8_3 = fma(eb, g3_12, o8_3);
            }
            { const double eb = bi[78];
              o8_3 = fma(eb, g3_22, o8_3);
            }
            { const double eb = bi[79];
              o9_3 = fma(eb, g3_0, o9_3);
            }
            { const double eb = bi[80];
              o9_3 = fma(eb, g3_2, o9_3);
            }
            { const double eb = bi[81];
              o9_3 = fma(eb, g3_6, o9_3);
            }
            { const double eb = bi[82];
              o9_3 = fma(eb, g3_13, o9_3);
            }
            { const double eb = bi[83];
              o9_3 = fma(eb, g3_3, o9_3);
            }
            { const double eb = bi[84];
              o9_3 = fma(eb, g3_8, o9_3);
            }
            { const double eb = bi[85];
              o9_3 = fma(eb, g3_16, o9_3);
            }
            { const double eb = bi[86];
              o9_3 = fma(eb, g3_28, o9_3);
            }
            { const double eb = bi[87];
              o10_3 = fma(eb, g3_0, o10_3);
            }
            { const double eb = bi[88];
              o10_3 = fma(eb, g3_1, o10_3);
            }
            { const double eb = bi[89];
              o10_3 = fma(eb, g3_2, o10_3);
            }
            { const double eb = bi[90];
              o10_3 = fma(eb, g3_5, o10_3);
            }
            { const double eb = bi[91];
              o10_3 = fma(eb, g3_6, o10_3);
            }
            { const double eb = bi[92];
              o10_3 = fma(eb, g3_12, o10_3);
            }
            { const double eb = bi[93];
              o10_3 = fma(eb, g3_3, o10_3);
            }
            { const double eb = bi[94];
              o10_3 = fma(eb, g3_7, o10_3);
            }
            { const double eb = bi[95];
              o10_3 = fma(eb, g3_8, o10_3);
            }
            { const double eb = bi[96];
              o10_3 = fma(eb, g3_15, o10_3);
            }
            { const double eb = bi[97];
              o10_3 = fma(eb, g3_16, o10_3);
            }
            { const double eb = bi[98];
              o10_3 = fma(eb, g3_27, o10_3);
            }
            { const double eb = bi[99];
              o11_3 = fma(eb, g3_0, o11_3);
            }
            { const double eb = bi[100];
              o11_3 = fma(eb, g3_1, o11_3);
            }
            { const double eb = bi[101];
              o11_3 = fma(eb, g3_2, o11_3);
            }
            { const double eb = bi[102];
              o11_3 = fma(eb, g3_5, o11_3);
            }
            { const double eb = bi[103];
              o11_3 = fma(eb, g3_6, o11_3);
            }
            { const double eb = bi[104];
              o11_3 = fma(eb, g3_12, o11_3);
            }
            { const double eb = bi[105];
              o11_3 = fma(eb, g3_13, o11_3);
            }
            { const double eb = bi[106];
              o11_3 = fma(eb, g3_23, o11_3);
            }
            { const double eb = bi[107];
              o12_3 = fma(eb, g3_0, o12_3);
            }
            { const double eb = bi[108];
              o12_3 = fma(eb, g3_1, o12_3);
            }
            { const double eb = bi[109];
              o12_3 = fma(eb, g3_4, o12_3);
            }
            { const double eb = bi[110];
              o12_3 = fma(eb, g3_3, o12_3);
            }
            { const double eb = bi[111];
              o12_3 = fma(eb, g3_7, o12_3);
            }
            { const double eb = bi[112];
              o12_3 = fma(eb, g3_14, o12_3);
            }
            { const double eb = bi[113];
              o12_3 = fma(eb, g3_9, o12_3);
            }
            { const double eb = bi[114];
              o12_3 = fma(eb, g3_17, o12_3);
            }
            { const double eb = bi[115];
              o12_3 = fma(eb, g3_29, o12_3);
            }
            { const double eb = bi[116];
              o13_3 = fma(eb, g3_0, o13_3);
            }
            { const double eb = bi[117];
              o13_3 = fma(eb, g3_1, o13_3);
            }
            { const double eb = bi[118];
              o13_3 = fma(eb, g3_4, o13_3);
            }
            { const double eb = bi[119];
              o13_3 = fma(eb, g3_2, o13_3);
            }
            { const double eb = bi[120];
              o13_3 = fma(eb, g3_5, o13_3);
            }
            { const double eb = bi[121];
              o13_3 = fma(eb, g3_11, o13_3);
            }
            { const double eb = bi[122];
              o13_3 = fma(eb, g3_6, o13_3);
            }
            { const double eb = bi[123];
              o13_3 = fma(eb, g3_12, o13_3);
            }
            { const double eb = bi[124];
              o13_3 = fma(eb, g3_22, o13_3);
            }
            { const double eb = bi[125];
              o14_3 = fma(eb, g3_0, o14_3);
            }
            { const double eb = bi[126];
              o14_3 = fma(eb, g3_1, o14_3);
            }
            { const double eb = bi[127];
              o14_3 = fma(eb, g3_4, o14_3);
            }
            { const double eb = bi[128];
              o14_3 = fma(eb, g3_10, o14_3);
            }
            { const double eb = bi[129];
              o14_3 = fma(eb, g3_20, o14_3);
            }
            { const double eb = bi[130];
              o15_3 = fma(eb, g3_0, o15_3);
            }
            { const double eb = bi[131];
              o15_3 = fma(eb, g3_1, o15_3);
            }
            { const double eb = bi[132];
              o15_3 = fma(eb, g3_4, o15_3);
            }
            { const double eb = bi[133];
              o15_3 = fma(eb, g3_2, o15_3);
            }
            { const double eb = bi[134];
              o15_3 = fma(eb, g3_5, o15_3);
            }
            { const double eb = bi[135];
              o15_3 = fma(eb, g3_11, o15_3);
            }
            { const double eb = bi[136];
              o15_3 = fma(eb, g3_3, o15_3);
            }
            { const double eb = bi[137];
              o15_3 = fma(eb, g3_7, o15_3);
            }
            { const double eb = bi[138];
              o15_3 = fma(eb, g3_14, o15_3);
            }
            { const double eb = bi[139];
              o15_3 = fma(eb, g3_8, o15_3);
            }
            { const double eb = bi[140];
              o15_3 = fma(eb, g3_15, o15_3);
            }
            { const double eb = bi[141];
              o15_3 = fma(eb, g3_26, o15_3);
            }
            { const double eb = bi[142];
              o16_3 = fma(eb, g3_0, o16_3);
            }
            { const double eb = bi[143];
              o16_3 = fma(eb, g3_1, o16_3);
            }
            { const double eb = bi[144];
              o16_3 = fma(eb, g3_4, o16_3);
            }
            { const double eb = bi[145];
              o16_3 = fma(eb, g3_10, o16_3);
            }
            { const double eb = bi[146];
              o16_3 = fma(eb, g3_3, o16_3);
            }
            { const double eb = bi[147];
              o16_3 = fma(eb, g3_7, o16_3);
            }
            { const double eb = bi[148];
              o16_3 = fma(eb, g3_14, o16_3);
            }
            { const double eb = bi[149];
              o16_3 = fma(eb, g3_25, o16_3);
            }
            { const double eb = bi[150];
              o17_3 = fma(eb, g3_0, o17_3);
            }
            { const double eb = bi[151];
              o17_3 = fma(eb, g3_1, o17_3);
            }
            { const double eb = bi[152];
              o17_3 = fma(eb, g3_4, o17_3);
            }
            { const double eb = bi[153];
              o17_3 = fma(eb, g3_10, o17_3);
            }
            { const double eb = bi[154];
              o17_3 = fma(eb, g3_2, o17_3);
            }
            { const double eb = bi[155];
              o17_3 = fma(eb, g3_5, o17_3);
            }
            { const double eb = bi[156];
              o17_3 = fma(eb, g3_11, o17_3);
            }
            { const double eb = bi[157];
              o17_3 = fma(eb, g3_21, o17_3);
            }
            { const double eb = bi[158];
              o18_3 = fma(eb, g3_0, o18_3);
            }
            { const double eb = bi[159];
              o18_3 = fma(eb, g3_2, o18_3);
            }
            { const double eb = bi[160];
              o18_3 = fma(eb, g3_3, o18_3);
            }
            { const double eb = bi[161];
              o18_3 = fma(eb, g3_8, o18_3);
            }
            { const double eb = bi[162];
              o18_3 = fma(eb, g3_9, o18_3);
            }
            { const double eb = bi[163];
              o18_3 = fma(eb, g3_18, o18_3);
            }
            { const double eb = bi[164];
              o18_3 = fma(eb, g3_19, o18_3);
            }
            { const double eb = bi[165];
              o18_3 = fma(eb, g3_33, o18_3);
            }
            { const double eb = bi[166];
              o19_3 = fma(eb, g3_0, o19_3);
            }
            { const double eb = bi[167];
              o19_3 = fma(eb, g3_2, o19_3);
            }
            { const double eb = bi[168];
              o19_3 = fma(eb, g3_6, o19_3);
            }
            { const double eb = bi[169];
              o19_3 = fma(eb, g3_13, o19_3);
            }
            { const double eb = bi[170];
              o19_3 = fma(eb, g3_3, o19_3);
            }
            { const double eb = bi[171];
              o19_3 = fma(eb, g3_8, o19_3);
            }
            { const double eb = bi[172];
              o19_3 = fma(eb, g3_16, o19_3);
            }
            { const double eb = bi[173];
              o19_3 = fma(eb, g3_28, o19_3);
            }
            { const double eb = bi[174];
              o20_3 = fma(eb, g3_0, o20_3);
            }
            { const double eb = bi[175];
              o20_3 = fma(eb, g3_1, o20_3);
            }
            { const double eb = bi[176];
              o20_3 = fma(eb, g3_4, o20_3);
            }
            { const double eb = bi[177];
              o20_3 = fma(eb, g3_2, o20_3);
            }
            { const double eb = bi[178];
              o20_3 = fma(eb, g3_5, o20_3);
            }
            { const double eb = bi[179];
              o20_3 = fma(eb, g3_11, o20_3);
            }
            { const double eb = bi[180];
              o20_3 = fma(eb, g3_3, o20_3);
            }
            { const double eb = bi[181];
              o20_3 = fma(eb, g3_7, o20_3);
            }
            { const double eb = bi[182];
              o20_3 = fma(eb, g3_14, o20_3);
            }
            { const double eb = bi[183];
              o20_3 = fma(eb, g3_8, o20_3);
            }
            { const double eb = bi[184];
              o20_3 = fma(eb, g3_15, o20_3);
            }
            { const double eb = bi[185];
              o20_3 = fma(eb, g3_26, o20_3);
            }
            { const double eb = bi[186];
              o21_3 = fma(eb, g3_0, o21_3);
            }
            { const double eb = bi[187];
              o21_3 = fma(eb, g3_2, o21_3);
            }
            { const double eb = bi[188];
              o21_3 = fma(eb, g3_6, o21_3);
            }
            { const double eb = bi[189];
              o21_3 = fma(eb, g3_3, o21_3);
            }
            { const double eb = bi[190];
              o21_3 = fma(eb, g3_8, o21_3);
            }
            { const double eb = bi[191];
              o21_3 = fma(eb, g3_16, o21_3);
            }
            { const double eb = bi[192];
              o21_3 = fma(eb, g3_9, o21_3);
            }
            { const double eb = bi[193];
              o21_3 = fma(eb, g3_18, o21_3);
            }
            { const double eb = bi[194];
              o21_3 = fma(eb, g3_31, o21_3);
            }
            { const double eb = bi[195];
              o22_3 = fma(eb, g3_0, o22_3);
            }
            { const double eb = bi[196];
              o22_3 = fma(eb, g3_1, o22_3);
            }
            { const double eb = bi[197];
              o22_3 = fma(eb, g3_2, o22_3);
            }
            { const double eb = bi[198];
              o22_3 = fma(eb, g3_5, o22_3);
            }
            { const double eb = bi[199];
              o22_3 = fma(eb, g3_3, o22_3);
            }
            { const double eb = bi[200];
              o22_3 = fma(eb, g3_7, o22_3);
            }
            { const double eb = bi[201];
              o22_3 = fma(eb, g3_8, o22_3);
            }
            { const double eb = bi[202];
              o22_3 = fma(eb, g3_15, o22_3);
            }
            { const double eb = bi[203];
              o22_3 = fma(eb, g3_9, o22_3);
            }
            { const double eb = bi[204];
              o22_3 = fma(eb, g3_17, o22_3);
            }
            { const double eb = bi[205];
              o22_3 = fma(eb, g3_18, o22_3);
            }
            { const double eb = bi[206];
              o22_3 = fma(eb, g3_30, o22_3);
            }
            { const double eb = bi[207];
              o23_3 = fma(eb, g3_0, o23_3);
            }
            { const double eb = bi[208];
              o23_3 = fma(eb, g3_1, o23_3);
            }
            { const double eb = bi[209];
              o23_3 = fma(eb, g3_2, o23_3);
            }
            { const double eb = bi[210];
              o23_3 = fma(eb, g3_5, o23_3);
            }
            { const double eb = bi[211];
              o23_3 = fma(eb, g3_6, o23_3);
            }
            { const double eb = bi[212];
              o23_3 = fma(eb, g3_12, o23_3);
            }
            { const double eb = bi[213];
              o23_3 = fma(eb, g3_3, o23_3);
            }
            { const double eb = bi[214];
              o23_3 = fma(eb, g3_7, o23_3);
            }
            { const double eb = bi[215];
              o23_3 = fma(eb, g3_8, o23_3);
            }
            { const double eb = bi[216];
              o23_3 = fma(eb, g3_15, o23_3);
            }
            { const double eb = bi[217];
              o23_3 = fma(eb, g3_16, o23_3);
            }
            { const double eb = bi[218];
              o23_3 = fma(eb, g3_27, o23_3);
            }
            { const double eb = bi[219];
              o24_3 = fma(eb, g3_0, o24_3);
            }
            { const double eb = bi[220];
              o24_3 = fma(eb, g3_1, o24_3);
            }
            { const double eb = bi[221];
              o24_3 = fma(eb, g3_3, o24_3);
            }
            { const double eb = bi[222];
              o24_3 = fma(eb, g3_7, o24_3);
            }
            { const double eb = bi[223];
              o24_3 = fma(eb, g3_9, o24_3);
            }
            { const double eb = bi[224];
              o24_3 = fma(eb, g3_17, o24_3);
            }
            { const double eb = bi[225];
              o24_3 = fma(eb, g3_19, o24_3);
            }
            { const double eb = bi[226];
              o24_3 = fma(eb, g3_32, o24_3);
            }
            { const double eb = bi[227];
              o25_3 = fma(eb, g3_0, o25_3);
            }
            { const double eb = bi[228];
              o25_3 = fma(eb, g3_1, o25_3);
            }
            { const double eb = bi[229];
              o25_3 = fma(eb, g3_2, o25_3);
            }
            { const double eb = bi[230];
              o25_3 = fma(eb, g3_5, o25_3);
            }
            { const double eb = bi[231];
              o25_3 = fma(eb, g3_6, o25_3);
            }
            { const double eb = bi[232];
              o25_3 = fma(eb, g3_12, o25_3);
            }
            { const double eb = bi[233];
              o25_3 = fma(eb, g3_3, o25_3);
            }
            { const double eb = bi[234];
              o25_3 = fma(eb, g3_7, o25_3);
            }
            { const double eb = bi[235];
              o25_3 = fma(eb, g3_8, o25_3);
            }
            { const double eb = bi[236];
              o25_3 = fma(eb, g3_15, o25_3);
            }
            { const double eb = bi[237];
              o25_3 = fma(eb, g3_16, o25_3);
            }
            { const double eb = bi[238];
              o25_3 = fma(eb, g3_27, o25_3);
            }
            { const double eb = bi[239];
              o26_3 = fma(eb, g3_0, o26_3);
            }
            { const double eb = bi[240];
              o26_3 = fma(eb, g3_1, o26_3);
            }
            { const double eb = bi[241];
              o26_3 = fma(eb, g3_4, o26_3);
            }
            { const double eb = bi[242];
              o26_3 = fma(eb, g3_10, o26_3);
            }
            { const double eb = bi[243];
              o26_3 = fma(eb, g3_3, o26_3);
            }
            { const double eb = bi[244];
              o26_3 = fma(eb, g3_7, o26_3);
            }
            { const double eb = bi[245];
              o26_3 = fma(eb, g3_14, o26_3);
            }
            { const double eb = bi[246];
              o26_3 = fma(eb, g3_25, o26_3);
            }
            { const double eb = bi[247];
              o27_3 = fma(eb, g3_0, o27_3);
            }
            { const double eb = bi[248];
              o27_3 = fma(eb, g3_1, o27_3);
            }
            { const double eb = bi[249];
              o27_3 = fma(eb, g3_2, o27_3);
            }
            { const double eb = bi[250];
              o27_3 = fma(eb, g3_5, o27_3);
            }
            { const double eb = bi[251];
              o27_3 = fma(eb, g3_3, o27_3);
            }
            { const double eb = bi[252];
              o27_3 = fma(eb, g3_7, o27_3);
            }
            { const double eb = bi[253];
              o27_3 = fma(eb, g3_8, o27_3);
            }
            { const double eb = bi[254];
              o27_3 = fma(eb, g3_15, o27_3);
            }
            { const double eb = bi[255];
              o27_3 = fma(eb, g3_9, o27_3);
            }
            { const double eb = bi[256];
              o27_3 = fma(eb, g3_17, o27_3);
            }
            { const double eb = bi[257];
              o27_3 = fma(eb, g3_18, o27_3);
            }
            { const double eb = bi[258];
              o27_3 = fma(eb, g3_30, o27_3);
            }
            { const double eb = bi[259];
              o28_3 = fma(eb, g3_0, o28_3);
            }
            { const double eb = bi[260];
              o28_3 = fma(eb, g3_1, o28_3);
            }
            { const double eb = bi[261];
              o28_3 = fma(eb, g3_4, o28_3);
            }
            { const double eb = bi[262];
              o28_3 = fma(eb, g3_3, o28_3);
            }
            { const double eb = bi[263];
              o28_3 = fma(eb, g3_7, o28_3);
            }
            { const double eb = bi[264];
              o28_3 = fma(eb, g3_14, o28_3);
            }
            { const double eb = bi[265];
              o28_3 = fma(eb, g3_9, o28_3);
            }
            { const double eb = bi[266];
              o28_3 = fma(eb, g3_17, o28_3);
            }
            { const double eb = bi[267];
              o28_3 = fma(eb, g3_29, o28_3);
            }
            { const double eb = bi[268];
              o29_3 = fma(eb, g3_0, o29_3);
            }
            { const double eb = bi[269];
              o29_3 = fma(eb, g3_1, o29_3);
            }
            { const double eb = bi[270];
              o29_3 = fma(eb, g3_4, o29_3);
            }
            { const double eb = bi[271];
              o29_3 = fma(eb, g3_2, o29_3);
            }
            { const double eb = bi[272];
              o29_3 = fma(eb, g3_5, o29_3);
            }
            { const double eb = bi[273];
              o29_3 = fma(eb, g3_11, o29_3);
            }
            { const double eb = bi[274];
              o29_3 = fma(eb, g3_3, o29_3);
            }
            { const double eb = bi[275];
              o29_3 = fma(eb, g3_7, o29_3);
            }
            { const double eb = bi[276];
              o29_3 = fma(eb, g3_14, o29_3);
            }
            { const double eb = bi[277];
              o29_3 = fma(eb, g3_8, o29_3);
            }
            { const double eb = bi[278];
              o29_3 = fma(eb, g3_15, o29_3);
            }
            { const double eb = bi[279];
              o29_3 = fma(eb, g3_26, o29_3);
            }
            { const double eb = bi[280];
              o30_3 = fma(eb, g3_0, o30_3);
            }
            { const double eb = bi[281];
              o30_3 = fma(eb, g3_1, o30_3);
            }
            { const double eb = bi[282];
              o30_3 = fma(eb, g3_2, o30_3);
            }
            { const double eb = bi[283];
              o30_3 = fma(eb, g3_5, o30_3);
            }
            { const double eb = bi[284];
              o30_3 = fma(eb, g3_3, o30_3);
            }
            { const double eb = bi[285];
              o30_3 = fma(eb, g3_7, o30_3);
            }
            { const double eb = bi[286];
              o30_3 = fma(eb, g3_8, o30_3);
            }
            { const double eb = bi[287];
              o30_3 = fma(eb, g3_15, o30_3);
            }
            { const double eb = bi[288];
              o30_3 = fma(eb, g3_9, o30_3);
            }
            { const double eb = bi[289];
              o30_3 = fma(eb, g3_17, o30_3);
            }
            { const double eb = bi[290];
              o30_3 = fma(eb, g3_18, o30_3);
            }
            { const double eb = bi[291];
              o30_3 = fma(eb, g3_30, o30_3);
            }
            { const double eb = bi[292];
              o31_3 = fma(eb, g3_0, o31_3);
            }
            { const double eb = bi[293];
              o31_3 = fma(eb, g3_1, o31_3);
            }
            { const double eb = bi[294];
              o31_3 = fma(eb, g3_2, o31_3);
            }
            { const double eb = bi[295];
              o31_3 = fma(eb, g3_5, o31_3);
            }
            { const double eb = bi[296];
              o31_3 = fma(eb, g3_6, o31_3);
            }
            { const double eb = bi[297];
              o31_3 = fma(eb, g3_12, o31_3);
            }
            { const double eb = bi[298];
              o31_3 = fma(eb, g3_13, o31_3);
            }
            { const double eb = bi[299];
              o31_3 = fma(eb, g3_23, o31_3);
            }
            { const double eb = bi[300];
              o32_3 = fma(eb, g3_0, o32_3);
            }
            { const double eb = bi[301];
              o32_3 = fma(eb, g3_1, o32_3);
            }
            { const double eb = bi[302];
              o32_3 = fma(eb, g3_4, o32_3);
            }
            { const double eb = bi[303];
              o32_3 = fma(eb, g3_10, o32_3);
            }
            { const double eb = bi[304];
              o32_3 = fma(eb, g3_2, o32_3);
            }
            { const double eb = bi[305];
              o32_3 = fma(eb, g3_5, o32_3);
            }
            { const double eb = bi[306];
              o32_3 = fma(eb, g3_11, o32_3);
            }
            { const double eb = bi[307];
              o32_3 = fma(eb, g3_21, o32_3);
            }
            { const double eb = bi[308];
              o33_3 = fma(eb, g3_0, o33_3);
            }
            { const double eb = bi[309];
              o33_3 = fma(eb, g3_1, o33_3);
            }
            { const double eb = bi[310];
              o33_3 = fma(eb, g3_2, o33_3);
            }
            { const double eb = bi[311];
              o33_3 = fma(eb, g3_5, o33_3);
            }
            { const double eb = bi[312];
              o33_3 = fma(eb, g3_6, o33_3);
            }
            { const double eb = bi[313];
              o33_3 = fma(eb, g3_12, o33_3);
            }
            { const double eb = bi[314];
              o33_3 = fma(eb, g3_3, o33_3);
            }
            { const double eb = bi[315];
              o33_3 = fma(eb, g3_7, o33_3);
            }
            { const double eb = bi[316];
              o33_3 = fma(eb, g3_8, o33_3);
            }
            { const double eb = bi[317];
              o33_3 = fma(eb, g3_15, o33_3);
            }
            { const double eb = bi[318];
              o33_3 = fma(eb, g3_16, o33_3);
            }
            { const double eb = bi[319];
              o33_3 = fma(eb, g3_27, o33_3);
            }
            { const double eb = bi[320];
              o34_3 = fma(eb, g3_0, o34_3);
            }
            { const double eb = bi[321];
              o34_3 = fma(eb, g3_1, o34_3);
            }
            { const double eb = bi[322];
              o34_3 = fma(eb, g3_4, o34_3);
            }
            { const double eb = bi[323];
              o34_3 = fma(eb, g3_2, o34_3);
            }
            { const double eb = bi[324];
              o34_3 = fma(eb, g3_5, o34_3);
            }
            { const double eb = bi[325];
              o34_3 = fma(eb, g3_11, o34_3);
            }
            { const double eb = bi[326];
              o34_3 = fma(eb, g3_3, o34_3);
            }
            { const double eb = bi[327];
              o34_3 = fma(eb, g3_7, o34_3);
            }
            { const double eb = bi[328];
              o34_3 = fma(eb, g3_14, o34_3);
            }
            { const double eb = bi[329];
              o34_3 = fma(eb, g3_8, o34_3);
            }
            { const double eb = bi[330];
              o34_3 = fma(eb, g3_15, o34_3);
            }
            { const double eb = bi[331];
              o34_3 = fma(eb, g3_26, o34_3);
            }
            { const double eb = bi[332];
              o35_3 = fma(eb, g3_0, o35_3);
            }
            { const double eb = bi[333];
              o35_3 = fma(eb, g3_1, o35_3);
            }
            { const double eb = bi[334];
              o35_3 = fma(eb, g3_4, o35_3);
            }
            { const double eb = bi[335];
              o35_3 = fma(eb, g3_2, o35_3);
            }
            { const double eb = bi[336];
              o35_3 = fma(eb, g3_5, o35_3);
            }
            { const double eb = bi[337];
              o35_3 = fma(eb, g3_11, o35_3);
            }
            { const double eb = bi[338];
              o35_3 = fma(eb, g3_6, o35_3);
            }
            { const double eb = bi[339];
              o35_3 = fma(eb, g3_12, o35_3);
            }
            { const double eb = bi[340];
              o35_3 = fma(eb, g3_22, o35_3);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 0);
            o1_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 0);
            o2_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 0);
            o3_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 0);
            o4_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 3, fJ + 0);
            o5_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 3, fJ + 0);
            o6_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 0);
            o7_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 0);
            o8_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 0);
            o9_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 0);
            o10_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 3, fJ + 0);
            o11_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 3, fJ + 0);
            o12_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 0);
            o13_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 0);
            o14_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 0);
            o15_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 0);
            o16_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 3, fJ + 0);
            o17_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 3, fJ + 0);
            o18_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 0);
            o19_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 0);
            o20_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 0);
            o21_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 0);
            o22_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 3, fJ + 0);
            o23_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 3, fJ + 0);
            o24_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 0);
            o25_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 0);
            o26_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 0);
            o27_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 0);
            o28_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 3, fJ + 0);
            o29_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 3, fJ + 0);
            o30_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 0);
            o31_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 0);
            o32_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 0);
            o33_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 0);
            o34_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 3, fJ + 0);
            o35_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 3, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o1_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o2_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o3_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o4_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o5_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o6_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o7_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o8_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o9_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o10_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o11_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o12_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o13_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o14_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o15_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o16_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o17_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o18_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o19_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o20_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o21_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o22_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o23_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o24_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o25_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o26_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o27_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o28_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o29_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o30_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o31_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o32_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o33_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o34_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o35_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 3, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk3 = PT[(fI + 3) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 0) * N + fQ + 4];
            const double ptb5 = PT[(fP + 0) * N + fQ + 5];
            const double ptb6 = PT[(fP + 1) * N + fQ + 0];
            const double ptb7 = PT[(fP + 1) * N + fQ + 1];
            const double ptb8 = PT[(fP + 1) * N + fQ + 2];
            const double ptb9 = PT[(fP + 1) * N + fQ + 3];
            const double ptb10 = PT[(fP + 1) * N + fQ + 4];
            const double ptb11 = PT[(fP + 1) * N + fQ + 5];
            const double ptb12 = PT[(fP + 2) * N + fQ + 0];
            const double ptb13 = PT[(fP + 2) * N + fQ + 1];
            const double ptb14 = PT[(fP + 2) * N + fQ + 2];
            const double ptb15 = PT[(fP + 2) * N + fQ + 3];
            const double ptb16 = PT[(fP + 2) * N + fQ + 4];
            const double ptb17 = PT[(fP + 2) * N + fQ + 5];
            const double ptb18 = PT[(fP + 3) * N + fQ + 0];
            const double ptb19 = PT[(fP + 3) * N + fQ + 1];
            const double ptb20 = PT[(fP + 3) * N + fQ + 2];
            const double ptb21 = PT[(fP + 3) * N + fQ + 3];
            const double ptb22 = PT[(fP + 3) * N + fQ + 4];
            const double ptb23 = PT[(fP + 3) * N + fQ + 5];
            const double ptb24 = PT[(fP + 4) * N + fQ + 0];
            const double ptb25 = PT[(fP + 4) * N + fQ + 1];
            const double ptb26 = PT[(fP + 4) * N + fQ + 2];
            const double ptb27 = PT[(fP + 4) * N + fQ + 3];
            const double ptb28 = PT[(fP + 4) * N + fQ + 4];
            const double ptb29 = PT[(fP + 4) * N + fQ + 5];
            const double ptb30 = PT[(fP + 5) * N + fQ + 0];
            const double ptb31 = PT[(fP + 5) * N + fQ + 1];
            const double ptb32 = PT[(fP + 5) * N + fQ + 2];
            const double ptb33 = PT[(fP + 5) * N + fQ + 3];
            const double ptb34 = PT[(fP + 5) * N + fQ + 4];
            const double ptb35 = PT[(fP + 5) * N + fQ + 5];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd4_0 = PA[(fQ + 4) * N + fJ + 0];
            const double Abd5_0 = PA[(fQ + 5) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_3 = PA[(fQ + 0) * N + fI + 3];
            const double Abc1_3 = PA[(fQ + 1) * N + fI + 3];
            const double Abc2_3 = PA[(fQ + 2) * N + fI + 3];
            const double Abc3_3 = PA[(fQ + 3) * N + fI + 3];
            const double Abc4_3 = PA[(fQ + 4) * N + fI + 3];
            const double Abc5_3 = PA[(fQ + 5) * N + fI + 3];
            const double Aac0_3 = PA[(fP + 0) * N + fI + 3];
            const double Aac1_3 = PA[(fP + 1) * N + fI + 3];
            const double Aac2_3 = PA[(fP + 2) * N + fI + 3];
            const double Aac3_3 = PA[(fP + 3) * N + fI + 3];
            const double Aac4_3 = PA[(fP + 4) * N + fI + 3];
            const double Aac5_3 = PA[(fP + 5) * N + fI + 3];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bbd4_0 = PB[(fQ + 4) * N + fJ + 0];
            const double Bbd5_0 = PB[(fQ + 5) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_3 = PB[(fQ + 0) * N + fI + 3];
            const double Bbc1_3 = PB[(fQ + 1) * N + fI + 3];
            const double Bbc2_3 = PB[(fQ + 2) * N + fI + 3];
            const double Bbc3_3 = PB[(fQ + 3) * N + fI + 3];
            const double Bbc4_3 = PB[(fQ + 4) * N + fI + 3];
            const double Bbc5_3 = PB[(fQ + 5) * N + fI + 3];
            const double Bac0_3 = PB[(fP + 0) * N + fI + 3];
            const double Bac1_3 = PB[(fP + 1) * N + fI + 3];
            const double Bac2_3 = PB[(fP + 2) * N + fI + 3];
            const double Bac3_3 = PB[(fP + 3) * N + fI + 3];
            const double Bac4_3 = PB[(fP + 4) * N + fI + 3];
            const double Bac5_3 = PB[(fP + 5) * N + fI + 3];
            jab0 += o0_3 * ptk3;
            jab1 += o1_3 * ptk3;
            jab2 += o2_3 * ptk3;
            jab3 += o3_3 * ptk3;
            jab4 += o4_3 * ptk3;
            jab5 += o5_3 * ptk3;
            jab6 += o6_3 * ptk3;
            jab7 += o7_3 * ptk3;
            jab8 += o8_3 * ptk3;
            jab9 += o9_3 * ptk3;
            jab10 += o10_3 * ptk3;
            jab11 += o11_3 * ptk3;
            jab12 += o12_3 * ptk3;
            jab13 += o13_3 * ptk3;
            jab14 += o14_3 * ptk3;
            jab15 += o15_3 * ptk3;
            jab16 += o16_3 * ptk3;
            jab17 += o17_3 * ptk3;
            jab18 += o18_3 * ptk3;
            jab19 += o19_3 * ptk3;
            jab20 += o20_3 * ptk3;
            jab21 += o21_3 * ptk3;
            jab22 += o22_3 * ptk3;
            jab23 += o23_3 * ptk3;
            jab24 += o24_3 * ptk3;
            jab25 += o25_3 * ptk3;
            jab26 += o26_3 * ptk3;
            jab27 += o27_3 * ptk3;
            jab28 += o28_3 * ptk3;
            jab29 += o29_3 * ptk3;
            jab30 += o30_3 * ptk3;
            jab31 += o31_3 * ptk3;
            jab32 += o32_3 * ptk3;
            jab33 += o33_3 * ptk3;
            jab34 += o34_3 * ptk3;
            jab35 += o35_3 * ptk3;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 0, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5 + o6_3 * ptb6 + o7_3 * ptb7 + o8_3 * ptb8 + o9_3 * ptb9 + o10_3 * ptb10 + o11_3 * ptb11 + o12_3 * ptb12 + o13_3 * ptb13 + o14_3 * ptb14 + o15_3 * ptb15 + o16_3 * ptb16 + o17_3 * ptb17 + o18_3 * ptb18 + o19_3 * ptb19 + o20_3 * ptb20 + o21_3 * ptb21 + o22_3 * ptb22 + o23_3 * ptb23 + o24_3 * ptb24 + o25_3 * ptb25 + o26_3 * ptb26 + o27_3 * ptb27 + o28_3 * ptb28 + o29_3 * ptb29 + o30_3 * ptb30 + o31_3 * ptb31 + o32_3 * ptb32 + o33_3 * ptb33 + o34_3 * ptb34 + o35_3 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_3 * Abd0_0 + o1_3 * Abd1_0 + o2_3 * Abd2_0 + o3_3 * Abd3_0 + o4_3 * Abd4_0 + o5_3 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_3 * Aad0_0 + o6_3 * Aad1_0 + o12_3 * Aad2_0 + o18_3 * Aad3_0 + o24_3 * Aad4_0 + o30_3 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_3 * Abc0_3 + o1_3 * Abc1_3 + o2_3 * Abc2_3 + o3_3 * Abc3_3 + o4_3 * Abc4_3 + o5_3 * Abc5_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_3 * Aac0_3 + o6_3 * Aac1_3 + o12_3 * Aac2_3 + o18_3 * Aac3_3 + o24_3 * Aac4_3 + o30_3 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_3 * Aad0_0 + o7_3 * Aad1_0 + o13_3 * Aad2_0 + o19_3 * Aad3_0 + o25_3 * Aad4_0 + o31_3 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_3 * Aac0_3 + o7_3 * Aac1_3 + o13_3 * Aac2_3 + o19_3 * Aac3_3 + o25_3 * Aac4_3 + o31_3 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_3 * Aad0_0 + o8_3 * Aad1_0 + o14_3 * Aad2_0 + o20_3 * Aad3_0 + o26_3 * Aad4_0 + o32_3 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_3 * Aac0_3 + o8_3 * Aac1_3 + o14_3 * Aac2_3 + o20_3 * Aac3_3 + o26_3 * Aac4_3 + o32_3 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_3 * Aad0_0 + o9_3 * Aad1_0 + o15_3 * Aad2_0 + o21_3 * Aad3_0 + o27_3 * Aad4_0 + o33_3 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_3 * Aac0_3 + o9_3 * Aac1_3 + o15_3 * Aac2_3 + o21_3 * Aac3_3 + o27_3 * Aac4_3 + o33_3 * Aac5_3));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 3, deg * (o4_3 * Aad0_0 + o10_3 * Aad1_0 + o16_3 * Aad2_0 + o22_3 * Aad3_0 + o28_3 * Aad4_0 + o34_3 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_3 * Aac0_3 + o10_3 * Aac1_3 + o16_3 * Aac2_3 + o22_3 * Aac3_3 + o28_3 * Aac4_3 + o34_3 * Aac5_3));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 3, deg * (o5_3 * Aad0_0 + o11_3 * Aad1_0 + o17_3 * Aad2_0 + o23_3 * Aad3_0 + o29_3 * Aad4_0 + o35_3 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_3 * Aac0_3 + o11_3 * Aac1_3 + o17_3 * Aac2_3 + o23_3 * Aac3_3 + o29_3 * Aac4_3 + o35_3 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o6_3 * Abd0_0 + o7_3 * Abd1_0 + o8_3 * Abd2_0 + o9_3 * Abd3_0 + o10_3 * Abd4_0 + o11_3 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_3 * Abc0_3 + o7_3 * Abc1_3 + o8_3 * Abc2_3 + o9_3 * Abc3_3 + o10_3 * Abc4_3 + o11_3 * Abc5_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o12_3 * Abd0_0 + o13_3 * Abd1_0 + o14_3 * Abd2_0 + o15_3 * Abd3_0 + o16_3 * Abd4_0 + o17_3 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_3 * Abc0_3 + o13_3 * Abc1_3 + o14_3 * Abc2_3 + o15_3 * Abc3_3 + o16_3 * Abc4_3 + o17_3 * Abc5_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o18_3 * Abd0_0 + o19_3 * Abd1_0 + o20_3 * Abd2_0 + o21_3 * Abd3_0 + o22_3 * Abd4_0 + o23_3 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_3 * Abc0_3 + o19_3 * Abc1_3 + o20_3 * Abc2_3 + o21_3 * Abc3_3 + o22_3 * Abc4_3 + o23_3 * Abc5_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o24_3 * Abd0_0 + o25_3 * Abd1_0 + o26_3 * Abd2_0 + o27_3 * Abd3_0 + o28_3 * Abd4_0 + o29_3 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_3 * Abc0_3 + o25_3 * Abc1_3 + o26_3 * Abc2_3 + o27_3 * Abc3_3 + o28_3 * Abc4_3 + o29_3 * Abc5_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o30_3 * Abd0_0 + o31_3 * Abd1_0 + o32_3 * Abd2_0 + o33_3 * Abd3_0 + o34_3 * Abd4_0 + o35_3 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_3 * Abc0_3 + o31_3 * Abc1_3 + o32_3 * Abc2_3 + o33_3 * Abc3_3 + o34_3 * Abc4_3 + o35_3 * Abc5_3));
            atomicAdd(KBacc + (fP + 0) * N + fI + 3, deg * (o0_3 * Bbd0_0 + o1_3 * Bbd1_0 + o2_3 * Bbd2_0 + o3_3 * Bbd3_0 + o4_3 * Bbd4_0 + o5_3 * Bbd5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 3, deg * (o0_3 * Bad0_0 + o6_3 * Bad1_0 + o12_3 * Bad2_0 + o18_3 * Bad3_0 + o24_3 * Bad4_0 + o30_3 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_3 * Bbc0_3 + o1_3 * Bbc1_3 + o2_3 * Bbc2_3 + o3_3 * Bbc3_3 + o4_3 * Bbc4_3 + o5_3 * Bbc5_3));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_3 * Bac0_3 + o6_3 * Bac1_3 + o12_3 * Bac2_3 + o18_3 * Bac3_3 + o24_3 * Bac4_3 + o30_3 * Bac5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 3, deg * (o1_3 * Bad0_0 + o7_3 * Bad1_0 + o13_3 * Bad2_0 + o19_3 * Bad3_0 + o25_3 * Bad4_0 + o31_3 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_3 * Bac0_3 + o7_3 * Bac1_3 + o13_3 * Bac2_3 + o19_3 * Bac3_3 + o25_3 * Bac4_3 + o31_3 * Bac5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 3, deg * (o2_3 * Bad0_0 + o8_3 * Bad1_0 + o14_3 * Bad2_0 + o20_3 * Bad3_0 + o26_3 * Bad4_0 + o32_3 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_3 * Bac0_3 + o8_3 * Bac1_3 + o14_3 * Bac2_3 + o20_3 * Bac3_3 + o26_3 * Bac4_3 + o32_3 * Bac5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 3, deg * (o3_3 * Bad0_0 + o9_3 * Bad1_0 + o15_3 * Bad2_0 + o21_3 * Bad3_0 + o27_3 * Bad4_0 + o33_3 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_3 * Bac0_3 + o9_3 * Bac1_3 + o15_3 * Bac2_3 + o21_3 * Bac3_3 + o27_3 * Bac4_3 + o33_3 * Bac5_3));
            atomicAdd(KBacc + (fQ + 4) * N + fI + 3, deg * (o4_3 * Bad0_0 + o10_3 * Bad1_0 + o16_3 * Bad2_0 + o22_3 * Bad3_0 + o28_3 * Bad4_0 + o34_3 * Bad5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fJ + 0, deg * (o4_3 * Bac0_3 + o10_3 * Bac1_3 + o16_3 * Bac2_3 + o22_3 * Bac3_3 + o28_3 * Bac4_3 + o34_3 * Bac5_3));
            atomicAdd(KBacc + (fQ + 5) * N + fI + 3, deg * (o5_3 * Bad0_0 + o11_3 * Bad1_0 + o17_3 * Bad2_0 + o23_3 * Bad3_0 + o29_3 * Bad4_0 + o35_3 * Bad5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fJ + 0, deg * (o5_3 * Bac0_3 + o11_3 * Bac1_3 + o17_3 * Bac2_3 + o23_3 * Bac3_3 + o29_3 * Bac4_3 + o35_3 * Bac5_3));
            atomicAdd(KBacc + (fP + 1) * N + fI + 3, deg * (o6_3 * Bbd0_0 + o7_3 * Bbd1_0 + o8_3 * Bbd2_0 + o9_3 * Bbd3_0 + o10_3 * Bbd4_0 + o11_3 * Bbd5_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o6_3 * Bbc0_3 + o7_3 * Bbc1_3 + o8_3 * Bbc2_3 + o9_3 * Bbc3_3 + o10_3 * Bbc4_3 + o11_3 * Bbc5_3));
            atomicAdd(KBacc + (fP + 2) * N + fI + 3, deg * (o12_3 * Bbd0_0 + o13_3 * Bbd1_0 + o14_3 * Bbd2_0 + o15_3 * Bbd3_0 + o16_3 * Bbd4_0 + o17_3 * Bbd5_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o12_3 * Bbc0_3 + o13_3 * Bbc1_3 + o14_3 * Bbc2_3 + o15_3 * Bbc3_3 + o16_3 * Bbc4_3 + o17_3 * Bbc5_3));
            atomicAdd(KBacc + (fP + 3) * N + fI + 3, deg * (o18_3 * Bbd0_0 + o19_3 * Bbd1_0 + o20_3 * Bbd2_0 + o21_3 * Bbd3_0 + o22_3 * Bbd4_0 + o23_3 * Bbd5_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o18_3 * Bbc0_3 + o19_3 * Bbc1_3 + o20_3 * Bbc2_3 + o21_3 * Bbc3_3 + o22_3 * Bbc4_3 + o23_3 * Bbc5_3));
            atomicAdd(KBacc + (fP + 4) * N + fI + 3, deg * (o24_3 * Bbd0_0 + o25_3 * Bbd1_0 + o26_3 * Bbd2_0 + o27_3 * Bbd3_0 + o28_3 * Bbd4_0 + o29_3 * Bbd5_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o24_3 * Bbc0_3 + o25_3 * Bbc1_3 + o26_3 * Bbc2_3 + o27_3 * Bbc3_3 + o28_3 * Bbc4_3 + o29_3 * Bbc5_3));
            atomicAdd(KBacc + (fP + 5) * N + fI + 3, deg * (o30_3 * Bbd0_0 + o31_3 * Bbd1_0 + o32_3 * Bbd2_0 + o33_3 * Bbd3_0 + o34_3 * Bbd4_0 + o35_3 * Bbd5_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o30_3 * Bbc0_3 + o31_3 * Bbc1_3 + o32_3 * Bbc2_3 + o33_3 * Bbc3_3 + o34_3 * Bbc4_3 + o35_3 * Bbc5_3));
          }
        } break;
        case 4: {  // ket functions [4]
          double o0_4 = 0;
          double o1_4 = 0;
          double o2_4 = 0;
          double o3_4 = 0;
          double o4_4 = 0;
          double o5_4 = 0;
          double o6_4 = 0;
          double o7_4 = 0;
          double o8_4 = 0;
          double o9_4 = 0;
          double o10_4 = 0;
          double o11_4 = 0;
          double o12_4 = 0;
          double o13_4 = 0;
          double o14_4 = 0;
          double o15_4 = 0;
          double o16_4 = 0;
          double o17_4 = 0;
          double o18_4 = 0;
          double o19_4 = 0;
          double o20_4 = 0;
          double o21_4 = 0;
          double o22_4 = 0;
          double o23_4 = 0;
          double o24_4 = 0;
          double o25_4 = 0;
          double o26_4 = 0;
          double o27_4 = 0;
          double o28_4 = 0;
          double o29_4 = 0;
          double o30_4 = 0;
          double o31_4 = 0;
          double o32_4 = 0;
          double o33_4 = 0;
          double o34_4 = 0;
          double o35_4 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 341;
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
            double g4_20 = 0;
            double g4_21 = 0;
            double g4_22 = 0;
            double g4_23 = 0;
            double g4_24 = 0;
            double g4_25 = 0;
            double g4_26 = 0;
            double g4_27 = 0;
            double g4_28 = 0;
            double g4_29 = 0;
            double g4_30 = 0;
            double g4_31 = 0;
            double g4_32 = 0;
            double g4_33 = 0;
            double g4_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 26 * kS;
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
              const double ek4_0 = kj[18 * kS];
              const double ek4_1 = -kj[19 * kS];
              const double ek4_2 = -kj[20 * kS];
              const double ek4_3 = kj[21 * kS];
              g4_0 = fma(ek4_0, b0, g4_0);
              const double r0_0_0_1 = Z * b1;
              g4_1 = fma(ek4_0, r0_0_0_1, g4_1);
              g4_0 = fma(ek4_1, r0_0_0_1, g4_0);
              const double r0_0_1_0 = Y * b1;
              g4_2 = fma(ek4_0, r0_0_1_0, g4_2);
              const double r0_1_0_0 = X * b1;
              g4_3 = fma(ek4_0, r0_1_0_0, g4_3);
              g4_0 = fma(ek4_2, r0_1_0_0, g4_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g4_4 = fma(ek4_0, r0_0_0_2, g4_4);
              g4_1 = fma(ek4_1, r0_0_0_2, g4_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g4_5 = fma(ek4_0, r0_0_1_1, g4_5);
              g4_2 = fma(ek4_1, r0_0_1_1, g4_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g4_6 = fma(ek4_0, r0_0_2_0, g4_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g4_7 = fma(ek4_0, r0_1_0_1, g4_7);
              g4_3 = fma(ek4_1, r0_1_0_1, g4_3);
              g4_1 = fma(ek4_2, r0_1_0_1, g4_1);
              g4_0 = fma(ek4_3, r0_1_0_1, g4_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g4_8 = fma(ek4_0, r0_1_1_0, g4_8);
              g4_2 = fma(ek4_2, r0_1_1_0, g4_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g4_9 = fma(ek4_0, r0_2_0_0, g4_9);
              g4_3 = fma(ek4_2, r0_2_0_0, g4_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g4_10 = fma(ek4_0, r0_0_0_3, g4_10);
              g4_4 = fma(ek4_1, r0_0_0_3, g4_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g4_11 = fma(ek4_0, r0_0_1_2, g4_11);
              g4_5 = fma(ek4_1, r0_0_1_2, g4_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g4_12 = fma(ek4_0, r0_0_2_1, g4_12);
              g4_6 = fma(ek4_1, r0_0_2_1, g4_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g4_13 = fma(ek4_0, r0_0_3_0, g4_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g4_14 = fma(ek4_0, r0_1_0_2, g4_14);
              g4_7 = fma(ek4_1, r0_1_0_2, g4_7);
              g4_4 = fma(ek4_2, r0_1_0_2, g4_4);
              g4_1 = fma(ek4_3, r0_1_0_2, g4_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g4_15 = fma(ek4_0, r0_1_1_1, g4_15);
              g4_8 = fma(ek4_1, r0_1_1_1, g4_8);
              g4_5 = fma(ek4_2, r0_1_1_1, g4_5);
              g4_2 = fma(ek4_3, r0_1_1_1, g4_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g4_16 = fma(ek4_0, r0_1_2_0, g4_16);
              g4_6 = fma(ek4_2, r0_1_2_0, g4_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g4_17 = fma(ek4_0, r0_2_0_1, g4_17);
              g4_9 = fma(ek4_1, r0_2_0_1, g4_9);
              g4_7 = fma(ek4_2, r0_2_0_1, g4_7);
              g4_3 = fma(ek4_3, r0_2_0_1, g4_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g4_18 = fma(ek4_0, r0_2_1_0, g4_18);
              g4_8 = fma(ek4_2, r0_2_1_0, g4_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g4_19 = fma(ek4_0, r0_3_0_0, g4_19);
              g4_9 = fma(ek4_2, r0_3_0_0, g4_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g4_20 = fma(ek4_0, r0_0_0_4, g4_20);
              g4_10 = fma(ek4_1, r0_0_0_4, g4_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g4_21 = fma(ek4_0, r0_0_1_3, g4_21);
              g4_11 = fma(ek4_1, r0_0_1_3, g4_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g4_22 = fma(ek4_0, r0_0_2_2, g4_22);
              g4_12 = fma(ek4_1, r0_0_2_2, g4_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g4_23 = fma(ek4_0, r0_0_3_1, g4_23);
              g4_13 = fma(ek4_1, r0_0_3_1, g4_13);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g4_24 = fma(ek4_0, r0_0_4_0, g4_24);
              const double r0_1_0_3 = X * r1_0_0_3;
              g4_25 = fma(ek4_0, r0_1_0_3, g4_25);
              g4_14 = fma(ek4_1, r0_1_0_3, g4_14);
              g4_10 = fma(ek4_2, r0_1_0_3, g4_10);
              g4_4 = fma(ek4_3, r0_1_0_3, g4_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g4_26 = fma(ek4_0, r0_1_1_2, g4_26);
              g4_15 = fma(ek4_1, r0_1_1_2, g4_15);
              g4_11 = fma(ek4_2, r0_1_1_2, g4_11);
              g4_5 = fma(ek4_3, r0_1_1_2, g4_5);
              const double r0_1_2_1 = X * r1_0_2_1;
              g4_27 = fma(ek4_0, r0_1_2_1, g4_27);
              g4_16 = fma(ek4_1, r0_1_2_1, g4_16);
              g4_12 = fma(ek4_2, r0_1_2_1, g4_12);
              g4_6 = fma(ek4_3, r0_1_2_1, g4_6);
              const double r0_1_3_0 = X * r1_0_3_0;
              g4_28 = fma(ek4_0, r0_1_3_0, g4_28);
              g4_13 = fma(ek4_2, r0_1_3_0, g4_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g4_29 = fma(ek4_0, r0_2_0_2, g4_29);
              g4_17 = fma(ek4_1, r0_2_0_2, g4_17);
              g4_14 = fma(ek4_2, r0_2_0_2, g4_14);
              g4_7 = fma(ek4_3, r0_2_0_2, g4_7);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g4_30 = fma(ek4_0, r0_2_1_1, g4_30);
              g4_18 = fma(ek4_1, r0_2_1_1, g4_18);
              g4_15 = fma(ek4_2, r0_2_1_1, g4_15);
              g4_8 = fma(ek4_3, r0_2_1_1, g4_8);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g4_31 = fma(ek4_0, r0_2_2_0, g4_31);
              g4_16 = fma(ek4_2, r0_2_2_0, g4_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g4_32 = fma(ek4_0, r0_3_0_1, g4_32);
              g4_19 = fma(ek4_1, r0_3_0_1, g4_19);
              g4_17 = fma(ek4_2, r0_3_0_1, g4_17);
              g4_9 = fma(ek4_3, r0_3_0_1, g4_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g4_33 = fma(ek4_0, r0_3_1_0, g4_33);
              g4_18 = fma(ek4_2, r0_3_1_0, g4_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g4_34 = fma(ek4_0, r0_4_0_0, g4_34);
              g4_19 = fma(ek4_2, r0_4_0_0, g4_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g4_20 = fma(ek4_1, r0_0_0_5, g4_20);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g4_21 = fma(ek4_1, r0_0_1_4, g4_21);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g4_22 = fma(ek4_1, r0_0_2_3, g4_22);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g4_23 = fma(ek4_1, r0_0_3_2, g4_23);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g4_24 = fma(ek4_1, r0_0_4_1, g4_24);
              const double r0_1_0_4 = X * r1_0_0_4;
              g4_25 = fma(ek4_1, r0_1_0_4, g4_25);
              g4_20 = fma(ek4_2, r0_1_0_4, g4_20);
              g4_10 = fma(ek4_3, r0_1_0_4, g4_10);
              const double r0_1_1_3 = X * r1_0_1_3;
              g4_26 = fma(ek4_1, r0_1_1_3, g4_26);
              g4_21 = fma(ek4_2, r0_1_1_3, g4_21);
              g4_11 = fma(ek4_3, r0_1_1_3, g4_11);
              const double r0_1_2_2 = X * r1_0_2_2;
              g4_27 = fma(ek4_1, r0_1_2_2, g4_27);
              g4_22 = fma(ek4_2, r0_1_2_2, g4_22);
              g4_12 = fma(ek4_3, r0_1_2_2, g4_12);
              const double r0_1_3_1 = X * r1_0_3_1;
              g4_28 = fma(ek4_1, r0_1_3_1, g4_28);
              g4_23 = fma(ek4_2, r0_1_3_1, g4_23);
              g4_13 = fma(ek4_3, r0_1_3_1, g4_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g4_24 = fma(ek4_2, r0_1_4_0, g4_24);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g4_29 = fma(ek4_1, r0_2_0_3, g4_29);
              g4_25 = fma(ek4_2, r0_2_0_3, g4_25);
              g4_14 = fma(ek4_3, r0_2_0_3, g4_14);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g4_30 = fma(ek4_1, r0_2_1_2, g4_30);
              g4_26 = fma(ek4_2, r0_2_1_2, g4_26);
              g4_15 = fma(ek4_3, r0_2_1_2, g4_15);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g4_31 = fma(ek4_1, r0_2_2_1, g4_31);
              g4_27 = fma(ek4_2, r0_2_2_1, g4_27);
              g4_16 = fma(ek4_3, r0_2_2_1, g4_16);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g4_28 = fma(ek4_2, r0_2_3_0, g4_28);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g4_32 = fma(ek4_1, r0_3_0_2, g4_32);
              g4_29 = fma(ek4_2, r0_3_0_2, g4_29);
              g4_17 = fma(ek4_3, r0_3_0_2, g4_17);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g4_33 = fma(ek4_1, r0_3_1_1, g4_33);
              g4_30 = fma(ek4_2, r0_3_1_1, g4_30);
              g4_18 = fma(ek4_3, r0_3_1_1, g4_18);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g4_31 = fma(ek4_2, r0_3_2_0, g4_31);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g4_34 = fma(ek4_1, r0_4_0_1, g4_34);
              g4_32 = fma(ek4_2, r0_4_0_1, g4_32);
              g4_19 = fma(ek4_3, r0_4_0_1, g4_19);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g4_33 = fma(ek4_2, r0_4_1_0, g4_33);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g4_34 = fma(ek4_2, r0_5_0_0, g4_34);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_1_0_5 = X * r1_0_0_5;
              g4_20 = fma(ek4_3, r0_1_0_5, g4_20);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_1_1_4 = X * r1_0_1_4;
              g4_21 = fma(ek4_3, r0_1_1_4, g4_21);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_1_2_3 = X * r1_0_2_3;
              g4_22 = fma(ek4_3, r0_1_2_3, g4_22);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_1_3_2 = X * r1_0_3_2;
              g4_23 = fma(ek4_3, r0_1_3_2, g4_23);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_1_4_1 = X * r1_0_4_1;
              g4_24 = fma(ek4_3, r0_1_4_1, g4_24);
              const double r1_1_0_4 = X * r2_0_0_4;
              const double r0_2_0_4 = fma(X, r1_1_0_4, r1_0_0_4);
              g4_25 = fma(ek4_3, r0_2_0_4, g4_25);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g4_26 = fma(ek4_3, r0_2_1_3, g4_26);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g4_27 = fma(ek4_3, r0_2_2_2, g4_27);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g4_28 = fma(ek4_3, r0_2_3_1, g4_28);
              const double r2_1_0_3 = X * r3_0_0_3;
              const double r1_2_0_3 = fma(X, r2_1_0_3, r2_0_0_3);
              const double r0_3_0_3 = fma(X, r1_2_0_3, 2.0 * r1_1_0_3);
              g4_29 = fma(ek4_3, r0_3_0_3, g4_29);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g4_30 = fma(ek4_3, r0_3_1_2, g4_30);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g4_31 = fma(ek4_3, r0_3_2_1, g4_31);
              const double r3_1_0_2 = X * r4_0_0_2;
              const double r2_2_0_2 = fma(X, r3_1_0_2, r3_0_0_2);
              const double r1_3_0_2 = fma(X, r2_2_0_2, 2.0 * r2_1_0_2);
              const double r0_4_0_2 = fma(X, r1_3_0_2, 3.0 * r1_2_0_2);
              g4_32 = fma(ek4_3, r0_4_0_2, g4_32);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g4_33 = fma(ek4_3, r0_4_1_1, g4_33);
              const double r4_1_0_1 = X * r5_0_0_1;
              const double r3_2_0_1 = fma(X, r4_1_0_1, r4_0_0_1);
              const double r2_3_0_1 = fma(X, r3_2_0_1, 2.0 * r3_1_0_1);
              const double r1_4_0_1 = fma(X, r2_3_0_1, 3.0 * r2_2_0_1);
              const double r0_5_0_1 = fma(X, r1_4_0_1, 4.0 * r1_3_0_1);
              g4_34 = fma(ek4_3, r0_5_0_1, g4_34);
            }
            { const double eb = bi[5];
              o0_4 = fma(eb, g4_0, o0_4);
            }
            { const double eb = bi[6];
              o0_4 = fma(eb, g4_3, o0_4);
            }
            { const double eb = bi[7];
              o0_4 = fma(eb, g4_9, o0_4);
            }
            { const double eb = bi[8];
              o0_4 = fma(eb, g4_19, o0_4);
            }
            { const double eb = bi[9];
              o0_4 = fma(eb, g4_34, o0_4);
            }
            { const double eb = bi[10];
              o1_4 = fma(eb, g4_0, o1_4);
            }
            { const double eb = bi[11];
              o1_4 = fma(eb, g4_2, o1_4);
            }
            { const double eb = bi[12];
              o1_4 = fma(eb, g4_6, o1_4);
            }
            { const double eb = bi[13];
              o1_4 = fma(eb, g4_3, o1_4);
            }
            { const double eb = bi[14];
              o1_4 = fma(eb, g4_8, o1_4);
            }
            { const double eb = bi[15];
              o1_4 = fma(eb, g4_16, o1_4);
            }
            { const double eb = bi[16];
              o1_4 = fma(eb, g4_9, o1_4);
            }
            { const double eb = bi[17];
              o1_4 = fma(eb, g4_18, o1_4);
            }
            { const double eb = bi[18];
              o1_4 = fma(eb, g4_31, o1_4);
            }
            { const double eb = bi[19];
              o2_4 = fma(eb, g4_0, o2_4);
            }
            { const double eb = bi[20];
              o2_4 = fma(eb, g4_1, o2_4);
            }
            { const double eb = bi[21];
              o2_4 = fma(eb, g4_4, o2_4);
            }
            { const double eb = bi[22];
              o2_4 = fma(eb, g4_3, o2_4);
            }
            { const double eb = bi[23];
              o2_4 = fma(eb, g4_7, o2_4);
            }
            { const double eb = bi[24];
              o2_4 = fma(eb, g4_14, o2_4);
            }
            { const double eb = bi[25];
              o2_4 = fma(eb, g4_9, o2_4);
            }
            { const double eb = bi[26];
              o2_4 = fma(eb, g4_17, o2_4);
            }
            { const double eb = bi[27];
              o2_4 = fma(eb, g4_29, o2_4);
            }
            { const double eb = bi[28];
              o3_4 = fma(eb, g4_0, o3_4);
            }
            { const double eb = bi[29];
              o3_4 = fma(eb, g4_2, o3_4);
            }
            { const double eb = bi[30];
              o3_4 = fma(eb, g4_3, o3_4);
            }
            { const double eb = bi[31];
              o3_4 = fma(eb, g4_8, o3_4);
            }
            { const double eb = bi[32];
              o3_4 = fma(eb, g4_9, o3_4);
            }
            { const double eb = bi[33];
              o3_4 = fma(eb, g4_18, o3_4);
            }
            { const double eb = bi[34];
              o3_4 = fma(eb, g4_19, o3_4);
            }
            { const double eb = bi[35];
              o3_4 = fma(eb, g4_33, o3_4);
            }
            { const double eb = bi[36];
              o4_4 = fma(eb, g4_0, o4_4);
            }
            { const double eb = bi[37];
              o4_4 = fma(eb, g4_1, o4_4);
            }
            { const double eb = bi[38];
              o4_4 = fma(eb, g4_3, o4_4);
            }
            { const double eb = bi[39];
              o4_4 = fma(eb, g4_7, o4_4);
            }
            { const double eb = bi[40];
              o4_4 = fma(eb, g4_9, o4_4);
            }
            { const double eb = bi[41];
              o4_4 = fma(eb, g4_17, o4_4);
            }
            { const double eb = bi[42];
              o4_4 = fma(eb, g4_19, o4_4);
            }
            { const double eb = bi[43];
              o4_4 = fma(eb, g4_32, o4_4);
            }
            { const double eb = bi[44];
              o5_4 = fma(eb, g4_0, o5_4);
            }
            { const double eb = bi[45];
              o5_4 = fma(eb, g4_1, o5_4);
            }
            { const double eb = bi[46];
              o5_4 = fma(eb, g4_2, o5_4);
            }
            { const double eb = bi[47];
              o5_4 = fma(eb, g4_5, o5_4);
            }
            { const double eb = bi[48];
              o5_4 = fma(eb, g4_3, o5_4);
            }
            { const double eb = bi[49];
              o5_4 = fma(eb, g4_7, o5_4);
            }
            { const double eb = bi[50];
              o5_4 = fma(eb, g4_8, o5_4);
            }
            { const double eb = bi[51];
              o5_4 = fma(eb, g4_15, o5_4);
            }
            { const double eb = bi[52];
              o5_4 = fma(eb, g4_9, o5_4);
            }
            { const double eb = bi[53];
              o5_4 = fma(eb, g4_17, o5_4);
            }
            { const double eb = bi[54];
              o5_4 = fma(eb, g4_18, o5_4);
            }
            { const double eb = bi[55];
              o5_4 = fma(eb, g4_30, o5_4);
            }
            { const double eb = bi[56];
              o6_4 = fma(eb, g4_0, o6_4);
            }
            { const double eb = bi[57];
              o6_4 = fma(eb, g4_2, o6_4);
            }
            { const double eb = bi[58];
              o6_4 = fma(eb, g4_6, o6_4);
            }
            { const double eb = bi[59];
              o6_4 = fma(eb, g4_3, o6_4);
            }
            { const double eb = bi[60];
              o6_4 = fma(eb, g4_8, o6_4);
            }
            { const double eb = bi[61];
              o6_4 = fma(eb, g4_16, o6_4);
            }
            { const double eb = bi[62];
              o6_4 = fma(eb, g4_9, o6_4);
            }
            { const double eb = bi[63];
              o6_4 = fma(eb, g4_18, o6_4);
            }
            { const double eb = bi[64];
              o6_4 = fma(eb, g4_31, o6_4);
            }
            { const double eb = bi[65];
              o7_4 = fma(eb, g4_0, o7_4);
            }
            { const double eb = bi[66];
              o7_4 = fma(eb, g4_2, o7_4);
            }
            { const double eb = bi[67];
              o7_4 = fma(eb, g4_6, o7_4);
            }
            { const double eb = bi[68];
              o7_4 = fma(eb, g4_13, o7_4);
            }
            { const double eb = bi[69];
              o7_4 = fma(eb, g4_24, o7_4);
            }
            { const double eb = bi[70];
              o8_4 = fma(eb, g4_0, o8_4);
            }
            { const double eb = bi[71];
              o8_4 = fma(eb, g4_1, o8_4);
            }
            { const double eb = bi[72];
              o8_4 = fma(eb, g4_4, o8_4);
            }
            { const double eb = bi[73];
              o8_4 = fma(eb, g4_2, o8_4);
            }
            { const double eb = bi[74];
              o8_4 = fma(eb, g4_5, o8_4);
            }
            { const double eb = bi[75];
              o8_4 = fma(eb, g4_11, o8_4);
            }
            { const double eb = bi[76];
              o8_4 = fma(eb, g4_6, o8_4);
            }
            { const double eb = bi[77];
              o8_4 = fma(eb, g4_12, o8_4);
            }
            { const double eb = bi[78];
              o8_4 = fma(eb, g4_22, o8_4);
            }
            { const double eb = bi[79];
              o9_4 = fma(eb, g4_0, o9_4);
            }
            { const double eb = bi[80];
              o9_4 = fma(eb, g4_2, o9_4);
            }
            { const double eb = bi[81];
              o9_4 = fma(eb, g4_6, o9_4);
            }
            { const double eb = bi[82];
              o9_4 = fma(eb, g4_13, o9_4);
            }
            { const double eb = bi[83];
              o9_4 = fma(eb, g4_3, o9_4);
            }
            { const double eb = bi[84];
              o9_4 = fma(eb, g4_8, o9_4);
            }
            { const double eb = bi[85];
              o9_4 = fma(eb, g4_16, o9_4);
            }
            { const double eb = bi[86];
              o9_4 = fma(eb, g4_28, o9_4);
            }
            { const double eb = bi[87];
              o10_4 = fma(eb, g4_0, o10_4);
            }
            { const double eb = bi[88];
              o10_4 = fma(eb, g4_1, o10_4);
            }
            { const double eb = bi[89];
              o10_4 = fma(eb, g4_2, o10_4);
            }
            { const double eb = bi[90];
              o10_4 = fma(eb, g4_5, o10_4);
            }
            { const double eb = bi[91];
              o10_4 = fma(eb, g4_6, o10_4);
            }
            { const double eb = bi[92];
              o10_4 = fma(eb, g4_12, o10_4);
            }
            { const double eb = bi[93];
              o10_4 = fma(eb, g4_3, o10_4);
            }
            { const double eb = bi[94];
              o10_4 = fma(eb, g4_7, o10_4);
            }
            { const double eb = bi[95];
              o10_4 = fma(eb, g4_8, o10_4);
            }
            { const double eb = bi[96];
              o10_4 = fma(eb, g4_15, o10_4);
            }
            { const double eb = bi[97];
              o10_4 = fma(eb, g4_16, o10_4);
            }
            { const double eb = bi[98];
              o10_4 = fma(eb, g4_27, o10_4);
            }
            { const double eb = bi[99];
              o11_4 = fma(eb, g4_0, o11_4);
            }
            { const double eb = bi[100];
              o11_4 = fma(eb, g4_1, o11_4);
            }
            { const double eb = bi[101];
              o11_4 = fma(eb, g4_2, o11_4);
            }
            { const double eb = bi[102];
              o11_4 = fma(eb, g4_5, o11_4);
            }
            { const double eb = bi[103];
              o11_4 = fma(eb, g4_6, o11_4);
            }
            { const double eb = bi[104];
              o11_4 = fma(eb, g4_12, o11_4);
            }
            { const double eb = bi[105];
              o11_4 = fma(eb, g4_13, o11_4);
            }
            { const double eb = bi[106];
              o11_4 = fma(eb, g4_23, o11_4);
            }
            { const double eb = bi[107];
              o12_4 = fma(eb, g4_0, o12_4);
            }
            { const double eb = bi[108];
              o12_4 = fma(eb, g4_1, o12_4);
            }
            { const double eb = bi[109];
              o12_4 = fma(eb, g4_4, o12_4);
            }
            { const double eb = bi[110];
              o12_4 = fma(eb, g4_3, o12_4);
            }
            { const double eb = bi[111];
              o12_4 = fma(eb, g4_7, o12_4);
            }
            { const double eb = bi[112];
              o12_4 = fma(eb, g4_14, o12_4);
            }
            { const double eb = bi[113];
              o12_4 = fma(eb, g4_9, o12_4);
            }
            { const double eb = bi[114];
              o12_4 = fma(eb, g4_17, o12_4);
            }
            { const double eb = bi[115];
              o12_4 = fma(eb, g4_29, o12_4);
            }
            { const double eb = bi[116];
              o13_4 = fma(eb, g4_0, o13_4);
            }
            { const double eb = bi[117];
              o13_4 = fma(eb, g4_1, o13_4);
            }
            { const double eb = bi[118];
              o13_4 = fma(eb, g4_4, o13_4);
            }
            { const double eb = bi[119];
              o13_4 = fma(eb, g4_2, o13_4);
            }
            { const double eb = bi[120];
              o13_4 = fma(eb, g4_5, o13_4);
            }
            { const double eb = bi[121];
              o13_4 = fma(eb, g4_11, o13_4);
            }
            { const double eb = bi[122];
              o13_4 = fma(eb, g4_6, o13_4);
            }
            { const double eb = bi[123];
              o13_4 = fma(eb, g4_12, o13_4);
            }
            { const double eb = bi[124];
              o13_4 = fma(eb, g4_22, o13_4);
            }
            { const double eb = bi[125];
              o14_4 = fma(eb, g4_0, o14_4);
            }
            { const double eb = bi[126];
              o14_4 = fma(eb, g4_1, o14_4);
            }
            { const double eb = bi[127];
              o14_4 = fma(eb, g4_4, o14_4);
            }
            { const double eb = bi[128];
              o14_4 = fma(eb, g4_10, o14_4);
            }
            { const double eb = bi[129];
              o14_4 = fma(eb, g4_20, o14_4);
            }
            { const double eb = bi[130];
              o15_4 = fma(eb, g4_0, o15_4);
            }
            { const double eb = bi[131];
              o15_4 = fma(eb, g4_1, o15_4);
            }
            { const double eb = bi[132];
              o15_4 = fma(eb, g4_4, o15_4);
            }
            { const double eb = bi[133];
              o15_4 = fma(eb, g4_2, o15_4);
            }
            { const double eb = bi[134];
              o15_4 = fma(eb, g4_5, o15_4);
            }
            { const double eb = bi[135];
              o15_4 = fma(eb, g4_11, o15_4);
            }
            { const double eb = bi[136];
              o15_4 = fma(eb, g4_3, o15_4);
            }
            { const double eb = bi[137];
              o15_4 = fma(eb, g4_7, o15_4);
            }
            { const double eb = bi[138];
              o15_4 = fma(eb, g4_14, o15_4);
            }
            { const double eb = bi[139];
              o15_4 = fma(eb, g4_8, o15_4);
            }
            { const double eb = bi[140];
              o15_4 = fma(eb, g4_15, o15_4);
            }
            { const double eb = bi[141];
              o15_4 = fma(eb, g4_26, o15_4);
            }
            { const double eb = bi[142];
              o16_4 = fma(eb, g4_0, o16_4);
            }
            { const double eb = bi[143];
              o16_4 = fma(eb, g4_1, o16_4);
            }
            { const double eb = bi[144];
              o16_4 = fma(eb, g4_4, o16_4);
            }
            { const double eb = bi[145];
              o16_4 = fma(eb, g4_10, o16_4);
            }
            { const double eb = bi[146];
              o16_4 = fma(eb, g4_3, o16_4);
            }
            { const double eb = bi[147];
              o16_4 = fma(eb, g4_7, o16_4);
            }
            { const double eb = bi[148];
              o16_4 = fma(eb, g4_14, o16_4);
            }
            { const double eb = bi[149];
              o16_4 = fma(eb, g4_25, o16_4);
            }
            { const double eb = bi[150];
              o17_4 = fma(eb, g4_0, o17_4);
            }
            { const double eb = bi[151];
              o17_4 = fma(eb, g4_1, o17_4);
            }
            { const double eb = bi[152];
              o17_4 = fma(eb, g4_4, o17_4);
            }
            { const double eb = bi[153];
              o17_4 = fma(eb, g4_10, o17_4);
            }
            { const double eb = bi[154];
              o17_4 = fma(eb, g4_2, o17_4);
            }
            { const double eb = bi[155];
              o17_4 = fma(eb, g4_5, o17_4);
            }
            { const double eb = bi[156];
              o17_4 = fma(eb, g4_11, o17_4);
            }
            { const double eb = bi[157];
              o17_4 = fma(eb, g4_21, o17_4);
            }
            { const double eb = bi[158];
              o18_4 = fma(eb, g4_0, o18_4);
            }
            { const double eb = bi[159];
              o18_4 = fma(eb, g4_2, o18_4);
            }
            { const double eb = bi[160];
              o18_4 = fma(eb, g4_3, o18_4);
            }
            { const double eb = bi[161];
              o18_4 = fma(eb, g4_8, o18_4);
            }
            { const double eb = bi[162];
              o18_4 = fma(eb, g4_9, o18_4);
            }
            { const double eb = bi[163];
              o18_4 = fma(eb, g4_18, o18_4);
            }
            { const double eb = bi[164];
              o18_4 = fma(eb, g4_19, o18_4);
            }
            { const double eb = bi[165];
              o18_4 = fma(eb, g4_33, o18_4);
            }
            { const double eb = bi[166];
              o19_4 = fma(eb, g4_0, o19_4);
            }
            { const double eb = bi[167];
              o19_4 = fma(eb, g4_2, o19_4);
            }
            { const double eb = bi[168];
              o19_4 = fma(eb, g4_6, o19_4);
            }
            { const double eb = bi[169];
              o19_4 = fma(eb, g4_13, o19_4);
            }
            { const double eb = bi[170];
              o19_4 = fma(eb, g4_3, o19_4);
            }
            { const double eb = bi[171];
              o19_4 = fma(eb, g4_8, o19_4);
            }
            { const double eb = bi[172];
              o19_4 = fma(eb, g4_16, o19_4);
            }
            { const double eb = bi[173];
              o19_4 = fma(eb, g4_28, o19_4);
            }
            { const double eb = bi[174];
              o20_4 = fma(eb, g4_0, o20_4);
            }
            { const double eb = bi[175];
              o20_4 = fma(eb, g4_1, o20_4);
            }
            { const double eb = bi[176];
              o20_4 = fma(eb, g4_4, o20_4);
            }
            { const double eb = bi[177];
              o20_4 = fma(eb, g4_2, o20_4);
            }
            { const double eb = bi[178];
              o20_4 = fma(eb, g4_5, o20_4);
            }
            { const double eb = bi[179];
              o20_4 = fma(eb, g4_11, o20_4);
            }
            { const double eb = bi[180];
              o20_4 = fma(eb, g4_3, o20_4);
            }
            { const double eb = bi[181];
              o20_4 = fma(eb, g4_7, o20_4);
            }
            { const double eb = bi[182];
              o20_4 = fma(eb, g4_14, o20_4);
            }
            { const double eb = bi[183];
              o20_4 = fma(eb, g4_8, o20_4);
            }
            { const double eb = bi[184];
              o20_4 = fma(eb, g4_15, o20_4);
            }
            { const double eb = bi[185];
              o20_4 = fma(eb, g4_26, o20_4);
            }
            { const double eb = bi[186];
              o21_4 = fma(eb, g4_0, o21_4);
            }
            { const double eb = bi[187];
              o21_4 = fma(eb, g4_2, o21_4);
            }
            { const double eb = bi[188];
              o21_4 = fma(eb, g4_6, o21_4);
            }
            { const double eb = bi[189];
              o21_4 = fma(eb, g4_3, o21_4);
            }
            { const double eb = bi[190];
              o21_4 = fma(eb, g4_8, o21_4);
            }
            { const double eb = bi[191];
              o21_4 = fma(eb, g4_16, o21_4);
            }
            { const double eb = bi[192];
              o21_4 = fma(eb, g4_9, o21_4);
            }
            { const double eb = bi[193];
              o21_4 = fma(eb, g4_18, o21_4);
            }
            { const double eb = bi[194];
              o21_4 = fma(eb, g4_31, o21_4);
            }
            { const double eb = bi[195];
              o22_4 = fma(eb, g4_0, o22_4);
            }
            { const double eb = bi[196];
              o22_4 = fma(eb, g4_1, o22_4);
            }
            { const double eb = bi[197];
              o22_4 = fma(eb, g4_2, o22_4);
            }
            { const double eb = bi[198];
              o22_4 = fma(eb, g4_5, o22_4);
            }
            { const double eb = bi[199];
              o22_4 = fma(eb, g4_3, o22_4);
            }
            { const double eb = bi[200];
              o22_4 = fma(eb, g4_7, o22_4);
            }
            { const double eb = bi[201];
              o22_4 = fma(eb, g4_8, o22_4);
            }
            { const double eb = bi[202];
              o22_4 = fma(eb, g4_15, o22_4);
            }
            { const double eb = bi[203];
              o22_4 = fma(eb, g4_9, o22_4);
            }
            { const double eb = bi[204];
              o22_4 = fma(eb, g4_17, o22_4);
            }
            { const double eb = bi[205];
              o22_4 = fma(eb, g4_18, o22_4);
            }
            { const double eb = bi[206];
              o22_4 = fma(eb, g4_30, o22_4);
            }
            { const double eb = bi[207];
              o23_4 = fma(eb, g4_0, o23_4);
            }
            { const double eb = bi[208];
              o23_4 = fma(eb, g4_1, o23_4);
            }
            { const double eb = bi[209];
              o23_4 = fma(eb, g4_2, o23_4);
            }
            { const double eb = bi[210];
              o23_4 = fma(eb, g4_5, o23_4);
            }
            { const double eb = bi[211];
              o23_4 = fma(eb, g4_6, o23_4);
            }
            { const double eb = bi[212];
              o23_4 = fma(eb, g4_12, o23_4);
            }
            { const double eb = bi[213];
              o23_4 = fma(eb, g4_3, o23_4);
            }
            { const double eb = bi[214];
              o23_4 = fma(eb, g4_7, o23_4);
            }
            { const double eb = bi[215];
              o23_4 = fma(eb, g4_8, o23_4);
            }
            { const double eb = bi[216];
              o23_4 = fma(eb, g4_15, o23_4);
            }
            { const double eb = bi[217];
              o23_4 = fma(eb, g4_16, o23_4);
            }
            { const double eb = bi[218];
              o23_4 = fma(eb, g4_27, o23_4);
            }
            { const double eb = bi[219];
              o24_4 = fma(eb, g4_0, o24_4);
            }
            { const double eb = bi[220];
              o24_4 = fma(eb, g4_1, o24_4);
            }
            { const double eb = bi[221];
              o24_4 = fma(eb, g4_3, o24_4);
            }
            { const double eb = bi[222];
              o24_4 = fma(eb, g4_7, o24_4);
            }
            { const double eb = bi[223];
              o24_4 = fma(eb, g4_9, o24_4);
            }
            { const double eb = bi[224];
              o24_4 = fma(eb, g4_17, o24_4);
            }
            { const double eb = bi[225];
              o24_4 = fma(eb, g4_19, o24_4);
            }
            { const double eb = bi[226];
              o24_4 = fma(eb, g4_32, o24_4);
            }
            { const double eb = bi[227];
              o25_4 = fma(eb, g4_0, o25_4);
            }
            { const double eb = bi[228];
              o25_4 = fma(eb, g4_1, o25_4);
            }
            { const double eb = bi[229];
              o25_4 = fma(eb, g4_2, o25_4);
            }
            { const double eb = bi[230];
              o25_4 = fma(eb, g4_5, o25_4);
            }
            { const double eb = bi[231];
              o25_4 = fma(eb, g4_6, o25_4);
            }
            { const double eb = bi[232];
              o25_4 = fma(eb, g4_12, o25_4);
            }
            { const double eb = bi[233];
              o25_4 = fma(eb, g4_3, o25_4);
            }
            { const double eb = bi[234];
              o25_4 = fma(eb, g4_7, o25_4);
            }
            { const double eb = bi[235];
              o25_4 = fma(eb, g4_8, o25_4);
            }
            { const double eb = bi[236];
              o25_4 = fma(eb, g4_15, o25_4);
            }
            { const double eb = bi[237];
              o25_4 = fma(eb, g4_16, o25_4);
            }
            { const double eb = bi[238];
              o25_4 = fma(eb, g4_27, o25_4);
            }
            { const double eb = bi[239];
              o26_4 = fma(eb, g4_0, o26_4);
            }
            { const double eb = bi[240];
              o26_4 = fma(eb, g4_1, o26_4);
            }
            { const double eb = bi[241];
              o26_4 = fma(eb, g4_4, o26_4);
            }
            { const double eb = bi[242];
              o26_4 = fma(eb, g4_10, o26_4);
            }
            { const double eb = bi[243];
              o26_4 = fma(eb, g4_3, o26_4);
            }
            { const double eb = bi[244];
              o26_4 = fma(eb, g4_7, o26_4);
            }
            { const double eb = bi[245];
              o26_4 = fma(eb, g4_14, o26_4);
            }
            { const double eb = bi[246];
              o26_4 = fma(eb, g4_25, o26_4);
            }
            { const double eb = bi[247];
              o27_4 = fma(eb, g4_0, o27_4);
            }
            { const double eb = bi[248];
              o27_4 = fma(eb, g4_1, o27_4);
            }
            { const double eb = bi[249];
              o27_4 = fma(eb, g4_2, o27_4);
            }
            { const double eb = bi[250];
              o27_4 = fma(eb, g4_5, o27_4);
            }
            { const double eb = bi[251];
              o27_4 = fma(eb, g4_3, o27_4);
            }
            { const double eb = bi[252];
              o27_4 = fma(eb, g4_7, o27_4);
            }
            { const double eb = bi[253];
              o27_4 = fma(eb, g4_8, o27_4);
            }
            { const double eb = bi[254];
              o27_4 = fma(eb, g4_15, o27_4);
            }
            { const double eb = bi[255];
              o27_4 = fma(eb, g4_9, o27_4);
            }
            { const double eb = bi[256];
              o27_4 = fma(eb, g4_17, o27_4);
            }
            { const double eb = bi[257];
              o27_4 = fma(eb, g4_18, o27_4);
            }
            { const double eb = bi[258];
              o27_4 = fma(eb, g4_30, o27_4);
            }
            { const double eb = bi[259];
              o28_4 = fma(eb, g4_0, o28_4);
            }
            { const double eb = bi[260];
              o28_4 = fma(eb, g4_1, o28_4);
            }
            { const double eb = bi[261];
              o28_4 = fma(eb, g4_4, o28_4);
            }
            { const double eb = bi[262];
              o28_4 = fma(eb, g4_3, o28_4);
            }
            { const double eb = bi[263];
              o28_4 = fma(eb, g4_7, o28_4);
            }
            { const double eb = bi[264];
              o28_4 = fma(eb, g4_14, o28_4);
            }
            { const double eb = bi[265];
              o28_4 = fma(eb, g4_9, o28_4);
            }
            { const double eb = bi[266];
              o28_4 = fma(eb, g4_17, o28_4);
            }
            { const double eb = bi[267];
              o28_4 = fma(eb, g4_29, o28_4);
            }
            { const double eb = bi[268];
              o29_4 = fma(eb, g4_0, o29_4);
            }
            { const double eb = bi[269];
              o29_4 = fma(eb, g4_1, o29_4);
            }
            { const double eb = bi[270];
              o29_4 = fma(eb, g4_4, o29_4);
            }
            { const double eb = bi[271];
              o29_4 = fma(eb, g4_2, o29_4);
            }
            { const double eb = bi[272];
              o29_4 = fma(eb, g4_5, o29_4);
            }
            { const double eb = bi[273];
              o29_4 = fma(eb, g4_11, o29_4);
            }
            { const double eb = bi[274];
              o29_4 = fma(eb, g4_3, o29_4);
            }
            { const double eb = bi[275];
              o29_4 = fma(eb, g4_7, o29_4);
            }
            { const double eb = bi[276];
              o29_4 = fma(eb, g4_14, o29_4);
            }
            { const double eb = bi[277];
              o29_4 = fma(eb, g4_8, o29_4);
            }
            { const double eb = bi[278];
              o29_4 = fma(eb, g4_15, o29_4);
            }
            { const double eb = bi[279];
              o29_4 = fma(eb, g4_26, o29_4);
            }
            { const double eb = bi[280];
              o30_4 = fma(eb, g4_0, o30_4);
            }
            { const double eb = bi[281];
              o30_4 = fma(eb, g4_1, o30_4);
            }
            { const double eb = bi[282];
              o30_4 = fma(eb, g4_2, o30_4);
            }
            { const double eb = bi[283];
              o30_4 = fma(eb, g4_5, o30_4);
            }
            { const double eb = bi[284];
              o30_4 = fma(eb, g4_3, o30_4);
            }
            { const double eb = bi[285];
              o30_4 = fma(eb, g4_7, o30_4);
            }
            { const double eb = bi[286];
              o30_4 = fma(eb, g4_8, o30_4);
            }
            { const double eb = bi[287];
              o30_4 = fma(eb, g4_15, o30_4);
            }
            { const double eb = bi[288];
              o30_4 = fma(eb, g4_9, o30_4);
            }
            { const double eb = bi[289];
              o30_4 = fma(eb, g4_17, o30_4);
            }
            { const double eb = bi[290];
              o30_4 = fma(eb, g4_18, o30_4);
            }
            { const double eb = bi[291];
              o30_4 = fma(eb, g4_30, o30_4);
            }
            { const double eb = bi[292];
              o31_4 = fma(eb, g4_0, o31_4);
            }
            { const double eb = bi[293];
              o31_4 = fma(eb, g4_1, o31_4);
            }
            { const double eb = bi[294];
              o31_4 = fma(eb, g4_2, o31_4);
            }
            { const double eb = bi[295];
              o31_4 = fma(eb, g4_5, o31_4);
            }
            { const double eb = bi[296];
              o31_4 = fma(eb, g4_6, o31_4);
            }
            { const double eb = bi[297];
              o31_4 = fma(eb, g4_12, o31_4);
            }
            { const double eb = bi[298];
              o31_4 = fma(eb, g4_13, o31_4);
            }
            { const double eb = bi[299];
              o31_4 = fma(eb, g4_23, o31_4);
            }
            { const double eb = bi[300];
              o32_4 = fma(eb, g4_0, o32_4);
            }
            { const double eb = bi[301];
              o32_4 = fma(eb, g4_1, o32_4);
            }
            { const double eb = bi[302];
              o32_4 = fma(eb, g4_4, o32_4);
            }
            { const double eb = bi[303];
              o32_4 = fma(eb, g4_10, o32_4);
            }
            { const double eb = bi[304];
              o32_4 = fma(eb, g4_2, o32_4);
            }
            { const double eb = bi[305];
              o32_4 = fma(eb, g4_5, o32_4);
            }
            { const double eb = bi[306];
              o32_4 = fma(eb, g4_11, o32_4);
            }
            { const double eb = bi[307];
              o32_4 = fma(eb, g4_21, o32_4);
            }
            { const double eb = bi[308];
              o33_4 = fma(eb, g4_0, o33_4);
            }
            { const double eb = bi[309];
              o33_4 = fma(eb, g4_1, o33_4);
            }
            { const double eb = bi[310];
              o33_4 = fma(eb, g4_2, o33_4);
            }
            { const double eb = bi[311];
              o33_4 = fma(eb, g4_5, o33_4);
            }
            { const double eb = bi[312];
              o33_4 = fma(eb, g4_6, o33_4);
            }
            { const double eb = bi[313];
              o33_4 = fma(eb, g4_12, o33_4);
            }
            { const double eb = bi[314];
              o33_4 = fma(eb, g4_3, o33_4);
            }
            { const double eb = bi[315];
              o33_4 = fma(eb, g4_7, o33_4);
            }
            { const double eb = bi[316];
              o33_4 = fma(eb, g4_8, o33_4);
            }
            { const double eb = bi[317];
              o33_4 = fma(eb, g4_15, o33_4);
            }
            { const double eb = bi[318];
              o33_4 = fma(eb, g4_16, o33_4);
            }
            { const double eb = bi[319];
              o33_4 = fma(eb, g4_27, o33_4);
            }
            { const double eb = bi[320];
              o34_4 = fma(eb, g4_0, o34_4);
            }
            { const double eb = bi[321];
              o34_4 = fma(eb, g4_1, o34_4);
            }
            { const double eb = bi[322];
              o34_4 = fma(eb, g4_4, o34_4);
            }
            { const double eb = bi[323];
              o34_4 = fma(eb, g4_2, o34_4);
            }
            { const double eb = bi[324];
              o34_4 = fma(eb, g4_5, o34_4);
            }
            { const double eb = bi[325];
              o34_4 = fma(eb, g4_11, o34_4);
            }
            { const double eb = bi[326];
              o34_4 = fma(eb, g4_3, o34_4);
            }
            { const double eb = bi[327];
              o34_4 = fma(eb, g4_7, o34_4);
            }
            { const double eb = bi[328];
              o34_4 = fma(eb, g4_14, o34_4);
            }
            { const double eb = bi[329];
              o34_4 = fma(eb, g4_8, o34_4);
            }
            { const double eb = bi[330];
              o34_4 = fma(eb, g4_15, o34_4);
            }
            { const double eb = bi[331];
              o34_4 = fma(eb, g4_26, o34_4);
            }
            { const double eb = bi[332];
              o35_4 = fma(eb, g4_0, o35_4);
            }
            { const double eb = bi[333];
              o35_4 = fma(eb, g4_1, o35_4);
            }
            { const double eb = bi[334];
              o35_4 = fma(eb, g4_4, o35_4);
            }
            { const double eb = bi[335];
              o35_4 = fma(eb, g4_2, o35_4);
            }
            { const double eb = bi[336];
              o35_4 = fma(eb, g4_5, o35_4);
            }
            { const double eb = bi[337];
              o35_4 = fma(eb, g4_11, o35_4);
            }
            { const double eb = bi[338];
              o35_4 = fma(eb, g4_6, o35_4);
            }
            { const double eb = bi[339];
              o35_4 = fma(eb, g4_12, o35_4);
            }
            { const double eb = bi[340];
              o35_4 = fma(eb, g4_22, o35_4);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 4, fJ + 0);
            o1_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 4, fJ + 0);
            o2_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 4, fJ + 0);
            o3_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 4, fJ + 0);
            o4_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 4, fJ + 0);
            o5_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 4, fJ + 0);
            o6_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 4, fJ + 0);
            o7_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 4, fJ + 0);
            o8_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 4, fJ + 0);
            o9_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 4, fJ + 0);
            o10_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 4, fJ + 0);
            o11_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 4, fJ + 0);
            o12_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 4, fJ + 0);
            o13_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 4, fJ + 0);
            o14_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 4, fJ + 0);
            o15_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 4, fJ + 0);
            o16_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 4, fJ + 0);
            o17_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 4, fJ + 0);
            o18_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 4, fJ + 0);
            o19_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 4, fJ + 0);
            o20_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 4, fJ + 0);
            o21_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 4, fJ + 0);
            o22_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 4, fJ + 0);
            o23_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 4, fJ + 0);
            o24_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 4, fJ + 0);
            o25_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 4, fJ + 0);
            o26_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 4, fJ + 0);
            o27_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 4, fJ + 0);
            o28_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 4, fJ + 0);
            o29_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 4, fJ + 0);
            o30_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 4, fJ + 0);
            o31_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 4, fJ + 0);
            o32_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 4, fJ + 0);
            o33_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 4, fJ + 0);
            o34_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 4, fJ + 0);
            o35_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 4, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o1_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o2_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o3_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o4_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o5_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o6_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o7_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o8_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o9_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o10_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o11_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o12_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o13_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o14_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o15_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o16_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o17_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o18_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o19_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o20_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o21_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o22_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o23_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o24_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o25_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o26_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o27_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o28_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o29_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o30_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o31_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o32_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o33_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o34_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 4, fJ + 0)));
            e = fmax(e, fabs(o35_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 4, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk4 = PT[(fI + 4) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 0) * N + fQ + 4];
            const double ptb5 = PT[(fP + 0) * N + fQ + 5];
            const double ptb6 = PT[(fP + 1) * N + fQ + 0];
            const double ptb7 = PT[(fP + 1) * N + fQ + 1];
            const double ptb8 = PT[(fP + 1) * N + fQ + 2];
            const double ptb9 = PT[(fP + 1) * N + fQ + 3];
            const double ptb10 = PT[(fP + 1) * N + fQ + 4];
            const double ptb11 = PT[(fP + 1) * N + fQ + 5];
            const double ptb12 = PT[(fP + 2) * N + fQ + 0];
            const double ptb13 = PT[(fP + 2) * N + fQ + 1];
            const double ptb14 = PT[(fP + 2) * N + fQ + 2];
            const double ptb15 = PT[(fP + 2) * N + fQ + 3];
            const double ptb16 = PT[(fP + 2) * N + fQ + 4];
            const double ptb17 = PT[(fP + 2) * N + fQ + 5];
            const double ptb18 = PT[(fP + 3) * N + fQ + 0];
            const double ptb19 = PT[(fP + 3) * N + fQ + 1];
            const double ptb20 = PT[(fP + 3) * N + fQ + 2];
            const double ptb21 = PT[(fP + 3) * N + fQ + 3];
            const double ptb22 = PT[(fP + 3) * N + fQ + 4];
            const double ptb23 = PT[(fP + 3) * N + fQ + 5];
            const double ptb24 = PT[(fP + 4) * N + fQ + 0];
            const double ptb25 = PT[(fP + 4) * N + fQ + 1];
            const double ptb26 = PT[(fP + 4) * N + fQ + 2];
            const double ptb27 = PT[(fP + 4) * N + fQ + 3];
            const double ptb28 = PT[(fP + 4) * N + fQ + 4];
            const double ptb29 = PT[(fP + 4) * N + fQ + 5];
            const double ptb30 = PT[(fP + 5) * N + fQ + 0];
            const double ptb31 = PT[(fP + 5) * N + fQ + 1];
            const double ptb32 = PT[(fP + 5) * N + fQ + 2];
            const double ptb33 = PT[(fP + 5) * N + fQ + 3];
            const double ptb34 = PT[(fP + 5) * N + fQ + 4];
            const double ptb35 = PT[(fP + 5) * N + fQ + 5];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd4_0 = PA[(fQ + 4) * N + fJ + 0];
            const double Abd5_0 = PA[(fQ + 5) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_4 = PA[(fQ + 0) * N + fI + 4];
            const double Abc1_4 = PA[(fQ + 1) * N + fI + 4];
            const double Abc2_4 = PA[(fQ + 2) * N + fI + 4];
            const double Abc3_4 = PA[(fQ + 3) * N + fI + 4];
            const double Abc4_4 = PA[(fQ + 4) * N + fI + 4];
            const double Abc5_4 = PA[(fQ + 5) * N + fI + 4];
            const double Aac0_4 = PA[(fP + 0) * N + fI + 4];
            const double Aac1_4 = PA[(fP + 1) * N + fI + 4];
            const double Aac2_4 = PA[(fP + 2) * N + fI + 4];
            const double Aac3_4 = PA[(fP + 3) * N + fI + 4];
            const double Aac4_4 = PA[(fP + 4) * N + fI + 4];
            const double Aac5_4 = PA[(fP + 5) * N + fI + 4];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bbd4_0 = PB[(fQ + 4) * N + fJ + 0];
            const double Bbd5_0 = PB[(fQ + 5) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_4 = PB[(fQ + 0) * N + fI + 4];
            const double Bbc1_4 = PB[(fQ + 1) * N + fI + 4];
            const double Bbc2_4 = PB[(fQ + 2) * N + fI + 4];
            const double Bbc3_4 = PB[(fQ + 3) * N + fI + 4];
            const double Bbc4_4 = PB[(fQ + 4) * N + fI + 4];
            const double Bbc5_4 = PB[(fQ + 5) * N + fI + 4];
            const double Bac0_4 = PB[(fP + 0) * N + fI + 4];
            const double Bac1_4 = PB[(fP + 1) * N + fI + 4];
            const double Bac2_4 = PB[(fP + 2) * N + fI + 4];
            const double Bac3_4 = PB[(fP + 3) * N + fI + 4];
            const double Bac4_4 = PB[(fP + 4) * N + fI + 4];
            const double Bac5_4 = PB[(fP + 5) * N + fI + 4];
            jab0 += o0_4 * ptk4;
            jab1 += o1_4 * ptk4;
            jab2 += o2_4 * ptk4;
            jab3 += o3_4 * ptk4;
            jab4 += o4_4 * ptk4;
            jab5 += o5_4 * ptk4;
            jab6 += o6_4 * ptk4;
            jab7 += o7_4 * ptk4;
            jab8 += o8_4 * ptk4;
            jab9 += o9_4 * ptk4;
            jab10 += o10_4 * ptk4;
            jab11 += o11_4 * ptk4;
            jab12 += o12_4 * ptk4;
            jab13 += o13_4 * ptk4;
            jab14 += o14_4 * ptk4;
            jab15 += o15_4 * ptk4;
            jab16 += o16_4 * ptk4;
            jab17 += o17_4 * ptk4;
            jab18 += o18_4 * ptk4;
            jab19 += o19_4 * ptk4;
            jab20 += o20_4 * ptk4;
            jab21 += o21_4 * ptk4;
            jab22 += o22_4 * ptk4;
            jab23 += o23_4 * ptk4;
            jab24 += o24_4 * ptk4;
            jab25 += o25_4 * ptk4;
            jab26 += o26_4 * ptk4;
            jab27 += o27_4 * ptk4;
            jab28 += o28_4 * ptk4;
            jab29 += o29_4 * ptk4;
            jab30 += o30_4 * ptk4;
            jab31 += o31_4 * ptk4;
            jab32 += o32_4 * ptk4;
            jab33 += o33_4 * ptk4;
            jab34 += o34_4 * ptk4;
            jab35 += o35_4 * ptk4;
            atomicAdd(Jacc + (fI + 4) * N + fJ + 0, 2.0 * deg * (o0_4 * ptb0 + o1_4 * ptb1 + o2_4 * ptb2 + o3_4 * ptb3 + o4_4 * ptb4 + o5_4 * ptb5 + o6_4 * ptb6 + o7_4 * ptb7 + o8_4 * ptb8 + o9_4 * ptb9 + o10_4 * ptb10 + o11_4 * ptb11 + o12_4 * ptb12 + o13_4 * ptb13 + o14_4 * ptb14 + o15_4 * ptb15 + o16_4 * ptb16 + o17_4 * ptb17 + o18_4 * ptb18 + o19_4 * ptb19 + o20_4 * ptb20 + o21_4 * ptb21 + o22_4 * ptb22 + o23_4 * ptb23 + o24_4 * ptb24 + o25_4 * ptb25 + o26_4 * ptb26 + o27_4 * ptb27 + o28_4 * ptb28 + o29_4 * ptb29 + o30_4 * ptb30 + o31_4 * ptb31 + o32_4 * ptb32 + o33_4 * ptb33 + o34_4 * ptb34 + o35_4 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 4, deg * (o0_4 * Abd0_0 + o1_4 * Abd1_0 + o2_4 * Abd2_0 + o3_4 * Abd3_0 + o4_4 * Abd4_0 + o5_4 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 4, deg * (o0_4 * Aad0_0 + o6_4 * Aad1_0 + o12_4 * Aad2_0 + o18_4 * Aad3_0 + o24_4 * Aad4_0 + o30_4 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Abc0_4 + o1_4 * Abc1_4 + o2_4 * Abc2_4 + o3_4 * Abc3_4 + o4_4 * Abc4_4 + o5_4 * Abc5_4));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Aac0_4 + o6_4 * Aac1_4 + o12_4 * Aac2_4 + o18_4 * Aac3_4 + o24_4 * Aac4_4 + o30_4 * Aac5_4));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 4, deg * (o1_4 * Aad0_0 + o7_4 * Aad1_0 + o13_4 * Aad2_0 + o19_4 * Aad3_0 + o25_4 * Aad4_0 + o31_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Aac0_4 + o7_4 * Aac1_4 + o13_4 * Aac2_4 + o19_4 * Aac3_4 + o25_4 * Aac4_4 + o31_4 * Aac5_4));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 4, deg * (o2_4 * Aad0_0 + o8_4 * Aad1_0 + o14_4 * Aad2_0 + o20_4 * Aad3_0 + o26_4 * Aad4_0 + o32_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Aac0_4 + o8_4 * Aac1_4 + o14_4 * Aac2_4 + o20_4 * Aac3_4 + o26_4 * Aac4_4 + o32_4 * Aac5_4));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 4, deg * (o3_4 * Aad0_0 + o9_4 * Aad1_0 + o15_4 * Aad2_0 + o21_4 * Aad3_0 + o27_4 * Aad4_0 + o33_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Aac0_4 + o9_4 * Aac1_4 + o15_4 * Aac2_4 + o21_4 * Aac3_4 + o27_4 * Aac4_4 + o33_4 * Aac5_4));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 4, deg * (o4_4 * Aad0_0 + o10_4 * Aad1_0 + o16_4 * Aad2_0 + o22_4 * Aad3_0 + o28_4 * Aad4_0 + o34_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_4 * Aac0_4 + o10_4 * Aac1_4 + o16_4 * Aac2_4 + o22_4 * Aac3_4 + o28_4 * Aac4_4 + o34_4 * Aac5_4));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 4, deg * (o5_4 * Aad0_0 + o11_4 * Aad1_0 + o17_4 * Aad2_0 + o23_4 * Aad3_0 + o29_4 * Aad4_0 + o35_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_4 * Aac0_4 + o11_4 * Aac1_4 + o17_4 * Aac2_4 + o23_4 * Aac3_4 + o29_4 * Aac4_4 + o35_4 * Aac5_4));
            atomicAdd(KAacc + (fP + 1) * N + fI + 4, deg * (o6_4 * Abd0_0 + o7_4 * Abd1_0 + o8_4 * Abd2_0 + o9_4 * Abd3_0 + o10_4 * Abd4_0 + o11_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_4 * Abc0_4 + o7_4 * Abc1_4 + o8_4 * Abc2_4 + o9_4 * Abc3_4 + o10_4 * Abc4_4 + o11_4 * Abc5_4));
            atomicAdd(KAacc + (fP + 2) * N + fI + 4, deg * (o12_4 * Abd0_0 + o13_4 * Abd1_0 + o14_4 * Abd2_0 + o15_4 * Abd3_0 + o16_4 * Abd4_0 + o17_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_4 * Abc0_4 + o13_4 * Abc1_4 + o14_4 * Abc2_4 + o15_4 * Abc3_4 + o16_4 * Abc4_4 + o17_4 * Abc5_4));
            atomicAdd(KAacc + (fP + 3) * N + fI + 4, deg * (o18_4 * Abd0_0 + o19_4 * Abd1_0 + o20_4 * Abd2_0 + o21_4 * Abd3_0 + o22_4 * Abd4_0 + o23_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_4 * Abc0_4 + o19_4 * Abc1_4 + o20_4 * Abc2_4 + o21_4 * Abc3_4 + o22_4 * Abc4_4 + o23_4 * Abc5_4));
            atomicAdd(KAacc + (fP + 4) * N + fI + 4, deg * (o24_4 * Abd0_0 + o25_4 * Abd1_0 + o26_4 * Abd2_0 + o27_4 * Abd3_0 + o28_4 * Abd4_0 + o29_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_4 * Abc0_4 + o25_4 * Abc1_4 + o26_4 * Abc2_4 + o27_4 * Abc3_4 + o28_4 * Abc4_4 + o29_4 * Abc5_4));
            atomicAdd(KAacc + (fP + 5) * N + fI + 4, deg * (o30_4 * Abd0_0 + o31_4 * Abd1_0 + o32_4 * Abd2_0 + o33_4 * Abd3_0 + o34_4 * Abd4_0 + o35_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_4 * Abc0_4 + o31_4 * Abc1_4 + o32_4 * Abc2_4 + o33_4 * Abc3_4 + o34_4 * Abc4_4 + o35_4 * Abc5_4));
            atomicAdd(KBacc + (fP + 0) * N + fI + 4, deg * (o0_4 * Bbd0_0 + o1_4 * Bbd1_0 + o2_4 * Bbd2_0 + o3_4 * Bbd3_0 + o4_4 * Bbd4_0 + o5_4 * Bbd5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 4, deg * (o0_4 * Bad0_0 + o6_4 * Bad1_0 + o12_4 * Bad2_0 + o18_4 * Bad3_0 + o24_4 * Bad4_0 + o30_4 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Bbc0_4 + o1_4 * Bbc1_4 + o2_4 * Bbc2_4 + o3_4 * Bbc3_4 + o4_4 * Bbc4_4 + o5_4 * Bbc5_4));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Bac0_4 + o6_4 * Bac1_4 + o12_4 * Bac2_4 + o18_4 * Bac3_4 + o24_4 * Bac4_4 + o30_4 * Bac5_4));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 4, deg * (o1_4 * Bad0_0 + o7_4 * Bad1_0 + o13_4 * Bad2_0 + o19_4 * Bad3_0 + o25_4 * Bad4_0 + o31_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Bac0_4 + o7_4 * Bac1_4 + o13_4 * Bac2_4 + o19_4 * Bac3_4 + o25_4 * Bac4_4 + o31_4 * Bac5_4));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 4, deg * (o2_4 * Bad0_0 + o8_4 * Bad1_0 + o14_4 * Bad2_0 + o20_4 * Bad3_0 + o26_4 * Bad4_0 + o32_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Bac0_4 + o8_4 * Bac1_4 + o14_4 * Bac2_4 + o20_4 * Bac3_4 + o26_4 * Bac4_4 + o32_4 * Bac5_4));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 4, deg * (o3_4 * Bad0_0 + o9_4 * Bad1_0 + o15_4 * Bad2_0 + o21_4 * Bad3_0 + o27_4 * Bad4_0 + o33_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Bac0_4 + o9_4 * Bac1_4 + o15_4 * Bac2_4 + o21_4 * Bac3_4 + o27_4 * Bac4_4 + o33_4 * Bac5_4));
            atomicAdd(KBacc + (fQ + 4) * N + fI + 4, deg * (o4_4 * Bad0_0 + o10_4 * Bad1_0 + o16_4 * Bad2_0 + o22_4 * Bad3_0 + o28_4 * Bad4_0 + o34_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fJ + 0, deg * (o4_4 * Bac0_4 + o10_4 * Bac1_4 + o16_4 * Bac2_4 + o22_4 * Bac3_4 + o28_4 * Bac4_4 + o34_4 * Bac5_4));
            atomicAdd(KBacc + (fQ + 5) * N + fI + 4, deg * (o5_4 * Bad0_0 + o11_4 * Bad1_0 + o17_4 * Bad2_0 + o23_4 * Bad3_0 + o29_4 * Bad4_0 + o35_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fJ + 0, deg * (o5_4 * Bac0_4 + o11_4 * Bac1_4 + o17_4 * Bac2_4 + o23_4 * Bac3_4 + o29_4 * Bac4_4 + o35_4 * Bac5_4));
            atomicAdd(KBacc + (fP + 1) * N + fI + 4, deg * (o6_4 * Bbd0_0 + o7_4 * Bbd1_0 + o8_4 * Bbd2_0 + o9_4 * Bbd3_0 + o10_4 * Bbd4_0 + o11_4 * Bbd5_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o6_4 * Bbc0_4 + o7_4 * Bbc1_4 + o8_4 * Bbc2_4 + o9_4 * Bbc3_4 + o10_4 * Bbc4_4 + o11_4 * Bbc5_4));
            atomicAdd(KBacc + (fP + 2) * N + fI + 4, deg * (o12_4 * Bbd0_0 + o13_4 * Bbd1_0 + o14_4 * Bbd2_0 + o15_4 * Bbd3_0 + o16_4 * Bbd4_0 + o17_4 * Bbd5_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o12_4 * Bbc0_4 + o13_4 * Bbc1_4 + o14_4 * Bbc2_4 + o15_4 * Bbc3_4 + o16_4 * Bbc4_4 + o17_4 * Bbc5_4));
            atomicAdd(KBacc + (fP + 3) * N + fI + 4, deg * (o18_4 * Bbd0_0 + o19_4 * Bbd1_0 + o20_4 * Bbd2_0 + o21_4 * Bbd3_0 + o22_4 * Bbd4_0 + o23_4 * Bbd5_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o18_4 * Bbc0_4 + o19_4 * Bbc1_4 + o20_4 * Bbc2_4 + o21_4 * Bbc3_4 + o22_4 * Bbc4_4 + o23_4 * Bbc5_4));
            atomicAdd(KBacc + (fP + 4) * N + fI + 4, deg * (o24_4 * Bbd0_0 + o25_4 * Bbd1_0 + o26_4 * Bbd2_0 + o27_4 * Bbd3_0 + o28_4 * Bbd4_0 + o29_4 * Bbd5_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o24_4 * Bbc0_4 + o25_4 * Bbc1_4 + o26_4 * Bbc2_4 + o27_4 * Bbc3_4 + o28_4 * Bbc4_4 + o29_4 * Bbc5_4));
            atomicAdd(KBacc + (fP + 5) * N + fI + 4, deg * (o30_4 * Bbd0_0 + o31_4 * Bbd1_0 + o32_4 * Bbd2_0 + o33_4 * Bbd3_0 + o34_4 * Bbd4_0 + o35_4 * Bbd5_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o30_4 * Bbc0_4 + o31_4 * Bbc1_4 + o32_4 * Bbc2_4 + o33_4 * Bbc3_4 + o34_4 * Bbc4_4 + o35_4 * Bbc5_4));
          }
        } break;
        case 5: {  // ket functions [5]
          double o0_5 = 0;
          double o1_5 = 0;
          double o2_5 = 0;
          double o3_5 = 0;
          double o4_5 = 0;
          double o5_5 = 0;
          double o6_5 = 0;
          double o7_5 = 0;
          double o8_5 = 0;
          double o9_5 = 0;
          double o10_5 = 0;
          double o11_5 = 0;
          double o12_5 = 0;
          double o13_5 = 0;
          double o14_5 = 0;
          double o15_5 = 0;
          double o16_5 = 0;
          double o17_5 = 0;
          double o18_5 = 0;
          double o19_5 = 0;
          double o20_5 = 0;
          double o21_5 = 0;
          double o22_5 = 0;
          double o23_5 = 0;
          double o24_5 = 0;
          double o25_5 = 0;
          double o26_5 = 0;
          double o27_5 = 0;
          double o28_5 = 0;
          double o29_5 = 0;
          double o30_5 = 0;
          double o31_5 = 0;
          double o32_5 = 0;
          double o33_5 = 0;
          double o34_5 = 0;
          double o35_5 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 341;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            double g5_20 = 0;
            double g5_21 = 0;
            double g5_22 = 0;
            double g5_23 = 0;
            double g5_24 = 0;
            double g5_25 = 0;
            double g5_26 = 0;
            double g5_27 = 0;
            double g5_28 = 0;
            double g5_29 = 0;
            double g5_30 = 0;
            double g5_31 = 0;
            double g5_32 = 0;
            double g5_33 = 0;
            double g5_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 26 * kS;
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
              const double ek5_0 = kj[22 * kS];
              const double ek5_1 = -kj[23 * kS];
              const double ek5_2 = -kj[24 * kS];
              const double ek5_3 = kj[25 * kS];
              g5_0 = fma(ek5_0, b0, g5_0);
              const double r0_0_0_1 = Z * b1;
              g5_1 = fma(ek5_0, r0_0_0_1, g5_1);
              g5_0 = fma(ek5_1, r0_0_0_1, g5_0);
              const double r0_0_1_0 = Y * b1;
              g5_2 = fma(ek5_0, r0_0_1_0, g5_2);
              g5_0 = fma(ek5_2, r0_0_1_0, g5_0);
              const double r0_1_0_0 = X * b1;
              g5_3 = fma(ek5_0, r0_1_0_0, g5_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g5_4 = fma(ek5_0, r0_0_0_2, g5_4);
              g5_1 = fma(ek5_1, r0_0_0_2, g5_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g5_5 = fma(ek5_0, r0_0_1_1, g5_5);
              g5_2 = fma(ek5_1, r0_0_1_1, g5_2);
              g5_1 = fma(ek5_2, r0_0_1_1, g5_1);
              g5_0 = fma(ek5_3, r0_0_1_1, g5_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g5_6 = fma(ek5_0, r0_0_2_0, g5_6);
              g5_2 = fma(ek5_2, r0_0_2_0, g5_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g5_7 = fma(ek5_0, r0_1_0_1, g5_7);
              g5_3 = fma(ek5_1, r0_1_0_1, g5_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g5_8 = fma(ek5_0, r0_1_1_0, g5_8);
              g5_3 = fma(ek5_2, r0_1_1_0, g5_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g5_9 = fma(ek5_0, r0_2_0_0, g5_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g5_10 = fma(ek5_0, r0_0_0_3, g5_10);
              g5_4 = fma(ek5_1, r0_0_0_3, g5_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g5_11 = fma(ek5_0, r0_0_1_2, g5_11);
              g5_5 = fma(ek5_1, r0_0_1_2, g5_5);
              g5_4 = fma(ek5_2, r0_0_1_2, g5_4);
              g5_1 = fma(ek5_3, r0_0_1_2, g5_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g5_12 = fma(ek5_0, r0_0_2_1, g5_12);
              g5_6 = fma(ek5_1, r0_0_2_1, g5_6);
              g5_5 = fma(ek5_2, r0_0_2_1, g5_5);
              g5_2 = fma(ek5_3, r0_0_2_1, g5_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g5_13 = fma(ek5_0, r0_0_3_0, g5_13);
              g5_6 = fma(ek5_2, r0_0_3_0, g5_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g5_14 = fma(ek5_0, r0_1_0_2, g5_14);
              g5_7 = fma(ek5_1, r0_1_0_2, g5_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g5_15 = fma(ek5_0, r0_1_1_1, g5_15);
              g5_8 = fma(ek5_1, r0_1_1_1, g5_8);
              g5_7 = fma(ek5_2, r0_1_1_1, g5_7);
              g5_3 = fma(ek5_3, r0_1_1_1, g5_3);
              const double r0_1_2_0 = X * r1_0_2_0;
              g5_16 = fma(ek5_0, r0_1_2_0, g5_16);
              g5_8 = fma(ek5_2, r0_1_2_0, g5_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g5_17 = fma(ek5_0, r0_2_0_1, g5_17);
              g5_9 = fma(ek5_1, r0_2_0_1, g5_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g5_18 = fma(ek5_0, r0_2_1_0, g5_18);
              g5_9 = fma(ek5_2, r0_2_1_0, g5_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g5_19 = fma(ek5_0, r0_3_0_0, g5_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g5_20 = fma(ek5_0, r0_0_0_4, g5_20);
              g5_10 = fma(ek5_1, r0_0_0_4, g5_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g5_21 = fma(ek5_0, r0_0_1_3, g5_21);
              g5_11 = fma(ek5_1, r0_0_1_3, g5_11);
              g5_10 = fma(ek5_2, r0_0_1_3, g5_10);
              g5_4 = fma(ek5_3, r0_0_1_3, g5_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g5_22 = fma(ek5_0, r0_0_2_2, g5_22);
              g5_12 = fma(ek5_1, r0_0_2_2, g5_12);
              g5_11 = fma(ek5_2, r0_0_2_2, g5_11);
              g5_5 = fma(ek5_3, r0_0_2_2, g5_5);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g5_23 = fma(ek5_0, r0_0_3_1, g5_23);
              g5_13 = fma(ek5_1, r0_0_3_1, g5_13);
              g5_12 = fma(ek5_2, r0_0_3_1, g5_12);
              g5_6 = fma(ek5_3, r0_0_3_1, g5_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g5_24 = fma(ek5_0, r0_0_4_0, g5_24);
              g5_13 = fma(ek5_2, r0_0_4_0, g5_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g5_25 = fma(ek5_0, r0_1_0_3, g5_25);
              g5_14 = fma(ek5_1, r0_1_0_3, g5_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g5_26 = fma(ek5_0, r0_1_1_2, g5_26);
              g5_15 = fma(ek5_1, r0_1_1_2, g5_15);
              g5_14 = fma(ek5_2, r0_1_1_2, g5_14);
              g5_7 = fma(ek5_3, r0_1_1_2, g5_7);
              const double r0_1_2_1 = X * r1_0_2_1;
              g5_27 = fma(ek5_0, r0_1_2_1, g5_27);
              g5_16 = fma(ek5_1, r0_1_2_1, g5_16);
              g5_15 = fma(ek5_2, r0_1_2_1, g5_15);
              g5_8 = fma(ek5_3, r0_1_2_1, g5_8);
              const double r0_1_3_0 = X * r1_0_3_0;
              g5_28 = fma(ek5_0, r0_1_3_0, g5_28);
              g5_16 = fma(ek5_2, r0_1_3_0, g5_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g5_29 = fma(ek5_0, r0_2_0_2, g5_29);
              g5_17 = fma(ek5_1, r0_2_0_2, g5_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g5_30 = fma(ek5_0, r0_2_1_1, g5_30);
              g5_18 = fma(ek5_1, r0_2_1_1, g5_18);
              g5_17 = fma(ek5_2, r0_2_1_1, g5_17);
              g5_9 = fma(ek5_3, r0_2_1_1, g5_9);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g5_31 = fma(ek5_0, r0_2_2_0, g5_31);
              g5_18 = fma(ek5_2, r0_2_2_0, g5_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g5_32 = fma(ek5_0, r0_3_0_1, g5_32);
              g5_19 = fma(ek5_1, r0_3_0_1, g5_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g5_33 = fma(ek5_0, r0_3_1_0, g5_33);
              g5_19 = fma(ek5_2, r0_3_1_0, g5_19);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g5_34 = fma(ek5_0, r0_4_0_0, g5_34);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g5_20 = fma(ek5_1, r0_0_0_5, g5_20);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g5_21 = fma(ek5_1, r0_0_1_4, g5_21);
              g5_20 = fma(ek5_2, r0_0_1_4, g5_20);
              g5_10 = fma(ek5_3, r0_0_1_4, g5_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g5_22 = fma(ek5_1, r0_0_2_3, g5_22);
              g5_21 = fma(ek5_2, r0_0_2_3, g5_21);
              g5_11 = fma(ek5_3, r0_0_2_3, g5_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g5_23 = fma(ek5_1, r0_0_3_2, g5_23);
              g5_22 = fma(ek5_2, r0_0_3_2, g5_22);
              g5_12 = fma(ek5_3, r0_0_3_2, g5_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g5_24 = fma(ek5_1, r0_0_4_1, g5_24);
              g5_23 = fma(ek5_2, r0_0_4_1, g5_23);
              g5_13 = fma(ek5_3, r0_0_4_1, g5_13);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g5_24 = fma(ek5_2, r0_0_5_0, g5_24);
              const double r0_1_0_4 = X * r1_0_0_4;
              g5_25 = fma(ek5_1, r0_1_0_4, g5_25);
              const double r0_1_1_3 = X * r1_0_1_3;
              g5_26 = fma(ek5_1, r0_1_1_3, g5_26);
              g5_25 = fma(ek5_2, r0_1_1_3, g5_25);
              g5_14 = fma(ek5_3, r0_1_1_3, g5_14);
              const double r0_1_2_2 = X * r1_0_2_2;
              g5_27 = fma(ek5_1, r0_1_2_2, g5_27);
              g5_26 = fma(ek5_2, r0_1_2_2, g5_26);
              g5_15 = fma(ek5_3, r0_1_2_2, g5_15);
              const double r0_1_3_1 = X * r1_0_3_1;
              g5_28 = fma(ek5_1, r0_1_3_1, g5_28);
              g5_27 = fma(ek5_2, r0_1_3_1, g5_27);
              g5_16 = fma(ek5_3, r0_1_3_1, g5_16);
              const double r0_1_4_0 = X * r1_0_4_0;
              g5_28 = fma(ek5_2, r0_1_4_0, g5_28);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g5_29 = fma(ek5_1, r0_2_0_3, g5_29);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g5_30 = fma(ek5_1, r0_2_1_2, g5_30);
              g5_29 = fma(ek5_2, r0_2_1_2, g5_29);
              g5_17 = fma(ek5_3, r0_2_1_2, g5_17);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g5_31 = fma(ek5_1, r0_2_2_1, g5_31);
              g5_30 = fma(ek5_2, r0_2_2_1, g5_30);
              g5_18 = fma(ek5_3, r0_2_2_1, g5_18);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g5_31 = fma(ek5_2, r0_2_3_0, g5_31);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g5_32 = fma(ek5_1, r0_3_0_2, g5_32);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g5_33 = fma(ek5_1, r0_3_1_1, g5_33);
              g5_32 = fma(ek5_2, r0_3_1_1, g5_32);
              g5_19 = fma(ek5_3, r0_3_1_1, g5_19);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g5_33 = fma(ek5_2, r0_3_2_0, g5_33);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g5_34 = fma(ek5_1, r0_4_0_1, g5_34);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g5_34 = fma(ek5_2, r0_4_1_0, g5_34);
              const double r5_0_0_1 = Z * b6;
              const double r4_0_0_2 = fma(Z, r5_0_0_1, b5);
              const double r3_0_0_3 = fma(Z, r4_0_0_2, 2.0 * r4_0_0_1);
              const double r2_0_0_4 = fma(Z, r3_0_0_3, 3.0 * r3_0_0_2);
              const double r1_0_0_5 = fma(Z, r2_0_0_4, 4.0 * r2_0_0_3);
              const double r0_0_1_5 = Y * r1_0_0_5;
              g5_20 = fma(ek5_3, r0_0_1_5, g5_20);
              const double r1_0_1_4 = Y * r2_0_0_4;
              const double r0_0_2_4 = fma(Y, r1_0_1_4, r1_0_0_4);
              g5_21 = fma(ek5_3, r0_0_2_4, g5_21);
              const double r2_0_1_3 = Y * r3_0_0_3;
              const double r1_0_2_3 = fma(Y, r2_0_1_3, r2_0_0_3);
              const double r0_0_3_3 = fma(Y, r1_0_2_3, 2.0 * r1_0_1_3);
              g5_22 = fma(ek5_3, r0_0_3_3, g5_22);
              const double r3_0_1_2 = Y * r4_0_0_2;
              const double r2_0_2_2 = fma(Y, r3_0_1_2, r3_0_0_2);
              const double r1_0_3_2 = fma(Y, r2_0_2_2, 2.0 * r2_0_1_2);
              const double r0_0_4_2 = fma(Y, r1_0_3_2, 3.0 * r1_0_2_2);
              g5_23 = fma(ek5_3, r0_0_4_2, g5_23);
              const double r4_0_1_1 = Y * r5_0_0_1;
              const double r3_0_2_1 = fma(Y, r4_0_1_1, r4_0_0_1);
              const double r2_0_3_1 = fma(Y, r3_0_2_1, 2.0 * r3_0_1_1);
              const double r1_0_4_1 = fma(Y, r2_0_3_1, 3.0 * r2_0_2_1);
              const double r0_0_5_1 = fma(Y, r1_0_4_1, 4.0 * r1_0_3_1);
              g5_24 = fma(ek5_3, r0_0_5_1, g5_24);
              const double r0_1_1_4 = X * r1_0_1_4;
              g5_25 = fma(ek5_3, r0_1_1_4, g5_25);
              const double r0_1_2_3 = X * r1_0_2_3;
              g5_26 = fma(ek5_3, r0_1_2_3, g5_26);
              const double r0_1_3_2 = X * r1_0_3_2;
              g5_27 = fma(ek5_3, r0_1_3_2, g5_27);
              const double r0_1_4_1 = X * r1_0_4_1;
              g5_28 = fma(ek5_3, r0_1_4_1, g5_28);
              const double r1_1_1_3 = X * r2_0_1_3;
              const double r0_2_1_3 = fma(X, r1_1_1_3, r1_0_1_3);
              g5_29 = fma(ek5_3, r0_2_1_3, g5_29);
              const double r1_1_2_2 = X * r2_0_2_2;
              const double r0_2_2_2 = fma(X, r1_1_2_2, r1_0_2_2);
              g5_30 = fma(ek5_3, r0_2_2_2, g5_30);
              const double r1_1_3_1 = X * r2_0_3_1;
              const double r0_2_3_1 = fma(X, r1_1_3_1, r1_0_3_1);
              g5_31 = fma(ek5_3, r0_2_3_1, g5_31);
              const double r2_1_1_2 = X * r3_0_1_2;
              const double r1_2_1_2 = fma(X, r2_1_1_2, r2_0_1_2);
              const double r0_3_1_2 = fma(X, r1_2_1_2, 2.0 * r1_1_1_2);
              g5_32 = fma(ek5_3, r0_3_1_2, g5_32);
              const double r2_1_2_1 = X * r3_0_2_1;
              const double r1_2_2_1 = fma(X, r2_1_2_1, r2_0_2_1);
              const double r0_3_2_1 = fma(X, r1_2_2_1, 2.0 * r1_1_2_1);
              g5_33 = fma(ek5_3, r0_3_2_1, g5_33);
              const double r3_1_1_1 = X * r4_0_1_1;
              const double r2_2_1_1 = fma(X, r3_1_1_1, r3_0_1_1);
              const double r1_3_1_1 = fma(X, r2_2_1_1, 2.0 * r2_1_1_1);
              const double r0_4_1_1 = fma(X, r1_3_1_1, 3.0 * r1_2_1_1);
              g5_34 = fma(ek5_3, r0_4_1_1, g5_34);
            }
            { const double eb = bi[5];
              o0_5 = fma(eb, g5_0, o0_5);
            }
            { const double eb = bi[6];
              o0_5 = fma(eb, g5_3, o0_5);
            }
            { const double eb = bi[7];
              o0_5 = fma(eb, g5_9, o0_5);
            }
            { const double eb = bi[8];
              o0_5 = fma(eb, g5_19, o0_5);
            }
            { const double eb = bi[9];
              o0_5 = fma(eb, g5_34, o0_5);
            }
            { const double eb = bi[10];
              o1_5 = fma(eb, g5_0, o1_5);
            }
            { const double eb = bi[11];
              o1_5 = fma(eb, g5_2, o1_5);
            }
            { const double eb = bi[12];
              o1_5 = fma(eb, g5_6, o1_5);
            }
            { const double eb = bi[13];
              o1_5 = fma(eb, g5_3, o1_5);
            }
            { const double eb = bi[14];
              o1_5 = fma(eb, g5_8, o1_5);
            }
            { const double eb = bi[15];
              o1_5 = fma(eb, g5_16, o1_5);
            }
            { const double eb = bi[16];
              o1_5 = fma(eb, g5_9, o1_5);
            }
            { const double eb = bi[17];
              o1_5 = fma(eb, g5_18, o1_5);
            }
            { const double eb = bi[18];
              o1_5 = fma(eb, g5_31, o1_5);
            }
            { const double eb = bi[19];
              o2_5 = fma(eb, g5_0, o2_5);
            }
            { const double eb = bi[20];
              o2_5 = fma(eb, g5_1, o2_5);
            }
            { const double eb = bi[21];
              o2_5 = fma(eb, g5_4, o2_5);
            }
            { const double eb = bi[22];
              o2_5 = fma(eb, g5_3, o2_5);
            }
            { const double eb = bi[23];
              o2_5 = fma(eb, g5_7, o2_5);
            }
            { const double eb = bi[24];
              o2_5 = fma(eb, g5_14, o2_5);
            }
            { const double eb = bi[25];
              o2_5 = fma(eb, g5_9, o2_5);
            }
            { const double eb = bi[26];
              o2_5 = fma(eb, g5_17, o2_5);
            }
            { const double eb = bi[27];
              o2_5 = fma(eb, g5_29, o2_5);
            }
            { const double eb = bi[28];
              o3_5 = fma(eb, g5_0, o3_5);
            }
            { const double eb = bi[29];
              o3_5 = fma(eb, g5_2, o3_5);
            }
            { const double eb = bi[30];
              o3_5 = fma(eb, g5_3, o3_5);
            }
            { const double eb = bi[31];
              o3_5 = fma(eb, g5_8, o3_5);
            }
            { const double eb = bi[32];
              o3_5 = fma(eb, g5_9, o3_5);
            }
            { const double eb = bi[33];
              o3_5 = fma(eb, g5_18, o3_5);
            }
            { const double eb = bi[34];
              o3_5 = fma(eb, g5_19, o3_5);
            }
            { const double eb = bi[35];
              o3_5 = fma(eb, g5_33, o3_5);
            }
            { const double eb = bi[36];
              o4_5 = fma(eb, g5_0, o4_5);
            }
            { const double eb = bi[37];
              o4_5 = fma(eb, g5_1, o4_5);
            }
            { const double eb = bi[38];
              o4_5 = fma(eb, g5_3, o4_5);
            }
            { const double eb = bi[39];
              o4_5 = fma(eb, g5_7, o4_5);
            }
            { const double eb = bi[40];
              o4_5 = fma(eb, g5_9, o4_5);
            }
            { const double eb = bi[41];
              o4_5 = fma(eb, g5_17, o4_5);
            }
            { const double eb = bi[42];
              o4_5 = fma(eb, g5_19, o4_5);
            }
            { const double eb = bi[43];
              o4_5 = fma(eb, g5_32, o4_5);
            }
            { const double eb = bi[44];
              o5_5 = fma(eb, g5_0, o5_5);
            }
            { const double eb = bi[45];
              o5_5 = fma(eb, g5_1, o5_5);
            }
            { const double eb = bi[46];
              o5_5 = fma(eb, g5_2, o5_5);
            }
            { const double eb = bi[47];
              o5_5 = fma(eb, g5_5, o5_5);
            }
            { const double eb = bi[48];
              o5_5 = fma(eb, g5_3, o5_5);
            }
            { const double eb = bi[49];
              o5_5 = fma(eb, g5_7, o5_5);
            }
            { const double eb = bi[50];
              o5_5 = fma(eb, g5_8, o5_5);
            }
            { const double eb = bi[51];
              o5_5 = fma(eb, g5_15, o5_5);
            }
            { const double eb = bi[52];
              o5_5 = fma(eb, g5_9, o5_5);
            }
            { const double eb = bi[53];
              o5_5 = fma(eb, g5_17, o5_5);
            }
            { const double eb = bi[54];
              o5_5 = fma(eb, g5_18, o5_5);
            }
            { const double eb = bi[55];
              o5_5 = fma(eb, g5_30, o5_5);
            }
            { const double eb = bi[56];
              o6_5 = fma(eb, g5_0, o6_5);
            }
            { const double eb = bi[57];
              o6_5 = fma(eb, g5_2, o6_5);
            }
            { const double eb = bi[58];
              o6_5 = fma(eb, g5_6, o6_5);
            }
            { const double eb = bi[59];
              o6_5 = fma(eb, g5_3, o6_5);
            }
            { const double eb = bi[60];
              o6_5 = fma(eb, g5_8, o6_5);
            }
            { const double eb = bi[61];
              o6_5 = fma(eb, g5_16, o6_5);
            }
            { const double eb = bi[62];
              o6_5 = fma(eb, g5_9, o6_5);
            }
            { const double eb = bi[63];
              o6_5 = fma(eb, g5_18, o6_5);
            }
            { const double eb = bi[64];
              o6_5 = fma(eb, g5_31, o6_5);
            }
            { const double eb = bi[65];
              o7_5 = fma(eb, g5_0, o7_5);
            }
            { const double eb = bi[66];
              o7_5 = fma(eb, g5_2, o7_5);
            }
            { const double eb = bi[67];
              o7_5 = fma(eb, g5_6, o7_5);
            }
            { const double eb = bi[68];
              o7_5 = fma(eb, g5_13, o7_5);
            }
            { const double eb = bi[69];
              o7_5 = fma(eb, g5_24, o7_5);
            }
            { const double eb = bi[70];
              o8_5 = fma(eb, g5_0, o8_5);
            }
            { const double eb = bi[71];
              o8_5 = fma(eb, g5_1, o8_5);
            }
            { const double eb = bi[72];
              o8_5 = fma(eb, g5_4, o8_5);
            }
            { const double eb = bi[73];
              o8_5 = fma(eb, g5_2, o8_5);
            }
            { const double eb = bi[74];
              o8_5 = fma(eb, g5_5, o8_5);
            }
            { const double eb = bi[75];
              o8_5 = fma(eb, g5_11, o8_5);
            }
            { const double eb = bi[76];
              o8_5 = fma(eb, g5_6, o8_5);
            }
            { const double eb = bi[77];
              o8_5 = fma(eb, g5_12, o8_5);
            }
            { const double eb = bi[78];
              o8_5 = fma(eb, g5_22, o8_5);
            }
            { const double eb = bi[79];
              o9_5 = fma(eb, g5_0, o9_5);
            }
            { const double eb = bi[80];
              o9_5 = fma(eb, g5_2, o9_5);
            }
            { const double eb = bi[81];
              o9_5 = fma(eb, g5_6, o9_5);
            }
            { const double eb = bi[82];
              o9_5 = fma(eb, g5_13, o9_5);
            }
            { const double eb = bi[83];
              o9_5 = fma(eb, g5_3, o9_5);
            }
            { const double eb = bi[84];
              o9_5 = fma(eb, g5_8, o9_5);
            }
            { const double eb = bi[85];
              o9_5 = fma(eb, g5_16, o9_5);
            }
            { const double eb = bi[86];
              o9_5 = fma(eb, g5_28, o9_5);
            }
            { const double eb = bi[87];
              o10_5 = fma(eb, g5_0, o10_5);
            }
            { const double eb = bi[88];
              o10_5 = fma(eb, g5_1, o10_5);
            }
            { const double eb = bi[89];
              o10_5 = fma(eb, g5_2, o10_5);
            }
            { const double eb = bi[90];
              o10_5 = fma(eb, g5_5, o10_5);
            }
            { const double eb = bi[91];
              o10_5 = fma(eb, g5_6, o10_5);
            }
            { const double eb = bi[92];
              o10_5 = fma(eb, g5_12, o10_5);
            }
            { const double eb = bi[93];
              o10_5 = fma(eb, g5_3, o10_5);
            }
            { const double eb = bi[94];
              o10_5 = fma(eb, g5_7, o10_5);
            }
            { const double eb = bi[95];
              o10_5 = fma(eb, g5_8, o10_5);
            }
            { const double eb = bi[96];
              o10_5 = fma(eb, g5_15, o10_5);
            }
            { const double eb = bi[97];
              o10_5 = fma(eb, g5_16, o10_5);
            }
            { const double eb = bi[98];
              o10_5 = fma(eb, g5_27, o10_5);
            }
            { const double eb = bi[99];
              o11_5 = fma(eb, g5_0, o11_5);
            }
            { const double eb = bi[100];
              o11_5 = fma(eb, g5_1, o11_5);
            }
            { const double eb = bi[101];
              o11_5 = fma(eb, g5_2, o11_5);
            }
            { const double eb = bi[102];
              o11_5 = fma(eb, g5_5, o11_5);
            }
            { const double eb = bi[103];
              o11_5 = fma(eb, g5_6, o11_5);
            }
            { const double eb = bi[104];
              o11_5 = fma(eb, g5_12, o11_5);
            }
            { const double eb = bi[105];
              o11_5 = fma(eb, g5_13, o11_5);
            }
            { const double eb = bi[106];
              o11_5 = fma(eb, g5_23, o11_5);
            }
            { const double eb = bi[107];
              o12_5 = fma(eb, g5_0, o12_5);
            }
            { const double eb = bi[108];
              o12_5 = fma(eb, g5_1, o12_5);
            }
            { const double eb = bi[109];
              o12_5 = fma(eb, g5_4, o12_5);
            }
            { const double eb = bi[110];
              o12_5 = fma(eb, g5_3, o12_5);
            }
            { const double eb = bi[111];
              o12_5 = fma(eb, g5_7, o12_5);
            }
            { const double eb = bi[112];
              o12_5 = fma(eb, g5_14, o12_5);
            }
            { const double eb = bi[113];
              o12_5 = fma(eb, g5_9, o12_5);
            }
            { const double eb = bi[114];
              o12_5 = fma(eb, g5_17, o12_5);
            }
            { const double eb = bi[115];
              o12_5 = fma(eb, g5_29, o12_5);
            }
            { const double eb = bi[116];
              o13_5 = fma(eb, g5_0, o13_5);
            }
            { const double eb = bi[117];
              o13_5 = fma(eb, g5_1, o13_5);
            }
            { const double eb = bi[118];
              o13_5 = fma(eb, g5_4, o13_5);
            }
            { const double eb = bi[119];
              o13_5 = fma(eb, g5_2, o13_5);
            }
            { const double eb = bi[120];
              o13_5 = fma(eb, g5_5, o13_5);
            }
            { const double eb = bi[121];
              o13_5 = fma(eb, g5_11, o13_5);
            }
            { const double eb = bi[122];
              o13_5 = fma(eb, g5_6, o13_5);
            }
            { const double eb = bi[123];
              o13_5 = fma(eb, g5_12, o13_5);
            }
            { const double eb = bi[124];
              o13_5 = fma(eb, g5_22, o13_5);
            }
            { const double eb = bi[125];
              o14_5 = fma(eb, g5_0, o14_5);
            }
            { const double eb = bi[126];
              o14_5 = fma(eb, g5_1, o14_5);
            }
            { const double eb = bi[127];
              o14_5 = fma(eb, g5_4, o14_5);
            }
            { const double eb = bi[128];
              o14_5 = fma(eb, g5_10, o14_5);
            }
            { const double eb = bi[129];
              o14_5 = fma(eb, g5_20, o14_5);
            }
            { const double eb = bi[130];
              o15_5 = fma(eb, g5_0, o15_5);
            }
            { const double eb = bi[131];
              o15_5 = fma(eb, g5_1, o15_5);
            }
            { const double eb = bi[132];
              o15_5 = fma(eb, g5_4, o15_5);
            }
            { const double eb = bi[133];
              o15_5 = fma(eb, g5_2, o15_5);
            }
            { const double eb = bi[134];
              o15_5 = fma(eb, g5_5, o15_5);
            }
            { const double eb = bi[135];
              o15_5 = fma(eb, g5_11, o15_5);
            }
            { const double eb = bi[136];
              o15_5 = fma(eb, g5_3, o15_5);
            }
            { const double eb = bi[137];
              o15_5 = fma(eb, g5_7, o15_5);
            }
            { const double eb = bi[138];
              o15_5 = fma(eb, g5_14, o15_5);
            }
            { const double eb = bi[139];
              o15_5 = fma(eb, g5_8, o15_5);
            }
            { const double eb = bi[140];
              o15_5 = fma(eb, g5_15, o15_5);
            }
            { const double eb = bi[141];
              o15_5 = fma(eb, g5_26, o15_5);
            }
            { const double eb = bi[142];
              o16_5 = fma(eb, g5_0, o16_5);
            }
            { const double eb = bi[143];
              o16_5 = fma(eb, g5_1, o16_5);
            }
            { const double eb = bi[144];
              o16_5 = fma(eb, g5_4, o16_5);
            }
            { const double eb = bi[145];
              o16_5 = fma(eb, g5_10, o16_5);
            }
            { const double eb = bi[146];
              o16_5 = fma(eb, g5_3, o16_5);
            }
            { const double eb = bi[147];
              o16_5 = fma(eb, g5_7, o16_5);
            }
            { const double eb = bi[148];
              o16_5 = fma(eb, g5_14, o16_5);
            }
            { const double eb = bi[149];
              o16_5 = fma(eb, g5_25, o16_5);
            }
            { const double eb = bi[150];
              o17_5 = fma(eb, g5_0, o17_5);
            }
            { const double eb = bi[151];
              o17_5 = fma(eb, g5_1, o17_5);
            }
            { const double eb = bi[152];
              o17_5 = fma(eb, g5_4, o17_5);
            }
            { const double eb = bi[153];
              o17_5 = fma(eb, g5_10, o17_5);
            }
            { const double eb = bi[154];
              o17_5 = fma(eb, g5_2, o17_5);
            }
            { const double eb = bi[155];
              o17_5 = fma(eb, g5_5, o17_5);
            }
            { const double eb = bi[156];
              o17_5 = fma(eb, g5_11, o17_5);
            }
            { const double eb = bi[157];
              o17_5 = fma(eb, g5_21, o17_5);
            }
            { const double eb = bi[158];
              o18_5 = fma(eb, g5_0, o18_5);
            }
            { const double eb = bi[159];
              o18_5 = fma(eb, g5_2, o18_5);
            }
            { const double eb = bi[160];
              o18_5 = fma(eb, g5_3, o18_5);
            }
            { const double eb = bi[161];
              o18_5 = fma(eb, g5_8, o18_5);
            }
            { const double eb = bi[162];
              o18_5 = fma(eb, g5_9, o18_5);
            }
            { const double eb = bi[163];
              o18_5 = fma(eb, g5_18, o18_5);
            }
            { const double eb = bi[164];
              o18_5 = fma(eb, g5_19, o18_5);
            }
            { const double eb = bi[165];
              o18_5 = fma(eb, g5_33, o18_5);
            }
            { const double eb = bi[166];
              o19_5 = fma(eb, g5_0, o19_5);
            }
            { const double eb = bi[167];
              o19_5 = fma(eb, g5_2, o19_5);
            }
            { const double eb = bi[168];
              o19_5 = fma(eb, g5_6, o19_5);
            }
            { const double eb = bi[169];
              o19_5 = fma(eb, g5_13, o19_5);
            }
            { const double eb = bi[170];
              o19_5 = fma(eb, g5_3, o19_5);
            }
            { const double eb = bi[171];
              o19_5 = fma(eb, g5_8, o19_5);
            }
            { const double eb = bi[172];
              o19_5 = fma(eb, g5_16, o19_5);
            }
            { const double eb = bi[173];
              o19_5 = fma(eb, g5_28, o19_5);
            }
            { const double eb = bi[174];
              o20_5 = fma(eb, g5_0, o20_5);
            }
            { const double eb = bi[175];
              o20_5 = fma(eb, g5_1, o20_5);
            }
            { const double eb = bi[176];
              o20_5 = fma(eb, g5_4, o20_5);
            }
            { const double eb = bi[177];
              o20_5 = fma(eb, g5_2, o20_5);
            }
            { const double eb = bi[178];
              o20_5 = fma(eb, g5_5, o20_5);
            }
            { const double eb = bi[179];
              o20_5 = fma(eb, g5_11, o20_5);
            }
            { const double eb = bi[180];
              o20_5 = fma(eb, g5_3, o20_5);
            }
            { const double eb = bi[181];
              o20_5 = fma(eb, g5_7, o20_5);
            }
            { const double eb = bi[182];
              o20_5 = fma(eb, g5_14, o20_5);
            }
            { const double eb = bi[183];
              o20_5 = fma(eb, g5_8, o20_5);
            }
            { const double eb = bi[184];
              o20_5 = fma(eb, g5_15, o20_5);
            }
            { const double eb = bi[185];
              o20_5 = fma(eb, g5_26, o20_5);
            }
            { const double eb = bi[186];
              o21_5 = fma(eb, g5_0, o21_5);
            }
            { const double eb = bi[187];
              o21_5 = fma(eb, g5_2, o21_5);
            }
            { const double eb = bi[188];
              o21_5 = fma(eb, g5_6, o21_5);
            }
            { const double eb = bi[189];
              o21_5 = fma(eb, g5_3, o21_5);
            }
            { const double eb = bi[190];
              o21_5 = fma(eb, g5_8, o21_5);
            }
            { const double eb = bi[191];
              o21_5 = fma(eb, g5_16, o21_5);
            }
            { const double eb = bi[192];
              o21_5 = fma(eb, g5_9, o21_5);
            }
            { const double eb = bi[193];
              o21_5 = fma(eb, g5_18, o21_5);
            }
            { const double eb = bi[194];
              o21_5 = fma(eb, g5_31, o21_5);
            }
            { const double eb = bi[195];
              o22_5 = fma(eb, g5_0, o22_5);
            }
            { const double eb = bi[196];
              o22_5 = fma(eb, g5_1, o22_5);
            }
            { const double eb = bi[197];
              o22_5 = fma(eb, g5_2, o22_5);
            }
            { const double eb = bi[198];
              o22_5 = fma(eb, g5_5, o22_5);
            }
            { const double eb = bi[199];
              o22_5 = fma(eb, g5_3, o22_5);
            }
            { const double eb = bi[200];
              o22_5 = fma(eb, g5_7, o22_5);
            }
            { const double eb = bi[201];
              o22_5 = fma(eb, g5_8, o22_5);
            }
            { const double eb = bi[202];
              o22_5 = fma(eb, g5_15, o22_5);
            }
            { const double eb = bi[203];
              o22_5 = fma(eb, g5_9, o22_5);
            }
            { const double eb = bi[204];
              o22_5 = fma(eb, g5_17, o22_5);
            }
            { const double eb = bi[205];
              o22_5 = fma(eb, g5_18, o22_5);
            }
            { const double eb = bi[206];
              o22_5 = fma(eb, g5_30, o22_5);
            }
            { const double eb = bi[207];
              o23_5 = fma(eb, g5_0, o23_5);
            }
            { const double eb = bi[208];
              o23_5 = fma(eb, g5_1, o23_5);
            }
            { const double eb = bi[209];
              o23_5 = fma(eb, g5_2, o23_5);
            }
            { const double eb = bi[210];
              o23_5 = fma(eb, g5_5, o23_5);
            }
            { const double eb = bi[211];
              o23_5 = fma(eb, g5_6, o23_5);
            }
            { const double eb = bi[212];
              o23_5 = fma(eb, g5_12, o23_5);
            }
            { const double eb = bi[213];
              o23_5 = fma(eb, g5_3, o23_5);
            }
            { const double eb = bi[214];
              o23_5 = fma(eb, g5_7, o23_5);
            }
            { const double eb = bi[215];
              o23_5 = fma(eb, g5_8, o23_5);
            }
            { const double eb = bi[216];
              o23_5 = fma(eb, g5_15, o23_5);
            }
            { const double eb = bi[217];
              o23_5 = fma(eb, g5_16, o23_5);
            }
            { const double eb = bi[218];
              o23_5 = fma(eb, g5_27, o23_5);
            }
            { const double eb = bi[219];
              o24_5 = fma(eb, g5_0, o24_5);
            }
            { const double eb = bi[220];
              o24_5 = fma(eb, g5_1, o24_5);
            }
            { const double eb = bi[221];
              o24_5 = fma(eb, g5_3, o24_5);
            }
            { const double eb = bi[222];
              o24_5 = fma(eb, g5_7, o24_5);
            }
            { const double eb = bi[223];
              o24_5 = fma(eb, g5_9, o24_5);
            }
            { const double eb = bi[224];
              o24_5 = fma(eb, g5_17, o24_5);
            }
            { const double eb = bi[225];
              o24_5 = fma(eb, g5_19, o24_5);
            }
            { const double eb = bi[226];
              o24_5 = fma(eb, g5_32, o24_5);
            }
            { const double eb = bi[227];
              o25_5 = fma(eb, g5_0, o25_5);
            }
            { const double eb = bi[228];
              o25_5 = fma(eb, g5_1, o25_5);
            }
            { const double eb = bi[229];
              o25_5 = fma(eb, g5_2, o25_5);
            }
            { const double eb = bi[230];
              o25_5 = fma(eb, g5_5, o25_5);
            }
            { const double eb = bi[231];
              o25_5 = fma(eb, g5_6, o25_5);
            }
            { const double eb = bi[232];
              o25_5 = fma(eb, g5_12, o25_5);
            }
            { const double eb = bi[233];
              o25_5 = fma(eb, g5_3, o25_5);
            }
            { const double eb = bi[234];
              o25_5 = fma(eb, g5_7, o25_5);
            }
            { const double eb = bi[235];
              o25_5 = fma(eb, g5_8, o25_5);
            }
            { const double eb = bi[236];
              o25_5 = fma(eb, g5_15, o25_5);
            }
            { const double eb = bi[237];
              o25_5 = fma(eb, g5_16, o25_5);
            }
            { const double eb = bi[238];
              o25_5 = fma(eb, g5_27, o25_5);
            }
            { const double eb = bi[239];
              o26_5 = fma(eb, g5_0, o26_5);
            }
            { const double eb = bi[240];
              o26_5 = fma(eb, g5_1, o26_5);
            }
            { const double eb = bi[241];
              o26_5 = fma(eb, g5_4, o26_5);
            }
            { const double eb = bi[242];
              o26_5 = fma(eb, g5_10, o26_5);
            }
            { const double eb = bi[243];
              o26_5 = fma(eb, g5_3, o26_5);
            }
            { const double eb = bi[244];
              o26_5 = fma(eb, g5_7, o26_5);
            }
            { const double eb = bi[245];
              o26_5 = fma(eb, g5_14, o26_5);
            }
            { const double eb = bi[246];
              o26_5 = fma(eb, g5_25, o26_5);
            }
            { const double eb = bi[247];
              o27_5 = fma(eb, g5_0, o27_5);
            }
            { const double eb = bi[248];
              o27_5 = fma(eb, g5_1, o27_5);
            }
            { const double eb = bi[249];
              o27_5 = fma(eb, g5_2, o27_5);
            }
            { const double eb = bi[250];
              o27_5 = fma(eb, g5_5, o27_5);
            }
            { const double eb = bi[251];
              o27_5 = fma(eb, g5_3, o27_5);
            }
            { const double eb = bi[252];
              o27_5 = fma(eb, g5_7, o27_5);
            }
            { const double eb = bi[253];
              o27_5 = fma(eb, g5_8, o27_5);
            }
            { const double eb = bi[254];
              o27_5 = fma(eb, g5_15, o27_5);
            }
            { const double eb = bi[255];
              o27_5 = fma(eb, g5_9, o27_5);
            }
            { const double eb = bi[256];
              o27_5 = fma(eb, g5_17, o27_5);
            }
            { const double eb = bi[257];
              o27_5 = fma(eb, g5_18, o27_5);
            }
            { const double eb = bi[258];
              o27_5 = fma(eb, g5_30, o27_5);
            }
            { const double eb = bi[259];
              o28_5 = fma(eb, g5_0, o28_5);
            }
            { const double eb = bi[260];
              o28_5 = fma(eb, g5_1, o28_5);
            }
            { const double eb = bi[261];
              o28_5 = fma(eb, g5_4, o28_5);
            }
            { const double eb = bi[262];
              o28_5 = fma(eb, g5_3, o28_5);
            }
            { const double eb = bi[263];
              o28_5 = fma(eb, g5_7, o28_5);
            }
            { const double eb = bi[264];
              o28_5 = fma(eb, g5_14, o28_5);
            }
            { const double eb = bi[265];
              o28_5 = fma(eb, g5_9, o28_5);
            }
            { const double eb = bi[266];
              o28_5 = fma(eb, g5_17, o28_5);
            }
            { const double eb = bi[267];
              o28_5 = fma(eb, g5_29, o28_5);
            }
            { const double eb = bi[268];
              o29_5 = fma(eb, g5_0, o29_5);
            }
            { const double eb = bi[269];
              o29_5 = fma(eb, g5_1, o29_5);
            }
            { const double eb = bi[270];
              o29_5 = fma(eb, g5_4, o29_5);
            }
            { const double eb = bi[271];
              o29_5 = fma(eb, g5_2, o29_5);
            }
            { const double eb = bi[272];
              o29_5 = fma(eb, g5_5, o29_5);
            }
            { const double eb = bi[273];
              o29_5 = fma(eb, g5_11, o29_5);
            }
            { const double eb = bi[274];
              o29_5 = fma(eb, g5_3, o29_5);
            }
            { const double eb = bi[275];
              o29_5 = fma(eb, g5_7, o29_5);
            }
            { const double eb = bi[276];
              o29_5 = fma(eb, g5_14, o29_5);
            }
            { const double eb = bi[277];
              o29_5 = fma(eb, g5_8, o29_5);
            }
            { const double eb = bi[278];
              o29_5 = fma(eb, g5_15, o29_5);
            }
            { const double eb = bi[279];
              o29_5 = fma(eb, g5_26, o29_5);
            }
            { const double eb = bi[280];
              o30_5 = fma(eb, g5_0, o30_5);
            }
            { const double eb = bi[281];
              o30_5 = fma(eb, g5_1, o30_5);
            }
            { const double eb = bi[282];
              o30_5 = fma(eb, g5_2, o30_5);
            }
            { const double eb = bi[283];
              o30_5 = fma(eb, g5_5, o30_5);
            }
            { const double eb = bi[284];
              o30_5 = fma(eb, g5_3, o30_5);
            }
            { const double eb = bi[285];
              o30_5 = fma(eb, g5_7, o30_5);
            }
            { const double eb = bi[286];
              o30_5 = fma(eb, g5_8, o30_5);
            }
            { const double eb = bi[287];
              o30_5 = fma(eb, g5_15, o30_5);
            }
            { const double eb = bi[288];
              o30_5 = fma(eb, g5_9, o30_5);
            }
            { const double eb = bi[289];
              o30_5 = fma(eb, g5_17, o30_5);
            }
            { const double eb = bi[290];
              o30_5 = fma(eb, g5_18, o30_5);
            }
            { const double eb = bi[291];
              o30_5 = fma(eb, g5_30, o30_5);
            }
            { const double eb = bi[292];
              o31_5 = fma(eb, g5_0, o31_5);
            }
            { const double eb = bi[293];
              o31_5 = fma(eb, g5_1, o31_5);
            }
            { const double eb = bi[294];
              o31_5 = fma(eb, g5_2, o31_5);
            }
            { const double eb = bi[295];
              o31_5 = fma(eb, g5_5, o31_5);
            }
            { const double eb = bi[296];
              o31_5 = fma(eb, g5_6, o31_5);
            }
            { const double eb = bi[297];
              o31_5 = fma(eb, g5_12, o31_5);
            }
            { const double eb = bi[298];
              o31_5 = fma(eb, g5_13, o31_5);
            }
            { const double eb = bi[299];
              o31_5 = fma(eb, g5_23, o31_5);
            }
            { const double eb = bi[300];
              o32_5 = fma(eb, g5_0, o32_5);
            }
            { const double eb = bi[301];
              o32_5 = fma(eb, g5_1, o32_5);
            }
            { const double eb = bi[302];
              o32_5 = fma(eb, g5_4, o32_5);
            }
            { const double eb = bi[303];
              o32_5 = fma(eb, g5_10, o32_5);
            }
            { const double eb = bi[304];
              o32_5 = fma(eb, g5_2, o32_5);
            }
            { const double eb = bi[305];
              o32_5 = fma(eb, g5_5, o32_5);
            }
            { const double eb = bi[306];
              o32_5 = fma(eb, g5_11, o32_5);
            }
            { const double eb = bi[307];
              o32_5 = fma(eb, g5_21, o32_5);
            }
            { const double eb = bi[308];
              o33_5 = fma(eb, g5_0, o33_5);
            }
            { const double eb = bi[309];
              o33_5 = fma(eb, g5_1, o33_5);
            }
            { const double eb = bi[310];
              o33_5 = fma(eb, g5_2, o33_5);
            }
            { const double eb = bi[311];
              o33_5 = fma(eb, g5_5, o33_5);
            }
            { const double eb = bi[312];
              o33_5 = fma(eb, g5_6, o33_5);
            }
            { const double eb = bi[313];
              o33_5 = fma(eb, g5_12, o33_5);
            }
            { const double eb = bi[314];
              o33_5 = fma(eb, g5_3, o33_5);
            }
            { const double eb = bi[315];
              o33_5 = fma(eb, g5_7, o33_5);
            }
            { const double eb = bi[316];
              o33_5 = fma(eb, g5_8, o33_5);
            }
            { const double eb = bi[317];
              o33_5 = fma(eb, g5_15, o33_5);
            }
            { const double eb = bi[318];
              o33_5 = fma(eb, g5_16, o33_5);
            }
            { const double eb = bi[319];
              o33_5 = fma(eb, g5_27, o33_5);
            }
            { const double eb = bi[320];
              o34_5 = fma(eb, g5_0, o34_5);
            }
            { const double eb = bi[321];
              o34_5 = fma(eb, g5_1, o34_5);
            }
            { const double eb = bi[322];
              o34_5 = fma(eb, g5_4, o34_5);
            }
            { const double eb = bi[323];
              o34_5 = fma(eb, g5_2, o34_5);
            }
            { const double eb = bi[324];
              o34_5 = fma(eb, g5_5, o34_5);
            }
            { const double eb = bi[325];
              o34_5 = fma(eb, g5_11, o34_5);
            }
            { const double eb = bi[326];
              o34_5 = fma(eb, g5_3, o34_5);
            }
            { const double eb = bi[327];
              o34_5 = fma(eb, g5_7, o34_5);
            }
            { const double eb = bi[328];
              o34_5 = fma(eb, g5_14, o34_5);
            }
            { const double eb = bi[329];
              o34_5 = fma(eb, g5_8, o34_5);
            }
            { const double eb = bi[330];
              o34_5 = fma(eb, g5_15, o34_5);
            }
            { const double eb = bi[331];
              o34_5 = fma(eb, g5_26, o34_5);
            }
            { const double eb = bi[332];
              o35_5 = fma(eb, g5_0, o35_5);
            }
            { const double eb = bi[333];
              o35_5 = fma(eb, g5_1, o35_5);
            }
            { const double eb = bi[334];
              o35_5 = fma(eb, g5_4, o35_5);
            }
            { const double eb = bi[335];
              o35_5 = fma(eb, g5_2, o35_5);
            }
            { const double eb = bi[336];
              o35_5 = fma(eb, g5_5, o35_5);
            }
            { const double eb = bi[337];
              o35_5 = fma(eb, g5_11, o35_5);
            }
            { const double eb = bi[338];
              o35_5 = fma(eb, g5_6, o35_5);
            }
            { const double eb = bi[339];
              o35_5 = fma(eb, g5_12, o35_5);
            }
            { const double eb = bi[340];
              o35_5 = fma(eb, g5_22, o35_5);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 5, fJ + 0);
            o1_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 5, fJ + 0);
            o2_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 5, fJ + 0);
            o3_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 5, fJ + 0);
            o4_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 5, fJ + 0);
            o5_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 5, fJ + 0);
            o6_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 5, fJ + 0);
            o7_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 5, fJ + 0);
            o8_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 5, fJ + 0);
            o9_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 5, fJ + 0);
            o10_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 5, fJ + 0);
            o11_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 5, fJ + 0);
            o12_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 5, fJ + 0);
            o13_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 5, fJ + 0);
            o14_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 5, fJ + 0);
            o15_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 5, fJ + 0);
            o16_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 5, fJ + 0);
            o17_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 5, fJ + 0);
            o18_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 5, fJ + 0);
            o19_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 5, fJ + 0);
            o20_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 5, fJ + 0);
            o21_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 5, fJ + 0);
            o22_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 5, fJ + 0);
            o23_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 5, fJ + 0);
            o24_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 5, fJ + 0);
            o25_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 5, fJ + 0);
            o26_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 5, fJ + 0);
            o27_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 5, fJ + 0);
            o28_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 5, fJ + 0);
            o29_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 5, fJ + 0);
            o30_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 5, fJ + 0);
            o31_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 5, fJ + 0);
            o32_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 5, fJ + 0);
            o33_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 5, fJ + 0);
            o34_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 5, fJ + 0);
            o35_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 5, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o1_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o2_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o3_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o4_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 4, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o5_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 5, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o6_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o7_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o8_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o9_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o10_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 4, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o11_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 5, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o12_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o13_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o14_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o15_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o16_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 4, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o17_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 5, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o18_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o19_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o20_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o21_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o22_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 4, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o23_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 5, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o24_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o25_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o26_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o27_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o28_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 4, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o29_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 5, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o30_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o31_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o32_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o33_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o34_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 4, fI + 5, fJ + 0)));
            e = fmax(e, fabs(o35_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 5, fI + 5, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk5 = PT[(fI + 5) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 0) * N + fQ + 1];
            const double ptb2 = PT[(fP + 0) * N + fQ + 2];
            const double ptb3 = PT[(fP + 0) * N + fQ + 3];
            const double ptb4 = PT[(fP + 0) * N + fQ + 4];
            const double ptb5 = PT[(fP + 0) * N + fQ + 5];
            const double ptb6 = PT[(fP + 1) * N + fQ + 0];
            const double ptb7 = PT[(fP + 1) * N + fQ + 1];
            const double ptb8 = PT[(fP + 1) * N + fQ + 2];
            const double ptb9 = PT[(fP + 1) * N + fQ + 3];
            const double ptb10 = PT[(fP + 1) * N + fQ + 4];
            const double ptb11 = PT[(fP + 1) * N + fQ + 5];
            const double ptb12 = PT[(fP + 2) * N + fQ + 0];
            const double ptb13 = PT[(fP + 2) * N + fQ + 1];
            const double ptb14 = PT[(fP + 2) * N + fQ + 2];
            const double ptb15 = PT[(fP + 2) * N + fQ + 3];
            const double ptb16 = PT[(fP + 2) * N + fQ + 4];
            const double ptb17 = PT[(fP + 2) * N + fQ + 5];
            const double ptb18 = PT[(fP + 3) * N + fQ + 0];
            const double ptb19 = PT[(fP + 3) * N + fQ + 1];
            const double ptb20 = PT[(fP + 3) * N + fQ + 2];
            const double ptb21 = PT[(fP + 3) * N + fQ + 3];
            const double ptb22 = PT[(fP + 3) * N + fQ + 4];
            const double ptb23 = PT[(fP + 3) * N + fQ + 5];
            const double ptb24 = PT[(fP + 4) * N + fQ + 0];
            const double ptb25 = PT[(fP + 4) * N + fQ + 1];
            const double ptb26 = PT[(fP + 4) * N + fQ + 2];
            const double ptb27 = PT[(fP + 4) * N + fQ + 3];
            const double ptb28 = PT[(fP + 4) * N + fQ + 4];
            const double ptb29 = PT[(fP + 4) * N + fQ + 5];
            const double ptb30 = PT[(fP + 5) * N + fQ + 0];
            const double ptb31 = PT[(fP + 5) * N + fQ + 1];
            const double ptb32 = PT[(fP + 5) * N + fQ + 2];
            const double ptb33 = PT[(fP + 5) * N + fQ + 3];
            const double ptb34 = PT[(fP + 5) * N + fQ + 4];
            const double ptb35 = PT[(fP + 5) * N + fQ + 5];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Abd4_0 = PA[(fQ + 4) * N + fJ + 0];
            const double Abd5_0 = PA[(fQ + 5) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_5 = PA[(fQ + 0) * N + fI + 5];
            const double Abc1_5 = PA[(fQ + 1) * N + fI + 5];
            const double Abc2_5 = PA[(fQ + 2) * N + fI + 5];
            const double Abc3_5 = PA[(fQ + 3) * N + fI + 5];
            const double Abc4_5 = PA[(fQ + 4) * N + fI + 5];
            const double Abc5_5 = PA[(fQ + 5) * N + fI + 5];
            const double Aac0_5 = PA[(fP + 0) * N + fI + 5];
            const double Aac1_5 = PA[(fP + 1) * N + fI + 5];
            const double Aac2_5 = PA[(fP + 2) * N + fI + 5];
            const double Aac3_5 = PA[(fP + 3) * N + fI + 5];
            const double Aac4_5 = PA[(fP + 4) * N + fI + 5];
            const double Aac5_5 = PA[(fP + 5) * N + fI + 5];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bbd4_0 = PB[(fQ + 4) * N + fJ + 0];
            const double Bbd5_0 = PB[(fQ + 5) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_5 = PB[(fQ + 0) * N + fI + 5];
            const double Bbc1_5 = PB[(fQ + 1) * N + fI + 5];
            const double Bbc2_5 = PB[(fQ + 2) * N + fI + 5];
            const double Bbc3_5 = PB[(fQ + 3) * N + fI + 5];
            const double Bbc4_5 = PB[(fQ + 4) * N + fI + 5];
            const double Bbc5_5 = PB[(fQ + 5) * N + fI + 5];
            const double Bac0_5 = PB[(fP + 0) * N + fI + 5];
            const double Bac1_5 = PB[(fP + 1) * N + fI + 5];
            const double Bac2_5 = PB[(fP + 2) * N + fI + 5];
            const double Bac3_5 = PB[(fP + 3) * N + fI + 5];
            const double Bac4_5 = PB[(fP + 4) * N + fI + 5];
            const double Bac5_5 = PB[(fP + 5) * N + fI + 5];
            jab0 += o0_5 * ptk5;
            jab1 += o1_5 * ptk5;
            jab2 += o2_5 * ptk5;
            jab3 += o3_5 * ptk5;
            jab4 += o4_5 * ptk5;
            jab5 += o5_5 * ptk5;
            jab6 += o6_5 * ptk5;
            jab7 += o7_5 * ptk5;
            jab8 += o8_5 * ptk5;
            jab9 += o9_5 * ptk5;
            jab10 += o10_5 * ptk5;
            jab11 += o11_5 * ptk5;
            jab12 += o12_5 * ptk5;
            jab13 += o13_5 * ptk5;
            jab14 += o14_5 * ptk5;
            jab15 += o15_5 * ptk5;
            jab16 += o16_5 * ptk5;
            jab17 += o17_5 * ptk5;
            jab18 += o18_5 * ptk5;
            jab19 += o19_5 * ptk5;
            jab20 += o20_5 * ptk5;
            jab21 += o21_5 * ptk5;
            jab22 += o22_5 * ptk5;
            jab23 += o23_5 * ptk5;
            jab24 += o24_5 * ptk5;
            jab25 += o25_5 * ptk5;
            jab26 += o26_5 * ptk5;
            jab27 += o27_5 * ptk5;
            jab28 += o28_5 * ptk5;
            jab29 += o29_5 * ptk5;
            jab30 += o30_5 * ptk5;
            jab31 += o31_5 * ptk5;
            jab32 += o32_5 * ptk5;
            jab33 += o33_5 * ptk5;
            jab34 += o34_5 * ptk5;
            jab35 += o35_5 * ptk5;
            atomicAdd(Jacc + (fI + 5) * N + fJ + 0, 2.0 * deg * (o0_5 * ptb0 + o1_5 * ptb1 + o2_5 * ptb2 + o3_5 * ptb3 + o4_5 * ptb4 + o5_5 * ptb5 + o6_5 * ptb6 + o7_5 * ptb7 + o8_5 * ptb8 + o9_5 * ptb9 + o10_5 * ptb10 + o11_5 * ptb11 + o12_5 * ptb12 + o13_5 * ptb13 + o14_5 * ptb14 + o15_5 * ptb15 + o16_5 * ptb16 + o17_5 * ptb17 + o18_5 * ptb18 + o19_5 * ptb19 + o20_5 * ptb20 + o21_5 * ptb21 + o22_5 * ptb22 + o23_5 * ptb23 + o24_5 * ptb24 + o25_5 * ptb25 + o26_5 * ptb26 + o27_5 * ptb27 + o28_5 * ptb28 + o29_5 * ptb29 + o30_5 * ptb30 + o31_5 * ptb31 + o32_5 * ptb32 + o33_5 * ptb33 + o34_5 * ptb34 + o35_5 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 5, deg * (o0_5 * Abd0_0 + o1_5 * Abd1_0 + o2_5 * Abd2_0 + o3_5 * Abd3_0 + o4_5 * Abd4_0 + o5_5 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 5, deg * (o0_5 * Aad0_0 + o6_5 * Aad1_0 + o12_5 * Aad2_0 + o18_5 * Aad3_0 + o24_5 * Aad4_0 + o30_5 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_5 * Abc0_5 + o1_5 * Abc1_5 + o2_5 * Abc2_5 + o3_5 * Abc3_5 + o4_5 * Abc4_5 + o5_5 * Abc5_5));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_5 * Aac0_5 + o6_5 * Aac1_5 + o12_5 * Aac2_5 + o18_5 * Aac3_5 + o24_5 * Aac4_5 + o30_5 * Aac5_5));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 5, deg * (o1_5 * Aad0_0 + o7_5 * Aad1_0 + o13_5 * Aad2_0 + o19_5 * Aad3_0 + o25_5 * Aad4_0 + o31_5 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_5 * Aac0_5 + o7_5 * Aac1_5 + o13_5 * Aac2_5 + o19_5 * Aac3_5 + o25_5 * Aac4_5 + o31_5 * Aac5_5));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 5, deg * (o2_5 * Aad0_0 + o8_5 * Aad1_0 + o14_5 * Aad2_0 + o20_5 * Aad3_0 + o26_5 * Aad4_0 + o32_5 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_5 * Aac0_5 + o8_5 * Aac1_5 + o14_5 * Aac2_5 + o20_5 * Aac3_5 + o26_5 * Aac4_5 + o32_5 * Aac5_5));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 5, deg * (o3_5 * Aad0_0 + o9_5 * Aad1_0 + o15_5 * Aad2_0 + o21_5 * Aad3_0 + o27_5 * Aad4_0 + o33_5 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_5 * Aac0_5 + o9_5 * Aac1_5 + o15_5 * Aac2_5 + o21_5 * Aac3_5 + o27_5 * Aac4_5 + o33_5 * Aac5_5));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 5, deg * (o4_5 * Aad0_0 + o10_5 * Aad1_0 + o16_5 * Aad2_0 + o22_5 * Aad3_0 + o28_5 * Aad4_0 + o34_5 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_5 * Aac0_5 + o10_5 * Aac1_5 + o16_5 * Aac2_5 + o22_5 * Aac3_5 + o28_5 * Aac4_5 + o34_5 * Aac5_5));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 5, deg * (o5_5 * Aad0_0 + o11_5 * Aad1_0 + o17_5 * Aad2_0 + o23_5 * Aad3_0 + o29_5 * Aad4_0 + o35_5 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_5 * Aac0_5 + o11_5 * Aac1_5 + o17_5 * Aac2_5 + o23_5 * Aac3_5 + o29_5 * Aac4_5 + o35_5 * Aac5_5));
            atomicAdd(KAacc + (fP + 1) * N + fI + 5, deg * (o6_5 * Abd0_0 + o7_5 * Abd1_0 + o8_5 * Abd2_0 + o9_5 * Abd3_0 + o10_5 * Abd4_0 + o11_5 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_5 * Abc0_5 + o7_5 * Abc1_5 + o8_5 * Abc2_5 + o9_5 * Abc3_5 + o10_5 * Abc4_5 + o11_5 * Abc5_5));
            atomicAdd(KAacc + (fP + 2) * N + fI + 5, deg * (o12_5 * Abd0_0 + o13_5 * Abd1_0 + o14_5 * Abd2_0 + o15_5 * Abd3_0 + o16_5 * Abd4_0 + o17_5 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_5 * Abc0_5 + o13_5 * Abc1_5 + o14_5 * Abc2_5 + o15_5 * Abc3_5 + o16_5 * Abc4_5 + o17_5 * Abc5_5));
            atomicAdd(KAacc + (fP + 3) * N + fI + 5, deg * (o18_5 * Abd0_0 + o19_5 * Abd1_0 + o20_5 * Abd2_0 + o21_5 * Abd3_0 + o22_5 * Abd4_0 + o23_5 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_5 * Abc0_5 + o19_5 * Abc1_5 + o20_5 * Abc2_5 + o21_5 * Abc3_5 + o22_5 * Abc4_5 + o23_5 * Abc5_5));
            atomicAdd(KAacc + (fP + 4) * N + fI + 5, deg * (o24_5 * Abd0_0 + o25_5 * Abd1_0 + o26_5 * Abd2_0 + o27_5 * Abd3_0 + o28_5 * Abd4_0 + o29_5 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_5 * Abc0_5 + o25_5 * Abc1_5 + o26_5 * Abc2_5 + o27_5 * Abc3_5 + o28_5 * Abc4_5 + o29_5 * Abc5_5));
            atomicAdd(KAacc + (fP + 5) * N + fI + 5, deg * (o30_5 * Abd0_0 + o31_5 * Abd1_0 + o32_5 * Abd2_0 + o33_5 * Abd3_0 + o34_5 * Abd4_0 + o35_5 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_5 * Abc0_5 + o31_5 * Abc1_5 + o32_5 * Abc2_5 + o33_5 * Abc3_5 + o34_5 * Abc4_5 + o35_5 * Abc5_5));
            atomicAdd(KBacc + (fP + 0) * N + fI + 5, deg * (o0_5 * Bbd0_0 + o1_5 * Bbd1_0 + o2_5 * Bbd2_0 + o3_5 * Bbd3_0 + o4_5 * Bbd4_0 + o5_5 * Bbd5_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 5, deg * (o0_5 * Bad0_0 + o6_5 * Bad1_0 + o12_5 * Bad2_0 + o18_5 * Bad3_0 + o24_5 * Bad4_0 + o30_5 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_5 * Bbc0_5 + o1_5 * Bbc1_5 + o2_5 * Bbc2_5 + o3_5 * Bbc3_5 + o4_5 * Bbc4_5 + o5_5 * Bbc5_5));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_5 * Bac0_5 + o6_5 * Bac1_5 + o12_5 * Bac2_5 + o18_5 * Bac3_5 + o24_5 * Bac4_5 + o30_5 * Bac5_5));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 5, deg * (o1_5 * Bad0_0 + o7_5 * Bad1_0 + o13_5 * Bad2_0 + o19_5 * Bad3_0 + o25_5 * Bad4_0 + o31_5 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_5 * Bac0_5 + o7_5 * Bac1_5 + o13_5 * Bac2_5 + o19_5 * Bac3_5 + o25_5 * Bac4_5 + o31_5 * Bac5_5));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 5, deg * (o2_5 * Bad0_0 + o8_5 * Bad1_0 + o14_5 * Bad2_0 + o20_5 * Bad3_0 + o26_5 * Bad4_0 + o32_5 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_5 * Bac0_5 + o8_5 * Bac1_5 + o14_5 * Bac2_5 + o20_5 * Bac3_5 + o26_5 * Bac4_5 + o32_5 * Bac5_5));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 5, deg * (o3_5 * Bad0_0 + o9_5 * Bad1_0 + o15_5 * Bad2_0 + o21_5 * Bad3_0 + o27_5 * Bad4_0 + o33_5 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_5 * Bac0_5 + o9_5 * Bac1_5 + o15_5 * Bac2_5 + o21_5 * Bac3_5 + o27_5 * Bac4_5 + o33_5 * Bac5_5));
            atomicAdd(KBacc + (fQ + 4) * N + fI + 5, deg * (o4_5 * Bad0_0 + o10_5 * Bad1_0 + o16_5 * Bad2_0 + o22_5 * Bad3_0 + o28_5 * Bad4_0 + o34_5 * Bad5_0));
            atomicAdd(KBacc + (fQ + 4) * N + fJ + 0, deg * (o4_5 * Bac0_5 + o10_5 * Bac1_5 + o16_5 * Bac2_5 + o22_5 * Bac3_5 + o28_5 * Bac4_5 + o34_5 * Bac5_5));
            atomicAdd(KBacc + (fQ + 5) * N + fI + 5, deg * (o5_5 * Bad0_0 + o11_5 * Bad1_0 + o17_5 * Bad2_0 + o23_5 * Bad3_0 + o29_5 * Bad4_0 + o35_5 * Bad5_0));
            atomicAdd(KBacc + (fQ + 5) * N + fJ + 0, deg * (o5_5 * Bac0_5 + o11_5 * Bac1_5 + o17_5 * Bac2_5 + o23_5 * Bac3_5 + o29_5 * Bac4_5 + o35_5 * Bac5_5));
            atomicAdd(KBacc + (fP + 1) * N + fI + 5, deg * (o6_5 * Bbd0_0 + o7_5 * Bbd1_0 + o8_5 * Bbd2_0 + o9_5 * Bbd3_0 + o10_5 * Bbd4_0 + o11_5 * Bbd5_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o6_5 * Bbc0_5 + o7_5 * Bbc1_5 + o8_5 * Bbc2_5 + o9_5 * Bbc3_5 + o10_5 * Bbc4_5 + o11_5 * Bbc5_5));
            atomicAdd(KBacc + (fP + 2) * N + fI + 5, deg * (o12_5 * Bbd0_0 + o13_5 * Bbd1_0 + o14_5 * Bbd2_0 + o15_5 * Bbd3_0 + o16_5 * Bbd4_0 + o17_5 * Bbd5_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o12_5 * Bbc0_5 + o13_5 * Bbc1_5 + o14_5 * Bbc2_5 + o15_5 * Bbc3_5 + o16_5 * Bbc4_5 + o17_5 * Bbc5_5));
            atomicAdd(KBacc + (fP + 3) * N + fI + 5, deg * (o18_5 * Bbd0_0 + o19_5 * Bbd1_0 + o20_5 * Bbd2_0 + o21_5 * Bbd3_0 + o22_5 * Bbd4_0 + o23_5 * Bbd5_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o18_5 * Bbc0_5 + o19_5 * Bbc1_5 + o20_5 * Bbc2_5 + o21_5 * Bbc3_5 + o22_5 * Bbc4_5 + o23_5 * Bbc5_5));
            atomicAdd(KBacc + (fP + 4) * N + fI + 5, deg * (o24_5 * Bbd0_0 + o25_5 * Bbd1_0 + o26_5 * Bbd2_0 + o27_5 * Bbd3_0 + o28_5 * Bbd4_0 + o29_5 * Bbd5_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o24_5 * Bbc0_5 + o25_5 * Bbc1_5 + o26_5 * Bbc2_5 + o27_5 * Bbc3_5 + o28_5 * Bbc4_5 + o29_5 * Bbc5_5));
            atomicAdd(KBacc + (fP + 5) * N + fI + 5, deg * (o30_5 * Bbd0_0 + o31_5 * Bbd1_0 + o32_5 * Bbd2_0 + o33_5 * Bbd3_0 + o34_5 * Bbd4_0 + o35_5 * Bbd5_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o30_5 * Bbc0_5 + o31_5 * Bbc1_5 + o32_5 * Bbc2_5 + o33_5 * Bbc3_5 + o34_5 * Bbc4_5 + o35_5 * Bbc5_5));
          }
        } break;
        }
      }
      {
        const double s2 = 2.0 * deg;
        double v[32] = {s2 * jab0, s2 * jab1, s2 * jab2, s2 * jab3, s2 * jab4, s2 * jab5, s2 * jab6, s2 * jab7, s2 * jab8, s2 * jab9, s2 * jab10, s2 * jab11, s2 * jab12, s2 * jab13, s2 * jab14, s2 * jab15, s2 * jab16, s2 * jab17, s2 * jab18, s2 * jab19, s2 * jab20, s2 * jab21, s2 * jab22, s2 * jab23, s2 * jab24, s2 * jab25, s2 * jab26, s2 * jab27, s2 * jab28, s2 * jab29, s2 * jab30, s2 * jab31};
        const double s = sqb::warp_sum_scatter<32>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 32 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 6) * N + bp.fQ + ab % 6, s);
      }
      {
        const double s2 = 2.0 * deg;
        double v[4] = {s2 * jab32, s2 * jab33, s2 * jab34, s2 * jab35};
        const double s = sqb::warp_sum_scatter<4>(v);
        const int l = threadIdx.x & 31, ab = l + 32;
        if (l < 4 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 6) * N + bp.fQ + ab % 6, s);
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
