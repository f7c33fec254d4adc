// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DP_PS_U(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fma(ek0_0, r0_2_1_0, g0_18);
              g0_8 = fma(ek0_1, r0_2_1_0, g0_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_19 = fma(ek0_0, r0_3_0_0, g0_19);
              g0_9 = fma(ek0_1, r0_3_0_0, g0_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_1_0_3 = X * r1_0_0_3;
              g0_10 = fma(ek0_1, r0_1_0_3, g0_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_1_1_2 = X * r1_0_1_2;
              g0_11 = fma(ek0_1, r0_1_1_2, g0_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g0_12 = fma(ek0_1, r0_1_2_1, g0_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g0_13 = fma(ek0_1, r0_1_3_0, g0_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g0_14 = fma(ek0_1, r0_2_0_2, g0_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g0_15 = fma(ek0_1, r0_2_1_1, g0_15);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g0_16 = fma(ek0_1, r0_2_2_0, g0_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g0_17 = fma(ek0_1, r0_3_0_1, g0_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g0_18 = fma(ek0_1, r0_3_1_0, g0_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g0_19 = fma(ek0_1, r0_4_0_0, g0_19);
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
              o1_0 = fma(eb, g0_0, o1_0);
            }
            { const double eb = bi[10];
              o1_0 = fma(eb, g0_2, o1_0);
            }
            { const double eb = bi[11];
              o1_0 = fma(eb, g0_3, o1_0);
            }
            { const double eb = bi[12];
              o1_0 = fma(eb, g0_8, o1_0);
            }
            { const double eb = bi[13];
              o1_0 = fma(eb, g0_9, o1_0);
            }
            { const double eb = bi[14];
              o1_0 = fma(eb, g0_18, o1_0);
            }
            { const double eb = bi[15];
              o2_0 = fma(eb, g0_0, o2_0);
            }
            { const double eb = bi[16];
              o2_0 = fma(eb, g0_1, o2_0);
            }
            { const double eb = bi[17];
              o2_0 = fma(eb, g0_3, o2_0);
            }
            { const double eb = bi[18];
              o2_0 = fma(eb, g0_7, o2_0);
            }
            { const double eb = bi[19];
              o2_0 = fma(eb, g0_9, o2_0);
            }
            { const double eb = bi[20];
              o2_0 = fma(eb, g0_17, o2_0);
            }
            { const double eb = bi[21];
              o3_0 = fma(eb, g0_0, o3_0);
            }
            { const double eb = bi[22];
              o3_0 = fma(eb, g0_2, o3_0);
            }
            { const double eb = bi[23];
              o3_0 = fma(eb, g0_6, o3_0);
            }
            { const double eb = bi[24];
              o3_0 = fma(eb, g0_3, o3_0);
            }
            { const double eb = bi[25];
              o3_0 = fma(eb, g0_8, o3_0);
            }
            { const double eb = bi[26];
              o3_0 = fma(eb, g0_16, o3_0);
            }
            { const double eb = bi[27];
              o4_0 = fma(eb, g0_0, o4_0);
            }
            { const double eb = bi[28];
              o4_0 = fma(eb, g0_2, o4_0);
            }
            { const double eb = bi[29];
              o4_0 = fma(eb, g0_6, o4_0);
            }
            { const double eb = bi[30];
              o4_0 = fma(eb, g0_13, o4_0);
            }
            { const double eb = bi[31];
              o5_0 = fma(eb, g0_0, o5_0);
            }
            { const double eb = bi[32];
              o5_0 = fma(eb, g0_1, o5_0);
            }
            { const double eb = bi[33];
              o5_0 = fma(eb, g0_2, o5_0);
            }
            { const double eb = bi[34];
              o5_0 = fma(eb, g0_5, o5_0);
            }
            { const double eb = bi[35];
              o5_0 = fma(eb, g0_6, o5_0);
            }
            { const double eb = bi[36];
              o5_0 = fma(eb, g0_12, o5_0);
            }
            { const double eb = bi[37];
              o6_0 = fma(eb, g0_0, o6_0);
            }
            { const double eb = bi[38];
              o6_0 = fma(eb, g0_1, o6_0);
            }
            { const double eb = bi[39];
              o6_0 = fma(eb, g0_4, o6_0);
            }
            { const double eb = bi[40];
              o6_0 = fma(eb, g0_3, o6_0);
            }
            { const double eb = bi[41];
              o6_0 = fma(eb, g0_7, o6_0);
            }
            { const double eb = bi[42];
              o6_0 = fma(eb, g0_14, o6_0);
            }
            { const double eb = bi[43];
              o7_0 = fma(eb, g0_0, o7_0);
            }
            { const double eb = bi[44];
              o7_0 = fma(eb, g0_1, o7_0);
            }
            { const double eb = bi[45];
              o7_0 = fma(eb, g0_4, o7_0);
            }
            { const double eb = bi[46];
              o7_0 = fma(eb, g0_2, o7_0);
            }
            { const double eb = bi[47];
              o7_0 = fma(eb, g0_5, o7_0);
            }
            { const double eb = bi[48];
              o7_0 = fma(eb, g0_11, o7_0);
            }
            { const double eb = bi[49];
              o8_0 = fma(eb, g0_0, o8_0);
            }
            { const double eb = bi[50];
              o8_0 = fma(eb, g0_1, o8_0);
            }
            { const double eb = bi[51];
              o8_0 = fma(eb, g0_4, o8_0);
            }
            { const double eb = bi[52];
              o8_0 = fma(eb, g0_10, o8_0);
            }
            { const double eb = bi[53];
              o9_0 = fma(eb, g0_0, o9_0);
            }
            { const double eb = bi[54];
              o9_0 = fma(eb, g0_2, o9_0);
            }
            { const double eb = bi[55];
              o9_0 = fma(eb, g0_3, o9_0);
            }
            { const double eb = bi[56];
              o9_0 = fma(eb, g0_8, o9_0);
            }
            { const double eb = bi[57];
              o9_0 = fma(eb, g0_9, o9_0);
            }
            { const double eb = bi[58];
              o9_0 = fma(eb, g0_18, o9_0);
            }
            { const double eb = bi[59];
              o10_0 = fma(eb, g0_0, o10_0);
            }
            { const double eb = bi[60];
              o10_0 = fma(eb, g0_2, o10_0);
            }
            { const double eb = bi[61];
              o10_0 = fma(eb, g0_6, o10_0);
            }
            { const double eb = bi[62];
              o10_0 = fma(eb, g0_3, o10_0);
            }
            { const double eb = bi[63];
              o10_0 = fma(eb, g0_8, o10_0);
            }
            { const double eb = bi[64];
              o10_0 = fma(eb, g0_16, o10_0);
            }
            { const double eb = bi[65];
              o11_0 = fma(eb, g0_0, o11_0);
            }
            { const double eb = bi[66];
              o11_0 = fma(eb, g0_1, o11_0);
            }
            { const double eb = bi[67];
              o11_0 = fma(eb, g0_2, o11_0);
            }
            { const double eb = bi[68];
              o11_0 = fma(eb, g0_5, o11_0);
            }
            { const double eb = bi[69];
              o11_0 = fma(eb, g0_3, o11_0);
            }
            { const double eb = bi[70];
              o11_0 = fma(eb, g0_7, o11_0);
            }
            { const double eb = bi[71];
              o11_0 = fma(eb, g0_8, o11_0);
            }
            { const double eb = bi[72];
              o11_0 = fma(eb, g0_15, o11_0);
            }
            { const double eb = bi[73];
              o12_0 = fma(eb, g0_0, o12_0);
            }
            { const double eb = bi[74];
              o12_0 = fma(eb, g0_1, o12_0);
            }
            { const double eb = bi[75];
              o12_0 = fma(eb, g0_3, o12_0);
            }
            { const double eb = bi[76];
              o12_0 = fma(eb, g0_7, o12_0);
            }
            { const double eb = bi[77];
              o12_0 = fma(eb, g0_9, o12_0);
            }
            { const double eb = bi[78];
              o12_0 = fma(eb, g0_17, o12_0);
            }
            { const double eb = bi[79];
              o13_0 = fma(eb, g0_0, o13_0);
            }
            { const double eb = bi[80];
              o13_0 = fma(eb, g0_1, o13_0);
            }
            { const double eb = bi[81];
              o13_0 = fma(eb, g0_2, o13_0);
            }
            { const double eb = bi[82];
              o13_0 = fma(eb, g0_5, o13_0);
            }
            { const double eb = bi[83];
              o13_0 = fma(eb, g0_3, o13_0);
            }
            { const double eb = bi[84];
              o13_0 = fma(eb, g0_7, o13_0);
            }
            { const double eb = bi[85];
              o13_0 = fma(eb, g0_8, o13_0);
            }
            { const double eb = bi[86];
              o13_0 = fma(eb, g0_15, o13_0);
            }
            { const double eb = bi[87];
              o14_0 = fma(eb, g0_0, o14_0);
            }
            { const double eb = bi[88];
              o14_0 = fma(eb, g0_1, o14_0);
            }
            { const double eb = bi[89];
              o14_0 = fma(eb, g0_4, o14_0);
            }
            { const double eb = bi[90];
              o14_0 = fma(eb, g0_3, o14_0);
            }
            { const double eb = bi[91];
              o14_0 = fma(eb, g0_7, o14_0);
            }
            { const double eb = bi[92];
              o14_0 = fma(eb, g0_14, o14_0);
            }
            { const double eb = bi[93];
              o15_0 = fma(eb, g0_0, o15_0);
            }
            { const double eb = bi[94];
              o15_0 = fma(eb, g0_1, o15_0);
            }
            { const double eb = bi[95];
              o15_0 = fma(eb, g0_2, o15_0);
            }
            { const double eb = bi[96];
              o15_0 = fma(eb, g0_5, o15_0);
            }
            { const double eb = bi[97];
              o15_0 = fma(eb, g0_3, o15_0);
            }
            { const double eb = bi[98];
              o15_0 = fma(eb, g0_7, o15_0);
            }
            { const double eb = bi[99];
              o15_0 = fma(eb, g0_8, o15_0);
            }
            { const double eb = bi[100];
              o15_0 = fma(eb, g0_15, o15_0);
            }
            { const double eb = bi[101];
              o16_0 = fma(eb, g0_0, o16_0);
            }
            { const double eb = bi[102];
              o16_0 = fma(eb, g0_1, o16_0);
            }
            { const double eb = bi[103];
              o16_0 = fma(eb, g0_2, o16_0);
            }
            { const double eb = bi[104];
              o16_0 = fma(eb, g0_5, o16_0);
            }
            { const double eb = bi[105];
              o16_0 = fma(eb, g0_6, o16_0);
            }
            { const double eb = bi[106];
              o16_0 = fma(eb, g0_12, o16_0);
            }
            { const double eb = bi[107];
              o17_0 = fma(eb, g0_0, o17_0);
            }
            { const double eb = bi[108];
              o17_0 = fma(eb, g0_1, o17_0);
            }
            { const double eb = bi[109];
              o17_0 = fma(eb, g0_4, o17_0);
            }
            { const double eb = bi[110];
              o17_0 = fma(eb, g0_2, o17_0);
            }
            { const double eb = bi[111];
              o17_0 = fma(eb, g0_5, o17_0);
            }
            { const double eb = bi[112];
              o17_0 = fma(eb, g0_11, o17_0);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0);
            o1_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 0);
            o2_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 0);
            o3_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0);
            o4_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 0);
            o5_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 0);
            o6_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0);
            o7_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 0);
            o8_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 0);
            o9_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0);
            o10_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 0);
            o11_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 0);
            o12_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0);
            o13_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 0);
            o14_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 0);
            o15_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0);
            o16_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 0);
            o17_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o1_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o2_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o3_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o4_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o5_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o6_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o7_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o8_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o9_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o10_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o11_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o12_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o13_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o14_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o15_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o16_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o17_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
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
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc1_0 = PB[(fQ + 1) * N + fI + 0];
            const double Bbc2_0 = PB[(fQ + 2) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15 + o16_0 * ptb16 + o17_0 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o3_0 * Aad1_0 + o6_0 * Aad2_0 + o9_0 * Aad3_0 + o12_0 * Aad4_0 + o15_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o1_0 * Abc1_0 + o2_0 * Abc2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o3_0 * Aac1_0 + o6_0 * Aac2_0 + o9_0 * Aac3_0 + o12_0 * Aac4_0 + o15_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o4_0 * Aad1_0 + o7_0 * Aad2_0 + o10_0 * Aad3_0 + o13_0 * Aad4_0 + o16_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o4_0 * Aac1_0 + o7_0 * Aac2_0 + o10_0 * Aac3_0 + o13_0 * Aac4_0 + o16_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o5_0 * Aad1_0 + o8_0 * Aad2_0 + o11_0 * Aad3_0 + o14_0 * Aad4_0 + o17_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o5_0 * Aac1_0 + o8_0 * Aac2_0 + o11_0 * Aac3_0 + o14_0 * Aac4_0 + o17_0 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o3_0 * Abd0_0 + o4_0 * Abd1_0 + o5_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o3_0 * Abc0_0 + o4_0 * Abc1_0 + o5_0 * Abc2_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o6_0 * Abd0_0 + o7_0 * Abd1_0 + o8_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o6_0 * Abc0_0 + o7_0 * Abc1_0 + o8_0 * Abc2_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o9_0 * Abd0_0 + o10_0 * Abd1_0 + o11_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o9_0 * Abc0_0 + o10_0 * Abc1_0 + o11_0 * Abc2_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o13_0 * Abc1_0 + o14_0 * Abc2_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o15_0 * Abd0_0 + o16_0 * Abd1_0 + o17_0 * Abd2_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o15_0 * Abc0_0 + o16_0 * Abc1_0 + o17_0 * Abc2_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Bbd0_0 + o1_0 * Bbd1_0 + o2_0 * Bbd2_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Bad0_0 + o3_0 * Bad1_0 + o6_0 * Bad2_0 + o9_0 * Bad3_0 + o12_0 * Bad4_0 + o15_0 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Bbc0_0 + o1_0 * Bbc1_0 + o2_0 * Bbc2_0));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Bac0_0 + o3_0 * Bac1_0 + o6_0 * Bac2_0 + o9_0 * Bac3_0 + o12_0 * Bac4_0 + o15_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Bad0_0 + o4_0 * Bad1_0 + o7_0 * Bad2_0 + o10_0 * Bad3_0 + o13_0 * Bad4_0 + o16_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Bac0_0 + o4_0 * Bac1_0 + o7_0 * Bac2_0 + o10_0 * Bac3_0 + o13_0 * Bac4_0 + o16_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Bad0_0 + o5_0 * Bad1_0 + o8_0 * Bad2_0 + o11_0 * Bad3_0 + o14_0 * Bad4_0 + o17_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Bac0_0 + o5_0 * Bac1_0 + o8_0 * Bac2_0 + o11_0 * Bac3_0 + o14_0 * Bac4_0 + o17_0 * Bac5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o3_0 * Bbd0_0 + o4_0 * Bbd1_0 + o5_0 * Bbd2_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o3_0 * Bbc0_0 + o4_0 * Bbc1_0 + o5_0 * Bbc2_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o6_0 * Bbd0_0 + o7_0 * Bbd1_0 + o8_0 * Bbd2_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o6_0 * Bbc0_0 + o7_0 * Bbc1_0 + o8_0 * Bbc2_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o9_0 * Bbd0_0 + o10_0 * Bbd1_0 + o11_0 * Bbd2_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o9_0 * Bbc0_0 + o10_0 * Bbc1_0 + o11_0 * Bbc2_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o12_0 * Bbd0_0 + o13_0 * Bbd1_0 + o14_0 * Bbd2_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o12_0 * Bbc0_0 + o13_0 * Bbc1_0 + o14_0 * Bbc2_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o15_0 * Bbd0_0 + o16_0 * Bbd1_0 + o17_0 * Bbd2_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o15_0 * Bbc0_0 + o16_0 * Bbc1_0 + o17_0 * Bbc2_0));
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
              const double ek1_0 = kj[7 * kS];
              const double ek1_1 = -kj[8 * kS];
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
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g1_13 = fma(ek1_0, r0_0_3_0, g1_13);
              g1_6 = fma(ek1_1, r0_0_3_0, g1_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g1_14 = fma(ek1_0, r0_1_0_2, g1_14);
              const double r0_1_1_1 = X * r1_0_1_1;
              g1_15 = fma(ek1_0, r0_1_1_1, g1_15);
              g1_7 = fma(ek1_1, r0_1_1_1, g1_7);
              const double r0_1_2_0 = X * r1_0_2_0;
              g1_16 = fma(ek1_0, r0_1_2_0, g1_16);
              g1_8 = fma(ek1_1, r0_1_2_0, g1_8);
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
              const double r0_1_1_2 = X * r1_0_1_2;
              g1_14 = fma(ek1_1, r0_1_1_2, g1_14);
              const double r0_1_2_1 = X * r1_0_2_1;
              g1_15 = fma(ek1_1, r0_1_2_1, g1_15);
              const double r0_1_3_0 = X * r1_0_3_0;
              g1_16 = fma(ek1_1, r0_1_3_0, g1_16);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g1_17 = fma(ek1_1, r0_2_1_1, g1_17);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g1_18 = fma(ek1_1, r0_2_2_0, g1_18);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g1_19 = fma(ek1_1, r0_3_1_0, g1_19);
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
              o1_1 = fma(eb, g1_0, o1_1);
            }
            { const double eb = bi[10];
              o1_1 = fma(eb, g1_2, o1_1);
            }
            { const double eb = bi[11];
              o1_1 = fma(eb, g1_3, o1_1);
            }
            { const double eb = bi[12];
              o1_1 = fma(eb, g1_8, o1_1);
            }
            { const double eb = bi[13];
              o1_1 = fma(eb, g1_9, o1_1);
            }
            { const double eb = bi[14];
              o1_1 = fma(eb, g1_18, o1_1);
            }
            { const double eb = bi[15];
              o2_1 = fma(eb, g1_0, o2_1);
            }
            { const double eb = bi[16];
              o2_1 = fma(eb, g1_1, o2_1);
            }
            { const double eb = bi[17];
              o2_1 = fma(eb, g1_3, o2_1);
            }
            { const double eb = bi[18];
              o2_1 = fma(eb, g1_7, o2_1);
            }
            { const double eb = bi[19];
              o2_1 = fma(eb, g1_9, o2_1);
            }
            { const double eb = bi[20];
              o2_1 = fma(eb, g1_17, o2_1);
            }
            { const double eb = bi[21];
              o3_1 = fma(eb, g1_0, o3_1);
            }
            { const double eb = bi[22];
              o3_1 = fma(eb, g1_2, o3_1);
            }
            { const double eb = bi[23];
              o3_1 = fma(eb, g1_6, o3_1);
            }
            { const double eb = bi[24];
              o3_1 = fma(eb, g1_3, o3_1);
            }
            { const double eb = bi[25];
              o3_1 = fma(eb, g1_8, o3_1);
            }
            { const double eb = bi[26];
              o3_1 = fma(eb, g1_16, o3_1);
            }
            { const double eb = bi[27];
              o4_1 = fma(eb, g1_0, o4_1);
            }
            { const double eb = bi[28];
              o4_1 = fma(eb, g1_2, o4_1);
            }
            { const double eb = bi[29];
              o4_1 = fma(eb, g1_6, o4_1);
            }
            { const double eb = bi[30];
              o4_1 = fma(eb, g1_13, o4_1);
            }
            { const double eb = bi[31];
              o5_1 = fma(eb, g1_0, o5_1);
            }
            { const double eb = bi[32];
              o5_1 = fma(eb, g1_1, o5_1);
            }
            { const double eb = bi[33];
              o5_1 = fma(eb, g1_2, o5_1);
            }
            { const double eb = bi[34];
              o5_1 = fma(eb, g1_5, o5_1);
            }
            { const double eb = bi[35];
              o5_1 = fma(eb, g1_6, o5_1);
            }
            { const double eb = bi[36];
              o5_1 = fma(eb, g1_12, o5_1);
            }
            { const double eb = bi[37];
              o6_1 = fma(eb, g1_0, o6_1);
            }
            { const double eb = bi[38];
              o6_1 = fma(eb, g1_1, o6_1);
            }
            { const double eb = bi[39];
              o6_1 = fma(eb, g1_4, o6_1);
            }
            { const double eb = bi[40];
              o6_1 = fma(eb, g1_3, o6_1);
            }
            { const double eb = bi[41];
              o6_1 = fma(eb, g1_7, o6_1);
            }
            { const double eb = bi[42];
              o6_1 = fma(eb, g1_14, o6_1);
            }
            { const double eb = bi[43];
              o7_1 = fma(eb, g1_0, o7_1);
            }
            { const double eb = bi[44];
              o7_1 = fma(eb, g1_1, o7_1);
            }
            { const double eb = bi[45];
              o7_1 = fma(eb, g1_4, o7_1);
            }
            { const double eb = bi[46];
              o7_1 = fma(eb, g1_2, o7_1);
            }
            { const double eb = bi[47];
              o7_1 = fma(eb, g1_5, o7_1);
            }
            { const double eb = bi[48];
              o7_1 = fma(eb, g1_11, o7_1);
            }
            { const double eb = bi[49];
              o8_1 = fma(eb, g1_0, o8_1);
            }
            { const double eb = bi[50];
              o8_1 = fma(eb, g1_1, o8_1);
            }
            { const double eb = bi[51];
              o8_1 = fma(eb, g1_4, o8_1);
            }
            { const double eb = bi[52];
              o8_1 = fma(eb, g1_10, o8_1);
            }
            { const double eb = bi[53];
              o9_1 = fma(eb, g1_0, o9_1);
            }
            { const double eb = bi[54];
              o9_1 = fma(eb, g1_2, o9_1);
            }
            { const double eb = bi[55];
              o9_1 = fma(eb, g1_3, o9_1);
            }
            { const double eb = bi[56];
              o9_1 = fma(eb, g1_8, o9_1);
            }
            { const double eb = bi[57];
              o9_1 = fma(eb, g1_9, o9_1);
            }
            { const double eb = bi[58];
              o9_1 = fma(eb, g1_18, o9_1);
            }
            { const double eb = bi[59];
              o10_1 = fma(eb, g1_0, o10_1);
            }
            { const double eb = bi[60];
              o10_1 = fma(eb, g1_2, o10_1);
            }
            { const double eb = bi[61];
              o10_1 = fma(eb, g1_6, o10_1);
            }
            { const double eb = bi[62];
              o10_1 = fma(eb, g1_3, o10_1);
            }
            { const double eb = bi[63];
              o10_1 = fma(eb, g1_8, o10_1);
            }
            { const double eb = bi[64];
              o10_1 = fma(eb, g1_16, o10_1);
            }
            { const double eb = bi[65];
              o11_1 = fma(eb, g1_0, o11_1);
            }
            { const double eb = bi[66];
              o11_1 = fma(eb, g1_1, o11_1);
            }
            { const double eb = bi[67];
              o11_1 = fma(eb, g1_2, o11_1);
            }
            { const double eb = bi[68];
              o11_1 = fma(eb, g1_5, o11_1);
            }
            { const double eb = bi[69];
              o11_1 = fma(eb, g1_3, o11_1);
            }
            { const double eb = bi[70];
              o11_1 = fma(eb, g1_7, o11_1);
            }
            { const double eb = bi[71];
              o11_1 = fma(eb, g1_8, o11_1);
            }
            { const double eb = bi[72];
              o11_1 = fma(eb, g1_15, o11_1);
            }
            { const double eb = bi[73];
              o12_1 = fma(eb, g1_0, o12_1);
            }
            { const double eb = bi[74];
              o12_1 = fma(eb, g1_1, o12_1);
            }
            { const double eb = bi[75];
              o12_1 = fma(eb, g1_3, o12_1);
            }
            { const double eb = bi[76];
              o12_1 = fma(eb, g1_7, o12_1);
            }
            { const double eb = bi[77];
              o12_1 = fma(eb, g1_9, o12_1);
            }
            { const double eb = bi[78];
              o12_1 = fma(eb, g1_17, o12_1);
            }
            { const double eb = bi[79];
              o13_1 = fma(eb, g1_0, o13_1);
            }
            { const double eb = bi[80];
              o13_1 = fma(eb, g1_1, o13_1);
            }
            { const double eb = bi[81];
              o13_1 = fma(eb, g1_2, o13_1);
            }
            { const double eb = bi[82];
              o13_1 = fma(eb, g1_5, o13_1);
            }
            { const double eb = bi[83];
              o13_1 = fma(eb, g1_3, o13_1);
            }
            { const double eb = bi[84];
              o13_1 = fma(eb, g1_7, o13_1);
            }
            { const double eb = bi[85];
              o13_1 = fma(eb, g1_8, o13_1);
            }
            { const double eb = bi[86];
              o13_1 = fma(eb, g1_15, o13_1);
            }
            { const double eb = bi[87];
              o14_1 = fma(eb, g1_0, o14_1);
            }
            { const double eb = bi[88];
              o14_1 = fma(eb, g1_1, o14_1);
            }
            { const double eb = bi[89];
              o14_1 = fma(eb, g1_4, o14_1);
            }
            { const double eb = bi[90];
              o14_1 = fma(eb, g1_3, o14_1);
            }
            { const double eb = bi[91];
              o14_1 = fma(eb, g1_7, o14_1);
            }
            { const double eb = bi[92];
              o14_1 = fma(eb, g1_14, o14_1);
            }
            { const double eb = bi[93];
              o15_1 = fma(eb, g1_0, o15_1);
            }
            { const double eb = bi[94];
              o15_1 = fma(eb, g1_1, o15_1);
            }
            { const double eb = bi[95];
              o15_1 = fma(eb, g1_2, o15_1);
            }
            { const double eb = bi[96];
              o15_1 = fma(eb, g1_5, o15_1);
            }
            { const double eb = bi[97];
              o15_1 = fma(eb, g1_3, o15_1);
            }
            { const double eb = bi[98];
              o15_1 = fma(eb, g1_7, o15_1);
            }
            { const double eb = bi[99];
              o15_1 = fma(eb, g1_8, o15_1);
            }
            { const double eb = bi[100];
              o15_1 = fma(eb, g1_15, o15_1);
            }
            { const double eb = bi[101];
              o16_1 = fma(eb, g1_0, o16_1);
            }
            { const double eb = bi[102];
              o16_1 = fma(eb, g1_1, o16_1);
            }
            { const double eb = bi[103];
              o16_1 = fma(eb, g1_2, o16_1);
            }
            { const double eb = bi[104];
              o16_1 = fma(eb, g1_5, o16_1);
            }
            { const double eb = bi[105];
              o16_1 = fma(eb, g1_6, o16_1);
            }
            { const double eb = bi[106];
              o16_1 = fma(eb, g1_12, o16_1);
            }
            { const double eb = bi[107];
              o17_1 = fma(eb, g1_0, o17_1);
            }
            { const double eb = bi[108];
              o17_1 = fma(eb, g1_1, o17_1);
            }
            { const double eb = bi[109];
              o17_1 = fma(eb, g1_4, o17_1);
            }
            { const double eb = bi[110];
              o17_1 = fma(eb, g1_2, o17_1);
            }
            { const double eb = bi[111];
              o17_1 = fma(eb, g1_5, o17_1);
            }
            { const double eb = bi[112];
              o17_1 = fma(eb, g1_11, o17_1);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0);
            o1_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 0);
            o2_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 0);
            o3_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0);
            o4_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 0);
            o5_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 0);
            o6_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0);
            o7_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 0);
            o8_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 0);
            o9_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0);
            o10_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 0);
            o11_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 0);
            o12_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0);
            o13_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 0);
            o14_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 0);
            o15_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0);
            o16_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 0);
            o17_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o1_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o2_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o3_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o4_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o5_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o6_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o7_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o8_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o9_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o10_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o11_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o12_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o13_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o14_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o15_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o16_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o17_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk1 = PT[(fI + 1) * N + fJ + 0];
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
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_1 = PB[(fQ + 0) * N + fI + 1];
            const double Bbc1_1 = PB[(fQ + 1) * N + fI + 1];
            const double Bbc2_1 = PB[(fQ + 2) * N + fI + 1];
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
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Abd0_0 + o1_1 * Abd1_0 + o2_1 * Abd2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Aad0_0 + o3_1 * Aad1_0 + o6_1 * Aad2_0 + o9_1 * Aad3_0 + o12_1 * Aad4_0 + o15_1 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_1 * Abc0_1 + o1_1 * Abc1_1 + o2_1 * Abc2_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_1 * Aac0_1 + o3_1 * Aac1_1 + o6_1 * Aac2_1 + o9_1 * Aac3_1 + o12_1 * Aac4_1 + o15_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_1 * Aad0_0 + o4_1 * Aad1_0 + o7_1 * Aad2_0 + o10_1 * Aad3_0 + o13_1 * Aad4_0 + o16_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_1 * Aac0_1 + o4_1 * Aac1_1 + o7_1 * Aac2_1 + o10_1 * Aac3_1 + o13_1 * Aac4_1 + o16_1 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_1 * Aad0_0 + o5_1 * Aad1_0 + o8_1 * Aad2_0 + o11_1 * Aad3_0 + o14_1 * Aad4_0 + o17_1 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_1 * Aac0_1 + o5_1 * Aac1_1 + o8_1 * Aac2_1 + o11_1 * Aac3_1 + o14_1 * Aac4_1 + o17_1 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o3_1 * Abd0_0 + o4_1 * Abd1_0 + o5_1 * Abd2_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o3_1 * Abc0_1 + o4_1 * Abc1_1 + o5_1 * Abc2_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o6_1 * Abd0_0 + o7_1 * Abd1_0 + o8_1 * Abd2_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o6_1 * Abc0_1 + o7_1 * Abc1_1 + o8_1 * Abc2_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o9_1 * Abd0_0 + o10_1 * Abd1_0 + o11_1 * Abd2_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o9_1 * Abc0_1 + o10_1 * Abc1_1 + o11_1 * Abc2_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o12_1 * Abd0_0 + o13_1 * Abd1_0 + o14_1 * Abd2_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o12_1 * Abc0_1 + o13_1 * Abc1_1 + o14_1 * Abc2_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o15_1 * Abd0_0 + o16_1 * Abd1_0 + o17_1 * Abd2_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o15_1 * Abc0_1 + o16_1 * Abc1_1 + o17_1 * Abc2_1));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Bbd0_0 + o1_1 * Bbd1_0 + o2_1 * Bbd2_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Bad0_0 + o3_1 * Bad1_0 + o6_1 * Bad2_0 + o9_1 * Bad3_0 + o12_1 * Bad4_0 + o15_1 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_1 * Bbc0_1 + o1_1 * Bbc1_1 + o2_1 * Bbc2_1));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_1 * Bac0_1 + o3_1 * Bac1_1 + o6_1 * Bac2_1 + o9_1 * Bac3_1 + o12_1 * Bac4_1 + o15_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 1, deg * (o1_1 * Bad0_0 + o4_1 * Bad1_0 + o7_1 * Bad2_0 + o10_1 * Bad3_0 + o13_1 * Bad4_0 + o16_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_1 * Bac0_1 + o4_1 * Bac1_1 + o7_1 * Bac2_1 + o10_1 * Bac3_1 + o13_1 * Bac4_1 + o16_1 * Bac5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 1, deg * (o2_1 * Bad0_0 + o5_1 * Bad1_0 + o8_1 * Bad2_0 + o11_1 * Bad3_0 + o14_1 * Bad4_0 + o17_1 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_1 * Bac0_1 + o5_1 * Bac1_1 + o8_1 * Bac2_1 + o11_1 * Bac3_1 + o14_1 * Bac4_1 + o17_1 * Bac5_1));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o3_1 * Bbd0_0 + o4_1 * Bbd1_0 + o5_1 * Bbd2_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o3_1 * Bbc0_1 + o4_1 * Bbc1_1 + o5_1 * Bbc2_1));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o6_1 * Bbd0_0 + o7_1 * Bbd1_0 + o8_1 * Bbd2_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o6_1 * Bbc0_1 + o7_1 * Bbc1_1 + o8_1 * Bbc2_1));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o9_1 * Bbd0_0 + o10_1 * Bbd1_0 + o11_1 * Bbd2_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o9_1 * Bbc0_1 + o10_1 * Bbc1_1 + o11_1 * Bbc2_1));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o12_1 * Bbd0_0 + o13_1 * Bbd1_0 + o14_1 * Bbd2_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o12_1 * Bbc0_1 + o13_1 * Bbc1_1 + o14_1 * Bbc2_1));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o15_1 * Bbd0_0 + o16_1 * Bbd1_0 + o17_1 * Bbd2_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o15_1 * Bbc0_1 + o16_1 * Bbc1_1 + o17_1 * Bbc2_1));
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
              o0_2 = fma(eb, g2_19, o0_2);
            }
            { const double eb = bi[9];
              o1_2 = fma(eb, g2_0, o1_2);
            }
            { const double eb = bi[10];
              o1_2 = fma(eb, g2_2, o1_2);
            }
            { const double eb = bi[11];
              o1_2 = fma(eb, g2_3, o1_2);
            }
            { const double eb = bi[12];
              o1_2 = fma(eb, g2_8, o1_2);
            }
            { const double eb = bi[13];
              o1_2 = fma(eb, g2_9, o1_2);
            }
            { const double eb = bi[14];
              o1_2 = fma(eb, g2_18, o1_2);
            }
            { const double eb = bi[15];
              o2_2 = fma(eb, g2_0, o2_2);
            }
            { const double eb = bi[16];
              o2_2 = fma(eb, g2_1, o2_2);
            }
            { const double eb = bi[17];
              o2_2 = fma(eb, g2_3, o2_2);
            }
            { const double eb = bi[18];
              o2_2 = fma(eb, g2_7, o2_2);
            }
            { const double eb = bi[19];
              o2_2 = fma(eb, g2_9, o2_2);
            }
            { const double eb = bi[20];
              o2_2 = fma(eb, g2_17, o2_2);
            }
            { const double eb = bi[21];
              o3_2 = fma(eb, g2_0, o3_2);
            }
            { const double eb = bi[22];
              o3_2 = fma(eb, g2_2, o3_2);
            }
            { const double eb = bi[23];
              o3_2 = fma(eb, g2_6, o3_2);
            }
            { const double eb = bi[24];
              o3_2 = fma(eb, g2_3, o3_2);
            }
            { const double eb = bi[25];
              o3_2 = fma(eb, g2_8, o3_2);
            }
            { const double eb = bi[26];
              o3_2 = fma(eb, g2_16, o3_2);
            }
            { const double eb = bi[27];
              o4_2 = fma(eb, g2_0, o4_2);
            }
            { const double eb = bi[28];
              o4_2 = fma(eb, g2_2, o4_2);
            }
            { const double eb = bi[29];
              o4_2 = fma(eb, g2_6, o4_2);
            }
            { const double eb = bi[30];
              o4_2 = fma(eb, g2_13, o4_2);
            }
            { const double eb = bi[31];
              o5_2 = fma(eb, g2_0, o5_2);
            }
            { const double eb = bi[32];
              o5_2 = fma(eb, g2_1, o5_2);
            }
            { const double eb = bi[33];
              o5_2 = fma(eb, g2_2, o5_2);
            }
            { const double eb = bi[34];
              o5_2 = fma(eb, g2_5, o5_2);
            }
            { const double eb = bi[35];
              o5_2 = fma(eb, g2_6, o5_2);
            }
            { const double eb = bi[36];
              o5_2 = fma(eb, g2_12, o5_2);
            }
            { const double eb = bi[37];
              o6_2 = fma(eb, g2_0, o6_2);
            }
            { const double eb = bi[38];
              o6_2 = fma(eb, g2_1, o6_2);
            }
            { const double eb = bi[39];
              o6_2 = fma(eb, g2_4, o6_2);
            }
            { const double eb = bi[40];
              o6_2 = fma(eb, g2_3, o6_2);
            }
            { const double eb = bi[41];
              o6_2 = fma(eb, g2_7, o6_2);
            }
            { const double eb = bi[42];
              o6_2 = fma(eb, g2_14, o6_2);
            }
            { const double eb = bi[43];
              o7_2 = fma(eb, g2_0, o7_2);
            }
            { const double eb = bi[44];
              o7_2 = fma(eb, g2_1, o7_2);
            }
            { const double eb = bi[45];
              o7_2 = fma(eb, g2_4, o7_2);
            }
            { const double eb = bi[46];
              o7_2 = fma(eb, g2_2, o7_2);
            }
            { const double eb = bi[47];
              o7_2 = fma(eb, g2_5, o7_2);
            }
            { const double eb = bi[48];
              o7_2 = fma(eb, g2_11, o7_2);
            }
            { const double eb = bi[49];
              o8_2 = fma(eb, g2_0, o8_2);
            }
            { const double eb = bi[50];
              o8_2 = fma(eb, g2_1, o8_2);
            }
            { const double eb = bi[51];
              o8_2 = fma(eb, g2_4, o8_2);
            }
            { const double eb = bi[52];
              o8_2 = fma(eb, g2_10, o8_2);
            }
            { const double eb = bi[53];
              o9_2 = fma(eb, g2_0, o9_2);
            }
            { const double eb = bi[54];
              o9_2 = fma(eb, g2_2, o9_2);
            }
            { const double eb = bi[55];
              o9_2 = fma(eb, g2_3, o9_2);
            }
            { const double eb = bi[56];
              o9_2 = fma(eb, g2_8, o9_2);
            }
            { const double eb = bi[57];
              o9_2 = fma(eb, g2_9, o9_2);
            }
            { const double eb = bi[58];
              o9_2 = fma(eb, g2_18, o9_2);
            }
            { const double eb = bi[59];
              o10_2 = fma(eb, g2_0, o10_2);
            }
            { const double eb = bi[60];
              o10_2 = fma(eb, g2_2, o10_2);
            }
            { const double eb = bi[61];
              o10_2 = fma(eb, g2_6, o10_2);
            }
            { const double eb = bi[62];
              o10_2 = fma(eb, g2_3, o10_2);
            }
            { const double eb = bi[63];
              o10_2 = fma(eb, g2_8, o10_2);
            }
            { const double eb = bi[64];
              o10_2 = fma(eb, g2_16, o10_2);
            }
            { const double eb = bi[65];
              o11_2 = fma(eb, g2_0, o11_2);
            }
            { const double eb = bi[66];
              o11_2 = fma(eb, g2_1, o11_2);
            }
            { const double eb = bi[67];
              o11_2 = fma(eb, g2_2, o11_2);
            }
            { const double eb = bi[68];
              o11_2 = fma(eb, g2_5, o11_2);
            }
            { const double eb = bi[69];
              o11_2 = fma(eb, g2_3, o11_2);
            }
            { const double eb = bi[70];
              o11_2 = fma(eb, g2_7, o11_2);
            }
            { const double eb = bi[71];
              o11_2 = fma(eb, g2_8, o11_2);
            }
            { const double eb = bi[72];
              o11_2 = fma(eb, g2_15, o11_2);
            }
            { const double eb = bi[73];
              o12_2 = fma(eb, g2_0, o12_2);
            }
            { const double eb = bi[74];
              o12_2 = fma(eb, g2_1, o12_2);
            }
            { const double eb = bi[75];
              o12_2 = fma(eb, g2_3, o12_2);
            }
            { const double eb = bi[76];
              o12_2 = fma(eb, g2_7, o12_2);
            }
            { const double eb = bi[77];
              o12_2 = fma(eb, g2_9, o12_2);
            }
            { const double eb = bi[78];
              o12_2 = fma(eb, g2_17, o12_2);
            }
            { const double eb = bi[79];
              o13_2 = fma(eb, g2_0, o13_2);
            }
            { const double eb = bi[80];
              o13_2 = fma(eb, g2_1, o13_2);
            }
            { const double eb = bi[81];
              o13_2 = fma(eb, g2_2, o13_2);
            }
            { const double eb = bi[82];
              o13_2 = fma(eb, g2_5, o13_2);
            }
            { const double eb = bi[83];
              o13_2 = fma(eb, g2_3, o13_2);
            }
            { const double eb = bi[84];
              o13_2 = fma(eb, g2_7, o13_2);
            }
            { const double eb = bi[85];
              o13_2 = fma(eb, g2_8, o13_2);
            }
            { const double eb = bi[86];
              o13_2 = fma(eb, g2_15, o13_2);
            }
            { const double eb = bi[87];
              o14_2 = fma(eb, g2_0, o14_2);
            }
            { const double eb = bi[88];
              o14_2 = fma(eb, g2_1, o14_2);
            }
            { const double eb = bi[89];
              o14_2 = fma(eb, g2_4, o14_2);
            }
            { const double eb = bi[90];
              o14_2 = fma(eb, g2_3, o14_2);
            }
            { const double eb = bi[91];
              o14_2 = fma(eb, g2_7, o14_2);
            }
            { const double eb = bi[92];
              o14_2 = fma(eb, g2_14, o14_2);
            }
            { const double eb = bi[93];
              o15_2 = fma(eb, g2_0, o15_2);
            }
            { const double eb = bi[94];
              o15_2 = fma(eb, g2_1, o15_2);
            }
            { const double eb = bi[95];
              o15_2 = fma(eb, g2_2, o15_2);
            }
            { const double eb = bi[96];
              o15_2 = fma(eb, g2_5, o15_2);
            }
            { const double eb = bi[97];
              o15_2 = fma(eb, g2_3, o15_2);
            }
            { const double eb = bi[98];
              o15_2 = fma(eb, g2_7, o15_2);
            }
            { const double eb = bi[99];
              o15_2 = fma(eb, g2_8, o15_2);
            }
            { const double eb = bi[100];
              o15_2 = fma(eb, g2_15, o15_2);
            }
            { const double eb = bi[101];
              o16_2 = fma(eb, g2_0, o16_2);
            }
            { const double eb = bi[102];
              o16_2 = fma(eb, g2_1, o16_2);
            }
            { const double eb = bi[103];
              o16_2 = fma(eb, g2_2, o16_2);
            }
            { const double eb = bi[104];
              o16_2 = fma(eb, g2_5, o16_2);
            }
            { const double eb = bi[105];
              o16_2 = fma(eb, g2_6, o16_2);
            }
            { const double eb = bi[106];
              o16_2 = fma(eb, g2_12, o16_2);
            }
            { const double eb = bi[107];
              o17_2 = fma(eb, g2_0, o17_2);
            }
            { const double eb = bi[108];
              o17_2 = fma(eb, g2_1, o17_2);
            }
            { const double eb = bi[109];
              o17_2 = fma(eb, g2_4, o17_2);
            }
            { const double eb = bi[110];
              o17_2 = fma(eb, g2_2, o17_2);
            }
            { const double eb = bi[111];
              o17_2 = fma(eb, g2_5, o17_2);
            }
            { const double eb = bi[112];
              o17_2 = fma(eb, g2_11, o17_2);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0);
            o1_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 0);
            o2_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 0);
            o3_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0);
            o4_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 0);
            o5_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 0);
            o6_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0);
            o7_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 0);
            o8_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 0);
            o9_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0);
            o10_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 0);
            o11_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 0);
            o12_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0);
            o13_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 0);
            o14_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 0);
            o15_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0);
            o16_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 0);
            o17_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o1_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o2_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o3_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o4_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o5_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o6_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o7_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o8_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o9_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o10_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o11_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o12_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o13_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o14_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o15_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o16_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o17_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 2) * N + fJ + 0];
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
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_2 = PB[(fQ + 0) * N + fI + 2];
            const double Bbc1_2 = PB[(fQ + 1) * N + fI + 2];
            const double Bbc2_2 = PB[(fQ + 2) * N + fI + 2];
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
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Abd0_0 + o1_2 * Abd1_0 + o2_2 * Abd2_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Aad0_0 + o3_2 * Aad1_0 + o6_2 * Aad2_0 + o9_2 * Aad3_0 + o12_2 * Aad4_0 + o15_2 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_2 * Abc0_2 + o1_2 * Abc1_2 + o2_2 * Abc2_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_2 * Aac0_2 + o3_2 * Aac1_2 + o6_2 * Aac2_2 + o9_2 * Aac3_2 + o12_2 * Aac4_2 + o15_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_2 * Aad0_0 + o4_2 * Aad1_0 + o7_2 * Aad2_0 + o10_2 * Aad3_0 + o13_2 * Aad4_0 + o16_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_2 * Aac0_2 + o4_2 * Aac1_2 + o7_2 * Aac2_2 + o10_2 * Aac3_2 + o13_2 * Aac4_2 + o16_2 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_2 * Aad0_0 + o5_2 * Aad1_0 + o8_2 * Aad2_0 + o11_2 * Aad3_0 + o14_2 * Aad4_0 + o17_2 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_2 * Aac0_2 + o5_2 * Aac1_2 + o8_2 * Aac2_2 + o11_2 * Aac3_2 + o14_2 * Aac4_2 + o17_2 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o3_2 * Abd0_0 + o4_2 * Abd1_0 + o5_2 * Abd2_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o3_2 * Abc0_2 + o4_2 * Abc1_2 + o5_2 * Abc2_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o6_2 * Abd0_0 + o7_2 * Abd1_0 + o8_2 * Abd2_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o6_2 * Abc0_2 + o7_2 * Abc1_2 + o8_2 * Abc2_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o9_2 * Abd0_0 + o10_2 * Abd1_0 + o11_2 * Abd2_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o9_2 * Abc0_2 + o10_2 * Abc1_2 + o11_2 * Abc2_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o12_2 * Abd0_0 + o13_2 * Abd1_0 + o14_2 * Abd2_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o12_2 * Abc0_2 + o13_2 * Abc1_2 + o14_2 * Abc2_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o15_2 * Abd0_0 + o16_2 * Abd1_0 + o17_2 * Abd2_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o15_2 * Abc0_2 + o16_2 * Abc1_2 + o17_2 * Abc2_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Bbd0_0 + o1_2 * Bbd1_0 + o2_2 * Bbd2_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Bad0_0 + o3_2 * Bad1_0 + o6_2 * Bad2_0 + o9_2 * Bad3_0 + o12_2 * Bad4_0 + o15_2 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_2 * Bbc0_2 + o1_2 * Bbc1_2 + o2_2 * Bbc2_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_2 * Bac0_2 + o3_2 * Bac1_2 + o6_2 * Bac2_2 + o9_2 * Bac3_2 + o12_2 * Bac4_2 + o15_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 2, deg * (o1_2 * Bad0_0 + o4_2 * Bad1_0 + o7_2 * Bad2_0 + o10_2 * Bad3_0 + o13_2 * Bad4_0 + o16_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_2 * Bac0_2 + o4_2 * Bac1_2 + o7_2 * Bac2_2 + o10_2 * Bac3_2 + o13_2 * Bac4_2 + o16_2 * Bac5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 2, deg * (o2_2 * Bad0_0 + o5_2 * Bad1_0 + o8_2 * Bad2_0 + o11_2 * Bad3_0 + o14_2 * Bad4_0 + o17_2 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_2 * Bac0_2 + o5_2 * Bac1_2 + o8_2 * Bac2_2 + o11_2 * Bac3_2 + o14_2 * Bac4_2 + o17_2 * Bac5_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o3_2 * Bbd0_0 + o4_2 * Bbd1_0 + o5_2 * Bbd2_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o3_2 * Bbc0_2 + o4_2 * Bbc1_2 + o5_2 * Bbc2_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o6_2 * Bbd0_0 + o7_2 * Bbd1_0 + o8_2 * Bbd2_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o6_2 * Bbc0_2 + o7_2 * Bbc1_2 + o8_2 * Bbc2_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o9_2 * Bbd0_0 + o10_2 * Bbd1_0 + o11_2 * Bbd2_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o9_2 * Bbc0_2 + o10_2 * Bbc1_2 + o11_2 * Bbc2_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o12_2 * Bbd0_0 + o13_2 * Bbd1_0 + o14_2 * Bbd2_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o12_2 * Bbc0_2 + o13_2 * Bbc1_2 + o14_2 * Bbc2_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o15_2 * Bbd0_0 + o16_2 * Bbd1_0 + o17_2 * Bbd2_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o15_2 * Bbc0_2 + o16_2 * Bbc1_2 + o17_2 * Bbc2_2));
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
