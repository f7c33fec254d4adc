// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DL_LL_U(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              ++nprimq;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[4];
              sqb::boys<3>(T, a.boys_tab, F);
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
              const double ek0_0 = kj[5 * kS];
              g0_0 = fma(ek0_0, b0, g0_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
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
              const double r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fma(ek0_0, r0_1_1_0, g0_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g0_9 = fma(ek0_0, r0_2_0_0, g0_9);
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
              const double r0_1_1_1 = X * r1_0_1_1;
              g0_15 = fma(ek0_0, r0_1_1_1, g0_15);
              const double r0_1_2_0 = X * r1_0_2_0;
              g0_16 = fma(ek0_0, r0_1_2_0, g0_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g0_17 = fma(ek0_0, r0_2_0_1, g0_17);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fma(ek0_0, r0_2_1_0, g0_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_19 = fma(ek0_0, r0_3_0_0, g0_19);
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
              o1_0 = fma(eb, g0_0, o1_0);
            }
            { const double eb = bi[9];
              o1_0 = fma(eb, g0_3, o1_0);
            }
            { const double eb = bi[10];
              o1_0 = fma(eb, g0_9, o1_0);
            }
            { const double eb = bi[11];
              o1_0 = fma(eb, g0_19, o1_0);
            }
            { const double eb = bi[12];
              o2_0 = fma(eb, g0_0, o2_0);
            }
            { const double eb = bi[13];
              o2_0 = fma(eb, g0_2, o2_0);
            }
            { const double eb = bi[14];
              o2_0 = fma(eb, g0_3, o2_0);
            }
            { const double eb = bi[15];
              o2_0 = fma(eb, g0_8, o2_0);
            }
            { const double eb = bi[16];
              o2_0 = fma(eb, g0_9, o2_0);
            }
            { const double eb = bi[17];
              o2_0 = fma(eb, g0_18, o2_0);
            }
            { const double eb = bi[18];
              o3_0 = fma(eb, g0_0, o3_0);
            }
            { const double eb = bi[19];
              o3_0 = fma(eb, g0_1, o3_0);
            }
            { const double eb = bi[20];
              o3_0 = fma(eb, g0_3, o3_0);
            }
            { const double eb = bi[21];
              o3_0 = fma(eb, g0_7, o3_0);
            }
            { const double eb = bi[22];
              o3_0 = fma(eb, g0_9, o3_0);
            }
            { const double eb = bi[23];
              o3_0 = fma(eb, g0_17, o3_0);
            }
            { const double eb = bi[24];
              o4_0 = fma(eb, g0_0, o4_0);
            }
            { const double eb = bi[25];
              o4_0 = fma(eb, g0_2, o4_0);
            }
            { const double eb = bi[26];
              o4_0 = fma(eb, g0_6, o4_0);
            }
            { const double eb = bi[27];
              o5_0 = fma(eb, g0_0, o5_0);
            }
            { const double eb = bi[28];
              o5_0 = fma(eb, g0_2, o5_0);
            }
            { const double eb = bi[29];
              o5_0 = fma(eb, g0_6, o5_0);
            }
            { const double eb = bi[30];
              o5_0 = fma(eb, g0_3, o5_0);
            }
            { const double eb = bi[31];
              o5_0 = fma(eb, g0_8, o5_0);
            }
            { const double eb = bi[32];
              o5_0 = fma(eb, g0_16, o5_0);
            }
            { const double eb = bi[33];
              o6_0 = fma(eb, g0_0, o6_0);
            }
            { const double eb = bi[34];
              o6_0 = fma(eb, g0_2, o6_0);
            }
            { const double eb = bi[35];
              o6_0 = fma(eb, g0_6, o6_0);
            }
            { const double eb = bi[36];
              o6_0 = fma(eb, g0_13, o6_0);
            }
            { const double eb = bi[37];
              o7_0 = fma(eb, g0_0, o7_0);
            }
            { const double eb = bi[38];
              o7_0 = fma(eb, g0_1, o7_0);
            }
            { const double eb = bi[39];
              o7_0 = fma(eb, g0_2, o7_0);
            }
            { const double eb = bi[40];
              o7_0 = fma(eb, g0_5, o7_0);
            }
            { const double eb = bi[41];
              o7_0 = fma(eb, g0_6, o7_0);
            }
            { const double eb = bi[42];
              o7_0 = fma(eb, g0_12, o7_0);
            }
            { const double eb = bi[43];
              o8_0 = fma(eb, g0_0, o8_0);
            }
            { const double eb = bi[44];
              o8_0 = fma(eb, g0_1, o8_0);
            }
            { const double eb = bi[45];
              o8_0 = fma(eb, g0_4, o8_0);
            }
            { const double eb = bi[46];
              o9_0 = fma(eb, g0_0, o9_0);
            }
            { const double eb = bi[47];
              o9_0 = fma(eb, g0_1, o9_0);
            }
            { const double eb = bi[48];
              o9_0 = fma(eb, g0_4, o9_0);
            }
            { const double eb = bi[49];
              o9_0 = fma(eb, g0_3, o9_0);
            }
            { const double eb = bi[50];
              o9_0 = fma(eb, g0_7, o9_0);
            }
            { const double eb = bi[51];
              o9_0 = fma(eb, g0_14, o9_0);
            }
            { const double eb = bi[52];
              o10_0 = fma(eb, g0_0, o10_0);
            }
            { const double eb = bi[53];
              o10_0 = fma(eb, g0_1, o10_0);
            }
            { const double eb = bi[54];
              o10_0 = fma(eb, g0_4, o10_0);
            }
            { const double eb = bi[55];
              o10_0 = fma(eb, g0_2, o10_0);
            }
            { const double eb = bi[56];
              o10_0 = fma(eb, g0_5, o10_0);
            }
            { const double eb = bi[57];
              o10_0 = fma(eb, g0_11, o10_0);
            }
            { const double eb = bi[58];
              o11_0 = fma(eb, g0_0, o11_0);
            }
            { const double eb = bi[59];
              o11_0 = fma(eb, g0_1, o11_0);
            }
            { const double eb = bi[60];
              o11_0 = fma(eb, g0_4, o11_0);
            }
            { const double eb = bi[61];
              o11_0 = fma(eb, g0_10, o11_0);
            }
            { const double eb = bi[62];
              o12_0 = fma(eb, g0_0, o12_0);
            }
            { const double eb = bi[63];
              o12_0 = fma(eb, g0_2, o12_0);
            }
            { const double eb = bi[64];
              o12_0 = fma(eb, g0_3, o12_0);
            }
            { const double eb = bi[65];
              o12_0 = fma(eb, g0_8, o12_0);
            }
            { const double eb = bi[66];
              o13_0 = fma(eb, g0_0, o13_0);
            }
            { const double eb = bi[67];
              o13_0 = fma(eb, g0_2, o13_0);
            }
            { const double eb = bi[68];
              o13_0 = fma(eb, g0_3, o13_0);
            }
            { const double eb = bi[69];
              o13_0 = fma(eb, g0_8, o13_0);
            }
            { const double eb = bi[70];
              o13_0 = fma(eb, g0_9, o13_0);
            }
            { const double eb = bi[71];
              o13_0 = fma(eb, g0_18, o13_0);
            }
            { const double eb = bi[72];
              o14_0 = fma(eb, g0_0, o14_0);
            }
            { const double eb = bi[73];
              o14_0 = fma(eb, g0_2, o14_0);
            }
            { const double eb = bi[74];
              o14_0 = fma(eb, g0_6, o14_0);
            }
            { const double eb = bi[75];
              o14_0 = fma(eb, g0_3, o14_0);
            }
            { const double eb = bi[76];
              o14_0 = fma(eb, g0_8, o14_0);
            }
            { const double eb = bi[77];
              o14_0 = fma(eb, g0_16, o14_0);
            }
            { const double eb = bi[78];
              o15_0 = fma(eb, g0_0, o15_0);
            }
            { const double eb = bi[79];
              o15_0 = fma(eb, g0_1, o15_0);
            }
            { const double eb = bi[80];
              o15_0 = fma(eb, g0_2, o15_0);
            }
            { const double eb = bi[81];
              o15_0 = fma(eb, g0_5, o15_0);
            }
            { const double eb = bi[82];
              o15_0 = fma(eb, g0_3, o15_0);
            }
            { const double eb = bi[83];
              o15_0 = fma(eb, g0_7, o15_0);
            }
            { const double eb = bi[84];
              o15_0 = fma(eb, g0_8, o15_0);
            }
            { const double eb = bi[85];
              o15_0 = fma(eb, g0_15, o15_0);
            }
            { const double eb = bi[86];
              o16_0 = fma(eb, g0_0, o16_0);
            }
            { const double eb = bi[87];
              o16_0 = fma(eb, g0_1, o16_0);
            }
            { const double eb = bi[88];
              o16_0 = fma(eb, g0_3, o16_0);
            }
            { const double eb = bi[89];
              o16_0 = fma(eb, g0_7, o16_0);
            }
            { const double eb = bi[90];
              o17_0 = fma(eb, g0_0, o17_0);
            }
            { const double eb = bi[91];
              o17_0 = fma(eb, g0_1, o17_0);
            }
            { const double eb = bi[92];
              o17_0 = fma(eb, g0_3, o17_0);
            }
            { const double eb = bi[93];
              o17_0 = fma(eb, g0_7, o17_0);
            }
            { const double eb = bi[94];
              o17_0 = fma(eb, g0_9, o17_0);
            }
            { const double eb = bi[95];
              o17_0 = fma(eb, g0_17, o17_0);
            }
            { const double eb = bi[96];
              o18_0 = fma(eb, g0_0, o18_0);
            }
            { const double eb = bi[97];
              o18_0 = fma(eb, g0_1, o18_0);
            }
            { const double eb = bi[98];
              o18_0 = fma(eb, g0_2, o18_0);
            }
            { const double eb = bi[99];
              o18_0 = fma(eb, g0_5, o18_0);
            }
            { const double eb = bi[100];
              o18_0 = fma(eb, g0_3, o18_0);
            }
            { const double eb = bi[101];
              o18_0 = fma(eb, g0_7, o18_0);
            }
            { const double eb = bi[102];
              o18_0 = fma(eb, g0_8, o18_0);
            }
            { const double eb = bi[103];
              o18_0 = fma(eb, g0_15, o18_0);
            }
            { const double eb = bi[104];
              o19_0 = fma(eb, g0_0, o19_0);
            }
            { const double eb = bi[105];
              o19_0 = fma(eb, g0_1, o19_0);
            }
            { const double eb = bi[106];
              o19_0 = fma(eb, g0_4, o19_0);
            }
            { const double eb = bi[107];
              o19_0 = fma(eb, g0_3, o19_0);
            }
            { const double eb = bi[108];
              o19_0 = fma(eb, g0_7, o19_0);
            }
            { const double eb = bi[109];
              o19_0 = fma(eb, g0_14, o19_0);
            }
            { const double eb = bi[110];
              o20_0 = fma(eb, g0_0, o20_0);
            }
            { const double eb = bi[111];
              o20_0 = fma(eb, g0_1, o20_0);
            }
            { const double eb = bi[112];
              o20_0 = fma(eb, g0_2, o20_0);
            }
            { const double eb = bi[113];
              o20_0 = fma(eb, g0_5, o20_0);
            }
            { const double eb = bi[114];
              o21_0 = fma(eb, g0_0, o21_0);
            }
            { const double eb = bi[115];
              o21_0 = fma(eb, g0_1, o21_0);
            }
            { const double eb = bi[116];
              o21_0 = fma(eb, g0_2, o21_0);
            }
            { const double eb = bi[117];
              o21_0 = fma(eb, g0_5, o21_0);
            }
            { const double eb = bi[118];
              o21_0 = fma(eb, g0_3, o21_0);
            }
            { const double eb = bi[119];
              o21_0 = fma(eb, g0_7, o21_0);
            }
            { const double eb = bi[120];
              o21_0 = fma(eb, g0_8, o21_0);
            }
            { const double eb = bi[121];
              o21_0 = fma(eb, g0_15, o21_0);
            }
            { const double eb = bi[122];
              o22_0 = fma(eb, g0_0, o22_0);
            }
            { const double eb = bi[123];
              o22_0 = fma(eb, g0_1, o22_0);
            }
            { const double eb = bi[124];
              o22_0 = fma(eb, g0_2, o22_0);
            }
            { const double eb = bi[125];
              o22_0 = fma(eb, g0_5, o22_0);
            }
            { const double eb = bi[126];
              o22_0 = fma(eb, g0_6, o22_0);
            }
            { const double eb = bi[127];
              o22_0 = fma(eb, g0_12, o22_0);
            }
            { const double eb = bi[128];
              o23_0 = fma(eb, g0_0, o23_0);
            }
            { const double eb = bi[129];
              o23_0 = fma(eb, g0_1, o23_0);
            }
            { const double eb = bi[130];
              o23_0 = fma(eb, g0_4, o23_0);
            }
            { const double eb = bi[131];
              o23_0 = fma(eb, g0_2, o23_0);
            }
            { const double eb = bi[132];
              o23_0 = fma(eb, g0_5, o23_0);
            }
            { const double eb = bi[133];
              o23_0 = fma(eb, g0_11, o23_0);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0);
            o1_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 0);
            o2_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 0);
            o3_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 0);
            o4_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0);
            o5_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 0);
            o6_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 0);
            o7_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 0);
            o8_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0);
            o9_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 0);
            o10_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 0);
            o11_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 0);
            o12_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0);
            o13_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 0);
            o14_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 0);
            o15_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 0);
            o16_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0);
            o17_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 0);
            o18_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 0);
            o19_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 0);
            o20_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0);
            o21_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 0);
            o22_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 0);
            o23_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o1_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o2_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o3_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o4_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o5_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o6_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o7_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o8_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o9_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o10_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o11_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o12_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o13_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o14_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o15_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o16_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o17_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o18_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o19_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o20_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o21_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o22_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o23_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
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
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15 + o16_0 * ptb16 + o17_0 * ptb17 + o18_0 * ptb18 + o19_0 * ptb19 + o20_0 * ptb20 + o21_0 * ptb21 + o22_0 * ptb22 + o23_0 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0 + o3_0 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o4_0 * Aad1_0 + o8_0 * Aad2_0 + o12_0 * Aad3_0 + o16_0 * Aad4_0 + o20_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o1_0 * Abc1_0 + o2_0 * Abc2_0 + o3_0 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o4_0 * Aac1_0 + o8_0 * Aac2_0 + o12_0 * Aac3_0 + o16_0 * Aac4_0 + o20_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o5_0 * Aad1_0 + o9_0 * Aad2_0 + o13_0 * Aad3_0 + o17_0 * Aad4_0 + o21_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o5_0 * Aac1_0 + o9_0 * Aac2_0 + o13_0 * Aac3_0 + o17_0 * Aac4_0 + o21_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o6_0 * Aad1_0 + o10_0 * Aad2_0 + o14_0 * Aad3_0 + o18_0 * Aad4_0 + o22_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o6_0 * Aac1_0 + o10_0 * Aac2_0 + o14_0 * Aac3_0 + o18_0 * Aac4_0 + o22_0 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Aad0_0 + o7_0 * Aad1_0 + o11_0 * Aad2_0 + o15_0 * Aad3_0 + o19_0 * Aad4_0 + o23_0 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Aac0_0 + o7_0 * Aac1_0 + o11_0 * Aac2_0 + o15_0 * Aac3_0 + o19_0 * Aac4_0 + o23_0 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Abd0_0 + o5_0 * Abd1_0 + o6_0 * Abd2_0 + o7_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o5_0 * Abc1_0 + o6_0 * Abc2_0 + o7_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Abd0_0 + o9_0 * Abd1_0 + o10_0 * Abd2_0 + o11_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Abc0_0 + o9_0 * Abc1_0 + o10_0 * Abc2_0 + o11_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0 + o15_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o13_0 * Abc1_0 + o14_0 * Abc2_0 + o15_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_0 * Abd0_0 + o17_0 * Abd1_0 + o18_0 * Abd2_0 + o19_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_0 * Abc0_0 + o17_0 * Abc1_0 + o18_0 * Abc2_0 + o19_0 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_0 * Abd0_0 + o21_0 * Abd1_0 + o22_0 * Abd2_0 + o23_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_0 * Abc0_0 + o21_0 * Abc1_0 + o22_0 * Abc2_0 + o23_0 * Abc3_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Bbd0_0 + o1_0 * Bbd1_0 + o2_0 * Bbd2_0 + o3_0 * Bbd3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Bad0_0 + o4_0 * Bad1_0 + o8_0 * Bad2_0 + o12_0 * Bad3_0 + o16_0 * Bad4_0 + o20_0 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Bbc0_0 + o1_0 * Bbc1_0 + o2_0 * Bbc2_0 + o3_0 * Bbc3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Bac0_0 + o4_0 * Bac1_0 + o8_0 * Bac2_0 + o12_0 * Bac3_0 + o16_0 * Bac4_0 + o20_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Bad0_0 + o5_0 * Bad1_0 + o9_0 * Bad2_0 + o13_0 * Bad3_0 + o17_0 * Bad4_0 + o21_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Bac0_0 + o5_0 * Bac1_0 + o9_0 * Bac2_0 + o13_0 * Bac3_0 + o17_0 * Bac4_0 + o21_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Bad0_0 + o6_0 * Bad1_0 + o10_0 * Bad2_0 + o14_0 * Bad3_0 + o18_0 * Bad4_0 + o22_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Bac0_0 + o6_0 * Bac1_0 + o10_0 * Bac2_0 + o14_0 * Bac3_0 + o18_0 * Bac4_0 + o22_0 * Bac5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Bad0_0 + o7_0 * Bad1_0 + o11_0 * Bad2_0 + o15_0 * Bad3_0 + o19_0 * Bad4_0 + o23_0 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Bac0_0 + o7_0 * Bac1_0 + o11_0 * Bac2_0 + o15_0 * Bac3_0 + o19_0 * Bac4_0 + o23_0 * Bac5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Bbd0_0 + o5_0 * Bbd1_0 + o6_0 * Bbd2_0 + o7_0 * Bbd3_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Bbc0_0 + o5_0 * Bbc1_0 + o6_0 * Bbc2_0 + o7_0 * Bbc3_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Bbd0_0 + o9_0 * Bbd1_0 + o10_0 * Bbd2_0 + o11_0 * Bbd3_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Bbc0_0 + o9_0 * Bbc1_0 + o10_0 * Bbc2_0 + o11_0 * Bbc3_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Bbd0_0 + o13_0 * Bbd1_0 + o14_0 * Bbd2_0 + o15_0 * Bbd3_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Bbc0_0 + o13_0 * Bbc1_0 + o14_0 * Bbc2_0 + o15_0 * Bbc3_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o16_0 * Bbd0_0 + o17_0 * Bbd1_0 + o18_0 * Bbd2_0 + o19_0 * Bbd3_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o16_0 * Bbc0_0 + o17_0 * Bbc1_0 + o18_0 * Bbc2_0 + o19_0 * Bbc3_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o20_0 * Bbd0_0 + o21_0 * Bbd1_0 + o22_0 * Bbd2_0 + o23_0 * Bbd3_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o20_0 * Bbc0_0 + o21_0 * Bbc1_0 + o22_0 * Bbc2_0 + o23_0 * Bbc3_0));
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
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek1_0 = kj[6 * kS];
              const double ek1_1 = -kj[7 * kS];
              g1_0 = fma(ek1_0, b0, g1_0);
              const double r0_0_0_1 = Z * b1;
              g1_1 = fma(ek1_0, r0_0_0_1, g1_1);
              const double r0_0_1_0 = Y * b1;
              g1_2 = fma(ek1_0, r0_0_1_0, g1_2);
              const double r0_1_0_0 = X * b1;
              g1_3 = fma(ek1_0, r0_1_0_0, g1_3);
              g1_0 = fma(ek1_1, r0_1_0_0, g1_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g1_4 = fma(ek1_0, r0_0_0_2, g1_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g1_5 = fma(ek1_0, r0_0_1_1, g1_5);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g1_6 = fma(ek1_0, r0_0_2_0, g1_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g1_7 = fma(ek1_0, r0_1_0_1, g1_7);
              g1_1 = fma(ek1_1, r0_1_0_1, g1_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g1_8 = fma(ek1_0, r0_1_1_0, g1_8);
              g1_2 = fma(ek1_1, r0_1_1_0, g1_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g1_9 = fma(ek1_0, r0_2_0_0, g1_9);
              g1_3 = fma(ek1_1, r0_2_0_0, g1_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g1_10 = fma(ek1_0, r0_0_0_3, g1_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g1_11 = fma(ek1_0, r0_0_1_2, g1_11);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g1_12 = fma(ek1_0, r0_0_2_1, g1_12);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g1_13 = fma(ek1_0, r0_0_3_0, g1_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g1_14 = fma(ek1_0, r0_1_0_2, g1_14);
              g1_4 = fma(ek1_1, r0_1_0_2, g1_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g1_15 = fma(ek1_0, r0_1_1_1, g1_15);
              g1_5 = fma(ek1_1, r0_1_1_1, g1_5);
              const double r0_1_2_0 = X * r1_0_2_0;
              g1_16 = fma(ek1_0, r0_1_2_0, g1_16);
              g1_6 = fma(ek1_1, r0_1_2_0, g1_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g1_17 = fma(ek1_0, r0_2_0_1, g1_17);
              g1_7 = fma(ek1_1, r0_2_0_1, g1_7);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g1_18 = fma(ek1_0, r0_2_1_0, g1_18);
              g1_8 = fma(ek1_1, r0_2_1_0, g1_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g1_19 = fma(ek1_0, r0_3_0_0, g1_19);
              g1_9 = fma(ek1_1, r0_3_0_0, g1_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_1_0_3 = X * r1_0_0_3;
              g1_10 = fma(ek1_1, r0_1_0_3, g1_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_1_1_2 = X * r1_0_1_2;
              g1_11 = fma(ek1_1, r0_1_1_2, g1_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g1_12 = fma(ek1_1, r0_1_2_1, g1_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g1_13 = fma(ek1_1, r0_1_3_0, g1_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g1_14 = fma(ek1_1, r0_2_0_2, g1_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g1_15 = fma(ek1_1, r0_2_1_1, g1_15);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g1_16 = fma(ek1_1, r0_2_2_0, g1_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g1_17 = fma(ek1_1, r0_3_0_1, g1_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g1_18 = fma(ek1_1, r0_3_1_0, g1_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g1_19 = fma(ek1_1, r0_4_0_0, g1_19);
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
              o1_1 = fma(eb, g1_0, o1_1);
            }
            { const double eb = bi[9];
              o1_1 = fma(eb, g1_3, o1_1);
            }
            { const double eb = bi[10];
              o1_1 = fma(eb, g1_9, o1_1);
            }
            { const double eb = bi[11];
              o1_1 = fma(eb, g1_19, o1_1);
            }
            { const double eb = bi[12];
              o2_1 = fma(eb, g1_0, o2_1);
            }
            { const double eb = bi[13];
              o2_1 = fma(eb, g1_2, o2_1);
            }
            { const double eb = bi[14];
              o2_1 = fma(eb, g1_3, o2_1);
            }
            { const double eb = bi[15];
              o2_1 = fma(eb, g1_8, o2_1);
            }
            { const double eb = bi[16];
              o2_1 = fma(eb, g1_9, o2_1);
            }
            { const double eb = bi[17];
              o2_1 = fma(eb, g1_18, o2_1);
            }
            { const double eb = bi[18];
              o3_1 = fma(eb, g1_0, o3_1);
            }
            { const double eb = bi[19];
              o3_1 = fma(eb, g1_1, o3_1);
            }
            { const double eb = bi[20];
              o3_1 = fma(eb, g1_3, o3_1);
            }
            { const double eb = bi[21];
              o3_1 = fma(eb, g1_7, o3_1);
            }
            { const double eb = bi[22];
              o3_1 = fma(eb, g1_9, o3_1);
            }
            { const double eb = bi[23];
              o3_1 = fma(eb, g1_17, o3_1);
            }
            { const double eb = bi[24];
              o4_1 = fma(eb, g1_0, o4_1);
            }
            { const double eb = bi[25];
              o4_1 = fma(eb, g1_2, o4_1);
            }
            { const double eb = bi[26];
              o4_1 = fma(eb, g1_6, o4_1);
            }
            { const double eb = bi[27];
              o5_1 = fma(eb, g1_0, o5_1);
            }
            { const double eb = bi[28];
              o5_1 = fma(eb, g1_2, o5_1);
            }
            { const double eb = bi[29];
              o5_1 = fma(eb, g1_6, o5_1);
            }
            { const double eb = bi[30];
              o5_1 = fma(eb, g1_3, o5_1);
            }
            { const double eb = bi[31];
              o5_1 = fma(eb, g1_8, o5_1);
            }
            { const double eb = bi[32];
              o5_1 = fma(eb, g1_16, o5_1);
            }
            { const double eb = bi[33];
              o6_1 = fma(eb, g1_0, o6_1);
            }
            { const double eb = bi[34];
              o6_1 = fma(eb, g1_2, o6_1);
            }
            { const double eb = bi[35];
              o6_1 = fma(eb, g1_6, o6_1);
            }
            { const double eb = bi[36];
              o6_1 = fma(eb, g1_13, o6_1);
            }
            { const double eb = bi[37];
              o7_1 = fma(eb, g1_0, o7_1);
            }
            { const double eb = bi[38];
              o7_1 = fma(eb, g1_1, o7_1);
            }
            { const double eb = bi[39];
              o7_1 = fma(eb, g1_2, o7_1);
            }
            { const double eb = bi[40];
              o7_1 = fma(eb, g1_5, o7_1);
            }
            { const double eb = bi[41];
              o7_1 = fma(eb, g1_6, o7_1);
            }
            { const double eb = bi[42];
              o7_1 = fma(eb, g1_12, o7_1);
            }
            { const double eb = bi[43];
              o8_1 = fma(eb, g1_0, o8_1);
            }
            { const double eb = bi[44];
              o8_1 = fma(eb, g1_1, o8_1);
            }
            { const double eb = bi[45];
              o8_1 = fma(eb, g1_4, o8_1);
            }
            { const double eb = bi[46];
              o9_1 = fma(eb, g1_0, o9_1);
            }
            { const double eb = bi[47];
              o9_1 = fma(eb, g1_1, o9_1);
            }
            { const double eb = bi[48];
              o9_1 = fma(eb, g1_4, o9_1);
            }
            { const double eb = bi[49];
              o9_1 = fma(eb, g1_3, o9_1);
            }
            { const double eb = bi[50];
              o9_1 = fma(eb, g1_7, o9_1);
            }
            { const double eb = bi[51];
              o9_1 = fma(eb, g1_14, o9_1);
            }
            { const double eb = bi[52];
              o10_1 = fma(eb, g1_0, o10_1);
            }
            { const double eb = bi[53];
              o10_1 = fma(eb, g1_1, o10_1);
            }
            { const double eb = bi[54];
              o10_1 = fma(eb, g1_4, o10_1);
            }
            { const double eb = bi[55];
              o10_1 = fma(eb, g1_2, o10_1);
            }
            { const double eb = bi[56];
              o10_1 = fma(eb, g1_5, o10_1);
            }
            { const double eb = bi[57];
              o10_1 = fma(eb, g1_11, o10_1);
            }
            { const double eb = bi[58];
              o11_1 = fma(eb, g1_0, o11_1);
            }
            { const double eb = bi[59];
              o11_1 = fma(eb, g1_1, o11_1);
            }
            { const double eb = bi[60];
              o11_1 = fma(eb, g1_4, o11_1);
            }
            { const double eb = bi[61];
              o11_1 = fma(eb, g1_10, o11_1);
            }
            { const double eb = bi[62];
              o12_1 = fma(eb, g1_0, o12_1);
            }
            { const double eb = bi[63];
              o12_1 = fma(eb, g1_2, o12_1);
            }
            { const double eb = bi[64];
              o12_1 = fma(eb, g1_3, o12_1);
            }
            { const double eb = bi[65];
              o12_1 = fma(eb, g1_8, o12_1);
            }
            { const double eb = bi[66];
              o13_1 = fma(eb, g1_0, o13_1);
            }
            { const double eb = bi[67];
              o13_1 = fma(eb, g1_2, o13_1);
            }
            { const double eb = bi[68];
              o13_1 = fma(eb, g1_3, o13_1);
            }
            { const double eb = bi[69];
              o13_1 = fma(eb, g1_8, o13_1);
            }
            { const double eb = bi[70];
              o13_1 = fma(eb, g1_9, o13_1);
            }
            { const double eb = bi[71];
              o13_1 = fma(eb, g1_18, o13_1);
            }
            { const double eb = bi[72];
              o14_1 = fma(eb, g1_0, o14_1);
            }
            { const double eb = bi[73];
              o14_1 = fma(eb, g1_2, o14_1);
            }
            { const double eb = bi[74];
              o14_1 = fma(eb, g1_6, o14_1);
            }
            { const double eb = bi[75];
              o14_1 = fma(eb, g1_3, o14_1);
            }
            { const double eb = bi[76];
              o14_1 = fma(eb, g1_8, o14_1);
            }
            { const double eb = bi[77];
              o14_1 = fma(eb, g1_16, o14_1);
            }
            { const double eb = bi[78];
              o15_1 = fma(eb, g1_0, o15_1);
            }
            { const double eb = bi[79];
              o15_1 = fma(eb, g1_1, o15_1);
            }
            { const double eb = bi[80];
              o15_1 = fma(eb, g1_2, o15_1);
            }
            { const double eb = bi[81];
              o15_1 = fma(eb, g1_5, o15_1);
            }
            { const double eb = bi[82];
              o15_1 = fma(eb, g1_3, o15_1);
            }
            { const double eb = bi[83];
              o15_1 = fma(eb, g1_7, o15_1);
            }
            { const double eb = bi[84];
              o15_1 = fma(eb, g1_8, o15_1);
            }
            { const double eb = bi[85];
              o15_1 = fma(eb, g1_15, o15_1);
            }
            { const double eb = bi[86];
              o16_1 = fma(eb, g1_0, o16_1);
            }
            { const double eb = bi[87];
              o16_1 = fma(eb, g1_1, o16_1);
            }
            { const double eb = bi[88];
              o16_1 = fma(eb, g1_3, o16_1);
            }
            { const double eb = bi[89];
              o16_1 = fma(eb, g1_7, o16_1);
            }
            { const double eb = bi[90];
              o17_1 = fma(eb, g1_0, o17_1);
            }
            { const double eb = bi[91];
              o17_1 = fma(eb, g1_1, o17_1);
            }
            { const double eb = bi[92];
              o17_1 = fma(eb, g1_3, o17_1);
            }
            { const double eb = bi[93];
              o17_1 = fma(eb, g1_7, o17_1);
            }
            { const double eb = bi[94];
              o17_1 = fma(eb, g1_9, o17_1);
            }
            { const double eb = bi[95];
              o17_1 = fma(eb, g1_17, o17_1);
            }
            { const double eb = bi[96];
              o18_1 = fma(eb, g1_0, o18_1);
            }
            { const double eb = bi[97];
              o18_1 = fma(eb, g1_1, o18_1);
            }
            { const double eb = bi[98];
              o18_1 = fma(eb, g1_2, o18_1);
            }
            { const double eb = bi[99];
              o18_1 = fma(eb, g1_5, o18_1);
            }
            { const double eb = bi[100];
              o18_1 = fma(eb, g1_3, o18_1);
            }
            { const double eb = bi[101];
              o18_1 = fma(eb, g1_7, o18_1);
            }
            { const double eb = bi[102];
              o18_1 = fma(eb, g1_8, o18_1);
            }
            { const double eb = bi[103];
              o18_1 = fma(eb, g1_15, o18_1);
            }
            { const double eb = bi[104];
              o19_1 = fma(eb, g1_0, o19_1);
            }
            { const double eb = bi[105];
              o19_1 = fma(eb, g1_1, o19_1);
            }
            { const double eb = bi[106];
              o19_1 = fma(eb, g1_4, o19_1);
            }
            { const double eb = bi[107];
              o19_1 = fma(eb, g1_3, o19_1);
            }
            { const double eb = bi[108];
              o19_1 = fma(eb, g1_7, o19_1);
            }
            { const double eb = bi[109];
              o19_1 = fma(eb, g1_14, o19_1);
            }
            { const double eb = bi[110];
              o20_1 = fma(eb, g1_0, o20_1);
            }
            { const double eb = bi[111];
              o20_1 = fma(eb, g1_1, o20_1);
            }
            { const double eb = bi[112];
              o20_1 = fma(eb, g1_2, o20_1);
            }
            { const double eb = bi[113];
              o20_1 = fma(eb, g1_5, o20_1);
            }
            { const double eb = bi[114];
              o21_1 = fma(eb, g1_0, o21_1);
            }
            { const double eb = bi[115];
              o21_1 = fma(eb, g1_1, o21_1);
            }
            { const double eb = bi[116];
              o21_1 = fma(eb, g1_2, o21_1);
            }
            { const double eb = bi[117];
              o21_1 = fma(eb, g1_5, o21_1);
            }
            { const double eb = bi[118];
              o21_1 = fma(eb, g1_3, o21_1);
            }
            { const double eb = bi[119];
              o21_1 = fma(eb, g1_7, o21_1);
            }
            { const double eb = bi[120];
              o21_1 = fma(eb, g1_8, o21_1);
            }
            { const double eb = bi[121];
              o21_1 = fma(eb, g1_15, o21_1);
            }
            { const double eb = bi[122];
              o22_1 = fma(eb, g1_0, o22_1);
            }
            { const double eb = bi[123];
              o22_1 = fma(eb, g1_1, o22_1);
            }
            { const double eb = bi[124];
              o22_1 = fma(eb, g1_2, o22_1);
            }
            { const double eb = bi[125];
              o22_1 = fma(eb, g1_5, o22_1);
            }
            { const double eb = bi[126];
              o22_1 = fma(eb, g1_6, o22_1);
            }
            { const double eb = bi[127];
              o22_1 = fma(eb, g1_12, o22_1);
            }
            { const double eb = bi[128];
              o23_1 = fma(eb, g1_0, o23_1);
            }
            { const double eb = bi[129];
              o23_1 = fma(eb, g1_1, o23_1);
            }
            { const double eb = bi[130];
              o23_1 = fma(eb, g1_4, o23_1);
            }
            { const double eb = bi[131];
              o23_1 = fma(eb, g1_2, o23_1);
            }
            { const double eb = bi[132];
              o23_1 = fma(eb, g1_5, o23_1);
            }
            { const double eb = bi[133];
              o23_1 = fma(eb, g1_11, o23_1);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 1);
            o1_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 1);
            o2_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 1);
            o3_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 1);
            o4_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 1);
            o5_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 1);
            o6_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 1);
            o7_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 1);
            o8_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 1);
            o9_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 1);
            o10_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 1);
            o11_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 1);
            o12_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 1);
            o13_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 1);
            o14_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 1);
            o15_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 1);
            o16_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 1);
            o17_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 1);
            o18_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 1);
            o19_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 1);
            o20_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 1);
            o21_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 1);
            o22_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 1);
            o23_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 1);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o1_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o2_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o3_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o4_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o5_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o6_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o7_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o8_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o9_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o10_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o11_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o12_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o13_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o14_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o15_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o16_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o17_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o18_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o19_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o20_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o21_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o22_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 1)));
            e = fmax(e, fabs(o23_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 1)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
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
            const double Bbd0_1 = PB[(fQ + 0) * N + fJ + 1];
            const double Bbd1_1 = PB[(fQ + 1) * N + fJ + 1];
            const double Bbd2_1 = PB[(fQ + 2) * N + fJ + 1];
            const double Bbd3_1 = PB[(fQ + 3) * N + fJ + 1];
            const double Bad0_1 = PB[(fP + 0) * N + fJ + 1];
            const double Bad1_1 = PB[(fP + 1) * N + fJ + 1];
            const double Bad2_1 = PB[(fP + 2) * N + fJ + 1];
            const double Bad3_1 = PB[(fP + 3) * N + fJ + 1];
            const double Bad4_1 = PB[(fP + 4) * N + fJ + 1];
            const double Bad5_1 = PB[(fP + 5) * N + fJ + 1];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc1_0 = PB[(fQ + 1) * N + fI + 0];
            const double Bbc2_0 = PB[(fQ + 2) * N + fI + 0];
            const double Bbc3_0 = PB[(fQ + 3) * N + fI + 0];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            const double Bac1_0 = PB[(fP + 1) * N + fI + 0];
            const double Bac2_0 = PB[(fP + 2) * N + fI + 0];
            const double Bac3_0 = PB[(fP + 3) * N + fI + 0];
            const double Bac4_0 = PB[(fP + 4) * N + fI + 0];
            const double Bac5_0 = PB[(fP + 5) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 1, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17 + o18_1 * ptb18 + o19_1 * ptb19 + o20_1 * ptb20 + o21_1 * ptb21 + o22_1 * ptb22 + o23_1 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_1 * Abd0_1 + o1_1 * Abd1_1 + o2_1 * Abd2_1 + o3_1 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_1 * Aad0_1 + o4_1 * Aad1_1 + o8_1 * Aad2_1 + o12_1 * Aad3_1 + o16_1 * Aad4_1 + o20_1 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_1 * Abc0_0 + o1_1 * Abc1_0 + o2_1 * Abc2_0 + o3_1 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_1 * Aac0_0 + o4_1 * Aac1_0 + o8_1 * Aac2_0 + o12_1 * Aac3_0 + o16_1 * Aac4_0 + o20_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_1 * Aad0_1 + o5_1 * Aad1_1 + o9_1 * Aad2_1 + o13_1 * Aad3_1 + o17_1 * Aad4_1 + o21_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_1 * Aac0_0 + o5_1 * Aac1_0 + o9_1 * Aac2_0 + o13_1 * Aac3_0 + o17_1 * Aac4_0 + o21_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_1 * Aad0_1 + o6_1 * Aad1_1 + o10_1 * Aad2_1 + o14_1 * Aad3_1 + o18_1 * Aad4_1 + o22_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_1 * Aac0_0 + o6_1 * Aac1_0 + o10_1 * Aac2_0 + o14_1 * Aac3_0 + o18_1 * Aac4_0 + o22_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_1 * Aad0_1 + o7_1 * Aad1_1 + o11_1 * Aad2_1 + o15_1 * Aad3_1 + o19_1 * Aad4_1 + o23_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_1 * Aac0_0 + o7_1 * Aac1_0 + o11_1 * Aac2_0 + o15_1 * Aac3_0 + o19_1 * Aac4_0 + o23_1 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_1 * Abd0_1 + o5_1 * Abd1_1 + o6_1 * Abd2_1 + o7_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_1 * Abc0_0 + o5_1 * Abc1_0 + o6_1 * Abc2_0 + o7_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_1 * Abd0_1 + o9_1 * Abd1_1 + o10_1 * Abd2_1 + o11_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_1 * Abc0_0 + o9_1 * Abc1_0 + o10_1 * Abc2_0 + o11_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_1 * Abd0_1 + o13_1 * Abd1_1 + o14_1 * Abd2_1 + o15_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_1 * Abc0_0 + o13_1 * Abc1_0 + o14_1 * Abc2_0 + o15_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_1 * Abd0_1 + o17_1 * Abd1_1 + o18_1 * Abd2_1 + o19_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_1 * Abc0_0 + o17_1 * Abc1_0 + o18_1 * Abc2_0 + o19_1 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_1 * Abd0_1 + o21_1 * Abd1_1 + o22_1 * Abd2_1 + o23_1 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_1 * Abc0_0 + o21_1 * Abc1_0 + o22_1 * Abc2_0 + o23_1 * Abc3_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_1 * Bbd0_1 + o1_1 * Bbd1_1 + o2_1 * Bbd2_1 + o3_1 * Bbd3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_1 * Bad0_1 + o4_1 * Bad1_1 + o8_1 * Bad2_1 + o12_1 * Bad3_1 + o16_1 * Bad4_1 + o20_1 * Bad5_1));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 1, deg * (o0_1 * Bbc0_0 + o1_1 * Bbc1_0 + o2_1 * Bbc2_0 + o3_1 * Bbc3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 1, deg * (o0_1 * Bac0_0 + o4_1 * Bac1_0 + o8_1 * Bac2_0 + o12_1 * Bac3_0 + o16_1 * Bac4_0 + o20_1 * Bac5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_1 * Bad0_1 + o5_1 * Bad1_1 + o9_1 * Bad2_1 + o13_1 * Bad3_1 + o17_1 * Bad4_1 + o21_1 * Bad5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 1, deg * (o1_1 * Bac0_0 + o5_1 * Bac1_0 + o9_1 * Bac2_0 + o13_1 * Bac3_0 + o17_1 * Bac4_0 + o21_1 * Bac5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_1 * Bad0_1 + o6_1 * Bad1_1 + o10_1 * Bad2_1 + o14_1 * Bad3_1 + o18_1 * Bad4_1 + o22_1 * Bad5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 1, deg * (o2_1 * Bac0_0 + o6_1 * Bac1_0 + o10_1 * Bac2_0 + o14_1 * Bac3_0 + o18_1 * Bac4_0 + o22_1 * Bac5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 0, deg * (o3_1 * Bad0_1 + o7_1 * Bad1_1 + o11_1 * Bad2_1 + o15_1 * Bad3_1 + o19_1 * Bad4_1 + o23_1 * Bad5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 1, deg * (o3_1 * Bac0_0 + o7_1 * Bac1_0 + o11_1 * Bac2_0 + o15_1 * Bac3_0 + o19_1 * Bac4_0 + o23_1 * Bac5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o4_1 * Bbd0_1 + o5_1 * Bbd1_1 + o6_1 * Bbd2_1 + o7_1 * Bbd3_1));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 1, deg * (o4_1 * Bbc0_0 + o5_1 * Bbc1_0 + o6_1 * Bbc2_0 + o7_1 * Bbc3_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o8_1 * Bbd0_1 + o9_1 * Bbd1_1 + o10_1 * Bbd2_1 + o11_1 * Bbd3_1));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 1, deg * (o8_1 * Bbc0_0 + o9_1 * Bbc1_0 + o10_1 * Bbc2_0 + o11_1 * Bbc3_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o12_1 * Bbd0_1 + o13_1 * Bbd1_1 + o14_1 * Bbd2_1 + o15_1 * Bbd3_1));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 1, deg * (o12_1 * Bbc0_0 + o13_1 * Bbc1_0 + o14_1 * Bbc2_0 + o15_1 * Bbc3_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o16_1 * Bbd0_1 + o17_1 * Bbd1_1 + o18_1 * Bbd2_1 + o19_1 * Bbd3_1));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 1, deg * (o16_1 * Bbc0_0 + o17_1 * Bbc1_0 + o18_1 * Bbc2_0 + o19_1 * Bbc3_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o20_1 * Bbd0_1 + o21_1 * Bbd1_1 + o22_1 * Bbd2_1 + o23_1 * Bbd3_1));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 1, deg * (o20_1 * Bbc0_0 + o21_1 * Bbc1_0 + o22_1 * Bbc2_0 + o23_1 * Bbc3_0));
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek2_0 = kj[8 * kS];
              const double ek2_1 = -kj[9 * kS];
              g2_0 = fma(ek2_0, b0, g2_0);
              const double r0_0_0_1 = Z * b1;
              g2_1 = fma(ek2_0, r0_0_0_1, g2_1);
              const double r0_0_1_0 = Y * b1;
              g2_2 = fma(ek2_0, r0_0_1_0, g2_2);
              g2_0 = fma(ek2_1, r0_0_1_0, g2_0);
              const double r0_1_0_0 = X * b1;
              g2_3 = fma(ek2_0, r0_1_0_0, g2_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g2_4 = fma(ek2_0, r0_0_0_2, g2_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g2_5 = fma(ek2_0, r0_0_1_1, g2_5);
              g2_1 = fma(ek2_1, r0_0_1_1, g2_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g2_6 = fma(ek2_0, r0_0_2_0, g2_6);
              g2_2 = fma(ek2_1, r0_0_2_0, g2_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g2_7 = fma(ek2_0, r0_1_0_1, g2_7);
              const double r0_1_1_0 = X * r1_0_1_0;
              g2_8 = fma(ek2_0, r0_1_1_0, g2_8);
              g2_3 = fma(ek2_1, r0_1_1_0, g2_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g2_9 = fma(ek2_0, r0_2_0_0, g2_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g2_10 = fma(ek2_0, r0_0_0_3, g2_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g2_11 = fma(ek2_0, r0_0_1_2, g2_11);
              g2_4 = fma(ek2_1, r0_0_1_2, g2_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g2_12 = fma(ek2_0, r0_0_2_1, g2_12);
              g2_5 = fma(ek2_1, r0_0_2_1, g2_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g2_13 = fma(ek2_0, r0_0_3_0, g2_13);
              g2_6 = fma(ek2_1, r0_0_3_0, g2_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g2_14 = fma(ek2_0, r0_1_0_2, g2_14);
              const double r0_1_1_1 = X * r1_0_1_1;
              g2_15 = fma(ek2_0, r0_1_1_1, g2_15);
              g2_7 = fma(ek2_1, r0_1_1_1, g2_7);
              const double r0_1_2_0 = X * r1_0_2_0;
              g2_16 = fma(ek2_0, r0_1_2_0, g2_16);
              g2_8 = fma(ek2_1, r0_1_2_0, g2_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g2_17 = fma(ek2_0, r0_2_0_1, g2_17);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g2_18 = fma(ek2_0, r0_2_1_0, g2_18);
              g2_9 = fma(ek2_1, r0_2_1_0, g2_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g2_19 = fma(ek2_0, r0_3_0_0, g2_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g2_10 = fma(ek2_1, r0_0_1_3, g2_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g2_11 = fma(ek2_1, r0_0_2_2, g2_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g2_12 = fma(ek2_1, r0_0_3_1, g2_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g2_13 = fma(ek2_1, r0_0_4_0, g2_13);
              const double r0_1_1_2 = X * r1_0_1_2;
              g2_14 = fma(ek2_1, r0_1_1_2, g2_14);
              const double r0_1_2_1 = X * r1_0_2_1;
              g2_15 = fma(ek2_1, r0_1_2_1, g2_15);
              const double r0_1_3_0 = X * r1_0_3_0;
              g2_16 = fma(ek2_1, r0_1_3_0, g2_16);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g2_17 = fma(ek2_1, r0_2_1_1, g2_17);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g2_18 = fma(ek2_1, r0_2_2_0, g2_18);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g2_19 = fma(ek2_1, r0_3_1_0, g2_19);
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
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 2);
            o1_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 2);
            o2_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 2);
            o3_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 2);
            o4_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 2);
            o5_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 2);
            o6_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 2);
            o7_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 2);
            o8_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 2);
            o9_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 2);
            o10_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 2);
            o11_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 2);
            o12_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 2);
            o13_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 2);
            o14_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 2);
            o15_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 2);
            o16_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 2);
            o17_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 2);
            o18_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 2);
            o19_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 2);
            o20_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 2);
            o21_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 2);
            o22_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 2);
            o23_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 2);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o1_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o2_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o3_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o4_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o5_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o6_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o7_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o8_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o9_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o10_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o11_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o12_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o13_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o14_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o15_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o16_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o17_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o18_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o19_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o20_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o21_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o22_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 2)));
            e = fmax(e, fabs(o23_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 2)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 0) * N + fJ + 2];
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
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
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
            const double Bbd0_2 = PB[(fQ + 0) * N + fJ + 2];
            const double Bbd1_2 = PB[(fQ + 1) * N + fJ + 2];
            const double Bbd2_2 = PB[(fQ + 2) * N + fJ + 2];
            const double Bbd3_2 = PB[(fQ + 3) * N + fJ + 2];
            const double Bad0_2 = PB[(fP + 0) * N + fJ + 2];
            const double Bad1_2 = PB[(fP + 1) * N + fJ + 2];
            const double Bad2_2 = PB[(fP + 2) * N + fJ + 2];
            const double Bad3_2 = PB[(fP + 3) * N + fJ + 2];
            const double Bad4_2 = PB[(fP + 4) * N + fJ + 2];
            const double Bad5_2 = PB[(fP + 5) * N + fJ + 2];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc1_0 = PB[(fQ + 1) * N + fI + 0];
            const double Bbc2_0 = PB[(fQ + 2) * N + fI + 0];
            const double Bbc3_0 = PB[(fQ + 3) * N + fI + 0];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            const double Bac1_0 = PB[(fP + 1) * N + fI + 0];
            const double Bac2_0 = PB[(fP + 2) * N + fI + 0];
            const double Bac3_0 = PB[(fP + 3) * N + fI + 0];
            const double Bac4_0 = PB[(fP + 4) * N + fI + 0];
            const double Bac5_0 = PB[(fP + 5) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 2, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17 + o18_2 * ptb18 + o19_2 * ptb19 + o20_2 * ptb20 + o21_2 * ptb21 + o22_2 * ptb22 + o23_2 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_2 * Abd0_2 + o1_2 * Abd1_2 + o2_2 * Abd2_2 + o3_2 * Abd3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_2 * Aad0_2 + o4_2 * Aad1_2 + o8_2 * Aad2_2 + o12_2 * Aad3_2 + o16_2 * Aad4_2 + o20_2 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_2 * Abc0_0 + o1_2 * Abc1_0 + o2_2 * Abc2_0 + o3_2 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_2 * Aac0_0 + o4_2 * Aac1_0 + o8_2 * Aac2_0 + o12_2 * Aac3_0 + o16_2 * Aac4_0 + o20_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_2 * Aad0_2 + o5_2 * Aad1_2 + o9_2 * Aad2_2 + o13_2 * Aad3_2 + o17_2 * Aad4_2 + o21_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_2 * Aac0_0 + o5_2 * Aac1_0 + o9_2 * Aac2_0 + o13_2 * Aac3_0 + o17_2 * Aac4_0 + o21_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_2 * Aad0_2 + o6_2 * Aad1_2 + o10_2 * Aad2_2 + o14_2 * Aad3_2 + o18_2 * Aad4_2 + o22_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_2 * Aac0_0 + o6_2 * Aac1_0 + o10_2 * Aac2_0 + o14_2 * Aac3_0 + o18_2 * Aac4_0 + o22_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_2 * Aad0_2 + o7_2 * Aad1_2 + o11_2 * Aad2_2 + o15_2 * Aad3_2 + o19_2 * Aad4_2 + o23_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_2 * Aac0_0 + o7_2 * Aac1_0 + o11_2 * Aac2_0 + o15_2 * Aac3_0 + o19_2 * Aac4_0 + o23_2 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_2 * Abd0_2 + o5_2 * Abd1_2 + o6_2 * Abd2_2 + o7_2 * Abd3_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_2 * Abc0_0 + o5_2 * Abc1_0 + o6_2 * Abc2_0 + o7_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_2 * Abd0_2 + o9_2 * Abd1_2 + o10_2 * Abd2_2 + o11_2 * Abd3_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_2 * Abc0_0 + o9_2 * Abc1_0 + o10_2 * Abc2_0 + o11_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_2 * Abd0_2 + o13_2 * Abd1_2 + o14_2 * Abd2_2 + o15_2 * Abd3_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_2 * Abc0_0 + o13_2 * Abc1_0 + o14_2 * Abc2_0 + o15_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_2 * Abd0_2 + o17_2 * Abd1_2 + o18_2 * Abd2_2 + o19_2 * Abd3_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_2 * Abc0_0 + o17_2 * Abc1_0 + o18_2 * Abc2_0 + o19_2 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_2 * Abd0_2 + o21_2 * Abd1_2 + o22_2 * Abd2_2 + o23_2 * Abd3_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_2 * Abc0_0 + o21_2 * Abc1_0 + o22_2 * Abc2_0 + o23_2 * Abc3_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_2 * Bbd0_2 + o1_2 * Bbd1_2 + o2_2 * Bbd2_2 + o3_2 * Bbd3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_2 * Bad0_2 + o4_2 * Bad1_2 + o8_2 * Bad2_2 + o12_2 * Bad3_2 + o16_2 * Bad4_2 + o20_2 * Bad5_2));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 2, deg * (o0_2 * Bbc0_0 + o1_2 * Bbc1_0 + o2_2 * Bbc2_0 + o3_2 * Bbc3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 2, deg * (o0_2 * Bac0_0 + o4_2 * Bac1_0 + o8_2 * Bac2_0 + o12_2 * Bac3_0 + o16_2 * Bac4_0 + o20_2 * Bac5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_2 * Bad0_2 + o5_2 * Bad1_2 + o9_2 * Bad2_2 + o13_2 * Bad3_2 + o17_2 * Bad4_2 + o21_2 * Bad5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 2, deg * (o1_2 * Bac0_0 + o5_2 * Bac1_0 + o9_2 * Bac2_0 + o13_2 * Bac3_0 + o17_2 * Bac4_0 + o21_2 * Bac5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_2 * Bad0_2 + o6_2 * Bad1_2 + o10_2 * Bad2_2 + o14_2 * Bad3_2 + o18_2 * Bad4_2 + o22_2 * Bad5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 2, deg * (o2_2 * Bac0_0 + o6_2 * Bac1_0 + o10_2 * Bac2_0 + o14_2 * Bac3_0 + o18_2 * Bac4_0 + o22_2 * Bac5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 0, deg * (o3_2 * Bad0_2 + o7_2 * Bad1_2 + o11_2 * Bad2_2 + o15_2 * Bad3_2 + o19_2 * Bad4_2 + o23_2 * Bad5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 2, deg * (o3_2 * Bac0_0 + o7_2 * Bac1_0 + o11_2 * Bac2_0 + o15_2 * Bac3_0 + o19_2 * Bac4_0 + o23_2 * Bac5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o4_2 * Bbd0_2 + o5_2 * Bbd1_2 + o6_2 * Bbd2_2 + o7_2 * Bbd3_2));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 2, deg * (o4_2 * Bbc0_0 + o5_2 * Bbc1_0 + o6_2 * Bbc2_0 + o7_2 * Bbc3_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o8_2 * Bbd0_2 + o9_2 * Bbd1_2 + o10_2 * Bbd2_2 + o11_2 * Bbd3_2));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 2, deg * (o8_2 * Bbc0_0 + o9_2 * Bbc1_0 + o10_2 * Bbc2_0 + o11_2 * Bbc3_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o12_2 * Bbd0_2 + o13_2 * Bbd1_2 + o14_2 * Bbd2_2 + o15_2 * Bbd3_2));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 2, deg * (o12_2 * Bbc0_0 + o13_2 * Bbc1_0 + o14_2 * Bbc2_0 + o15_2 * Bbc3_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o16_2 * Bbd0_2 + o17_2 * Bbd1_2 + o18_2 * Bbd2_2 + o19_2 * Bbd3_2));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 2, deg * (o16_2 * Bbc0_0 + o17_2 * Bbc1_0 + o18_2 * Bbc2_0 + o19_2 * Bbc3_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o20_2 * Bbd0_2 + o21_2 * Bbd1_2 + o22_2 * Bbd2_2 + o23_2 * Bbd3_2));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 2, deg * (o20_2 * Bbc0_0 + o21_2 * Bbc1_0 + o22_2 * Bbc2_0 + o23_2 * Bbc3_0));
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
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek3_0 = kj[10 * kS];
              const double ek3_1 = -kj[11 * kS];
              g3_0 = fma(ek3_0, b0, g3_0);
              const double r0_0_0_1 = Z * b1;
              g3_1 = fma(ek3_0, r0_0_0_1, g3_1);
              g3_0 = fma(ek3_1, r0_0_0_1, g3_0);
              const double r0_0_1_0 = Y * b1;
              g3_2 = fma(ek3_0, r0_0_1_0, g3_2);
              const double r0_1_0_0 = X * b1;
              g3_3 = fma(ek3_0, r0_1_0_0, g3_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g3_4 = fma(ek3_0, r0_0_0_2, g3_4);
              g3_1 = fma(ek3_1, r0_0_0_2, g3_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g3_5 = fma(ek3_0, r0_0_1_1, g3_5);
              g3_2 = fma(ek3_1, r0_0_1_1, g3_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g3_6 = fma(ek3_0, r0_0_2_0, g3_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g3_7 = fma(ek3_0, r0_1_0_1, g3_7);
              g3_3 = fma(ek3_1, r0_1_0_1, g3_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g3_8 = fma(ek3_0, r0_1_1_0, g3_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g3_9 = fma(ek3_0, r0_2_0_0, g3_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g3_10 = fma(ek3_0, r0_0_0_3, g3_10);
              g3_4 = fma(ek3_1, r0_0_0_3, g3_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g3_11 = fma(ek3_0, r0_0_1_2, g3_11);
              g3_5 = fma(ek3_1, r0_0_1_2, g3_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g3_12 = fma(ek3_0, r0_0_2_1, g3_12);
              g3_6 = fma(ek3_1, r0_0_2_1, g3_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g3_13 = fma(ek3_0, r0_0_3_0, g3_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g3_14 = fma(ek3_0, r0_1_0_2, g3_14);
              g3_7 = fma(ek3_1, r0_1_0_2, g3_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g3_15 = fma(ek3_0, r0_1_1_1, g3_15);
              g3_8 = fma(ek3_1, r0_1_1_1, g3_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g3_16 = fma(ek3_0, r0_1_2_0, g3_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g3_17 = fma(ek3_0, r0_2_0_1, g3_17);
              g3_9 = fma(ek3_1, r0_2_0_1, g3_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g3_18 = fma(ek3_0, r0_2_1_0, g3_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g3_19 = fma(ek3_0, r0_3_0_0, g3_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g3_10 = fma(ek3_1, r0_0_0_4, g3_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g3_11 = fma(ek3_1, r0_0_1_3, g3_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g3_12 = fma(ek3_1, r0_0_2_2, g3_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g3_13 = fma(ek3_1, r0_0_3_1, g3_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g3_14 = fma(ek3_1, r0_1_0_3, g3_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g3_15 = fma(ek3_1, r0_1_1_2, g3_15);
              const double r0_1_2_1 = X * r1_0_2_1;
              g3_16 = fma(ek3_1, r0_1_2_1, g3_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g3_17 = fma(ek3_1, r0_2_0_2, g3_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g3_18 = fma(ek3_1, r0_2_1_1, g3_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g3_19 = fma(ek3_1, r0_3_0_1, g3_19);
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
              o1_3 = fma(eb, g3_0, o1_3);
            }
            { const double eb = bi[9];
              o1_3 = fma(eb, g3_3, o1_3);
            }
            { const double eb = bi[10];
              o1_3 = fma(eb, g3_9, o1_3);
            }
            { const double eb = bi[11];
              o1_3 = fma(eb, g3_19, o1_3);
            }
            { const double eb = bi[12];
              o2_3 = fma(eb, g3_0, o2_3);
            }
            { const double eb = bi[13];
              o2_3 = fma(eb, g3_2, o2_3);
            }
            { const double eb = bi[14];
              o2_3 = fma(eb, g3_3, o2_3);
            }
            { const double eb = bi[15];
              o2_3 = fma(eb, g3_8, o2_3);
            }
            { const double eb = bi[16];
              o2_3 = fma(eb, g3_9, o2_3);
            }
            { const double eb = bi[17];
              o2_3 = fma(eb, g3_18, o2_3);
            }
            { const double eb = bi[18];
              o3_3 = fma(eb, g3_0, o3_3);
            }
            { const double eb = bi[19];
              o3_3 = fma(eb, g3_1, o3_3);
            }
            { const double eb = bi[20];
              o3_3 = fma(eb, g3_3, o3_3);
            }
            { const double eb = bi[21];
              o3_3 = fma(eb, g3_7, o3_3);
            }
            { const double eb = bi[22];
              o3_3 = fma(eb, g3_9, o3_3);
            }
            { const double eb = bi[23];
              o3_3 = fma(eb, g3_17, o3_3);
            }
            { const double eb = bi[24];
              o4_3 = fma(eb, g3_0, o4_3);
            }
            { const double eb = bi[25];
              o4_3 = fma(eb, g3_2, o4_3);
            }
            { const double eb = bi[26];
              o4_3 = fma(eb, g3_6, o4_3);
            }
            { const double eb = bi[27];
              o5_3 = fma(eb, g3_0, o5_3);
            }
            { const double eb = bi[28];
              o5_3 = fma(eb, g3_2, o5_3);
            }
            { const double eb = bi[29];
              o5_3 = fma(eb, g3_6, o5_3);
            }
            { const double eb = bi[30];
              o5_3 = fma(eb, g3_3, o5_3);
            }
            { const double eb = bi[31];
              o5_3 = fma(eb, g3_8, o5_3);
            }
            { const double eb = bi[32];
              o5_3 = fma(eb, g3_16, o5_3);
            }
            { const double eb = bi[33];
              o6_3 = fma(eb, g3_0, o6_3);
            }
            { const double eb = bi[34];
              o6_3 = fma(eb, g3_2, o6_3);
            }
            { const double eb = bi[35];
              o6_3 = fma(eb, g3_6, o6_3);
            }
            { const double eb = bi[36];
              o6_3 = fma(eb, g3_13, o6_3);
            }
            { const double eb = bi[37];
              o7_3 = fma(eb, g3_0, o7_3);
            }
            { const double eb = bi[38];
              o7_3 = fma(eb, g3_1, o7_3);
            }
            { const double eb = bi[39];
              o7_3 = fma(eb, g3_2, o7_3);
            }
            { const double eb = bi[40];
              o7_3 = fma(eb, g3_5, o7_3);
            }
            { const double eb = bi[41];
              o7_3 = fma(eb, g3_6, o7_3);
            }
            { const double eb = bi[42];
              o7_3 = fma(eb, g3_12, o7_3);
            }
            { const double eb = bi[43];
              o8_3 = fma(eb, g3_0, o8_3);
            }
            { const double eb = bi[44];
              o8_3 = fma(eb, g3_1, o8_3);
            }
            { const double eb = bi[45];
              o8_3 = fma(eb, g3_4, o8_3);
            }
            { const double eb = bi[46];
              o9_3 = fma(eb, g3_0, o9_3);
            }
            { const double eb = bi[47];
              o9_3 = fma(eb, g3_1, o9_3);
            }
            { const double eb = bi[48];
              o9_3 = fma(eb, g3_4, o9_3);
            }
            { const double eb = bi[49];
              o9_3 = fma(eb, g3_3, o9_3);
            }
            { const double eb = bi[50];
              o9_3 = fma(eb, g3_7, o9_3);
            }
            { const double eb = bi[51];
              o9_3 = fma(eb, g3_14, o9_3);
            }
            { const double eb = bi[52];
              o10_3 = fma(eb, g3_0, o10_3);
            }
            { const double eb = bi[53];
              o10_3 = fma(eb, g3_1, o10_3);
            }
            { const double eb = bi[54];
              o10_3 = fma(eb, g3_4, o10_3);
            }
            { const double eb = bi[55];
              o10_3 = fma(eb, g3_2, o10_3);
            }
            { const double eb = bi[56];
              o10_3 = fma(eb, g3_5, o10_3);
            }
            { const double eb = bi[57];
              o10_3 = fma(eb, g3_11, o10_3);
            }
            { const double eb = bi[58];
              o11_3 = fma(eb, g3_0, o11_3);
            }
            { const double eb = bi[59];
              o11_3 = fma(eb, g3_1, o11_3);
            }
            { const double eb = bi[60];
              o11_3 = fma(eb, g3_4, o11_3);
            }
            { const double eb = bi[61];
              o11_3 = fma(eb, g3_10, o11_3);
            }
            { const double eb = bi[62];
              o12_3 = fma(eb, g3_0, o12_3);
            }
            { const double eb = bi[63];
              o12_3 = fma(eb, g3_2, o12_3);
            }
            { const double eb = bi[64];
              o12_3 = fma(eb, g3_3, o12_3);
            }
            { const double eb = bi[65];
              o12_3 = fma(eb, g3_8, o12_3);
            }
            { const double eb = bi[66];
              o13_3 = fma(eb, g3_0, o13_3);
            }
            { const double eb = bi[67];
              o13_3 = fma(eb, g3_2, o13_3);
            }
            { const double eb = bi[68];
              o13_3 = fma(eb, g3_3, o13_3);
            }
            { const double eb = bi[69];
              o13_3 = fma(eb, g3_8, o13_3);
            }
            { const double eb = bi[70];
              o13_3 = fma(eb, g3_9, o13_3);
            }
            { const double eb = bi[71];
              o13_3 = fma(eb, g3_18, o13_3);
            }
            { const double eb = bi[72];
              o14_3 = fma(eb, g3_0, o14_3);
            }
            { const double eb = bi[73];
              o14_3 = fma(eb, g3_2, o14_3);
            }
            { const double eb = bi[74];
              o14_3 = fma(eb, g3_6, o14_3);
            }
            { const double eb = bi[75];
              o14_3 = fma(eb, g3_3, o14_3);
            }
            { const double eb = bi[76];
              o14_3 = fma(eb, g3_8, o14_3);
            }
            { const double eb = bi[77];
              o14_3 = fma(eb, g3_16, o14_3);
            }
            { const double eb = bi[78];
              o15_3 = fma(eb, g3_0, o15_3);
            }
            { const double eb = bi[79];
              o15_3 = fma(eb, g3_1, o15_3);
            }
            { const double eb = bi[80];
              o15_3 = fma(eb, g3_2, o15_3);
            }
            { const double eb = bi[81];
              o15_3 = fma(eb, g3_5, o15_3);
            }
            { const double eb = bi[82];
              o15_3 = fma(eb, g3_3, o15_3);
            }
            { const double eb = bi[83];
              o15_3 = fma(eb, g3_7, o15_3);
            }
            { const double eb = bi[84];
              o15_3 = fma(eb, g3_8, o15_3);
            }
            { const double eb = bi[85];
              o15_3 = fma(eb, g3_15, o15_3);
            }
            { const double eb = bi[86];
              o16_3 = fma(eb, g3_0, o16_3);
            }
            { const double eb = bi[87];
              o16_3 = fma(eb, g3_1, o16_3);
            }
            { const double eb = bi[88];
              o16_3 = fma(eb, g3_3, o16_3);
            }
            { const double eb = bi[89];
              o16_3 = fma(eb, g3_7, o16_3);
            }
            { const double eb = bi[90];
              o17_3 = fma(eb, g3_0, o17_3);
            }
            { const double eb = bi[91];
              o17_3 = fma(eb, g3_1, o17_3);
            }
            { const double eb = bi[92];
              o17_3 = fma(eb, g3_3, o17_3);
            }
            { const double eb = bi[93];
              o17_3 = fma(eb, g3_7, o17_3);
            }
            { const double eb = bi[94];
              o17_3 = fma(eb, g3_9, o17_3);
            }
            { const double eb = bi[95];
              o17_3 = fma(eb, g3_17, o17_3);
            }
            { const double eb = bi[96];
              o18_3 = fma(eb, g3_0, o18_3);
            }
            { const double eb = bi[97];
              o18_3 = fma(eb, g3_1, o18_3);
            }
            { const double eb = bi[98];
              o18_3 = fma(eb, g3_2, o18_3);
            }
            { const double eb = bi[99];
              o18_3 = fma(eb, g3_5, o18_3);
            }
            { const double eb = bi[100];
              o18_3 = fma(eb, g3_3, o18_3);
            }
            { const double eb = bi[101];
              o18_3 = fma(eb, g3_7, o18_3);
            }
            { const double eb = bi[102];
              o18_3 = fma(eb, g3_8, o18_3);
            }
            { const double eb = bi[103];
              o18_3 = fma(eb, g3_15, o18_3);
            }
            { const double eb = bi[104];
              o19_3 = fma(eb, g3_0, o19_3);
            }
            { const double eb = bi[105];
              o19_3 = fma(eb, g3_1, o19_3);
            }
            { const double eb = bi[106];
              o19_3 = fma(eb, g3_4, o19_3);
            }
            { const double eb = bi[107];
              o19_3 = fma(eb, g3_3, o19_3);
            }
            { const double eb = bi[108];
              o19_3 = fma(eb, g3_7, o19_3);
            }
            { const double eb = bi[109];
              o19_3 = fma(eb, g3_14, o19_3);
            }
            { const double eb = bi[110];
              o20_3 = fma(eb, g3_0, o20_3);
            }
            { const double eb = bi[111];
              o20_3 = fma(eb, g3_1, o20_3);
            }
            { const double eb = bi[112];
              o20_3 = fma(eb, g3_2, o20_3);
            }
            { const double eb = bi[113];
              o20_3 = fma(eb, g3_5, o20_3);
            }
            { const double eb = bi[114];
              o21_3 = fma(eb, g3_0, o21_3);
            }
            { const double eb = bi[115];
              o21_3 = fma(eb, g3_1, o21_3);
            }
            { const double eb = bi[116];
              o21_3 = fma(eb, g3_2, o21_3);
            }
            { const double eb = bi[117];
              o21_3 = fma(eb, g3_5, o21_3);
            }
            { const double eb = bi[118];
              o21_3 = fma(eb, g3_3, o21_3);
            }
            { const double eb = bi[119];
              o21_3 = fma(eb, g3_7, o21_3);
            }
            { const double eb = bi[120];
              o21_3 = fma(eb, g3_8, o21_3);
            }
            { const double eb = bi[121];
              o21_3 = fma(eb, g3_15, o21_3);
            }
            { const double eb = bi[122];
              o22_3 = fma(eb, g3_0, o22_3);
            }
            { const double eb = bi[123];
              o22_3 = fma(eb, g3_1, o22_3);
            }
            { const double eb = bi[124];
              o22_3 = fma(eb, g3_2, o22_3);
            }
            { const double eb = bi[125];
              o22_3 = fma(eb, g3_5, o22_3);
            }
            { const double eb = bi[126];
              o22_3 = fma(eb, g3_6, o22_3);
            }
            { const double eb = bi[127];
              o22_3 = fma(eb, g3_12, o22_3);
            }
            { const double eb = bi[128];
              o23_3 = fma(eb, g3_0, o23_3);
            }
            { const double eb = bi[129];
              o23_3 = fma(eb, g3_1, o23_3);
            }
            { const double eb = bi[130];
              o23_3 = fma(eb, g3_4, o23_3);
            }
            { const double eb = bi[131];
              o23_3 = fma(eb, g3_2, o23_3);
            }
            { const double eb = bi[132];
              o23_3 = fma(eb, g3_5, o23_3);
            }
            { const double eb = bi[133];
              o23_3 = fma(eb, g3_11, o23_3);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 3);
            o1_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 3);
            o2_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 3);
            o3_3 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 3);
            o4_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 3);
            o5_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 3);
            o6_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 3);
            o7_3 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 3);
            o8_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 3);
            o9_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 3);
            o10_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 3);
            o11_3 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 3);
            o12_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 3);
            o13_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 3);
            o14_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 3);
            o15_3 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 3);
            o16_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 3);
            o17_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 3);
            o18_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 3);
            o19_3 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 3);
            o20_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 3);
            o21_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 3);
            o22_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 3);
            o23_3 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 3);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o1_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o2_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o3_3 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o4_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o5_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o6_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o7_3 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o8_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o9_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o10_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o11_3 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o12_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o13_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o14_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o15_3 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o16_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o17_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o18_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o19_3 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o20_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o21_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o22_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 0, fJ + 3)));
            e = fmax(e, fabs(o23_3 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 0, fJ + 3)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
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
            const double Bbd0_3 = PB[(fQ + 0) * N + fJ + 3];
            const double Bbd1_3 = PB[(fQ + 1) * N + fJ + 3];
            const double Bbd2_3 = PB[(fQ + 2) * N + fJ + 3];
            const double Bbd3_3 = PB[(fQ + 3) * N + fJ + 3];
            const double Bad0_3 = PB[(fP + 0) * N + fJ + 3];
            const double Bad1_3 = PB[(fP + 1) * N + fJ + 3];
            const double Bad2_3 = PB[(fP + 2) * N + fJ + 3];
            const double Bad3_3 = PB[(fP + 3) * N + fJ + 3];
            const double Bad4_3 = PB[(fP + 4) * N + fJ + 3];
            const double Bad5_3 = PB[(fP + 5) * N + fJ + 3];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc1_0 = PB[(fQ + 1) * N + fI + 0];
            const double Bbc2_0 = PB[(fQ + 2) * N + fI + 0];
            const double Bbc3_0 = PB[(fQ + 3) * N + fI + 0];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            const double Bac1_0 = PB[(fP + 1) * N + fI + 0];
            const double Bac2_0 = PB[(fP + 2) * N + fI + 0];
            const double Bac3_0 = PB[(fP + 3) * N + fI + 0];
            const double Bac4_0 = PB[(fP + 4) * N + fI + 0];
            const double Bac5_0 = PB[(fP + 5) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 3, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5 + o6_3 * ptb6 + o7_3 * ptb7 + o8_3 * ptb8 + o9_3 * ptb9 + o10_3 * ptb10 + o11_3 * ptb11 + o12_3 * ptb12 + o13_3 * ptb13 + o14_3 * ptb14 + o15_3 * ptb15 + o16_3 * ptb16 + o17_3 * ptb17 + o18_3 * ptb18 + o19_3 * ptb19 + o20_3 * ptb20 + o21_3 * ptb21 + o22_3 * ptb22 + o23_3 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_3 * Abd0_3 + o1_3 * Abd1_3 + o2_3 * Abd2_3 + o3_3 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_3 * Aad0_3 + o4_3 * Aad1_3 + o8_3 * Aad2_3 + o12_3 * Aad3_3 + o16_3 * Aad4_3 + o20_3 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_3 * Abc0_0 + o1_3 * Abc1_0 + o2_3 * Abc2_0 + o3_3 * Abc3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_3 * Aac0_0 + o4_3 * Aac1_0 + o8_3 * Aac2_0 + o12_3 * Aac3_0 + o16_3 * Aac4_0 + o20_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_3 * Aad0_3 + o5_3 * Aad1_3 + o9_3 * Aad2_3 + o13_3 * Aad3_3 + o17_3 * Aad4_3 + o21_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_3 * Aac0_0 + o5_3 * Aac1_0 + o9_3 * Aac2_0 + o13_3 * Aac3_0 + o17_3 * Aac4_0 + o21_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_3 * Aad0_3 + o6_3 * Aad1_3 + o10_3 * Aad2_3 + o14_3 * Aad3_3 + o18_3 * Aad4_3 + o22_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_3 * Aac0_0 + o6_3 * Aac1_0 + o10_3 * Aac2_0 + o14_3 * Aac3_0 + o18_3 * Aac4_0 + o22_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_3 * Aad0_3 + o7_3 * Aad1_3 + o11_3 * Aad2_3 + o15_3 * Aad3_3 + o19_3 * Aad4_3 + o23_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_3 * Aac0_0 + o7_3 * Aac1_0 + o11_3 * Aac2_0 + o15_3 * Aac3_0 + o19_3 * Aac4_0 + o23_3 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_3 * Abd0_3 + o5_3 * Abd1_3 + o6_3 * Abd2_3 + o7_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_3 * Abc0_0 + o5_3 * Abc1_0 + o6_3 * Abc2_0 + o7_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_3 * Abd0_3 + o9_3 * Abd1_3 + o10_3 * Abd2_3 + o11_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_3 * Abc0_0 + o9_3 * Abc1_0 + o10_3 * Abc2_0 + o11_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_3 * Abd0_3 + o13_3 * Abd1_3 + o14_3 * Abd2_3 + o15_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_3 * Abc0_0 + o13_3 * Abc1_0 + o14_3 * Abc2_0 + o15_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o16_3 * Abd0_3 + o17_3 * Abd1_3 + o18_3 * Abd2_3 + o19_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_3 * Abc0_0 + o17_3 * Abc1_0 + o18_3 * Abc2_0 + o19_3 * Abc3_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o20_3 * Abd0_3 + o21_3 * Abd1_3 + o22_3 * Abd2_3 + o23_3 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_3 * Abc0_0 + o21_3 * Abc1_0 + o22_3 * Abc2_0 + o23_3 * Abc3_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_3 * Bbd0_3 + o1_3 * Bbd1_3 + o2_3 * Bbd2_3 + o3_3 * Bbd3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_3 * Bad0_3 + o4_3 * Bad1_3 + o8_3 * Bad2_3 + o12_3 * Bad3_3 + o16_3 * Bad4_3 + o20_3 * Bad5_3));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 3, deg * (o0_3 * Bbc0_0 + o1_3 * Bbc1_0 + o2_3 * Bbc2_0 + o3_3 * Bbc3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 3, deg * (o0_3 * Bac0_0 + o4_3 * Bac1_0 + o8_3 * Bac2_0 + o12_3 * Bac3_0 + o16_3 * Bac4_0 + o20_3 * Bac5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_3 * Bad0_3 + o5_3 * Bad1_3 + o9_3 * Bad2_3 + o13_3 * Bad3_3 + o17_3 * Bad4_3 + o21_3 * Bad5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 3, deg * (o1_3 * Bac0_0 + o5_3 * Bac1_0 + o9_3 * Bac2_0 + o13_3 * Bac3_0 + o17_3 * Bac4_0 + o21_3 * Bac5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_3 * Bad0_3 + o6_3 * Bad1_3 + o10_3 * Bad2_3 + o14_3 * Bad3_3 + o18_3 * Bad4_3 + o22_3 * Bad5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 3, deg * (o2_3 * Bac0_0 + o6_3 * Bac1_0 + o10_3 * Bac2_0 + o14_3 * Bac3_0 + o18_3 * Bac4_0 + o22_3 * Bac5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 0, deg * (o3_3 * Bad0_3 + o7_3 * Bad1_3 + o11_3 * Bad2_3 + o15_3 * Bad3_3 + o19_3 * Bad4_3 + o23_3 * Bad5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 3, deg * (o3_3 * Bac0_0 + o7_3 * Bac1_0 + o11_3 * Bac2_0 + o15_3 * Bac3_0 + o19_3 * Bac4_0 + o23_3 * Bac5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o4_3 * Bbd0_3 + o5_3 * Bbd1_3 + o6_3 * Bbd2_3 + o7_3 * Bbd3_3));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 3, deg * (o4_3 * Bbc0_0 + o5_3 * Bbc1_0 + o6_3 * Bbc2_0 + o7_3 * Bbc3_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o8_3 * Bbd0_3 + o9_3 * Bbd1_3 + o10_3 * Bbd2_3 + o11_3 * Bbd3_3));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 3, deg * (o8_3 * Bbc0_0 + o9_3 * Bbc1_0 + o10_3 * Bbc2_0 + o11_3 * Bbc3_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o12_3 * Bbd0_3 + o13_3 * Bbd1_3 + o14_3 * Bbd2_3 + o15_3 * Bbd3_3));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 3, deg * (o12_3 * Bbc0_0 + o13_3 * Bbc1_0 + o14_3 * Bbc2_0 + o15_3 * Bbc3_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o16_3 * Bbd0_3 + o17_3 * Bbd1_3 + o18_3 * Bbd2_3 + o19_3 * Bbd3_3));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 3, deg * (o16_3 * Bbc0_0 + o17_3 * Bbc1_0 + o18_3 * Bbc2_0 + o19_3 * Bbc3_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o20_3 * Bbd0_3 + o21_3 * Bbd1_3 + o22_3 * Bbd2_3 + o23_3 * Bbd3_3));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 3, deg * (o20_3 * Bbc0_0 + o21_3 * Bbc1_0 + o22_3 * Bbc2_0 + o23_3 * Bbc3_0));
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek4_0 = kj[12 * kS];
              const double ek4_1 = -kj[13 * kS];
              g4_0 = fma(ek4_0, b0, g4_0);
              const double r0_0_0_1 = Z * b1;
              g4_1 = fma(ek4_0, r0_0_0_1, g4_1);
              const double r0_0_1_0 = Y * b1;
              g4_2 = fma(ek4_0, r0_0_1_0, g4_2);
              const double r0_1_0_0 = X * b1;
              g4_3 = fma(ek4_0, r0_1_0_0, g4_3);
              g4_0 = fma(ek4_1, r0_1_0_0, g4_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g4_4 = fma(ek4_0, r0_0_0_2, g4_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g4_5 = fma(ek4_0, r0_0_1_1, g4_5);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g4_6 = fma(ek4_0, r0_0_2_0, g4_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g4_7 = fma(ek4_0, r0_1_0_1, g4_7);
              g4_1 = fma(ek4_1, r0_1_0_1, g4_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g4_8 = fma(ek4_0, r0_1_1_0, g4_8);
              g4_2 = fma(ek4_1, r0_1_1_0, g4_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g4_9 = fma(ek4_0, r0_2_0_0, g4_9);
              g4_3 = fma(ek4_1, r0_2_0_0, g4_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g4_10 = fma(ek4_0, r0_0_0_3, g4_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g4_11 = fma(ek4_0, r0_0_1_2, g4_11);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g4_12 = fma(ek4_0, r0_0_2_1, g4_12);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g4_13 = fma(ek4_0, r0_0_3_0, g4_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g4_14 = fma(ek4_0, r0_1_0_2, g4_14);
              g4_4 = fma(ek4_1, r0_1_0_2, g4_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g4_15 = fma(ek4_0, r0_1_1_1, g4_15);
              g4_5 = fma(ek4_1, r0_1_1_1, g4_5);
              const double r0_1_2_0 = X * r1_0_2_0;
              g4_16 = fma(ek4_0, r0_1_2_0, g4_16);
              g4_6 = fma(ek4_1, r0_1_2_0, g4_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g4_17 = fma(ek4_0, r0_2_0_1, g4_17);
              g4_7 = fma(ek4_1, r0_2_0_1, g4_7);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g4_18 = fma(ek4_0, r0_2_1_0, g4_18);
              g4_8 = fma(ek4_1, r0_2_1_0, g4_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g4_19 = fma(ek4_0, r0_3_0_0, g4_19);
              g4_9 = fma(ek4_1, r0_3_0_0, g4_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_1_0_3 = X * r1_0_0_3;
              g4_10 = fma(ek4_1, r0_1_0_3, g4_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_1_1_2 = X * r1_0_1_2;
              g4_11 = fma(ek4_1, r0_1_1_2, g4_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g4_12 = fma(ek4_1, r0_1_2_1, g4_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g4_13 = fma(ek4_1, r0_1_3_0, g4_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g4_14 = fma(ek4_1, r0_2_0_2, g4_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g4_15 = fma(ek4_1, r0_2_1_1, g4_15);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g4_16 = fma(ek4_1, r0_2_2_0, g4_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g4_17 = fma(ek4_1, r0_3_0_1, g4_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g4_18 = fma(ek4_1, r0_3_1_0, g4_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g4_19 = fma(ek4_1, r0_4_0_0, g4_19);
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
              o1_4 = fma(eb, g4_0, o1_4);
            }
            { const double eb = bi[9];
              o1_4 = fma(eb, g4_3, o1_4);
            }
            { const double eb = bi[10];
              o1_4 = fma(eb, g4_9, o1_4);
            }
            { const double eb = bi[11];
              o1_4 = fma(eb, g4_19, o1_4);
            }
            { const double eb = bi[12];
              o2_4 = fma(eb, g4_0, o2_4);
            }
            { const double eb = bi[13];
              o2_4 = fma(eb, g4_2, o2_4);
            }
            { const double eb = bi[14];
              o2_4 = fma(eb, g4_3, o2_4);
            }
            { const double eb = bi[15];
              o2_4 = fma(eb, g4_8, o2_4);
            }
            { const double eb = bi[16];
              o2_4 = fma(eb, g4_9, o2_4);
            }
            { const double eb = bi[17];
              o2_4 = fma(eb, g4_18, o2_4);
            }
            { const double eb = bi[18];
              o3_4 = fma(eb, g4_0, o3_4);
            }
            { const double eb = bi[19];
              o3_4 = fma(eb, g4_1, o3_4);
            }
            { const double eb = bi[20];
              o3_4 = fma(eb, g4_3, o3_4);
            }
            { const double eb = bi[21];
              o3_4 = fma(eb, g4_7, o3_4);
            }
            { const double eb = bi[22];
              o3_4 = fma(eb, g4_9, o3_4);
            }
            { const double eb = bi[23];
              o3_4 = fma(eb, g4_17, o3_4);
            }
            { const double eb = bi[24];
              o4_4 = fma(eb, g4_0, o4_4);
            }
            { const double eb = bi[25];
              o4_4 = fma(eb, g4_2, o4_4);
            }
            { const double eb = bi[26];
              o4_4 = fma(eb, g4_6, o4_4);
            }
            { const double eb = bi[27];
              o5_4 = fma(eb, g4_0, o5_4);
            }
            { const double eb = bi[28];
              o5_4 = fma(eb, g4_2, o5_4);
            }
            { const double eb = bi[29];
              o5_4 = fma(eb, g4_6, o5_4);
            }
            { const double eb = bi[30];
              o5_4 = fma(eb, g4_3, o5_4);
            }
            { const double eb = bi[31];
              o5_4 = fma(eb, g4_8, o5_4);
            }
            { const double eb = bi[32];
              o5_4 = fma(eb, g4_16, o5_4);
            }
            { const double eb = bi[33];
              o6_4 = fma(eb, g4_0, o6_4);
            }
            { const double eb = bi[34];
              o6_4 = fma(eb, g4_2, o6_4);
            }
            { const double eb = bi[35];
              o6_4 = fma(eb, g4_6, o6_4);
            }
            { const double eb = bi[36];
              o6_4 = fma(eb, g4_13, o6_4);
            }
            { const double eb = bi[37];
              o7_4 = fma(eb, g4_0, o7_4);
            }
            { const double eb = bi[38];
              o7_4 = fma(eb, g4_1, o7_4);
            }
            { const double eb = bi[39];
              o7_4 = fma(eb, g4_2, o7_4);
            }
            { const double eb = bi[40];
              o7_4 = fma(eb, g4_5, o7_4);
            }
            { const double eb = bi[41];
              o7_4 = fma(eb, g4_6, o7_4);
            }
            { const double eb = bi[42];
              o7_4 = fma(eb, g4_12, o7_4);
            }
            { const double eb = bi[43];
              o8_4 = fma(eb, g4_0, o8_4);
            }
            { const double eb = bi[44];
              o8_4 = fma(eb, g4_1, o8_4);
            }
            { const double eb = bi[45];
              o8_4 = fma(eb, g4_4, o8_4);
            }
            { const double eb = bi[46];
              o9_4 = fma(eb, g4_0, o9_4);
            }
            { const double eb = bi[47];
              o9_4 = fma(eb, g4_1, o9_4);
            }
            { const double eb = bi[48];
              o9_4 = fma(eb, g4_4, o9_4);
            }
            { const double eb = bi[49];
              o9_4 = fma(eb, g4_3, o9_4);
            }
            { const double eb = bi[50];
              o9_4 = fma(eb, g4_7, o9_4);
            }
            { const double eb = bi[51];
              o9_4 = fma(eb, g4_14, o9_4);
            }
            { const double eb = bi[52];
              o10_4 = fma(eb, g4_0, o10_4);
            }
            { const double eb = bi[53];
              o10_4 = fma(eb, g4_1, o10_4);
            }
            { const double eb = bi[54];
              o10_4 = fma(eb, g4_4, o10_4);
            }
            { const double eb = bi[55];
              o10_4 = fma(eb, g4_2, o10_4);
            }
            { const double eb = bi[56];
              o10_4 = fma(eb, g4_5, o10_4);
            }
            { const double eb = bi[57];
              o10_4 = fma(eb, g4_11, o10_4);
            }
            { const double eb = bi[58];
              o11_4 = fma(eb, g4_0, o11_4);
            }
            { const double eb = bi[59];
              o11_4 = fma(eb, g4_1, o11_4);
            }
            { const double eb = bi[60];
              o11_4 = fma(eb, g4_4, o11_4);
            }
            { const double eb = bi[61];
              o11_4 = fma(eb, g4_10, o11_4);
            }
            { const double eb = bi[62];
              o12_4 = fma(eb, g4_0, o12_4);
            }
            { const double eb = bi[63];
              o12_4 = fma(eb, g4_2, o12_4);
            }
            { const double eb = bi[64];
              o12_4 = fma(eb, g4_3, o12_4);
            }
            { const double eb = bi[65];
              o12_4 = fma(eb, g4_8, o12_4);
            }
            { const double eb = bi[66];
              o13_4 = fma(eb, g4_0, o13_4);
            }
            { const double eb = bi[67];
              o13_4 = fma(eb, g4_2, o13_4);
            }
            { const double eb = bi[68];
              o13_4 = fma(eb, g4_3, o13_4);
            }
            { const double eb = bi[69];
              o13_4 = fma(eb, g4_8, o13_4);
            }
            { const double eb = bi[70];
              o13_4 = fma(eb, g4_9, o13_4);
            }
            { const double eb = bi[71];
              o13_4 = fma(eb, g4_18, o13_4);
            }
            { const double eb = bi[72];
              o14_4 = fma(eb, g4_0, o14_4);
            }
            { const double eb = bi[73];
              o14_4 = fma(eb, g4_2, o14_4);
            }
            { const double eb = bi[74];
              o14_4 = fma(eb, g4_6, o14_4);
            }
            { const double eb = bi[75];
              o14_4 = fma(eb, g4_3, o14_4);
            }
            { const double eb = bi[76];
              o14_4 = fma(eb, g4_8, o14_4);
            }
            { const double eb = bi[77];
              o14_4 = fma(eb, g4_16, o14_4);
            }
            { const double eb = bi[78];
              o15_4 = fma(eb, g4_0, o15_4);
            }
            { const double eb = bi[79];
              o15_4 = fma(eb, g4_1, o15_4);
            }
            { const double eb = bi[80];
              o15_4 = fma(eb, g4_2, o15_4);
            }
            { const double eb = bi[81];
              o15_4 = fma(eb, g4_5, o15_4);
            }
            { const double eb = bi[82];
              o15_4 = fma(eb, g4_3, o15_4);
            }
            { const double eb = bi[83];
              o15_4 = fma(eb, g4_7, o15_4);
            }
            { const double eb = bi[84];
              o15_4 = fma(eb, g4_8, o15_4);
            }
            { const double eb = bi[85];
              o15_4 = fma(eb, g4_15, o15_4);
            }
            { const double eb = bi[86];
              o16_4 = fma(eb, g4_0, o16_4);
            }
            { const double eb = bi[87];
              o16_4 = fma(eb, g4_1, o16_4);
            }
            { const double eb = bi[88];
              o16_4 = fma(eb, g4_3, o16_4);
            }
            { const double eb = bi[89];
              o16_4 = fma(eb, g4_7, o16_4);
            }
            { const double eb = bi[90];
              o17_4 = fma(eb, g4_0, o17_4);
            }
            { const double eb = bi[91];
              o17_4 = fma(eb, g4_1, o17_4);
            }
            { const double eb = bi[92];
              o17_4 = fma(eb, g4_3, o17_4);
            }
            { const double eb = bi[93];
              o17_4 = fma(eb, g4_7, o17_4);
            }
            { const double eb = bi[94];
              o17_4 = fma(eb, g4_9, o17_4);
            }
            { const double eb = bi[95];
              o17_4 = fma(eb, g4_17, o17_4);
            }
            { const double eb = bi[96];
              o18_4 = fma(eb, g4_0, o18_4);
            }
            { const double eb = bi[97];
              o18_4 = fma(eb, g4_1, o18_4);
            }
            { const double eb = bi[98];
              o18_4 = fma(eb, g4_2, o18_4);
            }
            { const double eb = bi[99];
              o18_4 = fma(eb, g4_5, o18_4);
            }
            { const double eb = bi[100];
              o18_4 = fma(eb, g4_3, o18_4);
            }
            { const double eb = bi[101];
              o18_4 = fma(eb, g4_7, o18_4);
            }
            { const double eb = bi[102];
              o18_4 = fma(eb, g4_8, o18_4);
            }
            { const double eb = bi[103];
              o18_4 = fma(eb, g4_15, o18_4);
            }
            { const double eb = bi[104];
              o19_4 = fma(eb, g4_0, o19_4);
            }
            { const double eb = bi[105];
              o19_4 = fma(eb, g4_1, o19_4);
            }
            { const double eb = bi[106];
              o19_4 = fma(eb, g4_4, o19_4);
            }
            { const double eb = bi[107];
              o19_4 = fma(eb, g4_3, o19_4);
            }
            { const double eb = bi[108];
              o19_4 = fma(eb, g4_7, o19_4);
            }
            { const double eb = bi[109];
              o19_4 = fma(eb, g4_14, o19_4);
            }
            { const double eb = bi[110];
              o20_4 = fma(eb, g4_0, o20_4);
            }
            { const double eb = bi[111];
              o20_4 = fma(eb, g4_1, o20_4);
            }
            { const double eb = bi[112];
              o20_4 = fma(eb, g4_2, o20_4);
            }
            { const double eb = bi[113];
              o20_4 = fma(eb, g4_5, o20_4);
            }
            { const double eb = bi[114];
              o21_4 = fma(eb, g4_0, o21_4);
            }
            { const double eb = bi[115];
              o21_4 = fma(eb, g4_1, o21_4);
            }
            { const double eb = bi[116];
              o21_4 = fma(eb, g4_2, o21_4);
            }
            { const double eb = bi[117];
              o21_4 = fma(eb, g4_5, o21_4);
            }
            { const double eb = bi[118];
              o21_4 = fma(eb, g4_3, o21_4);
            }
            { const double eb = bi[119];
              o21_4 = fma(eb, g4_7, o21_4);
            }
            { const double eb = bi[120];
              o21_4 = fma(eb, g4_8, o21_4);
            }
            { const double eb = bi[121];
              o21_4 = fma(eb, g4_15, o21_4);
            }
            { const double eb = bi[122];
              o22_4 = fma(eb, g4_0, o22_4);
            }
            { const double eb = bi[123];
              o22_4 = fma(eb, g4_1, o22_4);
            }
            { const double eb = bi[124];
              o22_4 = fma(eb, g4_2, o22_4);
            }
            { const double eb = bi[125];
              o22_4 = fma(eb, g4_5, o22_4);
            }
            { const double eb = bi[126];
              o22_4 = fma(eb, g4_6, o22_4);
            }
            { const double eb = bi[127];
              o22_4 = fma(eb, g4_12, o22_4);
            }
            { const double eb = bi[128];
              o23_4 = fma(eb, g4_0, o23_4);
            }
            { const double eb = bi[129];
              o23_4 = fma(eb, g4_1, o23_4);
            }
            { const double eb = bi[130];
              o23_4 = fma(eb, g4_4, o23_4);
            }
            { const double eb = bi[131];
              o23_4 = fma(eb, g4_2, o23_4);
            }
            { const double eb = bi[132];
              o23_4 = fma(eb, g4_5, o23_4);
            }
            { const double eb = bi[133];
              o23_4 = fma(eb, g4_11, o23_4);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0);
            o1_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 0);
            o2_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 0);
            o3_4 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 0);
            o4_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0);
            o5_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 0);
            o6_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 0);
            o7_4 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 0);
            o8_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0);
            o9_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 0);
            o10_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 0);
            o11_4 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 0);
            o12_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0);
            o13_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 0);
            o14_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 0);
            o15_4 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 0);
            o16_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0);
            o17_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 0);
            o18_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 0);
            o19_4 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 0);
            o20_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0);
            o21_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 0);
            o22_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 0);
            o23_4 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o1_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o2_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o3_4 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o4_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o5_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o6_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o7_4 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o8_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o9_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o10_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o11_4 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o12_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o13_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o14_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o15_4 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o16_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o17_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o18_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o19_4 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o20_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o21_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o22_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o23_4 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk4 = PT[(fI + 1) * N + fJ + 0];
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
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
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
            const double Bac0_1 = PB[(fP + 0) * N + fI + 1];
            const double Bac1_1 = PB[(fP + 1) * N + fI + 1];
            const double Bac2_1 = PB[(fP + 2) * N + fI + 1];
            const double Bac3_1 = PB[(fP + 3) * N + fI + 1];
            const double Bac4_1 = PB[(fP + 4) * N + fI + 1];
            const double Bac5_1 = PB[(fP + 5) * N + fI + 1];
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
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_4 * ptb0 + o1_4 * ptb1 + o2_4 * ptb2 + o3_4 * ptb3 + o4_4 * ptb4 + o5_4 * ptb5 + o6_4 * ptb6 + o7_4 * ptb7 + o8_4 * ptb8 + o9_4 * ptb9 + o10_4 * ptb10 + o11_4 * ptb11 + o12_4 * ptb12 + o13_4 * ptb13 + o14_4 * ptb14 + o15_4 * ptb15 + o16_4 * ptb16 + o17_4 * ptb17 + o18_4 * ptb18 + o19_4 * ptb19 + o20_4 * ptb20 + o21_4 * ptb21 + o22_4 * ptb22 + o23_4 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_4 * Abd0_0 + o1_4 * Abd1_0 + o2_4 * Abd2_0 + o3_4 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_4 * Aad0_0 + o4_4 * Aad1_0 + o8_4 * Aad2_0 + o12_4 * Aad3_0 + o16_4 * Aad4_0 + o20_4 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Abc0_1 + o1_4 * Abc1_1 + o2_4 * Abc2_1 + o3_4 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Aac0_1 + o4_4 * Aac1_1 + o8_4 * Aac2_1 + o12_4 * Aac3_1 + o16_4 * Aac4_1 + o20_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_4 * Aad0_0 + o5_4 * Aad1_0 + o9_4 * Aad2_0 + o13_4 * Aad3_0 + o17_4 * Aad4_0 + o21_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Aac0_1 + o5_4 * Aac1_1 + o9_4 * Aac2_1 + o13_4 * Aac3_1 + o17_4 * Aac4_1 + o21_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_4 * Aad0_0 + o6_4 * Aad1_0 + o10_4 * Aad2_0 + o14_4 * Aad3_0 + o18_4 * Aad4_0 + o22_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Aac0_1 + o6_4 * Aac1_1 + o10_4 * Aac2_1 + o14_4 * Aac3_1 + o18_4 * Aac4_1 + o22_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_4 * Aad0_0 + o7_4 * Aad1_0 + o11_4 * Aad2_0 + o15_4 * Aad3_0 + o19_4 * Aad4_0 + o23_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Aac0_1 + o7_4 * Aac1_1 + o11_4 * Aac2_1 + o15_4 * Aac3_1 + o19_4 * Aac4_1 + o23_4 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_4 * Abd0_0 + o5_4 * Abd1_0 + o6_4 * Abd2_0 + o7_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_4 * Abc0_1 + o5_4 * Abc1_1 + o6_4 * Abc2_1 + o7_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_4 * Abd0_0 + o9_4 * Abd1_0 + o10_4 * Abd2_0 + o11_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_4 * Abc0_1 + o9_4 * Abc1_1 + o10_4 * Abc2_1 + o11_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_4 * Abd0_0 + o13_4 * Abd1_0 + o14_4 * Abd2_0 + o15_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_4 * Abc0_1 + o13_4 * Abc1_1 + o14_4 * Abc2_1 + o15_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_4 * Abd0_0 + o17_4 * Abd1_0 + o18_4 * Abd2_0 + o19_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_4 * Abc0_1 + o17_4 * Abc1_1 + o18_4 * Abc2_1 + o19_4 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_4 * Abd0_0 + o21_4 * Abd1_0 + o22_4 * Abd2_0 + o23_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_4 * Abc0_1 + o21_4 * Abc1_1 + o22_4 * Abc2_1 + o23_4 * Abc3_1));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_4 * Bbd0_0 + o1_4 * Bbd1_0 + o2_4 * Bbd2_0 + o3_4 * Bbd3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_4 * Bad0_0 + o4_4 * Bad1_0 + o8_4 * Bad2_0 + o12_4 * Bad3_0 + o16_4 * Bad4_0 + o20_4 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Bbc0_1 + o1_4 * Bbc1_1 + o2_4 * Bbc2_1 + o3_4 * Bbc3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Bac0_1 + o4_4 * Bac1_1 + o8_4 * Bac2_1 + o12_4 * Bac3_1 + o16_4 * Bac4_1 + o20_4 * Bac5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 1, deg * (o1_4 * Bad0_0 + o5_4 * Bad1_0 + o9_4 * Bad2_0 + o13_4 * Bad3_0 + o17_4 * Bad4_0 + o21_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Bac0_1 + o5_4 * Bac1_1 + o9_4 * Bac2_1 + o13_4 * Bac3_1 + o17_4 * Bac4_1 + o21_4 * Bac5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 1, deg * (o2_4 * Bad0_0 + o6_4 * Bad1_0 + o10_4 * Bad2_0 + o14_4 * Bad3_0 + o18_4 * Bad4_0 + o22_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Bac0_1 + o6_4 * Bac1_1 + o10_4 * Bac2_1 + o14_4 * Bac3_1 + o18_4 * Bac4_1 + o22_4 * Bac5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 1, deg * (o3_4 * Bad0_0 + o7_4 * Bad1_0 + o11_4 * Bad2_0 + o15_4 * Bad3_0 + o19_4 * Bad4_0 + o23_4 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Bac0_1 + o7_4 * Bac1_1 + o11_4 * Bac2_1 + o15_4 * Bac3_1 + o19_4 * Bac4_1 + o23_4 * Bac5_1));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o4_4 * Bbd0_0 + o5_4 * Bbd1_0 + o6_4 * Bbd2_0 + o7_4 * Bbd3_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o4_4 * Bbc0_1 + o5_4 * Bbc1_1 + o6_4 * Bbc2_1 + o7_4 * Bbc3_1));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o8_4 * Bbd0_0 + o9_4 * Bbd1_0 + o10_4 * Bbd2_0 + o11_4 * Bbd3_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o8_4 * Bbc0_1 + o9_4 * Bbc1_1 + o10_4 * Bbc2_1 + o11_4 * Bbc3_1));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o12_4 * Bbd0_0 + o13_4 * Bbd1_0 + o14_4 * Bbd2_0 + o15_4 * Bbd3_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o12_4 * Bbc0_1 + o13_4 * Bbc1_1 + o14_4 * Bbc2_1 + o15_4 * Bbc3_1));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o16_4 * Bbd0_0 + o17_4 * Bbd1_0 + o18_4 * Bbd2_0 + o19_4 * Bbd3_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o16_4 * Bbc0_1 + o17_4 * Bbc1_1 + o18_4 * Bbc2_1 + o19_4 * Bbc3_1));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o20_4 * Bbd0_0 + o21_4 * Bbd1_0 + o22_4 * Bbd2_0 + o23_4 * Bbd3_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o20_4 * Bbc0_1 + o21_4 * Bbc1_1 + o22_4 * Bbc2_1 + o23_4 * Bbc3_1));
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
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek5_0 = kj[14 * kS];
              const double ek5_1 = -kj[15 * kS];
              const double ek5_2 = kj[16 * kS];
              g5_0 = fma(ek5_0, b0, g5_0);
              const double r0_0_0_1 = Z * b1;
              g5_1 = fma(ek5_0, r0_0_0_1, g5_1);
              const double r0_0_1_0 = Y * b1;
              g5_2 = fma(ek5_0, r0_0_1_0, g5_2);
              const double r0_1_0_0 = X * b1;
              g5_3 = fma(ek5_0, r0_1_0_0, g5_3);
              g5_0 = fma(ek5_1, r0_1_0_0, g5_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g5_4 = fma(ek5_0, r0_0_0_2, g5_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g5_5 = fma(ek5_0, r0_0_1_1, g5_5);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g5_6 = fma(ek5_0, r0_0_2_0, g5_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g5_7 = fma(ek5_0, r0_1_0_1, g5_7);
              g5_1 = fma(ek5_1, r0_1_0_1, g5_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g5_8 = fma(ek5_0, r0_1_1_0, g5_8);
              g5_2 = fma(ek5_1, r0_1_1_0, g5_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g5_9 = fma(ek5_0, r0_2_0_0, g5_9);
              g5_3 = fma(ek5_1, r0_2_0_0, g5_3);
              g5_0 = fma(ek5_2, r0_2_0_0, g5_0);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g5_10 = fma(ek5_0, r0_0_0_3, g5_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g5_11 = fma(ek5_0, r0_0_1_2, g5_11);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g5_12 = fma(ek5_0, r0_0_2_1, g5_12);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g5_13 = fma(ek5_0, r0_0_3_0, g5_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g5_14 = fma(ek5_0, r0_1_0_2, g5_14);
              g5_4 = fma(ek5_1, r0_1_0_2, g5_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g5_15 = fma(ek5_0, r0_1_1_1, g5_15);
              g5_5 = fma(ek5_1, r0_1_1_1, g5_5);
              const double r0_1_2_0 = X * r1_0_2_0;
              g5_16 = fma(ek5_0, r0_1_2_0, g5_16);
              g5_6 = fma(ek5_1, r0_1_2_0, g5_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g5_17 = fma(ek5_0, r0_2_0_1, g5_17);
              g5_7 = fma(ek5_1, r0_2_0_1, g5_7);
              g5_1 = fma(ek5_2, r0_2_0_1, g5_1);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g5_18 = fma(ek5_0, r0_2_1_0, g5_18);
              g5_8 = fma(ek5_1, r0_2_1_0, g5_8);
              g5_2 = fma(ek5_2, r0_2_1_0, g5_2);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g5_19 = fma(ek5_0, r0_3_0_0, g5_19);
              g5_9 = fma(ek5_1, r0_3_0_0, g5_9);
              g5_3 = fma(ek5_2, r0_3_0_0, g5_3);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_1_0_3 = X * r1_0_0_3;
              g5_10 = fma(ek5_1, r0_1_0_3, g5_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_1_1_2 = X * r1_0_1_2;
              g5_11 = fma(ek5_1, r0_1_1_2, g5_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_1_2_1 = X * r1_0_2_1;
              g5_12 = fma(ek5_1, r0_1_2_1, g5_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g5_13 = fma(ek5_1, r0_1_3_0, g5_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g5_14 = fma(ek5_1, r0_2_0_2, g5_14);
              g5_4 = fma(ek5_2, r0_2_0_2, g5_4);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g5_15 = fma(ek5_1, r0_2_1_1, g5_15);
              g5_5 = fma(ek5_2, r0_2_1_1, g5_5);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g5_16 = fma(ek5_1, r0_2_2_0, g5_16);
              g5_6 = fma(ek5_2, r0_2_2_0, g5_6);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g5_17 = fma(ek5_1, r0_3_0_1, g5_17);
              g5_7 = fma(ek5_2, r0_3_0_1, g5_7);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g5_18 = fma(ek5_1, r0_3_1_0, g5_18);
              g5_8 = fma(ek5_2, r0_3_1_0, g5_8);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g5_19 = fma(ek5_1, r0_4_0_0, g5_19);
              g5_9 = fma(ek5_2, r0_4_0_0, g5_9);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g5_10 = fma(ek5_2, r0_2_0_3, g5_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g5_11 = fma(ek5_2, r0_2_1_2, g5_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g5_12 = fma(ek5_2, r0_2_2_1, g5_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g5_13 = fma(ek5_2, r0_2_3_0, g5_13);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g5_14 = fma(ek5_2, r0_3_0_2, g5_14);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g5_15 = fma(ek5_2, r0_3_1_1, g5_15);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g5_16 = fma(ek5_2, r0_3_2_0, g5_16);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g5_17 = fma(ek5_2, r0_4_0_1, g5_17);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g5_18 = fma(ek5_2, r0_4_1_0, g5_18);
              const double r4_1_0_0 = X * b5;
              const double r3_2_0_0 = fma(X, r4_1_0_0, b4);
              const double r2_3_0_0 = fma(X, r3_2_0_0, 2.0 * r3_1_0_0);
              const double r1_4_0_0 = fma(X, r2_3_0_0, 3.0 * r2_2_0_0);
              const double r0_5_0_0 = fma(X, r1_4_0_0, 4.0 * r1_3_0_0);
              g5_19 = fma(ek5_2, r0_5_0_0, g5_19);
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
              o1_5 = fma(eb, g5_0, o1_5);
            }
            { const double eb = bi[9];
              o1_5 = fma(eb, g5_3, o1_5);
            }
            { const double eb = bi[10];
              o1_5 = fma(eb, g5_9, o1_5);
            }
            { const double eb = bi[11];
              o1_5 = fma(eb, g5_19, o1_5);
            }
            { const double eb = bi[12];
              o2_5 = fma(eb, g5_0, o2_5);
            }
            { const double eb = bi[13];
              o2_5 = fma(eb, g5_2, o2_5);
            }
            { const double eb = bi[14];
              o2_5 = fma(eb, g5_3, o2_5);
            }
            { const double eb = bi[15];
              o2_5 = fma(eb, g5_8, o2_5);
            }
            { const double eb = bi[16];
              o2_5 = fma(eb, g5_9, o2_5);
            }
            { const double eb = bi[17];
              o2_5 = fma(eb, g5_18, o2_5);
            }
            { const double eb = bi[18];
              o3_5 = fma(eb, g5_0, o3_5);
            }
            { const double eb = bi[19];
              o3_5 = fma(eb, g5_1, o3_5);
            }
            { const double eb = bi[20];
              o3_5 = fma(eb, g5_3, o3_5);
            }
            { const double eb = bi[21];
              o3_5 = fma(eb, g5_7, o3_5);
            }
            { const double eb = bi[22];
              o3_5 = fma(eb, g5_9, o3_5);
            }
            { const double eb = bi[23];
              o3_5 = fma(eb, g5_17, o3_5);
            }
            { const double eb = bi[24];
              o4_5 = fma(eb, g5_0, o4_5);
            }
            { const double eb = bi[25];
              o4_5 = fma(eb, g5_2, o4_5);
            }
            { const double eb = bi[26];
              o4_5 = fma(eb, g5_6, o4_5);
            }
            { const double eb = bi[27];
              o5_5 = fma(eb, g5_0, o5_5);
            }
            { const double eb = bi[28];
              o5_5 = fma(eb, g5_2, o5_5);
            }
            { const double eb = bi[29];
              o5_5 = fma(eb, g5_6, o5_5);
            }
            { const double eb = bi[30];
              o5_5 = fma(eb, g5_3, o5_5);
            }
            { const double eb = bi[31];
              o5_5 = fma(eb, g5_8, o5_5);
            }
            { const double eb = bi[32];
              o5_5 = fma(eb, g5_16, o5_5);
            }
            { const double eb = bi[33];
              o6_5 = fma(eb, g5_0, o6_5);
            }
            { const double eb = bi[34];
              o6_5 = fma(eb, g5_2, o6_5);
            }
            { const double eb = bi[35];
              o6_5 = fma(eb, g5_6, o6_5);
            }
            { const double eb = bi[36];
              o6_5 = fma(eb, g5_13, o6_5);
            }
            { const double eb = bi[37];
              o7_5 = fma(eb, g5_0, o7_5);
            }
            { const double eb = bi[38];
              o7_5 = fma(eb, g5_1, o7_5);
            }
            { const double eb = bi[39];
              o7_5 = fma(eb, g5_2, o7_5);
            }
            { const double eb = bi[40];
              o7_5 = fma(eb, g5_5, o7_5);
            }
            { const double eb = bi[41];
              o7_5 = fma(eb, g5_6, o7_5);
            }
            { const double eb = bi[42];
              o7_5 = fma(eb, g5_12, o7_5);
            }
            { const double eb = bi[43];
              o8_5 = fma(eb, g5_0, o8_5);
            }
            { const double eb = bi[44];
              o8_5 = fma(eb, g5_1, o8_5);
            }
            { const double eb = bi[45];
              o8_5 = fma(eb, g5_4, o8_5);
            }
            { const double eb = bi[46];
              o9_5 = fma(eb, g5_0, o9_5);
            }
            { const double eb = bi[47];
              o9_5 = fma(eb, g5_1, o9_5);
            }
            { const double eb = bi[48];
              o9_5 = fma(eb, g5_4, o9_5);
            }
            { const double eb = bi[49];
              o9_5 = fma(eb, g5_3, o9_5);
            }
            { const double eb = bi[50];
              o9_5 = fma(eb, g5_7, o9_5);
            }
            { const double eb = bi[51];
              o9_5 = fma(eb, g5_14, o9_5);
            }
            { const double eb = bi[52];
              o10_5 = fma(eb, g5_0, o10_5);
            }
            { const double eb = bi[53];
              o10_5 = fma(eb, g5_1, o10_5);
            }
            { const double eb = bi[54];
              o10_5 = fma(eb, g5_4, o10_5);
            }
            { const double eb = bi[55];
              o10_5 = fma(eb, g5_2, o10_5);
            }
            { const double eb = bi[56];
              o10_5 = fma(eb, g5_5, o10_5);
            }
            { const double eb = bi[57];
              o10_5 = fma(eb, g5_11, o10_5);
            }
            { const double eb = bi[58];
              o11_5 = fma(eb, g5_0, o11_5);
            }
            { const double eb = bi[59];
              o11_5 = fma(eb, g5_1, o11_5);
            }
            { const double eb = bi[60];
              o11_5 = fma(eb, g5_4, o11_5);
            }
            { const double eb = bi[61];
              o11_5 = fma(eb, g5_10, o11_5);
            }
            { const double eb = bi[62];
              o12_5 = fma(eb, g5_0, o12_5);
            }
            { const double eb = bi[63];
              o12_5 = fma(eb, g5_2, o12_5);
            }
            { const double eb = bi[64];
              o12_5 = fma(eb, g5_3, o12_5);
            }
            { const double eb = bi[65];
              o12_5 = fma(eb, g5_8, o12_5);
            }
            { const double eb = bi[66];
              o13_5 = fma(eb, g5_0, o13_5);
            }
            { const double eb = bi[67];
              o13_5 = fma(eb, g5_2, o13_5);
            }
            { const double eb = bi[68];
              o13_5 = fma(eb, g5_3, o13_5);
            }
            { const double eb = bi[69];
              o13_5 = fma(eb, g5_8, o13_5);
            }
            { const double eb = bi[70];
              o13_5 = fma(eb, g5_9, o13_5);
            }
            { const double eb = bi[71];
              o13_5 = fma(eb, g5_18, o13_5);
            }
            { const double eb = bi[72];
              o14_5 = fma(eb, g5_0, o14_5);
            }
            { const double eb = bi[73];
              o14_5 = fma(eb, g5_2, o14_5);
            }
            { const double eb = bi[74];
              o14_5 = fma(eb, g5_6, o14_5);
            }
            { const double eb = bi[75];
              o14_5 = fma(eb, g5_3, o14_5);
            }
            { const double eb = bi[76];
              o14_5 = fma(eb, g5_8, o14_5);
            }
            { const double eb = bi[77];
              o14_5 = fma(eb, g5_16, o14_5);
            }
            { const double eb = bi[78];
              o15_5 = fma(eb, g5_0, o15_5);
            }
            { const double eb = bi[79];
              o15_5 = fma(eb, g5_1, o15_5);
            }
            { const double eb = bi[80];
              o15_5 = fma(eb, g5_2, o15_5);
            }
            { const double eb = bi[81];
              o15_5 = fma(eb, g5_5, o15_5);
            }
            { const double eb = bi[82];
              o15_5 = fma(eb, g5_3, o15_5);
            }
            { const double eb = bi[83];
              o15_5 = fma(eb, g5_7, o15_5);
            }
            { const double eb = bi[84];
              o15_5 = fma(eb, g5_8, o15_5);
            }
            { const double eb = bi[85];
              o15_5 = fma(eb, g5_15, o15_5);
            }
            { const double eb = bi[86];
              o16_5 = fma(eb, g5_0, o16_5);
            }
            { const double eb = bi[87];
              o16_5 = fma(eb, g5_1, o16_5);
            }
            { const double eb = bi[88];
              o16_5 = fma(eb, g5_3, o16_5);
            }
            { const double eb = bi[89];
              o16_5 = fma(eb, g5_7, o16_5);
            }
            { const double eb = bi[90];
              o17_5 = fma(eb, g5_0, o17_5);
            }
            { const double eb = bi[91];
              o17_5 = fma(eb, g5_1, o17_5);
            }
            { const double eb = bi[92];
              o17_5 = fma(eb, g5_3, o17_5);
            }
            { const double eb = bi[93];
              o17_5 = fma(eb, g5_7, o17_5);
            }
            { const double eb = bi[94];
              o17_5 = fma(eb, g5_9, o17_5);
            }
            { const double eb = bi[95];
              o17_5 = fma(eb, g5_17, o17_5);
            }
            { const double eb = bi[96];
              o18_5 = fma(eb, g5_0, o18_5);
            }
            { const double eb = bi[97];
              o18_5 = fma(eb, g5_1, o18_5);
            }
            { const double eb = bi[98];
              o18_5 = fma(eb, g5_2, o18_5);
            }
            { const double eb = bi[99];
              o18_5 = fma(eb, g5_5, o18_5);
            }
            { const double eb = bi[100];
              o18_5 = fma(eb, g5_3, o18_5);
            }
            { const double eb = bi[101];
              o18_5 = fma(eb, g5_7, o18_5);
            }
            { const double eb = bi[102];
              o18_5 = fma(eb, g5_8, o18_5);
            }
            { const double eb = bi[103];
              o18_5 = fma(eb, g5_15, o18_5);
            }
            { const double eb = bi[104];
              o19_5 = fma(eb, g5_0, o19_5);
            }
            { const double eb = bi[105];
              o19_5 = fma(eb, g5_1, o19_5);
            }
            { const double eb = bi[106];
              o19_5 = fma(eb, g5_4, o19_5);
            }
            { const double eb = bi[107];
              o19_5 = fma(eb, g5_3, o19_5);
            }
            { const double eb = bi[108];
              o19_5 = fma(eb, g5_7, o19_5);
            }
            { const double eb = bi[109];
              o19_5 = fma(eb, g5_14, o19_5);
            }
            { const double eb = bi[110];
              o20_5 = fma(eb, g5_0, o20_5);
            }
            { const double eb = bi[111];
              o20_5 = fma(eb, g5_1, o20_5);
            }
            { const double eb = bi[112];
              o20_5 = fma(eb, g5_2, o20_5);
            }
            { const double eb = bi[113];
              o20_5 = fma(eb, g5_5, o20_5);
            }
            { const double eb = bi[114];
              o21_5 = fma(eb, g5_0, o21_5);
            }
            { const double eb = bi[115];
              o21_5 = fma(eb, g5_1, o21_5);
            }
            { const double eb = bi[116];
              o21_5 = fma(eb, g5_2, o21_5);
            }
            { const double eb = bi[117];
              o21_5 = fma(eb, g5_5, o21_5);
            }
            { const double eb = bi[118];
              o21_5 = fma(eb, g5_3, o21_5);
            }
            { const double eb = bi[119];
              o21_5 = fma(eb, g5_7, o21_5);
            }
            { const double eb = bi[120];
              o21_5 = fma(eb, g5_8, o21_5);
            }
            { const double eb = bi[121];
              o21_5 = fma(eb, g5_15, o21_5);
            }
            { const double eb = bi[122];
              o22_5 = fma(eb, g5_0, o22_5);
            }
            { const double eb = bi[123];
              o22_5 = fma(eb, g5_1, o22_5);
            }
            { const double eb = bi[124];
              o22_5 = fma(eb, g5_2, o22_5);
            }
            { const double eb = bi[125];
              o22_5 = fma(eb, g5_5, o22_5);
            }
            { const double eb = bi[126];
              o22_5 = fma(eb, g5_6, o22_5);
            }
            { const double eb = bi[127];
              o22_5 = fma(eb, g5_12, o22_5);
            }
            { const double eb = bi[128];
              o23_5 = fma(eb, g5_0, o23_5);
            }
            { const double eb = bi[129];
              o23_5 = fma(eb, g5_1, o23_5);
            }
            { const double eb = bi[130];
              o23_5 = fma(eb, g5_4, o23_5);
            }
            { const double eb = bi[131];
              o23_5 = fma(eb, g5_2, o23_5);
            }
            { const double eb = bi[132];
              o23_5 = fma(eb, g5_5, o23_5);
            }
            { const double eb = bi[133];
              o23_5 = fma(eb, g5_11, o23_5);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 1);
            o1_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 1);
            o2_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 1);
            o3_5 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 1);
            o4_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 1);
            o5_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 1);
            o6_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 1);
            o7_5 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 1);
            o8_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 1);
            o9_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 1);
            o10_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 1);
            o11_5 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 1);
            o12_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 1);
            o13_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 1);
            o14_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 1);
            o15_5 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 1);
            o16_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 1);
            o17_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 1);
            o18_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 1);
            o19_5 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 1);
            o20_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 1);
            o21_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 1);
            o22_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 1);
            o23_5 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 1);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o1_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o2_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o3_5 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o4_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o5_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o6_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o7_5 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o8_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o9_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o10_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o11_5 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o12_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o13_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o14_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o15_5 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o16_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o17_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o18_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o19_5 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o20_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o21_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o22_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 1)));
            e = fmax(e, fabs(o23_5 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 1)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
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
            const double Bbd0_1 = PB[(fQ + 0) * N + fJ + 1];
            const double Bbd1_1 = PB[(fQ + 1) * N + fJ + 1];
            const double Bbd2_1 = PB[(fQ + 2) * N + fJ + 1];
            const double Bbd3_1 = PB[(fQ + 3) * N + fJ + 1];
            const double Bad0_1 = PB[(fP + 0) * N + fJ + 1];
            const double Bad1_1 = PB[(fP + 1) * N + fJ + 1];
            const double Bad2_1 = PB[(fP + 2) * N + fJ + 1];
            const double Bad3_1 = PB[(fP + 3) * N + fJ + 1];
            const double Bad4_1 = PB[(fP + 4) * N + fJ + 1];
            const double Bad5_1 = PB[(fP + 5) * N + fJ + 1];
            const double Bbc0_1 = PB[(fQ + 0) * N + fI + 1];
            const double Bbc1_1 = PB[(fQ + 1) * N + fI + 1];
            const double Bbc2_1 = PB[(fQ + 2) * N + fI + 1];
            const double Bbc3_1 = PB[(fQ + 3) * N + fI + 1];
            const double Bac0_1 = PB[(fP + 0) * N + fI + 1];
            const double Bac1_1 = PB[(fP + 1) * N + fI + 1];
            const double Bac2_1 = PB[(fP + 2) * N + fI + 1];
            const double Bac3_1 = PB[(fP + 3) * N + fI + 1];
            const double Bac4_1 = PB[(fP + 4) * N + fI + 1];
            const double Bac5_1 = PB[(fP + 5) * N + fI + 1];
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
            atomicAdd(Jacc + (fI + 1) * N + fJ + 1, 2.0 * deg * (o0_5 * ptb0 + o1_5 * ptb1 + o2_5 * ptb2 + o3_5 * ptb3 + o4_5 * ptb4 + o5_5 * ptb5 + o6_5 * ptb6 + o7_5 * ptb7 + o8_5 * ptb8 + o9_5 * ptb9 + o10_5 * ptb10 + o11_5 * ptb11 + o12_5 * ptb12 + o13_5 * ptb13 + o14_5 * ptb14 + o15_5 * ptb15 + o16_5 * ptb16 + o17_5 * ptb17 + o18_5 * ptb18 + o19_5 * ptb19 + o20_5 * ptb20 + o21_5 * ptb21 + o22_5 * ptb22 + o23_5 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_5 * Abd0_1 + o1_5 * Abd1_1 + o2_5 * Abd2_1 + o3_5 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_5 * Aad0_1 + o4_5 * Aad1_1 + o8_5 * Aad2_1 + o12_5 * Aad3_1 + o16_5 * Aad4_1 + o20_5 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_5 * Abc0_1 + o1_5 * Abc1_1 + o2_5 * Abc2_1 + o3_5 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_5 * Aac0_1 + o4_5 * Aac1_1 + o8_5 * Aac2_1 + o12_5 * Aac3_1 + o16_5 * Aac4_1 + o20_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_5 * Aad0_1 + o5_5 * Aad1_1 + o9_5 * Aad2_1 + o13_5 * Aad3_1 + o17_5 * Aad4_1 + o21_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_5 * Aac0_1 + o5_5 * Aac1_1 + o9_5 * Aac2_1 + o13_5 * Aac3_1 + o17_5 * Aac4_1 + o21_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_5 * Aad0_1 + o6_5 * Aad1_1 + o10_5 * Aad2_1 + o14_5 * Aad3_1 + o18_5 * Aad4_1 + o22_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_5 * Aac0_1 + o6_5 * Aac1_1 + o10_5 * Aac2_1 + o14_5 * Aac3_1 + o18_5 * Aac4_1 + o22_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_5 * Aad0_1 + o7_5 * Aad1_1 + o11_5 * Aad2_1 + o15_5 * Aad3_1 + o19_5 * Aad4_1 + o23_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_5 * Aac0_1 + o7_5 * Aac1_1 + o11_5 * Aac2_1 + o15_5 * Aac3_1 + o19_5 * Aac4_1 + o23_5 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_5 * Abd0_1 + o5_5 * Abd1_1 + o6_5 * Abd2_1 + o7_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_5 * Abc0_1 + o5_5 * Abc1_1 + o6_5 * Abc2_1 + o7_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_5 * Abd0_1 + o9_5 * Abd1_1 + o10_5 * Abd2_1 + o11_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_5 * Abc0_1 + o9_5 * Abc1_1 + o10_5 * Abc2_1 + o11_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_5 * Abd0_1 + o13_5 * Abd1_1 + o14_5 * Abd2_1 + o15_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_5 * Abc0_1 + o13_5 * Abc1_1 + o14_5 * Abc2_1 + o15_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_5 * Abd0_1 + o17_5 * Abd1_1 + o18_5 * Abd2_1 + o19_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_5 * Abc0_1 + o17_5 * Abc1_1 + o18_5 * Abc2_1 + o19_5 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_5 * Abd0_1 + o21_5 * Abd1_1 + o22_5 * Abd2_1 + o23_5 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_5 * Abc0_1 + o21_5 * Abc1_1 + o22_5 * Abc2_1 + o23_5 * Abc3_1));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_5 * Bbd0_1 + o1_5 * Bbd1_1 + o2_5 * Bbd2_1 + o3_5 * Bbd3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_5 * Bad0_1 + o4_5 * Bad1_1 + o8_5 * Bad2_1 + o12_5 * Bad3_1 + o16_5 * Bad4_1 + o20_5 * Bad5_1));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 1, deg * (o0_5 * Bbc0_1 + o1_5 * Bbc1_1 + o2_5 * Bbc2_1 + o3_5 * Bbc3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 1, deg * (o0_5 * Bac0_1 + o4_5 * Bac1_1 + o8_5 * Bac2_1 + o12_5 * Bac3_1 + o16_5 * Bac4_1 + o20_5 * Bac5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 1, deg * (o1_5 * Bad0_1 + o5_5 * Bad1_1 + o9_5 * Bad2_1 + o13_5 * Bad3_1 + o17_5 * Bad4_1 + o21_5 * Bad5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 1, deg * (o1_5 * Bac0_1 + o5_5 * Bac1_1 + o9_5 * Bac2_1 + o13_5 * Bac3_1 + o17_5 * Bac4_1 + o21_5 * Bac5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 1, deg * (o2_5 * Bad0_1 + o6_5 * Bad1_1 + o10_5 * Bad2_1 + o14_5 * Bad3_1 + o18_5 * Bad4_1 + o22_5 * Bad5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 1, deg * (o2_5 * Bac0_1 + o6_5 * Bac1_1 + o10_5 * Bac2_1 + o14_5 * Bac3_1 + o18_5 * Bac4_1 + o22_5 * Bac5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 1, deg * (o3_5 * Bad0_1 + o7_5 * Bad1_1 + o11_5 * Bad2_1 + o15_5 * Bad3_1 + o19_5 * Bad4_1 + o23_5 * Bad5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 1, deg * (o3_5 * Bac0_1 + o7_5 * Bac1_1 + o11_5 * Bac2_1 + o15_5 * Bac3_1 + o19_5 * Bac4_1 + o23_5 * Bac5_1));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o4_5 * Bbd0_1 + o5_5 * Bbd1_1 + o6_5 * Bbd2_1 + o7_5 * Bbd3_1));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 1, deg * (o4_5 * Bbc0_1 + o5_5 * Bbc1_1 + o6_5 * Bbc2_1 + o7_5 * Bbc3_1));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o8_5 * Bbd0_1 + o9_5 * Bbd1_1 + o10_5 * Bbd2_1 + o11_5 * Bbd3_1));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 1, deg * (o8_5 * Bbc0_1 + o9_5 * Bbc1_1 + o10_5 * Bbc2_1 + o11_5 * Bbc3_1));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o12_5 * Bbd0_1 + o13_5 * Bbd1_1 + o14_5 * Bbd2_1 + o15_5 * Bbd3_1));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 1, deg * (o12_5 * Bbc0_1 + o13_5 * Bbc1_1 + o14_5 * Bbc2_1 + o15_5 * Bbc3_1));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o16_5 * Bbd0_1 + o17_5 * Bbd1_1 + o18_5 * Bbd2_1 + o19_5 * Bbd3_1));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 1, deg * (o16_5 * Bbc0_1 + o17_5 * Bbc1_1 + o18_5 * Bbc2_1 + o19_5 * Bbc3_1));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o20_5 * Bbd0_1 + o21_5 * Bbd1_1 + o22_5 * Bbd2_1 + o23_5 * Bbd3_1));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 1, deg * (o20_5 * Bbc0_1 + o21_5 * Bbc1_1 + o22_5 * Bbc2_1 + o23_5 * Bbc3_1));
          }
        } break;
        case 6: {  // ket functions [6]
          double o0_6 = 0;
          double o1_6 = 0;
          double o2_6 = 0;
          double o3_6 = 0;
          double o4_6 = 0;
          double o5_6 = 0;
          double o6_6 = 0;
          double o7_6 = 0;
          double o8_6 = 0;
          double o9_6 = 0;
          double o10_6 = 0;
          double o11_6 = 0;
          double o12_6 = 0;
          double o13_6 = 0;
          double o14_6 = 0;
          double o15_6 = 0;
          double o16_6 = 0;
          double o17_6 = 0;
          double o18_6 = 0;
          double o19_6 = 0;
          double o20_6 = 0;
          double o21_6 = 0;
          double o22_6 = 0;
          double o23_6 = 0;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek6_0 = kj[17 * kS];
              const double ek6_1 = -kj[18 * kS];
              const double ek6_2 = -kj[19 * kS];
              const double ek6_3 = kj[20 * kS];
              g6_0 = fma(ek6_0, b0, g6_0);
              const double r0_0_0_1 = Z * b1;
              g6_1 = fma(ek6_0, r0_0_0_1, g6_1);
              const double r0_0_1_0 = Y * b1;
              g6_2 = fma(ek6_0, r0_0_1_0, g6_2);
              g6_0 = fma(ek6_1, r0_0_1_0, g6_0);
              const double r0_1_0_0 = X * b1;
              g6_3 = fma(ek6_0, r0_1_0_0, g6_3);
              g6_0 = fma(ek6_2, r0_1_0_0, g6_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g6_4 = fma(ek6_0, r0_0_0_2, g6_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g6_5 = fma(ek6_0, r0_0_1_1, g6_5);
              g6_1 = fma(ek6_1, r0_0_1_1, g6_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g6_6 = fma(ek6_0, r0_0_2_0, g6_6);
              g6_2 = fma(ek6_1, r0_0_2_0, g6_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g6_7 = fma(ek6_0, r0_1_0_1, g6_7);
              g6_1 = fma(ek6_2, r0_1_0_1, g6_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g6_8 = fma(ek6_0, r0_1_1_0, g6_8);
              g6_3 = fma(ek6_1, r0_1_1_0, g6_3);
              g6_2 = fma(ek6_2, r0_1_1_0, g6_2);
              g6_0 = fma(ek6_3, r0_1_1_0, g6_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g6_9 = fma(ek6_0, r0_2_0_0, g6_9);
              g6_3 = fma(ek6_2, r0_2_0_0, g6_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g6_10 = fma(ek6_0, r0_0_0_3, g6_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g6_11 = fma(ek6_0, r0_0_1_2, g6_11);
              g6_4 = fma(ek6_1, r0_0_1_2, g6_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g6_12 = fma(ek6_0, r0_0_2_1, g6_12);
              g6_5 = fma(ek6_1, r0_0_2_1, g6_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g6_13 = fma(ek6_0, r0_0_3_0, g6_13);
              g6_6 = fma(ek6_1, r0_0_3_0, g6_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g6_14 = fma(ek6_0, r0_1_0_2, g6_14);
              g6_4 = fma(ek6_2, r0_1_0_2, g6_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g6_15 = fma(ek6_0, r0_1_1_1, g6_15);
              g6_7 = fma(ek6_1, r0_1_1_1, g6_7);
              g6_5 = fma(ek6_2, r0_1_1_1, g6_5);
              g6_1 = fma(ek6_3, r0_1_1_1, g6_1);
              const double r0_1_2_0 = X * r1_0_2_0;
              g6_16 = fma(ek6_0, r0_1_2_0, g6_16);
              g6_8 = fma(ek6_1, r0_1_2_0, g6_8);
              g6_6 = fma(ek6_2, r0_1_2_0, g6_6);
              g6_2 = fma(ek6_3, r0_1_2_0, g6_2);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g6_17 = fma(ek6_0, r0_2_0_1, g6_17);
              g6_7 = fma(ek6_2, r0_2_0_1, g6_7);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g6_18 = fma(ek6_0, r0_2_1_0, g6_18);
              g6_9 = fma(ek6_1, r0_2_1_0, g6_9);
              g6_8 = fma(ek6_2, r0_2_1_0, g6_8);
              g6_3 = fma(ek6_3, r0_2_1_0, g6_3);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g6_19 = fma(ek6_0, r0_3_0_0, g6_19);
              g6_9 = fma(ek6_2, r0_3_0_0, g6_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g6_10 = fma(ek6_1, r0_0_1_3, g6_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g6_11 = fma(ek6_1, r0_0_2_2, g6_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g6_12 = fma(ek6_1, r0_0_3_1, g6_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g6_13 = fma(ek6_1, r0_0_4_0, g6_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g6_10 = fma(ek6_2, r0_1_0_3, g6_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g6_14 = fma(ek6_1, r0_1_1_2, g6_14);
              g6_11 = fma(ek6_2, r0_1_1_2, g6_11);
              g6_4 = fma(ek6_3, r0_1_1_2, g6_4);
              const double r0_1_2_1 = X * r1_0_2_1;
              g6_15 = fma(ek6_1, r0_1_2_1, g6_15);
              g6_12 = fma(ek6_2, r0_1_2_1, g6_12);
              g6_5 = fma(ek6_3, r0_1_2_1, g6_5);
              const double r0_1_3_0 = X * r1_0_3_0;
              g6_16 = fma(ek6_1, r0_1_3_0, g6_16);
              g6_13 = fma(ek6_2, r0_1_3_0, g6_13);
              g6_6 = fma(ek6_3, r0_1_3_0, g6_6);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g6_14 = fma(ek6_2, r0_2_0_2, g6_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g6_17 = fma(ek6_1, r0_2_1_1, g6_17);
              g6_15 = fma(ek6_2, r0_2_1_1, g6_15);
              g6_7 = fma(ek6_3, r0_2_1_1, g6_7);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g6_18 = fma(ek6_1, r0_2_2_0, g6_18);
              g6_16 = fma(ek6_2, r0_2_2_0, g6_16);
              g6_8 = fma(ek6_3, r0_2_2_0, g6_8);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g6_17 = fma(ek6_2, r0_3_0_1, g6_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g6_19 = fma(ek6_1, r0_3_1_0, g6_19);
              g6_18 = fma(ek6_2, r0_3_1_0, g6_18);
              g6_9 = fma(ek6_3, r0_3_1_0, g6_9);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g6_19 = fma(ek6_2, r0_4_0_0, g6_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g6_10 = fma(ek6_3, r0_1_1_3, g6_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g6_11 = fma(ek6_3, r0_1_2_2, g6_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g6_12 = fma(ek6_3, r0_1_3_1, g6_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g6_13 = fma(ek6_3, r0_1_4_0, g6_13);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g6_14 = fma(ek6_3, r0_2_1_2, g6_14);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g6_15 = fma(ek6_3, r0_2_2_1, g6_15);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g6_16 = fma(ek6_3, r0_2_3_0, g6_16);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g6_17 = fma(ek6_3, r0_3_1_1, g6_17);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g6_18 = fma(ek6_3, r0_3_2_0, g6_18);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g6_19 = fma(ek6_3, r0_4_1_0, g6_19);
            }
            { const double eb = bi[5];
              o0_6 = fma(eb, g6_0, o0_6);
            }
            { const double eb = bi[6];
              o0_6 = fma(eb, g6_3, o0_6);
            }
            { const double eb = bi[7];
              o0_6 = fma(eb, g6_9, o0_6);
            }
            { const double eb = bi[8];
              o1_6 = fma(eb, g6_0, o1_6);
            }
            { const double eb = bi[9];
              o1_6 = fma(eb, g6_3, o1_6);
            }
            { const double eb = bi[10];
              o1_6 = fma(eb, g6_9, o1_6);
            }
            { const double eb = bi[11];
              o1_6 = fma(eb, g6_19, o1_6);
            }
            { const double eb = bi[12];
              o2_6 = fma(eb, g6_0, o2_6);
            }
            { const double eb = bi[13];
              o2_6 = fma(eb, g6_2, o2_6);
            }
            { const double eb = bi[14];
              o2_6 = fma(eb, g6_3, o2_6);
            }
            { const double eb = bi[15];
              o2_6 = fma(eb, g6_8, o2_6);
            }
            { const double eb = bi[16];
              o2_6 = fma(eb, g6_9, o2_6);
            }
            { const double eb = bi[17];
              o2_6 = fma(eb, g6_18, o2_6);
            }
            { const double eb = bi[18];
              o3_6 = fma(eb, g6_0, o3_6);
            }
            { const double eb = bi[19];
              o3_6 = fma(eb, g6_1, o3_6);
            }
            { const double eb = bi[20];
              o3_6 = fma(eb, g6_3, o3_6);
            }
            { const double eb = bi[21];
              o3_6 = fma(eb, g6_7, o3_6);
            }
            { const double eb = bi[22];
              o3_6 = fma(eb, g6_9, o3_6);
            }
            { const double eb = bi[23];
              o3_6 = fma(eb, g6_17, o3_6);
            }
            { const double eb = bi[24];
              o4_6 = fma(eb, g6_0, o4_6);
            }
            { const double eb = bi[25];
              o4_6 = fma(eb, g6_2, o4_6);
            }
            { const double eb = bi[26];
              o4_6 = fma(eb, g6_6, o4_6);
            }
            { const double eb = bi[27];
              o5_6 = fma(eb, g6_0, o5_6);
            }
            { const double eb = bi[28];
              o5_6 = fma(eb, g6_2, o5_6);
            }
            { const double eb = bi[29];
              o5_6 = fma(eb, g6_6, o5_6);
            }
            { const double eb = bi[30];
              o5_6 = fma(eb, g6_3, o5_6);
            }
            { const double eb = bi[31];
              o5_6 = fma(eb, g6_8, o5_6);
            }
            { const double eb = bi[32];
              o5_6 = fma(eb, g6_16, o5_6);
            }
            { const double eb = bi[33];
              o6_6 = fma(eb, g6_0, o6_6);
            }
            { const double eb = bi[34];
              o6_6 = fma(eb, g6_2, o6_6);
            }
            { const double eb = bi[35];
              o6_6 = fma(eb, g6_6, o6_6);
            }
            { const double eb = bi[36];
              o6_6 = fma(eb, g6_13, o6_6);
            }
            { const double eb = bi[37];
              o7_6 = fma(eb, g6_0, o7_6);
            }
            { const double eb = bi[38];
              o7_6 = fma(eb, g6_1, o7_6);
            }
            { const double eb = bi[39];
              o7_6 = fma(eb, g6_2, o7_6);
            }
            { const double eb = bi[40];
              o7_6 = fma(eb, g6_5, o7_6);
            }
            { const double eb = bi[41];
              o7_6 = fma(eb, g6_6, o7_6);
            }
            { const double eb = bi[42];
              o7_6 = fma(eb, g6_12, o7_6);
            }
            { const double eb = bi[43];
              o8_6 = fma(eb, g6_0, o8_6);
            }
            { const double eb = bi[44];
              o8_6 = fma(eb, g6_1, o8_6);
            }
            { const double eb = bi[45];
              o8_6 = fma(eb, g6_4, o8_6);
            }
            { const double eb = bi[46];
              o9_6 = fma(eb, g6_0, o9_6);
            }
            { const double eb = bi[47];
              o9_6 = fma(eb, g6_1, o9_6);
            }
            { const double eb = bi[48];
              o9_6 = fma(eb, g6_4, o9_6);
            }
            { const double eb = bi[49];
              o9_6 = fma(eb, g6_3, o9_6);
            }
            { const double eb = bi[50];
              o9_6 = fma(eb, g6_7, o9_6);
            }
            { const double eb = bi[51];
              o9_6 = fma(eb, g6_14, o9_6);
            }
            { const double eb = bi[52];
              o10_6 = fma(eb, g6_0, o10_6);
            }
            { const double eb = bi[53];
              o10_6 = fma(eb, g6_1, o10_6);
            }
            { const double eb = bi[54];
              o10_6 = fma(eb, g6_4, o10_6);
            }
            { const double eb = bi[55];
              o10_6 = fma(eb, g6_2, o10_6);
            }
            { const double eb = bi[56];
              o10_6 = fma(eb, g6_5, o10_6);
            }
            { const double eb = bi[57];
              o10_6 = fma(eb, g6_11, o10_6);
            }
            { const double eb = bi[58];
              o11_6 = fma(eb, g6_0, o11_6);
            }
            { const double eb = bi[59];
              o11_6 = fma(eb, g6_1, o11_6);
            }
            { const double eb = bi[60];
              o11_6 = fma(eb, g6_4, o11_6);
            }
            { const double eb = bi[61];
              o11_6 = fma(eb, g6_10, o11_6);
            }
            { const double eb = bi[62];
              o12_6 = fma(eb, g6_0, o12_6);
            }
            { const double eb = bi[63];
              o12_6 = fma(eb, g6_2, o12_6);
            }
            { const double eb = bi[64];
              o12_6 = fma(eb, g6_3, o12_6);
            }
            { const double eb = bi[65];
              o12_6 = fma(eb, g6_8, o12_6);
            }
            { const double eb = bi[66];
              o13_6 = fma(eb, g6_0, o13_6);
            }
            { const double eb = bi[67];
              o13_6 = fma(eb, g6_2, o13_6);
            }
            { const double eb = bi[68];
              o13_6 = fma(eb, g6_3, o13_6);
            }
            { const double eb = bi[69];
              o13_6 = fma(eb, g6_8, o13_6);
            }
            { const double eb = bi[70];
              o13_6 = fma(eb, g6_9, o13_6);
            }
            { const double eb = bi[71];
              o13_6 = fma(eb, g6_18, o13_6);
            }
            { const double eb = bi[72];
              o14_6 = fma(eb, g6_0, o14_6);
            }
            { const double eb = bi[73];
              o14_6 = fma(eb, g6_2, o14_6);
            }
            { const double eb = bi[74];
              o14_6 = fma(eb, g6_6, o14_6);
            }
            { const double eb = bi[75];
              o14_6 = fma(eb, g6_3, o14_6);
            }
            { const double eb = bi[76];
              o14_6 = fma(eb, g6_8, o14_6);
            }
            { const double eb = bi[77];
              o14_6 = fma(eb, g6_16, o14_6);
            }
            { const double eb = bi[78];
              o15_6 = fma(eb, g6_0, o15_6);
            }
            { const double eb = bi[79];
              o15_6 = fma(eb, g6_1, o15_6);
            }
            { const double eb = bi[80];
              o15_6 = fma(eb, g6_2, o15_6);
            }
            { const double eb = bi[81];
              o15_6 = fma(eb, g6_5, o15_6);
            }
            { const double eb = bi[82];
              o15_6 = fma(eb, g6_3, o15_6);
            }
            { const double eb = bi[83];
              o15_6 = fma(eb, g6_7, o15_6);
            }
            { const double eb = bi[84];
              o15_6 = fma(eb, g6_8, o15_6);
            }
            { const double eb = bi[85];
              o15_6 = fma(eb, g6_15, o15_6);
            }
            { const double eb = bi[86];
              o16_6 = fma(eb, g6_0, o16_6);
            }
            { const double eb = bi[87];
              o16_6 = fma(eb, g6_1, o16_6);
            }
            { const double eb = bi[88];
              o16_6 = fma(eb, g6_3, o16_6);
            }
            { const double eb = bi[89];
              o16_6 = fma(eb, g6_7, o16_6);
            }
            { const double eb = bi[90];
              o17_6 = fma(eb, g6_0, o17_6);
            }
            { const double eb = bi[91];
              o17_6 = fma(eb, g6_1, o17_6);
            }
            { const double eb = bi[92];
              o17_6 = fma(eb, g6_3, o17_6);
            }
            { const double eb = bi[93];
              o17_6 = fma(eb, g6_7, o17_6);
            }
            { const double eb = bi[94];
              o17_6 = fma(eb, g6_9, o17_6);
            }
            { const double eb = bi[95];
              o17_6 = fma(eb, g6_17, o17_6);
            }
            { const double eb = bi[96];
              o18_6 = fma(eb, g6_0, o18_6);
            }
            { const double eb = bi[97];
              o18_6 = fma(eb, g6_1, o18_6);
            }
            { const double eb = bi[98];
              o18_6 = fma(eb, g6_2, o18_6);
            }
            { const double eb = bi[99];
              o18_6 = fma(eb, g6_5, o18_6);
            }
            { const double eb = bi[100];
              o18_6 = fma(eb, g6_3, o18_6);
            }
            { const double eb = bi[101];
              o18_6 = fma(eb, g6_7, o18_6);
            }
            { const double eb = bi[102];
              o18_6 = fma(eb, g6_8, o18_6);
            }
            { const double eb = bi[103];
              o18_6 = fma(eb, g6_15, o18_6);
            }
            { const double eb = bi[104];
              o19_6 = fma(eb, g6_0, o19_6);
            }
            { const double eb = bi[105];
              o19_6 = fma(eb, g6_1, o19_6);
            }
            { const double eb = bi[106];
              o19_6 = fma(eb, g6_4, o19_6);
            }
            { const double eb = bi[107];
              o19_6 = fma(eb, g6_3, o19_6);
            }
            { const double eb = bi[108];
              o19_6 = fma(eb, g6_7, o19_6);
            }
            { const double eb = bi[109];
              o19_6 = fma(eb, g6_14, o19_6);
            }
            { const double eb = bi[110];
              o20_6 = fma(eb, g6_0, o20_6);
            }
            { const double eb = bi[111];
              o20_6 = fma(eb, g6_1, o20_6);
            }
            { const double eb = bi[112];
              o20_6 = fma(eb, g6_2, o20_6);
            }
            { const double eb = bi[113];
              o20_6 = fma(eb, g6_5, o20_6);
            }
            { const double eb = bi[114];
              o21_6 = fma(eb, g6_0, o21_6);
            }
            { const double eb = bi[115];
              o21_6 = fma(eb, g6_1, o21_6);
            }
            { const double eb = bi[116];
              o21_6 = fma(eb, g6_2, o21_6);
            }
            { const double eb = bi[117];
              o21_6 = fma(eb, g6_5, o21_6);
            }
            { const double eb = bi[118];
              o21_6 = fma(eb, g6_3, o21_6);
            }
            { const double eb = bi[119];
              o21_6 = fma(eb, g6_7, o21_6);
            }
            { const double eb = bi[120];
              o21_6 = fma(eb, g6_8, o21_6);
            }
            { const double eb = bi[121];
              o21_6 = fma(eb, g6_15, o21_6);
            }
            { const double eb = bi[122];
              o22_6 = fma(eb, g6_0, o22_6);
            }
            { const double eb = bi[123];
              o22_6 = fma(eb, g6_1, o22_6);
            }
            { const double eb = bi[124];
              o22_6 = fma(eb, g6_2, o22_6);
            }
            { const double eb = bi[125];
              o22_6 = fma(eb, g6_5, o22_6);
            }
            { const double eb = bi[126];
              o22_6 = fma(eb, g6_6, o22_6);
            }
            { const double eb = bi[127];
              o22_6 = fma(eb, g6_12, o22_6);
            }
            { const double eb = bi[128];
              o23_6 = fma(eb, g6_0, o23_6);
            }
            { const double eb = bi[129];
              o23_6 = fma(eb, g6_1, o23_6);
            }
            { const double eb = bi[130];
              o23_6 = fma(eb, g6_4, o23_6);
            }
            { const double eb = bi[131];
              o23_6 = fma(eb, g6_2, o23_6);
            }
            { const double eb = bi[132];
              o23_6 = fma(eb, g6_5, o23_6);
            }
            { const double eb = bi[133];
              o23_6 = fma(eb, g6_11, o23_6);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_6 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 2);
            o1_6 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 2);
            o2_6 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 2);
            o3_6 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 2);
            o4_6 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 2);
            o5_6 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 2);
            o6_6 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 2);
            o7_6 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 2);
            o8_6 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 2);
            o9_6 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 2);
            o10_6 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 2);
            o11_6 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 2);
            o12_6 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 2);
            o13_6 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 2);
            o14_6 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 2);
            o15_6 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 2);
            o16_6 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 2);
            o17_6 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 2);
            o18_6 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 2);
            o19_6 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 2);
            o20_6 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 2);
            o21_6 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 2);
            o22_6 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 2);
            o23_6 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 2);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_6 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o1_6 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o2_6 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o3_6 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o4_6 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o5_6 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o6_6 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o7_6 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o8_6 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o9_6 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o10_6 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o11_6 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o12_6 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o13_6 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o14_6 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o15_6 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o16_6 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o17_6 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o18_6 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o19_6 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o20_6 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o21_6 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o22_6 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 2)));
            e = fmax(e, fabs(o23_6 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 2)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk6 = PT[(fI + 1) * N + fJ + 2];
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
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
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
            const double Bbd0_2 = PB[(fQ + 0) * N + fJ + 2];
            const double Bbd1_2 = PB[(fQ + 1) * N + fJ + 2];
            const double Bbd2_2 = PB[(fQ + 2) * N + fJ + 2];
            const double Bbd3_2 = PB[(fQ + 3) * N + fJ + 2];
            const double Bad0_2 = PB[(fP + 0) * N + fJ + 2];
            const double Bad1_2 = PB[(fP + 1) * N + fJ + 2];
            const double Bad2_2 = PB[(fP + 2) * N + fJ + 2];
            const double Bad3_2 = PB[(fP + 3) * N + fJ + 2];
            const double Bad4_2 = PB[(fP + 4) * N + fJ + 2];
            const double Bad5_2 = PB[(fP + 5) * N + fJ + 2];
            const double Bbc0_1 = PB[(fQ + 0) * N + fI + 1];
            const double Bbc1_1 = PB[(fQ + 1) * N + fI + 1];
            const double Bbc2_1 = PB[(fQ + 2) * N + fI + 1];
            const double Bbc3_1 = PB[(fQ + 3) * N + fI + 1];
            const double Bac0_1 = PB[(fP + 0) * N + fI + 1];
            const double Bac1_1 = PB[(fP + 1) * N + fI + 1];
            const double Bac2_1 = PB[(fP + 2) * N + fI + 1];
            const double Bac3_1 = PB[(fP + 3) * N + fI + 1];
            const double Bac4_1 = PB[(fP + 4) * N + fI + 1];
            const double Bac5_1 = PB[(fP + 5) * N + fI + 1];
            jab0 += o0_6 * ptk6;
            jab1 += o1_6 * ptk6;
            jab2 += o2_6 * ptk6;
            jab3 += o3_6 * ptk6;
            jab4 += o4_6 * ptk6;
            jab5 += o5_6 * ptk6;
            jab6 += o6_6 * ptk6;
            jab7 += o7_6 * ptk6;
            jab8 += o8_6 * ptk6;
            jab9 += o9_6 * ptk6;
            jab10 += o10_6 * ptk6;
            jab11 += o11_6 * ptk6;
            jab12 += o12_6 * ptk6;
            jab13 += o13_6 * ptk6;
            jab14 += o14_6 * ptk6;
            jab15 += o15_6 * ptk6;
            jab16 += o16_6 * ptk6;
            jab17 += o17_6 * ptk6;
            jab18 += o18_6 * ptk6;
            jab19 += o19_6 * ptk6;
            jab20 += o20_6 * ptk6;
            jab21 += o21_6 * ptk6;
            jab22 += o22_6 * ptk6;
            jab23 += o23_6 * ptk6;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 2, 2.0 * deg * (o0_6 * ptb0 + o1_6 * ptb1 + o2_6 * ptb2 + o3_6 * ptb3 + o4_6 * ptb4 + o5_6 * ptb5 + o6_6 * ptb6 + o7_6 * ptb7 + o8_6 * ptb8 + o9_6 * ptb9 + o10_6 * ptb10 + o11_6 * ptb11 + o12_6 * ptb12 + o13_6 * ptb13 + o14_6 * ptb14 + o15_6 * ptb15 + o16_6 * ptb16 + o17_6 * ptb17 + o18_6 * ptb18 + o19_6 * ptb19 + o20_6 * ptb20 + o21_6 * ptb21 + o22_6 * ptb22 + o23_6 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_6 * Abd0_2 + o1_6 * Abd1_2 + o2_6 * Abd2_2 + o3_6 * Abd3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_6 * Aad0_2 + o4_6 * Aad1_2 + o8_6 * Aad2_2 + o12_6 * Aad3_2 + o16_6 * Aad4_2 + o20_6 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_6 * Abc0_1 + o1_6 * Abc1_1 + o2_6 * Abc2_1 + o3_6 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_6 * Aac0_1 + o4_6 * Aac1_1 + o8_6 * Aac2_1 + o12_6 * Aac3_1 + o16_6 * Aac4_1 + o20_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_6 * Aad0_2 + o5_6 * Aad1_2 + o9_6 * Aad2_2 + o13_6 * Aad3_2 + o17_6 * Aad4_2 + o21_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_6 * Aac0_1 + o5_6 * Aac1_1 + o9_6 * Aac2_1 + o13_6 * Aac3_1 + o17_6 * Aac4_1 + o21_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_6 * Aad0_2 + o6_6 * Aad1_2 + o10_6 * Aad2_2 + o14_6 * Aad3_2 + o18_6 * Aad4_2 + o22_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_6 * Aac0_1 + o6_6 * Aac1_1 + o10_6 * Aac2_1 + o14_6 * Aac3_1 + o18_6 * Aac4_1 + o22_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_6 * Aad0_2 + o7_6 * Aad1_2 + o11_6 * Aad2_2 + o15_6 * Aad3_2 + o19_6 * Aad4_2 + o23_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_6 * Aac0_1 + o7_6 * Aac1_1 + o11_6 * Aac2_1 + o15_6 * Aac3_1 + o19_6 * Aac4_1 + o23_6 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_6 * Abd0_2 + o5_6 * Abd1_2 + o6_6 * Abd2_2 + o7_6 * Abd3_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_6 * Abc0_1 + o5_6 * Abc1_1 + o6_6 * Abc2_1 + o7_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_6 * Abd0_2 + o9_6 * Abd1_2 + o10_6 * Abd2_2 + o11_6 * Abd3_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_6 * Abc0_1 + o9_6 * Abc1_1 + o10_6 * Abc2_1 + o11_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_6 * Abd0_2 + o13_6 * Abd1_2 + o14_6 * Abd2_2 + o15_6 * Abd3_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_6 * Abc0_1 + o13_6 * Abc1_1 + o14_6 * Abc2_1 + o15_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_6 * Abd0_2 + o17_6 * Abd1_2 + o18_6 * Abd2_2 + o19_6 * Abd3_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_6 * Abc0_1 + o17_6 * Abc1_1 + o18_6 * Abc2_1 + o19_6 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_6 * Abd0_2 + o21_6 * Abd1_2 + o22_6 * Abd2_2 + o23_6 * Abd3_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_6 * Abc0_1 + o21_6 * Abc1_1 + o22_6 * Abc2_1 + o23_6 * Abc3_1));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_6 * Bbd0_2 + o1_6 * Bbd1_2 + o2_6 * Bbd2_2 + o3_6 * Bbd3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_6 * Bad0_2 + o4_6 * Bad1_2 + o8_6 * Bad2_2 + o12_6 * Bad3_2 + o16_6 * Bad4_2 + o20_6 * Bad5_2));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 2, deg * (o0_6 * Bbc0_1 + o1_6 * Bbc1_1 + o2_6 * Bbc2_1 + o3_6 * Bbc3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 2, deg * (o0_6 * Bac0_1 + o4_6 * Bac1_1 + o8_6 * Bac2_1 + o12_6 * Bac3_1 + o16_6 * Bac4_1 + o20_6 * Bac5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 1, deg * (o1_6 * Bad0_2 + o5_6 * Bad1_2 + o9_6 * Bad2_2 + o13_6 * Bad3_2 + o17_6 * Bad4_2 + o21_6 * Bad5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 2, deg * (o1_6 * Bac0_1 + o5_6 * Bac1_1 + o9_6 * Bac2_1 + o13_6 * Bac3_1 + o17_6 * Bac4_1 + o21_6 * Bac5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 1, deg * (o2_6 * Bad0_2 + o6_6 * Bad1_2 + o10_6 * Bad2_2 + o14_6 * Bad3_2 + o18_6 * Bad4_2 + o22_6 * Bad5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 2, deg * (o2_6 * Bac0_1 + o6_6 * Bac1_1 + o10_6 * Bac2_1 + o14_6 * Bac3_1 + o18_6 * Bac4_1 + o22_6 * Bac5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 1, deg * (o3_6 * Bad0_2 + o7_6 * Bad1_2 + o11_6 * Bad2_2 + o15_6 * Bad3_2 + o19_6 * Bad4_2 + o23_6 * Bad5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 2, deg * (o3_6 * Bac0_1 + o7_6 * Bac1_1 + o11_6 * Bac2_1 + o15_6 * Bac3_1 + o19_6 * Bac4_1 + o23_6 * Bac5_1));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o4_6 * Bbd0_2 + o5_6 * Bbd1_2 + o6_6 * Bbd2_2 + o7_6 * Bbd3_2));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 2, deg * (o4_6 * Bbc0_1 + o5_6 * Bbc1_1 + o6_6 * Bbc2_1 + o7_6 * Bbc3_1));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o8_6 * Bbd0_2 + o9_6 * Bbd1_2 + o10_6 * Bbd2_2 + o11_6 * Bbd3_2));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 2, deg * (o8_6 * Bbc0_1 + o9_6 * Bbc1_1 + o10_6 * Bbc2_1 + o11_6 * Bbc3_1));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o12_6 * Bbd0_2 + o13_6 * Bbd1_2 + o14_6 * Bbd2_2 + o15_6 * Bbd3_2));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 2, deg * (o12_6 * Bbc0_1 + o13_6 * Bbc1_1 + o14_6 * Bbc2_1 + o15_6 * Bbc3_1));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o16_6 * Bbd0_2 + o17_6 * Bbd1_2 + o18_6 * Bbd2_2 + o19_6 * Bbd3_2));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 2, deg * (o16_6 * Bbc0_1 + o17_6 * Bbc1_1 + o18_6 * Bbc2_1 + o19_6 * Bbc3_1));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o20_6 * Bbd0_2 + o21_6 * Bbd1_2 + o22_6 * Bbd2_2 + o23_6 * Bbd3_2));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 2, deg * (o20_6 * Bbc0_1 + o21_6 * Bbc1_1 + o22_6 * Bbc2_1 + o23_6 * Bbc3_1));
          }
        } break;
        case 7: {  // ket functions [7]
          double o0_7 = 0;
          double o1_7 = 0;
          double o2_7 = 0;
          double o3_7 = 0;
          double o4_7 = 0;
          double o5_7 = 0;
          double o6_7 = 0;
          double o7_7 = 0;
          double o8_7 = 0;
          double o9_7 = 0;
          double o10_7 = 0;
          double o11_7 = 0;
          double o12_7 = 0;
          double o13_7 = 0;
          double o14_7 = 0;
          double o15_7 = 0;
          double o16_7 = 0;
          double o17_7 = 0;
          double o18_7 = 0;
          double o19_7 = 0;
          double o20_7 = 0;
          double o21_7 = 0;
          double o22_7 = 0;
          double o23_7 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek7_0 = kj[21 * kS];
              const double ek7_1 = -kj[22 * kS];
              const double ek7_2 = -kj[23 * kS];
              const double ek7_3 = kj[24 * kS];
              g7_0 = fma(ek7_0, b0, g7_0);
              const double r0_0_0_1 = Z * b1;
              g7_1 = fma(ek7_0, r0_0_0_1, g7_1);
              g7_0 = fma(ek7_1, r0_0_0_1, g7_0);
              const double r0_0_1_0 = Y * b1;
              g7_2 = fma(ek7_0, r0_0_1_0, g7_2);
              const double r0_1_0_0 = X * b1;
              g7_3 = fma(ek7_0, r0_1_0_0, g7_3);
              g7_0 = fma(ek7_2, r0_1_0_0, g7_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g7_4 = fma(ek7_0, r0_0_0_2, g7_4);
              g7_1 = fma(ek7_1, r0_0_0_2, g7_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g7_5 = fma(ek7_0, r0_0_1_1, g7_5);
              g7_2 = fma(ek7_1, r0_0_1_1, g7_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g7_6 = fma(ek7_0, r0_0_2_0, g7_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g7_7 = fma(ek7_0, r0_1_0_1, g7_7);
              g7_3 = fma(ek7_1, r0_1_0_1, g7_3);
              g7_1 = fma(ek7_2, r0_1_0_1, g7_1);
              g7_0 = fma(ek7_3, r0_1_0_1, g7_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g7_8 = fma(ek7_0, r0_1_1_0, g7_8);
              g7_2 = fma(ek7_2, r0_1_1_0, g7_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g7_9 = fma(ek7_0, r0_2_0_0, g7_9);
              g7_3 = fma(ek7_2, r0_2_0_0, g7_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g7_10 = fma(ek7_0, r0_0_0_3, g7_10);
              g7_4 = fma(ek7_1, r0_0_0_3, g7_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g7_11 = fma(ek7_0, r0_0_1_2, g7_11);
              g7_5 = fma(ek7_1, r0_0_1_2, g7_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g7_12 = fma(ek7_0, r0_0_2_1, g7_12);
              g7_6 = fma(ek7_1, r0_0_2_1, g7_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g7_13 = fma(ek7_0, r0_0_3_0, g7_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g7_14 = fma(ek7_0, r0_1_0_2, g7_14);
              g7_7 = fma(ek7_1, r0_1_0_2, g7_7);
              g7_4 = fma(ek7_2, r0_1_0_2, g7_4);
              g7_1 = fma(ek7_3, r0_1_0_2, g7_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g7_15 = fma(ek7_0, r0_1_1_1, g7_15);
              g7_8 = fma(ek7_1, r0_1_1_1, g7_8);
              g7_5 = fma(ek7_2, r0_1_1_1, g7_5);
              g7_2 = fma(ek7_3, r0_1_1_1, g7_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g7_16 = fma(ek7_0, r0_1_2_0, g7_16);
              g7_6 = fma(ek7_2, r0_1_2_0, g7_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g7_17 = fma(ek7_0, r0_2_0_1, g7_17);
              g7_9 = fma(ek7_1, r0_2_0_1, g7_9);
              g7_7 = fma(ek7_2, r0_2_0_1, g7_7);
              g7_3 = fma(ek7_3, r0_2_0_1, g7_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g7_18 = fma(ek7_0, r0_2_1_0, g7_18);
              g7_8 = fma(ek7_2, r0_2_1_0, g7_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g7_19 = fma(ek7_0, r0_3_0_0, g7_19);
              g7_9 = fma(ek7_2, r0_3_0_0, g7_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g7_10 = fma(ek7_1, r0_0_0_4, g7_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g7_11 = fma(ek7_1, r0_0_1_3, g7_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g7_12 = fma(ek7_1, r0_0_2_2, g7_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g7_13 = fma(ek7_1, r0_0_3_1, g7_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g7_14 = fma(ek7_1, r0_1_0_3, g7_14);
              g7_10 = fma(ek7_2, r0_1_0_3, g7_10);
              g7_4 = fma(ek7_3, r0_1_0_3, g7_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g7_15 = fma(ek7_1, r0_1_1_2, g7_15);
              g7_11 = fma(ek7_2, r0_1_1_2, g7_11);
              g7_5 = fma(ek7_3, r0_1_1_2, g7_5);
              const double r0_1_2_1 = X * r1_0_2_1;
              g7_16 = fma(ek7_1, r0_1_2_1, g7_16);
              g7_12 = fma(ek7_2, r0_1_2_1, g7_12);
              g7_6 = fma(ek7_3, r0_1_2_1, g7_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g7_13 = fma(ek7_2, r0_1_3_0, g7_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g7_17 = fma(ek7_1, r0_2_0_2, g7_17);
              g7_14 = fma(ek7_2, r0_2_0_2, g7_14);
              g7_7 = fma(ek7_3, r0_2_0_2, g7_7);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g7_18 = fma(ek7_1, r0_2_1_1, g7_18);
              g7_15 = fma(ek7_2, r0_2_1_1, g7_15);
              g7_8 = fma(ek7_3, r0_2_1_1, g7_8);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g7_16 = fma(ek7_2, r0_2_2_0, g7_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g7_19 = fma(ek7_1, r0_3_0_1, g7_19);
              g7_17 = fma(ek7_2, r0_3_0_1, g7_17);
              g7_9 = fma(ek7_3, r0_3_0_1, g7_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g7_18 = fma(ek7_2, r0_3_1_0, g7_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g7_19 = fma(ek7_2, r0_4_0_0, g7_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_1_0_4 = X * r1_0_0_4;
              g7_10 = fma(ek7_3, r0_1_0_4, g7_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g7_11 = fma(ek7_3, r0_1_1_3, g7_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g7_12 = fma(ek7_3, r0_1_2_2, g7_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g7_13 = fma(ek7_3, r0_1_3_1, g7_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g7_14 = fma(ek7_3, r0_2_0_3, g7_14);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g7_15 = fma(ek7_3, r0_2_1_2, g7_15);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g7_16 = fma(ek7_3, r0_2_2_1, g7_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g7_17 = fma(ek7_3, r0_3_0_2, g7_17);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g7_18 = fma(ek7_3, r0_3_1_1, g7_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g7_19 = fma(ek7_3, r0_4_0_1, g7_19);
            }
            { const double eb = bi[5];
              o0_7 = fma(eb, g7_0, o0_7);
            }
            { const double eb = bi[6];
              o0_7 = fma(eb, g7_3, o0_7);
            }
            { const double eb = bi[7];
              o0_7 = fma(eb, g7_9, o0_7);
            }
            { const double eb = bi[8];
              o1_7 = fma(eb, g7_0, o1_7);
            }
            { const double eb = bi[9];
              o1_7 = fma(eb, g7_3, o1_7);
            }
            { const double eb = bi[10];
              o1_7 = fma(eb, g7_9, o1_7);
            }
            { const double eb = bi[11];
              o1_7 = fma(eb, g7_19, o1_7);
            }
            { const double eb = bi[12];
              o2_7 = fma(eb, g7_0, o2_7);
            }
            { const double eb = bi[13];
              o2_7 = fma(eb, g7_2, o2_7);
            }
            { const double eb = bi[14];
              o2_7 = fma(eb, g7_3, o2_7);
            }
            { const double eb = bi[15];
              o2_7 = fma(eb, g7_8, o2_7);
            }
            { const double eb = bi[16];
              o2_7 = fma(eb, g7_9, o2_7);
            }
            { const double eb = bi[17];
              o2_7 = fma(eb, g7_18, o2_7);
            }
            { const double eb = bi[18];
              o3_7 = fma(eb, g7_0, o3_7);
            }
            { const double eb = bi[19];
              o3_7 = fma(eb, g7_1, o3_7);
            }
            { const double eb = bi[20];
              o3_7 = fma(eb, g7_3, o3_7);
            }
            { const double eb = bi[21];
              o3_7 = fma(eb, g7_7, o3_7);
            }
            { const double eb = bi[22];
              o3_7 = fma(eb, g7_9, o3_7);
            }
            { const double eb = bi[23];
              o3_7 = fma(eb, g7_17, o3_7);
            }
            { const double eb = bi[24];
              o4_7 = fma(eb, g7_0, o4_7);
            }
            { const double eb = bi[25];
              o4_7 = fma(eb, g7_2, o4_7);
            }
            { const double eb = bi[26];
              o4_7 = fma(eb, g7_6, o4_7);
            }
            { const double eb = bi[27];
              o5_7 = fma(eb, g7_0, o5_7);
            }
            { const double eb = bi[28];
              o5_7 = fma(eb, g7_2, o5_7);
            }
            { const double eb = bi[29];
              o5_7 = fma(eb, g7_6, o5_7);
            }
            { const double eb = bi[30];
              o5_7 = fma(eb, g7_3, o5_7);
            }
            { const double eb = bi[31];
              o5_7 = fma(eb, g7_8, o5_7);
            }
            { const double eb = bi[32];
              o5_7 = fma(eb, g7_16, o5_7);
            }
            { const double eb = bi[33];
              o6_7 = fma(eb, g7_0, o6_7);
            }
            { const double eb = bi[34];
              o6_7 = fma(eb, g7_2, o6_7);
            }
            { const double eb = bi[35];
              o6_7 = fma(eb, g7_6, o6_7);
            }
            { const double eb = bi[36];
              o6_7 = fma(eb, g7_13, o6_7);
            }
            { const double eb = bi[37];
              o7_7 = fma(eb, g7_0, o7_7);
            }
            { const double eb = bi[38];
              o7_7 = fma(eb, g7_1, o7_7);
            }
            { const double eb = bi[39];
              o7_7 = fma(eb, g7_2, o7_7);
            }
            { const double eb = bi[40];
              o7_7 = fma(eb, g7_5, o7_7);
            }
            { const double eb = bi[41];
              o7_7 = fma(eb, g7_6, o7_7);
            }
            { const double eb = bi[42];
              o7_7 = fma(eb, g7_12, o7_7);
            }
            { const double eb = bi[43];
              o8_7 = fma(eb, g7_0, o8_7);
            }
            { const double eb = bi[44];
              o8_7 = fma(eb, g7_1, o8_7);
            }
            { const double eb = bi[45];
              o8_7 = fma(eb, g7_4, o8_7);
            }
            { const double eb = bi[46];
              o9_7 = fma(eb, g7_0, o9_7);
            }
            { const double eb = bi[47];
              o9_7 = fma(eb, g7_1, o9_7);
            }
            { const double eb = bi[48];
              o9_7 = fma(eb, g7_4, o9_7);
            }
            { const double eb = bi[49];
              o9_7 = fma(eb, g7_3, o9_7);
            }
            { const double eb = bi[50];
              o9_7 = fma(eb, g7_7, o9_7);
            }
            { const double eb = bi[51];
              o9_7 = fma(eb, g7_14, o9_7);
            }
            { const double eb = bi[52];
              o10_7 = fma(eb, g7_0, o10_7);
            }
            { const double eb = bi[53];
              o10_7 = fma(eb, g7_1, o10_7);
            }
            { const double eb = bi[54];
              o10_7 = fma(eb, g7_4, o10_7);
            }
            { const double eb = bi[55];
              o10_7 = fma(eb, g7_2, o10_7);
            }
            { const double eb = bi[56];
              o10_7 = fma(eb, g7_5, o10_7);
            }
            { const double eb = bi[57];
              o10_7 = fma(eb, g7_11, o10_7);
            }
            { const double eb = bi[58];
              o11_7 = fma(eb, g7_0, o11_7);
            }
            { const double eb = bi[59];
              o11_7 = fma(eb, g7_1, o11_7);
            }
            { const double eb = bi[60];
              o11_7 = fma(eb, g7_4, o11_7);
            }
            { const double eb = bi[61];
              o11_7 = fma(eb, g7_10, o11_7);
            }
            { const double eb = bi[62];
              o12_7 = fma(eb, g7_0, o12_7);
            }
            { const double eb = bi[63];
              o12_7 = fma(eb, g7_2, o12_7);
            }
            { const double eb = bi[64];
              o12_7 = fma(eb, g7_3, o12_7);
            }
            { const double eb = bi[65];
              o12_7 = fma(eb, g7_8, o12_7);
            }
            { const double eb = bi[66];
              o13_7 = fma(eb, g7_0, o13_7);
            }
            { const double eb = bi[67];
              o13_7 = fma(eb, g7_2, o13_7);
            }
            { const double eb = bi[68];
              o13_7 = fma(eb, g7_3, o13_7);
            }
            { const double eb = bi[69];
              o13_7 = fma(eb, g7_8, o13_7);
            }
            { const double eb = bi[70];
              o13_7 = fma(eb, g7_9, o13_7);
            }
            { const double eb = bi[71];
              o13_7 = fma(eb, g7_18, o13_7);
            }
            { const double eb = bi[72];
              o14_7 = fma(eb, g7_0, o14_7);
            }
            { const double eb = bi[73];
              o14_7 = fma(eb, g7_2, o14_7);
            }
            { const double eb = bi[74];
              o14_7 = fma(eb, g7_6, o14_7);
            }
            { const double eb = bi[75];
              o14_7 = fma(eb, g7_3, o14_7);
            }
            { const double eb = bi[76];
              o14_7 = fma(eb, g7_8, o14_7);
            }
            { const double eb = bi[77];
              o14_7 = fma(eb, g7_16, o14_7);
            }
            { const double eb = bi[78];
              o15_7 = fma(eb, g7_0, o15_7);
            }
            { const double eb = bi[79];
              o15_7 = fma(eb, g7_1, o15_7);
            }
            { const double eb = bi[80];
              o15_7 = fma(eb, g7_2, o15_7);
            }
            { const double eb = bi[81];
              o15_7 = fma(eb, g7_5, o15_7);
            }
            { const double eb = bi[82];
              o15_7 = fma(eb, g7_3, o15_7);
            }
            { const double eb = bi[83];
              o15_7 = fma(eb, g7_7, o15_7);
            }
            { const double eb = bi[84];
              o15_7 = fma(eb, g7_8, o15_7);
            }
            { const double eb = bi[85];
              o15_7 = fma(eb, g7_15, o15_7);
            }
            { const double eb = bi[86];
              o16_7 = fma(eb, g7_0, o16_7);
            }
            { const double eb = bi[87];
              o16_7 = fma(eb, g7_1, o16_7);
            }
            { const double eb = bi[88];
              o16_7 = fma(eb, g7_3, o16_7);
            }
            { const double eb = bi[89];
              o16_7 = fma(eb, g7_7, o16_7);
            }
            { const double eb = bi[90];
              o17_7 = fma(eb, g7_0, o17_7);
            }
            { const double eb = bi[91];
              o17_7 = fma(eb, g7_1, o17_7);
            }
            { const double eb = bi[92];
              o17_7 = fma(eb, g7_3, o17_7);
            }
            { const double eb = bi[93];
              o17_7 = fma(eb, g7_7, o17_7);
            }
            { const double eb = bi[94];
              o17_7 = fma(eb, g7_9, o17_7);
            }
            { const double eb = bi[95];
              o17_7 = fma(eb, g7_17, o17_7);
            }
            { const double eb = bi[96];
              o18_7 = fma(eb, g7_0, o18_7);
            }
            { const double eb = bi[97];
              o18_7 = fma(eb, g7_1, o18_7);
            }
            { const double eb = bi[98];
              o18_7 = fma(eb, g7_2, o18_7);
            }
            { const double eb = bi[99];
              o18_7 = fma(eb, g7_5, o18_7);
            }
            { const double eb = bi[100];
              o18_7 = fma(eb, g7_3, o18_7);
            }
            { const double eb = bi[101];
              o18_7 = fma(eb, g7_7, o18_7);
            }
            { const double eb = bi[102];
              o18_7 = fma(eb, g7_8, o18_7);
            }
            { const double eb = bi[103];
              o18_7 = fma(eb, g7_15, o18_7);
            }
            { const double eb = bi[104];
              o19_7 = fma(eb, g7_0, o19_7);
            }
            { const double eb = bi[105];
              o19_7 = fma(eb, g7_1, o19_7);
            }
            { const double eb = bi[106];
              o19_7 = fma(eb, g7_4, o19_7);
            }
            { const double eb = bi[107];
              o19_7 = fma(eb, g7_3, o19_7);
            }
            { const double eb = bi[108];
              o19_7 = fma(eb, g7_7, o19_7);
            }
            { const double eb = bi[109];
              o19_7 = fma(eb, g7_14, o19_7);
            }
            { const double eb = bi[110];
              o20_7 = fma(eb, g7_0, o20_7);
            }
            { const double eb = bi[111];
              o20_7 = fma(eb, g7_1, o20_7);
            }
            { const double eb = bi[112];
              o20_7 = fma(eb, g7_2, o20_7);
            }
            { const double eb = bi[113];
              o20_7 = fma(eb, g7_5, o20_7);
            }
            { const double eb = bi[114];
              o21_7 = fma(eb, g7_0, o21_7);
            }
            { const double eb = bi[115];
              o21_7 = fma(eb, g7_1, o21_7);
            }
            { const double eb = bi[116];
              o21_7 = fma(eb, g7_2, o21_7);
            }
            { const double eb = bi[117];
              o21_7 = fma(eb, g7_5, o21_7);
            }
            { const double eb = bi[118];
              o21_7 = fma(eb, g7_3, o21_7);
            }
            { const double eb = bi[119];
              o21_7 = fma(eb, g7_7, o21_7);
            }
            { const double eb = bi[120];
              o21_7 = fma(eb, g7_8, o21_7);
            }
            { const double eb = bi[121];
              o21_7 = fma(eb, g7_15, o21_7);
            }
            { const double eb = bi[122];
              o22_7 = fma(eb, g7_0, o22_7);
            }
            { const double eb = bi[123];
              o22_7 = fma(eb, g7_1, o22_7);
            }
            { const double eb = bi[124];
              o22_7 = fma(eb, g7_2, o22_7);
            }
            { const double eb = bi[125];
              o22_7 = fma(eb, g7_5, o22_7);
            }
            { const double eb = bi[126];
              o22_7 = fma(eb, g7_6, o22_7);
            }
            { const double eb = bi[127];
              o22_7 = fma(eb, g7_12, o22_7);
            }
            { const double eb = bi[128];
              o23_7 = fma(eb, g7_0, o23_7);
            }
            { const double eb = bi[129];
              o23_7 = fma(eb, g7_1, o23_7);
            }
            { const double eb = bi[130];
              o23_7 = fma(eb, g7_4, o23_7);
            }
            { const double eb = bi[131];
              o23_7 = fma(eb, g7_2, o23_7);
            }
            { const double eb = bi[132];
              o23_7 = fma(eb, g7_5, o23_7);
            }
            { const double eb = bi[133];
              o23_7 = fma(eb, g7_11, o23_7);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_7 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 3);
            o1_7 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 3);
            o2_7 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 3);
            o3_7 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 3);
            o4_7 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 3);
            o5_7 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 3);
            o6_7 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 3);
            o7_7 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 3);
            o8_7 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 3);
            o9_7 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 3);
            o10_7 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 3);
            o11_7 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 3);
            o12_7 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 3);
            o13_7 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 3);
            o14_7 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 3);
            o15_7 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 3);
            o16_7 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 3);
            o17_7 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 3);
            o18_7 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 3);
            o19_7 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 3);
            o20_7 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 3);
            o21_7 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 3);
            o22_7 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 3);
            o23_7 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 3);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_7 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o1_7 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o2_7 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o3_7 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o4_7 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o5_7 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o6_7 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o7_7 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o8_7 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o9_7 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o10_7 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o11_7 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o12_7 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o13_7 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o14_7 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o15_7 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o16_7 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o17_7 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o18_7 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o19_7 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o20_7 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o21_7 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o22_7 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 1, fJ + 3)));
            e = fmax(e, fabs(o23_7 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 1, fJ + 3)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
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
            const double Bbd0_3 = PB[(fQ + 0) * N + fJ + 3];
            const double Bbd1_3 = PB[(fQ + 1) * N + fJ + 3];
            const double Bbd2_3 = PB[(fQ + 2) * N + fJ + 3];
            const double Bbd3_3 = PB[(fQ + 3) * N + fJ + 3];
            const double Bad0_3 = PB[(fP + 0) * N + fJ + 3];
            const double Bad1_3 = PB[(fP + 1) * N + fJ + 3];
            const double Bad2_3 = PB[(fP + 2) * N + fJ + 3];
            const double Bad3_3 = PB[(fP + 3) * N + fJ + 3];
            const double Bad4_3 = PB[(fP + 4) * N + fJ + 3];
            const double Bad5_3 = PB[(fP + 5) * N + fJ + 3];
            const double Bbc0_1 = PB[(fQ + 0) * N + fI + 1];
            const double Bbc1_1 = PB[(fQ + 1) * N + fI + 1];
            const double Bbc2_1 = PB[(fQ + 2) * N + fI + 1];
            const double Bbc3_1 = PB[(fQ + 3) * N + fI + 1];
            const double Bac0_1 = PB[(fP + 0) * N + fI + 1];
            const double Bac1_1 = PB[(fP + 1) * N + fI + 1];
            const double Bac2_1 = PB[(fP + 2) * N + fI + 1];
            const double Bac3_1 = PB[(fP + 3) * N + fI + 1];
            const double Bac4_1 = PB[(fP + 4) * N + fI + 1];
            const double Bac5_1 = PB[(fP + 5) * N + fI + 1];
            jab0 += o0_7 * ptk7;
            jab1 += o1_7 * ptk7;
            jab2 += o2_7 * ptk7;
            jab3 += o3_7 * ptk7;
            jab4 += o4_7 * ptk7;
            jab5 += o5_7 * ptk7;
            jab6 += o6_7 * ptk7;
            jab7 += o7_7 * ptk7;
            jab8 += o8_7 * ptk7;
            jab9 += o9_7 * ptk7;
            jab10 += o10_7 * ptk7;
            jab11 += o11_7 * ptk7;
            jab12 += o12_7 * ptk7;
            jab13 += o13_7 * ptk7;
            jab14 += o14_7 * ptk7;
            jab15 += o15_7 * ptk7;
            jab16 += o16_7 * ptk7;
            jab17 += o17_7 * ptk7;
            jab18 += o18_7 * ptk7;
            jab19 += o19_7 * ptk7;
            jab20 += o20_7 * ptk7;
            jab21 += o21_7 * ptk7;
            jab22 += o22_7 * ptk7;
            jab23 += o23_7 * ptk7;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 3, 2.0 * deg * (o0_7 * ptb0 + o1_7 * ptb1 + o2_7 * ptb2 + o3_7 * ptb3 + o4_7 * ptb4 + o5_7 * ptb5 + o6_7 * ptb6 + o7_7 * ptb7 + o8_7 * ptb8 + o9_7 * ptb9 + o10_7 * ptb10 + o11_7 * ptb11 + o12_7 * ptb12 + o13_7 * ptb13 + o14_7 * ptb14 + o15_7 * ptb15 + o16_7 * ptb16 + o17_7 * ptb17 + o18_7 * ptb18 + o19_7 * ptb19 + o20_7 * ptb20 + o21_7 * ptb21 + o22_7 * ptb22 + o23_7 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_7 * Abd0_3 + o1_7 * Abd1_3 + o2_7 * Abd2_3 + o3_7 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_7 * Aad0_3 + o4_7 * Aad1_3 + o8_7 * Aad2_3 + o12_7 * Aad3_3 + o16_7 * Aad4_3 + o20_7 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_7 * Abc0_1 + o1_7 * Abc1_1 + o2_7 * Abc2_1 + o3_7 * Abc3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_7 * Aac0_1 + o4_7 * Aac1_1 + o8_7 * Aac2_1 + o12_7 * Aac3_1 + o16_7 * Aac4_1 + o20_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_7 * Aad0_3 + o5_7 * Aad1_3 + o9_7 * Aad2_3 + o13_7 * Aad3_3 + o17_7 * Aad4_3 + o21_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_7 * Aac0_1 + o5_7 * Aac1_1 + o9_7 * Aac2_1 + o13_7 * Aac3_1 + o17_7 * Aac4_1 + o21_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_7 * Aad0_3 + o6_7 * Aad1_3 + o10_7 * Aad2_3 + o14_7 * Aad3_3 + o18_7 * Aad4_3 + o22_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_7 * Aac0_1 + o6_7 * Aac1_1 + o10_7 * Aac2_1 + o14_7 * Aac3_1 + o18_7 * Aac4_1 + o22_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_7 * Aad0_3 + o7_7 * Aad1_3 + o11_7 * Aad2_3 + o15_7 * Aad3_3 + o19_7 * Aad4_3 + o23_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_7 * Aac0_1 + o7_7 * Aac1_1 + o11_7 * Aac2_1 + o15_7 * Aac3_1 + o19_7 * Aac4_1 + o23_7 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_7 * Abd0_3 + o5_7 * Abd1_3 + o6_7 * Abd2_3 + o7_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_7 * Abc0_1 + o5_7 * Abc1_1 + o6_7 * Abc2_1 + o7_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_7 * Abd0_3 + o9_7 * Abd1_3 + o10_7 * Abd2_3 + o11_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_7 * Abc0_1 + o9_7 * Abc1_1 + o10_7 * Abc2_1 + o11_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_7 * Abd0_3 + o13_7 * Abd1_3 + o14_7 * Abd2_3 + o15_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_7 * Abc0_1 + o13_7 * Abc1_1 + o14_7 * Abc2_1 + o15_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o16_7 * Abd0_3 + o17_7 * Abd1_3 + o18_7 * Abd2_3 + o19_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_7 * Abc0_1 + o17_7 * Abc1_1 + o18_7 * Abc2_1 + o19_7 * Abc3_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o20_7 * Abd0_3 + o21_7 * Abd1_3 + o22_7 * Abd2_3 + o23_7 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_7 * Abc0_1 + o21_7 * Abc1_1 + o22_7 * Abc2_1 + o23_7 * Abc3_1));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_7 * Bbd0_3 + o1_7 * Bbd1_3 + o2_7 * Bbd2_3 + o3_7 * Bbd3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_7 * Bad0_3 + o4_7 * Bad1_3 + o8_7 * Bad2_3 + o12_7 * Bad3_3 + o16_7 * Bad4_3 + o20_7 * Bad5_3));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 3, deg * (o0_7 * Bbc0_1 + o1_7 * Bbc1_1 + o2_7 * Bbc2_1 + o3_7 * Bbc3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 3, deg * (o0_7 * Bac0_1 + o4_7 * Bac1_1 + o8_7 * Bac2_1 + o12_7 * Bac3_1 + o16_7 * Bac4_1 + o20_7 * Bac5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 1, deg * (o1_7 * Bad0_3 + o5_7 * Bad1_3 + o9_7 * Bad2_3 + o13_7 * Bad3_3 + o17_7 * Bad4_3 + o21_7 * Bad5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 3, deg * (o1_7 * Bac0_1 + o5_7 * Bac1_1 + o9_7 * Bac2_1 + o13_7 * Bac3_1 + o17_7 * Bac4_1 + o21_7 * Bac5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 1, deg * (o2_7 * Bad0_3 + o6_7 * Bad1_3 + o10_7 * Bad2_3 + o14_7 * Bad3_3 + o18_7 * Bad4_3 + o22_7 * Bad5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 3, deg * (o2_7 * Bac0_1 + o6_7 * Bac1_1 + o10_7 * Bac2_1 + o14_7 * Bac3_1 + o18_7 * Bac4_1 + o22_7 * Bac5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 1, deg * (o3_7 * Bad0_3 + o7_7 * Bad1_3 + o11_7 * Bad2_3 + o15_7 * Bad3_3 + o19_7 * Bad4_3 + o23_7 * Bad5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 3, deg * (o3_7 * Bac0_1 + o7_7 * Bac1_1 + o11_7 * Bac2_1 + o15_7 * Bac3_1 + o19_7 * Bac4_1 + o23_7 * Bac5_1));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o4_7 * Bbd0_3 + o5_7 * Bbd1_3 + o6_7 * Bbd2_3 + o7_7 * Bbd3_3));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 3, deg * (o4_7 * Bbc0_1 + o5_7 * Bbc1_1 + o6_7 * Bbc2_1 + o7_7 * Bbc3_1));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o8_7 * Bbd0_3 + o9_7 * Bbd1_3 + o10_7 * Bbd2_3 + o11_7 * Bbd3_3));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 3, deg * (o8_7 * Bbc0_1 + o9_7 * Bbc1_1 + o10_7 * Bbc2_1 + o11_7 * Bbc3_1));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o12_7 * Bbd0_3 + o13_7 * Bbd1_3 + o14_7 * Bbd2_3 + o15_7 * Bbd3_3));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 3, deg * (o12_7 * Bbc0_1 + o13_7 * Bbc1_1 + o14_7 * Bbc2_1 + o15_7 * Bbc3_1));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o16_7 * Bbd0_3 + o17_7 * Bbd1_3 + o18_7 * Bbd2_3 + o19_7 * Bbd3_3));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 3, deg * (o16_7 * Bbc0_1 + o17_7 * Bbc1_1 + o18_7 * Bbc2_1 + o19_7 * Bbc3_1));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o20_7 * Bbd0_3 + o21_7 * Bbd1_3 + o22_7 * Bbd2_3 + o23_7 * Bbd3_3));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 3, deg * (o20_7 * Bbc0_1 + o21_7 * Bbc1_1 + o22_7 * Bbc2_1 + o23_7 * Bbc3_1));
          }
        } break;
        case 8: {  // ket functions [8]
          double o0_8 = 0;
          double o1_8 = 0;
          double o2_8 = 0;
          double o3_8 = 0;
          double o4_8 = 0;
          double o5_8 = 0;
          double o6_8 = 0;
          double o7_8 = 0;
          double o8_8 = 0;
          double o9_8 = 0;
          double o10_8 = 0;
          double o11_8 = 0;
          double o12_8 = 0;
          double o13_8 = 0;
          double o14_8 = 0;
          double o15_8 = 0;
          double o16_8 = 0;
          double o17_8 = 0;
          double o18_8 = 0;
          double o19_8 = 0;
          double o20_8 = 0;
          double o21_8 = 0;
          double o22_8 = 0;
          double o23_8 = 0;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek8_0 = kj[25 * kS];
              const double ek8_1 = -kj[26 * kS];
              g8_0 = fma(ek8_0, b0, g8_0);
              const double r0_0_0_1 = Z * b1;
              g8_1 = fma(ek8_0, r0_0_0_1, g8_1);
              const double r0_0_1_0 = Y * b1;
              g8_2 = fma(ek8_0, r0_0_1_0, g8_2);
              g8_0 = fma(ek8_1, r0_0_1_0, g8_0);
              const double r0_1_0_0 = X * b1;
              g8_3 = fma(ek8_0, r0_1_0_0, g8_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g8_4 = fma(ek8_0, r0_0_0_2, g8_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g8_5 = fma(ek8_0, r0_0_1_1, g8_5);
              g8_1 = fma(ek8_1, r0_0_1_1, g8_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g8_6 = fma(ek8_0, r0_0_2_0, g8_6);
              g8_2 = fma(ek8_1, r0_0_2_0, g8_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g8_7 = fma(ek8_0, r0_1_0_1, g8_7);
              const double r0_1_1_0 = X * r1_0_1_0;
              g8_8 = fma(ek8_0, r0_1_1_0, g8_8);
              g8_3 = fma(ek8_1, r0_1_1_0, g8_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g8_9 = fma(ek8_0, r0_2_0_0, g8_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g8_10 = fma(ek8_0, r0_0_0_3, g8_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g8_11 = fma(ek8_0, r0_0_1_2, g8_11);
              g8_4 = fma(ek8_1, r0_0_1_2, g8_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g8_12 = fma(ek8_0, r0_0_2_1, g8_12);
              g8_5 = fma(ek8_1, r0_0_2_1, g8_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g8_13 = fma(ek8_0, r0_0_3_0, g8_13);
              g8_6 = fma(ek8_1, r0_0_3_0, g8_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g8_14 = fma(ek8_0, r0_1_0_2, g8_14);
              const double r0_1_1_1 = X * r1_0_1_1;
              g8_15 = fma(ek8_0, r0_1_1_1, g8_15);
              g8_7 = fma(ek8_1, r0_1_1_1, g8_7);
              const double r0_1_2_0 = X * r1_0_2_0;
              g8_16 = fma(ek8_0, r0_1_2_0, g8_16);
              g8_8 = fma(ek8_1, r0_1_2_0, g8_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g8_17 = fma(ek8_0, r0_2_0_1, g8_17);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g8_18 = fma(ek8_0, r0_2_1_0, g8_18);
              g8_9 = fma(ek8_1, r0_2_1_0, g8_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g8_19 = fma(ek8_0, r0_3_0_0, g8_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g8_10 = fma(ek8_1, r0_0_1_3, g8_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g8_11 = fma(ek8_1, r0_0_2_2, g8_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g8_12 = fma(ek8_1, r0_0_3_1, g8_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g8_13 = fma(ek8_1, r0_0_4_0, g8_13);
              const double r0_1_1_2 = X * r1_0_1_2;
              g8_14 = fma(ek8_1, r0_1_1_2, g8_14);
              const double r0_1_2_1 = X * r1_0_2_1;
              g8_15 = fma(ek8_1, r0_1_2_1, g8_15);
              const double r0_1_3_0 = X * r1_0_3_0;
              g8_16 = fma(ek8_1, r0_1_3_0, g8_16);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g8_17 = fma(ek8_1, r0_2_1_1, g8_17);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g8_18 = fma(ek8_1, r0_2_2_0, g8_18);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g8_19 = fma(ek8_1, r0_3_1_0, g8_19);
            }
            { const double eb = bi[5];
              o0_8 = fma(eb, g8_0, o0_8);
            }
            { const double eb = bi[6];
              o0_8 = fma(eb, g8_3, o0_8);
            }
            { const double eb = bi[7];
              o0_8 = fma(eb, g8_9, o0_8);
            }
            { const double eb = bi[8];
              o1_8 = fma(eb, g8_0, o1_8);
            }
            { const double eb = bi[9];
              o1_8 = fma(eb, g8_3, o1_8);
            }
            { const double eb = bi[10];
              o1_8 = fma(eb, g8_9, o1_8);
            }
            { const double eb = bi[11];
              o1_8 = fma(eb, g8_19, o1_8);
            }
            { const double eb = bi[12];
              o2_8 = fma(eb, g8_0, o2_8);
            }
            { const double eb = bi[13];
              o2_8 = fma(eb, g8_2, o2_8);
            }
            { const double eb = bi[14];
              o2_8 = fma(eb, g8_3, o2_8);
            }
            { const double eb = bi[15];
              o2_8 = fma(eb, g8_8, o2_8);
            }
            { const double eb = bi[16];
              o2_8 = fma(eb, g8_9, o2_8);
            }
            { const double eb = bi[17];
              o2_8 = fma(eb, g8_18, o2_8);
            }
            { const double eb = bi[18];
              o3_8 = fma(eb, g8_0, o3_8);
            }
            { const double eb = bi[19];
              o3_8 = fma(eb, g8_1, o3_8);
            }
            { const double eb = bi[20];
              o3_8 = fma(eb, g8_3, o3_8);
            }
            { const double eb = bi[21];
              o3_8 = fma(eb, g8_7, o3_8);
            }
            { const double eb = bi[22];
              o3_8 = fma(eb, g8_9, o3_8);
            }
            { const double eb = bi[23];
              o3_8 = fma(eb, g8_17, o3_8);
            }
            { const double eb = bi[24];
              o4_8 = fma(eb, g8_0, o4_8);
            }
            { const double eb = bi[25];
              o4_8 = fma(eb, g8_2, o4_8);
            }
            { const double eb = bi[26];
              o4_8 = fma(eb, g8_6, o4_8);
            }
            { const double eb = bi[27];
              o5_8 = fma(eb, g8_0, o5_8);
            }
            { const double eb = bi[28];
              o5_8 = fma(eb, g8_2, o5_8);
            }
            { const double eb = bi[29];
              o5_8 = fma(eb, g8_6, o5_8);
            }
            { const double eb = bi[30];
              o5_8 = fma(eb, g8_3, o5_8);
            }
            { const double eb = bi[31];
              o5_8 = fma(eb, g8_8, o5_8);
            }
            { const double eb = bi[32];
              o5_8 = fma(eb, g8_16, o5_8);
            }
            { const double eb = bi[33];
              o6_8 = fma(eb, g8_0, o6_8);
            }
            { const double eb = bi[34];
              o6_8 = fma(eb, g8_2, o6_8);
            }
            { const double eb = bi[35];
              o6_8 = fma(eb, g8_6, o6_8);
            }
            { const double eb = bi[36];
              o6_8 = fma(eb, g8_13, o6_8);
            }
            { const double eb = bi[37];
              o7_8 = fma(eb, g8_0, o7_8);
            }
            { const double eb = bi[38];
              o7_8 = fma(eb, g8_1, o7_8);
            }
            { const double eb = bi[39];
              o7_8 = fma(eb, g8_2, o7_8);
            }
            { const double eb = bi[40];
              o7_8 = fma(eb, g8_5, o7_8);
            }
            { const double eb = bi[41];
              o7_8 = fma(eb, g8_6, o7_8);
            }
            { const double eb = bi[42];
              o7_8 = fma(eb, g8_12, o7_8);
            }
            { const double eb = bi[43];
              o8_8 = fma(eb, g8_0, o8_8);
            }
            { const double eb = bi[44];
              o8_8 = fma(eb, g8_1, o8_8);
            }
            { const double eb = bi[45];
              o8_8 = fma(eb, g8_4, o8_8);
            }
            { const double eb = bi[46];
              o9_8 = fma(eb, g8_0, o9_8);
            }
            { const double eb = bi[47];
              o9_8 = fma(eb, g8_1, o9_8);
            }
            { const double eb = bi[48];
              o9_8 = fma(eb, g8_4, o9_8);
            }
            { const double eb = bi[49];
              o9_8 = fma(eb, g8_3, o9_8);
            }
            { const double eb = bi[50];
              o9_8 = fma(eb, g8_7, o9_8);
            }
            { const double eb = bi[51];
              o9_8 = fma(eb, g8_14, o9_8);
            }
            { const double eb = bi[52];
              o10_8 = fma(eb, g8_0, o10_8);
            }
            { const double eb = bi[53];
              o10_8 = fma(eb, g8_1, o10_8);
            }
            { const double eb = bi[54];
              o10_8 = fma(eb, g8_4, o10_8);
            }
            { const double eb = bi[55];
              o10_8 = fma(eb, g8_2, o10_8);
            }
            { const double eb = bi[56];
              o10_8 = fma(eb, g8_5, o10_8);
            }
            { const double eb = bi[57];
              o10_8 = fma(eb, g8_11, o10_8);
            }
            { const double eb = bi[58];
              o11_8 = fma(eb, g8_0, o11_8);
            }
            { const double eb = bi[59];
              o11_8 = fma(eb, g8_1, o11_8);
            }
            { const double eb = bi[60];
              o11_8 = fma(eb, g8_4, o11_8);
            }
            { const double eb = bi[61];
              o11_8 = fma(eb, g8_10, o11_8);
            }
            { const double eb = bi[62];
              o12_8 = fma(eb, g8_0, o12_8);
            }
            { const double eb = bi[63];
              o12_8 = fma(eb, g8_2, o12_8);
            }
            { const double eb = bi[64];
              o12_8 = fma(eb, g8_3, o12_8);
            }
            { const double eb = bi[65];
              o12_8 = fma(eb, g8_8, o12_8);
            }
            { const double eb = bi[66];
              o13_8 = fma(eb, g8_0, o13_8);
            }
            { const double eb = bi[67];
              o13_8 = fma(eb, g8_2, o13_8);
            }
            { const double eb = bi[68];
              o13_8 = fma(eb, g8_3, o13_8);
            }
            { const double eb = bi[69];
              o13_8 = fma(eb, g8_8, o13_8);
            }
            { const double eb = bi[70];
              o13_8 = fma(eb, g8_9, o13_8);
            }
            { const double eb = bi[71];
              o13_8 = fma(eb, g8_18, o13_8);
            }
            { const double eb = bi[72];
              o14_8 = fma(eb, g8_0, o14_8);
            }
            { const double eb = bi[73];
              o14_8 = fma(eb, g8_2, o14_8);
            }
            { const double eb = bi[74];
              o14_8 = fma(eb, g8_6, o14_8);
            }
            { const double eb = bi[75];
              o14_8 = fma(eb, g8_3, o14_8);
            }
            { const double eb = bi[76];
              o14_8 = fma(eb, g8_8, o14_8);
            }
            { const double eb = bi[77];
              o14_8 = fma(eb, g8_16, o14_8);
            }
            { const double eb = bi[78];
              o15_8 = fma(eb, g8_0, o15_8);
            }
            { const double eb = bi[79];
              o15_8 = fma(eb, g8_1, o15_8);
            }
            { const double eb = bi[80];
              o15_8 = fma(eb, g8_2, o15_8);
            }
            { const double eb = bi[81];
              o15_8 = fma(eb, g8_5, o15_8);
            }
            { const double eb = bi[82];
              o15_8 = fma(eb, g8_3, o15_8);
            }
            { const double eb = bi[83];
              o15_8 = fma(eb, g8_7, o15_8);
            }
            { const double eb = bi[84];
              o15_8 = fma(eb, g8_8, o15_8);
            }
            { const double eb = bi[85];
              o15_8 = fma(eb, g8_15, o15_8);
            }
            { const double eb = bi[86];
              o16_8 = fma(eb, g8_0, o16_8);
            }
            { const double eb = bi[87];
              o16_8 = fma(eb, g8_1, o16_8);
            }
            { const double eb = bi[88];
              o16_8 = fma(eb, g8_3, o16_8);
            }
            { const double eb = bi[89];
              o16_8 = fma(eb, g8_7, o16_8);
            }
            { const double eb = bi[90];
              o17_8 = fma(eb, g8_0, o17_8);
            }
            { const double eb = bi[91];
              o17_8 = fma(eb, g8_1, o17_8);
            }
            { const double eb = bi[92];
              o17_8 = fma(eb, g8_3, o17_8);
            }
            { const double eb = bi[93];
              o17_8 = fma(eb, g8_7, o17_8);
            }
            { const double eb = bi[94];
              o17_8 = fma(eb, g8_9, o17_8);
            }
            { const double eb = bi[95];
              o17_8 = fma(eb, g8_17, o17_8);
            }
            { const double eb = bi[96];
              o18_8 = fma(eb, g8_0, o18_8);
            }
            { const double eb = bi[97];
              o18_8 = fma(eb, g8_1, o18_8);
            }
            { const double eb = bi[98];
              o18_8 = fma(eb, g8_2, o18_8);
            }
            { const double eb = bi[99];
              o18_8 = fma(eb, g8_5, o18_8);
            }
            { const double eb = bi[100];
              o18_8 = fma(eb, g8_3, o18_8);
            }
            { const double eb = bi[101];
              o18_8 = fma(eb, g8_7, o18_8);
            }
            { const double eb = bi[102];
              o18_8 = fma(eb, g8_8, o18_8);
            }
            { const double eb = bi[103];
              o18_8 = fma(eb, g8_15, o18_8);
            }
            { const double eb = bi[104];
              o19_8 = fma(eb, g8_0, o19_8);
            }
            { const double eb = bi[105];
              o19_8 = fma(eb, g8_1, o19_8);
            }
            { const double eb = bi[106];
              o19_8 = fma(eb, g8_4, o19_8);
            }
            { const double eb = bi[107];
              o19_8 = fma(eb, g8_3, o19_8);
            }
            { const double eb = bi[108];
              o19_8 = fma(eb, g8_7, o19_8);
            }
            { const double eb = bi[109];
              o19_8 = fma(eb, g8_14, o19_8);
            }
            { const double eb = bi[110];
              o20_8 = fma(eb, g8_0, o20_8);
            }
            { const double eb = bi[111];
              o20_8 = fma(eb, g8_1, o20_8);
            }
            { const double eb = bi[112];
              o20_8 = fma(eb, g8_2, o20_8);
            }
            { const double eb = bi[113];
              o20_8 = fma(eb, g8_5, o20_8);
            }
            { const double eb = bi[114];
              o21_8 = fma(eb, g8_0, o21_8);
            }
            { const double eb = bi[115];
              o21_8 = fma(eb, g8_1, o21_8);
            }
            { const double eb = bi[116];
              o21_8 = fma(eb, g8_2, o21_8);
            }
            { const double eb = bi[117];
              o21_8 = fma(eb, g8_5, o21_8);
            }
            { const double eb = bi[118];
              o21_8 = fma(eb, g8_3, o21_8);
            }
            { const double eb = bi[119];
              o21_8 = fma(eb, g8_7, o21_8);
            }
            { const double eb = bi[120];
              o21_8 = fma(eb, g8_8, o21_8);
            }
            { const double eb = bi[121];
              o21_8 = fma(eb, g8_15, o21_8);
            }
            { const double eb = bi[122];
              o22_8 = fma(eb, g8_0, o22_8);
            }
            { const double eb = bi[123];
              o22_8 = fma(eb, g8_1, o22_8);
            }
            { const double eb = bi[124];
              o22_8 = fma(eb, g8_2, o22_8);
            }
            { const double eb = bi[125];
              o22_8 = fma(eb, g8_5, o22_8);
            }
            { const double eb = bi[126];
              o22_8 = fma(eb, g8_6, o22_8);
            }
            { const double eb = bi[127];
              o22_8 = fma(eb, g8_12, o22_8);
            }
            { const double eb = bi[128];
              o23_8 = fma(eb, g8_0, o23_8);
            }
            { const double eb = bi[129];
              o23_8 = fma(eb, g8_1, o23_8);
            }
            { const double eb = bi[130];
              o23_8 = fma(eb, g8_4, o23_8);
            }
            { const double eb = bi[131];
              o23_8 = fma(eb, g8_2, o23_8);
            }
            { const double eb = bi[132];
              o23_8 = fma(eb, g8_5, o23_8);
            }
            { const double eb = bi[133];
              o23_8 = fma(eb, g8_11, o23_8);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_8 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0);
            o1_8 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 0);
            o2_8 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 0);
            o3_8 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 0);
            o4_8 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0);
            o5_8 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 0);
            o6_8 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 0);
            o7_8 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 0);
            o8_8 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0);
            o9_8 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 0);
            o10_8 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 0);
            o11_8 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 0);
            o12_8 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0);
            o13_8 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 0);
            o14_8 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 0);
            o15_8 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 0);
            o16_8 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0);
            o17_8 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 0);
            o18_8 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 0);
            o19_8 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 0);
            o20_8 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0);
            o21_8 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 0);
            o22_8 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 0);
            o23_8 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_8 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o1_8 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o2_8 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o3_8 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o4_8 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o5_8 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o6_8 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o7_8 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o8_8 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o9_8 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o10_8 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o11_8 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o12_8 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o13_8 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o14_8 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o15_8 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o16_8 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o17_8 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o18_8 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o19_8 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o20_8 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o21_8 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o22_8 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o23_8 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk8 = PT[(fI + 2) * N + fJ + 0];
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
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
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
            const double Bac0_2 = PB[(fP + 0) * N + fI + 2];
            const double Bac1_2 = PB[(fP + 1) * N + fI + 2];
            const double Bac2_2 = PB[(fP + 2) * N + fI + 2];
            const double Bac3_2 = PB[(fP + 3) * N + fI + 2];
            const double Bac4_2 = PB[(fP + 4) * N + fI + 2];
            const double Bac5_2 = PB[(fP + 5) * N + fI + 2];
            jab0 += o0_8 * ptk8;
            jab1 += o1_8 * ptk8;
            jab2 += o2_8 * ptk8;
            jab3 += o3_8 * ptk8;
            jab4 += o4_8 * ptk8;
            jab5 += o5_8 * ptk8;
            jab6 += o6_8 * ptk8;
            jab7 += o7_8 * ptk8;
            jab8 += o8_8 * ptk8;
            jab9 += o9_8 * ptk8;
            jab10 += o10_8 * ptk8;
            jab11 += o11_8 * ptk8;
            jab12 += o12_8 * ptk8;
            jab13 += o13_8 * ptk8;
            jab14 += o14_8 * ptk8;
            jab15 += o15_8 * ptk8;
            jab16 += o16_8 * ptk8;
            jab17 += o17_8 * ptk8;
            jab18 += o18_8 * ptk8;
            jab19 += o19_8 * ptk8;
            jab20 += o20_8 * ptk8;
            jab21 += o21_8 * ptk8;
            jab22 += o22_8 * ptk8;
            jab23 += o23_8 * ptk8;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_8 * ptb0 + o1_8 * ptb1 + o2_8 * ptb2 + o3_8 * ptb3 + o4_8 * ptb4 + o5_8 * ptb5 + o6_8 * ptb6 + o7_8 * ptb7 + o8_8 * ptb8 + o9_8 * ptb9 + o10_8 * ptb10 + o11_8 * ptb11 + o12_8 * ptb12 + o13_8 * ptb13 + o14_8 * ptb14 + o15_8 * ptb15 + o16_8 * ptb16 + o17_8 * ptb17 + o18_8 * ptb18 + o19_8 * ptb19 + o20_8 * ptb20 + o21_8 * ptb21 + o22_8 * ptb22 + o23_8 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_8 * Abd0_0 + o1_8 * Abd1_0 + o2_8 * Abd2_0 + o3_8 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_8 * Aad0_0 + o4_8 * Aad1_0 + o8_8 * Aad2_0 + o12_8 * Aad3_0 + o16_8 * Aad4_0 + o20_8 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_8 * Abc0_2 + o1_8 * Abc1_2 + o2_8 * Abc2_2 + o3_8 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_8 * Aac0_2 + o4_8 * Aac1_2 + o8_8 * Aac2_2 + o12_8 * Aac3_2 + o16_8 * Aac4_2 + o20_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_8 * Aad0_0 + o5_8 * Aad1_0 + o9_8 * Aad2_0 + o13_8 * Aad3_0 + o17_8 * Aad4_0 + o21_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_8 * Aac0_2 + o5_8 * Aac1_2 + o9_8 * Aac2_2 + o13_8 * Aac3_2 + o17_8 * Aac4_2 + o21_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_8 * Aad0_0 + o6_8 * Aad1_0 + o10_8 * Aad2_0 + o14_8 * Aad3_0 + o18_8 * Aad4_0 + o22_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_8 * Aac0_2 + o6_8 * Aac1_2 + o10_8 * Aac2_2 + o14_8 * Aac3_2 + o18_8 * Aac4_2 + o22_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_8 * Aad0_0 + o7_8 * Aad1_0 + o11_8 * Aad2_0 + o15_8 * Aad3_0 + o19_8 * Aad4_0 + o23_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_8 * Aac0_2 + o7_8 * Aac1_2 + o11_8 * Aac2_2 + o15_8 * Aac3_2 + o19_8 * Aac4_2 + o23_8 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_8 * Abd0_0 + o5_8 * Abd1_0 + o6_8 * Abd2_0 + o7_8 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_8 * Abc0_2 + o5_8 * Abc1_2 + o6_8 * Abc2_2 + o7_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_8 * Abd0_0 + o9_8 * Abd1_0 + o10_8 * Abd2_0 + o11_8 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_8 * Abc0_2 + o9_8 * Abc1_2 + o10_8 * Abc2_2 + o11_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_8 * Abd0_0 + o13_8 * Abd1_0 + o14_8 * Abd2_0 + o15_8 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_8 * Abc0_2 + o13_8 * Abc1_2 + o14_8 * Abc2_2 + o15_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_8 * Abd0_0 + o17_8 * Abd1_0 + o18_8 * Abd2_0 + o19_8 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_8 * Abc0_2 + o17_8 * Abc1_2 + o18_8 * Abc2_2 + o19_8 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_8 * Abd0_0 + o21_8 * Abd1_0 + o22_8 * Abd2_0 + o23_8 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_8 * Abc0_2 + o21_8 * Abc1_2 + o22_8 * Abc2_2 + o23_8 * Abc3_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_8 * Bbd0_0 + o1_8 * Bbd1_0 + o2_8 * Bbd2_0 + o3_8 * Bbd3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_8 * Bad0_0 + o4_8 * Bad1_0 + o8_8 * Bad2_0 + o12_8 * Bad3_0 + o16_8 * Bad4_0 + o20_8 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_8 * Bbc0_2 + o1_8 * Bbc1_2 + o2_8 * Bbc2_2 + o3_8 * Bbc3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_8 * Bac0_2 + o4_8 * Bac1_2 + o8_8 * Bac2_2 + o12_8 * Bac3_2 + o16_8 * Bac4_2 + o20_8 * Bac5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 2, deg * (o1_8 * Bad0_0 + o5_8 * Bad1_0 + o9_8 * Bad2_0 + o13_8 * Bad3_0 + o17_8 * Bad4_0 + o21_8 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_8 * Bac0_2 + o5_8 * Bac1_2 + o9_8 * Bac2_2 + o13_8 * Bac3_2 + o17_8 * Bac4_2 + o21_8 * Bac5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 2, deg * (o2_8 * Bad0_0 + o6_8 * Bad1_0 + o10_8 * Bad2_0 + o14_8 * Bad3_0 + o18_8 * Bad4_0 + o22_8 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_8 * Bac0_2 + o6_8 * Bac1_2 + o10_8 * Bac2_2 + o14_8 * Bac3_2 + o18_8 * Bac4_2 + o22_8 * Bac5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 2, deg * (o3_8 * Bad0_0 + o7_8 * Bad1_0 + o11_8 * Bad2_0 + o15_8 * Bad3_0 + o19_8 * Bad4_0 + o23_8 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_8 * Bac0_2 + o7_8 * Bac1_2 + o11_8 * Bac2_2 + o15_8 * Bac3_2 + o19_8 * Bac4_2 + o23_8 * Bac5_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o4_8 * Bbd0_0 + o5_8 * Bbd1_0 + o6_8 * Bbd2_0 + o7_8 * Bbd3_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o4_8 * Bbc0_2 + o5_8 * Bbc1_2 + o6_8 * Bbc2_2 + o7_8 * Bbc3_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o8_8 * Bbd0_0 + o9_8 * Bbd1_0 + o10_8 * Bbd2_0 + o11_8 * Bbd3_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o8_8 * Bbc0_2 + o9_8 * Bbc1_2 + o10_8 * Bbc2_2 + o11_8 * Bbc3_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o12_8 * Bbd0_0 + o13_8 * Bbd1_0 + o14_8 * Bbd2_0 + o15_8 * Bbd3_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o12_8 * Bbc0_2 + o13_8 * Bbc1_2 + o14_8 * Bbc2_2 + o15_8 * Bbc3_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o16_8 * Bbd0_0 + o17_8 * Bbd1_0 + o18_8 * Bbd2_0 + o19_8 * Bbd3_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o16_8 * Bbc0_2 + o17_8 * Bbc1_2 + o18_8 * Bbc2_2 + o19_8 * Bbc3_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o20_8 * Bbd0_0 + o21_8 * Bbd1_0 + o22_8 * Bbd2_0 + o23_8 * Bbd3_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o20_8 * Bbc0_2 + o21_8 * Bbc1_2 + o22_8 * Bbc2_2 + o23_8 * Bbc3_2));
          }
        } break;
        case 9: {  // ket functions [9]
          double o0_9 = 0;
          double o1_9 = 0;
          double o2_9 = 0;
          double o3_9 = 0;
          double o4_9 = 0;
          double o5_9 = 0;
          double o6_9 = 0;
          double o7_9 = 0;
          double o8_9 = 0;
          double o9_9 = 0;
          double o10_9 = 0;
          double o11_9 = 0;
          double o12_9 = 0;
          double o13_9 = 0;
          double o14_9 = 0;
          double o15_9 = 0;
          double o16_9 = 0;
          double o17_9 = 0;
          double o18_9 = 0;
          double o19_9 = 0;
          double o20_9 = 0;
          double o21_9 = 0;
          double o22_9 = 0;
          double o23_9 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek9_0 = kj[27 * kS];
              const double ek9_1 = -kj[28 * kS];
              const double ek9_2 = -kj[29 * kS];
              const double ek9_3 = kj[30 * kS];
              g9_0 = fma(ek9_0, b0, g9_0);
              const double r0_0_0_1 = Z * b1;
              g9_1 = fma(ek9_0, r0_0_0_1, g9_1);
              const double r0_0_1_0 = Y * b1;
              g9_2 = fma(ek9_0, r0_0_1_0, g9_2);
              g9_0 = fma(ek9_1, r0_0_1_0, g9_0);
              const double r0_1_0_0 = X * b1;
              g9_3 = fma(ek9_0, r0_1_0_0, g9_3);
              g9_0 = fma(ek9_2, r0_1_0_0, g9_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g9_4 = fma(ek9_0, r0_0_0_2, g9_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g9_5 = fma(ek9_0, r0_0_1_1, g9_5);
              g9_1 = fma(ek9_1, r0_0_1_1, g9_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g9_6 = fma(ek9_0, r0_0_2_0, g9_6);
              g9_2 = fma(ek9_1, r0_0_2_0, g9_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g9_7 = fma(ek9_0, r0_1_0_1, g9_7);
              g9_1 = fma(ek9_2, r0_1_0_1, g9_1);
              const double r0_1_1_0 = X * r1_0_1_0;
              g9_8 = fma(ek9_0, r0_1_1_0, g9_8);
              g9_3 = fma(ek9_1, r0_1_1_0, g9_3);
              g9_2 = fma(ek9_2, r0_1_1_0, g9_2);
              g9_0 = fma(ek9_3, r0_1_1_0, g9_0);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g9_9 = fma(ek9_0, r0_2_0_0, g9_9);
              g9_3 = fma(ek9_2, r0_2_0_0, g9_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g9_10 = fma(ek9_0, r0_0_0_3, g9_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g9_11 = fma(ek9_0, r0_0_1_2, g9_11);
              g9_4 = fma(ek9_1, r0_0_1_2, g9_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g9_12 = fma(ek9_0, r0_0_2_1, g9_12);
              g9_5 = fma(ek9_1, r0_0_2_1, g9_5);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g9_13 = fma(ek9_0, r0_0_3_0, g9_13);
              g9_6 = fma(ek9_1, r0_0_3_0, g9_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g9_14 = fma(ek9_0, r0_1_0_2, g9_14);
              g9_4 = fma(ek9_2, r0_1_0_2, g9_4);
              const double r0_1_1_1 = X * r1_0_1_1;
              g9_15 = fma(ek9_0, r0_1_1_1, g9_15);
              g9_7 = fma(ek9_1, r0_1_1_1, g9_7);
              g9_5 = fma(ek9_2, r0_1_1_1, g9_5);
              g9_1 = fma(ek9_3, r0_1_1_1, g9_1);
              const double r0_1_2_0 = X * r1_0_2_0;
              g9_16 = fma(ek9_0, r0_1_2_0, g9_16);
              g9_8 = fma(ek9_1, r0_1_2_0, g9_8);
              g9_6 = fma(ek9_2, r0_1_2_0, g9_6);
              g9_2 = fma(ek9_3, r0_1_2_0, g9_2);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g9_17 = fma(ek9_0, r0_2_0_1, g9_17);
              g9_7 = fma(ek9_2, r0_2_0_1, g9_7);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g9_18 = fma(ek9_0, r0_2_1_0, g9_18);
              g9_9 = fma(ek9_1, r0_2_1_0, g9_9);
              g9_8 = fma(ek9_2, r0_2_1_0, g9_8);
              g9_3 = fma(ek9_3, r0_2_1_0, g9_3);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g9_19 = fma(ek9_0, r0_3_0_0, g9_19);
              g9_9 = fma(ek9_2, r0_3_0_0, g9_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g9_10 = fma(ek9_1, r0_0_1_3, g9_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g9_11 = fma(ek9_1, r0_0_2_2, g9_11);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g9_12 = fma(ek9_1, r0_0_3_1, g9_12);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g9_13 = fma(ek9_1, r0_0_4_0, g9_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g9_10 = fma(ek9_2, r0_1_0_3, g9_10);
              const double r0_1_1_2 = X * r1_0_1_2;
              g9_14 = fma(ek9_1, r0_1_1_2, g9_14);
              g9_11 = fma(ek9_2, r0_1_1_2, g9_11);
              g9_4 = fma(ek9_3, r0_1_1_2, g9_4);
              const double r0_1_2_1 = X * r1_0_2_1;
              g9_15 = fma(ek9_1, r0_1_2_1, g9_15);
              g9_12 = fma(ek9_2, r0_1_2_1, g9_12);
              g9_5 = fma(ek9_3, r0_1_2_1, g9_5);
              const double r0_1_3_0 = X * r1_0_3_0;
              g9_16 = fma(ek9_1, r0_1_3_0, g9_16);
              g9_13 = fma(ek9_2, r0_1_3_0, g9_13);
              g9_6 = fma(ek9_3, r0_1_3_0, g9_6);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g9_14 = fma(ek9_2, r0_2_0_2, g9_14);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g9_17 = fma(ek9_1, r0_2_1_1, g9_17);
              g9_15 = fma(ek9_2, r0_2_1_1, g9_15);
              g9_7 = fma(ek9_3, r0_2_1_1, g9_7);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g9_18 = fma(ek9_1, r0_2_2_0, g9_18);
              g9_16 = fma(ek9_2, r0_2_2_0, g9_16);
              g9_8 = fma(ek9_3, r0_2_2_0, g9_8);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g9_17 = fma(ek9_2, r0_3_0_1, g9_17);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g9_19 = fma(ek9_1, r0_3_1_0, g9_19);
              g9_18 = fma(ek9_2, r0_3_1_0, g9_18);
              g9_9 = fma(ek9_3, r0_3_1_0, g9_9);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g9_19 = fma(ek9_2, r0_4_0_0, g9_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g9_10 = fma(ek9_3, r0_1_1_3, g9_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g9_11 = fma(ek9_3, r0_1_2_2, g9_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g9_12 = fma(ek9_3, r0_1_3_1, g9_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_1_4_0 = X * r1_0_4_0;
              g9_13 = fma(ek9_3, r0_1_4_0, g9_13);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g9_14 = fma(ek9_3, r0_2_1_2, g9_14);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g9_15 = fma(ek9_3, r0_2_2_1, g9_15);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g9_16 = fma(ek9_3, r0_2_3_0, g9_16);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g9_17 = fma(ek9_3, r0_3_1_1, g9_17);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g9_18 = fma(ek9_3, r0_3_2_0, g9_18);
              const double r3_1_1_0 = X * r4_0_1_0;
              const double r2_2_1_0 = fma(X, r3_1_1_0, r3_0_1_0);
              const double r1_3_1_0 = fma(X, r2_2_1_0, 2.0 * r2_1_1_0);
              const double r0_4_1_0 = fma(X, r1_3_1_0, 3.0 * r1_2_1_0);
              g9_19 = fma(ek9_3, r0_4_1_0, g9_19);
            }
            { const double eb = bi[5];
              o0_9 = fma(eb, g9_0, o0_9);
            }
            { const double eb = bi[6];
              o0_9 = fma(eb, g9_3, o0_9);
            }
            { const double eb = bi[7];
              o0_9 = fma(eb, g9_9, o0_9);
            }
            { const double eb = bi[8];
              o1_9 = fma(eb, g9_0, o1_9);
            }
            { const double eb = bi[9];
              o1_9 = fma(eb, g9_3, o1_9);
            }
            { const double eb = bi[10];
              o1_9 = fma(eb, g9_9, o1_9);
            }
            { const double eb = bi[11];
              o1_9 = fma(eb, g9_19, o1_9);
            }
            { const double eb = bi[12];
              o2_9 = fma(eb, g9_0, o2_9);
            }
            { const double eb = bi[13];
              o2_9 = fma(eb, g9_2, o2_9);
            }
            { const double eb = bi[14];
              o2_9 = fma(eb, g9_3, o2_9);
            }
            { const double eb = bi[15];
              o2_9 = fma(eb, g9_8, o2_9);
            }
            { const double eb = bi[16];
              o2_9 = fma(eb, g9_9, o2_9);
            }
            { const double eb = bi[17];
              o2_9 = fma(eb, g9_18, o2_9);
            }
            { const double eb = bi[18];
              o3_9 = fma(eb, g9_0, o3_9);
            }
            { const double eb = bi[19];
              o3_9 = fma(eb, g9_1, o3_9);
            }
            { const double eb = bi[20];
              o3_9 = fma(eb, g9_3, o3_9);
            }
            { const double eb = bi[21];
              o3_9 = fma(eb, g9_7, o3_9);
            }
            { const double eb = bi[22];
              o3_9 = fma(eb, g9_9, o3_9);
            }
            { const double eb = bi[23];
              o3_9 = fma(eb, g9_17, o3_9);
            }
            { const double eb = bi[24];
              o4_9 = fma(eb, g9_0, o4_9);
            }
            { const double eb = bi[25];
              o4_9 = fma(eb, g9_2, o4_9);
            }
            { const double eb = bi[26];
              o4_9 = fma(eb, g9_6, o4_9);
            }
            { const double eb = bi[27];
              o5_9 = fma(eb, g9_0, o5_9);
            }
            { const double eb = bi[28];
              o5_9 = fma(eb, g9_2, o5_9);
            }
            { const double eb = bi[29];
              o5_9 = fma(eb, g9_6, o5_9);
            }
            { const double eb = bi[30];
              o5_9 = fma(eb, g9_3, o5_9);
            }
            { const double eb = bi[31];
              o5_9 = fma(eb, g9_8, o5_9);
            }
            { const double eb = bi[32];
              o5_9 = fma(eb, g9_16, o5_9);
            }
            { const double eb = bi[33];
              o6_9 = fma(eb, g9_0, o6_9);
            }
            { const double eb = bi[34];
              o6_9 = fma(eb, g9_2, o6_9);
            }
            { const double eb = bi[35];
              o6_9 = fma(eb, g9_6, o6_9);
            }
            { const double eb = bi[36];
              o6_9 = fma(eb, g9_13, o6_9);
            }
            { const double eb = bi[37];
              o7_9 = fma(eb, g9_0, o7_9);
            }
            { const double eb = bi[38];
              o7_9 = fma(eb, g9_1, o7_9);
            }
            { const double eb = bi[39];
              o7_9 = fma(eb, g9_2, o7_9);
            }
            { const double eb = bi[40];
              o7_9 = fma(eb, g9_5, o7_9);
            }
            { const double eb = bi[41];
              o7_9 = fma(eb, g9_6, o7_9);
            }
            { const double eb = bi[42];
              o7_9 = fma(eb, g9_12, o7_9);
            }
            { const double eb = bi[43];
              o8_9 = fma(eb, g9_0, o8_9);
            }
            { const double eb = bi[44];
              o8_9 = fma(eb, g9_1, o8_9);
            }
            { const double eb = bi[45];
              o8_9 = fma(eb, g9_4, o8_9);
            }
            { const double eb = bi[46];
              o9_9 = fma(eb, g9_0, o9_9);
            }
            { const double eb = bi[47];
              o9_9 = fma(eb, g9_1, o9_9);
            }
            { const double eb = bi[48];
              o9_9 = fma(eb, g9_4, o9_9);
            }
            { const double eb = bi[49];
              o9_9 = fma(eb, g9_3, o9_9);
            }
            { const double eb = bi[50];
              o9_9 = fma(eb, g9_7, o9_9);
            }
            { const double eb = bi[51];
              o9_9 = fma(eb, g9_14, o9_9);
            }
            { const double eb = bi[52];
              o10_9 = fma(eb, g9_0, o10_9);
            }
            { const double eb = bi[53];
              o10_9 = fma(eb, g9_1, o10_9);
            }
            { const double eb = bi[54];
              o10_9 = fma(eb, g9_4, o10_9);
            }
            { const double eb = bi[55];
              o10_9 = fma(eb, g9_2, o10_9);
            }
            { const double eb = bi[56];
              o10_9 = fma(eb, g9_5, o10_9);
            }
            { const double eb = bi[57];
              o10_9 = fma(eb, g9_11, o10_9);
            }
            { const double eb = bi[58];
              o11_9 = fma(eb, g9_0, o11_9);
            }
            { const double eb = bi[59];
              o11_9 = fma(eb, g9_1, o11_9);
            }
            { const double eb = bi[60];
              o11_9 = fma(eb, g9_4, o11_9);
            }
            { const double eb = bi[61];
              o11_9 = fma(eb, g9_10, o11_9);
            }
            { const double eb = bi[62];
              o12_9 = fma(eb, g9_0, o12_9);
            }
            { const double eb = bi[63];
              o12_9 = fma(eb, g9_2, o12_9);
            }
            { const double eb = bi[64];
              o12_9 = fma(eb, g9_3, o12_9);
            }
            { const double eb = bi[65];
              o12_9 = fma(eb, g9_8, o12_9);
            }
            { const double eb = bi[66];
              o13_9 = fma(eb, g9_0, o13_9);
            }
            { const double eb = bi[67];
              o13_9 = fma(eb, g9_2, o13_9);
            }
            { const double eb = bi[68];
              o13_9 = fma(eb, g9_3, o13_9);
            }
            { const double eb = bi[69];
              o13_9 = fma(eb, g9_8, o13_9);
            }
            { const double eb = bi[70];
              o13_9 = fma(eb, g9_9, o13_9);
            }
            { const double eb = bi[71];
              o13_9 = fma(eb, g9_18, o13_9);
            }
            { const double eb = bi[72];
              o14_9 = fma(eb, g9_0, o14_9);
            }
            { const double eb = bi[73];
              o14_9 = fma(eb, g9_2, o14_9);
            }
            { const double eb = bi[74];
              o14_9 = fma(eb, g9_6, o14_9);
            }
            { const double eb = bi[75];
              o14_9 = fma(eb, g9_3, o14_9);
            }
            { const double eb = bi[76];
              o14_9 = fma(eb, g9_8, o14_9);
            }
            { const double eb = bi[77];
              o14_9 = fma(eb, g9_16, o14_9);
            }
            { const double eb = bi[78];
              o15_9 = fma(eb, g9_0, o15_9);
            }
            { const double eb = bi[79];
              o15_9 = fma(eb, g9_1, o15_9);
            }
            { const double eb = bi[80];
              o15_9 = fma(eb, g9_2, o15_9);
            }
            { const double eb = bi[81];
              o15_9 = fma(eb, g9_5, o15_9);
            }
            { const double eb = bi[82];
              o15_9 = fma(eb, g9_3, o15_9);
            }
            { const double eb = bi[83];
              o15_9 = fma(eb, g9_7, o15_9);
            }
            { const double eb = bi[84];
              o15_9 = fma(eb, g9_8, o15_9);
            }
            { const double eb = bi[85];
              o15_9 = fma(eb, g9_15, o15_9);
            }
            { const double eb = bi[86];
              o16_9 = fma(eb, g9_0, o16_9);
            }
            { const double eb = bi[87];
              o16_9 = fma(eb, g9_1, o16_9);
            }
            { const double eb = bi[88];
              o16_9 = fma(eb, g9_3, o16_9);
            }
            { const double eb = bi[89];
              o16_9 = fma(eb, g9_7, o16_9);
            }
            { const double eb = bi[90];
              o17_9 = fma(eb, g9_0, o17_9);
            }
            { const double eb = bi[91];
              o17_9 = fma(eb, g9_1, o17_9);
            }
            { const double eb = bi[92];
              o17_9 = fma(eb, g9_3, o17_9);
            }
            { const double eb = bi[93];
              o17_9 = fma(eb, g9_7, o17_9);
            }
            { const double eb = bi[94];
              o17_9 = fma(eb, g9_9, o17_9);
            }
            { const double eb = bi[95];
              o17_9 = fma(eb, g9_17, o17_9);
            }
            { const double eb = bi[96];
              o18_9 = fma(eb, g9_0, o18_9);
            }
            { const double eb = bi[97];
              o18_9 = fma(eb, g9_1, o18_9);
            }
            { const double eb = bi[98];
              o18_9 = fma(eb, g9_2, o18_9);
            }
            { const double eb = bi[99];
              o18_9 = fma(eb, g9_5, o18_9);
            }
            { const double eb = bi[100];
              o18_9 = fma(eb, g9_3, o18_9);
            }
            { const double eb = bi[101];
              o18_9 = fma(eb, g9_7, o18_9);
            }
            { const double eb = bi[102];
              o18_9 = fma(eb, g9_8, o18_9);
            }
            { const double eb = bi[103];
              o18_9 = fma(eb, g9_15, o18_9);
            }
            { const double eb = bi[104];
              o19_9 = fma(eb, g9_0, o19_9);
            }
            { const double eb = bi[105];
              o19_9 = fma(eb, g9_1, o19_9);
            }
            { const double eb = bi[106];
              o19_9 = fma(eb, g9_4, o19_9);
            }
            { const double eb = bi[107];
              o19_9 = fma(eb, g9_3, o19_9);
            }
            { const double eb = bi[108];
              o19_9 = fma(eb, g9_7, o19_9);
            }
            { const double eb = bi[109];
              o19_9 = fma(eb, g9_14, o19_9);
            }
            { const double eb = bi[110];
              o20_9 = fma(eb, g9_0, o20_9);
            }
            { const double eb = bi[111];
              o20_9 = fma(eb, g9_1, o20_9);
            }
            { const double eb = bi[112];
              o20_9 = fma(eb, g9_2, o20_9);
            }
            { const double eb = bi[113];
              o20_9 = fma(eb, g9_5, o20_9);
            }
            { const double eb = bi[114];
              o21_9 = fma(eb, g9_0, o21_9);
            }
            { const double eb = bi[115];
              o21_9 = fma(eb, g9_1, o21_9);
            }
            { const double eb = bi[116];
              o21_9 = fma(eb, g9_2, o21_9);
            }
            { const double eb = bi[117];
              o21_9 = fma(eb, g9_5, o21_9);
            }
            { const double eb = bi[118];
              o21_9 = fma(eb, g9_3, o21_9);
            }
            { const double eb = bi[119];
              o21_9 = fma(eb, g9_7, o21_9);
            }
            { const double eb = bi[120];
              o21_9 = fma(eb, g9_8, o21_9);
            }
            { const double eb = bi[121];
              o21_9 = fma(eb, g9_15, o21_9);
            }
            { const double eb = bi[122];
              o22_9 = fma(eb, g9_0, o22_9);
            }
            { const double eb = bi[123];
              o22_9 = fma(eb, g9_1, o22_9);
            }
            { const double eb = bi[124];
              o22_9 = fma(eb, g9_2, o22_9);
            }
            { const double eb = bi[125];
              o22_9 = fma(eb, g9_5, o22_9);
            }
            { const double eb = bi[126];
              o22_9 = fma(eb, g9_6, o22_9);
            }
            { const double eb = bi[127];
              o22_9 = fma(eb, g9_12, o22_9);
            }
            { const double eb = bi[128];
              o23_9 = fma(eb, g9_0, o23_9);
            }
            { const double eb = bi[129];
              o23_9 = fma(eb, g9_1, o23_9);
            }
            { const double eb = bi[130];
              o23_9 = fma(eb, g9_4, o23_9);
            }
            { const double eb = bi[131];
              o23_9 = fma(eb, g9_2, o23_9);
            }
            { const double eb = bi[132];
              o23_9 = fma(eb, g9_5, o23_9);
            }
            { const double eb = bi[133];
              o23_9 = fma(eb, g9_11, o23_9);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_9 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 1);
            o1_9 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 1);
            o2_9 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 1);
            o3_9 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 1);
            o4_9 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 1);
            o5_9 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 1);
            o6_9 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 1);
            o7_9 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 1);
            o8_9 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 1);
            o9_9 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 1);
            o10_9 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 1);
            o11_9 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 1);
            o12_9 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 1);
            o13_9 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 1);
            o14_9 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 1);
            o15_9 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 1);
            o16_9 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 1);
            o17_9 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 1);
            o18_9 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 1);
            o19_9 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 1);
            o20_9 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 1);
            o21_9 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 1);
            o22_9 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 1);
            o23_9 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 1);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_9 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o1_9 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o2_9 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o3_9 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o4_9 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o5_9 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o6_9 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o7_9 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o8_9 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o9_9 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o10_9 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o11_9 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o12_9 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o13_9 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o14_9 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o15_9 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o16_9 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o17_9 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o18_9 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o19_9 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o20_9 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o21_9 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o22_9 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 1)));
            e = fmax(e, fabs(o23_9 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 1)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
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
            const double Bbd0_1 = PB[(fQ + 0) * N + fJ + 1];
            const double Bbd1_1 = PB[(fQ + 1) * N + fJ + 1];
            const double Bbd2_1 = PB[(fQ + 2) * N + fJ + 1];
            const double Bbd3_1 = PB[(fQ + 3) * N + fJ + 1];
            const double Bad0_1 = PB[(fP + 0) * N + fJ + 1];
            const double Bad1_1 = PB[(fP + 1) * N + fJ + 1];
            const double Bad2_1 = PB[(fP + 2) * N + fJ + 1];
            const double Bad3_1 = PB[(fP + 3) * N + fJ + 1];
            const double Bad4_1 = PB[(fP + 4) * N + fJ + 1];
            const double Bad5_1 = PB[(fP + 5) * N + fJ + 1];
            const double Bbc0_2 = PB[(fQ + 0) * N + fI + 2];
            const double Bbc1_2 = PB[(fQ + 1) * N + fI + 2];
            const double Bbc2_2 = PB[(fQ + 2) * N + fI + 2];
            const double Bbc3_2 = PB[(fQ + 3) * N + fI + 2];
            const double Bac0_2 = PB[(fP + 0) * N + fI + 2];
            const double Bac1_2 = PB[(fP + 1) * N + fI + 2];
            const double Bac2_2 = PB[(fP + 2) * N + fI + 2];
            const double Bac3_2 = PB[(fP + 3) * N + fI + 2];
            const double Bac4_2 = PB[(fP + 4) * N + fI + 2];
            const double Bac5_2 = PB[(fP + 5) * N + fI + 2];
            jab0 += o0_9 * ptk9;
            jab1 += o1_9 * ptk9;
            jab2 += o2_9 * ptk9;
            jab3 += o3_9 * ptk9;
            jab4 += o4_9 * ptk9;
            jab5 += o5_9 * ptk9;
            jab6 += o6_9 * ptk9;
            jab7 += o7_9 * ptk9;
            jab8 += o8_9 * ptk9;
            jab9 += o9_9 * ptk9;
            jab10 += o10_9 * ptk9;
            jab11 += o11_9 * ptk9;
            jab12 += o12_9 * ptk9;
            jab13 += o13_9 * ptk9;
            jab14 += o14_9 * ptk9;
            jab15 += o15_9 * ptk9;
            jab16 += o16_9 * ptk9;
            jab17 += o17_9 * ptk9;
            jab18 += o18_9 * ptk9;
            jab19 += o19_9 * ptk9;
            jab20 += o20_9 * ptk9;
            jab21 += o21_9 * ptk9;
            jab22 += o22_9 * ptk9;
            jab23 += o23_9 * ptk9;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 1, 2.0 * deg * (o0_9 * ptb0 + o1_9 * ptb1 + o2_9 * ptb2 + o3_9 * ptb3 + o4_9 * ptb4 + o5_9 * ptb5 + o6_9 * ptb6 + o7_9 * ptb7 + o8_9 * ptb8 + o9_9 * ptb9 + o10_9 * ptb10 + o11_9 * ptb11 + o12_9 * ptb12 + o13_9 * ptb13 + o14_9 * ptb14 + o15_9 * ptb15 + o16_9 * ptb16 + o17_9 * ptb17 + o18_9 * ptb18 + o19_9 * ptb19 + o20_9 * ptb20 + o21_9 * ptb21 + o22_9 * ptb22 + o23_9 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_9 * Abd0_1 + o1_9 * Abd1_1 + o2_9 * Abd2_1 + o3_9 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_9 * Aad0_1 + o4_9 * Aad1_1 + o8_9 * Aad2_1 + o12_9 * Aad3_1 + o16_9 * Aad4_1 + o20_9 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_9 * Abc0_2 + o1_9 * Abc1_2 + o2_9 * Abc2_2 + o3_9 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_9 * Aac0_2 + o4_9 * Aac1_2 + o8_9 * Aac2_2 + o12_9 * Aac3_2 + o16_9 * Aac4_2 + o20_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_9 * Aad0_1 + o5_9 * Aad1_1 + o9_9 * Aad2_1 + o13_9 * Aad3_1 + o17_9 * Aad4_1 + o21_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_9 * Aac0_2 + o5_9 * Aac1_2 + o9_9 * Aac2_2 + o13_9 * Aac3_2 + o17_9 * Aac4_2 + o21_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_9 * Aad0_1 + o6_9 * Aad1_1 + o10_9 * Aad2_1 + o14_9 * Aad3_1 + o18_9 * Aad4_1 + o22_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_9 * Aac0_2 + o6_9 * Aac1_2 + o10_9 * Aac2_2 + o14_9 * Aac3_2 + o18_9 * Aac4_2 + o22_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_9 * Aad0_1 + o7_9 * Aad1_1 + o11_9 * Aad2_1 + o15_9 * Aad3_1 + o19_9 * Aad4_1 + o23_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_9 * Aac0_2 + o7_9 * Aac1_2 + o11_9 * Aac2_2 + o15_9 * Aac3_2 + o19_9 * Aac4_2 + o23_9 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_9 * Abd0_1 + o5_9 * Abd1_1 + o6_9 * Abd2_1 + o7_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_9 * Abc0_2 + o5_9 * Abc1_2 + o6_9 * Abc2_2 + o7_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_9 * Abd0_1 + o9_9 * Abd1_1 + o10_9 * Abd2_1 + o11_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_9 * Abc0_2 + o9_9 * Abc1_2 + o10_9 * Abc2_2 + o11_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_9 * Abd0_1 + o13_9 * Abd1_1 + o14_9 * Abd2_1 + o15_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_9 * Abc0_2 + o13_9 * Abc1_2 + o14_9 * Abc2_2 + o15_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_9 * Abd0_1 + o17_9 * Abd1_1 + o18_9 * Abd2_1 + o19_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_9 * Abc0_2 + o17_9 * Abc1_2 + o18_9 * Abc2_2 + o19_9 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_9 * Abd0_1 + o21_9 * Abd1_1 + o22_9 * Abd2_1 + o23_9 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_9 * Abc0_2 + o21_9 * Abc1_2 + o22_9 * Abc2_2 + o23_9 * Abc3_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_9 * Bbd0_1 + o1_9 * Bbd1_1 + o2_9 * Bbd2_1 + o3_9 * Bbd3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_9 * Bad0_1 + o4_9 * Bad1_1 + o8_9 * Bad2_1 + o12_9 * Bad3_1 + o16_9 * Bad4_1 + o20_9 * Bad5_1));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 1, deg * (o0_9 * Bbc0_2 + o1_9 * Bbc1_2 + o2_9 * Bbc2_2 + o3_9 * Bbc3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 1, deg * (o0_9 * Bac0_2 + o4_9 * Bac1_2 + o8_9 * Bac2_2 + o12_9 * Bac3_2 + o16_9 * Bac4_2 + o20_9 * Bac5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 2, deg * (o1_9 * Bad0_1 + o5_9 * Bad1_1 + o9_9 * Bad2_1 + o13_9 * Bad3_1 + o17_9 * Bad4_1 + o21_9 * Bad5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 1, deg * (o1_9 * Bac0_2 + o5_9 * Bac1_2 + o9_9 * Bac2_2 + o13_9 * Bac3_2 + o17_9 * Bac4_2 + o21_9 * Bac5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 2, deg * (o2_9 * Bad0_1 + o6_9 * Bad1_1 + o10_9 * Bad2_1 + o14_9 * Bad3_1 + o18_9 * Bad4_1 + o22_9 * Bad5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 1, deg * (o2_9 * Bac0_2 + o6_9 * Bac1_2 + o10_9 * Bac2_2 + o14_9 * Bac3_2 + o18_9 * Bac4_2 + o22_9 * Bac5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 2, deg * (o3_9 * Bad0_1 + o7_9 * Bad1_1 + o11_9 * Bad2_1 + o15_9 * Bad3_1 + o19_9 * Bad4_1 + o23_9 * Bad5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 1, deg * (o3_9 * Bac0_2 + o7_9 * Bac1_2 + o11_9 * Bac2_2 + o15_9 * Bac3_2 + o19_9 * Bac4_2 + o23_9 * Bac5_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o4_9 * Bbd0_1 + o5_9 * Bbd1_1 + o6_9 * Bbd2_1 + o7_9 * Bbd3_1));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 1, deg * (o4_9 * Bbc0_2 + o5_9 * Bbc1_2 + o6_9 * Bbc2_2 + o7_9 * Bbc3_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o8_9 * Bbd0_1 + o9_9 * Bbd1_1 + o10_9 * Bbd2_1 + o11_9 * Bbd3_1));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 1, deg * (o8_9 * Bbc0_2 + o9_9 * Bbc1_2 + o10_9 * Bbc2_2 + o11_9 * Bbc3_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o12_9 * Bbd0_1 + o13_9 * Bbd1_1 + o14_9 * Bbd2_1 + o15_9 * Bbd3_1));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 1, deg * (o12_9 * Bbc0_2 + o13_9 * Bbc1_2 + o14_9 * Bbc2_2 + o15_9 * Bbc3_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o16_9 * Bbd0_1 + o17_9 * Bbd1_1 + o18_9 * Bbd2_1 + o19_9 * Bbd3_1));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 1, deg * (o16_9 * Bbc0_2 + o17_9 * Bbc1_2 + o18_9 * Bbc2_2 + o19_9 * Bbc3_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o20_9 * Bbd0_1 + o21_9 * Bbd1_1 + o22_9 * Bbd2_1 + o23_9 * Bbd3_1));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 1, deg * (o20_9 * Bbc0_2 + o21_9 * Bbc1_2 + o22_9 * Bbc2_2 + o23_9 * Bbc3_2));
          }
        } break;
        case 10: {  // ket functions [10]
          double o0_10 = 0;
          double o1_10 = 0;
          double o2_10 = 0;
          double o3_10 = 0;
          double o4_10 = 0;
          double o5_10 = 0;
          double o6_10 = 0;
          double o7_10 = 0;
          double o8_10 = 0;
          double o9_10 = 0;
          double o10_10 = 0;
          double o11_10 = 0;
          double o12_10 = 0;
          double o13_10 = 0;
          double o14_10 = 0;
          double o15_10 = 0;
          double o16_10 = 0;
          double o17_10 = 0;
          double o18_10 = 0;
          double o19_10 = 0;
          double o20_10 = 0;
          double o21_10 = 0;
          double o22_10 = 0;
          double o23_10 = 0;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek10_0 = kj[31 * kS];
              const double ek10_1 = -kj[32 * kS];
              const double ek10_2 = kj[33 * kS];
              g10_0 = fma(ek10_0, b0, g10_0);
              const double r0_0_0_1 = Z * b1;
              g10_1 = fma(ek10_0, r0_0_0_1, g10_1);
              const double r0_0_1_0 = Y * b1;
              g10_2 = fma(ek10_0, r0_0_1_0, g10_2);
              g10_0 = fma(ek10_1, r0_0_1_0, g10_0);
              const double r0_1_0_0 = X * b1;
              g10_3 = fma(ek10_0, r0_1_0_0, g10_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g10_4 = fma(ek10_0, r0_0_0_2, g10_4);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g10_5 = fma(ek10_0, r0_0_1_1, g10_5);
              g10_1 = fma(ek10_1, r0_0_1_1, g10_1);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g10_6 = fma(ek10_0, r0_0_2_0, g10_6);
              g10_2 = fma(ek10_1, r0_0_2_0, g10_2);
              g10_0 = fma(ek10_2, r0_0_2_0, g10_0);
              const double r0_1_0_1 = X * r1_0_0_1;
              g10_7 = fma(ek10_0, r0_1_0_1, g10_7);
              const double r0_1_1_0 = X * r1_0_1_0;
              g10_8 = fma(ek10_0, r0_1_1_0, g10_8);
              g10_3 = fma(ek10_1, r0_1_1_0, g10_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g10_9 = fma(ek10_0, r0_2_0_0, g10_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g10_10 = fma(ek10_0, r0_0_0_3, g10_10);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g10_11 = fma(ek10_0, r0_0_1_2, g10_11);
              g10_4 = fma(ek10_1, r0_0_1_2, g10_4);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g10_12 = fma(ek10_0, r0_0_2_1, g10_12);
              g10_5 = fma(ek10_1, r0_0_2_1, g10_5);
              g10_1 = fma(ek10_2, r0_0_2_1, g10_1);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g10_13 = fma(ek10_0, r0_0_3_0, g10_13);
              g10_6 = fma(ek10_1, r0_0_3_0, g10_6);
              g10_2 = fma(ek10_2, r0_0_3_0, g10_2);
              const double r0_1_0_2 = X * r1_0_0_2;
              g10_14 = fma(ek10_0, r0_1_0_2, g10_14);
              const double r0_1_1_1 = X * r1_0_1_1;
              g10_15 = fma(ek10_0, r0_1_1_1, g10_15);
              g10_7 = fma(ek10_1, r0_1_1_1, g10_7);
              const double r0_1_2_0 = X * r1_0_2_0;
              g10_16 = fma(ek10_0, r0_1_2_0, g10_16);
              g10_8 = fma(ek10_1, r0_1_2_0, g10_8);
              g10_3 = fma(ek10_2, r0_1_2_0, g10_3);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g10_17 = fma(ek10_0, r0_2_0_1, g10_17);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g10_18 = fma(ek10_0, r0_2_1_0, g10_18);
              g10_9 = fma(ek10_1, r0_2_1_0, g10_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g10_19 = fma(ek10_0, r0_3_0_0, g10_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g10_10 = fma(ek10_1, r0_0_1_3, g10_10);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g10_11 = fma(ek10_1, r0_0_2_2, g10_11);
              g10_4 = fma(ek10_2, r0_0_2_2, g10_4);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g10_12 = fma(ek10_1, r0_0_3_1, g10_12);
              g10_5 = fma(ek10_2, r0_0_3_1, g10_5);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g10_13 = fma(ek10_1, r0_0_4_0, g10_13);
              g10_6 = fma(ek10_2, r0_0_4_0, g10_6);
              const double r0_1_1_2 = X * r1_0_1_2;
              g10_14 = fma(ek10_1, r0_1_1_2, g10_14);
              const double r0_1_2_1 = X * r1_0_2_1;
              g10_15 = fma(ek10_1, r0_1_2_1, g10_15);
              g10_7 = fma(ek10_2, r0_1_2_1, g10_7);
              const double r0_1_3_0 = X * r1_0_3_0;
              g10_16 = fma(ek10_1, r0_1_3_0, g10_16);
              g10_8 = fma(ek10_2, r0_1_3_0, g10_8);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g10_17 = fma(ek10_1, r0_2_1_1, g10_17);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g10_18 = fma(ek10_1, r0_2_2_0, g10_18);
              g10_9 = fma(ek10_2, r0_2_2_0, g10_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g10_19 = fma(ek10_1, r0_3_1_0, g10_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g10_10 = fma(ek10_2, r0_0_2_3, g10_10);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g10_11 = fma(ek10_2, r0_0_3_2, g10_11);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g10_12 = fma(ek10_2, r0_0_4_1, g10_12);
              const double r4_0_1_0 = Y * b5;
              const double r3_0_2_0 = fma(Y, r4_0_1_0, b4);
              const double r2_0_3_0 = fma(Y, r3_0_2_0, 2.0 * r3_0_1_0);
              const double r1_0_4_0 = fma(Y, r2_0_3_0, 3.0 * r2_0_2_0);
              const double r0_0_5_0 = fma(Y, r1_0_4_0, 4.0 * r1_0_3_0);
              g10_13 = fma(ek10_2, r0_0_5_0, g10_13);
              const double r0_1_2_2 = X * r1_0_2_2;
              g10_14 = fma(ek10_2, r0_1_2_2, g10_14);
              const double r0_1_3_1 = X * r1_0_3_1;
              g10_15 = fma(ek10_2, r0_1_3_1, g10_15);
              const double r0_1_4_0 = X * r1_0_4_0;
              g10_16 = fma(ek10_2, r0_1_4_0, g10_16);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g10_17 = fma(ek10_2, r0_2_2_1, g10_17);
              const double r1_1_3_0 = X * r2_0_3_0;
              const double r0_2_3_0 = fma(X, r1_1_3_0, r1_0_3_0);
              g10_18 = fma(ek10_2, r0_2_3_0, g10_18);
              const double r2_1_2_0 = X * r3_0_2_0;
              const double r1_2_2_0 = fma(X, r2_1_2_0, r2_0_2_0);
              const double r0_3_2_0 = fma(X, r1_2_2_0, 2.0 * r1_1_2_0);
              g10_19 = fma(ek10_2, r0_3_2_0, g10_19);
            }
            { const double eb = bi[5];
              o0_10 = fma(eb, g10_0, o0_10);
            }
            { const double eb = bi[6];
              o0_10 = fma(eb, g10_3, o0_10);
            }
            { const double eb = bi[7];
              o0_10 = fma(eb, g10_9, o0_10);
            }
            { const double eb = bi[8];
              o1_10 = fma(eb, g10_0, o1_10);
            }
            { const double eb = bi[9];
              o1_10 = fma(eb, g10_3, o1_10);
            }
            { const double eb = bi[10];
              o1_10 = fma(eb, g10_9, o1_10);
            }
            { const double eb = bi[11];
              o1_10 = fma(eb, g10_19, o1_10);
            }
            { const double eb = bi[12];
              o2_10 = fma(eb, g10_0, o2_10);
            }
            { const double eb = bi[13];
              o2_10 = fma(eb, g10_2, o2_10);
            }
            { const double eb = bi[14];
              o2_10 = fma(eb, g10_3, o2_10);
            }
            { const double eb = bi[15];
              o2_10 = fma(eb, g10_8, o2_10);
            }
            { const double eb = bi[16];
              o2_10 = fma(eb, g10_9, o2_10);
            }
            { const double eb = bi[17];
              o2_10 = fma(eb, g10_18, o2_10);
            }
            { const double eb = bi[18];
              o3_10 = fma(eb, g10_0, o3_10);
            }
            { const double eb = bi[19];
              o3_10 = fma(eb, g10_1, o3_10);
            }
            { const double eb = bi[20];
              o3_10 = fma(eb, g10_3, o3_10);
            }
            { const double eb = bi[21];
              o3_10 = fma(eb, g10_7, o3_10);
            }
            { const double eb = bi[22];
              o3_10 = fma(eb, g10_9, o3_10);
            }
            { const double eb = bi[23];
              o3_10 = fma(eb, g10_17, o3_10);
            }
            { const double eb = bi[24];
              o4_10 = fma(eb, g10_0, o4_10);
            }
            { const double eb = bi[25];
              o4_10 = fma(eb, g10_2, o4_10);
            }
            { const double eb = bi[26];
              o4_10 = fma(eb, g10_6, o4_10);
            }
            { const double eb = bi[27];
              o5_10 = fma(eb, g10_0, o5_10);
            }
            { const double eb = bi[28];
              o5_10 = fma(eb, g10_2, o5_10);
            }
            { const double eb = bi[29];
              o5_10 = fma(eb, g10_6, o5_10);
            }
            { const double eb = bi[30];
              o5_10 = fma(eb, g10_3, o5_10);
            }
            { const double eb = bi[31];
              o5_10 = fma(eb, g10_8, o5_10);
            }
            { const double eb = bi[32];
              o5_10 = fma(eb, g10_16, o5_10);
            }
            { const double eb = bi[33];
              o6_10 = fma(eb, g10_0, o6_10);
            }
            { const double eb = bi[34];
              o6_10 = fma(eb, g10_2, o6_10);
            }
            { const double eb = bi[35];
              o6_10 = fma(eb, g10_6, o6_10);
            }
            { const double eb = bi[36];
              o6_10 = fma(eb, g10_13, o6_10);
            }
            { const double eb = bi[37];
              o7_10 = fma(eb, g10_0, o7_10);
            }
            { const double eb = bi[38];
              o7_10 = fma(eb, g10_1, o7_10);
            }
            { const double eb = bi[39];
              o7_10 = fma(eb, g10_2, o7_10);
            }
            { const double eb = bi[40];
              o7_10 = fma(eb, g10_5, o7_10);
            }
            { const double eb = bi[41];
              o7_10 = fma(eb, g10_6, o7_10);
            }
            { const double eb = bi[42];
              o7_10 = fma(eb, g10_12, o7_10);
            }
            { const double eb = bi[43];
              o8_10 = fma(eb, g10_0, o8_10);
            }
            { const double eb = bi[44];
              o8_10 = fma(eb, g10_1, o8_10);
            }
            { const double eb = bi[45];
              o8_10 = fma(eb, g10_4, o8_10);
            }
            { const double eb = bi[46];
              o9_10 = fma(eb, g10_0, o9_10);
            }
            { const double eb = bi[47];
              o9_10 = fma(eb, g10_1, o9_10);
            }
            { const double eb = bi[48];
              o9_10 = fma(eb, g10_4, o9_10);
            }
            { const double eb = bi[49];
              o9_10 = fma(eb, g10_3, o9_10);
            }
            { const double eb = bi[50];
              o9_10 = fma(eb, g10_7, o9_10);
            }
            { const double eb = bi[51];
              o9_10 = fma(eb, g10_14, o9_10);
            }
            { const double eb = bi[52];
              o10_10 = fma(eb, g10_0, o10_10);
            }
            { const double eb = bi[53];
              o10_10 = fma(eb, g10_1, o10_10);
            }
            { const double eb = bi[54];
              o10_10 = fma(eb, g10_4, o10_10);
            }
            { const double eb = bi[55];
              o10_10 = fma(eb, g10_2, o10_10);
            }
            { const double eb = bi[56];
              o10_10 = fma(eb, g10_5, o10_10);
            }
            { const double eb = bi[57];
              o10_10 = fma(eb, g10_11, o10_10);
            }
            { const double eb = bi[58];
              o11_10 = fma(eb, g10_0, o11_10);
            }
            { const double eb = bi[59];
              o11_10 = fma(eb, g10_1, o11_10);
            }
            { const double eb = bi[60];
              o11_10 = fma(eb, g10_4, o11_10);
            }
            { const double eb = bi[61];
              o11_10 = fma(eb, g10_10, o11_10);
            }
            { const double eb = bi[62];
              o12_10 = fma(eb, g10_0, o12_10);
            }
            { const double eb = bi[63];
              o12_10 = fma(eb, g10_2, o12_10);
            }
            { const double eb = bi[64];
              o12_10 = fma(eb, g10_3, o12_10);
            }
            { const double eb = bi[65];
              o12_10 = fma(eb, g10_8, o12_10);
            }
            { const double eb = bi[66];
              o13_10 = fma(eb, g10_0, o13_10);
            }
            { const double eb = bi[67];
              o13_10 = fma(eb, g10_2, o13_10);
            }
            { const double eb = bi[68];
              o13_10 = fma(eb, g10_3, o13_10);
            }
            { const double eb = bi[69];
              o13_10 = fma(eb, g10_8, o13_10);
            }
            { const double eb = bi[70];
              o13_10 = fma(eb, g10_9, o13_10);
            }
            { const double eb = bi[71];
              o13_10 = fma(eb, g10_18, o13_10);
            }
            { const double eb = bi[72];
              o14_10 = fma(eb, g10_0, o14_10);
            }
            { const double eb = bi[73];
              o14_10 = fma(eb, g10_2, o14_10);
            }
            { const double eb = bi[74];
              o14_10 = fma(eb, g10_6, o14_10);
            }
            { const double eb = bi[75];
              o14_10 = fma(eb, g10_3, o14_10);
            }
            { const double eb = bi[76];
              o14_10 = fma(eb, g10_8, o14_10);
            }
            { const double eb = bi[77];
              o14_10 = fma(eb, g10_16, o14_10);
            }
            { const double eb = bi[78];
              o15_10 = fma(eb, g10_0, o15_10);
            }
            { const double eb = bi[79];
              o15_10 = fma(eb, g10_1, o15_10);
            }
            { const double eb = bi[80];
              o15_10 = fma(eb, g10_2, o15_10);
            }
            { const double eb = bi[81];
              o15_10 = fma(eb, g10_5, o15_10);
            }
            { const double eb = bi[82];
              o15_10 = fma(eb, g10_3, o15_10);
            }
            { const double eb = bi[83];
              o15_10 = fma(eb, g10_7, o15_10);
            }
            { const double eb = bi[84];
              o15_10 = fma(eb, g10_8, o15_10);
            }
            { const double eb = bi[85];
              o15_10 = fma(eb, g10_15, o15_10);
            }
            { const double eb = bi[86];
              o16_10 = fma(eb, g10_0, o16_10);
            }
            { const double eb = bi[87];
              o16_10 = fma(eb, g10_1, o16_10);
            }
            { const double eb = bi[88];
              o16_10 = fma(eb, g10_3, o16_10);
            }
            { const double eb = bi[89];
              o16_10 = fma(eb, g10_7, o16_10);
            }
            { const double eb = bi[90];
              o17_10 = fma(eb, g10_0, o17_10);
            }
            { const double eb = bi[91];
              o17_10 = fma(eb, g10_1, o17_10);
            }
            { const double eb = bi[92];
              o17_10 = fma(eb, g10_3, o17_10);
            }
            { const double eb = bi[93];
              o17_10 = fma(eb, g10_7, o17_10);
            }
            { const double eb = bi[94];
              o17_10 = fma(eb, g10_9, o17_10);
            }
            { const double eb = bi[95];
              o17_10 = fma(eb, g10_17, o17_10);
            }
            { const double eb = bi[96];
              o18_10 = fma(eb, g10_0, o18_10);
            }
            { const double eb = bi[97];
              o18_10 = fma(eb, g10_1, o18_10);
            }
            { const double eb = bi[98];
              o18_10 = fma(eb, g10_2, o18_10);
            }
            { const double eb = bi[99];
              o18_10 = fma(eb, g10_5, o18_10);
            }
            { const double eb = bi[100];
              o18_10 = fma(eb, g10_3, o18_10);
            }
            { const double eb = bi[101];
              o18_10 = fma(eb, g10_7, o18_10);
            }
            { const double eb = bi[102];
              o18_10 = fma(eb, g10_8, o18_10);
            }
            { const double eb = bi[103];
              o18_10 = fma(eb, g10_15, o18_10);
            }
            { const double eb = bi[104];
              o19_10 = fma(eb, g10_0, o19_10);
            }
            { const double eb = bi[105];
              o19_10 = fma(eb, g10_1, o19_10);
            }
            { const double eb = bi[106];
              o19_10 = fma(eb, g10_4, o19_10);
            }
            { const double eb = bi[107];
              o19_10 = fma(eb, g10_3, o19_10);
            }
            { const double eb = bi[108];
              o19_10 = fma(eb, g10_7, o19_10);
            }
            { const double eb = bi[109];
              o19_10 = fma(eb, g10_14, o19_10);
            }
            { const double eb = bi[110];
              o20_10 = fma(eb, g10_0, o20_10);
            }
            { const double eb = bi[111];
              o20_10 = fma(eb, g10_1, o20_10);
            }
            { const double eb = bi[112];
              o20_10 = fma(eb, g10_2, o20_10);
            }
            { const double eb = bi[113];
              o20_10 = fma(eb, g10_5, o20_10);
            }
            { const double eb = bi[114];
              o21_10 = fma(eb, g10_0, o21_10);
            }
            { const double eb = bi[115];
              o21_10 = fma(eb, g10_1, o21_10);
            }
            { const double eb = bi[116];
              o21_10 = fma(eb, g10_2, o21_10);
            }
            { const double eb = bi[117];
              o21_10 = fma(eb, g10_5, o21_10);
            }
            { const double eb = bi[118];
              o21_10 = fma(eb, g10_3, o21_10);
            }
            { const double eb = bi[119];
              o21_10 = fma(eb, g10_7, o21_10);
            }
            { const double eb = bi[120];
              o21_10 = fma(eb, g10_8, o21_10);
            }
            { const double eb = bi[121];
              o21_10 = fma(eb, g10_15, o21_10);
            }
            { const double eb = bi[122];
              o22_10 = fma(eb, g10_0, o22_10);
            }
            { const double eb = bi[123];
              o22_10 = fma(eb, g10_1, o22_10);
            }
            { const double eb = bi[124];
              o22_10 = fma(eb, g10_2, o22_10);
            }
            { const double eb = bi[125];
              o22_10 = fma(eb, g10_5, o22_10);
            }
            { const double eb = bi[126];
              o22_10 = fma(eb, g10_6, o22_10);
            }
            { const double eb = bi[127];
              o22_10 = fma(eb, g10_12, o22_10);
            }
            { const double eb = bi[128];
              o23_10 = fma(eb, g10_0, o23_10);
            }
            { const double eb = bi[129];
              o23_10 = fma(eb, g10_1, o23_10);
            }
            { const double eb = bi[130];
              o23_10 = fma(eb, g10_4, o23_10);
            }
            { const double eb = bi[131];
              o23_10 = fma(eb, g10_2, o23_10);
            }
            { const double eb = bi[132];
              o23_10 = fma(eb, g10_5, o23_10);
            }
            { const double eb = bi[133];
              o23_10 = fma(eb, g10_11, o23_10);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_10 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 2);
            o1_10 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 2);
            o2_10 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 2);
            o3_10 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 2);
            o4_10 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 2);
            o5_10 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 2);
            o6_10 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 2);
            o7_10 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 2);
            o8_10 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 2);
            o9_10 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 2);
            o10_10 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 2);
            o11_10 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 2);
            o12_10 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 2);
            o13_10 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 2);
            o14_10 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 2);
            o15_10 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 2);
            o16_10 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 2);
            o17_10 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 2);
            o18_10 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 2);
            o19_10 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 2);
            o20_10 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 2);
            o21_10 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 2);
            o22_10 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 2);
            o23_10 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 2);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_10 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o1_10 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o2_10 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o3_10 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o4_10 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o5_10 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o6_10 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o7_10 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o8_10 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o9_10 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o10_10 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o11_10 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o12_10 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o13_10 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o14_10 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o15_10 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o16_10 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o17_10 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o18_10 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o19_10 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o20_10 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o21_10 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o22_10 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 2)));
            e = fmax(e, fabs(o23_10 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 2)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk10 = PT[(fI + 2) * N + fJ + 2];
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
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
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
            const double Bbd0_2 = PB[(fQ + 0) * N + fJ + 2];
            const double Bbd1_2 = PB[(fQ + 1) * N + fJ + 2];
            const double Bbd2_2 = PB[(fQ + 2) * N + fJ + 2];
            const double Bbd3_2 = PB[(fQ + 3) * N + fJ + 2];
            const double Bad0_2 = PB[(fP + 0) * N + fJ + 2];
            const double Bad1_2 = PB[(fP + 1) * N + fJ + 2];
            const double Bad2_2 = PB[(fP + 2) * N + fJ + 2];
            const double Bad3_2 = PB[(fP + 3) * N + fJ + 2];
            const double Bad4_2 = PB[(fP + 4) * N + fJ + 2];
            const double Bad5_2 = PB[(fP + 5) * N + fJ + 2];
            const double Bbc0_2 = PB[(fQ + 0) * N + fI + 2];
            const double Bbc1_2 = PB[(fQ + 1) * N + fI + 2];
            const double Bbc2_2 = PB[(fQ + 2) * N + fI + 2];
            const double Bbc3_2 = PB[(fQ + 3) * N + fI + 2];
            const double Bac0_2 = PB[(fP + 0) * N + fI + 2];
            const double Bac1_2 = PB[(fP + 1) * N + fI + 2];
            const double Bac2_2 = PB[(fP + 2) * N + fI + 2];
            const double Bac3_2 = PB[(fP + 3) * N + fI + 2];
            const double Bac4_2 = PB[(fP + 4) * N + fI + 2];
            const double Bac5_2 = PB[(fP + 5) * N + fI + 2];
            jab0 += o0_10 * ptk10;
            jab1 += o1_10 * ptk10;
            jab2 += o2_10 * ptk10;
            jab3 += o3_10 * ptk10;
            jab4 += o4_10 * ptk10;
            jab5 += o5_10 * ptk10;
            jab6 += o6_10 * ptk10;
            jab7 += o7_10 * ptk10;
            jab8 += o8_10 * ptk10;
            jab9 += o9_10 * ptk10;
            jab10 += o10_10 * ptk10;
            jab11 += o11_10 * ptk10;
            jab12 += o12_10 * ptk10;
            jab13 += o13_10 * ptk10;
            jab14 += o14_10 * ptk10;
            jab15 += o15_10 * ptk10;
            jab16 += o16_10 * ptk10;
            jab17 += o17_10 * ptk10;
            jab18 += o18_10 * ptk10;
            jab19 += o19_10 * ptk10;
            jab20 += o20_10 * ptk10;
            jab21 += o21_10 * ptk10;
            jab22 += o22_10 * ptk10;
            jab23 += o23_10 * ptk10;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 2, 2.0 * deg * (o0_10 * ptb0 + o1_10 * ptb1 + o2_10 * ptb2 + o3_10 * ptb3 + o4_10 * ptb4 + o5_10 * ptb5 + o6_10 * ptb6 + o7_10 * ptb7 + o8_10 * ptb8 + o9_10 * ptb9 + o10_10 * ptb10 + o11_10 * ptb11 + o12_10 * ptb12 + o13_10 * ptb13 + o14_10 * ptb14 + o15_10 * ptb15 + o16_10 * ptb16 + o17_10 * ptb17 + o18_10 * ptb18 + o19_10 * ptb19 + o20_10 * ptb20 + o21_10 * ptb21 + o22_10 * ptb22 + o23_10 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_10 * Abd0_2 + o1_10 * Abd1_2 + o2_10 * Abd2_2 + o3_10 * Abd3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_10 * Aad0_2 + o4_10 * Aad1_2 + o8_10 * Aad2_2 + o12_10 * Aad3_2 + o16_10 * Aad4_2 + o20_10 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_10 * Abc0_2 + o1_10 * Abc1_2 + o2_10 * Abc2_2 + o3_10 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_10 * Aac0_2 + o4_10 * Aac1_2 + o8_10 * Aac2_2 + o12_10 * Aac3_2 + o16_10 * Aac4_2 + o20_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_10 * Aad0_2 + o5_10 * Aad1_2 + o9_10 * Aad2_2 + o13_10 * Aad3_2 + o17_10 * Aad4_2 + o21_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_10 * Aac0_2 + o5_10 * Aac1_2 + o9_10 * Aac2_2 + o13_10 * Aac3_2 + o17_10 * Aac4_2 + o21_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_10 * Aad0_2 + o6_10 * Aad1_2 + o10_10 * Aad2_2 + o14_10 * Aad3_2 + o18_10 * Aad4_2 + o22_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_10 * Aac0_2 + o6_10 * Aac1_2 + o10_10 * Aac2_2 + o14_10 * Aac3_2 + o18_10 * Aac4_2 + o22_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_10 * Aad0_2 + o7_10 * Aad1_2 + o11_10 * Aad2_2 + o15_10 * Aad3_2 + o19_10 * Aad4_2 + o23_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_10 * Aac0_2 + o7_10 * Aac1_2 + o11_10 * Aac2_2 + o15_10 * Aac3_2 + o19_10 * Aac4_2 + o23_10 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_10 * Abd0_2 + o5_10 * Abd1_2 + o6_10 * Abd2_2 + o7_10 * Abd3_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_10 * Abc0_2 + o5_10 * Abc1_2 + o6_10 * Abc2_2 + o7_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_10 * Abd0_2 + o9_10 * Abd1_2 + o10_10 * Abd2_2 + o11_10 * Abd3_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_10 * Abc0_2 + o9_10 * Abc1_2 + o10_10 * Abc2_2 + o11_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_10 * Abd0_2 + o13_10 * Abd1_2 + o14_10 * Abd2_2 + o15_10 * Abd3_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_10 * Abc0_2 + o13_10 * Abc1_2 + o14_10 * Abc2_2 + o15_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_10 * Abd0_2 + o17_10 * Abd1_2 + o18_10 * Abd2_2 + o19_10 * Abd3_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_10 * Abc0_2 + o17_10 * Abc1_2 + o18_10 * Abc2_2 + o19_10 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_10 * Abd0_2 + o21_10 * Abd1_2 + o22_10 * Abd2_2 + o23_10 * Abd3_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_10 * Abc0_2 + o21_10 * Abc1_2 + o22_10 * Abc2_2 + o23_10 * Abc3_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_10 * Bbd0_2 + o1_10 * Bbd1_2 + o2_10 * Bbd2_2 + o3_10 * Bbd3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_10 * Bad0_2 + o4_10 * Bad1_2 + o8_10 * Bad2_2 + o12_10 * Bad3_2 + o16_10 * Bad4_2 + o20_10 * Bad5_2));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 2, deg * (o0_10 * Bbc0_2 + o1_10 * Bbc1_2 + o2_10 * Bbc2_2 + o3_10 * Bbc3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 2, deg * (o0_10 * Bac0_2 + o4_10 * Bac1_2 + o8_10 * Bac2_2 + o12_10 * Bac3_2 + o16_10 * Bac4_2 + o20_10 * Bac5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 2, deg * (o1_10 * Bad0_2 + o5_10 * Bad1_2 + o9_10 * Bad2_2 + o13_10 * Bad3_2 + o17_10 * Bad4_2 + o21_10 * Bad5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 2, deg * (o1_10 * Bac0_2 + o5_10 * Bac1_2 + o9_10 * Bac2_2 + o13_10 * Bac3_2 + o17_10 * Bac4_2 + o21_10 * Bac5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 2, deg * (o2_10 * Bad0_2 + o6_10 * Bad1_2 + o10_10 * Bad2_2 + o14_10 * Bad3_2 + o18_10 * Bad4_2 + o22_10 * Bad5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 2, deg * (o2_10 * Bac0_2 + o6_10 * Bac1_2 + o10_10 * Bac2_2 + o14_10 * Bac3_2 + o18_10 * Bac4_2 + o22_10 * Bac5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 2, deg * (o3_10 * Bad0_2 + o7_10 * Bad1_2 + o11_10 * Bad2_2 + o15_10 * Bad3_2 + o19_10 * Bad4_2 + o23_10 * Bad5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 2, deg * (o3_10 * Bac0_2 + o7_10 * Bac1_2 + o11_10 * Bac2_2 + o15_10 * Bac3_2 + o19_10 * Bac4_2 + o23_10 * Bac5_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o4_10 * Bbd0_2 + o5_10 * Bbd1_2 + o6_10 * Bbd2_2 + o7_10 * Bbd3_2));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 2, deg * (o4_10 * Bbc0_2 + o5_10 * Bbc1_2 + o6_10 * Bbc2_2 + o7_10 * Bbc3_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o8_10 * Bbd0_2 + o9_10 * Bbd1_2 + o10_10 * Bbd2_2 + o11_10 * Bbd3_2));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 2, deg * (o8_10 * Bbc0_2 + o9_10 * Bbc1_2 + o10_10 * Bbc2_2 + o11_10 * Bbc3_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o12_10 * Bbd0_2 + o13_10 * Bbd1_2 + o14_10 * Bbd2_2 + o15_10 * Bbd3_2));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 2, deg * (o12_10 * Bbc0_2 + o13_10 * Bbc1_2 + o14_10 * Bbc2_2 + o15_10 * Bbc3_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o16_10 * Bbd0_2 + o17_10 * Bbd1_2 + o18_10 * Bbd2_2 + o19_10 * Bbd3_2));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 2, deg * (o16_10 * Bbc0_2 + o17_10 * Bbc1_2 + o18_10 * Bbc2_2 + o19_10 * Bbc3_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o20_10 * Bbd0_2 + o21_10 * Bbd1_2 + o22_10 * Bbd2_2 + o23_10 * Bbd3_2));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 2, deg * (o20_10 * Bbc0_2 + o21_10 * Bbc1_2 + o22_10 * Bbc2_2 + o23_10 * Bbc3_2));
          }
        } break;
        case 11: {  // ket functions [11]
          double o0_11 = 0;
          double o1_11 = 0;
          double o2_11 = 0;
          double o3_11 = 0;
          double o4_11 = 0;
          double o5_11 = 0;
          double o6_11 = 0;
          double o7_11 = 0;
          double o8_11 = 0;
          double o9_11 = 0;
          double o10_11 = 0;
          double o11_11 = 0;
          double o12_11 = 0;
          double o13_11 = 0;
          double o14_11 = 0;
          double o15_11 = 0;
          double o16_11 = 0;
          double o17_11 = 0;
          double o18_11 = 0;
          double o19_11 = 0;
          double o20_11 = 0;
          double o21_11 = 0;
          double o22_11 = 0;
          double o23_11 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek11_0 = kj[34 * kS];
              const double ek11_1 = -kj[35 * kS];
              const double ek11_2 = -kj[36 * kS];
              const double ek11_3 = kj[37 * kS];
              g11_0 = fma(ek11_0, b0, g11_0);
              const double r0_0_0_1 = Z * b1;
              g11_1 = fma(ek11_0, r0_0_0_1, g11_1);
              g11_0 = fma(ek11_1, r0_0_0_1, g11_0);
              const double r0_0_1_0 = Y * b1;
              g11_2 = fma(ek11_0, r0_0_1_0, g11_2);
              g11_0 = fma(ek11_2, r0_0_1_0, g11_0);
              const double r0_1_0_0 = X * b1;
              g11_3 = fma(ek11_0, r0_1_0_0, g11_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g11_4 = fma(ek11_0, r0_0_0_2, g11_4);
              g11_1 = fma(ek11_1, r0_0_0_2, g11_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g11_5 = fma(ek11_0, r0_0_1_1, g11_5);
              g11_2 = fma(ek11_1, r0_0_1_1, g11_2);
              g11_1 = fma(ek11_2, r0_0_1_1, g11_1);
              g11_0 = fma(ek11_3, r0_0_1_1, g11_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g11_6 = fma(ek11_0, r0_0_2_0, g11_6);
              g11_2 = fma(ek11_2, r0_0_2_0, g11_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g11_7 = fma(ek11_0, r0_1_0_1, g11_7);
              g11_3 = fma(ek11_1, r0_1_0_1, g11_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g11_8 = fma(ek11_0, r0_1_1_0, g11_8);
              g11_3 = fma(ek11_2, r0_1_1_0, g11_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g11_9 = fma(ek11_0, r0_2_0_0, g11_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g11_10 = fma(ek11_0, r0_0_0_3, g11_10);
              g11_4 = fma(ek11_1, r0_0_0_3, g11_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g11_11 = fma(ek11_0, r0_0_1_2, g11_11);
              g11_5 = fma(ek11_1, r0_0_1_2, g11_5);
              g11_4 = fma(ek11_2, r0_0_1_2, g11_4);
              g11_1 = fma(ek11_3, r0_0_1_2, g11_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g11_12 = fma(ek11_0, r0_0_2_1, g11_12);
              g11_6 = fma(ek11_1, r0_0_2_1, g11_6);
              g11_5 = fma(ek11_2, r0_0_2_1, g11_5);
              g11_2 = fma(ek11_3, r0_0_2_1, g11_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g11_13 = fma(ek11_0, r0_0_3_0, g11_13);
              g11_6 = fma(ek11_2, r0_0_3_0, g11_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g11_14 = fma(ek11_0, r0_1_0_2, g11_14);
              g11_7 = fma(ek11_1, r0_1_0_2, g11_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g11_15 = fma(ek11_0, r0_1_1_1, g11_15);
              g11_8 = fma(ek11_1, r0_1_1_1, g11_8);
              g11_7 = fma(ek11_2, r0_1_1_1, g11_7);
              g11_3 = fma(ek11_3, r0_1_1_1, g11_3);
              const double r0_1_2_0 = X * r1_0_2_0;
              g11_16 = fma(ek11_0, r0_1_2_0, g11_16);
              g11_8 = fma(ek11_2, r0_1_2_0, g11_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g11_17 = fma(ek11_0, r0_2_0_1, g11_17);
              g11_9 = fma(ek11_1, r0_2_0_1, g11_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g11_18 = fma(ek11_0, r0_2_1_0, g11_18);
              g11_9 = fma(ek11_2, r0_2_1_0, g11_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g11_19 = fma(ek11_0, r0_3_0_0, g11_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g11_10 = fma(ek11_1, r0_0_0_4, g11_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g11_11 = fma(ek11_1, r0_0_1_3, g11_11);
              g11_10 = fma(ek11_2, r0_0_1_3, g11_10);
              g11_4 = fma(ek11_3, r0_0_1_3, g11_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g11_12 = fma(ek11_1, r0_0_2_2, g11_12);
              g11_11 = fma(ek11_2, r0_0_2_2, g11_11);
              g11_5 = fma(ek11_3, r0_0_2_2, g11_5);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g11_13 = fma(ek11_1, r0_0_3_1, g11_13);
              g11_12 = fma(ek11_2, r0_0_3_1, g11_12);
              g11_6 = fma(ek11_3, r0_0_3_1, g11_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g11_13 = fma(ek11_2, r0_0_4_0, g11_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g11_14 = fma(ek11_1, r0_1_0_3, g11_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g11_15 = fma(ek11_1, r0_1_1_2, g11_15);
              g11_14 = fma(ek11_2, r0_1_1_2, g11_14);
              g11_7 = fma(ek11_3, r0_1_1_2, g11_7);
              const double r0_1_2_1 = X * r1_0_2_1;
              g11_16 = fma(ek11_1, r0_1_2_1, g11_16);
              g11_15 = fma(ek11_2, r0_1_2_1, g11_15);
              g11_8 = fma(ek11_3, r0_1_2_1, g11_8);
              const double r0_1_3_0 = X * r1_0_3_0;
              g11_16 = fma(ek11_2, r0_1_3_0, g11_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g11_17 = fma(ek11_1, r0_2_0_2, g11_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g11_18 = fma(ek11_1, r0_2_1_1, g11_18);
              g11_17 = fma(ek11_2, r0_2_1_1, g11_17);
              g11_9 = fma(ek11_3, r0_2_1_1, g11_9);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g11_18 = fma(ek11_2, r0_2_2_0, g11_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g11_19 = fma(ek11_1, r0_3_0_1, g11_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g11_19 = fma(ek11_2, r0_3_1_0, g11_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g11_10 = fma(ek11_3, r0_0_1_4, g11_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g11_11 = fma(ek11_3, r0_0_2_3, g11_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g11_12 = fma(ek11_3, r0_0_3_2, g11_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g11_13 = fma(ek11_3, r0_0_4_1, g11_13);
              const double r0_1_1_3 = X * r1_0_1_3;
              g11_14 = fma(ek11_3, r0_1_1_3, g11_14);
              const double r0_1_2_2 = X * r1_0_2_2;
              g11_15 = fma(ek11_3, r0_1_2_2, g11_15);
              const double r0_1_3_1 = X * r1_0_3_1;
              g11_16 = fma(ek11_3, r0_1_3_1, g11_16);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g11_17 = fma(ek11_3, r0_2_1_2, g11_17);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g11_18 = fma(ek11_3, r0_2_2_1, g11_18);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g11_19 = fma(ek11_3, r0_3_1_1, g11_19);
            }
            { const double eb = bi[5];
              o0_11 = fma(eb, g11_0, o0_11);
            }
            { const double eb = bi[6];
              o0_11 = fma(eb, g11_3, o0_11);
            }
            { const double eb = bi[7];
              o0_11 = fma(eb, g11_9, o0_11);
            }
            { const double eb = bi[8];
              o1_11 = fma(eb, g11_0, o1_11);
            }
            { const double eb = bi[9];
              o1_11 = fma(eb, g11_3, o1_11);
            }
            { const double eb = bi[10];
              o1_11 = fma(eb, g11_9, o1_11);
            }
            { const double eb = bi[11];
              o1_11 = fma(eb, g11_19, o1_11);
            }
            { const double eb = bi[12];
              o2_11 = fma(eb, g11_0, o2_11);
            }
            { const double eb = bi[13];
              o2_11 = fma(eb, g11_2, o2_11);
            }
            { const double eb = bi[14];
              o2_11 = fma(eb, g11_3, o2_11);
            }
            { const double eb = bi[15];
              o2_11 = fma(eb, g11_8, o2_11);
            }
            { const double eb = bi[16];
              o2_11 = fma(eb, g11_9, o2_11);
            }
            { const double eb = bi[17];
              o2_11 = fma(eb, g11_18, o2_11);
            }
            { const double eb = bi[18];
              o3_11 = fma(eb, g11_0, o3_11);
            }
            { const double eb = bi[19];
              o3_11 = fma(eb, g11_1, o3_11);
            }
            { const double eb = bi[20];
              o3_11 = fma(eb, g11_3, o3_11);
            }
            { const double eb = bi[21];
              o3_11 = fma(eb, g11_7, o3_11);
            }
            { const double eb = bi[22];
              o3_11 = fma(eb, g11_9, o3_11);
            }
            { const double eb = bi[23];
              o3_11 = fma(eb, g11_17, o3_11);
            }
            { const double eb = bi[24];
              o4_11 = fma(eb, g11_0, o4_11);
            }
            { const double eb = bi[25];
              o4_11 = fma(eb, g11_2, o4_11);
            }
            { const double eb = bi[26];
              o4_11 = fma(eb, g11_6, o4_11);
            }
            { const double eb = bi[27];
              o5_11 = fma(eb, g11_0, o5_11);
            }
            { const double eb = bi[28];
              o5_11 = fma(eb, g11_2, o5_11);
            }
            { const double eb = bi[29];
              o5_11 = fma(eb, g11_6, o5_11);
            }
            { const double eb = bi[30];
              o5_11 = fma(eb, g11_3, o5_11);
            }
            { const double eb = bi[31];
              o5_11 = fma(eb, g11_8, o5_11);
            }
            { const double eb = bi[32];
              o5_11 = fma(eb, g11_16, o5_11);
            }
            { const double eb = bi[33];
              o6_11 = fma(eb, g11_0, o6_11);
            }
            { const double eb = bi[34];
              o6_11 = fma(eb, g11_2, o6_11);
            }
            { const double eb = bi[35];
              o6_11 = fma(eb, g11_6, o6_11);
            }
            { const double eb = bi[36];
              o6_11 = fma(eb, g11_13, o6_11);
            }
            { const double eb = bi[37];
              o7_11 = fma(eb, g11_0, o7_11);
            }
            { const double eb = bi[38];
              o7_11 = fma(eb, g11_1, o7_11);
            }
            { const double eb = bi[39];
              o7_11 = fma(eb, g11_2, o7_11);
            }
            { const double eb = bi[40];
              o7_11 = fma(eb, g11_5, o7_11);
            }
            { const double eb = bi[41];
              o7_11 = fma(eb, g11_6, o7_11);
            }
            { const double eb = bi[42];
              o7_11 = fma(eb, g11_12, o7_11);
            }
            { const double eb = bi[43];
              o8_11 = fma(eb, g11_0, o8_11);
            }
            { const double eb = bi[44];
              o8_11 = fma(eb, g11_1, o8_11);
            }
            { const double eb = bi[45];
              o8_11 = fma(eb, g11_4, o8_11);
            }
            { const double eb = bi[46];
              o9_11 = fma(eb, g11_0, o9_11);
            }
            { const double eb = bi[47];
              o9_11 = fma(eb, g11_1, o9_11);
            }
            { const double eb = bi[48];
              o9_11 = fma(eb, g11_4, o9_11);
            }
            { const double eb = bi[49];
              o9_11 = fma(eb, g11_3, o9_11);
            }
            { const double eb = bi[50];
              o9_11 = fma(eb, g11_7, o9_11);
            }
            { const double eb = bi[51];
              o9_11 = fma(eb, g11_14, o9_11);
            }
            { const double eb = bi[52];
              o10_11 = fma(eb, g11_0, o10_11);
            }
            { const double eb = bi[53];
              o10_11 = fma(eb, g11_1, o10_11);
            }
            { const double eb = bi[54];
              o10_11 = fma(eb, g11_4, o10_11);
            }
            { const double eb = bi[55];
              o10_11 = fma(eb, g11_2, o10_11);
            }
            { const double eb = bi[56];
              o10_11 = fma(eb, g11_5, o10_11);
            }
            { const double eb = bi[57];
              o10_11 = fma(eb, g11_11, o10_11);
            }
            { const double eb = bi[58];
              o11_11 = fma(eb, g11_0, o11_11);
            }
            { const double eb = bi[59];
              o11_11 = fma(eb, g11_1, o11_11);
            }
            { const double eb = bi[60];
              o11_11 = fma(eb, g11_4, o11_11);
            }
            { const double eb = bi[61];
              o11_11 = fma(eb, g11_10, o11_11);
            }
            { const double eb = bi[62];
              o12_11 = fma(eb, g11_0, o12_11);
            }
            { const double eb = bi[63];
              o12_11 = fma(eb, g11_2, o12_11);
            }
            { const double eb = bi[64];
              o12_11 = fma(eb, g11_3, o12_11);
            }
            { const double eb = bi[65];
              o12_11 = fma(eb, g11_8, o12_11);
            }
            { const double eb = bi[66];
              o13_11 = fma(eb, g11_0, o13_11);
            }
            { const double eb = bi[67];
              o13_11 = fma(eb, g11_2, o13_11);
            }
            { const double eb = bi[68];
              o13_11 = fma(eb, g11_3, o13_11);
            }
            { const double eb = bi[69];
              o13_11 = fma(eb, g11_8, o13_11);
            }
            { const double eb = bi[70];
              o13_11 = fma(eb, g11_9, o13_11);
            }
            { const double eb = bi[71];
              o13_11 = fma(eb, g11_18, o13_11);
            }
            { const double eb = bi[72];
              o14_11 = fma(eb, g11_0, o14_11);
            }
            { const double eb = bi[73];
              o14_11 = fma(eb, g11_2, o14_11);
            }
            { const double eb = bi[74];
              o14_11 = fma(eb, g11_6, o14_11);
            }
            { const double eb = bi[75];
              o14_11 = fma(eb, g11_3, o14_11);
            }
            { const double eb = bi[76];
              o14_11 = fma(eb, g11_8, o14_11);
            }
            { const double eb = bi[77];
              o14_11 = fma(eb, g11_16, o14_11);
            }
            { const double eb = bi[78];
              o15_11 = fma(eb, g11_0, o15_11);
            }
            { const double eb = bi[79];
              o15_11 = fma(eb, g11_1, o15_11);
            }
            { const double eb = bi[80];
              o15_11 = fma(eb, g11_2, o15_11);
            }
            { const double eb = bi[81];
              o15_11 = fma(eb, g11_5, o15_11);
            }
            { const double eb = bi[82];
              o15_11 = fma(eb, g11_3, o15_11);
            }
            { const double eb = bi[83];
              o15_11 = fma(eb, g11_7, o15_11);
            }
            { const double eb = bi[84];
              o15_11 = fma(eb, g11_8, o15_11);
            }
            { const double eb = bi[85];
              o15_11 = fma(eb, g11_15, o15_11);
            }
            { const double eb = bi[86];
              o16_11 = fma(eb, g11_0, o16_11);
            }
            { const double eb = bi[87];
              o16_11 = fma(eb, g11_1, o16_11);
            }
            { const double eb = bi[88];
              o16_11 = fma(eb, g11_3, o16_11);
            }
            { const double eb = bi[89];
              o16_11 = fma(eb, g11_7, o16_11);
            }
            { const double eb = bi[90];
              o17_11 = fma(eb, g11_0, o17_11);
            }
            { const double eb = bi[91];
              o17_11 = fma(eb, g11_1, o17_11);
            }
            { const double eb = bi[92];
              o17_11 = fma(eb, g11_3, o17_11);
            }
            { const double eb = bi[93];
              o17_11 = fma(eb, g11_7, o17_11);
            }
            { const double eb = bi[94];
              o17_11 = fma(eb, g11_9, o17_11);
            }
            { const double eb = bi[95];
              o17_11 = fma(eb, g11_17, o17_11);
            }
            { const double eb = bi[96];
              o18_11 = fma(eb, g11_0, o18_11);
            }
            { const double eb = bi[97];
              o18_11 = fma(eb, g11_1, o18_11);
            }
            { const double eb = bi[98];
              o18_11 = fma(eb, g11_2, o18_11);
            }
            { const double eb = bi[99];
              o18_11 = fma(eb, g11_5, o18_11);
            }
            { const double eb = bi[100];
              o18_11 = fma(eb, g11_3, o18_11);
            }
            { const double eb = bi[101];
              o18_11 = fma(eb, g11_7, o18_11);
            }
            { const double eb = bi[102];
              o18_11 = fma(eb, g11_8, o18_11);
            }
            { const double eb = bi[103];
              o18_11 = fma(eb, g11_15, o18_11);
            }
            { const double eb = bi[104];
              o19_11 = fma(eb, g11_0, o19_11);
            }
            { const double eb = bi[105];
              o19_11 = fma(eb, g11_1, o19_11);
            }
            { const double eb = bi[106];
              o19_11 = fma(eb, g11_4, o19_11);
            }
            { const double eb = bi[107];
              o19_11 = fma(eb, g11_3, o19_11);
            }
            { const double eb = bi[108];
              o19_11 = fma(eb, g11_7, o19_11);
            }
            { const double eb = bi[109];
              o19_11 = fma(eb, g11_14, o19_11);
            }
            { const double eb = bi[110];
              o20_11 = fma(eb, g11_0, o20_11);
            }
            { const double eb = bi[111];
              o20_11 = fma(eb, g11_1, o20_11);
            }
            { const double eb = bi[112];
              o20_11 = fma(eb, g11_2, o20_11);
            }
            { const double eb = bi[113];
              o20_11 = fma(eb, g11_5, o20_11);
            }
            { const double eb = bi[114];
              o21_11 = fma(eb, g11_0, o21_11);
            }
            { const double eb = bi[115];
              o21_11 = fma(eb, g11_1, o21_11);
            }
            { const double eb = bi[116];
              o21_11 = fma(eb, g11_2, o21_11);
            }
            { const double eb = bi[117];
              o21_11 = fma(eb, g11_5, o21_11);
            }
            { const double eb = bi[118];
              o21_11 = fma(eb, g11_3, o21_11);
            }
            { const double eb = bi[119];
              o21_11 = fma(eb, g11_7, o21_11);
            }
            { const double eb = bi[120];
              o21_11 = fma(eb, g11_8, o21_11);
            }
            { const double eb = bi[121];
              o21_11 = fma(eb, g11_15, o21_11);
            }
            { const double eb = bi[122];
              o22_11 = fma(eb, g11_0, o22_11);
            }
            { const double eb = bi[123];
              o22_11 = fma(eb, g11_1, o22_11);
            }
            { const double eb = bi[124];
              o22_11 = fma(eb, g11_2, o22_11);
            }
            { const double eb = bi[125];
              o22_11 = fma(eb, g11_5, o22_11);
            }
            { const double eb = bi[126];
              o22_11 = fma(eb, g11_6, o22_11);
            }
            { const double eb = bi[127];
              o22_11 = fma(eb, g11_12, o22_11);
            }
            { const double eb = bi[128];
              o23_11 = fma(eb, g11_0, o23_11);
            }
            { const double eb = bi[129];
              o23_11 = fma(eb, g11_1, o23_11);
            }
            { const double eb = bi[130];
              o23_11 = fma(eb, g11_4, o23_11);
            }
            { const double eb = bi[131];
              o23_11 = fma(eb, g11_2, o23_11);
            }
            { const double eb = bi[132];
              o23_11 = fma(eb, g11_5, o23_11);
            }
            { const double eb = bi[133];
              o23_11 = fma(eb, g11_11, o23_11);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_11 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 3);
            o1_11 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 3);
            o2_11 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 3);
            o3_11 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 3);
            o4_11 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 3);
            o5_11 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 3);
            o6_11 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 3);
            o7_11 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 3);
            o8_11 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 3);
            o9_11 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 3);
            o10_11 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 3);
            o11_11 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 3);
            o12_11 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 3);
            o13_11 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 3);
            o14_11 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 3);
            o15_11 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 3);
            o16_11 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 3);
            o17_11 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 3);
            o18_11 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 3);
            o19_11 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 3);
            o20_11 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 3);
            o21_11 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 3);
            o22_11 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 3);
            o23_11 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 3);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_11 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o1_11 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o2_11 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o3_11 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o4_11 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o5_11 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o6_11 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o7_11 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o8_11 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o9_11 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o10_11 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o11_11 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o12_11 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o13_11 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o14_11 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o15_11 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o16_11 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o17_11 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o18_11 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o19_11 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o20_11 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o21_11 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o22_11 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 2, fJ + 3)));
            e = fmax(e, fabs(o23_11 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 2, fJ + 3)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
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
            const double Bbd0_3 = PB[(fQ + 0) * N + fJ + 3];
            const double Bbd1_3 = PB[(fQ + 1) * N + fJ + 3];
            const double Bbd2_3 = PB[(fQ + 2) * N + fJ + 3];
            const double Bbd3_3 = PB[(fQ + 3) * N + fJ + 3];
            const double Bad0_3 = PB[(fP + 0) * N + fJ + 3];
            const double Bad1_3 = PB[(fP + 1) * N + fJ + 3];
            const double Bad2_3 = PB[(fP + 2) * N + fJ + 3];
            const double Bad3_3 = PB[(fP + 3) * N + fJ + 3];
            const double Bad4_3 = PB[(fP + 4) * N + fJ + 3];
            const double Bad5_3 = PB[(fP + 5) * N + fJ + 3];
            const double Bbc0_2 = PB[(fQ + 0) * N + fI + 2];
            const double Bbc1_2 = PB[(fQ + 1) * N + fI + 2];
            const double Bbc2_2 = PB[(fQ + 2) * N + fI + 2];
            const double Bbc3_2 = PB[(fQ + 3) * N + fI + 2];
            const double Bac0_2 = PB[(fP + 0) * N + fI + 2];
            const double Bac1_2 = PB[(fP + 1) * N + fI + 2];
            const double Bac2_2 = PB[(fP + 2) * N + fI + 2];
            const double Bac3_2 = PB[(fP + 3) * N + fI + 2];
            const double Bac4_2 = PB[(fP + 4) * N + fI + 2];
            const double Bac5_2 = PB[(fP + 5) * N + fI + 2];
            jab0 += o0_11 * ptk11;
            jab1 += o1_11 * ptk11;
            jab2 += o2_11 * ptk11;
            jab3 += o3_11 * ptk11;
            jab4 += o4_11 * ptk11;
            jab5 += o5_11 * ptk11;
            jab6 += o6_11 * ptk11;
            jab7 += o7_11 * ptk11;
            jab8 += o8_11 * ptk11;
            jab9 += o9_11 * ptk11;
            jab10 += o10_11 * ptk11;
            jab11 += o11_11 * ptk11;
            jab12 += o12_11 * ptk11;
            jab13 += o13_11 * ptk11;
            jab14 += o14_11 * ptk11;
            jab15 += o15_11 * ptk11;
            jab16 += o16_11 * ptk11;
            jab17 += o17_11 * ptk11;
            jab18 += o18_11 * ptk11;
            jab19 += o19_11 * ptk11;
            jab20 += o20_11 * ptk11;
            jab21 += o21_11 * ptk11;
            jab22 += o22_11 * ptk11;
            jab23 += o23_11 * ptk11;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 3, 2.0 * deg * (o0_11 * ptb0 + o1_11 * ptb1 + o2_11 * ptb2 + o3_11 * ptb3 + o4_11 * ptb4 + o5_11 * ptb5 + o6_11 * ptb6 + o7_11 * ptb7 + o8_11 * ptb8 + o9_11 * ptb9 + o10_11 * ptb10 + o11_11 * ptb11 + o12_11 * ptb12 + o13_11 * ptb13 + o14_11 * ptb14 + o15_11 * ptb15 + o16_11 * ptb16 + o17_11 * ptb17 + o18_11 * ptb18 + o19_11 * ptb19 + o20_11 * ptb20 + o21_11 * ptb21 + o22_11 * ptb22 + o23_11 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_11 * Abd0_3 + o1_11 * Abd1_3 + o2_11 * Abd2_3 + o3_11 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_11 * Aad0_3 + o4_11 * Aad1_3 + o8_11 * Aad2_3 + o12_11 * Aad3_3 + o16_11 * Aad4_3 + o20_11 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_11 * Abc0_2 + o1_11 * Abc1_2 + o2_11 * Abc2_2 + o3_11 * Abc3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_11 * Aac0_2 + o4_11 * Aac1_2 + o8_11 * Aac2_2 + o12_11 * Aac3_2 + o16_11 * Aac4_2 + o20_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_11 * Aad0_3 + o5_11 * Aad1_3 + o9_11 * Aad2_3 + o13_11 * Aad3_3 + o17_11 * Aad4_3 + o21_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_11 * Aac0_2 + o5_11 * Aac1_2 + o9_11 * Aac2_2 + o13_11 * Aac3_2 + o17_11 * Aac4_2 + o21_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_11 * Aad0_3 + o6_11 * Aad1_3 + o10_11 * Aad2_3 + o14_11 * Aad3_3 + o18_11 * Aad4_3 + o22_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_11 * Aac0_2 + o6_11 * Aac1_2 + o10_11 * Aac2_2 + o14_11 * Aac3_2 + o18_11 * Aac4_2 + o22_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_11 * Aad0_3 + o7_11 * Aad1_3 + o11_11 * Aad2_3 + o15_11 * Aad3_3 + o19_11 * Aad4_3 + o23_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_11 * Aac0_2 + o7_11 * Aac1_2 + o11_11 * Aac2_2 + o15_11 * Aac3_2 + o19_11 * Aac4_2 + o23_11 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_11 * Abd0_3 + o5_11 * Abd1_3 + o6_11 * Abd2_3 + o7_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_11 * Abc0_2 + o5_11 * Abc1_2 + o6_11 * Abc2_2 + o7_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_11 * Abd0_3 + o9_11 * Abd1_3 + o10_11 * Abd2_3 + o11_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_11 * Abc0_2 + o9_11 * Abc1_2 + o10_11 * Abc2_2 + o11_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_11 * Abd0_3 + o13_11 * Abd1_3 + o14_11 * Abd2_3 + o15_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_11 * Abc0_2 + o13_11 * Abc1_2 + o14_11 * Abc2_2 + o15_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o16_11 * Abd0_3 + o17_11 * Abd1_3 + o18_11 * Abd2_3 + o19_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_11 * Abc0_2 + o17_11 * Abc1_2 + o18_11 * Abc2_2 + o19_11 * Abc3_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o20_11 * Abd0_3 + o21_11 * Abd1_3 + o22_11 * Abd2_3 + o23_11 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_11 * Abc0_2 + o21_11 * Abc1_2 + o22_11 * Abc2_2 + o23_11 * Abc3_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_11 * Bbd0_3 + o1_11 * Bbd1_3 + o2_11 * Bbd2_3 + o3_11 * Bbd3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_11 * Bad0_3 + o4_11 * Bad1_3 + o8_11 * Bad2_3 + o12_11 * Bad3_3 + o16_11 * Bad4_3 + o20_11 * Bad5_3));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 3, deg * (o0_11 * Bbc0_2 + o1_11 * Bbc1_2 + o2_11 * Bbc2_2 + o3_11 * Bbc3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 3, deg * (o0_11 * Bac0_2 + o4_11 * Bac1_2 + o8_11 * Bac2_2 + o12_11 * Bac3_2 + o16_11 * Bac4_2 + o20_11 * Bac5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 2, deg * (o1_11 * Bad0_3 + o5_11 * Bad1_3 + o9_11 * Bad2_3 + o13_11 * Bad3_3 + o17_11 * Bad4_3 + o21_11 * Bad5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 3, deg * (o1_11 * Bac0_2 + o5_11 * Bac1_2 + o9_11 * Bac2_2 + o13_11 * Bac3_2 + o17_11 * Bac4_2 + o21_11 * Bac5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 2, deg * (o2_11 * Bad0_3 + o6_11 * Bad1_3 + o10_11 * Bad2_3 + o14_11 * Bad3_3 + o18_11 * Bad4_3 + o22_11 * Bad5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 3, deg * (o2_11 * Bac0_2 + o6_11 * Bac1_2 + o10_11 * Bac2_2 + o14_11 * Bac3_2 + o18_11 * Bac4_2 + o22_11 * Bac5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 2, deg * (o3_11 * Bad0_3 + o7_11 * Bad1_3 + o11_11 * Bad2_3 + o15_11 * Bad3_3 + o19_11 * Bad4_3 + o23_11 * Bad5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 3, deg * (o3_11 * Bac0_2 + o7_11 * Bac1_2 + o11_11 * Bac2_2 + o15_11 * Bac3_2 + o19_11 * Bac4_2 + o23_11 * Bac5_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o4_11 * Bbd0_3 + o5_11 * Bbd1_3 + o6_11 * Bbd2_3 + o7_11 * Bbd3_3));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 3, deg * (o4_11 * Bbc0_2 + o5_11 * Bbc1_2 + o6_11 * Bbc2_2 + o7_11 * Bbc3_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o8_11 * Bbd0_3 + o9_11 * Bbd1_3 + o10_11 * Bbd2_3 + o11_11 * Bbd3_3));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 3, deg * (o8_11 * Bbc0_2 + o9_11 * Bbc1_2 + o10_11 * Bbc2_2 + o11_11 * Bbc3_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o12_11 * Bbd0_3 + o13_11 * Bbd1_3 + o14_11 * Bbd2_3 + o15_11 * Bbd3_3));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 3, deg * (o12_11 * Bbc0_2 + o13_11 * Bbc1_2 + o14_11 * Bbc2_2 + o15_11 * Bbc3_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o16_11 * Bbd0_3 + o17_11 * Bbd1_3 + o18_11 * Bbd2_3 + o19_11 * Bbd3_3));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 3, deg * (o16_11 * Bbc0_2 + o17_11 * Bbc1_2 + o18_11 * Bbc2_2 + o19_11 * Bbc3_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o20_11 * Bbd0_3 + o21_11 * Bbd1_3 + o22_11 * Bbd2_3 + o23_11 * Bbd3_3));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 3, deg * (o20_11 * Bbc0_2 + o21_11 * Bbc1_2 + o22_11 * Bbc2_2 + o23_11 * Bbc3_2));
          }
        } break;
        case 12: {  // ket functions [12]
          double o0_12 = 0;
          double o1_12 = 0;
          double o2_12 = 0;
          double o3_12 = 0;
          double o4_12 = 0;
          double o5_12 = 0;
          double o6_12 = 0;
          double o7_12 = 0;
          double o8_12 = 0;
          double o9_12 = 0;
          double o10_12 = 0;
          double o11_12 = 0;
          double o12_12 = 0;
          double o13_12 = 0;
          double o14_12 = 0;
          double o15_12 = 0;
          double o16_12 = 0;
          double o17_12 = 0;
          double o18_12 = 0;
          double o19_12 = 0;
          double o20_12 = 0;
          double o21_12 = 0;
          double o22_12 = 0;
          double o23_12 = 0;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek12_0 = kj[38 * kS];
              const double ek12_1 = -kj[39 * kS];
              g12_0 = fma(ek12_0, b0, g12_0);
              const double r0_0_0_1 = Z * b1;
              g12_1 = fma(ek12_0, r0_0_0_1, g12_1);
              g12_0 = fma(ek12_1, r0_0_0_1, g12_0);
              const double r0_0_1_0 = Y * b1;
              g12_2 = fma(ek12_0, r0_0_1_0, g12_2);
              const double r0_1_0_0 = X * b1;
              g12_3 = fma(ek12_0, r0_1_0_0, g12_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g12_4 = fma(ek12_0, r0_0_0_2, g12_4);
              g12_1 = fma(ek12_1, r0_0_0_2, g12_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g12_5 = fma(ek12_0, r0_0_1_1, g12_5);
              g12_2 = fma(ek12_1, r0_0_1_1, g12_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g12_6 = fma(ek12_0, r0_0_2_0, g12_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g12_7 = fma(ek12_0, r0_1_0_1, g12_7);
              g12_3 = fma(ek12_1, r0_1_0_1, g12_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g12_8 = fma(ek12_0, r0_1_1_0, g12_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g12_9 = fma(ek12_0, r0_2_0_0, g12_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g12_10 = fma(ek12_0, r0_0_0_3, g12_10);
              g12_4 = fma(ek12_1, r0_0_0_3, g12_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g12_11 = fma(ek12_0, r0_0_1_2, g12_11);
              g12_5 = fma(ek12_1, r0_0_1_2, g12_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g12_12 = fma(ek12_0, r0_0_2_1, g12_12);
              g12_6 = fma(ek12_1, r0_0_2_1, g12_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g12_13 = fma(ek12_0, r0_0_3_0, g12_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g12_14 = fma(ek12_0, r0_1_0_2, g12_14);
              g12_7 = fma(ek12_1, r0_1_0_2, g12_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g12_15 = fma(ek12_0, r0_1_1_1, g12_15);
              g12_8 = fma(ek12_1, r0_1_1_1, g12_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g12_16 = fma(ek12_0, r0_1_2_0, g12_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g12_17 = fma(ek12_0, r0_2_0_1, g12_17);
              g12_9 = fma(ek12_1, r0_2_0_1, g12_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g12_18 = fma(ek12_0, r0_2_1_0, g12_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g12_19 = fma(ek12_0, r0_3_0_0, g12_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g12_10 = fma(ek12_1, r0_0_0_4, g12_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g12_11 = fma(ek12_1, r0_0_1_3, g12_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g12_12 = fma(ek12_1, r0_0_2_2, g12_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g12_13 = fma(ek12_1, r0_0_3_1, g12_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g12_14 = fma(ek12_1, r0_1_0_3, g12_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g12_15 = fma(ek12_1, r0_1_1_2, g12_15);
              const double r0_1_2_1 = X * r1_0_2_1;
              g12_16 = fma(ek12_1, r0_1_2_1, g12_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g12_17 = fma(ek12_1, r0_2_0_2, g12_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g12_18 = fma(ek12_1, r0_2_1_1, g12_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g12_19 = fma(ek12_1, r0_3_0_1, g12_19);
            }
            { const double eb = bi[5];
              o0_12 = fma(eb, g12_0, o0_12);
            }
            { const double eb = bi[6];
              o0_12 = fma(eb, g12_3, o0_12);
            }
            { const double eb = bi[7];
              o0_12 = fma(eb, g12_9, o0_12);
            }
            { const double eb = bi[8];
              o1_12 = fma(eb, g12_0, o1_12);
            }
            { const double eb = bi[9];
              o1_12 = fma(eb, g12_3, o1_12);
            }
            { const double eb = bi[10];
              o1_12 = fma(eb, g12_9, o1_12);
            }
            { const double eb = bi[11];
              o1_12 = fma(eb, g12_19, o1_12);
            }
            { const double eb = bi[12];
              o2_12 = fma(eb, g12_0, o2_12);
            }
            { const double eb = bi[13];
              o2_12 = fma(eb, g12_2, o2_12);
            }
            { const double eb = bi[14];
              o2_12 = fma(eb, g12_3, o2_12);
            }
            { const double eb = bi[15];
              o2_12 = fma(eb, g12_8, o2_12);
            }
            { const double eb = bi[16];
              o2_12 = fma(eb, g12_9, o2_12);
            }
            { const double eb = bi[17];
              o2_12 = fma(eb, g12_18, o2_12);
            }
            { const double eb = bi[18];
              o3_12 = fma(eb, g12_0, o3_12);
            }
            { const double eb = bi[19];
              o3_12 = fma(eb, g12_1, o3_12);
            }
            { const double eb = bi[20];
              o3_12 = fma(eb, g12_3, o3_12);
            }
            { const double eb = bi[21];
              o3_12 = fma(eb, g12_7, o3_12);
            }
            { const double eb = bi[22];
              o3_12 = fma(eb, g12_9, o3_12);
            }
            { const double eb = bi[23];
              o3_12 = fma(eb, g12_17, o3_12);
            }
            { const double eb = bi[24];
              o4_12 = fma(eb, g12_0, o4_12);
            }
            { const double eb = bi[25];
              o4_12 = fma(eb, g12_2, o4_12);
            }
            { const double eb = bi[26];
              o4_12 = fma(eb, g12_6, o4_12);
            }
            { const double eb = bi[27];
              o5_12 = fma(eb, g12_0, o5_12);
            }
            { const double eb = bi[28];
              o5_12 = fma(eb, g12_2, o5_12);
            }
            { const double eb = bi[29];
              o5_12 = fma(eb, g12_6, o5_12);
            }
            { const double eb = bi[30];
              o5_12 = fma(eb, g12_3, o5_12);
            }
            { const double eb = bi[31];
              o5_12 = fma(eb, g12_8, o5_12);
            }
            { const double eb = bi[32];
              o5_12 = fma(eb, g12_16, o5_12);
            }
            { const double eb = bi[33];
              o6_12 = fma(eb, g12_0, o6_12);
            }
            { const double eb = bi[34];
              o6_12 = fma(eb, g12_2, o6_12);
            }
            { const double eb = bi[35];
              o6_12 = fma(eb, g12_6, o6_12);
            }
            { const double eb = bi[36];
              o6_12 = fma(eb, g12_13, o6_12);
            }
            { const double eb = bi[37];
              o7_12 = fma(eb, g12_0, o7_12);
            }
            { const double eb = bi[38];
              o7_12 = fma(eb, g12_1, o7_12);
            }
            { const double eb = bi[39];
              o7_12 = fma(eb, g12_2, o7_12);
            }
            { const double eb = bi[40];
              o7_12 = fma(eb, g12_5, o7_12);
            }
            { const double eb = bi[41];
              o7_12 = fma(eb, g12_6, o7_12);
            }
            { const double eb = bi[42];
              o7_12 = fma(eb, g12_12, o7_12);
            }
            { const double eb = bi[43];
              o8_12 = fma(eb, g12_0, o8_12);
            }
            { const double eb = bi[44];
              o8_12 = fma(eb, g12_1, o8_12);
            }
            { const double eb = bi[45];
              o8_12 = fma(eb, g12_4, o8_12);
            }
            { const double eb = bi[46];
              o9_12 = fma(eb, g12_0, o9_12);
            }
            { const double eb = bi[47];
              o9_12 = fma(eb, g12_1, o9_12);
            }
            { const double eb = bi[48];
              o9_12 = fma(eb, g12_4, o9_12);
            }
            { const double eb = bi[49];
              o9_12 = fma(eb, g12_3, o9_12);
            }
            { const double eb = bi[50];
              o9_12 = fma(eb, g12_7, o9_12);
            }
            { const double eb = bi[51];
              o9_12 = fma(eb, g12_14, o9_12);
            }
            { const double eb = bi[52];
              o10_12 = fma(eb, g12_0, o10_12);
            }
            { const double eb = bi[53];
              o10_12 = fma(eb, g12_1, o10_12);
            }
            { const double eb = bi[54];
              o10_12 = fma(eb, g12_4, o10_12);
            }
            { const double eb = bi[55];
              o10_12 = fma(eb, g12_2, o10_12);
            }
            { const double eb = bi[56];
              o10_12 = fma(eb, g12_5, o10_12);
            }
            { const double eb = bi[57];
              o10_12 = fma(eb, g12_11, o10_12);
            }
            { const double eb = bi[58];
              o11_12 = fma(eb, g12_0, o11_12);
            }
            { const double eb = bi[59];
              o11_12 = fma(eb, g12_1, o11_12);
            }
            { const double eb = bi[60];
              o11_12 = fma(eb, g12_4, o11_12);
            }
            { const double eb = bi[61];
              o11_12 = fma(eb, g12_10, o11_12);
            }
            { const double eb = bi[62];
              o12_12 = fma(eb, g12_0, o12_12);
            }
            { const double eb = bi[63];
              o12_12 = fma(eb, g12_2, o12_12);
            }
            { const double eb = bi[64];
              o12_12 = fma(eb, g12_3, o12_12);
            }
            { const double eb = bi[65];
              o12_12 = fma(eb, g12_8, o12_12);
            }
            { const double eb = bi[66];
              o13_12 = fma(eb, g12_0, o13_12);
            }
            { const double eb = bi[67];
              o13_12 = fma(eb, g12_2, o13_12);
            }
            { const double eb = bi[68];
              o13_12 = fma(eb, g12_3, o13_12);
            }
            { const double eb = bi[69];
              o13_12 = fma(eb, g12_8, o13_12);
            }
            { const double eb = bi[70];
              o13_12 = fma(eb, g12_9, o13_12);
            }
            { const double eb = bi[71];
              o13_12 = fma(eb, g12_18, o13_12);
            }
            { const double eb = bi[72];
              o14_12 = fma(eb, g12_0, o14_12);
            }
            { const double eb = bi[73];
              o14_12 = fma(eb, g12_2, o14_12);
            }
            { const double eb = bi[74];
              o14_12 = fma(eb, g12_6, o14_12);
            }
            { const double eb = bi[75];
              o14_12 = fma(eb, g12_3, o14_12);
            }
            { const double eb = bi[76];
              o14_12 = fma(eb, g12_8, o14_12);
            }
            { const double eb = bi[77];
              o14_12 = fma(eb, g12_16, o14_12);
            }
            { const double eb = bi[78];
              o15_12 = fma(eb, g12_0, o15_12);
            }
            { const double eb = bi[79];
              o15_12 = fma(eb, g12_1, o15_12);
            }
            { const double eb = bi[80];
              o15_12 = fma(eb, g12_2, o15_12);
            }
            { const double eb = bi[81];
              o15_12 = fma(eb, g12_5, o15_12);
            }
            { const double eb = bi[82];
              o15_12 = fma(eb, g12_3, o15_12);
            }
            { const double eb = bi[83];
              o15_12 = fma(eb, g12_7, o15_12);
            }
            { const double eb = bi[84];
              o15_12 = fma(eb, g12_8, o15_12);
            }
            { const double eb = bi[85];
              o15_12 = fma(eb, g12_15, o15_12);
            }
            { const double eb = bi[86];
              o16_12 = fma(eb, g12_0, o16_12);
            }
            { const double eb = bi[87];
              o16_12 = fma(eb, g12_1, o16_12);
            }
            { const double eb = bi[88];
              o16_12 = fma(eb, g12_3, o16_12);
            }
            { const double eb = bi[89];
              o16_12 = fma(eb, g12_7, o16_12);
            }
            { const double eb = bi[90];
              o17_12 = fma(eb, g12_0, o17_12);
            }
            { const double eb = bi[91];
              o17_12 = fma(eb, g12_1, o17_12);
            }
            { const double eb = bi[92];
              o17_12 = fma(eb, g12_3, o17_12);
            }
            { const double eb = bi[93];
              o17_12 = fma(eb, g12_7, o17_12);
            }
            { const double eb = bi[94];
              o17_12 = fma(eb, g12_9, o17_12);
            }
            { const double eb = bi[95];
              o17_12 = fma(eb, g12_17, o17_12);
            }
            { const double eb = bi[96];
              o18_12 = fma(eb, g12_0, o18_12);
            }
            { const double eb = bi[97];
              o18_12 = fma(eb, g12_1, o18_12);
            }
            { const double eb = bi[98];
              o18_12 = fma(eb, g12_2, o18_12);
            }
            { const double eb = bi[99];
              o18_12 = fma(eb, g12_5, o18_12);
            }
            { const double eb = bi[100];
              o18_12 = fma(eb, g12_3, o18_12);
            }
            { const double eb = bi[101];
              o18_12 = fma(eb, g12_7, o18_12);
            }
            { const double eb = bi[102];
              o18_12 = fma(eb, g12_8, o18_12);
            }
            { const double eb = bi[103];
              o18_12 = fma(eb, g12_15, o18_12);
            }
            { const double eb = bi[104];
              o19_12 = fma(eb, g12_0, o19_12);
            }
            { const double eb = bi[105];
              o19_12 = fma(eb, g12_1, o19_12);
            }
            { const double eb = bi[106];
              o19_12 = fma(eb, g12_4, o19_12);
            }
            { const double eb = bi[107];
              o19_12 = fma(eb, g12_3, o19_12);
            }
            { const double eb = bi[108];
              o19_12 = fma(eb, g12_7, o19_12);
            }
            { const double eb = bi[109];
              o19_12 = fma(eb, g12_14, o19_12);
            }
            { const double eb = bi[110];
              o20_12 = fma(eb, g12_0, o20_12);
            }
            { const double eb = bi[111];
              o20_12 = fma(eb, g12_1, o20_12);
            }
            { const double eb = bi[112];
              o20_12 = fma(eb, g12_2, o20_12);
            }
            { const double eb = bi[113];
              o20_12 = fma(eb, g12_5, o20_12);
            }
            { const double eb = bi[114];
              o21_12 = fma(eb, g12_0, o21_12);
            }
            { const double eb = bi[115];
              o21_12 = fma(eb, g12_1, o21_12);
            }
            { const double eb = bi[116];
              o21_12 = fma(eb, g12_2, o21_12);
            }
            { const double eb = bi[117];
              o21_12 = fma(eb, g12_5, o21_12);
            }
            { const double eb = bi[118];
              o21_12 = fma(eb, g12_3, o21_12);
            }
            { const double eb = bi[119];
              o21_12 = fma(eb, g12_7, o21_12);
            }
            { const double eb = bi[120];
              o21_12 = fma(eb, g12_8, o21_12);
            }
            { const double eb = bi[121];
              o21_12 = fma(eb, g12_15, o21_12);
            }
            { const double eb = bi[122];
              o22_12 = fma(eb, g12_0, o22_12);
            }
            { const double eb = bi[123];
              o22_12 = fma(eb, g12_1, o22_12);
            }
            { const double eb = bi[124];
              o22_12 = fma(eb, g12_2, o22_12);
            }
            { const double eb = bi[125];
              o22_12 = fma(eb, g12_5, o22_12);
            }
            { const double eb = bi[126];
              o22_12 = fma(eb, g12_6, o22_12);
            }
            { const double eb = bi[127];
              o22_12 = fma(eb, g12_12, o22_12);
            }
            { const double eb = bi[128];
              o23_12 = fma(eb, g12_0, o23_12);
            }
            { const double eb = bi[129];
              o23_12 = fma(eb, g12_1, o23_12);
            }
            { const double eb = bi[130];
              o23_12 = fma(eb, g12_4, o23_12);
            }
            { const double eb = bi[131];
              o23_12 = fma(eb, g12_2, o23_12);
            }
            { const double eb = bi[132];
              o23_12 = fma(eb, g12_5, o23_12);
            }
            { const double eb = bi[133];
              o23_12 = fma(eb, g12_11, o23_12);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_12 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 0);
            o1_12 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 0);
            o2_12 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 0);
            o3_12 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 0);
            o4_12 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 0);
            o5_12 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 0);
            o6_12 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 0);
            o7_12 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 0);
            o8_12 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 0);
            o9_12 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 0);
            o10_12 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 0);
            o11_12 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 0);
            o12_12 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 0);
            o13_12 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 0);
            o14_12 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 0);
            o15_12 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 0);
            o16_12 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 0);
            o17_12 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 0);
            o18_12 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 0);
            o19_12 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 0);
            o20_12 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 0);
            o21_12 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 0);
            o22_12 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 0);
            o23_12 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_12 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o1_12 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o2_12 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o3_12 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o4_12 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o5_12 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o6_12 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o7_12 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o8_12 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o9_12 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o10_12 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o11_12 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o12_12 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o13_12 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o14_12 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o15_12 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o16_12 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o17_12 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o18_12 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o19_12 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o20_12 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o21_12 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o22_12 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 0)));
            e = fmax(e, fabs(o23_12 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk12 = PT[(fI + 3) * N + fJ + 0];
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
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
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
            const double Bac0_3 = PB[(fP + 0) * N + fI + 3];
            const double Bac1_3 = PB[(fP + 1) * N + fI + 3];
            const double Bac2_3 = PB[(fP + 2) * N + fI + 3];
            const double Bac3_3 = PB[(fP + 3) * N + fI + 3];
            const double Bac4_3 = PB[(fP + 4) * N + fI + 3];
            const double Bac5_3 = PB[(fP + 5) * N + fI + 3];
            jab0 += o0_12 * ptk12;
            jab1 += o1_12 * ptk12;
            jab2 += o2_12 * ptk12;
            jab3 += o3_12 * ptk12;
            jab4 += o4_12 * ptk12;
            jab5 += o5_12 * ptk12;
            jab6 += o6_12 * ptk12;
            jab7 += o7_12 * ptk12;
            jab8 += o8_12 * ptk12;
            jab9 += o9_12 * ptk12;
            jab10 += o10_12 * ptk12;
            jab11 += o11_12 * ptk12;
            jab12 += o12_12 * ptk12;
            jab13 += o13_12 * ptk12;
            jab14 += o14_12 * ptk12;
            jab15 += o15_12 * ptk12;
            jab16 += o16_12 * ptk12;
            jab17 += o17_12 * ptk12;
            jab18 += o18_12 * ptk12;
            jab19 += o19_12 * ptk12;
            jab20 += o20_12 * ptk12;
            jab21 += o21_12 * ptk12;
            jab22 += o22_12 * ptk12;
            jab23 += o23_12 * ptk12;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 0, 2.0 * deg * (o0_12 * ptb0 + o1_12 * ptb1 + o2_12 * ptb2 + o3_12 * ptb3 + o4_12 * ptb4 + o5_12 * ptb5 + o6_12 * ptb6 + o7_12 * ptb7 + o8_12 * ptb8 + o9_12 * ptb9 + o10_12 * ptb10 + o11_12 * ptb11 + o12_12 * ptb12 + o13_12 * ptb13 + o14_12 * ptb14 + o15_12 * ptb15 + o16_12 * ptb16 + o17_12 * ptb17 + o18_12 * ptb18 + o19_12 * ptb19 + o20_12 * ptb20 + o21_12 * ptb21 + o22_12 * ptb22 + o23_12 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_12 * Abd0_0 + o1_12 * Abd1_0 + o2_12 * Abd2_0 + o3_12 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_12 * Aad0_0 + o4_12 * Aad1_0 + o8_12 * Aad2_0 + o12_12 * Aad3_0 + o16_12 * Aad4_0 + o20_12 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_12 * Abc0_3 + o1_12 * Abc1_3 + o2_12 * Abc2_3 + o3_12 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_12 * Aac0_3 + o4_12 * Aac1_3 + o8_12 * Aac2_3 + o12_12 * Aac3_3 + o16_12 * Aac4_3 + o20_12 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_12 * Aad0_0 + o5_12 * Aad1_0 + o9_12 * Aad2_0 + o13_12 * Aad3_0 + o17_12 * Aad4_0 + o21_12 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_12 * Aac0_3 + o5_12 * Aac1_3 + o9_12 * Aac2_3 + o13_12 * Aac3_3 + o17_12 * Aac4_3 + o21_12 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_12 * Aad0_0 + o6_12 * Aad1_0 + o10_12 * Aad2_0 + o14_12 * Aad3_0 + o18_12 * Aad4_0 + o22_12 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_12 * Aac0_3 + o6_12 * Aac1_3 + o10_12 * Aac2_3 + o14_12 * Aac3_3 + o18_12 * Aac4_3 + o22_12 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_12 * Aad0_0 + o7_12 * Aad1_0 + o11_12 * Aad2_0 + o15_12 * Aad3_0 + o19_12 * Aad4_0 + o23_12 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_12 * Aac0_3 + o7_12 * Aac1_3 + o11_12 * Aac2_3 + o15_12 * Aac3_3 + o19_12 * Aac4_3 + o23_12 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_12 * Abd0_0 + o5_12 * Abd1_0 + o6_12 * Abd2_0 + o7_12 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_12 * Abc0_3 + o5_12 * Abc1_3 + o6_12 * Abc2_3 + o7_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_12 * Abd0_0 + o9_12 * Abd1_0 + o10_12 * Abd2_0 + o11_12 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_12 * Abc0_3 + o9_12 * Abc1_3 + o10_12 * Abc2_3 + o11_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_12 * Abd0_0 + o13_12 * Abd1_0 + o14_12 * Abd2_0 + o15_12 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_12 * Abc0_3 + o13_12 * Abc1_3 + o14_12 * Abc2_3 + o15_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o16_12 * Abd0_0 + o17_12 * Abd1_0 + o18_12 * Abd2_0 + o19_12 * Abd3_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o16_12 * Abc0_3 + o17_12 * Abc1_3 + o18_12 * Abc2_3 + o19_12 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o20_12 * Abd0_0 + o21_12 * Abd1_0 + o22_12 * Abd2_0 + o23_12 * Abd3_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o20_12 * Abc0_3 + o21_12 * Abc1_3 + o22_12 * Abc2_3 + o23_12 * Abc3_3));
            atomicAdd(KBacc + (fP + 0) * N + fI + 3, deg * (o0_12 * Bbd0_0 + o1_12 * Bbd1_0 + o2_12 * Bbd2_0 + o3_12 * Bbd3_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 3, deg * (o0_12 * Bad0_0 + o4_12 * Bad1_0 + o8_12 * Bad2_0 + o12_12 * Bad3_0 + o16_12 * Bad4_0 + o20_12 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_12 * Bbc0_3 + o1_12 * Bbc1_3 + o2_12 * Bbc2_3 + o3_12 * Bbc3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_12 * Bac0_3 + o4_12 * Bac1_3 + o8_12 * Bac2_3 + o12_12 * Bac3_3 + o16_12 * Bac4_3 + o20_12 * Bac5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 3, deg * (o1_12 * Bad0_0 + o5_12 * Bad1_0 + o9_12 * Bad2_0 + o13_12 * Bad3_0 + o17_12 * Bad4_0 + o21_12 * Bad5_0));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_12 * Bac0_3 + o5_12 * Bac1_3 + o9_12 * Bac2_3 + o13_12 * Bac3_3 + o17_12 * Bac4_3 + o21_12 * Bac5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 3, deg * (o2_12 * Bad0_0 + o6_12 * Bad1_0 + o10_12 * Bad2_0 + o14_12 * Bad3_0 + o18_12 * Bad4_0 + o22_12 * Bad5_0));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_12 * Bac0_3 + o6_12 * Bac1_3 + o10_12 * Bac2_3 + o14_12 * Bac3_3 + o18_12 * Bac4_3 + o22_12 * Bac5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 3, deg * (o3_12 * Bad0_0 + o7_12 * Bad1_0 + o11_12 * Bad2_0 + o15_12 * Bad3_0 + o19_12 * Bad4_0 + o23_12 * Bad5_0));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_12 * Bac0_3 + o7_12 * Bac1_3 + o11_12 * Bac2_3 + o15_12 * Bac3_3 + o19_12 * Bac4_3 + o23_12 * Bac5_3));
            atomicAdd(KBacc + (fP + 1) * N + fI + 3, deg * (o4_12 * Bbd0_0 + o5_12 * Bbd1_0 + o6_12 * Bbd2_0 + o7_12 * Bbd3_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o4_12 * Bbc0_3 + o5_12 * Bbc1_3 + o6_12 * Bbc2_3 + o7_12 * Bbc3_3));
            atomicAdd(KBacc + (fP + 2) * N + fI + 3, deg * (o8_12 * Bbd0_0 + o9_12 * Bbd1_0 + o10_12 * Bbd2_0 + o11_12 * Bbd3_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o8_12 * Bbc0_3 + o9_12 * Bbc1_3 + o10_12 * Bbc2_3 + o11_12 * Bbc3_3));
            atomicAdd(KBacc + (fP + 3) * N + fI + 3, deg * (o12_12 * Bbd0_0 + o13_12 * Bbd1_0 + o14_12 * Bbd2_0 + o15_12 * Bbd3_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o12_12 * Bbc0_3 + o13_12 * Bbc1_3 + o14_12 * Bbc2_3 + o15_12 * Bbc3_3));
            atomicAdd(KBacc + (fP + 4) * N + fI + 3, deg * (o16_12 * Bbd0_0 + o17_12 * Bbd1_0 + o18_12 * Bbd2_0 + o19_12 * Bbd3_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o16_12 * Bbc0_3 + o17_12 * Bbc1_3 + o18_12 * Bbc2_3 + o19_12 * Bbc3_3));
            atomicAdd(KBacc + (fP + 5) * N + fI + 3, deg * (o20_12 * Bbd0_0 + o21_12 * Bbd1_0 + o22_12 * Bbd2_0 + o23_12 * Bbd3_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o20_12 * Bbc0_3 + o21_12 * Bbc1_3 + o22_12 * Bbc2_3 + o23_12 * Bbc3_3));
          }
        } break;
        case 13: {  // ket functions [13]
          double o0_13 = 0;
          double o1_13 = 0;
          double o2_13 = 0;
          double o3_13 = 0;
          double o4_13 = 0;
          double o5_13 = 0;
          double o6_13 = 0;
          double o7_13 = 0;
          double o8_13 = 0;
          double o9_13 = 0;
          double o10_13 = 0;
          double o11_13 = 0;
          double o12_13 = 0;
          double o13_13 = 0;
          double o14_13 = 0;
          double o15_13 = 0;
          double o16_13 = 0;
          double o17_13 = 0;
          double o18_13 = 0;
          double o19_13 = 0;
          double o20_13 = 0;
          double o21_13 = 0;
          double o22_13 = 0;
          double o23_13 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek13_0 = kj[40 * kS];
              const double ek13_1 = -kj[41 * kS];
              const double ek13_2 = -kj[42 * kS];
              const double ek13_3 = kj[43 * kS];
              g13_0 = fma(ek13_0, b0, g13_0);
              const double r0_0_0_1 = Z * b1;
              g13_1 = fma(ek13_0, r0_0_0_1, g13_1);
              g13_0 = fma(ek13_1, r0_0_0_1, g13_0);
              const double r0_0_1_0 = Y * b1;
              g13_2 = fma(ek13_0, r0_0_1_0, g13_2);
              const double r0_1_0_0 = X * b1;
              g13_3 = fma(ek13_0, r0_1_0_0, g13_3);
              g13_0 = fma(ek13_2, r0_1_0_0, g13_0);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g13_4 = fma(ek13_0, r0_0_0_2, g13_4);
              g13_1 = fma(ek13_1, r0_0_0_2, g13_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g13_5 = fma(ek13_0, r0_0_1_1, g13_5);
              g13_2 = fma(ek13_1, r0_0_1_1, g13_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g13_6 = fma(ek13_0, r0_0_2_0, g13_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g13_7 = fma(ek13_0, r0_1_0_1, g13_7);
              g13_3 = fma(ek13_1, r0_1_0_1, g13_3);
              g13_1 = fma(ek13_2, r0_1_0_1, g13_1);
              g13_0 = fma(ek13_3, r0_1_0_1, g13_0);
              const double r0_1_1_0 = X * r1_0_1_0;
              g13_8 = fma(ek13_0, r0_1_1_0, g13_8);
              g13_2 = fma(ek13_2, r0_1_1_0, g13_2);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g13_9 = fma(ek13_0, r0_2_0_0, g13_9);
              g13_3 = fma(ek13_2, r0_2_0_0, g13_3);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g13_10 = fma(ek13_0, r0_0_0_3, g13_10);
              g13_4 = fma(ek13_1, r0_0_0_3, g13_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g13_11 = fma(ek13_0, r0_0_1_2, g13_11);
              g13_5 = fma(ek13_1, r0_0_1_2, g13_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g13_12 = fma(ek13_0, r0_0_2_1, g13_12);
              g13_6 = fma(ek13_1, r0_0_2_1, g13_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g13_13 = fma(ek13_0, r0_0_3_0, g13_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g13_14 = fma(ek13_0, r0_1_0_2, g13_14);
              g13_7 = fma(ek13_1, r0_1_0_2, g13_7);
              g13_4 = fma(ek13_2, r0_1_0_2, g13_4);
              g13_1 = fma(ek13_3, r0_1_0_2, g13_1);
              const double r0_1_1_1 = X * r1_0_1_1;
              g13_15 = fma(ek13_0, r0_1_1_1, g13_15);
              g13_8 = fma(ek13_1, r0_1_1_1, g13_8);
              g13_5 = fma(ek13_2, r0_1_1_1, g13_5);
              g13_2 = fma(ek13_3, r0_1_1_1, g13_2);
              const double r0_1_2_0 = X * r1_0_2_0;
              g13_16 = fma(ek13_0, r0_1_2_0, g13_16);
              g13_6 = fma(ek13_2, r0_1_2_0, g13_6);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g13_17 = fma(ek13_0, r0_2_0_1, g13_17);
              g13_9 = fma(ek13_1, r0_2_0_1, g13_9);
              g13_7 = fma(ek13_2, r0_2_0_1, g13_7);
              g13_3 = fma(ek13_3, r0_2_0_1, g13_3);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g13_18 = fma(ek13_0, r0_2_1_0, g13_18);
              g13_8 = fma(ek13_2, r0_2_1_0, g13_8);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g13_19 = fma(ek13_0, r0_3_0_0, g13_19);
              g13_9 = fma(ek13_2, r0_3_0_0, g13_9);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g13_10 = fma(ek13_1, r0_0_0_4, g13_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g13_11 = fma(ek13_1, r0_0_1_3, g13_11);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g13_12 = fma(ek13_1, r0_0_2_2, g13_12);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g13_13 = fma(ek13_1, r0_0_3_1, g13_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g13_14 = fma(ek13_1, r0_1_0_3, g13_14);
              g13_10 = fma(ek13_2, r0_1_0_3, g13_10);
              g13_4 = fma(ek13_3, r0_1_0_3, g13_4);
              const double r0_1_1_2 = X * r1_0_1_2;
              g13_15 = fma(ek13_1, r0_1_1_2, g13_15);
              g13_11 = fma(ek13_2, r0_1_1_2, g13_11);
              g13_5 = fma(ek13_3, r0_1_1_2, g13_5);
              const double r0_1_2_1 = X * r1_0_2_1;
              g13_16 = fma(ek13_1, r0_1_2_1, g13_16);
              g13_12 = fma(ek13_2, r0_1_2_1, g13_12);
              g13_6 = fma(ek13_3, r0_1_2_1, g13_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_1_3_0 = X * r1_0_3_0;
              g13_13 = fma(ek13_2, r0_1_3_0, g13_13);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g13_17 = fma(ek13_1, r0_2_0_2, g13_17);
              g13_14 = fma(ek13_2, r0_2_0_2, g13_14);
              g13_7 = fma(ek13_3, r0_2_0_2, g13_7);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g13_18 = fma(ek13_1, r0_2_1_1, g13_18);
              g13_15 = fma(ek13_2, r0_2_1_1, g13_15);
              g13_8 = fma(ek13_3, r0_2_1_1, g13_8);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g13_16 = fma(ek13_2, r0_2_2_0, g13_16);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g13_19 = fma(ek13_1, r0_3_0_1, g13_19);
              g13_17 = fma(ek13_2, r0_3_0_1, g13_17);
              g13_9 = fma(ek13_3, r0_3_0_1, g13_9);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g13_18 = fma(ek13_2, r0_3_1_0, g13_18);
              const double r3_1_0_0 = X * b4;
              const double r2_2_0_0 = fma(X, r3_1_0_0, b3);
              const double r1_3_0_0 = fma(X, r2_2_0_0, 2.0 * r2_1_0_0);
              const double r0_4_0_0 = fma(X, r1_3_0_0, 3.0 * r1_2_0_0);
              g13_19 = fma(ek13_2, r0_4_0_0, g13_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_1_0_4 = X * r1_0_0_4;
              g13_10 = fma(ek13_3, r0_1_0_4, g13_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_1_1_3 = X * r1_0_1_3;
              g13_11 = fma(ek13_3, r0_1_1_3, g13_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_1_2_2 = X * r1_0_2_2;
              g13_12 = fma(ek13_3, r0_1_2_2, g13_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_1_3_1 = X * r1_0_3_1;
              g13_13 = fma(ek13_3, r0_1_3_1, g13_13);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g13_14 = fma(ek13_3, r0_2_0_3, g13_14);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g13_15 = fma(ek13_3, r0_2_1_2, g13_15);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g13_16 = fma(ek13_3, r0_2_2_1, g13_16);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g13_17 = fma(ek13_3, r0_3_0_2, g13_17);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g13_18 = fma(ek13_3, r0_3_1_1, g13_18);
              const double r3_1_0_1 = X * r4_0_0_1;
              const double r2_2_0_1 = fma(X, r3_1_0_1, r3_0_0_1);
              const double r1_3_0_1 = fma(X, r2_2_0_1, 2.0 * r2_1_0_1);
              const double r0_4_0_1 = fma(X, r1_3_0_1, 3.0 * r1_2_0_1);
              g13_19 = fma(ek13_3, r0_4_0_1, g13_19);
            }
            { const double eb = bi[5];
              o0_13 = fma(eb, g13_0, o0_13);
            }
            { const double eb = bi[6];
              o0_13 = fma(eb, g13_3, o0_13);
            }
            { const double eb = bi[7];
              o0_13 = fma(eb, g13_9, o0_13);
            }
            { const double eb = bi[8];
              o1_13 = fma(eb, g13_0, o1_13);
            }
            { const double eb = bi[9];
              o1_13 = fma(eb, g13_3, o1_13);
            }
            { const double eb = bi[10];
              o1_13 = fma(eb, g13_9, o1_13);
            }
            { const double eb = bi[11];
              o1_13 = fma(eb, g13_19, o1_13);
            }
            { const double eb = bi[12];
              o2_13 = fma(eb, g13_0, o2_13);
            }
            { const double eb = bi[13];
              o2_13 = fma(eb, g13_2, o2_13);
            }
            { const double eb = bi[14];
              o2_13 = fma(eb, g13_3, o2_13);
            }
            { const double eb = bi[15];
              o2_13 = fma(eb, g13_8, o2_13);
            }
            { const double eb = bi[16];
              o2_13 = fma(eb, g13_9, o2_13);
            }
            { const double eb = bi[17];
              o2_13 = fma(eb, g13_18, o2_13);
            }
            { const double eb = bi[18];
              o3_13 = fma(eb, g13_0, o3_13);
            }
            { const double eb = bi[19];
              o3_13 = fma(eb, g13_1, o3_13);
            }
            { const double eb = bi[20];
              o3_13 = fma(eb, g13_3, o3_13);
            }
            { const double eb = bi[21];
              o3_13 = fma(eb, g13_7, o3_13);
            }
            { const double eb = bi[22];
              o3_13 = fma(eb, g13_9, o3_13);
            }
            { const double eb = bi[23];
              o3_13 = fma(eb, g13_17, o3_13);
            }
            { const double eb = bi[24];
              o4_13 = fma(eb, g13_0, o4_13);
            }
            { const double eb = bi[25];
              o4_13 = fma(eb, g13_2, o4_13);
            }
            { const double eb = bi[26];
              o4_13 = fma(eb, g13_6, o4_13);
            }
            { const double eb = bi[27];
              o5_13 = fma(eb, g13_0, o5_13);
            }
            { const double eb = bi[28];
              o5_13 = fma(eb, g13_2, o5_13);
            }
            { const double eb = bi[29];
              o5_13 = fma(eb, g13_6, o5_13);
            }
            { const double eb = bi[30];
              o5_13 = fma(eb, g13_3, o5_13);
            }
            { const double eb = bi[31];
              o5_13 = fma(eb, g13_8, o5_13);
            }
            { const double eb = bi[32];
              o5_13 = fma(eb, g13_16, o5_13);
            }
            { const double eb = bi[33];
              o6_13 = fma(eb, g13_0, o6_13);
            }
            { const double eb = bi[34];
              o6_13 = fma(eb, g13_2, o6_13);
            }
            { const double eb = bi[35];
              o6_13 = fma(eb, g13_6, o6_13);
            }
            { const double eb = bi[36];
              o6_13 = fma(eb, g13_13, o6_13);
            }
            { const double eb = bi[37];
              o7_13 = fma(eb, g13_0, o7_13);
            }
            { const double eb = bi[38];
              o7_13 = fma(eb, g13_1, o7_13);
            }
            { const double eb = bi[39];
              o7_13 = fma(eb, g13_2, o7_13);
            }
            { const double eb = bi[40];
              o7_13 = fma(eb, g13_5, o7_13);
            }
            { const double eb = bi[41];
              o7_13 = fma(eb, g13_6, o7_13);
            }
            { const double eb = bi[42];
              o7_13 = fma(eb, g13_12, o7_13);
            }
            { const double eb = bi[43];
              o8_13 = fma(eb, g13_0, o8_13);
            }
            { const double eb = bi[44];
              o8_13 = fma(eb, g13_1, o8_13);
            }
            { const double eb = bi[45];
              o8_13 = fma(eb, g13_4, o8_13);
            }
            { const double eb = bi[46];
              o9_13 = fma(eb, g13_0, o9_13);
            }
            { const double eb = bi[47];
              o9_13 = fma(eb, g13_1, o9_13);
            }
            { const double eb = bi[48];
              o9_13 = fma(eb, g13_4, o9_13);
            }
            { const double eb = bi[49];
              o9_13 = fma(eb, g13_3, o9_13);
            }
            { const double eb = bi[50];
              o9_13 = fma(eb, g13_7, o9_13);
            }
            { const double eb = bi[51];
              o9_13 = fma(eb, g13_14, o9_13);
            }
            { const double eb = bi[52];
              o10_13 = fma(eb, g13_0, o10_13);
            }
            { const double eb = bi[53];
              o10_13 = fma(eb, g13_1, o10_13);
            }
            { const double eb = bi[54];
              o10_13 = fma(eb, g13_4, o10_13);
            }
            { const double eb = bi[55];
              o10_13 = fma(eb, g13_2, o10_13);
            }
            { const double eb = bi[56];
              o10_13 = fma(eb, g13_5, o10_13);
            }
            { const double eb = bi[57];
              o10_13 = fma(eb, g13_11, o10_13);
            }
            { const double eb = bi[58];
              o11_13 = fma(eb, g13_0, o11_13);
            }
            { const double eb = bi[59];
              o11_13 = fma(eb, g13_1, o11_13);
            }
            { const double eb = bi[60];
              o11_13 = fma(eb, g13_4, o11_13);
            }
            { const double eb = bi[61];
              o11_13 = fma(eb, g13_10, o11_13);
            }
            { const double eb = bi[62];
              o12_13 = fma(eb, g13_0, o12_13);
            }
            { const double eb = bi[63];
              o12_13 = fma(eb, g13_2, o12_13);
            }
            { const double eb = bi[64];
              o12_13 = fma(eb, g13_3, o12_13);
            }
            { const double eb = bi[65];
              o12_13 = fma(eb, g13_8, o12_13);
            }
            { const double eb = bi[66];
              o13_13 = fma(eb, g13_0, o13_13);
            }
            { const double eb = bi[67];
              o13_13 = fma(eb, g13_2, o13_13);
            }
            { const double eb = bi[68];
              o13_13 = fma(eb, g13_3, o13_13);
            }
            { const double eb = bi[69];
              o13_13 = fma(eb, g13_8, o13_13);
            }
            { const double eb = bi[70];
              o13_13 = fma(eb, g13_9, o13_13);
            }
            { const double eb = bi[71];
              o13_13 = fma(eb, g13_18, o13_13);
            }
            { const double eb = bi[72];
              o14_13 = fma(eb, g13_0, o14_13);
            }
            { const double eb = bi[73];
              o14_13 = fma(eb, g13_2, o14_13);
            }
            { const double eb = bi[74];
              o14_13 = fma(eb, g13_6, o14_13);
            }
            { const double eb = bi[75];
              o14_13 = fma(eb, g13_3, o14_13);
            }
            { const double eb = bi[76];
              o14_13 = fma(eb, g13_8, o14_13);
            }
            { const double eb = bi[77];
              o14_13 = fma(eb, g13_16, o14_13);
            }
            { const double eb = bi[78];
              o15_13 = fma(eb, g13_0, o15_13);
            }
            { const double eb = bi[79];
              o15_13 = fma(eb, g13_1, o15_13);
            }
            { const double eb = bi[80];
              o15_13 = fma(eb, g13_2, o15_13);
            }
            { const double eb = bi[81];
              o15_13 = fma(eb, g13_5, o15_13);
            }
            { const double eb = bi[82];
              o15_13 = fma(eb, g13_3, o15_13);
            }
            { const double eb = bi[83];
              o15_13 = fma(eb, g13_7, o15_13);
            }
            { const double eb = bi[84];
              o15_13 = fma(eb, g13_8, o15_13);
            }
            { const double eb = bi[85];
              o15_13 = fma(eb, g13_15, o15_13);
            }
            { const double eb = bi[86];
              o16_13 = fma(eb, g13_0, o16_13);
            }
            { const double eb = bi[87];
              o16_13 = fma(eb, g13_1, o16_13);
            }
            { const double eb = bi[88];
              o16_13 = fma(eb, g13_3, o16_13);
            }
            { const double eb = bi[89];
              o16_13 = fma(eb, g13_7, o16_13);
            }
            { const double eb = bi[90];
              o17_13 = fma(eb, g13_0, o17_13);
            }
            { const double eb = bi[91];
              o17_13 = fma(eb, g13_1, o17_13);
            }
            { const double eb = bi[92];
              o17_13 = fma(eb, g13_3, o17_13);
            }
            { const double eb = bi[93];
              o17_13 = fma(eb, g13_7, o17_13);
            }
            { const double eb = bi[94];
              o17_13 = fma(eb, g13_9, o17_13);
            }
            { const double eb = bi[95];
              o17_13 = fma(eb, g13_17, o17_13);
            }
            { const double eb = bi[96];
              o18_13 = fma(eb, g13_0, o18_13);
            }
            { const double eb = bi[97];
              o18_13 = fma(eb, g13_1, o18_13);
            }
            { const double eb = bi[98];
              o18_13 = fma(eb, g13_2, o18_13);
            }
            { const double eb = bi[99];
              o18_13 = fma(eb, g13_5, o18_13);
            }
            { const double eb = bi[100];
              o18_13 = fma(eb, g13_3, o18_13);
            }
            { const double eb = bi[101];
              o18_13 = fma(eb, g13_7, o18_13);
            }
            { const double eb = bi[102];
              o18_13 = fma(eb, g13_8, o18_13);
            }
            { const double eb = bi[103];
              o18_13 = fma(eb, g13_15, o18_13);
            }
            { const double eb = bi[104];
              o19_13 = fma(eb, g13_0, o19_13);
            }
            { const double eb = bi[105];
              o19_13 = fma(eb, g13_1, o19_13);
            }
            { const double eb = bi[106];
              o19_13 = fma(eb, g13_4, o19_13);
            }
            { const double eb = bi[107];
              o19_13 = fma(eb, g13_3, o19_13);
            }
            { const double eb = bi[108];
              o19_13 = fma(eb, g13_7, o19_13);
            }
            { const double eb = bi[109];
              o19_13 = fma(eb, g13_14, o19_13);
            }
            { const double eb = bi[110];
              o20_13 = fma(eb, g13_0, o20_13);
            }
            { const double eb = bi[111];
              o20_13 = fma(eb, g13_1, o20_13);
            }
            { const double eb = bi[112];
              o20_13 = fma(eb, g13_2, o20_13);
            }
            { const double eb = bi[113];
              o20_13 = fma(eb, g13_5, o20_13);
            }
            { const double eb = bi[114];
              o21_13 = fma(eb, g13_0, o21_13);
            }
            { const double eb = bi[115];
              o21_13 = fma(eb, g13_1, o21_13);
            }
            { const double eb = bi[116];
              o21_13 = fma(eb, g13_2, o21_13);
            }
            { const double eb = bi[117];
              o21_13 = fma(eb, g13_5, o21_13);
            }
            { const double eb = bi[118];
              o21_13 = fma(eb, g13_3, o21_13);
            }
            { const double eb = bi[119];
              o21_13 = fma(eb, g13_7, o21_13);
            }
            { const double eb = bi[120];
              o21_13 = fma(eb, g13_8, o21_13);
            }
            { const double eb = bi[121];
              o21_13 = fma(eb, g13_15, o21_13);
            }
            { const double eb = bi[122];
              o22_13 = fma(eb, g13_0, o22_13);
            }
            { const double eb = bi[123];
              o22_13 = fma(eb, g13_1, o22_13);
            }
            { const double eb = bi[124];
              o22_13 = fma(eb, g13_2, o22_13);
            }
            { const double eb = bi[125];
              o22_13 = fma(eb, g13_5, o22_13);
            }
            { const double eb = bi[126];
              o22_13 = fma(eb, g13_6, o22_13);
            }
            { const double eb = bi[127];
              o22_13 = fma(eb, g13_12, o22_13);
            }
            { const double eb = bi[128];
              o23_13 = fma(eb, g13_0, o23_13);
            }
            { const double eb = bi[129];
              o23_13 = fma(eb, g13_1, o23_13);
            }
            { const double eb = bi[130];
              o23_13 = fma(eb, g13_4, o23_13);
            }
            { const double eb = bi[131];
              o23_13 = fma(eb, g13_2, o23_13);
            }
            { const double eb = bi[132];
              o23_13 = fma(eb, g13_5, o23_13);
            }
            { const double eb = bi[133];
              o23_13 = fma(eb, g13_11, o23_13);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_13 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 1);
            o1_13 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 1);
            o2_13 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 1);
            o3_13 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 1);
            o4_13 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 1);
            o5_13 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 1);
            o6_13 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 1);
            o7_13 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 1);
            o8_13 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 1);
            o9_13 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 1);
            o10_13 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 1);
            o11_13 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 1);
            o12_13 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 1);
            o13_13 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 1);
            o14_13 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 1);
            o15_13 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 1);
            o16_13 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 1);
            o17_13 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 1);
            o18_13 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 1);
            o19_13 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 1);
            o20_13 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 1);
            o21_13 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 1);
            o22_13 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 1);
            o23_13 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 1);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_13 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o1_13 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o2_13 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o3_13 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o4_13 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o5_13 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o6_13 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o7_13 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o8_13 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o9_13 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o10_13 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o11_13 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o12_13 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o13_13 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o14_13 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o15_13 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o16_13 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o17_13 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o18_13 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o19_13 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o20_13 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o21_13 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o22_13 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 1)));
            e = fmax(e, fabs(o23_13 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 1)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Aad0_1 = PA[(fP + 0) * N + fJ + 1];
            const double Aad1_1 = PA[(fP + 1) * N + fJ + 1];
            const double Aad2_1 = PA[(fP + 2) * N + fJ + 1];
            const double Aad3_1 = PA[(fP + 3) * N + fJ + 1];
            const double Aad4_1 = PA[(fP + 4) * N + fJ + 1];
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
            const double Bbd0_1 = PB[(fQ + 0) * N + fJ + 1];
            const double Bbd1_1 = PB[(fQ + 1) * N + fJ + 1];
            const double Bbd2_1 = PB[(fQ + 2) * N + fJ + 1];
            const double Bbd3_1 = PB[(fQ + 3) * N + fJ + 1];
            const double Bad0_1 = PB[(fP + 0) * N + fJ + 1];
            const double Bad1_1 = PB[(fP + 1) * N + fJ + 1];
            const double Bad2_1 = PB[(fP + 2) * N + fJ + 1];
            const double Bad3_1 = PB[(fP + 3) * N + fJ + 1];
            const double Bad4_1 = PB[(fP + 4) * N + fJ + 1];
            const double Bad5_1 = PB[(fP + 5) * N + fJ + 1];
            const double Bbc0_3 = PB[(fQ + 0) * N + fI + 3];
            const double Bbc1_3 = PB[(fQ + 1) * N + fI + 3];
            const double Bbc2_3 = PB[(fQ + 2) * N + fI + 3];
            const double Bbc3_3 = PB[(fQ + 3) * N + fI + 3];
            const double Bac0_3 = PB[(fP + 0) * N + fI + 3];
            const double Bac1_3 = PB[(fP + 1) * N + fI + 3];
            const double Bac2_3 = PB[(fP + 2) * N + fI + 3];
            const double Bac3_3 = PB[(fP + 3) * N + fI + 3];
            const double Bac4_3 = PB[(fP + 4) * N + fI + 3];
            const double Bac5_3 = PB[(fP + 5) * N + fI + 3];
            jab0 += o0_13 * ptk13;
            jab1 += o1_13 * ptk13;
            jab2 += o2_13 * ptk13;
            jab3 += o3_13 * ptk13;
            jab4 += o4_13 * ptk13;
            jab5 += o5_13 * ptk13;
            jab6 += o6_13 * ptk13;
            jab7 += o7_13 * ptk13;
            jab8 += o8_13 * ptk13;
            jab9 += o9_13 * ptk13;
            jab10 += o10_13 * ptk13;
            jab11 += o11_13 * ptk13;
            jab12 += o12_13 * ptk13;
            jab13 += o13_13 * ptk13;
            jab14 += o14_13 * ptk13;
            jab15 += o15_13 * ptk13;
            jab16 += o16_13 * ptk13;
            jab17 += o17_13 * ptk13;
            jab18 += o18_13 * ptk13;
            jab19 += o19_13 * ptk13;
            jab20 += o20_13 * ptk13;
            jab21 += o21_13 * ptk13;
            jab22 += o22_13 * ptk13;
            jab23 += o23_13 * ptk13;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 1, 2.0 * deg * (o0_13 * ptb0 + o1_13 * ptb1 + o2_13 * ptb2 + o3_13 * ptb3 + o4_13 * ptb4 + o5_13 * ptb5 + o6_13 * ptb6 + o7_13 * ptb7 + o8_13 * ptb8 + o9_13 * ptb9 + o10_13 * ptb10 + o11_13 * ptb11 + o12_13 * ptb12 + o13_13 * ptb13 + o14_13 * ptb14 + o15_13 * ptb15 + o16_13 * ptb16 + o17_13 * ptb17 + o18_13 * ptb18 + o19_13 * ptb19 + o20_13 * ptb20 + o21_13 * ptb21 + o22_13 * ptb22 + o23_13 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_13 * Abd0_1 + o1_13 * Abd1_1 + o2_13 * Abd2_1 + o3_13 * Abd3_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_13 * Aad0_1 + o4_13 * Aad1_1 + o8_13 * Aad2_1 + o12_13 * Aad3_1 + o16_13 * Aad4_1 + o20_13 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_13 * Abc0_3 + o1_13 * Abc1_3 + o2_13 * Abc2_3 + o3_13 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_13 * Aac0_3 + o4_13 * Aac1_3 + o8_13 * Aac2_3 + o12_13 * Aac3_3 + o16_13 * Aac4_3 + o20_13 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_13 * Aad0_1 + o5_13 * Aad1_1 + o9_13 * Aad2_1 + o13_13 * Aad3_1 + o17_13 * Aad4_1 + o21_13 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_13 * Aac0_3 + o5_13 * Aac1_3 + o9_13 * Aac2_3 + o13_13 * Aac3_3 + o17_13 * Aac4_3 + o21_13 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_13 * Aad0_1 + o6_13 * Aad1_1 + o10_13 * Aad2_1 + o14_13 * Aad3_1 + o18_13 * Aad4_1 + o22_13 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_13 * Aac0_3 + o6_13 * Aac1_3 + o10_13 * Aac2_3 + o14_13 * Aac3_3 + o18_13 * Aac4_3 + o22_13 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_13 * Aad0_1 + o7_13 * Aad1_1 + o11_13 * Aad2_1 + o15_13 * Aad3_1 + o19_13 * Aad4_1 + o23_13 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_13 * Aac0_3 + o7_13 * Aac1_3 + o11_13 * Aac2_3 + o15_13 * Aac3_3 + o19_13 * Aac4_3 + o23_13 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_13 * Abd0_1 + o5_13 * Abd1_1 + o6_13 * Abd2_1 + o7_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o4_13 * Abc0_3 + o5_13 * Abc1_3 + o6_13 * Abc2_3 + o7_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_13 * Abd0_1 + o9_13 * Abd1_1 + o10_13 * Abd2_1 + o11_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o8_13 * Abc0_3 + o9_13 * Abc1_3 + o10_13 * Abc2_3 + o11_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_13 * Abd0_1 + o13_13 * Abd1_1 + o14_13 * Abd2_1 + o15_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o12_13 * Abc0_3 + o13_13 * Abc1_3 + o14_13 * Abc2_3 + o15_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o16_13 * Abd0_1 + o17_13 * Abd1_1 + o18_13 * Abd2_1 + o19_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o16_13 * Abc0_3 + o17_13 * Abc1_3 + o18_13 * Abc2_3 + o19_13 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o20_13 * Abd0_1 + o21_13 * Abd1_1 + o22_13 * Abd2_1 + o23_13 * Abd3_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o20_13 * Abc0_3 + o21_13 * Abc1_3 + o22_13 * Abc2_3 + o23_13 * Abc3_3));
            atomicAdd(KBacc + (fP + 0) * N + fI + 3, deg * (o0_13 * Bbd0_1 + o1_13 * Bbd1_1 + o2_13 * Bbd2_1 + o3_13 * Bbd3_1));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 3, deg * (o0_13 * Bad0_1 + o4_13 * Bad1_1 + o8_13 * Bad2_1 + o12_13 * Bad3_1 + o16_13 * Bad4_1 + o20_13 * Bad5_1));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 1, deg * (o0_13 * Bbc0_3 + o1_13 * Bbc1_3 + o2_13 * Bbc2_3 + o3_13 * Bbc3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 1, deg * (o0_13 * Bac0_3 + o4_13 * Bac1_3 + o8_13 * Bac2_3 + o12_13 * Bac3_3 + o16_13 * Bac4_3 + o20_13 * Bac5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 3, deg * (o1_13 * Bad0_1 + o5_13 * Bad1_1 + o9_13 * Bad2_1 + o13_13 * Bad3_1 + o17_13 * Bad4_1 + o21_13 * Bad5_1));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 1, deg * (o1_13 * Bac0_3 + o5_13 * Bac1_3 + o9_13 * Bac2_3 + o13_13 * Bac3_3 + o17_13 * Bac4_3 + o21_13 * Bac5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 3, deg * (o2_13 * Bad0_1 + o6_13 * Bad1_1 + o10_13 * Bad2_1 + o14_13 * Bad3_1 + o18_13 * Bad4_1 + o22_13 * Bad5_1));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 1, deg * (o2_13 * Bac0_3 + o6_13 * Bac1_3 + o10_13 * Bac2_3 + o14_13 * Bac3_3 + o18_13 * Bac4_3 + o22_13 * Bac5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 3, deg * (o3_13 * Bad0_1 + o7_13 * Bad1_1 + o11_13 * Bad2_1 + o15_13 * Bad3_1 + o19_13 * Bad4_1 + o23_13 * Bad5_1));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 1, deg * (o3_13 * Bac0_3 + o7_13 * Bac1_3 + o11_13 * Bac2_3 + o15_13 * Bac3_3 + o19_13 * Bac4_3 + o23_13 * Bac5_3));
            atomicAdd(KBacc + (fP + 1) * N + fI + 3, deg * (o4_13 * Bbd0_1 + o5_13 * Bbd1_1 + o6_13 * Bbd2_1 + o7_13 * Bbd3_1));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 1, deg * (o4_13 * Bbc0_3 + o5_13 * Bbc1_3 + o6_13 * Bbc2_3 + o7_13 * Bbc3_3));
            atomicAdd(KBacc + (fP + 2) * N + fI + 3, deg * (o8_13 * Bbd0_1 + o9_13 * Bbd1_1 + o10_13 * Bbd2_1 + o11_13 * Bbd3_1));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 1, deg * (o8_13 * Bbc0_3 + o9_13 * Bbc1_3 + o10_13 * Bbc2_3 + o11_13 * Bbc3_3));
            atomicAdd(KBacc + (fP + 3) * N + fI + 3, deg * (o12_13 * Bbd0_1 + o13_13 * Bbd1_1 + o14_13 * Bbd2_1 + o15_13 * Bbd3_1));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 1, deg * (o12_13 * Bbc0_3 + o13_13 * Bbc1_3 + o14_13 * Bbc2_3 + o15_13 * Bbc3_3));
            atomicAdd(KBacc + (fP + 4) * N + fI + 3, deg * (o16_13 * Bbd0_1 + o17_13 * Bbd1_1 + o18_13 * Bbd2_1 + o19_13 * Bbd3_1));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 1, deg * (o16_13 * Bbc0_3 + o17_13 * Bbc1_3 + o18_13 * Bbc2_3 + o19_13 * Bbc3_3));
            atomicAdd(KBacc + (fP + 5) * N + fI + 3, deg * (o20_13 * Bbd0_1 + o21_13 * Bbd1_1 + o22_13 * Bbd2_1 + o23_13 * Bbd3_1));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 1, deg * (o20_13 * Bbc0_3 + o21_13 * Bbc1_3 + o22_13 * Bbc2_3 + o23_13 * Bbc3_3));
          }
        } break;
        case 14: {  // ket functions [14]
          double o0_14 = 0;
          double o1_14 = 0;
          double o2_14 = 0;
          double o3_14 = 0;
          double o4_14 = 0;
          double o5_14 = 0;
          double o6_14 = 0;
          double o7_14 = 0;
          double o8_14 = 0;
          double o9_14 = 0;
          double o10_14 = 0;
          double o11_14 = 0;
          double o12_14 = 0;
          double o13_14 = 0;
          double o14_14 = 0;
          double o15_14 = 0;
          double o16_14 = 0;
          double o17_14 = 0;
          double o18_14 = 0;
          double o19_14 = 0;
          double o20_14 = 0;
          double o21_14 = 0;
          double o22_14 = 0;
          double o23_14 = 0;
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
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek14_0 = kj[44 * kS];
              const double ek14_1 = -kj[45 * kS];
              const double ek14_2 = -kj[46 * kS];
              const double ek14_3 = kj[47 * kS];
              g14_0 = fma(ek14_0, b0, g14_0);
              const double r0_0_0_1 = Z * b1;
              g14_1 = fma(ek14_0, r0_0_0_1, g14_1);
              g14_0 = fma(ek14_1, r0_0_0_1, g14_0);
              const double r0_0_1_0 = Y * b1;
              g14_2 = fma(ek14_0, r0_0_1_0, g14_2);
              g14_0 = fma(ek14_2, r0_0_1_0, g14_0);
              const double r0_1_0_0 = X * b1;
              g14_3 = fma(ek14_0, r0_1_0_0, g14_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g14_4 = fma(ek14_0, r0_0_0_2, g14_4);
              g14_1 = fma(ek14_1, r0_0_0_2, g14_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g14_5 = fma(ek14_0, r0_0_1_1, g14_5);
              g14_2 = fma(ek14_1, r0_0_1_1, g14_2);
              g14_1 = fma(ek14_2, r0_0_1_1, g14_1);
              g14_0 = fma(ek14_3, r0_0_1_1, g14_0);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g14_6 = fma(ek14_0, r0_0_2_0, g14_6);
              g14_2 = fma(ek14_2, r0_0_2_0, g14_2);
              const double r0_1_0_1 = X * r1_0_0_1;
              g14_7 = fma(ek14_0, r0_1_0_1, g14_7);
              g14_3 = fma(ek14_1, r0_1_0_1, g14_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g14_8 = fma(ek14_0, r0_1_1_0, g14_8);
              g14_3 = fma(ek14_2, r0_1_1_0, g14_3);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g14_9 = fma(ek14_0, r0_2_0_0, g14_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g14_10 = fma(ek14_0, r0_0_0_3, g14_10);
              g14_4 = fma(ek14_1, r0_0_0_3, g14_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g14_11 = fma(ek14_0, r0_0_1_2, g14_11);
              g14_5 = fma(ek14_1, r0_0_1_2, g14_5);
              g14_4 = fma(ek14_2, r0_0_1_2, g14_4);
              g14_1 = fma(ek14_3, r0_0_1_2, g14_1);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g14_12 = fma(ek14_0, r0_0_2_1, g14_12);
              g14_6 = fma(ek14_1, r0_0_2_1, g14_6);
              g14_5 = fma(ek14_2, r0_0_2_1, g14_5);
              g14_2 = fma(ek14_3, r0_0_2_1, g14_2);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g14_13 = fma(ek14_0, r0_0_3_0, g14_13);
              g14_6 = fma(ek14_2, r0_0_3_0, g14_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g14_14 = fma(ek14_0, r0_1_0_2, g14_14);
              g14_7 = fma(ek14_1, r0_1_0_2, g14_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g14_15 = fma(ek14_0, r0_1_1_1, g14_15);
              g14_8 = fma(ek14_1, r0_1_1_1, g14_8);
              g14_7 = fma(ek14_2, r0_1_1_1, g14_7);
              g14_3 = fma(ek14_3, r0_1_1_1, g14_3);
              const double r0_1_2_0 = X * r1_0_2_0;
              g14_16 = fma(ek14_0, r0_1_2_0, g14_16);
              g14_8 = fma(ek14_2, r0_1_2_0, g14_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g14_17 = fma(ek14_0, r0_2_0_1, g14_17);
              g14_9 = fma(ek14_1, r0_2_0_1, g14_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g14_18 = fma(ek14_0, r0_2_1_0, g14_18);
              g14_9 = fma(ek14_2, r0_2_1_0, g14_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g14_19 = fma(ek14_0, r0_3_0_0, g14_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g14_10 = fma(ek14_1, r0_0_0_4, g14_10);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g14_11 = fma(ek14_1, r0_0_1_3, g14_11);
              g14_10 = fma(ek14_2, r0_0_1_3, g14_10);
              g14_4 = fma(ek14_3, r0_0_1_3, g14_4);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g14_12 = fma(ek14_1, r0_0_2_2, g14_12);
              g14_11 = fma(ek14_2, r0_0_2_2, g14_11);
              g14_5 = fma(ek14_3, r0_0_2_2, g14_5);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g14_13 = fma(ek14_1, r0_0_3_1, g14_13);
              g14_12 = fma(ek14_2, r0_0_3_1, g14_12);
              g14_6 = fma(ek14_3, r0_0_3_1, g14_6);
              const double r3_0_1_0 = Y * b4;
              const double r2_0_2_0 = fma(Y, r3_0_1_0, b3);
              const double r1_0_3_0 = fma(Y, r2_0_2_0, 2.0 * r2_0_1_0);
              const double r0_0_4_0 = fma(Y, r1_0_3_0, 3.0 * r1_0_2_0);
              g14_13 = fma(ek14_2, r0_0_4_0, g14_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g14_14 = fma(ek14_1, r0_1_0_3, g14_14);
              const double r0_1_1_2 = X * r1_0_1_2;
              g14_15 = fma(ek14_1, r0_1_1_2, g14_15);
              g14_14 = fma(ek14_2, r0_1_1_2, g14_14);
              g14_7 = fma(ek14_3, r0_1_1_2, g14_7);
              const double r0_1_2_1 = X * r1_0_2_1;
              g14_16 = fma(ek14_1, r0_1_2_1, g14_16);
              g14_15 = fma(ek14_2, r0_1_2_1, g14_15);
              g14_8 = fma(ek14_3, r0_1_2_1, g14_8);
              const double r0_1_3_0 = X * r1_0_3_0;
              g14_16 = fma(ek14_2, r0_1_3_0, g14_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g14_17 = fma(ek14_1, r0_2_0_2, g14_17);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g14_18 = fma(ek14_1, r0_2_1_1, g14_18);
              g14_17 = fma(ek14_2, r0_2_1_1, g14_17);
              g14_9 = fma(ek14_3, r0_2_1_1, g14_9);
              const double r1_1_2_0 = X * r2_0_2_0;
              const double r0_2_2_0 = fma(X, r1_1_2_0, r1_0_2_0);
              g14_18 = fma(ek14_2, r0_2_2_0, g14_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g14_19 = fma(ek14_1, r0_3_0_1, g14_19);
              const double r2_1_1_0 = X * r3_0_1_0;
              const double r1_2_1_0 = fma(X, r2_1_1_0, r2_0_1_0);
              const double r0_3_1_0 = fma(X, r1_2_1_0, 2.0 * r1_1_1_0);
              g14_19 = fma(ek14_2, r0_3_1_0, g14_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g14_10 = fma(ek14_3, r0_0_1_4, g14_10);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g14_11 = fma(ek14_3, r0_0_2_3, g14_11);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g14_12 = fma(ek14_3, r0_0_3_2, g14_12);
              const double r3_0_1_1 = Y * r4_0_0_1;
              const double r2_0_2_1 = fma(Y, r3_0_1_1, r3_0_0_1);
              const double r1_0_3_1 = fma(Y, r2_0_2_1, 2.0 * r2_0_1_1);
              const double r0_0_4_1 = fma(Y, r1_0_3_1, 3.0 * r1_0_2_1);
              g14_13 = fma(ek14_3, r0_0_4_1, g14_13);
              const double r0_1_1_3 = X * r1_0_1_3;
              g14_14 = fma(ek14_3, r0_1_1_3, g14_14);
              const double r0_1_2_2 = X * r1_0_2_2;
              g14_15 = fma(ek14_3, r0_1_2_2, g14_15);
              const double r0_1_3_1 = X * r1_0_3_1;
              g14_16 = fma(ek14_3, r0_1_3_1, g14_16);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g14_17 = fma(ek14_3, r0_2_1_2, g14_17);
              const double r1_1_2_1 = X * r2_0_2_1;
              const double r0_2_2_1 = fma(X, r1_1_2_1, r1_0_2_1);
              g14_18 = fma(ek14_3, r0_2_2_1, g14_18);
              const double r2_1_1_1 = X * r3_0_1_1;
              const double r1_2_1_1 = fma(X, r2_1_1_1, r2_0_1_1);
              const double r0_3_1_1 = fma(X, r1_2_1_1, 2.0 * r1_1_1_1);
              g14_19 = fma(ek14_3, r0_3_1_1, g14_19);
            }
            { const double eb = bi[5];
              o0_14 = fma(eb, g14_0, o0_14);
            }
            { const double eb = bi[6];
              o0_14 = fma(eb, g14_3, o0_14);
            }
            { const double eb = bi[7];
              o0_14 = fma(eb, g14_9, o0_14);
            }
            { const double eb = bi[8];
              o1_14 = fma(eb, g14_0, o1_14);
            }
            { const double eb = bi[9];
              o1_14 = fma(eb, g14_3, o1_14);
            }
            { const double eb = bi[10];
              o1_14 = fma(eb, g14_9, o1_14);
            }
            { const double eb = bi[11];
              o1_14 = fma(eb, g14_19, o1_14);
            }
            { const double eb = bi[12];
              o2_14 = fma(eb, g14_0, o2_14);
            }
            { const double eb = bi[13];
              o2_14 = fma(eb, g14_2, o2_14);
            }
            { const double eb = bi[14];
              o2_14 = fma(eb, g14_3, o2_14);
            }
            { const double eb = bi[15];
              o2_14 = fma(eb, g14_8, o2_14);
            }
            { const double eb = bi[16];
              o2_14 = fma(eb, g14_9, o2_14);
            }
            { const double eb = bi[17];
              o2_14 = fma(eb, g14_18, o2_14);
            }
            { const double eb = bi[18];
              o3_14 = fma(eb, g14_0, o3_14);
            }
            { const double eb = bi[19];
              o3_14 = fma(eb, g14_1, o3_14);
            }
            { const double eb = bi[20];
              o3_14 = fma(eb, g14_3, o3_14);
            }
            { const double eb = bi[21];
              o3_14 = fma(eb, g14_7, o3_14);
            }
            { const double eb = bi[22];
              o3_14 = fma(eb, g14_9, o3_14);
            }
            { const double eb = bi[23];
              o3_14 = fma(eb, g14_17, o3_14);
            }
            { const double eb = bi[24];
              o4_14 = fma(eb, g14_0, o4_14);
            }
            { const double eb = bi[25];
              o4_14 = fma(eb, g14_2, o4_14);
            }
            { const double eb = bi[26];
              o4_14 = fma(eb, g14_6, o4_14);
            }
            { const double eb = bi[27];
              o5_14 = fma(eb, g14_0, o5_14);
            }
            { const double eb = bi[28];
              o5_14 = fma(eb, g14_2, o5_14);
            }
            { const double eb = bi[29];
              o5_14 = fma(eb, g14_6, o5_14);
            }
            { const double eb = bi[30];
              o5_14 = fma(eb, g14_3, o5_14);
            }
            { const double eb = bi[31];
              o5_14 = fma(eb, g14_8, o5_14);
            }
            { const double eb = bi[32];
              o5_14 = fma(eb, g14_16, o5_14);
            }
            { const double eb = bi[33];
              o6_14 = fma(eb, g14_0, o6_14);
            }
            { const double eb = bi[34];
              o6_14 = fma(eb, g14_2, o6_14);
            }
            { const double eb = bi[35];
              o6_14 = fma(eb, g14_6, o6_14);
            }
            { const double eb = bi[36];
              o6_14 = fma(eb, g14_13, o6_14);
            }
            { const double eb = bi[37];
              o7_14 = fma(eb, g14_0, o7_14);
            }
            { const double eb = bi[38];
              o7_14 = fma(eb, g14_1, o7_14);
            }
            { const double eb = bi[39];
              o7_14 = fma(eb, g14_2, o7_14);
            }
            { const double eb = bi[40];
              o7_14 = fma(eb, g14_5, o7_14);
            }
            { const double eb = bi[41];
              o7_14 = fma(eb, g14_6, o7_14);
            }
            { const double eb = bi[42];
              o7_14 = fma(eb, g14_12, o7_14);
            }
            { const double eb = bi[43];
              o8_14 = fma(eb, g14_0, o8_14);
            }
            { const double eb = bi[44];
              o8_14 = fma(eb, g14_1, o8_14);
            }
            { const double eb = bi[45];
              o8_14 = fma(eb, g14_4, o8_14);
            }
            { const double eb = bi[46];
              o9_14 = fma(eb, g14_0, o9_14);
            }
            { const double eb = bi[47];
              o9_14 = fma(eb, g14_1, o9_14);
            }
            { const double eb = bi[48];
              o9_14 = fma(eb, g14_4, o9_14);
            }
            { const double eb = bi[49];
              o9_14 = fma(eb, g14_3, o9_14);
            }
            { const double eb = bi[50];
              o9_14 = fma(eb, g14_7, o9_14);
            }
            { const double eb = bi[51];
              o9_14 = fma(eb, g14_14, o9_14);
            }
            { const double eb = bi[52];
              o10_14 = fma(eb, g14_0, o10_14);
            }
            { const double eb = bi[53];
              o10_14 = fma(eb, g14_1, o10_14);
            }
            { const double eb = bi[54];
              o10_14 = fma(eb, g14_4, o10_14);
            }
            { const double eb = bi[55];
              o10_14 = fma(eb, g14_2, o10_14);
            }
            { const double eb = bi[56];
              o10_14 = fma(eb, g14_5, o10_14);
            }
            { const double eb = bi[57];
              o10_14 = fma(eb, g14_11, o10_14);
            }
            { const double eb = bi[58];
              o11_14 = fma(eb, g14_0, o11_14);
            }
            { const double eb = bi[59];
              o11_14 = fma(eb, g14_1, o11_14);
            }
            { const double eb = bi[60];
              o11_14 = fma(eb, g14_4, o11_14);
            }
            { const double eb = bi[61];
              o11_14 = fma(eb, g14_10, o11_14);
            }
            { const double eb = bi[62];
              o12_14 = fma(eb, g14_0, o12_14);
            }
            { const double eb = bi[63];
              o12_14 = fma(eb, g14_2, o12_14);
            }
            { const double eb = bi[64];
              o12_14 = fma(eb, g14_3, o12_14);
            }
            { const double eb = bi[65];
              o12_14 = fma(eb, g14_8, o12_14);
            }
            { const double eb = bi[66];
              o13_14 = fma(eb, g14_0, o13_14);
            }
            { const double eb = bi[67];
              o13_14 = fma(eb, g14_2, o13_14);
            }
            { const double eb = bi[68];
              o13_14 = fma(eb, g14_3, o13_14);
            }
            { const double eb = bi[69];
              o13_14 = fma(eb, g14_8, o13_14);
            }
            { const double eb = bi[70];
              o13_14 = fma(eb, g14_9, o13_14);
            }
            { const double eb = bi[71];
              o13_14 = fma(eb, g14_18, o13_14);
            }
            { const double eb = bi[72];
              o14_14 = fma(eb, g14_0, o14_14);
            }
            { const double eb = bi[73];
              o14_14 = fma(eb, g14_2, o14_14);
            }
            { const double eb = bi[74];
              o14_14 = fma(eb, g14_6, o14_14);
            }
            { const double eb = bi[75];
              o14_14 = fma(eb, g14_3, o14_14);
            }
            { const double eb = bi[76];
              o14_14 = fma(eb, g14_8, o14_14);
            }
            { const double eb = bi[77];
              o14_14 = fma(eb, g14_16, o14_14);
            }
            { const double eb = bi[78];
              o15_14 = fma(eb, g14_0, o15_14);
            }
            { const double eb = bi[79];
              o15_14 = fma(eb, g14_1, o15_14);
            }
            { const double eb = bi[80];
              o15_14 = fma(eb, g14_2, o15_14);
            }
            { const double eb = bi[81];
              o15_14 = fma(eb, g14_5, o15_14);
            }
            { const double eb = bi[82];
              o15_14 = fma(eb, g14_3, o15_14);
            }
            { const double eb = bi[83];
              o15_14 = fma(eb, g14_7, o15_14);
            }
            { const double eb = bi[84];
              o15_14 = fma(eb, g14_8, o15_14);
            }
            { const double eb = bi[85];
              o15_14 = fma(eb, g14_15, o15_14);
            }
            { const double eb = bi[86];
              o16_14 = fma(eb, g14_0, o16_14);
            }
            { const double eb = bi[87];
              o16_14 = fma(eb, g14_1, o16_14);
            }
            { const double eb = bi[88];
              o16_14 = fma(eb, g14_3, o16_14);
            }
            { const double eb = bi[89];
              o16_14 = fma(eb, g14_7, o16_14);
            }
            { const double eb = bi[90];
              o17_14 = fma(eb, g14_0, o17_14);
            }
            { const double eb = bi[91];
              o17_14 = fma(eb, g14_1, o17_14);
            }
            { const double eb = bi[92];
              o17_14 = fma(eb, g14_3, o17_14);
            }
            { const double eb = bi[93];
              o17_14 = fma(eb, g14_7, o17_14);
            }
            { const double eb = bi[94];
              o17_14 = fma(eb, g14_9, o17_14);
            }
            { const double eb = bi[95];
              o17_14 = fma(eb, g14_17, o17_14);
            }
            { const double eb = bi[96];
              o18_14 = fma(eb, g14_0, o18_14);
            }
            { const double eb = bi[97];
              o18_14 = fma(eb, g14_1, o18_14);
            }
            { const double eb = bi[98];
              o18_14 = fma(eb, g14_2, o18_14);
            }
            { const double eb = bi[99];
              o18_14 = fma(eb, g14_5, o18_14);
            }
            { const double eb = bi[100];
              o18_14 = fma(eb, g14_3, o18_14);
            }
            { const double eb = bi[101];
              o18_14 = fma(eb, g14_7, o18_14);
            }
            { const double eb = bi[102];
              o18_14 = fma(eb, g14_8, o18_14);
            }
            { const double eb = bi[103];
              o18_14 = fma(eb, g14_15, o18_14);
            }
            { const double eb = bi[104];
              o19_14 = fma(eb, g14_0, o19_14);
            }
            { const double eb = bi[105];
              o19_14 = fma(eb, g14_1, o19_14);
            }
            { const double eb = bi[106];
              o19_14 = fma(eb, g14_4, o19_14);
            }
            { const double eb = bi[107];
              o19_14 = fma(eb, g14_3, o19_14);
            }
            { const double eb = bi[108];
              o19_14 = fma(eb, g14_7, o19_14);
            }
            { const double eb = bi[109];
              o19_14 = fma(eb, g14_14, o19_14);
            }
            { const double eb = bi[110];
              o20_14 = fma(eb, g14_0, o20_14);
            }
            { const double eb = bi[111];
              o20_14 = fma(eb, g14_1, o20_14);
            }
            { const double eb = bi[112];
              o20_14 = fma(eb, g14_2, o20_14);
            }
            { const double eb = bi[113];
              o20_14 = fma(eb, g14_5, o20_14);
            }
            { const double eb = bi[114];
              o21_14 = fma(eb, g14_0, o21_14);
            }
            { const double eb = bi[115];
              o21_14 = fma(eb, g14_1, o21_14);
            }
            { const double eb = bi[116];
              o21_14 = fma(eb, g14_2, o21_14);
            }
            { const double eb = bi[117];
              o21_14 = fma(eb, g14_5, o21_14);
            }
            { const double eb = bi[118];
              o21_14 = fma(eb, g14_3, o21_14);
            }
            { const double eb = bi[119];
              o21_14 = fma(eb, g14_7, o21_14);
            }
            { const double eb = bi[120];
              o21_14 = fma(eb, g14_8, o21_14);
            }
            { const double eb = bi[121];
              o21_14 = fma(eb, g14_15, o21_14);
            }
            { const double eb = bi[122];
              o22_14 = fma(eb, g14_0, o22_14);
            }
            { const double eb = bi[123];
              o22_14 = fma(eb, g14_1, o22_14);
            }
            { const double eb = bi[124];
              o22_14 = fma(eb, g14_2, o22_14);
            }
            { const double eb = bi[125];
              o22_14 = fma(eb, g14_5, o22_14);
            }
            { const double eb = bi[126];
              o22_14 = fma(eb, g14_6, o22_14);
            }
            { const double eb = bi[127];
              o22_14 = fma(eb, g14_12, o22_14);
            }
            { const double eb = bi[128];
              o23_14 = fma(eb, g14_0, o23_14);
            }
            { const double eb = bi[129];
              o23_14 = fma(eb, g14_1, o23_14);
            }
            { const double eb = bi[130];
              o23_14 = fma(eb, g14_4, o23_14);
            }
            { const double eb = bi[131];
              o23_14 = fma(eb, g14_2, o23_14);
            }
            { const double eb = bi[132];
              o23_14 = fma(eb, g14_5, o23_14);
            }
            { const double eb = bi[133];
              o23_14 = fma(eb, g14_11, o23_14);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_14 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 2);
            o1_14 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 2);
            o2_14 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 2);
            o3_14 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 2);
            o4_14 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 2);
            o5_14 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 2);
            o6_14 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 2);
            o7_14 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 2);
            o8_14 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 2);
            o9_14 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 2);
            o10_14 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 2);
            o11_14 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 2);
            o12_14 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 2);
            o13_14 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 2);
            o14_14 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 2);
            o15_14 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 2);
            o16_14 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 2);
            o17_14 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 2);
            o18_14 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 2);
            o19_14 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 2);
            o20_14 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 2);
            o21_14 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 2);
            o22_14 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 2);
            o23_14 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 2);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_14 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o1_14 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o2_14 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o3_14 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o4_14 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o5_14 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o6_14 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o7_14 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o8_14 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o9_14 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o10_14 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o11_14 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o12_14 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o13_14 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o14_14 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o15_14 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o16_14 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o17_14 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o18_14 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o19_14 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o20_14 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o21_14 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o22_14 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 2)));
            e = fmax(e, fabs(o23_14 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 2)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk14 = PT[(fI + 3) * N + fJ + 2];
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
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Aad0_2 = PA[(fP + 0) * N + fJ + 2];
            const double Aad1_2 = PA[(fP + 1) * N + fJ + 2];
            const double Aad2_2 = PA[(fP + 2) * N + fJ + 2];
            const double Aad3_2 = PA[(fP + 3) * N + fJ + 2];
            const double Aad4_2 = PA[(fP + 4) * N + fJ + 2];
            const double Aad5_2 = PA[(fP + 5) * N + fJ + 2];
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
            const double Bbd0_2 = PB[(fQ + 0) * N + fJ + 2];
            const double Bbd1_2 = PB[(fQ + 1) * N + fJ + 2];
            const double Bbd2_2 = PB[(fQ + 2) * N + fJ + 2];
            const double Bbd3_2 = PB[(fQ + 3) * N + fJ + 2];
            const double Bad0_2 = PB[(fP + 0) * N + fJ + 2];
            const double Bad1_2 = PB[(fP + 1) * N + fJ + 2];
            const double Bad2_2 = PB[(fP + 2) * N + fJ + 2];
            const double Bad3_2 = PB[(fP + 3) * N + fJ + 2];
            const double Bad4_2 = PB[(fP + 4) * N + fJ + 2];
            const double Bad5_2 = PB[(fP + 5) * N + fJ + 2];
            const double Bbc0_3 = PB[(fQ + 0) * N + fI + 3];
            const double Bbc1_3 = PB[(fQ + 1) * N + fI + 3];
            const double Bbc2_3 = PB[(fQ + 2) * N + fI + 3];
            const double Bbc3_3 = PB[(fQ + 3) * N + fI + 3];
            const double Bac0_3 = PB[(fP + 0) * N + fI + 3];
            const double Bac1_3 = PB[(fP + 1) * N + fI + 3];
            const double Bac2_3 = PB[(fP + 2) * N + fI + 3];
            const double Bac3_3 = PB[(fP + 3) * N + fI + 3];
            const double Bac4_3 = PB[(fP + 4) * N + fI + 3];
            const double Bac5_3 = PB[(fP + 5) * N + fI + 3];
            jab0 += o0_14 * ptk14;
            jab1 += o1_14 * ptk14;
            jab2 += o2_14 * ptk14;
            jab3 += o3_14 * ptk14;
            jab4 += o4_14 * ptk14;
            jab5 += o5_14 * ptk14;
            jab6 += o6_14 * ptk14;
            jab7 += o7_14 * ptk14;
            jab8 += o8_14 * ptk14;
            jab9 += o9_14 * ptk14;
            jab10 += o10_14 * ptk14;
            jab11 += o11_14 * ptk14;
            jab12 += o12_14 * ptk14;
            jab13 += o13_14 * ptk14;
            jab14 += o14_14 * ptk14;
            jab15 += o15_14 * ptk14;
            jab16 += o16_14 * ptk14;
            jab17 += o17_14 * ptk14;
            jab18 += o18_14 * ptk14;
            jab19 += o19_14 * ptk14;
            jab20 += o20_14 * ptk14;
            jab21 += o21_14 * ptk14;
            jab22 += o22_14 * ptk14;
            jab23 += o23_14 * ptk14;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 2, 2.0 * deg * (o0_14 * ptb0 + o1_14 * ptb1 + o2_14 * ptb2 + o3_14 * ptb3 + o4_14 * ptb4 + o5_14 * ptb5 + o6_14 * ptb6 + o7_14 * ptb7 + o8_14 * ptb8 + o9_14 * ptb9 + o10_14 * ptb10 + o11_14 * ptb11 + o12_14 * ptb12 + o13_14 * ptb13 + o14_14 * ptb14 + o15_14 * ptb15 + o16_14 * ptb16 + o17_14 * ptb17 + o18_14 * ptb18 + o19_14 * ptb19 + o20_14 * ptb20 + o21_14 * ptb21 + o22_14 * ptb22 + o23_14 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_14 * Abd0_2 + o1_14 * Abd1_2 + o2_14 * Abd2_2 + o3_14 * Abd3_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_14 * Aad0_2 + o4_14 * Aad1_2 + o8_14 * Aad2_2 + o12_14 * Aad3_2 + o16_14 * Aad4_2 + o20_14 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_14 * Abc0_3 + o1_14 * Abc1_3 + o2_14 * Abc2_3 + o3_14 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_14 * Aac0_3 + o4_14 * Aac1_3 + o8_14 * Aac2_3 + o12_14 * Aac3_3 + o16_14 * Aac4_3 + o20_14 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_14 * Aad0_2 + o5_14 * Aad1_2 + o9_14 * Aad2_2 + o13_14 * Aad3_2 + o17_14 * Aad4_2 + o21_14 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_14 * Aac0_3 + o5_14 * Aac1_3 + o9_14 * Aac2_3 + o13_14 * Aac3_3 + o17_14 * Aac4_3 + o21_14 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_14 * Aad0_2 + o6_14 * Aad1_2 + o10_14 * Aad2_2 + o14_14 * Aad3_2 + o18_14 * Aad4_2 + o22_14 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_14 * Aac0_3 + o6_14 * Aac1_3 + o10_14 * Aac2_3 + o14_14 * Aac3_3 + o18_14 * Aac4_3 + o22_14 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_14 * Aad0_2 + o7_14 * Aad1_2 + o11_14 * Aad2_2 + o15_14 * Aad3_2 + o19_14 * Aad4_2 + o23_14 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_14 * Aac0_3 + o7_14 * Aac1_3 + o11_14 * Aac2_3 + o15_14 * Aac3_3 + o19_14 * Aac4_3 + o23_14 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_14 * Abd0_2 + o5_14 * Abd1_2 + o6_14 * Abd2_2 + o7_14 * Abd3_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o4_14 * Abc0_3 + o5_14 * Abc1_3 + o6_14 * Abc2_3 + o7_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_14 * Abd0_2 + o9_14 * Abd1_2 + o10_14 * Abd2_2 + o11_14 * Abd3_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o8_14 * Abc0_3 + o9_14 * Abc1_3 + o10_14 * Abc2_3 + o11_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_14 * Abd0_2 + o13_14 * Abd1_2 + o14_14 * Abd2_2 + o15_14 * Abd3_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o12_14 * Abc0_3 + o13_14 * Abc1_3 + o14_14 * Abc2_3 + o15_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o16_14 * Abd0_2 + o17_14 * Abd1_2 + o18_14 * Abd2_2 + o19_14 * Abd3_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o16_14 * Abc0_3 + o17_14 * Abc1_3 + o18_14 * Abc2_3 + o19_14 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o20_14 * Abd0_2 + o21_14 * Abd1_2 + o22_14 * Abd2_2 + o23_14 * Abd3_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o20_14 * Abc0_3 + o21_14 * Abc1_3 + o22_14 * Abc2_3 + o23_14 * Abc3_3));
            atomicAdd(KBacc + (fP + 0) * N + fI + 3, deg * (o0_14 * Bbd0_2 + o1_14 * Bbd1_2 + o2_14 * Bbd2_2 + o3_14 * Bbd3_2));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 3, deg * (o0_14 * Bad0_2 + o4_14 * Bad1_2 + o8_14 * Bad2_2 + o12_14 * Bad3_2 + o16_14 * Bad4_2 + o20_14 * Bad5_2));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 2, deg * (o0_14 * Bbc0_3 + o1_14 * Bbc1_3 + o2_14 * Bbc2_3 + o3_14 * Bbc3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 2, deg * (o0_14 * Bac0_3 + o4_14 * Bac1_3 + o8_14 * Bac2_3 + o12_14 * Bac3_3 + o16_14 * Bac4_3 + o20_14 * Bac5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 3, deg * (o1_14 * Bad0_2 + o5_14 * Bad1_2 + o9_14 * Bad2_2 + o13_14 * Bad3_2 + o17_14 * Bad4_2 + o21_14 * Bad5_2));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 2, deg * (o1_14 * Bac0_3 + o5_14 * Bac1_3 + o9_14 * Bac2_3 + o13_14 * Bac3_3 + o17_14 * Bac4_3 + o21_14 * Bac5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 3, deg * (o2_14 * Bad0_2 + o6_14 * Bad1_2 + o10_14 * Bad2_2 + o14_14 * Bad3_2 + o18_14 * Bad4_2 + o22_14 * Bad5_2));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 2, deg * (o2_14 * Bac0_3 + o6_14 * Bac1_3 + o10_14 * Bac2_3 + o14_14 * Bac3_3 + o18_14 * Bac4_3 + o22_14 * Bac5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 3, deg * (o3_14 * Bad0_2 + o7_14 * Bad1_2 + o11_14 * Bad2_2 + o15_14 * Bad3_2 + o19_14 * Bad4_2 + o23_14 * Bad5_2));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 2, deg * (o3_14 * Bac0_3 + o7_14 * Bac1_3 + o11_14 * Bac2_3 + o15_14 * Bac3_3 + o19_14 * Bac4_3 + o23_14 * Bac5_3));
            atomicAdd(KBacc + (fP + 1) * N + fI + 3, deg * (o4_14 * Bbd0_2 + o5_14 * Bbd1_2 + o6_14 * Bbd2_2 + o7_14 * Bbd3_2));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 2, deg * (o4_14 * Bbc0_3 + o5_14 * Bbc1_3 + o6_14 * Bbc2_3 + o7_14 * Bbc3_3));
            atomicAdd(KBacc + (fP + 2) * N + fI + 3, deg * (o8_14 * Bbd0_2 + o9_14 * Bbd1_2 + o10_14 * Bbd2_2 + o11_14 * Bbd3_2));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 2, deg * (o8_14 * Bbc0_3 + o9_14 * Bbc1_3 + o10_14 * Bbc2_3 + o11_14 * Bbc3_3));
            atomicAdd(KBacc + (fP + 3) * N + fI + 3, deg * (o12_14 * Bbd0_2 + o13_14 * Bbd1_2 + o14_14 * Bbd2_2 + o15_14 * Bbd3_2));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 2, deg * (o12_14 * Bbc0_3 + o13_14 * Bbc1_3 + o14_14 * Bbc2_3 + o15_14 * Bbc3_3));
            atomicAdd(KBacc + (fP + 4) * N + fI + 3, deg * (o16_14 * Bbd0_2 + o17_14 * Bbd1_2 + o18_14 * Bbd2_2 + o19_14 * Bbd3_2));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 2, deg * (o16_14 * Bbc0_3 + o17_14 * Bbc1_3 + o18_14 * Bbc2_3 + o19_14 * Bbc3_3));
            atomicAdd(KBacc + (fP + 5) * N + fI + 3, deg * (o20_14 * Bbd0_2 + o21_14 * Bbd1_2 + o22_14 * Bbd2_2 + o23_14 * Bbd3_2));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 2, deg * (o20_14 * Bbc0_3 + o21_14 * Bbc1_3 + o22_14 * Bbc2_3 + o23_14 * Bbc3_3));
          }
        } break;
        case 15: {  // ket functions [15]
          double o0_15 = 0;
          double o1_15 = 0;
          double o2_15 = 0;
          double o3_15 = 0;
          double o4_15 = 0;
          double o5_15 = 0;
          double o6_15 = 0;
          double o7_15 = 0;
          double o8_15 = 0;
          double o9_15 = 0;
          double o10_15 = 0;
          double o11_15 = 0;
          double o12_15 = 0;
          double o13_15 = 0;
          double o14_15 = 0;
          double o15_15 = 0;
          double o16_15 = 0;
          double o17_15 = 0;
          double o18_15 = 0;
          double o19_15 = 0;
          double o20_15 = 0;
          double o21_15 = 0;
          double o22_15 = 0;
          double o23_15 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 134;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
              const double* __restrict__ kj = kprim + (long long)j * 51 * kS;
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
              const double ek15_0 = kj[48 * kS];
              const double ek15_1 = -kj[49 * kS];
              const double ek15_2 = kj[50 * kS];
              g15_0 = fma(ek15_0, b0, g15_0);
              const double r0_0_0_1 = Z * b1;
              g15_1 = fma(ek15_0, r0_0_0_1, g15_1);
              g15_0 = fma(ek15_1, r0_0_0_1, g15_0);
              const double r0_0_1_0 = Y * b1;
              g15_2 = fma(ek15_0, r0_0_1_0, g15_2);
              const double r0_1_0_0 = X * b1;
              g15_3 = fma(ek15_0, r0_1_0_0, g15_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g15_4 = fma(ek15_0, r0_0_0_2, g15_4);
              g15_1 = fma(ek15_1, r0_0_0_2, g15_1);
              g15_0 = fma(ek15_2, r0_0_0_2, g15_0);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g15_5 = fma(ek15_0, r0_0_1_1, g15_5);
              g15_2 = fma(ek15_1, r0_0_1_1, g15_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g15_6 = fma(ek15_0, r0_0_2_0, g15_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g15_7 = fma(ek15_0, r0_1_0_1, g15_7);
              g15_3 = fma(ek15_1, r0_1_0_1, g15_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g15_8 = fma(ek15_0, r0_1_1_0, g15_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g15_9 = fma(ek15_0, r0_2_0_0, g15_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g15_10 = fma(ek15_0, r0_0_0_3, g15_10);
              g15_4 = fma(ek15_1, r0_0_0_3, g15_4);
              g15_1 = fma(ek15_2, r0_0_0_3, g15_1);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g15_11 = fma(ek15_0, r0_0_1_2, g15_11);
              g15_5 = fma(ek15_1, r0_0_1_2, g15_5);
              g15_2 = fma(ek15_2, r0_0_1_2, g15_2);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g15_12 = fma(ek15_0, r0_0_2_1, g15_12);
              g15_6 = fma(ek15_1, r0_0_2_1, g15_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g15_13 = fma(ek15_0, r0_0_3_0, g15_13);
              const double r0_1_0_2 = X * r1_0_0_2;
              g15_14 = fma(ek15_0, r0_1_0_2, g15_14);
              g15_7 = fma(ek15_1, r0_1_0_2, g15_7);
              g15_3 = fma(ek15_2, r0_1_0_2, g15_3);
              const double r0_1_1_1 = X * r1_0_1_1;
              g15_15 = fma(ek15_0, r0_1_1_1, g15_15);
              g15_8 = fma(ek15_1, r0_1_1_1, g15_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g15_16 = fma(ek15_0, r0_1_2_0, g15_16);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g15_17 = fma(ek15_0, r0_2_0_1, g15_17);
              g15_9 = fma(ek15_1, r0_2_0_1, g15_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g15_18 = fma(ek15_0, r0_2_1_0, g15_18);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g15_19 = fma(ek15_0, r0_3_0_0, g15_19);
              const double r3_0_0_1 = Z * b4;
              const double r2_0_0_2 = fma(Z, r3_0_0_1, b3);
              const double r1_0_0_3 = fma(Z, r2_0_0_2, 2.0 * r2_0_0_1);
              const double r0_0_0_4 = fma(Z, r1_0_0_3, 3.0 * r1_0_0_2);
              g15_10 = fma(ek15_1, r0_0_0_4, g15_10);
              g15_4 = fma(ek15_2, r0_0_0_4, g15_4);
              const double r0_0_1_3 = Y * r1_0_0_3;
              g15_11 = fma(ek15_1, r0_0_1_3, g15_11);
              g15_5 = fma(ek15_2, r0_0_1_3, g15_5);
              const double r1_0_1_2 = Y * r2_0_0_2;
              const double r0_0_2_2 = fma(Y, r1_0_1_2, r1_0_0_2);
              g15_12 = fma(ek15_1, r0_0_2_2, g15_12);
              g15_6 = fma(ek15_2, r0_0_2_2, g15_6);
              const double r2_0_1_1 = Y * r3_0_0_1;
              const double r1_0_2_1 = fma(Y, r2_0_1_1, r2_0_0_1);
              const double r0_0_3_1 = fma(Y, r1_0_2_1, 2.0 * r1_0_1_1);
              g15_13 = fma(ek15_1, r0_0_3_1, g15_13);
              const double r0_1_0_3 = X * r1_0_0_3;
              g15_14 = fma(ek15_1, r0_1_0_3, g15_14);
              g15_7 = fma(ek15_2, r0_1_0_3, g15_7);
              const double r0_1_1_2 = X * r1_0_1_2;
              g15_15 = fma(ek15_1, r0_1_1_2, g15_15);
              g15_8 = fma(ek15_2, r0_1_1_2, g15_8);
              const double r0_1_2_1 = X * r1_0_2_1;
              g15_16 = fma(ek15_1, r0_1_2_1, g15_16);
              const double r1_1_0_2 = X * r2_0_0_2;
              const double r0_2_0_2 = fma(X, r1_1_0_2, r1_0_0_2);
              g15_17 = fma(ek15_1, r0_2_0_2, g15_17);
              g15_9 = fma(ek15_2, r0_2_0_2, g15_9);
              const double r1_1_1_1 = X * r2_0_1_1;
              const double r0_2_1_1 = fma(X, r1_1_1_1, r1_0_1_1);
              g15_18 = fma(ek15_1, r0_2_1_1, g15_18);
              const double r2_1_0_1 = X * r3_0_0_1;
              const double r1_2_0_1 = fma(X, r2_1_0_1, r2_0_0_1);
              const double r0_3_0_1 = fma(X, r1_2_0_1, 2.0 * r1_1_0_1);
              g15_19 = fma(ek15_1, r0_3_0_1, g15_19);
              const double r4_0_0_1 = Z * b5;
              const double r3_0_0_2 = fma(Z, r4_0_0_1, b4);
              const double r2_0_0_3 = fma(Z, r3_0_0_2, 2.0 * r3_0_0_1);
              const double r1_0_0_4 = fma(Z, r2_0_0_3, 3.0 * r2_0_0_2);
              const double r0_0_0_5 = fma(Z, r1_0_0_4, 4.0 * r1_0_0_3);
              g15_10 = fma(ek15_2, r0_0_0_5, g15_10);
              const double r0_0_1_4 = Y * r1_0_0_4;
              g15_11 = fma(ek15_2, r0_0_1_4, g15_11);
              const double r1_0_1_3 = Y * r2_0_0_3;
              const double r0_0_2_3 = fma(Y, r1_0_1_3, r1_0_0_3);
              g15_12 = fma(ek15_2, r0_0_2_3, g15_12);
              const double r2_0_1_2 = Y * r3_0_0_2;
              const double r1_0_2_2 = fma(Y, r2_0_1_2, r2_0_0_2);
              const double r0_0_3_2 = fma(Y, r1_0_2_2, 2.0 * r1_0_1_2);
              g15_13 = fma(ek15_2, r0_0_3_2, g15_13);
              const double r0_1_0_4 = X * r1_0_0_4;
              g15_14 = fma(ek15_2, r0_1_0_4, g15_14);
              const double r0_1_1_3 = X * r1_0_1_3;
              g15_15 = fma(ek15_2, r0_1_1_3, g15_15);
              const double r0_1_2_2 = X * r1_0_2_2;
              g15_16 = fma(ek15_2, r0_1_2_2, g15_16);
              const double r1_1_0_3 = X * r2_0_0_3;
              const double r0_2_0_3 = fma(X, r1_1_0_3, r1_0_0_3);
              g15_17 = fma(ek15_2, r0_2_0_3, g15_17);
              const double r1_1_1_2 = X * r2_0_1_2;
              const double r0_2_1_2 = fma(X, r1_1_1_2, r1_0_1_2);
              g15_18 = fma(ek15_2, r0_2_1_2, g15_18);
              const double r2_1_0_2 = X * r3_0_0_2;
              const double r1_2_0_2 = fma(X, r2_1_0_2, r2_0_0_2);
              const double r0_3_0_2 = fma(X, r1_2_0_2, 2.0 * r1_1_0_2);
              g15_19 = fma(ek15_2, r0_3_0_2, g15_19);
            }
            { const double eb = bi[5];
              o0_15 = fma(eb, g15_0, o0_15);
            }
            { const double eb = bi[6];
              o0_15 = fma(eb, g15_3, o0_15);
            }
            { const double eb = bi[7];
              o0_15 = fma(eb, g15_9, o0_15);
            }
            { const double eb = bi[8];
              o1_15 = fma(eb, g15_0, o1_15);
            }
            { const double eb = bi[9];
              o1_15 = fma(eb, g15_3, o1_15);
            }
            { const double eb = bi[10];
              o1_15 = fma(eb, g15_9, o1_15);
            }
            { const double eb = bi[11];
              o1_15 = fma(eb, g15_19, o1_15);
            }
            { const double eb = bi[12];
              o2_15 = fma(eb, g15_0, o2_15);
            }
            { const double eb = bi[13];
              o2_15 = fma(eb, g15_2, o2_15);
            }
            { const double eb = bi[14];
              o2_15 = fma(eb, g15_3, o2_15);
            }
            { const double eb = bi[15];
              o2_15 = fma(eb, g15_8, o2_15);
            }
            { const double eb = bi[16];
              o2_15 = fma(eb, g15_9, o2_15);
            }
            { const double eb = bi[17];
              o2_15 = fma(eb, g15_18, o2_15);
            }
            { const double eb = bi[18];
              o3_15 = fma(eb, g15_0, o3_15);
            }
            { const double eb = bi[19];
              o3_15 = fma(eb, g15_1, o3_15);
            }
            { const double eb = bi[20];
              o3_15 = fma(eb, g15_3, o3_15);
            }
            { const double eb = bi[21];
              o3_15 = fma(eb, g15_7, o3_15);
            }
            { const double eb = bi[22];
              o3_15 = fma(eb, g15_9, o3_15);
            }
            { const double eb = bi[23];
              o3_15 = fma(eb, g15_17, o3_15);
            }
            { const double eb = bi[24];
              o4_15 = fma(eb, g15_0, o4_15);
            }
            { const double eb = bi[25];
              o4_15 = fma(eb, g15_2, o4_15);
            }
            { const double eb = bi[26];
              o4_15 = fma(eb, g15_6, o4_15);
            }
            { const double eb = bi[27];
              o5_15 = fma(eb, g15_0, o5_15);
            }
            { const double eb = bi[28];
              o5_15 = fma(eb, g15_2, o5_15);
            }
            { const double eb = bi[29];
              o5_15 = fma(eb, g15_6, o5_15);
            }
            { const double eb = bi[30];
              o5_15 = fma(eb, g15_3, o5_15);
            }
            { const double eb = bi[31];
              o5_15 = fma(eb, g15_8, o5_15);
            }
            { const double eb = bi[32];
              o5_15 = fma(eb, g15_16, o5_15);
            }
            { const double eb = bi[33];
              o6_15 = fma(eb, g15_0, o6_15);
            }
            { const double eb = bi[34];
              o6_15 = fma(eb, g15_2, o6_15);
            }
            { const double eb = bi[35];
              o6_15 = fma(eb, g15_6, o6_15);
            }
            { const double eb = bi[36];
              o6_15 = fma(eb, g15_13, o6_15);
            }
            { const double eb = bi[37];
              o7_15 = fma(eb, g15_0, o7_15);
            }
            { const double eb = bi[38];
              o7_15 = fma(eb, g15_1, o7_15);
            }
            { const double eb = bi[39];
              o7_15 = fma(eb, g15_2, o7_15);
            }
            { const double eb = bi[40];
              o7_15 = fma(eb, g15_5, o7_15);
            }
            { const double eb = bi[41];
              o7_15 = fma(eb, g15_6, o7_15);
            }
            { const double eb = bi[42];
              o7_15 = fma(eb, g15_12, o7_15);
            }
            { const double eb = bi[43];
              o8_15 = fma(eb, g15_0, o8_15);
            }
            { const double eb = bi[44];
              o8_15 = fma(eb, g15_1, o8_15);
            }
            { const double eb = bi[45];
              o8_15 = fma(eb, g15_4, o8_15);
            }
            { const double eb = bi[46];
              o9_15 = fma(eb, g15_0, o9_15);
            }
            { const double eb = bi[47];
              o9_15 = fma(eb, g15_1, o9_15);
            }
            { const double eb = bi[48];
              o9_15 = fma(eb, g15_4, o9_15);
            }
            { const double eb = bi[49];
              o9_15 = fma(eb, g15_3, o9_15);
            }
            { const double eb = bi[50];
              o9_15 = fma(eb, g15_7, o9_15);
            }
            { const double eb = bi[51];
              o9_15 = fma(eb, g15_14, o9_15);
            }
            { const double eb = bi[52];
              o10_15 = fma(eb, g15_0, o10_15);
            }
            { const double eb = bi[53];
              o10_15 = fma(eb, g15_1, o10_15);
            }
            { const double eb = bi[54];
              o10_15 = fma(eb, g15_4, o10_15);
            }
            { const double eb = bi[55];
              o10_15 = fma(eb, g15_2, o10_15);
            }
            { const double eb = bi[56];
              o10_15 = fma(eb, g15_5, o10_15);
            }
            { const double eb = bi[57];
              o10_15 = fma(eb, g15_11, o10_15);
            }
            { const double eb = bi[58];
              o11_15 = fma(eb, g15_0, o11_15);
            }
            { const double eb = bi[59];
              o11_15 = fma(eb, g15_1, o11_15);
            }
            { const double eb = bi[60];
              o11_15 = fma(eb, g15_4, o11_15);
            }
            { const double eb = bi[61];
              o11_15 = fma(eb, g15_10, o11_15);
            }
            { const double eb = bi[62];
              o12_15 = fma(eb, g15_0, o12_15);
            }
            { const double eb = bi[63];
              o12_15 = fma(eb, g15_2, o12_15);
            }
            { const double eb = bi[64];
              o12_15 = fma(eb, g15_3, o12_15);
            }
            { const double eb = bi[65];
              o12_15 = fma(eb, g15_8, o12_15);
            }
            { const double eb = bi[66];
              o13_15 = fma(eb, g15_0, o13_15);
            }
            { const double eb = bi[67];
              o13_15 = fma(eb, g15_2, o13_15);
            }
            { const double eb = bi[68];
              o13_15 = fma(eb, g15_3, o13_15);
            }
            { const double eb = bi[69];
              o13_15 = fma(eb, g15_8, o13_15);
            }
            { const double eb = bi[70];
              o13_15 = fma(eb, g15_9, o13_15);
            }
            { const double eb = bi[71];
              o13_15 = fma(eb, g15_18, o13_15);
            }
            { const double eb = bi[72];
              o14_15 = fma(eb, g15_0, o14_15);
            }
            { const double eb = bi[73];
              o14_15 = fma(eb, g15_2, o14_15);
            }
            { const double eb = bi[74];
              o14_15 = fma(eb, g15_6, o14_15);
            }
            { const double eb = bi[75];
              o14_15 = fma(eb, g15_3, o14_15);
            }
            { const double eb = bi[76];
              o14_15 = fma(eb, g15_8, o14_15);
            }
            { const double eb = bi[77];
              o14_15 = fma(eb, g15_16, o14_15);
            }
            { const double eb = bi[78];
              o15_15 = fma(eb, g15_0, o15_15);
            }
            { const double eb = bi[79];
              o15_15 = fma(eb, g15_1, o15_15);
            }
            { const double eb = bi[80];
              o15_15 = fma(eb, g15_2, o15_15);
            }
            { const double eb = bi[81];
              o15_15 = fma(eb, g15_5, o15_15);
            }
            { const double eb = bi[82];
              o15_15 = fma(eb, g15_3, o15_15);
            }
            { const double eb = bi[83];
              o15_15 = fma(eb, g15_7, o15_15);
            }
            { const double eb = bi[84];
              o15_15 = fma(eb, g15_8, o15_15);
            }
            { const double eb = bi[85];
              o15_15 = fma(eb, g15_15, o15_15);
            }
            { const double eb = bi[86];
              o16_15 = fma(eb, g15_0, o16_15);
            }
            { const double eb = bi[87];
              o16_15 = fma(eb, g15_1, o16_15);
            }
            { const double eb = bi[88];
              o16_15 = fma(eb, g15_3, o16_15);
            }
            { const double eb = bi[89];
              o16_15 = fma(eb, g15_7, o16_15);
            }
            { const double eb = bi[90];
              o17_15 = fma(eb, g15_0, o17_15);
            }
            { const double eb = bi[91];
              o17_15 = fma(eb, g15_1, o17_15);
            }
            { const double eb = bi[92];
              o17_15 = fma(eb, g15_3, o17_15);
            }
            { const double eb = bi[93];
              o17_15 = fma(eb, g15_7, o17_15);
            }
            { const double eb = bi[94];
              o17_15 = fma(eb, g15_9, o17_15);
            }
            { const double eb = bi[95];
              o17_15 = fma(eb, g15_17, o17_15);
            }
            { const double eb = bi[96];
              o18_15 = fma(eb, g15_0, o18_15);
            }
            { const double eb = bi[97];
              o18_15 = fma(eb, g15_1, o18_15);
            }
            { const double eb = bi[98];
              o18_15 = fma(eb, g15_2, o18_15);
            }
            { const double eb = bi[99];
              o18_15 = fma(eb, g15_5, o18_15);
            }
            { const double eb = bi[100];
              o18_15 = fma(eb, g15_3, o18_15);
            }
            { const double eb = bi[101];
              o18_15 = fma(eb, g15_7, o18_15);
            }
            { const double eb = bi[102];
              o18_15 = fma(eb, g15_8, o18_15);
            }
            { const double eb = bi[103];
              o18_15 = fma(eb, g15_15, o18_15);
            }
            { const double eb = bi[104];
              o19_15 = fma(eb, g15_0, o19_15);
            }
            { const double eb = bi[105];
              o19_15 = fma(eb, g15_1, o19_15);
            }
            { const double eb = bi[106];
              o19_15 = fma(eb, g15_4, o19_15);
            }
            { const double eb = bi[107];
              o19_15 = fma(eb, g15_3, o19_15);
            }
            { const double eb = bi[108];
              o19_15 = fma(eb, g15_7, o19_15);
            }
            { const double eb = bi[109];
              o19_15 = fma(eb, g15_14, o19_15);
            }
            { const double eb = bi[110];
              o20_15 = fma(eb, g15_0, o20_15);
            }
            { const double eb = bi[111];
              o20_15 = fma(eb, g15_1, o20_15);
            }
            { const double eb = bi[112];
              o20_15 = fma(eb, g15_2, o20_15);
            }
            { const double eb = bi[113];
              o20_15 = fma(eb, g15_5, o20_15);
            }
            { const double eb = bi[114];
              o21_15 = fma(eb, g15_0, o21_15);
            }
            { const double eb = bi[115];
              o21_15 = fma(eb, g15_1, o21_15);
            }
            { const double eb = bi[116];
              o21_15 = fma(eb, g15_2, o21_15);
            }
            { const double eb = bi[117];
              o21_15 = fma(eb, g15_5, o21_15);
            }
            { const double eb = bi[118];
              o21_15 = fma(eb, g15_3, o21_15);
            }
            { const double eb = bi[119];
              o21_15 = fma(eb, g15_7, o21_15);
            }
            { const double eb = bi[120];
              o21_15 = fma(eb, g15_8, o21_15);
            }
            { const double eb = bi[121];
              o21_15 = fma(eb, g15_15, o21_15);
            }
            { const double eb = bi[122];
              o22_15 = fma(eb, g15_0, o22_15);
            }
            { const double eb = bi[123];
              o22_15 = fma(eb, g15_1, o22_15);
            }
            { const double eb = bi[124];
              o22_15 = fma(eb, g15_2, o22_15);
            }
            { const double eb = bi[125];
              o22_15 = fma(eb, g15_5, o22_15);
            }
            { const double eb = bi[126];
              o22_15 = fma(eb, g15_6, o22_15);
            }
            { const double eb = bi[127];
              o22_15 = fma(eb, g15_12, o22_15);
            }
            { const double eb = bi[128];
              o23_15 = fma(eb, g15_0, o23_15);
            }
            { const double eb = bi[129];
              o23_15 = fma(eb, g15_1, o23_15);
            }
            { const double eb = bi[130];
              o23_15 = fma(eb, g15_4, o23_15);
            }
            { const double eb = bi[131];
              o23_15 = fma(eb, g15_2, o23_15);
            }
            { const double eb = bi[132];
              o23_15 = fma(eb, g15_5, o23_15);
            }
            { const double eb = bi[133];
              o23_15 = fma(eb, g15_11, o23_15);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_15 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 3);
            o1_15 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 3);
            o2_15 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 3);
            o3_15 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 3);
            o4_15 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 3);
            o5_15 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 3);
            o6_15 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 3);
            o7_15 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 3);
            o8_15 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 3);
            o9_15 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 3);
            o10_15 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 3);
            o11_15 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 3);
            o12_15 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 3);
            o13_15 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 3);
            o14_15 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 3);
            o15_15 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 3);
            o16_15 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 3);
            o17_15 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 3);
            o18_15 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 3);
            o19_15 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 3);
            o20_15 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 3);
            o21_15 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 3);
            o22_15 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 3);
            o23_15 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 3);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_15 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o1_15 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 1, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o2_15 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 2, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o3_15 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 3, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o4_15 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o5_15 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 1, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o6_15 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 2, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o7_15 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 3, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o8_15 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o9_15 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 1, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o10_15 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 2, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o11_15 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 3, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o12_15 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o13_15 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 1, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o14_15 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 2, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o15_15 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 3, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o16_15 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o17_15 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 1, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o18_15 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 2, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o19_15 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 3, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o20_15 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o21_15 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 1, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o22_15 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 2, fI + 3, fJ + 3)));
            e = fmax(e, fabs(o23_15 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 3, fI + 3, fJ + 3)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Aad0_3 = PA[(fP + 0) * N + fJ + 3];
            const double Aad1_3 = PA[(fP + 1) * N + fJ + 3];
            const double Aad2_3 = PA[(fP + 2) * N + fJ + 3];
            const double Aad3_3 = PA[(fP + 3) * N + fJ + 3];
            const double Aad4_3 = PA[(fP + 4) * N + fJ + 3];
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
            const double Bbd0_3 = PB[(fQ + 0) * N + fJ + 3];
            const double Bbd1_3 = PB[(fQ + 1) * N + fJ + 3];
            const double Bbd2_3 = PB[(fQ + 2) * N + fJ + 3];
            const double Bbd3_3 = PB[(fQ + 3) * N + fJ + 3];
            const double Bad0_3 = PB[(fP + 0) * N + fJ + 3];
            const double Bad1_3 = PB[(fP + 1) * N + fJ + 3];
            const double Bad2_3 = PB[(fP + 2) * N + fJ + 3];
            const double Bad3_3 = PB[(fP + 3) * N + fJ + 3];
            const double Bad4_3 = PB[(fP + 4) * N + fJ + 3];
            const double Bad5_3 = PB[(fP + 5) * N + fJ + 3];
            const double Bbc0_3 = PB[(fQ + 0) * N + fI + 3];
            const double Bbc1_3 = PB[(fQ + 1) * N + fI + 3];
            const double Bbc2_3 = PB[(fQ + 2) * N + fI + 3];
            const double Bbc3_3 = PB[(fQ + 3) * N + fI + 3];
            const double Bac0_3 = PB[(fP + 0) * N + fI + 3];
            const double Bac1_3 = PB[(fP + 1) * N + fI + 3];
            const double Bac2_3 = PB[(fP + 2) * N + fI + 3];
            const double Bac3_3 = PB[(fP + 3) * N + fI + 3];
            const double Bac4_3 = PB[(fP + 4) * N + fI + 3];
            const double Bac5_3 = PB[(fP + 5) * N + fI + 3];
            jab0 += o0_15 * ptk15;
            jab1 += o1_15 * ptk15;
            jab2 += o2_15 * ptk15;
            jab3 += o3_15 * ptk15;
            jab4 += o4_15 * ptk15;
            jab5 += o5_15 * ptk15;
            jab6 += o6_15 * ptk15;
            jab7 += o7_15 * ptk15;
            jab8 += o8_15 * ptk15;
            jab9 += o9_15 * ptk15;
            jab10 += o10_15 * ptk15;
            jab11 += o11_15 * ptk15;
            jab12 += o12_15 * ptk15;
            jab13 += o13_15 * ptk15;
            jab14 += o14_15 * ptk15;
            jab15 += o15_15 * ptk15;
            jab16 += o16_15 * ptk15;
            jab17 += o17_15 * ptk15;
            jab18 += o18_15 * ptk15;
            jab19 += o19_15 * ptk15;
            jab20 += o20_15 * ptk15;
            jab21 += o21_15 * ptk15;
            jab22 += o22_15 * ptk15;
            jab23 += o23_15 * ptk15;
            atomicAdd(Jacc + (fI + 3) * N + fJ + 3, 2.0 * deg * (o0_15 * ptb0 + o1_15 * ptb1 + o2_15 * ptb2 + o3_15 * ptb3 + o4_15 * ptb4 + o5_15 * ptb5 + o6_15 * ptb6 + o7_15 * ptb7 + o8_15 * ptb8 + o9_15 * ptb9 + o10_15 * ptb10 + o11_15 * ptb11 + o12_15 * ptb12 + o13_15 * ptb13 + o14_15 * ptb14 + o15_15 * ptb15 + o16_15 * ptb16 + o17_15 * ptb17 + o18_15 * ptb18 + o19_15 * ptb19 + o20_15 * ptb20 + o21_15 * ptb21 + o22_15 * ptb22 + o23_15 * ptb23));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_15 * Abd0_3 + o1_15 * Abd1_3 + o2_15 * Abd2_3 + o3_15 * Abd3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_15 * Aad0_3 + o4_15 * Aad1_3 + o8_15 * Aad2_3 + o12_15 * Aad3_3 + o16_15 * Aad4_3 + o20_15 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_15 * Abc0_3 + o1_15 * Abc1_3 + o2_15 * Abc2_3 + o3_15 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_15 * Aac0_3 + o4_15 * Aac1_3 + o8_15 * Aac2_3 + o12_15 * Aac3_3 + o16_15 * Aac4_3 + o20_15 * Aac5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_15 * Aad0_3 + o5_15 * Aad1_3 + o9_15 * Aad2_3 + o13_15 * Aad3_3 + o17_15 * Aad4_3 + o21_15 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_15 * Aac0_3 + o5_15 * Aac1_3 + o9_15 * Aac2_3 + o13_15 * Aac3_3 + o17_15 * Aac4_3 + o21_15 * Aac5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_15 * Aad0_3 + o6_15 * Aad1_3 + o10_15 * Aad2_3 + o14_15 * Aad3_3 + o18_15 * Aad4_3 + o22_15 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_15 * Aac0_3 + o6_15 * Aac1_3 + o10_15 * Aac2_3 + o14_15 * Aac3_3 + o18_15 * Aac4_3 + o22_15 * Aac5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_15 * Aad0_3 + o7_15 * Aad1_3 + o11_15 * Aad2_3 + o15_15 * Aad3_3 + o19_15 * Aad4_3 + o23_15 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_15 * Aac0_3 + o7_15 * Aac1_3 + o11_15 * Aac2_3 + o15_15 * Aac3_3 + o19_15 * Aac4_3 + o23_15 * Aac5_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_15 * Abd0_3 + o5_15 * Abd1_3 + o6_15 * Abd2_3 + o7_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o4_15 * Abc0_3 + o5_15 * Abc1_3 + o6_15 * Abc2_3 + o7_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_15 * Abd0_3 + o9_15 * Abd1_3 + o10_15 * Abd2_3 + o11_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o8_15 * Abc0_3 + o9_15 * Abc1_3 + o10_15 * Abc2_3 + o11_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_15 * Abd0_3 + o13_15 * Abd1_3 + o14_15 * Abd2_3 + o15_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o12_15 * Abc0_3 + o13_15 * Abc1_3 + o14_15 * Abc2_3 + o15_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o16_15 * Abd0_3 + o17_15 * Abd1_3 + o18_15 * Abd2_3 + o19_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o16_15 * Abc0_3 + o17_15 * Abc1_3 + o18_15 * Abc2_3 + o19_15 * Abc3_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o20_15 * Abd0_3 + o21_15 * Abd1_3 + o22_15 * Abd2_3 + o23_15 * Abd3_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o20_15 * Abc0_3 + o21_15 * Abc1_3 + o22_15 * Abc2_3 + o23_15 * Abc3_3));
            atomicAdd(KBacc + (fP + 0) * N + fI + 3, deg * (o0_15 * Bbd0_3 + o1_15 * Bbd1_3 + o2_15 * Bbd2_3 + o3_15 * Bbd3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 3, deg * (o0_15 * Bad0_3 + o4_15 * Bad1_3 + o8_15 * Bad2_3 + o12_15 * Bad3_3 + o16_15 * Bad4_3 + o20_15 * Bad5_3));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 3, deg * (o0_15 * Bbc0_3 + o1_15 * Bbc1_3 + o2_15 * Bbc2_3 + o3_15 * Bbc3_3));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 3, deg * (o0_15 * Bac0_3 + o4_15 * Bac1_3 + o8_15 * Bac2_3 + o12_15 * Bac3_3 + o16_15 * Bac4_3 + o20_15 * Bac5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fI + 3, deg * (o1_15 * Bad0_3 + o5_15 * Bad1_3 + o9_15 * Bad2_3 + o13_15 * Bad3_3 + o17_15 * Bad4_3 + o21_15 * Bad5_3));
            atomicAdd(KBacc + (fQ + 1) * N + fJ + 3, deg * (o1_15 * Bac0_3 + o5_15 * Bac1_3 + o9_15 * Bac2_3 + o13_15 * Bac3_3 + o17_15 * Bac4_3 + o21_15 * Bac5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fI + 3, deg * (o2_15 * Bad0_3 + o6_15 * Bad1_3 + o10_15 * Bad2_3 + o14_15 * Bad3_3 + o18_15 * Bad4_3 + o22_15 * Bad5_3));
            atomicAdd(KBacc + (fQ + 2) * N + fJ + 3, deg * (o2_15 * Bac0_3 + o6_15 * Bac1_3 + o10_15 * Bac2_3 + o14_15 * Bac3_3 + o18_15 * Bac4_3 + o22_15 * Bac5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fI + 3, deg * (o3_15 * Bad0_3 + o7_15 * Bad1_3 + o11_15 * Bad2_3 + o15_15 * Bad3_3 + o19_15 * Bad4_3 + o23_15 * Bad5_3));
            atomicAdd(KBacc + (fQ + 3) * N + fJ + 3, deg * (o3_15 * Bac0_3 + o7_15 * Bac1_3 + o11_15 * Bac2_3 + o15_15 * Bac3_3 + o19_15 * Bac4_3 + o23_15 * Bac5_3));
            atomicAdd(KBacc + (fP + 1) * N + fI + 3, deg * (o4_15 * Bbd0_3 + o5_15 * Bbd1_3 + o6_15 * Bbd2_3 + o7_15 * Bbd3_3));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 3, deg * (o4_15 * Bbc0_3 + o5_15 * Bbc1_3 + o6_15 * Bbc2_3 + o7_15 * Bbc3_3));
            atomicAdd(KBacc + (fP + 2) * N + fI + 3, deg * (o8_15 * Bbd0_3 + o9_15 * Bbd1_3 + o10_15 * Bbd2_3 + o11_15 * Bbd3_3));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 3, deg * (o8_15 * Bbc0_3 + o9_15 * Bbc1_3 + o10_15 * Bbc2_3 + o11_15 * Bbc3_3));
            atomicAdd(KBacc + (fP + 3) * N + fI + 3, deg * (o12_15 * Bbd0_3 + o13_15 * Bbd1_3 + o14_15 * Bbd2_3 + o15_15 * Bbd3_3));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 3, deg * (o12_15 * Bbc0_3 + o13_15 * Bbc1_3 + o14_15 * Bbc2_3 + o15_15 * Bbc3_3));
            atomicAdd(KBacc + (fP + 4) * N + fI + 3, deg * (o16_15 * Bbd0_3 + o17_15 * Bbd1_3 + o18_15 * Bbd2_3 + o19_15 * Bbd3_3));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 3, deg * (o16_15 * Bbc0_3 + o17_15 * Bbc1_3 + o18_15 * Bbc2_3 + o19_15 * Bbc3_3));
            atomicAdd(KBacc + (fP + 5) * N + fI + 3, deg * (o20_15 * Bbd0_3 + o21_15 * Bbd1_3 + o22_15 * Bbd2_3 + o23_15 * Bbd3_3));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 3, deg * (o20_15 * Bbc0_3 + o21_15 * Bbc1_3 + o22_15 * Bbc2_3 + o23_15 * Bbc3_3));
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
