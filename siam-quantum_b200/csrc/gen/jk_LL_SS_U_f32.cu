// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_LL_SS_U_f32(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      extern __shared__ float sbra_f32[];
      float* __restrict__ sbra = sbra_f32;
      const sqb::WorkItem it = items[qi_];
      const sqb::PairRec bp = a.bra_pairs[it.bra];
      const sqb::MolRec mr = a.mols[it.mol];        // the molecule of this work item
      const long long acc0 = mr.moff + (qi_ & a.copy_mask) * a.copy_stride;   // this item's copy
      double* __restrict__ Jacc = a.Jacc + acc0;
      double* __restrict__ KAacc = a.KAacc + acc0;
      double* __restrict__ KBacc = a.KBacc + acc0;
      const int N = mr.nbf;
      for (int x = threadIdx.x; x < bp.nprim * 51; x += blockDim.x) sbra[x] = a.bra_prims_f[bp.poff + (long long)x * bp.kstride];
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
      unsigned long long nprimq = 0, nflush = 0;
      if (ok) {
        const float* __restrict__ kprim = a.ket_prims_f + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
        const double* __restrict__ PB = a.PB + mr.moff;
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // ket functions [0]
          float o0_0 = 0;
          float o1_0 = 0;
          float o2_0 = 0;
          float o3_0 = 0;
          float o4_0 = 0;
          float o5_0 = 0;
          float o6_0 = 0;
          float o7_0 = 0;
          float o8_0 = 0;
          float o9_0 = 0;
          float o10_0 = 0;
          float o11_0 = 0;
          float o12_0 = 0;
          float o13_0 = 0;
          float o14_0 = 0;
          float o15_0 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 51;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g0_0 = 0;
            float g0_1 = 0;
            float g0_2 = 0;
            float g0_3 = 0;
            float g0_4 = 0;
            float g0_5 = 0;
            float g0_6 = 0;
            float g0_7 = 0;
            float g0_8 = 0;
            float g0_9 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 6 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              ++nprimq;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[3];
              sqb::boysf<2>(T, a.boys_tab_f, F);
              const float s0 = TWO_PI_2_5F * rs;
              const float m2a = -2.0f * alpha;
              float w = s0;
              const float b0 = w * F[0];
              w *= m2a;
              const float b1 = w * F[1];
              w *= m2a;
              const float b2 = w * F[2];
              const float ek0_0 = kj[5 * kS];
              g0_0 = fmaf(ek0_0, b0, g0_0);
              const float r0_0_0_1 = Z * b1;
              g0_1 = fmaf(ek0_0, r0_0_0_1, g0_1);
              const float r0_0_1_0 = Y * b1;
              g0_2 = fmaf(ek0_0, r0_0_1_0, g0_2);
              const float r0_1_0_0 = X * b1;
              g0_3 = fmaf(ek0_0, r0_1_0_0, g0_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g0_4 = fmaf(ek0_0, r0_0_0_2, g0_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fmaf(ek0_0, r0_0_1_1, g0_5);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g0_6 = fmaf(ek0_0, r0_0_2_0, g0_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fmaf(ek0_0, r0_1_0_1, g0_7);
              const float r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fmaf(ek0_0, r0_1_1_0, g0_8);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g0_9 = fmaf(ek0_0, r0_2_0_0, g0_9);
            }
            { const float eb = bi[5];
              o0_0 = fmaf(eb, g0_0, o0_0);
            }
            { const float eb = bi[6];
              o1_0 = fmaf(eb, g0_0, o1_0);
            }
            { const float eb = bi[7];
              o1_0 = fmaf(eb, g0_3, o1_0);
            }
            { const float eb = bi[8];
              o2_0 = fmaf(eb, g0_0, o2_0);
            }
            { const float eb = bi[9];
              o2_0 = fmaf(eb, g0_2, o2_0);
            }
            { const float eb = bi[10];
              o3_0 = fmaf(eb, g0_0, o3_0);
            }
            { const float eb = bi[11];
              o3_0 = fmaf(eb, g0_1, o3_0);
            }
            { const float eb = bi[12];
              o4_0 = fmaf(eb, g0_0, o4_0);
            }
            { const float eb = bi[13];
              o4_0 = fmaf(eb, g0_3, o4_0);
            }
            { const float eb = bi[14];
              o5_0 = fmaf(eb, g0_0, o5_0);
            }
            { const float eb = bi[15];
              o5_0 = fmaf(eb, g0_3, o5_0);
            }
            { const float eb = bi[16];
              o5_0 = fmaf(eb, g0_9, o5_0);
            }
            { const float eb = bi[17];
              o6_0 = fmaf(eb, g0_0, o6_0);
            }
            { const float eb = bi[18];
              o6_0 = fmaf(eb, g0_2, o6_0);
            }
            { const float eb = bi[19];
              o6_0 = fmaf(eb, g0_3, o6_0);
            }
            { const float eb = bi[20];
              o6_0 = fmaf(eb, g0_8, o6_0);
            }
            { const float eb = bi[21];
              o7_0 = fmaf(eb, g0_0, o7_0);
            }
            { const float eb = bi[22];
              o7_0 = fmaf(eb, g0_1, o7_0);
            }
            { const float eb = bi[23];
              o7_0 = fmaf(eb, g0_3, o7_0);
            }
            { const float eb = bi[24];
              o7_0 = fmaf(eb, g0_7, o7_0);
            }
            { const float eb = bi[25];
              o8_0 = fmaf(eb, g0_0, o8_0);
            }
            { const float eb = bi[26];
              o8_0 = fmaf(eb, g0_2, o8_0);
            }
            { const float eb = bi[27];
              o9_0 = fmaf(eb, g0_0, o9_0);
            }
            { const float eb = bi[28];
              o9_0 = fmaf(eb, g0_2, o9_0);
            }
            { const float eb = bi[29];
              o9_0 = fmaf(eb, g0_3, o9_0);
            }
            { const float eb = bi[30];
              o9_0 = fmaf(eb, g0_8, o9_0);
            }
            { const float eb = bi[31];
              o10_0 = fmaf(eb, g0_0, o10_0);
            }
            { const float eb = bi[32];
              o10_0 = fmaf(eb, g0_2, o10_0);
            }
            { const float eb = bi[33];
              o10_0 = fmaf(eb, g0_6, o10_0);
            }
            { const float eb = bi[34];
              o11_0 = fmaf(eb, g0_0, o11_0);
            }
            { const float eb = bi[35];
              o11_0 = fmaf(eb, g0_1, o11_0);
            }
            { const float eb = bi[36];
              o11_0 = fmaf(eb, g0_2, o11_0);
            }
            { const float eb = bi[37];
              o11_0 = fmaf(eb, g0_5, o11_0);
            }
            { const float eb = bi[38];
              o12_0 = fmaf(eb, g0_0, o12_0);
            }
            { const float eb = bi[39];
              o12_0 = fmaf(eb, g0_1, o12_0);
            }
            { const float eb = bi[40];
              o13_0 = fmaf(eb, g0_0, o13_0);
            }
            { const float eb = bi[41];
              o13_0 = fmaf(eb, g0_1, o13_0);
            }
            { const float eb = bi[42];
              o13_0 = fmaf(eb, g0_3, o13_0);
            }
            { const float eb = bi[43];
              o13_0 = fmaf(eb, g0_7, o13_0);
            }
            { const float eb = bi[44];
              o14_0 = fmaf(eb, g0_0, o14_0);
            }
            { const float eb = bi[45];
              o14_0 = fmaf(eb, g0_1, o14_0);
            }
            { const float eb = bi[46];
              o14_0 = fmaf(eb, g0_2, o14_0);
            }
            { const float eb = bi[47];
              o14_0 = fmaf(eb, g0_5, o14_0);
            }
            { const float eb = bi[48];
              o15_0 = fmaf(eb, g0_0, o15_0);
            }
            { const float eb = bi[49];
              o15_0 = fmaf(eb, g0_1, o15_0);
            }
            { const float eb = bi[50];
              o15_0 = fmaf(eb, g0_4, o15_0);
            }
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
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Abd1_0 = PA[(fQ + 1) * N + fJ + 0];
            const double Abd2_0 = PA[(fQ + 2) * N + fJ + 0];
            const double Abd3_0 = PA[(fQ + 3) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bbd1_0 = PB[(fQ + 1) * N + fJ + 0];
            const double Bbd2_0 = PB[(fQ + 2) * N + fJ + 0];
            const double Bbd3_0 = PB[(fQ + 3) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc1_0 = PB[(fQ + 1) * N + fI + 0];
            const double Bbc2_0 = PB[(fQ + 2) * N + fI + 0];
            const double Bbc3_0 = PB[(fQ + 3) * N + fI + 0];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            const double Bac1_0 = PB[(fP + 1) * N + fI + 0];
            const double Bac2_0 = PB[(fP + 2) * N + fI + 0];
            const double Bac3_0 = PB[(fP + 3) * N + fI + 0];
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
            sqb::group_add(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0 + o3_0 * Abd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o4_0 * Aad1_0 + o8_0 * Aad2_0 + o12_0 * Aad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o1_0 * Abc1_0 + o2_0 * Abc2_0 + o3_0 * Abc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o4_0 * Aac1_0 + o8_0 * Aac2_0 + o12_0 * Aac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o5_0 * Aad1_0 + o9_0 * Aad2_0 + o13_0 * Aad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o5_0 * Aac1_0 + o9_0 * Aac2_0 + o13_0 * Aac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o6_0 * Aad1_0 + o10_0 * Aad2_0 + o14_0 * Aad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o6_0 * Aac1_0 + o10_0 * Aac2_0 + o14_0 * Aac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Aad0_0 + o7_0 * Aad1_0 + o11_0 * Aad2_0 + o15_0 * Aad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Aac0_0 + o7_0 * Aac1_0 + o11_0 * Aac2_0 + o15_0 * Aac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Abd0_0 + o5_0 * Abd1_0 + o6_0 * Abd2_0 + o7_0 * Abd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o5_0 * Abc1_0 + o6_0 * Abc2_0 + o7_0 * Abc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Abd0_0 + o9_0 * Abd1_0 + o10_0 * Abd2_0 + o11_0 * Abd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Abc0_0 + o9_0 * Abc1_0 + o10_0 * Abc2_0 + o11_0 * Abc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0 + o15_0 * Abd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o13_0 * Abc1_0 + o14_0 * Abc2_0 + o15_0 * Abc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Bbd0_0 + o1_0 * Bbd1_0 + o2_0 * Bbd2_0 + o3_0 * Bbd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Bad0_0 + o4_0 * Bad1_0 + o8_0 * Bad2_0 + o12_0 * Bad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Bbc0_0 + o1_0 * Bbc1_0 + o2_0 * Bbc2_0 + o3_0 * Bbc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Bac0_0 + o4_0 * Bac1_0 + o8_0 * Bac2_0 + o12_0 * Bac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Bad0_0 + o5_0 * Bad1_0 + o9_0 * Bad2_0 + o13_0 * Bad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Bac0_0 + o5_0 * Bac1_0 + o9_0 * Bac2_0 + o13_0 * Bac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Bad0_0 + o6_0 * Bad1_0 + o10_0 * Bad2_0 + o14_0 * Bad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Bac0_0 + o6_0 * Bac1_0 + o10_0 * Bac2_0 + o14_0 * Bac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Bad0_0 + o7_0 * Bad1_0 + o11_0 * Bad2_0 + o15_0 * Bad3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Bac0_0 + o7_0 * Bac1_0 + o11_0 * Bac2_0 + o15_0 * Bac3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Bbd0_0 + o5_0 * Bbd1_0 + o6_0 * Bbd2_0 + o7_0 * Bbd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Bbc0_0 + o5_0 * Bbc1_0 + o6_0 * Bbc2_0 + o7_0 * Bbc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Bbd0_0 + o9_0 * Bbd1_0 + o10_0 * Bbd2_0 + o11_0 * Bbd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Bbc0_0 + o9_0 * Bbc1_0 + o10_0 * Bbc2_0 + o11_0 * Bbc3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Bbd0_0 + o13_0 * Bbd1_0 + o14_0 * Bbd2_0 + o15_0 * Bbd3_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Bbc0_0 + o13_0 * Bbc1_0 + o14_0 * Bbc2_0 + o15_0 * Bbc3_0), isplit, gmask, grp == 0);
          }
        } break;
        }
      }
      {
        const double s2 = 2.0 * deg;
        double v[16] = {s2 * jab0, s2 * jab1, s2 * jab2, s2 * jab3, s2 * jab4, s2 * jab5, s2 * jab6, s2 * jab7, s2 * jab8, s2 * jab9, s2 * jab10, s2 * jab11, s2 * jab12, s2 * jab13, s2 * jab14, s2 * jab15};
        const double s = sqb::warp_sum_scatter<16>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 16 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 4) * N + bp.fQ + ab % 4, s);
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
