// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_LL_DS_R_f32(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // ket functions [0, 1, 2, 3]
          float o0_0 = 0;
          float o0_1 = 0;
          float o0_2 = 0;
          float o0_3 = 0;
          float o1_0 = 0;
          float o1_1 = 0;
          float o1_2 = 0;
          float o1_3 = 0;
          float o2_0 = 0;
          float o2_1 = 0;
          float o2_2 = 0;
          float o2_3 = 0;
          float o3_0 = 0;
          float o3_1 = 0;
          float o3_2 = 0;
          float o3_3 = 0;
          float o4_0 = 0;
          float o4_1 = 0;
          float o4_2 = 0;
          float o4_3 = 0;
          float o5_0 = 0;
          float o5_1 = 0;
          float o5_2 = 0;
          float o5_3 = 0;
          float o6_0 = 0;
          float o6_1 = 0;
          float o6_2 = 0;
          float o6_3 = 0;
          float o7_0 = 0;
          float o7_1 = 0;
          float o7_2 = 0;
          float o7_3 = 0;
          float o8_0 = 0;
          float o8_1 = 0;
          float o8_2 = 0;
          float o8_3 = 0;
          float o9_0 = 0;
          float o9_1 = 0;
          float o9_2 = 0;
          float o9_3 = 0;
          float o10_0 = 0;
          float o10_1 = 0;
          float o10_2 = 0;
          float o10_3 = 0;
          float o11_0 = 0;
          float o11_1 = 0;
          float o11_2 = 0;
          float o11_3 = 0;
          float o12_0 = 0;
          float o12_1 = 0;
          float o12_2 = 0;
          float o12_3 = 0;
          float o13_0 = 0;
          float o13_1 = 0;
          float o13_2 = 0;
          float o13_3 = 0;
          float o14_0 = 0;
          float o14_1 = 0;
          float o14_2 = 0;
          float o14_3 = 0;
          float o15_0 = 0;
          float o15_1 = 0;
          float o15_2 = 0;
          float o15_3 = 0;
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
            float g1_0 = 0;
            float g1_1 = 0;
            float g1_2 = 0;
            float g1_3 = 0;
            float g1_4 = 0;
            float g1_5 = 0;
            float g1_6 = 0;
            float g1_7 = 0;
            float g1_8 = 0;
            float g1_9 = 0;
            float g2_0 = 0;
            float g2_1 = 0;
            float g2_2 = 0;
            float g2_3 = 0;
            float g2_4 = 0;
            float g2_5 = 0;
            float g2_6 = 0;
            float g2_7 = 0;
            float g2_8 = 0;
            float g2_9 = 0;
            float g3_0 = 0;
            float g3_1 = 0;
            float g3_2 = 0;
            float g3_3 = 0;
            float g3_4 = 0;
            float g3_5 = 0;
            float g3_6 = 0;
            float g3_7 = 0;
            float g3_8 = 0;
            float g3_9 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 26 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              ++nprimq;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[5];
              sqb::boysf<4>(T, a.boys_tab_f, F);
              const float s0 = TWO_PI_2_5F * rs;
              const float m2a = -2.0f * alpha;
              float w = s0;
              const float b0 = w * F[0];
              w *= m2a;
              const float b1 = w * F[1];
              w *= m2a;
              const float b2 = w * F[2];
              w *= m2a;
              const float b3 = w * F[3];
              w *= m2a;
              const float b4 = w * F[4];
              const float ek0_0 = kj[5 * kS];
              const float ek0_1 = -kj[6 * kS];
              const float ek0_2 = kj[7 * kS];
              const float ek1_0 = kj[8 * kS];
              const float ek1_1 = -kj[9 * kS];
              const float ek1_2 = kj[10 * kS];
              const float ek2_0 = kj[11 * kS];
              const float ek2_1 = -kj[12 * kS];
              const float ek2_2 = kj[13 * kS];
              const float ek3_0 = kj[14 * kS];
              const float ek3_1 = -kj[15 * kS];
              const float ek3_2 = -kj[16 * kS];
              const float ek3_3 = kj[17 * kS];
              g0_0 = fmaf(ek0_0, b0, g0_0);
              g1_0 = fmaf(ek1_0, b0, g1_0);
              g2_0 = fmaf(ek2_0, b0, g2_0);
              g3_0 = fmaf(ek3_0, b0, g3_0);
              const float r0_0_0_1 = Z * b1;
              g0_1 = fmaf(ek0_0, r0_0_0_1, g0_1);
              g1_1 = fmaf(ek1_0, r0_0_0_1, g1_1);
              g2_1 = fmaf(ek2_0, r0_0_0_1, g2_1);
              g2_0 = fmaf(ek2_1, r0_0_0_1, g2_0);
              g3_1 = fmaf(ek3_0, r0_0_0_1, g3_1);
              const float r0_0_1_0 = Y * b1;
              g0_2 = fmaf(ek0_0, r0_0_1_0, g0_2);
              g1_2 = fmaf(ek1_0, r0_0_1_0, g1_2);
              g1_0 = fmaf(ek1_1, r0_0_1_0, g1_0);
              g2_2 = fmaf(ek2_0, r0_0_1_0, g2_2);
              g3_2 = fmaf(ek3_0, r0_0_1_0, g3_2);
              g3_0 = fmaf(ek3_1, r0_0_1_0, g3_0);
              const float r0_1_0_0 = X * b1;
              g0_3 = fmaf(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fmaf(ek0_1, r0_1_0_0, g0_0);
              g1_3 = fmaf(ek1_0, r0_1_0_0, g1_3);
              g2_3 = fmaf(ek2_0, r0_1_0_0, g2_3);
              g3_3 = fmaf(ek3_0, r0_1_0_0, g3_3);
              g3_0 = fmaf(ek3_2, r0_1_0_0, g3_0);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g0_4 = fmaf(ek0_0, r0_0_0_2, g0_4);
              g1_4 = fmaf(ek1_0, r0_0_0_2, g1_4);
              g2_4 = fmaf(ek2_0, r0_0_0_2, g2_4);
              g2_1 = fmaf(ek2_1, r0_0_0_2, g2_1);
              g2_0 = fmaf(ek2_2, r0_0_0_2, g2_0);
              g3_4 = fmaf(ek3_0, r0_0_0_2, g3_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fmaf(ek0_0, r0_0_1_1, g0_5);
              g1_5 = fmaf(ek1_0, r0_0_1_1, g1_5);
              g1_1 = fmaf(ek1_1, r0_0_1_1, g1_1);
              g2_5 = fmaf(ek2_0, r0_0_1_1, g2_5);
              g2_2 = fmaf(ek2_1, r0_0_1_1, g2_2);
              g3_5 = fmaf(ek3_0, r0_0_1_1, g3_5);
              g3_1 = fmaf(ek3_1, r0_0_1_1, g3_1);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g0_6 = fmaf(ek0_0, r0_0_2_0, g0_6);
              g1_6 = fmaf(ek1_0, r0_0_2_0, g1_6);
              g1_2 = fmaf(ek1_1, r0_0_2_0, g1_2);
              g1_0 = fmaf(ek1_2, r0_0_2_0, g1_0);
              g2_6 = fmaf(ek2_0, r0_0_2_0, g2_6);
              g3_6 = fmaf(ek3_0, r0_0_2_0, g3_6);
              g3_2 = fmaf(ek3_1, r0_0_2_0, g3_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fmaf(ek0_0, r0_1_0_1, g0_7);
              g0_1 = fmaf(ek0_1, r0_1_0_1, g0_1);
              g1_7 = fmaf(ek1_0, r0_1_0_1, g1_7);
              g2_7 = fmaf(ek2_0, r0_1_0_1, g2_7);
              g2_3 = fmaf(ek2_1, r0_1_0_1, g2_3);
              g3_7 = fmaf(ek3_0, r0_1_0_1, g3_7);
              g3_1 = fmaf(ek3_2, r0_1_0_1, g3_1);
              const float r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fmaf(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fmaf(ek0_1, r0_1_1_0, g0_2);
              g1_8 = fmaf(ek1_0, r0_1_1_0, g1_8);
              g1_3 = fmaf(ek1_1, r0_1_1_0, g1_3);
              g2_8 = fmaf(ek2_0, r0_1_1_0, g2_8);
              g3_8 = fmaf(ek3_0, r0_1_1_0, g3_8);
              g3_3 = fmaf(ek3_1, r0_1_1_0, g3_3);
              g3_2 = fmaf(ek3_2, r0_1_1_0, g3_2);
              g3_0 = fmaf(ek3_3, r0_1_1_0, g3_0);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g0_9 = fmaf(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fmaf(ek0_1, r0_2_0_0, g0_3);
              g0_0 = fmaf(ek0_2, r0_2_0_0, g0_0);
              g1_9 = fmaf(ek1_0, r0_2_0_0, g1_9);
              g2_9 = fmaf(ek2_0, r0_2_0_0, g2_9);
              g3_9 = fmaf(ek3_0, r0_2_0_0, g3_9);
              g3_3 = fmaf(ek3_2, r0_2_0_0, g3_3);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g2_4 = fmaf(ek2_1, r0_0_0_3, g2_4);
              g2_1 = fmaf(ek2_2, r0_0_0_3, g2_1);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g1_4 = fmaf(ek1_1, r0_0_1_2, g1_4);
              g2_5 = fmaf(ek2_1, r0_0_1_2, g2_5);
              g2_2 = fmaf(ek2_2, r0_0_1_2, g2_2);
              g3_4 = fmaf(ek3_1, r0_0_1_2, g3_4);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g1_5 = fmaf(ek1_1, r0_0_2_1, g1_5);
              g1_1 = fmaf(ek1_2, r0_0_2_1, g1_1);
              g2_6 = fmaf(ek2_1, r0_0_2_1, g2_6);
              g3_5 = fmaf(ek3_1, r0_0_2_1, g3_5);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g1_6 = fmaf(ek1_1, r0_0_3_0, g1_6);
              g1_2 = fmaf(ek1_2, r0_0_3_0, g1_2);
              g3_6 = fmaf(ek3_1, r0_0_3_0, g3_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g0_4 = fmaf(ek0_1, r0_1_0_2, g0_4);
              g2_7 = fmaf(ek2_1, r0_1_0_2, g2_7);
              g2_3 = fmaf(ek2_2, r0_1_0_2, g2_3);
              g3_4 = fmaf(ek3_2, r0_1_0_2, g3_4);
              const float r0_1_1_1 = X * r1_0_1_1;
              g0_5 = fmaf(ek0_1, r0_1_1_1, g0_5);
              g1_7 = fmaf(ek1_1, r0_1_1_1, g1_7);
              g2_8 = fmaf(ek2_1, r0_1_1_1, g2_8);
              g3_7 = fmaf(ek3_1, r0_1_1_1, g3_7);
              g3_5 = fmaf(ek3_2, r0_1_1_1, g3_5);
              g3_1 = fmaf(ek3_3, r0_1_1_1, g3_1);
              const float r0_1_2_0 = X * r1_0_2_0;
              g0_6 = fmaf(ek0_1, r0_1_2_0, g0_6);
              g1_8 = fmaf(ek1_1, r0_1_2_0, g1_8);
              g1_3 = fmaf(ek1_2, r0_1_2_0, g1_3);
              g3_8 = fmaf(ek3_1, r0_1_2_0, g3_8);
              g3_6 = fmaf(ek3_2, r0_1_2_0, g3_6);
              g3_2 = fmaf(ek3_3, r0_1_2_0, g3_2);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g0_7 = fmaf(ek0_1, r0_2_0_1, g0_7);
              g0_1 = fmaf(ek0_2, r0_2_0_1, g0_1);
              g2_9 = fmaf(ek2_1, r0_2_0_1, g2_9);
              g3_7 = fmaf(ek3_2, r0_2_0_1, g3_7);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g0_8 = fmaf(ek0_1, r0_2_1_0, g0_8);
              g0_2 = fmaf(ek0_2, r0_2_1_0, g0_2);
              g1_9 = fmaf(ek1_1, r0_2_1_0, g1_9);
              g3_9 = fmaf(ek3_1, r0_2_1_0, g3_9);
              g3_8 = fmaf(ek3_2, r0_2_1_0, g3_8);
              g3_3 = fmaf(ek3_3, r0_2_1_0, g3_3);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g0_9 = fmaf(ek0_1, r0_3_0_0, g0_9);
              g0_3 = fmaf(ek0_2, r0_3_0_0, g0_3);
              g3_9 = fmaf(ek3_2, r0_3_0_0, g3_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g2_4 = fmaf(ek2_2, r0_0_0_4, g2_4);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g2_5 = fmaf(ek2_2, r0_0_1_3, g2_5);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g1_4 = fmaf(ek1_2, r0_0_2_2, g1_4);
              g2_6 = fmaf(ek2_2, r0_0_2_2, g2_6);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g1_5 = fmaf(ek1_2, r0_0_3_1, g1_5);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g1_6 = fmaf(ek1_2, r0_0_4_0, g1_6);
              const float r0_1_0_3 = X * r1_0_0_3;
              g2_7 = fmaf(ek2_2, r0_1_0_3, g2_7);
              const float r0_1_1_2 = X * r1_0_1_2;
              g2_8 = fmaf(ek2_2, r0_1_1_2, g2_8);
              g3_4 = fmaf(ek3_3, r0_1_1_2, g3_4);
              const float r0_1_2_1 = X * r1_0_2_1;
              g1_7 = fmaf(ek1_2, r0_1_2_1, g1_7);
              g3_5 = fmaf(ek3_3, r0_1_2_1, g3_5);
              const float r0_1_3_0 = X * r1_0_3_0;
              g1_8 = fmaf(ek1_2, r0_1_3_0, g1_8);
              g3_6 = fmaf(ek3_3, r0_1_3_0, g3_6);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g0_4 = fmaf(ek0_2, r0_2_0_2, g0_4);
              g2_9 = fmaf(ek2_2, r0_2_0_2, g2_9);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g0_5 = fmaf(ek0_2, r0_2_1_1, g0_5);
              g3_7 = fmaf(ek3_3, r0_2_1_1, g3_7);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g0_6 = fmaf(ek0_2, r0_2_2_0, g0_6);
              g1_9 = fmaf(ek1_2, r0_2_2_0, g1_9);
              g3_8 = fmaf(ek3_3, r0_2_2_0, g3_8);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g0_7 = fmaf(ek0_2, r0_3_0_1, g0_7);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g0_8 = fmaf(ek0_2, r0_3_1_0, g0_8);
              g3_9 = fmaf(ek3_3, r0_3_1_0, g3_9);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g0_9 = fmaf(ek0_2, r0_4_0_0, g0_9);
            }
            { const float eb = bi[5];
              o0_0 = fmaf(eb, g0_0, o0_0);
              o0_1 = fmaf(eb, g1_0, o0_1);
              o0_2 = fmaf(eb, g2_0, o0_2);
              o0_3 = fmaf(eb, g3_0, o0_3);
            }
            { const float eb = bi[6];
              o1_0 = fmaf(eb, g0_0, o1_0);
              o1_1 = fmaf(eb, g1_0, o1_1);
              o1_2 = fmaf(eb, g2_0, o1_2);
              o1_3 = fmaf(eb, g3_0, o1_3);
            }
            { const float eb = bi[7];
              o1_0 = fmaf(eb, g0_3, o1_0);
              o1_1 = fmaf(eb, g1_3, o1_1);
              o1_2 = fmaf(eb, g2_3, o1_2);
              o1_3 = fmaf(eb, g3_3, o1_3);
            }
            { const float eb = bi[8];
              o2_0 = fmaf(eb, g0_0, o2_0);
              o2_1 = fmaf(eb, g1_0, o2_1);
              o2_2 = fmaf(eb, g2_0, o2_2);
              o2_3 = fmaf(eb, g3_0, o2_3);
            }
            { const float eb = bi[9];
              o2_0 = fmaf(eb, g0_2, o2_0);
              o2_1 = fmaf(eb, g1_2, o2_1);
              o2_2 = fmaf(eb, g2_2, o2_2);
              o2_3 = fmaf(eb, g3_2, o2_3);
            }
            { const float eb = bi[10];
              o3_0 = fmaf(eb, g0_0, o3_0);
              o3_1 = fmaf(eb, g1_0, o3_1);
              o3_2 = fmaf(eb, g2_0, o3_2);
              o3_3 = fmaf(eb, g3_0, o3_3);
            }
            { const float eb = bi[11];
              o3_0 = fmaf(eb, g0_1, o3_0);
              o3_1 = fmaf(eb, g1_1, o3_1);
              o3_2 = fmaf(eb, g2_1, o3_2);
              o3_3 = fmaf(eb, g3_1, o3_3);
            }
            { const float eb = bi[12];
              o4_0 = fmaf(eb, g0_0, o4_0);
              o4_1 = fmaf(eb, g1_0, o4_1);
              o4_2 = fmaf(eb, g2_0, o4_2);
              o4_3 = fmaf(eb, g3_0, o4_3);
            }
            { const float eb = bi[13];
              o4_0 = fmaf(eb, g0_3, o4_0);
              o4_1 = fmaf(eb, g1_3, o4_1);
              o4_2 = fmaf(eb, g2_3, o4_2);
              o4_3 = fmaf(eb, g3_3, o4_3);
            }
            { const float eb = bi[14];
              o5_0 = fmaf(eb, g0_0, o5_0);
              o5_1 = fmaf(eb, g1_0, o5_1);
              o5_2 = fmaf(eb, g2_0, o5_2);
              o5_3 = fmaf(eb, g3_0, o5_3);
            }
            { const float eb = bi[15];
              o5_0 = fmaf(eb, g0_3, o5_0);
              o5_1 = fmaf(eb, g1_3, o5_1);
              o5_2 = fmaf(eb, g2_3, o5_2);
              o5_3 = fmaf(eb, g3_3, o5_3);
            }
            { const float eb = bi[16];
              o5_0 = fmaf(eb, g0_9, o5_0);
              o5_1 = fmaf(eb, g1_9, o5_1);
              o5_2 = fmaf(eb, g2_9, o5_2);
              o5_3 = fmaf(eb, g3_9, o5_3);
            }
            { const float eb = bi[17];
              o6_0 = fmaf(eb, g0_0, o6_0);
              o6_1 = fmaf(eb, g1_0, o6_1);
              o6_2 = fmaf(eb, g2_0, o6_2);
              o6_3 = fmaf(eb, g3_0, o6_3);
            }
            { const float eb = bi[18];
              o6_0 = fmaf(eb, g0_2, o6_0);
              o6_1 = fmaf(eb, g1_2, o6_1);
              o6_2 = fmaf(eb, g2_2, o6_2);
              o6_3 = fmaf(eb, g3_2, o6_3);
            }
            { const float eb = bi[19];
              o6_0 = fmaf(eb, g0_3, o6_0);
              o6_1 = fmaf(eb, g1_3, o6_1);
              o6_2 = fmaf(eb, g2_3, o6_2);
              o6_3 = fmaf(eb, g3_3, o6_3);
            }
            { const float eb = bi[20];
              o6_0 = fmaf(eb, g0_8, o6_0);
              o6_1 = fmaf(eb, g1_8, o6_1);
              o6_2 = fmaf(eb, g2_8, o6_2);
              o6_3 = fmaf(eb, g3_8, o6_3);
            }
            { const float eb = bi[21];
              o7_0 = fmaf(eb, g0_0, o7_0);
              o7_1 = fmaf(eb, g1_0, o7_1);
              o7_2 = fmaf(eb, g2_0, o7_2);
              o7_3 = fmaf(eb, g3_0, o7_3);
            }
            { const float eb = bi[22];
              o7_0 = fmaf(eb, g0_1, o7_0);
              o7_1 = fmaf(eb, g1_1, o7_1);
              o7_2 = fmaf(eb, g2_1, o7_2);
              o7_3 = fmaf(eb, g3_1, o7_3);
            }
            { const float eb = bi[23];
              o7_0 = fmaf(eb, g0_3, o7_0);
              o7_1 = fmaf(eb, g1_3, o7_1);
              o7_2 = fmaf(eb, g2_3, o7_2);
              o7_3 = fmaf(eb, g3_3, o7_3);
            }
            { const float eb = bi[24];
              o7_0 = fmaf(eb, g0_7, o7_0);
              o7_1 = fmaf(eb, g1_7, o7_1);
              o7_2 = fmaf(eb, g2_7, o7_2);
              o7_3 = fmaf(eb, g3_7, o7_3);
            }
            { const float eb = bi[25];
              o8_0 = fmaf(eb, g0_0, o8_0);
              o8_1 = fmaf(eb, g1_0, o8_1);
              o8_2 = fmaf(eb, g2_0, o8_2);
              o8_3 = fmaf(eb, g3_0, o8_3);
            }
            { const float eb = bi[26];
              o8_0 = fmaf(eb, g0_2, o8_0);
              o8_1 = fmaf(eb, g1_2, o8_1);
              o8_2 = fmaf(eb, g2_2, o8_2);
              o8_3 = fmaf(eb, g3_2, o8_3);
            }
            { const float eb = bi[27];
              o9_0 = fmaf(eb, g0_0, o9_0);
              o9_1 = fmaf(eb, g1_0, o9_1);
              o9_2 = fmaf(eb, g2_0, o9_2);
              o9_3 = fmaf(eb, g3_0, o9_3);
            }
            { const float eb = bi[28];
              o9_0 = fmaf(eb, g0_2, o9_0);
              o9_1 = fmaf(eb, g1_2, o9_1);
              o9_2 = fmaf(eb, g2_2, o9_2);
              o9_3 = fmaf(eb, g3_2, o9_3);
            }
            { const float eb = bi[29];
              o9_0 = fmaf(eb, g0_3, o9_0);
              o9_1 = fmaf(eb, g1_3, o9_1);
              o9_2 = fmaf(eb, g2_3, o9_2);
              o9_3 = fmaf(eb, g3_3, o9_3);
            }
            { const float eb = bi[30];
              o9_0 = fmaf(eb, g0_8, o9_0);
              o9_1 = fmaf(eb, g1_8, o9_1);
              o9_2 = fmaf(eb, g2_8, o9_2);
              o9_3 = fmaf(eb, g3_8, o9_3);
            }
            { const float eb = bi[31];
              o10_0 = fmaf(eb, g0_0, o10_0);
              o10_1 = fmaf(eb, g1_0, o10_1);
              o10_2 = fmaf(eb, g2_0, o10_2);
              o10_3 = fmaf(eb, g3_0, o10_3);
            }
            { const float eb = bi[32];
              o10_0 = fmaf(eb, g0_2, o10_0);
              o10_1 = fmaf(eb, g1_2, o10_1);
              o10_2 = fmaf(eb, g2_2, o10_2);
              o10_3 = fmaf(eb, g3_2, o10_3);
            }
            { const float eb = bi[33];
              o10_0 = fmaf(eb, g0_6, o10_0);
              o10_1 = fmaf(eb, g1_6, o10_1);
              o10_2 = fmaf(eb, g2_6, o10_2);
              o10_3 = fmaf(eb, g3_6, o10_3);
            }
            { const float eb = bi[34];
              o11_0 = fmaf(eb, g0_0, o11_0);
              o11_1 = fmaf(eb, g1_0, o11_1);
              o11_2 = fmaf(eb, g2_0, o11_2);
              o11_3 = fmaf(eb, g3_0, o11_3);
            }
            { const float eb = bi[35];
              o11_0 = fmaf(eb, g0_1, o11_0);
              o11_1 = fmaf(eb, g1_1, o11_1);
              o11_2 = fmaf(eb, g2_1, o11_2);
              o11_3 = fmaf(eb, g3_1, o11_3);
            }
            { const float eb = bi[36];
              o11_0 = fmaf(eb, g0_2, o11_0);
              o11_1 = fmaf(eb, g1_2, o11_1);
              o11_2 = fmaf(eb, g2_2, o11_2);
              o11_3 = fmaf(eb, g3_2, o11_3);
            }
            { const float eb = bi[37];
              o11_0 = fmaf(eb, g0_5, o11_0);
              o11_1 = fmaf(eb, g1_5, o11_1);
              o11_2 = fmaf(eb, g2_5, o11_2);
              o11_3 = fmaf(eb, g3_5, o11_3);
            }
            { const float eb = bi[38];
              o12_0 = fmaf(eb, g0_0, o12_0);
              o12_1 = fmaf(eb, g1_0, o12_1);
              o12_2 = fmaf(eb, g2_0, o12_2);
              o12_3 = fmaf(eb, g3_0, o12_3);
            }
            { const float eb = bi[39];
              o12_0 = fmaf(eb, g0_1, o12_0);
              o12_1 = fmaf(eb, g1_1, o12_1);
              o12_2 = fmaf(eb, g2_1, o12_2);
              o12_3 = fmaf(eb, g3_1, o12_3);
            }
            { const float eb = bi[40];
              o13_0 = fmaf(eb, g0_0, o13_0);
              o13_1 = fmaf(eb, g1_0, o13_1);
              o13_2 = fmaf(eb, g2_0, o13_2);
              o13_3 = fmaf(eb, g3_0, o13_3);
            }
            { const float eb = bi[41];
              o13_0 = fmaf(eb, g0_1, o13_0);
              o13_1 = fmaf(eb, g1_1, o13_1);
              o13_2 = fmaf(eb, g2_1, o13_2);
              o13_3 = fmaf(eb, g3_1, o13_3);
            }
            { const float eb = bi[42];
              o13_0 = fmaf(eb, g0_3, o13_0);
              o13_1 = fmaf(eb, g1_3, o13_1);
              o13_2 = fmaf(eb, g2_3, o13_2);
              o13_3 = fmaf(eb, g3_3, o13_3);
            }
            { const float eb = bi[43];
              o13_0 = fmaf(eb, g0_7, o13_0);
              o13_1 = fmaf(eb, g1_7, o13_1);
              o13_2 = fmaf(eb, g2_7, o13_2);
              o13_3 = fmaf(eb, g3_7, o13_3);
            }
            { const float eb = bi[44];
              o14_0 = fmaf(eb, g0_0, o14_0);
              o14_1 = fmaf(eb, g1_0, o14_1);
              o14_2 = fmaf(eb, g2_0, o14_2);
              o14_3 = fmaf(eb, g3_0, o14_3);
            }
            { const float eb = bi[45];
              o14_0 = fmaf(eb, g0_1, o14_0);
              o14_1 = fmaf(eb, g1_1, o14_1);
              o14_2 = fmaf(eb, g2_1, o14_2);
              o14_3 = fmaf(eb, g3_1, o14_3);
            }
            { const float eb = bi[46];
              o14_0 = fmaf(eb, g0_2, o14_0);
              o14_1 = fmaf(eb, g1_2, o14_1);
              o14_2 = fmaf(eb, g2_2, o14_2);
              o14_3 = fmaf(eb, g3_2, o14_3);
            }
            { const float eb = bi[47];
              o14_0 = fmaf(eb, g0_5, o14_0);
              o14_1 = fmaf(eb, g1_5, o14_1);
              o14_2 = fmaf(eb, g2_5, o14_2);
              o14_3 = fmaf(eb, g3_5, o14_3);
            }
            { const float eb = bi[48];
              o15_0 = fmaf(eb, g0_0, o15_0);
              o15_1 = fmaf(eb, g1_0, o15_1);
              o15_2 = fmaf(eb, g2_0, o15_2);
              o15_3 = fmaf(eb, g3_0, o15_3);
            }
            { const float eb = bi[49];
              o15_0 = fmaf(eb, g0_1, o15_0);
              o15_1 = fmaf(eb, g1_1, o15_1);
              o15_2 = fmaf(eb, g2_1, o15_2);
              o15_3 = fmaf(eb, g3_1, o15_3);
            }
            { const float eb = bi[50];
              o15_0 = fmaf(eb, g0_4, o15_0);
              o15_1 = fmaf(eb, g1_4, o15_1);
              o15_2 = fmaf(eb, g2_4, o15_2);
              o15_3 = fmaf(eb, g3_4, o15_3);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptk1 = PT[(fI + 1) * N + fJ + 0];
            const double ptk2 = PT[(fI + 2) * N + fJ + 0];
            const double ptk3 = PT[(fI + 3) * N + fJ + 0];
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
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc0_3 = PA[(fQ + 0) * N + fI + 3];
            const double Abc1_0 = PA[(fQ + 1) * N + fI + 0];
            const double Abc1_1 = PA[(fQ + 1) * N + fI + 1];
            const double Abc1_2 = PA[(fQ + 1) * N + fI + 2];
            const double Abc1_3 = PA[(fQ + 1) * N + fI + 3];
            const double Abc2_0 = PA[(fQ + 2) * N + fI + 0];
            const double Abc2_1 = PA[(fQ + 2) * N + fI + 1];
            const double Abc2_2 = PA[(fQ + 2) * N + fI + 2];
            const double Abc2_3 = PA[(fQ + 2) * N + fI + 3];
            const double Abc3_0 = PA[(fQ + 3) * N + fI + 0];
            const double Abc3_1 = PA[(fQ + 3) * N + fI + 1];
            const double Abc3_2 = PA[(fQ + 3) * N + fI + 2];
            const double Abc3_3 = PA[(fQ + 3) * N + fI + 3];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac0_3 = PA[(fP + 0) * N + fI + 3];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac1_3 = PA[(fP + 1) * N + fI + 3];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac2_3 = PA[(fP + 2) * N + fI + 3];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac3_3 = PA[(fP + 3) * N + fI + 3];
            jab0 += o0_0 * ptk0 + o0_1 * ptk1 + o0_2 * ptk2 + o0_3 * ptk3;
            jab1 += o1_0 * ptk0 + o1_1 * ptk1 + o1_2 * ptk2 + o1_3 * ptk3;
            jab2 += o2_0 * ptk0 + o2_1 * ptk1 + o2_2 * ptk2 + o2_3 * ptk3;
            jab3 += o3_0 * ptk0 + o3_1 * ptk1 + o3_2 * ptk2 + o3_3 * ptk3;
            jab4 += o4_0 * ptk0 + o4_1 * ptk1 + o4_2 * ptk2 + o4_3 * ptk3;
            jab5 += o5_0 * ptk0 + o5_1 * ptk1 + o5_2 * ptk2 + o5_3 * ptk3;
            jab6 += o6_0 * ptk0 + o6_1 * ptk1 + o6_2 * ptk2 + o6_3 * ptk3;
            jab7 += o7_0 * ptk0 + o7_1 * ptk1 + o7_2 * ptk2 + o7_3 * ptk3;
            jab8 += o8_0 * ptk0 + o8_1 * ptk1 + o8_2 * ptk2 + o8_3 * ptk3;
            jab9 += o9_0 * ptk0 + o9_1 * ptk1 + o9_2 * ptk2 + o9_3 * ptk3;
            jab10 += o10_0 * ptk0 + o10_1 * ptk1 + o10_2 * ptk2 + o10_3 * ptk3;
            jab11 += o11_0 * ptk0 + o11_1 * ptk1 + o11_2 * ptk2 + o11_3 * ptk3;
            jab12 += o12_0 * ptk0 + o12_1 * ptk1 + o12_2 * ptk2 + o12_3 * ptk3;
            jab13 += o13_0 * ptk0 + o13_1 * ptk1 + o13_2 * ptk2 + o13_3 * ptk3;
            jab14 += o14_0 * ptk0 + o14_1 * ptk1 + o14_2 * ptk2 + o14_3 * ptk3;
            jab15 += o15_0 * ptk0 + o15_1 * ptk1 + o15_2 * ptk2 + o15_3 * ptk3;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5 + o6_0 * ptb6 + o7_0 * ptb7 + o8_0 * ptb8 + o9_0 * ptb9 + o10_0 * ptb10 + o11_0 * ptb11 + o12_0 * ptb12 + o13_0 * ptb13 + o14_0 * ptb14 + o15_0 * ptb15));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15));
            atomicAdd(Jacc + (fI + 3) * N + fJ + 0, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5 + o6_3 * ptb6 + o7_3 * ptb7 + o8_3 * ptb8 + o9_3 * ptb9 + o10_3 * ptb10 + o11_3 * ptb11 + o12_3 * ptb12 + o13_3 * ptb13 + o14_3 * ptb14 + o15_3 * ptb15));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0 + o1_0 * Abd1_0 + o2_0 * Abd2_0 + o3_0 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o4_0 * Aad1_0 + o8_0 * Aad2_0 + o12_0 * Aad3_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o0_1 * Abc0_1 + o0_2 * Abc0_2 + o0_3 * Abc0_3 + o1_0 * Abc1_0 + o1_1 * Abc1_1 + o1_2 * Abc1_2 + o1_3 * Abc1_3 + o2_0 * Abc2_0 + o2_1 * Abc2_1 + o2_2 * Abc2_2 + o2_3 * Abc2_3 + o3_0 * Abc3_0 + o3_1 * Abc3_1 + o3_2 * Abc3_2 + o3_3 * Abc3_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o0_1 * Aac0_1 + o0_2 * Aac0_2 + o0_3 * Aac0_3 + o4_0 * Aac1_0 + o4_1 * Aac1_1 + o4_2 * Aac1_2 + o4_3 * Aac1_3 + o8_0 * Aac2_0 + o8_1 * Aac2_1 + o8_2 * Aac2_2 + o8_3 * Aac2_3 + o12_0 * Aac3_0 + o12_1 * Aac3_1 + o12_2 * Aac3_2 + o12_3 * Aac3_3));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Abd0_0 + o1_1 * Abd1_0 + o2_1 * Abd2_0 + o3_1 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Aad0_0 + o4_1 * Aad1_0 + o8_1 * Aad2_0 + o12_1 * Aad3_0));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Abd0_0 + o1_2 * Abd1_0 + o2_2 * Abd2_0 + o3_2 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Aad0_0 + o4_2 * Aad1_0 + o8_2 * Aad2_0 + o12_2 * Aad3_0));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_3 * Abd0_0 + o1_3 * Abd1_0 + o2_3 * Abd2_0 + o3_3 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_3 * Aad0_0 + o4_3 * Aad1_0 + o8_3 * Aad2_0 + o12_3 * Aad3_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_0 * Aad0_0 + o5_0 * Aad1_0 + o9_0 * Aad2_0 + o13_0 * Aad3_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_0 * Aac0_0 + o1_1 * Aac0_1 + o1_2 * Aac0_2 + o1_3 * Aac0_3 + o5_0 * Aac1_0 + o5_1 * Aac1_1 + o5_2 * Aac1_2 + o5_3 * Aac1_3 + o9_0 * Aac2_0 + o9_1 * Aac2_1 + o9_2 * Aac2_2 + o9_3 * Aac2_3 + o13_0 * Aac3_0 + o13_1 * Aac3_1 + o13_2 * Aac3_2 + o13_3 * Aac3_3));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_1 * Aad0_0 + o5_1 * Aad1_0 + o9_1 * Aad2_0 + o13_1 * Aad3_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_2 * Aad0_0 + o5_2 * Aad1_0 + o9_2 * Aad2_0 + o13_2 * Aad3_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 3, deg * (o1_3 * Aad0_0 + o5_3 * Aad1_0 + o9_3 * Aad2_0 + o13_3 * Aad3_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_0 * Aad0_0 + o6_0 * Aad1_0 + o10_0 * Aad2_0 + o14_0 * Aad3_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_0 * Aac0_0 + o2_1 * Aac0_1 + o2_2 * Aac0_2 + o2_3 * Aac0_3 + o6_0 * Aac1_0 + o6_1 * Aac1_1 + o6_2 * Aac1_2 + o6_3 * Aac1_3 + o10_0 * Aac2_0 + o10_1 * Aac2_1 + o10_2 * Aac2_2 + o10_3 * Aac2_3 + o14_0 * Aac3_0 + o14_1 * Aac3_1 + o14_2 * Aac3_2 + o14_3 * Aac3_3));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_1 * Aad0_0 + o6_1 * Aad1_0 + o10_1 * Aad2_0 + o14_1 * Aad3_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_2 * Aad0_0 + o6_2 * Aad1_0 + o10_2 * Aad2_0 + o14_2 * Aad3_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 3, deg * (o2_3 * Aad0_0 + o6_3 * Aad1_0 + o10_3 * Aad2_0 + o14_3 * Aad3_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_0 * Aad0_0 + o7_0 * Aad1_0 + o11_0 * Aad2_0 + o15_0 * Aad3_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_0 * Aac0_0 + o3_1 * Aac0_1 + o3_2 * Aac0_2 + o3_3 * Aac0_3 + o7_0 * Aac1_0 + o7_1 * Aac1_1 + o7_2 * Aac1_2 + o7_3 * Aac1_3 + o11_0 * Aac2_0 + o11_1 * Aac2_1 + o11_2 * Aac2_2 + o11_3 * Aac2_3 + o15_0 * Aac3_0 + o15_1 * Aac3_1 + o15_2 * Aac3_2 + o15_3 * Aac3_3));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_1 * Aad0_0 + o7_1 * Aad1_0 + o11_1 * Aad2_0 + o15_1 * Aad3_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_2 * Aad0_0 + o7_2 * Aad1_0 + o11_2 * Aad2_0 + o15_2 * Aad3_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 3, deg * (o3_3 * Aad0_0 + o7_3 * Aad1_0 + o11_3 * Aad2_0 + o15_3 * Aad3_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o4_0 * Abd0_0 + o5_0 * Abd1_0 + o6_0 * Abd2_0 + o7_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o4_1 * Abc0_1 + o4_2 * Abc0_2 + o4_3 * Abc0_3 + o5_0 * Abc1_0 + o5_1 * Abc1_1 + o5_2 * Abc1_2 + o5_3 * Abc1_3 + o6_0 * Abc2_0 + o6_1 * Abc2_1 + o6_2 * Abc2_2 + o6_3 * Abc2_3 + o7_0 * Abc3_0 + o7_1 * Abc3_1 + o7_2 * Abc3_2 + o7_3 * Abc3_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o4_1 * Abd0_0 + o5_1 * Abd1_0 + o6_1 * Abd2_0 + o7_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o4_2 * Abd0_0 + o5_2 * Abd1_0 + o6_2 * Abd2_0 + o7_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o4_3 * Abd0_0 + o5_3 * Abd1_0 + o6_3 * Abd2_0 + o7_3 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o8_0 * Abd0_0 + o9_0 * Abd1_0 + o10_0 * Abd2_0 + o11_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_0 * Abc0_0 + o8_1 * Abc0_1 + o8_2 * Abc0_2 + o8_3 * Abc0_3 + o9_0 * Abc1_0 + o9_1 * Abc1_1 + o9_2 * Abc1_2 + o9_3 * Abc1_3 + o10_0 * Abc2_0 + o10_1 * Abc2_1 + o10_2 * Abc2_2 + o10_3 * Abc2_3 + o11_0 * Abc3_0 + o11_1 * Abc3_1 + o11_2 * Abc3_2 + o11_3 * Abc3_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o8_1 * Abd0_0 + o9_1 * Abd1_0 + o10_1 * Abd2_0 + o11_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o8_2 * Abd0_0 + o9_2 * Abd1_0 + o10_2 * Abd2_0 + o11_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o8_3 * Abd0_0 + o9_3 * Abd1_0 + o10_3 * Abd2_0 + o11_3 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o12_0 * Abd0_0 + o13_0 * Abd1_0 + o14_0 * Abd2_0 + o15_0 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_0 * Abc0_0 + o12_1 * Abc0_1 + o12_2 * Abc0_2 + o12_3 * Abc0_3 + o13_0 * Abc1_0 + o13_1 * Abc1_1 + o13_2 * Abc1_2 + o13_3 * Abc1_3 + o14_0 * Abc2_0 + o14_1 * Abc2_1 + o14_2 * Abc2_2 + o14_3 * Abc2_3 + o15_0 * Abc3_0 + o15_1 * Abc3_1 + o15_2 * Abc3_2 + o15_3 * Abc3_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o12_1 * Abd0_0 + o13_1 * Abd1_0 + o14_1 * Abd2_0 + o15_1 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o12_2 * Abd0_0 + o13_2 * Abd1_0 + o14_2 * Abd2_0 + o15_2 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o12_3 * Abd0_0 + o13_3 * Abd1_0 + o14_3 * Abd2_0 + o15_3 * Abd3_0));
          }
        } break;
        case 1: {  // ket functions [4, 5]
          float o0_4 = 0;
          float o0_5 = 0;
          float o1_4 = 0;
          float o1_5 = 0;
          float o2_4 = 0;
          float o2_5 = 0;
          float o3_4 = 0;
          float o3_5 = 0;
          float o4_4 = 0;
          float o4_5 = 0;
          float o5_4 = 0;
          float o5_5 = 0;
          float o6_4 = 0;
          float o6_5 = 0;
          float o7_4 = 0;
          float o7_5 = 0;
          float o8_4 = 0;
          float o8_5 = 0;
          float o9_4 = 0;
          float o9_5 = 0;
          float o10_4 = 0;
          float o10_5 = 0;
          float o11_4 = 0;
          float o11_5 = 0;
          float o12_4 = 0;
          float o12_5 = 0;
          float o13_4 = 0;
          float o13_5 = 0;
          float o14_4 = 0;
          float o14_5 = 0;
          float o15_4 = 0;
          float o15_5 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 51;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g4_0 = 0;
            float g4_1 = 0;
            float g4_2 = 0;
            float g4_3 = 0;
            float g4_4 = 0;
            float g4_5 = 0;
            float g4_6 = 0;
            float g4_7 = 0;
            float g4_8 = 0;
            float g4_9 = 0;
            float g5_0 = 0;
            float g5_1 = 0;
            float g5_2 = 0;
            float g5_3 = 0;
            float g5_4 = 0;
            float g5_5 = 0;
            float g5_6 = 0;
            float g5_7 = 0;
            float g5_8 = 0;
            float g5_9 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 26 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[5];
              sqb::boysf<4>(T, a.boys_tab_f, F);
              const float s0 = TWO_PI_2_5F * rs;
              const float m2a = -2.0f * alpha;
              float w = s0;
              const float b0 = w * F[0];
              w *= m2a;
              const float b1 = w * F[1];
              w *= m2a;
              const float b2 = w * F[2];
              w *= m2a;
              const float b3 = w * F[3];
              w *= m2a;
              const float b4 = w * F[4];
              const float ek4_0 = kj[18 * kS];
              const float ek4_1 = -kj[19 * kS];
              const float ek4_2 = -kj[20 * kS];
              const float ek4_3 = kj[21 * kS];
              const float ek5_0 = kj[22 * kS];
              const float ek5_1 = -kj[23 * kS];
              const float ek5_2 = -kj[24 * kS];
              const float ek5_3 = kj[25 * kS];
              g4_0 = fmaf(ek4_0, b0, g4_0);
              g5_0 = fmaf(ek5_0, b0, g5_0);
              const float r0_0_0_1 = Z * b1;
              g4_1 = fmaf(ek4_0, r0_0_0_1, g4_1);
              g4_0 = fmaf(ek4_1, r0_0_0_1, g4_0);
              g5_1 = fmaf(ek5_0, r0_0_0_1, g5_1);
              g5_0 = fmaf(ek5_1, r0_0_0_1, g5_0);
              const float r0_0_1_0 = Y * b1;
              g4_2 = fmaf(ek4_0, r0_0_1_0, g4_2);
              g5_2 = fmaf(ek5_0, r0_0_1_0, g5_2);
              g5_0 = fmaf(ek5_2, r0_0_1_0, g5_0);
              const float r0_1_0_0 = X * b1;
              g4_3 = fmaf(ek4_0, r0_1_0_0, g4_3);
              g4_0 = fmaf(ek4_2, r0_1_0_0, g4_0);
              g5_3 = fmaf(ek5_0, r0_1_0_0, g5_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g4_4 = fmaf(ek4_0, r0_0_0_2, g4_4);
              g4_1 = fmaf(ek4_1, r0_0_0_2, g4_1);
              g5_4 = fmaf(ek5_0, r0_0_0_2, g5_4);
              g5_1 = fmaf(ek5_1, r0_0_0_2, g5_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g4_5 = fmaf(ek4_0, r0_0_1_1, g4_5);
              g4_2 = fmaf(ek4_1, r0_0_1_1, g4_2);
              g5_5 = fmaf(ek5_0, r0_0_1_1, g5_5);
              g5_2 = fmaf(ek5_1, r0_0_1_1, g5_2);
              g5_1 = fmaf(ek5_2, r0_0_1_1, g5_1);
              g5_0 = fmaf(ek5_3, r0_0_1_1, g5_0);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g4_6 = fmaf(ek4_0, r0_0_2_0, g4_6);
              g5_6 = fmaf(ek5_0, r0_0_2_0, g5_6);
              g5_2 = fmaf(ek5_2, r0_0_2_0, g5_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g4_7 = fmaf(ek4_0, r0_1_0_1, g4_7);
              g4_3 = fmaf(ek4_1, r0_1_0_1, g4_3);
              g4_1 = fmaf(ek4_2, r0_1_0_1, g4_1);
              g4_0 = fmaf(ek4_3, r0_1_0_1, g4_0);
              g5_7 = fmaf(ek5_0, r0_1_0_1, g5_7);
              g5_3 = fmaf(ek5_1, r0_1_0_1, g5_3);
              const float r0_1_1_0 = X * r1_0_1_0;
              g4_8 = fmaf(ek4_0, r0_1_1_0, g4_8);
              g4_2 = fmaf(ek4_2, r0_1_1_0, g4_2);
              g5_8 = fmaf(ek5_0, r0_1_1_0, g5_8);
              g5_3 = fmaf(ek5_2, r0_1_1_0, g5_3);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g4_9 = fmaf(ek4_0, r0_2_0_0, g4_9);
              g4_3 = fmaf(ek4_2, r0_2_0_0, g4_3);
              g5_9 = fmaf(ek5_0, r0_2_0_0, g5_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g4_4 = fmaf(ek4_1, r0_0_0_3, g4_4);
              g5_4 = fmaf(ek5_1, r0_0_0_3, g5_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g4_5 = fmaf(ek4_1, r0_0_1_2, g4_5);
              g5_5 = fmaf(ek5_1, r0_0_1_2, g5_5);
              g5_4 = fmaf(ek5_2, r0_0_1_2, g5_4);
              g5_1 = fmaf(ek5_3, r0_0_1_2, g5_1);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g4_6 = fmaf(ek4_1, r0_0_2_1, g4_6);
              g5_6 = fmaf(ek5_1, r0_0_2_1, g5_6);
              g5_5 = fmaf(ek5_2, r0_0_2_1, g5_5);
              g5_2 = fmaf(ek5_3, r0_0_2_1, g5_2);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g5_6 = fmaf(ek5_2, r0_0_3_0, g5_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g4_7 = fmaf(ek4_1, r0_1_0_2, g4_7);
              g4_4 = fmaf(ek4_2, r0_1_0_2, g4_4);
              g4_1 = fmaf(ek4_3, r0_1_0_2, g4_1);
              g5_7 = fmaf(ek5_1, r0_1_0_2, g5_7);
              const float r0_1_1_1 = X * r1_0_1_1;
              g4_8 = fmaf(ek4_1, r0_1_1_1, g4_8);
              g4_5 = fmaf(ek4_2, r0_1_1_1, g4_5);
              g4_2 = fmaf(ek4_3, r0_1_1_1, g4_2);
              g5_8 = fmaf(ek5_1, r0_1_1_1, g5_8);
              g5_7 = fmaf(ek5_2, r0_1_1_1, g5_7);
              g5_3 = fmaf(ek5_3, r0_1_1_1, g5_3);
              const float r0_1_2_0 = X * r1_0_2_0;
              g4_6 = fmaf(ek4_2, r0_1_2_0, g4_6);
              g5_8 = fmaf(ek5_2, r0_1_2_0, g5_8);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g4_9 = fmaf(ek4_1, r0_2_0_1, g4_9);
              g4_7 = fmaf(ek4_2, r0_2_0_1, g4_7);
              g4_3 = fmaf(ek4_3, r0_2_0_1, g4_3);
              g5_9 = fmaf(ek5_1, r0_2_0_1, g5_9);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g4_8 = fmaf(ek4_2, r0_2_1_0, g4_8);
              g5_9 = fmaf(ek5_2, r0_2_1_0, g5_9);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g4_9 = fmaf(ek4_2, r0_3_0_0, g4_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g5_4 = fmaf(ek5_3, r0_0_1_3, g5_4);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g5_5 = fmaf(ek5_3, r0_0_2_2, g5_5);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g5_6 = fmaf(ek5_3, r0_0_3_1, g5_6);
              const float r0_1_0_3 = X * r1_0_0_3;
              g4_4 = fmaf(ek4_3, r0_1_0_3, g4_4);
              const float r0_1_1_2 = X * r1_0_1_2;
              g4_5 = fmaf(ek4_3, r0_1_1_2, g4_5);
              g5_7 = fmaf(ek5_3, r0_1_1_2, g5_7);
              const float r0_1_2_1 = X * r1_0_2_1;
              g4_6 = fmaf(ek4_3, r0_1_2_1, g4_6);
              g5_8 = fmaf(ek5_3, r0_1_2_1, g5_8);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g4_7 = fmaf(ek4_3, r0_2_0_2, g4_7);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g4_8 = fmaf(ek4_3, r0_2_1_1, g4_8);
              g5_9 = fmaf(ek5_3, r0_2_1_1, g5_9);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g4_9 = fmaf(ek4_3, r0_3_0_1, g4_9);
            }
            { const float eb = bi[5];
              o0_4 = fmaf(eb, g4_0, o0_4);
              o0_5 = fmaf(eb, g5_0, o0_5);
            }
            { const float eb = bi[6];
              o1_4 = fmaf(eb, g4_0, o1_4);
              o1_5 = fmaf(eb, g5_0, o1_5);
            }
            { const float eb = bi[7];
              o1_4 = fmaf(eb, g4_3, o1_4);
              o1_5 = fmaf(eb, g5_3, o1_5);
            }
            { const float eb = bi[8];
              o2_4 = fmaf(eb, g4_0, o2_4);
              o2_5 = fmaf(eb, g5_0, o2_5);
            }
            { const float eb = bi[9];
              o2_4 = fmaf(eb, g4_2, o2_4);
              o2_5 = fmaf(eb, g5_2, o2_5);
            }
            { const float eb = bi[10];
              o3_4 = fmaf(eb, g4_0, o3_4);
              o3_5 = fmaf(eb, g5_0, o3_5);
            }
            { const float eb = bi[11];
              o3_4 = fmaf(eb, g4_1, o3_4);
              o3_5 = fmaf(eb, g5_1, o3_5);
            }
            { const float eb = bi[12];
              o4_4 = fmaf(eb, g4_0, o4_4);
              o4_5 = fmaf(eb, g5_0, o4_5);
            }
            { const float eb = bi[13];
              o4_4 = fmaf(eb, g4_3, o4_4);
              o4_5 = fmaf(eb, g5_3, o4_5);
            }
            { const float eb = bi[14];
              o5_4 = fmaf(eb, g4_0, o5_4);
              o5_5 = fmaf(eb, g5_0, o5_5);
            }
            { const float eb = bi[15];
              o5_4 = fmaf(eb, g4_3, o5_4);
              o5_5 = fmaf(eb, g5_3, o5_5);
            }
            { const float eb = bi[16];
              o5_4 = fmaf(eb, g4_9, o5_4);
              o5_5 = fmaf(eb, g5_9, o5_5);
            }
            { const float eb = bi[17];
              o6_4 = fmaf(eb, g4_0, o6_4);
              o6_5 = fmaf(eb, g5_0, o6_5);
            }
            { const float eb = bi[18];
              o6_4 = fmaf(eb, g4_2, o6_4);
              o6_5 = fmaf(eb, g5_2, o6_5);
            }
            { const float eb = bi[19];
              o6_4 = fmaf(eb, g4_3, o6_4);
              o6_5 = fmaf(eb, g5_3, o6_5);
            }
            { const float eb = bi[20];
              o6_4 = fmaf(eb, g4_8, o6_4);
              o6_5 = fmaf(eb, g5_8, o6_5);
            }
            { const float eb = bi[21];
              o7_4 = fmaf(eb, g4_0, o7_4);
              o7_5 = fmaf(eb, g5_0, o7_5);
            }
            { const float eb = bi[22];
              o7_4 = fmaf(eb, g4_1, o7_4);
              o7_5 = fmaf(eb, g5_1, o7_5);
            }
            { const float eb = bi[23];
              o7_4 = fmaf(eb, g4_3, o7_4);
              o7_5 = fmaf(eb, g5_3, o7_5);
            }
            { const float eb = bi[24];
              o7_4 = fmaf(eb, g4_7, o7_4);
              o7_5 = fmaf(eb, g5_7, o7_5);
            }
            { const float eb = bi[25];
              o8_4 = fmaf(eb, g4_0, o8_4);
              o8_5 = fmaf(eb, g5_0, o8_5);
            }
            { const float eb = bi[26];
              o8_4 = fmaf(eb, g4_2, o8_4);
              o8_5 = fmaf(eb, g5_2, o8_5);
            }
            { const float eb = bi[27];
              o9_4 = fmaf(eb, g4_0, o9_4);
              o9_5 = fmaf(eb, g5_0, o9_5);
            }
            { const float eb = bi[28];
              o9_4 = fmaf(eb, g4_2, o9_4);
              o9_5 = fmaf(eb, g5_2, o9_5);
            }
            { const float eb = bi[29];
              o9_4 = fmaf(eb, g4_3, o9_4);
              o9_5 = fmaf(eb, g5_3, o9_5);
            }
            { const float eb = bi[30];
              o9_4 = fmaf(eb, g4_8, o9_4);
              o9_5 = fmaf(eb, g5_8, o9_5);
            }
            { const float eb = bi[31];
              o10_4 = fmaf(eb, g4_0, o10_4);
              o10_5 = fmaf(eb, g5_0, o10_5);
            }
            { const float eb = bi[32];
              o10_4 = fmaf(eb, g4_2, o10_4);
              o10_5 = fmaf(eb, g5_2, o10_5);
            }
            { const float eb = bi[33];
              o10_4 = fmaf(eb, g4_6, o10_4);
              o10_5 = fmaf(eb, g5_6, o10_5);
            }
            { const float eb = bi[34];
              o11_4 = fmaf(eb, g4_0, o11_4);
              o11_5 = fmaf(eb, g5_0, o11_5);
            }
            { const float eb = bi[35];
              o11_4 = fmaf(eb, g4_1, o11_4);
              o11_5 = fmaf(eb, g5_1, o11_5);
            }
            { const float eb = bi[36];
              o11_4 = fmaf(eb, g4_2, o11_4);
              o11_5 = fmaf(eb, g5_2, o11_5);
            }
            { const float eb = bi[37];
              o11_4 = fmaf(eb, g4_5, o11_4);
              o11_5 = fmaf(eb, g5_5, o11_5);
            }
            { const float eb = bi[38];
              o12_4 = fmaf(eb, g4_0, o12_4);
              o12_5 = fmaf(eb, g5_0, o12_5);
            }
            { const float eb = bi[39];
              o12_4 = fmaf(eb, g4_1, o12_4);
              o12_5 = fmaf(eb, g5_1, o12_5);
            }
            { const float eb = bi[40];
              o13_4 = fmaf(eb, g4_0, o13_4);
              o13_5 = fmaf(eb, g5_0, o13_5);
            }
            { const float eb = bi[41];
              o13_4 = fmaf(eb, g4_1, o13_4);
              o13_5 = fmaf(eb, g5_1, o13_5);
            }
            { const float eb = bi[42];
              o13_4 = fmaf(eb, g4_3, o13_4);
              o13_5 = fmaf(eb, g5_3, o13_5);
            }
            { const float eb = bi[43];
              o13_4 = fmaf(eb, g4_7, o13_4);
              o13_5 = fmaf(eb, g5_7, o13_5);
            }
            { const float eb = bi[44];
              o14_4 = fmaf(eb, g4_0, o14_4);
              o14_5 = fmaf(eb, g5_0, o14_5);
            }
            { const float eb = bi[45];
              o14_4 = fmaf(eb, g4_1, o14_4);
              o14_5 = fmaf(eb, g5_1, o14_5);
            }
            { const float eb = bi[46];
              o14_4 = fmaf(eb, g4_2, o14_4);
              o14_5 = fmaf(eb, g5_2, o14_5);
            }
            { const float eb = bi[47];
              o14_4 = fmaf(eb, g4_5, o14_4);
              o14_5 = fmaf(eb, g5_5, o14_5);
            }
            { const float eb = bi[48];
              o15_4 = fmaf(eb, g4_0, o15_4);
              o15_5 = fmaf(eb, g5_0, o15_5);
            }
            { const float eb = bi[49];
              o15_4 = fmaf(eb, g4_1, o15_4);
              o15_5 = fmaf(eb, g5_1, o15_5);
            }
            { const float eb = bi[50];
              o15_4 = fmaf(eb, g4_4, o15_4);
              o15_5 = fmaf(eb, g5_4, o15_5);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk4 = PT[(fI + 4) * N + fJ + 0];
            const double ptk5 = PT[(fI + 5) * N + fJ + 0];
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
            const double Abc0_4 = PA[(fQ + 0) * N + fI + 4];
            const double Abc0_5 = PA[(fQ + 0) * N + fI + 5];
            const double Abc1_4 = PA[(fQ + 1) * N + fI + 4];
            const double Abc1_5 = PA[(fQ + 1) * N + fI + 5];
            const double Abc2_4 = PA[(fQ + 2) * N + fI + 4];
            const double Abc2_5 = PA[(fQ + 2) * N + fI + 5];
            const double Abc3_4 = PA[(fQ + 3) * N + fI + 4];
            const double Abc3_5 = PA[(fQ + 3) * N + fI + 5];
            const double Aac0_4 = PA[(fP + 0) * N + fI + 4];
            const double Aac0_5 = PA[(fP + 0) * N + fI + 5];
            const double Aac1_4 = PA[(fP + 1) * N + fI + 4];
            const double Aac1_5 = PA[(fP + 1) * N + fI + 5];
            const double Aac2_4 = PA[(fP + 2) * N + fI + 4];
            const double Aac2_5 = PA[(fP + 2) * N + fI + 5];
            const double Aac3_4 = PA[(fP + 3) * N + fI + 4];
            const double Aac3_5 = PA[(fP + 3) * N + fI + 5];
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
            atomicAdd(Jacc + (fI + 4) * N + fJ + 0, 2.0 * deg * (o0_4 * ptb0 + o1_4 * ptb1 + o2_4 * ptb2 + o3_4 * ptb3 + o4_4 * ptb4 + o5_4 * ptb5 + o6_4 * ptb6 + o7_4 * ptb7 + o8_4 * ptb8 + o9_4 * ptb9 + o10_4 * ptb10 + o11_4 * ptb11 + o12_4 * ptb12 + o13_4 * ptb13 + o14_4 * ptb14 + o15_4 * ptb15));
            atomicAdd(Jacc + (fI + 5) * N + fJ + 0, 2.0 * deg * (o0_5 * ptb0 + o1_5 * ptb1 + o2_5 * ptb2 + o3_5 * ptb3 + o4_5 * ptb4 + o5_5 * ptb5 + o6_5 * ptb6 + o7_5 * ptb7 + o8_5 * ptb8 + o9_5 * ptb9 + o10_5 * ptb10 + o11_5 * ptb11 + o12_5 * ptb12 + o13_5 * ptb13 + o14_5 * ptb14 + o15_5 * ptb15));
            atomicAdd(KAacc + (fP + 0) * N + fI + 4, deg * (o0_4 * Abd0_0 + o1_4 * Abd1_0 + o2_4 * Abd2_0 + o3_4 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 4, deg * (o0_4 * Aad0_0 + o4_4 * Aad1_0 + o8_4 * Aad2_0 + o12_4 * Aad3_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Abc0_4 + o0_5 * Abc0_5 + o1_4 * Abc1_4 + o1_5 * Abc1_5 + o2_4 * Abc2_4 + o2_5 * Abc2_5 + o3_4 * Abc3_4 + o3_5 * Abc3_5));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Aac0_4 + o0_5 * Aac0_5 + o4_4 * Aac1_4 + o4_5 * Aac1_5 + o8_4 * Aac2_4 + o8_5 * Aac2_5 + o12_4 * Aac3_4 + o12_5 * Aac3_5));
            atomicAdd(KAacc + (fP + 0) * N + fI + 5, deg * (o0_5 * Abd0_0 + o1_5 * Abd1_0 + o2_5 * Abd2_0 + o3_5 * Abd3_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 5, deg * (o0_5 * Aad0_0 + o4_5 * Aad1_0 + o8_5 * Aad2_0 + o12_5 * Aad3_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 4, deg * (o1_4 * Aad0_0 + o5_4 * Aad1_0 + o9_4 * Aad2_0 + o13_4 * Aad3_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Aac0_4 + o1_5 * Aac0_5 + o5_4 * Aac1_4 + o5_5 * Aac1_5 + o9_4 * Aac2_4 + o9_5 * Aac2_5 + o13_4 * Aac3_4 + o13_5 * Aac3_5));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 5, deg * (o1_5 * Aad0_0 + o5_5 * Aad1_0 + o9_5 * Aad2_0 + o13_5 * Aad3_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 4, deg * (o2_4 * Aad0_0 + o6_4 * Aad1_0 + o10_4 * Aad2_0 + o14_4 * Aad3_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Aac0_4 + o2_5 * Aac0_5 + o6_4 * Aac1_4 + o6_5 * Aac1_5 + o10_4 * Aac2_4 + o10_5 * Aac2_5 + o14_4 * Aac3_4 + o14_5 * Aac3_5));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 5, deg * (o2_5 * Aad0_0 + o6_5 * Aad1_0 + o10_5 * Aad2_0 + o14_5 * Aad3_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 4, deg * (o3_4 * Aad0_0 + o7_4 * Aad1_0 + o11_4 * Aad2_0 + o15_4 * Aad3_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Aac0_4 + o3_5 * Aac0_5 + o7_4 * Aac1_4 + o7_5 * Aac1_5 + o11_4 * Aac2_4 + o11_5 * Aac2_5 + o15_4 * Aac3_4 + o15_5 * Aac3_5));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 5, deg * (o3_5 * Aad0_0 + o7_5 * Aad1_0 + o11_5 * Aad2_0 + o15_5 * Aad3_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 4, deg * (o4_4 * Abd0_0 + o5_4 * Abd1_0 + o6_4 * Abd2_0 + o7_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o4_4 * Abc0_4 + o4_5 * Abc0_5 + o5_4 * Abc1_4 + o5_5 * Abc1_5 + o6_4 * Abc2_4 + o6_5 * Abc2_5 + o7_4 * Abc3_4 + o7_5 * Abc3_5));
            atomicAdd(KAacc + (fP + 1) * N + fI + 5, deg * (o4_5 * Abd0_0 + o5_5 * Abd1_0 + o6_5 * Abd2_0 + o7_5 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 4, deg * (o8_4 * Abd0_0 + o9_4 * Abd1_0 + o10_4 * Abd2_0 + o11_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o8_4 * Abc0_4 + o8_5 * Abc0_5 + o9_4 * Abc1_4 + o9_5 * Abc1_5 + o10_4 * Abc2_4 + o10_5 * Abc2_5 + o11_4 * Abc3_4 + o11_5 * Abc3_5));
            atomicAdd(KAacc + (fP + 2) * N + fI + 5, deg * (o8_5 * Abd0_0 + o9_5 * Abd1_0 + o10_5 * Abd2_0 + o11_5 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 4, deg * (o12_4 * Abd0_0 + o13_4 * Abd1_0 + o14_4 * Abd2_0 + o15_4 * Abd3_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o12_4 * Abc0_4 + o12_5 * Abc0_5 + o13_4 * Abc1_4 + o13_5 * Abc1_5 + o14_4 * Abc2_4 + o14_5 * Abc2_5 + o15_4 * Abc3_4 + o15_5 * Abc3_5));
            atomicAdd(KAacc + (fP + 3) * N + fI + 5, deg * (o12_5 * Abd0_0 + o13_5 * Abd1_0 + o14_5 * Abd2_0 + o15_5 * Abd3_0));
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
