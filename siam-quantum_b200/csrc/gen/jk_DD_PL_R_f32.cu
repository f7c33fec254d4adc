// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DD_PL_R_f32(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 341; x += blockDim.x) sbra[x] = a.bra_prims_f[bp.poff + (long long)x * bp.kstride];
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
        const float* __restrict__ kprim = a.ket_prims_f + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
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
          float o16_0 = 0;
          float o17_0 = 0;
          float o18_0 = 0;
          float o19_0 = 0;
          float o20_0 = 0;
          float o21_0 = 0;
          float o22_0 = 0;
          float o23_0 = 0;
          float o24_0 = 0;
          float o25_0 = 0;
          float o26_0 = 0;
          float o27_0 = 0;
          float o28_0 = 0;
          float o29_0 = 0;
          float o30_0 = 0;
          float o31_0 = 0;
          float o32_0 = 0;
          float o33_0 = 0;
          float o34_0 = 0;
          float o35_0 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
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
            float g0_10 = 0;
            float g0_11 = 0;
            float g0_12 = 0;
            float g0_13 = 0;
            float g0_14 = 0;
            float g0_15 = 0;
            float g0_16 = 0;
            float g0_17 = 0;
            float g0_18 = 0;
            float g0_19 = 0;
            float g0_20 = 0;
            float g0_21 = 0;
            float g0_22 = 0;
            float g0_23 = 0;
            float g0_24 = 0;
            float g0_25 = 0;
            float g0_26 = 0;
            float g0_27 = 0;
            float g0_28 = 0;
            float g0_29 = 0;
            float g0_30 = 0;
            float g0_31 = 0;
            float g0_32 = 0;
            float g0_33 = 0;
            float g0_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              ++nprimq;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[6];
              sqb::boysf<5>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              const float ek0_0 = kj[5 * kS];
              const float ek0_1 = -kj[6 * kS];
              g0_0 = fmaf(ek0_0, b0, g0_0);
              const float r0_0_0_1 = Z * b1;
              g0_1 = fmaf(ek0_0, r0_0_0_1, g0_1);
              const float r0_0_1_0 = Y * b1;
              g0_2 = fmaf(ek0_0, r0_0_1_0, g0_2);
              const float r0_1_0_0 = X * b1;
              g0_3 = fmaf(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fmaf(ek0_1, r0_1_0_0, g0_0);
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
              g0_1 = fmaf(ek0_1, r0_1_0_1, g0_1);
              const float r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fmaf(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fmaf(ek0_1, r0_1_1_0, g0_2);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g0_9 = fmaf(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fmaf(ek0_1, r0_2_0_0, g0_3);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g0_10 = fmaf(ek0_0, r0_0_0_3, g0_10);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g0_11 = fmaf(ek0_0, r0_0_1_2, g0_11);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g0_12 = fmaf(ek0_0, r0_0_2_1, g0_12);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g0_13 = fmaf(ek0_0, r0_0_3_0, g0_13);
              const float r0_1_0_2 = X * r1_0_0_2;
              g0_14 = fmaf(ek0_0, r0_1_0_2, g0_14);
              g0_4 = fmaf(ek0_1, r0_1_0_2, g0_4);
              const float r0_1_1_1 = X * r1_0_1_1;
              g0_15 = fmaf(ek0_0, r0_1_1_1, g0_15);
              g0_5 = fmaf(ek0_1, r0_1_1_1, g0_5);
              const float r0_1_2_0 = X * r1_0_2_0;
              g0_16 = fmaf(ek0_0, r0_1_2_0, g0_16);
              g0_6 = fmaf(ek0_1, r0_1_2_0, g0_6);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g0_17 = fmaf(ek0_0, r0_2_0_1, g0_17);
              g0_7 = fmaf(ek0_1, r0_2_0_1, g0_7);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g0_18 = fmaf(ek0_0, r0_2_1_0, g0_18);
              g0_8 = fmaf(ek0_1, r0_2_1_0, g0_8);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g0_19 = fmaf(ek0_0, r0_3_0_0, g0_19);
              g0_9 = fmaf(ek0_1, r0_3_0_0, g0_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g0_20 = fmaf(ek0_0, r0_0_0_4, g0_20);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g0_21 = fmaf(ek0_0, r0_0_1_3, g0_21);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g0_22 = fmaf(ek0_0, r0_0_2_2, g0_22);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g0_23 = fmaf(ek0_0, r0_0_3_1, g0_23);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g0_24 = fmaf(ek0_0, r0_0_4_0, g0_24);
              const float r0_1_0_3 = X * r1_0_0_3;
              g0_25 = fmaf(ek0_0, r0_1_0_3, g0_25);
              g0_10 = fmaf(ek0_1, r0_1_0_3, g0_10);
              const float r0_1_1_2 = X * r1_0_1_2;
              g0_26 = fmaf(ek0_0, r0_1_1_2, g0_26);
              g0_11 = fmaf(ek0_1, r0_1_1_2, g0_11);
              const float r0_1_2_1 = X * r1_0_2_1;
              g0_27 = fmaf(ek0_0, r0_1_2_1, g0_27);
              g0_12 = fmaf(ek0_1, r0_1_2_1, g0_12);
              const float r0_1_3_0 = X * r1_0_3_0;
              g0_28 = fmaf(ek0_0, r0_1_3_0, g0_28);
              g0_13 = fmaf(ek0_1, r0_1_3_0, g0_13);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g0_29 = fmaf(ek0_0, r0_2_0_2, g0_29);
              g0_14 = fmaf(ek0_1, r0_2_0_2, g0_14);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g0_30 = fmaf(ek0_0, r0_2_1_1, g0_30);
              g0_15 = fmaf(ek0_1, r0_2_1_1, g0_15);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g0_31 = fmaf(ek0_0, r0_2_2_0, g0_31);
              g0_16 = fmaf(ek0_1, r0_2_2_0, g0_16);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g0_32 = fmaf(ek0_0, r0_3_0_1, g0_32);
              g0_17 = fmaf(ek0_1, r0_3_0_1, g0_17);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g0_33 = fmaf(ek0_0, r0_3_1_0, g0_33);
              g0_18 = fmaf(ek0_1, r0_3_1_0, g0_18);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g0_34 = fmaf(ek0_0, r0_4_0_0, g0_34);
              g0_19 = fmaf(ek0_1, r0_4_0_0, g0_19);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_1_0_4 = X * r1_0_0_4;
              g0_20 = fmaf(ek0_1, r0_1_0_4, g0_20);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_1_1_3 = X * r1_0_1_3;
              g0_21 = fmaf(ek0_1, r0_1_1_3, g0_21);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_1_2_2 = X * r1_0_2_2;
              g0_22 = fmaf(ek0_1, r0_1_2_2, g0_22);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_1_3_1 = X * r1_0_3_1;
              g0_23 = fmaf(ek0_1, r0_1_3_1, g0_23);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_1_4_0 = X * r1_0_4_0;
              g0_24 = fmaf(ek0_1, r0_1_4_0, g0_24);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g0_25 = fmaf(ek0_1, r0_2_0_3, g0_25);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g0_26 = fmaf(ek0_1, r0_2_1_2, g0_26);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g0_27 = fmaf(ek0_1, r0_2_2_1, g0_27);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g0_28 = fmaf(ek0_1, r0_2_3_0, g0_28);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g0_29 = fmaf(ek0_1, r0_3_0_2, g0_29);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g0_30 = fmaf(ek0_1, r0_3_1_1, g0_30);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g0_31 = fmaf(ek0_1, r0_3_2_0, g0_31);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g0_32 = fmaf(ek0_1, r0_4_0_1, g0_32);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g0_33 = fmaf(ek0_1, r0_4_1_0, g0_33);
              const float r4_1_0_0 = X * b5;
              const float r3_2_0_0 = fmaf(X, r4_1_0_0, b4);
              const float r2_3_0_0 = fmaf(X, r3_2_0_0, 2.0f * r3_1_0_0);
              const float r1_4_0_0 = fmaf(X, r2_3_0_0, 3.0f * r2_2_0_0);
              const float r0_5_0_0 = fmaf(X, r1_4_0_0, 4.0f * r1_3_0_0);
              g0_34 = fmaf(ek0_1, r0_5_0_0, g0_34);
            }
            { const float eb = bi[5];
              o0_0 = fmaf(eb, g0_0, o0_0);
            }
            { const float eb = bi[6];
              o0_0 = fmaf(eb, g0_3, o0_0);
            }
            { const float eb = bi[7];
              o0_0 = fmaf(eb, g0_9, o0_0);
            }
            { const float eb = bi[8];
              o0_0 = fmaf(eb, g0_19, o0_0);
            }
            { const float eb = bi[9];
              o0_0 = fmaf(eb, g0_34, o0_0);
            }
            { const float eb = bi[10];
              o1_0 = fmaf(eb, g0_0, o1_0);
            }
            { const float eb = bi[11];
              o1_0 = fmaf(eb, g0_2, o1_0);
            }
            { const float eb = bi[12];
              o1_0 = fmaf(eb, g0_6, o1_0);
            }
            { const float eb = bi[13];
              o1_0 = fmaf(eb, g0_3, o1_0);
            }
            { const float eb = bi[14];
              o1_0 = fmaf(eb, g0_8, o1_0);
            }
            { const float eb = bi[15];
              o1_0 = fmaf(eb, g0_16, o1_0);
            }
            { const float eb = bi[16];
              o1_0 = fmaf(eb, g0_9, o1_0);
            }
            { const float eb = bi[17];
              o1_0 = fmaf(eb, g0_18, o1_0);
            }
            { const float eb = bi[18];
              o1_0 = fmaf(eb, g0_31, o1_0);
            }
            { const float eb = bi[19];
              o2_0 = fmaf(eb, g0_0, o2_0);
            }
            { const float eb = bi[20];
              o2_0 = fmaf(eb, g0_1, o2_0);
            }
            { const float eb = bi[21];
              o2_0 = fmaf(eb, g0_4, o2_0);
            }
            { const float eb = bi[22];
              o2_0 = fmaf(eb, g0_3, o2_0);
            }
            { const float eb = bi[23];
              o2_0 = fmaf(eb, g0_7, o2_0);
            }
            { const float eb = bi[24];
              o2_0 = fmaf(eb, g0_14, o2_0);
            }
            { const float eb = bi[25];
              o2_0 = fmaf(eb, g0_9, o2_0);
            }
            { const float eb = bi[26];
              o2_0 = fmaf(eb, g0_17, o2_0);
            }
            { const float eb = bi[27];
              o2_0 = fmaf(eb, g0_29, o2_0);
            }
            { const float eb = bi[28];
              o3_0 = fmaf(eb, g0_0, o3_0);
            }
            { const float eb = bi[29];
              o3_0 = fmaf(eb, g0_2, o3_0);
            }
            { const float eb = bi[30];
              o3_0 = fmaf(eb, g0_3, o3_0);
            }
            { const float eb = bi[31];
              o3_0 = fmaf(eb, g0_8, o3_0);
            }
            { const float eb = bi[32];
              o3_0 = fmaf(eb, g0_9, o3_0);
            }
            { const float eb = bi[33];
              o3_0 = fmaf(eb, g0_18, o3_0);
            }
            { const float eb = bi[34];
              o3_0 = fmaf(eb, g0_19, o3_0);
            }
            { const float eb = bi[35];
              o3_0 = fmaf(eb, g0_33, o3_0);
            }
            { const float eb = bi[36];
              o4_0 = fmaf(eb, g0_0, o4_0);
            }
            { const float eb = bi[37];
              o4_0 = fmaf(eb, g0_1, o4_0);
            }
            { const float eb = bi[38];
              o4_0 = fmaf(eb, g0_3, o4_0);
            }
            { const float eb = bi[39];
              o4_0 = fmaf(eb, g0_7, o4_0);
            }
            { const float eb = bi[40];
              o4_0 = fmaf(eb, g0_9, o4_0);
            }
            { const float eb = bi[41];
              o4_0 = fmaf(eb, g0_17, o4_0);
            }
            { const float eb = bi[42];
              o4_0 = fmaf(eb, g0_19, o4_0);
            }
            { const float eb = bi[43];
              o4_0 = fmaf(eb, g0_32, o4_0);
            }
            { const float eb = bi[44];
              o5_0 = fmaf(eb, g0_0, o5_0);
            }
            { const float eb = bi[45];
              o5_0 = fmaf(eb, g0_1, o5_0);
            }
            { const float eb = bi[46];
              o5_0 = fmaf(eb, g0_2, o5_0);
            }
            { const float eb = bi[47];
              o5_0 = fmaf(eb, g0_5, o5_0);
            }
            { const float eb = bi[48];
              o5_0 = fmaf(eb, g0_3, o5_0);
            }
            { const float eb = bi[49];
              o5_0 = fmaf(eb, g0_7, o5_0);
            }
            { const float eb = bi[50];
              o5_0 = fmaf(eb, g0_8, o5_0);
            }
            { const float eb = bi[51];
              o5_0 = fmaf(eb, g0_15, o5_0);
            }
            { const float eb = bi[52];
              o5_0 = fmaf(eb, g0_9, o5_0);
            }
            { const float eb = bi[53];
              o5_0 = fmaf(eb, g0_17, o5_0);
            }
            { const float eb = bi[54];
              o5_0 = fmaf(eb, g0_18, o5_0);
            }
            { const float eb = bi[55];
              o5_0 = fmaf(eb, g0_30, o5_0);
            }
            { const float eb = bi[56];
              o6_0 = fmaf(eb, g0_0, o6_0);
            }
            { const float eb = bi[57];
              o6_0 = fmaf(eb, g0_2, o6_0);
            }
            { const float eb = bi[58];
              o6_0 = fmaf(eb, g0_6, o6_0);
            }
            { const float eb = bi[59];
              o6_0 = fmaf(eb, g0_3, o6_0);
            }
            { const float eb = bi[60];
              o6_0 = fmaf(eb, g0_8, o6_0);
            }
            { const float eb = bi[61];
              o6_0 = fmaf(eb, g0_16, o6_0);
            }
            { const float eb = bi[62];
              o6_0 = fmaf(eb, g0_9, o6_0);
            }
            { const float eb = bi[63];
              o6_0 = fmaf(eb, g0_18, o6_0);
            }
            { const float eb = bi[64];
              o6_0 = fmaf(eb, g0_31, o6_0);
            }
            { const float eb = bi[65];
              o7_0 = fmaf(eb, g0_0, o7_0);
            }
            { const float eb = bi[66];
              o7_0 = fmaf(eb, g0_2, o7_0);
            }
            { const float eb = bi[67];
              o7_0 = fmaf(eb, g0_6, o7_0);
            }
            { const float eb = bi[68];
              o7_0 = fmaf(eb, g0_13, o7_0);
            }
            { const float eb = bi[69];
              o7_0 = fmaf(eb, g0_24, o7_0);
            }
            { const float eb = bi[70];
              o8_0 = fmaf(eb, g0_0, o8_0);
            }
            { const float eb = bi[71];
              o8_0 = fmaf(eb, g0_1, o8_0);
            }
            { const float eb = bi[72];
              o8_0 = fmaf(eb, g0_4, o8_0);
            }
            { const float eb = bi[73];
              o8_0 = fmaf(eb, g0_2, o8_0);
            }
            { const float eb = bi[74];
              o8_0 = fmaf(eb, g0_5, o8_0);
            }
            { const float eb = bi[75];
              o8_0 = fmaf(eb, g0_11, o8_0);
            }
            { const float eb = bi[76];
              o8_0 = fmaf(eb, g0_6, o8_0);
            }
            { const float eb = bi[77];
              o8_0 = fmaf(eb, g0_12, o8_0);
            }
            { const float eb = bi[78];
              o8_0 = fmaf(eb, g0_22, o8_0);
            }
            { const float eb = bi[79];
              o9_0 = fmaf(eb, g0_0, o9_0);
            }
            { const float eb = bi[80];
              o9_0 = fmaf(eb, g0_2, o9_0);
            }
            { const float eb = bi[81];
              o9_0 = fmaf(eb, g0_6, o9_0);
            }
            { const float eb = bi[82];
              o9_0 = fmaf(eb, g0_13, o9_0);
            }
            { const float eb = bi[83];
              o9_0 = fmaf(eb, g0_3, o9_0);
            }
            { const float eb = bi[84];
              o9_0 = fmaf(eb, g0_8, o9_0);
            }
            { const float eb = bi[85];
              o9_0 = fmaf(eb, g0_16, o9_0);
            }
            { const float eb = bi[86];
              o9_0 = fmaf(eb, g0_28, o9_0);
            }
            { const float eb = bi[87];
              o10_0 = fmaf(eb, g0_0, o10_0);
            }
            { const float eb = bi[88];
              o10_0 = fmaf(eb, g0_1, o10_0);
            }
            { const float eb = bi[89];
              o10_0 = fmaf(eb, g0_2, o10_0);
            }
            { const float eb = bi[90];
              o10_0 = fmaf(eb, g0_5, o10_0);
            }
            { const float eb = bi[91];
              o10_0 = fmaf(eb, g0_6, o10_0);
            }
            { const float eb = bi[92];
              o10_0 = fmaf(eb, g0_12, o10_0);
            }
            { const float eb = bi[93];
              o10_0 = fmaf(eb, g0_3, o10_0);
            }
            { const float eb = bi[94];
              o10_0 = fmaf(eb, g0_7, o10_0);
            }
            { const float eb = bi[95];
              o10_0 = fmaf(eb, g0_8, o10_0);
            }
            { const float eb = bi[96];
              o10_0 = fmaf(eb, g0_15, o10_0);
            }
            { const float eb = bi[97];
              o10_0 = fmaf(eb, g0_16, o10_0);
            }
            { const float eb = bi[98];
              o10_0 = fmaf(eb, g0_27, o10_0);
            }
            { const float eb = bi[99];
              o11_0 = fmaf(eb, g0_0, o11_0);
            }
            { const float eb = bi[100];
              o11_0 = fmaf(eb, g0_1, o11_0);
            }
            { const float eb = bi[101];
              o11_0 = fmaf(eb, g0_2, o11_0);
            }
            { const float eb = bi[102];
              o11_0 = fmaf(eb, g0_5, o11_0);
            }
            { const float eb = bi[103];
              o11_0 = fmaf(eb, g0_6, o11_0);
            }
            { const float eb = bi[104];
              o11_0 = fmaf(eb, g0_12, o11_0);
            }
            { const float eb = bi[105];
              o11_0 = fmaf(eb, g0_13, o11_0);
            }
            { const float eb = bi[106];
              o11_0 = fmaf(eb, g0_23, o11_0);
            }
            { const float eb = bi[107];
              o12_0 = fmaf(eb, g0_0, o12_0);
            }
            { const float eb = bi[108];
              o12_0 = fmaf(eb, g0_1, o12_0);
            }
            { const float eb = bi[109];
              o12_0 = fmaf(eb, g0_4, o12_0);
            }
            { const float eb = bi[110];
              o12_0 = fmaf(eb, g0_3, o12_0);
            }
            { const float eb = bi[111];
              o12_0 = fmaf(eb, g0_7, o12_0);
            }
            { const float eb = bi[112];
              o12_0 = fmaf(eb, g0_14, o12_0);
            }
            { const float eb = bi[113];
              o12_0 = fmaf(eb, g0_9, o12_0);
            }
            { const float eb = bi[114];
              o12_0 = fmaf(eb, g0_17, o12_0);
            }
            { const float eb = bi[115];
              o12_0 = fmaf(eb, g0_29, o12_0);
            }
            { const float eb = bi[116];
              o13_0 = fmaf(eb, g0_0, o13_0);
            }
            { const float eb = bi[117];
              o13_0 = fmaf(eb, g0_1, o13_0);
            }
            { const float eb = bi[118];
              o13_0 = fmaf(eb, g0_4, o13_0);
            }
            { const float eb = bi[119];
              o13_0 = fmaf(eb, g0_2, o13_0);
            }
            { const float eb = bi[120];
              o13_0 = fmaf(eb, g0_5, o13_0);
            }
            { const float eb = bi[121];
              o13_0 = fmaf(eb, g0_11, o13_0);
            }
            { const float eb = bi[122];
              o13_0 = fmaf(eb, g0_6, o13_0);
            }
            { const float eb = bi[123];
              o13_0 = fmaf(eb, g0_12, o13_0);
            }
            { const float eb = bi[124];
              o13_0 = fmaf(eb, g0_22, o13_0);
            }
            { const float eb = bi[125];
              o14_0 = fmaf(eb, g0_0, o14_0);
            }
            { const float eb = bi[126];
              o14_0 = fmaf(eb, g0_1, o14_0);
            }
            { const float eb = bi[127];
              o14_0 = fmaf(eb, g0_4, o14_0);
            }
            { const float eb = bi[128];
              o14_0 = fmaf(eb, g0_10, o14_0);
            }
            { const float eb = bi[129];
              o14_0 = fmaf(eb, g0_20, o14_0);
            }
            { const float eb = bi[130];
              o15_0 = fmaf(eb, g0_0, o15_0);
            }
            { const float eb = bi[131];
              o15_0 = fmaf(eb, g0_1, o15_0);
            }
            { const float eb = bi[132];
              o15_0 = fmaf(eb, g0_4, o15_0);
            }
            { const float eb = bi[133];
              o15_0 = fmaf(eb, g0_2, o15_0);
            }
            { const float eb = bi[134];
              o15_0 = fmaf(eb, g0_5, o15_0);
            }
            { const float eb = bi[135];
              o15_0 = fmaf(eb, g0_11, o15_0);
            }
            { const float eb = bi[136];
              o15_0 = fmaf(eb, g0_3, o15_0);
            }
            { const float eb = bi[137];
              o15_0 = fmaf(eb, g0_7, o15_0);
            }
            { const float eb = bi[138];
              o15_0 = fmaf(eb, g0_14, o15_0);
            }
            { const float eb = bi[139];
              o15_0 = fmaf(eb, g0_8, o15_0);
            }
            { const float eb = bi[140];
              o15_0 = fmaf(eb, g0_15, o15_0);
            }
            { const float eb = bi[141];
              o15_0 = fmaf(eb, g0_26, o15_0);
            }
            { const float eb = bi[142];
              o16_0 = fmaf(eb, g0_0, o16_0);
            }
            { const float eb = bi[143];
              o16_0 = fmaf(eb, g0_1, o16_0);
            }
            { const float eb = bi[144];
              o16_0 = fmaf(eb, g0_4, o16_0);
            }
            { const float eb = bi[145];
              o16_0 = fmaf(eb, g0_10, o16_0);
            }
            { const float eb = bi[146];
              o16_0 = fmaf(eb, g0_3, o16_0);
            }
            { const float eb = bi[147];
              o16_0 = fmaf(eb, g0_7, o16_0);
            }
            { const float eb = bi[148];
              o16_0 = fmaf(eb, g0_14, o16_0);
            }
            { const float eb = bi[149];
              o16_0 = fmaf(eb, g0_25, o16_0);
            }
            { const float eb = bi[150];
              o17_0 = fmaf(eb, g0_0, o17_0);
            }
            { const float eb = bi[151];
              o17_0 = fmaf(eb, g0_1, o17_0);
            }
            { const float eb = bi[152];
              o17_0 = fmaf(eb, g0_4, o17_0);
            }
            { const float eb = bi[153];
              o17_0 = fmaf(eb, g0_10, o17_0);
            }
            { const float eb = bi[154];
              o17_0 = fmaf(eb, g0_2, o17_0);
            }
            { const float eb = bi[155];
              o17_0 = fmaf(eb, g0_5, o17_0);
            }
            { const float eb = bi[156];
              o17_0 = fmaf(eb, g0_11, o17_0);
            }
            { const float eb = bi[157];
              o17_0 = fmaf(eb, g0_21, o17_0);
            }
            { const float eb = bi[158];
              o18_0 = fmaf(eb, g0_0, o18_0);
            }
            { const float eb = bi[159];
              o18_0 = fmaf(eb, g0_2, o18_0);
            }
            { const float eb = bi[160];
              o18_0 = fmaf(eb, g0_3, o18_0);
            }
            { const float eb = bi[161];
              o18_0 = fmaf(eb, g0_8, o18_0);
            }
            { const float eb = bi[162];
              o18_0 = fmaf(eb, g0_9, o18_0);
            }
            { const float eb = bi[163];
              o18_0 = fmaf(eb, g0_18, o18_0);
            }
            { const float eb = bi[164];
              o18_0 = fmaf(eb, g0_19, o18_0);
            }
            { const float eb = bi[165];
              o18_0 = fmaf(eb, g0_33, o18_0);
            }
            { const float eb = bi[166];
              o19_0 = fmaf(eb, g0_0, o19_0);
            }
            { const float eb = bi[167];
              o19_0 = fmaf(eb, g0_2, o19_0);
            }
            { const float eb = bi[168];
              o19_0 = fmaf(eb, g0_6, o19_0);
            }
            { const float eb = bi[169];
              o19_0 = fmaf(eb, g0_13, o19_0);
            }
            { const float eb = bi[170];
              o19_0 = fmaf(eb, g0_3, o19_0);
            }
            { const float eb = bi[171];
              o19_0 = fmaf(eb, g0_8, o19_0);
            }
            { const float eb = bi[172];
              o19_0 = fmaf(eb, g0_16, o19_0);
            }
            { const float eb = bi[173];
              o19_0 = fmaf(eb, g0_28, o19_0);
            }
            { const float eb = bi[174];
              o20_0 = fmaf(eb, g0_0, o20_0);
            }
            { const float eb = bi[175];
              o20_0 = fmaf(eb, g0_1, o20_0);
            }
            { const float eb = bi[176];
              o20_0 = fmaf(eb, g0_4, o20_0);
            }
            { const float eb = bi[177];
              o20_0 = fmaf(eb, g0_2, o20_0);
            }
            { const float eb = bi[178];
              o20_0 = fmaf(eb, g0_5, o20_0);
            }
            { const float eb = bi[179];
              o20_0 = fmaf(eb, g0_11, o20_0);
            }
            { const float eb = bi[180];
              o20_0 = fmaf(eb, g0_3, o20_0);
            }
            { const float eb = bi[181];
              o20_0 = fmaf(eb, g0_7, o20_0);
            }
            { const float eb = bi[182];
              o20_0 = fmaf(eb, g0_14, o20_0);
            }
            { const float eb = bi[183];
              o20_0 = fmaf(eb, g0_8, o20_0);
            }
            { const float eb = bi[184];
              o20_0 = fmaf(eb, g0_15, o20_0);
            }
            { const float eb = bi[185];
              o20_0 = fmaf(eb, g0_26, o20_0);
            }
            { const float eb = bi[186];
              o21_0 = fmaf(eb, g0_0, o21_0);
            }
            { const float eb = bi[187];
              o21_0 = fmaf(eb, g0_2, o21_0);
            }
            { const float eb = bi[188];
              o21_0 = fmaf(eb, g0_6, o21_0);
            }
            { const float eb = bi[189];
              o21_0 = fmaf(eb, g0_3, o21_0);
            }
            { const float eb = bi[190];
              o21_0 = fmaf(eb, g0_8, o21_0);
            }
            { const float eb = bi[191];
              o21_0 = fmaf(eb, g0_16, o21_0);
            }
            { const float eb = bi[192];
              o21_0 = fmaf(eb, g0_9, o21_0);
            }
            { const float eb = bi[193];
              o21_0 = fmaf(eb, g0_18, o21_0);
            }
            { const float eb = bi[194];
              o21_0 = fmaf(eb, g0_31, o21_0);
            }
            { const float eb = bi[195];
              o22_0 = fmaf(eb, g0_0, o22_0);
            }
            { const float eb = bi[196];
              o22_0 = fmaf(eb, g0_1, o22_0);
            }
            { const float eb = bi[197];
              o22_0 = fmaf(eb, g0_2, o22_0);
            }
            { const float eb = bi[198];
              o22_0 = fmaf(eb, g0_5, o22_0);
            }
            { const float eb = bi[199];
              o22_0 = fmaf(eb, g0_3, o22_0);
            }
            { const float eb = bi[200];
              o22_0 = fmaf(eb, g0_7, o22_0);
            }
            { const float eb = bi[201];
              o22_0 = fmaf(eb, g0_8, o22_0);
            }
            { const float eb = bi[202];
              o22_0 = fmaf(eb, g0_15, o22_0);
            }
            { const float eb = bi[203];
              o22_0 = fmaf(eb, g0_9, o22_0);
            }
            { const float eb = bi[204];
              o22_0 = fmaf(eb, g0_17, o22_0);
            }
            { const float eb = bi[205];
              o22_0 = fmaf(eb, g0_18, o22_0);
            }
            { const float eb = bi[206];
              o22_0 = fmaf(eb, g0_30, o22_0);
            }
            { const float eb = bi[207];
              o23_0 = fmaf(eb, g0_0, o23_0);
            }
            { const float eb = bi[208];
              o23_0 = fmaf(eb, g0_1, o23_0);
            }
            { const float eb = bi[209];
              o23_0 = fmaf(eb, g0_2, o23_0);
            }
            { const float eb = bi[210];
              o23_0 = fmaf(eb, g0_5, o23_0);
            }
            { const float eb = bi[211];
              o23_0 = fmaf(eb, g0_6, o23_0);
            }
            { const float eb = bi[212];
              o23_0 = fmaf(eb, g0_12, o23_0);
            }
            { const float eb = bi[213];
              o23_0 = fmaf(eb, g0_3, o23_0);
            }
            { const float eb = bi[214];
              o23_0 = fmaf(eb, g0_7, o23_0);
            }
            { const float eb = bi[215];
              o23_0 = fmaf(eb, g0_8, o23_0);
            }
            { const float eb = bi[216];
              o23_0 = fmaf(eb, g0_15, o23_0);
            }
            { const float eb = bi[217];
              o23_0 = fmaf(eb, g0_16, o23_0);
            }
            { const float eb = bi[218];
              o23_0 = fmaf(eb, g0_27, o23_0);
            }
            { const float eb = bi[219];
              o24_0 = fmaf(eb, g0_0, o24_0);
            }
            { const float eb = bi[220];
              o24_0 = fmaf(eb, g0_1, o24_0);
            }
            { const float eb = bi[221];
              o24_0 = fmaf(eb, g0_3, o24_0);
            }
            { const float eb = bi[222];
              o24_0 = fmaf(eb, g0_7, o24_0);
            }
            { const float eb = bi[223];
              o24_0 = fmaf(eb, g0_9, o24_0);
            }
            { const float eb = bi[224];
              o24_0 = fmaf(eb, g0_17, o24_0);
            }
            { const float eb = bi[225];
              o24_0 = fmaf(eb, g0_19, o24_0);
            }
            { const float eb = bi[226];
              o24_0 = fmaf(eb, g0_32, o24_0);
            }
            { const float eb = bi[227];
              o25_0 = fmaf(eb, g0_0, o25_0);
            }
            { const float eb = bi[228];
              o25_0 = fmaf(eb, g0_1, o25_0);
            }
            { const float eb = bi[229];
              o25_0 = fmaf(eb, g0_2, o25_0);
            }
            { const float eb = bi[230];
              o25_0 = fmaf(eb, g0_5, o25_0);
            }
            { const float eb = bi[231];
              o25_0 = fmaf(eb, g0_6, o25_0);
            }
            { const float eb = bi[232];
              o25_0 = fmaf(eb, g0_12, o25_0);
            }
            { const float eb = bi[233];
              o25_0 = fmaf(eb, g0_3, o25_0);
            }
            { const float eb = bi[234];
              o25_0 = fmaf(eb, g0_7, o25_0);
            }
            { const float eb = bi[235];
              o25_0 = fmaf(eb, g0_8, o25_0);
            }
            { const float eb = bi[236];
              o25_0 = fmaf(eb, g0_15, o25_0);
            }
            { const float eb = bi[237];
              o25_0 = fmaf(eb, g0_16, o25_0);
            }
            { const float eb = bi[238];
              o25_0 = fmaf(eb, g0_27, o25_0);
            }
            { const float eb = bi[239];
              o26_0 = fmaf(eb, g0_0, o26_0);
            }
            { const float eb = bi[240];
              o26_0 = fmaf(eb, g0_1, o26_0);
            }
            { const float eb = bi[241];
              o26_0 = fmaf(eb, g0_4, o26_0);
            }
            { const float eb = bi[242];
              o26_0 = fmaf(eb, g0_10, o26_0);
            }
            { const float eb = bi[243];
              o26_0 = fmaf(eb, g0_3, o26_0);
            }
            { const float eb = bi[244];
              o26_0 = fmaf(eb, g0_7, o26_0);
            }
            { const float eb = bi[245];
              o26_0 = fmaf(eb, g0_14, o26_0);
            }
            { const float eb = bi[246];
              o26_0 = fmaf(eb, g0_25, o26_0);
            }
            { const float eb = bi[247];
              o27_0 = fmaf(eb, g0_0, o27_0);
            }
            { const float eb = bi[248];
              o27_0 = fmaf(eb, g0_1, o27_0);
            }
            { const float eb = bi[249];
              o27_0 = fmaf(eb, g0_2, o27_0);
            }
            { const float eb = bi[250];
              o27_0 = fmaf(eb, g0_5, o27_0);
            }
            { const float eb = bi[251];
              o27_0 = fmaf(eb, g0_3, o27_0);
            }
            { const float eb = bi[252];
              o27_0 = fmaf(eb, g0_7, o27_0);
            }
            { const float eb = bi[253];
              o27_0 = fmaf(eb, g0_8, o27_0);
            }
            { const float eb = bi[254];
              o27_0 = fmaf(eb, g0_15, o27_0);
            }
            { const float eb = bi[255];
              o27_0 = fmaf(eb, g0_9, o27_0);
            }
            { const float eb = bi[256];
              o27_0 = fmaf(eb, g0_17, o27_0);
            }
            { const float eb = bi[257];
              o27_0 = fmaf(eb, g0_18, o27_0);
            }
            { const float eb = bi[258];
              o27_0 = fmaf(eb, g0_30, o27_0);
            }
            { const float eb = bi[259];
              o28_0 = fmaf(eb, g0_0, o28_0);
            }
            { const float eb = bi[260];
              o28_0 = fmaf(eb, g0_1, o28_0);
            }
            { const float eb = bi[261];
              o28_0 = fmaf(eb, g0_4, o28_0);
            }
            { const float eb = bi[262];
              o28_0 = fmaf(eb, g0_3, o28_0);
            }
            { const float eb = bi[263];
              o28_0 = fmaf(eb, g0_7, o28_0);
            }
            { const float eb = bi[264];
              o28_0 = fmaf(eb, g0_14, o28_0);
            }
            { const float eb = bi[265];
              o28_0 = fmaf(eb, g0_9, o28_0);
            }
            { const float eb = bi[266];
              o28_0 = fmaf(eb, g0_17, o28_0);
            }
            { const float eb = bi[267];
              o28_0 = fmaf(eb, g0_29, o28_0);
            }
            { const float eb = bi[268];
              o29_0 = fmaf(eb, g0_0, o29_0);
            }
            { const float eb = bi[269];
              o29_0 = fmaf(eb, g0_1, o29_0);
            }
            { const float eb = bi[270];
              o29_0 = fmaf(eb, g0_4, o29_0);
            }
            { const float eb = bi[271];
              o29_0 = fmaf(eb, g0_2, o29_0);
            }
            { const float eb = bi[272];
              o29_0 = fmaf(eb, g0_5, o29_0);
            }
            { const float eb = bi[273];
              o29_0 = fmaf(eb, g0_11, o29_0);
            }
            { const float eb = bi[274];
              o29_0 = fmaf(eb, g0_3, o29_0);
            }
            { const float eb = bi[275];
              o29_0 = fmaf(eb, g0_7, o29_0);
            }
            { const float eb = bi[276];
              o29_0 = fmaf(eb, g0_14, o29_0);
            }
            { const float eb = bi[277];
              o29_0 = fmaf(eb, g0_8, o29_0);
            }
            { const float eb = bi[278];
              o29_0 = fmaf(eb, g0_15, o29_0);
            }
            { const float eb = bi[279];
              o29_0 = fmaf(eb, g0_26, o29_0);
            }
            { const float eb = bi[280];
              o30_0 = fmaf(eb, g0_0, o30_0);
            }
            { const float eb = bi[281];
              o30_0 = fmaf(eb, g0_1, o30_0);
            }
            { const float eb = bi[282];
              o30_0 = fmaf(eb, g0_2, o30_0);
            }
            { const float eb = bi[283];
              o30_0 = fmaf(eb, g0_5, o30_0);
            }
            { const float eb = bi[284];
              o30_0 = fmaf(eb, g0_3, o30_0);
            }
            { const float eb = bi[285];
              o30_0 = fmaf(eb, g0_7, o30_0);
            }
            { const float eb = bi[286];
              o30_0 = fmaf(eb, g0_8, o30_0);
            }
            { const float eb = bi[287];
              o30_0 = fmaf(eb, g0_15, o30_0);
            }
            { const float eb = bi[288];
              o30_0 = fmaf(eb, g0_9, o30_0);
            }
            { const float eb = bi[289];
              o30_0 = fmaf(eb, g0_17, o30_0);
            }
            { const float eb = bi[290];
              o30_0 = fmaf(eb, g0_18, o30_0);
            }
            { const float eb = bi[291];
              o30_0 = fmaf(eb, g0_30, o30_0);
            }
            { const float eb = bi[292];
              o31_0 = fmaf(eb, g0_0, o31_0);
            }
            { const float eb = bi[293];
              o31_0 = fmaf(eb, g0_1, o31_0);
            }
            { const float eb = bi[294];
              o31_0 = fmaf(eb, g0_2, o31_0);
            }
            { const float eb = bi[295];
              o31_0 = fmaf(eb, g0_5, o31_0);
            }
            { const float eb = bi[296];
              o31_0 = fmaf(eb, g0_6, o31_0);
            }
            { const float eb = bi[297];
              o31_0 = fmaf(eb, g0_12, o31_0);
            }
            { const float eb = bi[298];
              o31_0 = fmaf(eb, g0_13, o31_0);
            }
            { const float eb = bi[299];
              o31_0 = fmaf(eb, g0_23, o31_0);
            }
            { const float eb = bi[300];
              o32_0 = fmaf(eb, g0_0, o32_0);
            }
            { const float eb = bi[301];
              o32_0 = fmaf(eb, g0_1, o32_0);
            }
            { const float eb = bi[302];
              o32_0 = fmaf(eb, g0_4, o32_0);
            }
            { const float eb = bi[303];
              o32_0 = fmaf(eb, g0_10, o32_0);
            }
            { const float eb = bi[304];
              o32_0 = fmaf(eb, g0_2, o32_0);
            }
            { const float eb = bi[305];
              o32_0 = fmaf(eb, g0_5, o32_0);
            }
            { const float eb = bi[306];
              o32_0 = fmaf(eb, g0_11, o32_0);
            }
            { const float eb = bi[307];
              o32_0 = fmaf(eb, g0_21, o32_0);
            }
            { const float eb = bi[308];
              o33_0 = fmaf(eb, g0_0, o33_0);
            }
            { const float eb = bi[309];
              o33_0 = fmaf(eb, g0_1, o33_0);
            }
            { const float eb = bi[310];
              o33_0 = fmaf(eb, g0_2, o33_0);
            }
            { const float eb = bi[311];
              o33_0 = fmaf(eb, g0_5, o33_0);
            }
            { const float eb = bi[312];
              o33_0 = fmaf(eb, g0_6, o33_0);
            }
            { const float eb = bi[313];
              o33_0 = fmaf(eb, g0_12, o33_0);
            }
            { const float eb = bi[314];
              o33_0 = fmaf(eb, g0_3, o33_0);
            }
            { const float eb = bi[315];
              o33_0 = fmaf(eb, g0_7, o33_0);
            }
            { const float eb = bi[316];
              o33_0 = fmaf(eb, g0_8, o33_0);
            }
            { const float eb = bi[317];
              o33_0 = fmaf(eb, g0_15, o33_0);
            }
            { const float eb = bi[318];
              o33_0 = fmaf(eb, g0_16, o33_0);
            }
            { const float eb = bi[319];
              o33_0 = fmaf(eb, g0_27, o33_0);
            }
            { const float eb = bi[320];
              o34_0 = fmaf(eb, g0_0, o34_0);
            }
            { const float eb = bi[321];
              o34_0 = fmaf(eb, g0_1, o34_0);
            }
            { const float eb = bi[322];
              o34_0 = fmaf(eb, g0_4, o34_0);
            }
            { const float eb = bi[323];
              o34_0 = fmaf(eb, g0_2, o34_0);
            }
            { const float eb = bi[324];
              o34_0 = fmaf(eb, g0_5, o34_0);
            }
            { const float eb = bi[325];
              o34_0 = fmaf(eb, g0_11, o34_0);
            }
            { const float eb = bi[326];
              o34_0 = fmaf(eb, g0_3, o34_0);
            }
            { const float eb = bi[327];
              o34_0 = fmaf(eb, g0_7, o34_0);
            }
            { const float eb = bi[328];
              o34_0 = fmaf(eb, g0_14, o34_0);
            }
            { const float eb = bi[329];
              o34_0 = fmaf(eb, g0_8, o34_0);
            }
            { const float eb = bi[330];
              o34_0 = fmaf(eb, g0_15, o34_0);
            }
            { const float eb = bi[331];
              o34_0 = fmaf(eb, g0_26, o34_0);
            }
            { const float eb = bi[332];
              o35_0 = fmaf(eb, g0_0, o35_0);
            }
            { const float eb = bi[333];
              o35_0 = fmaf(eb, g0_1, o35_0);
            }
            { const float eb = bi[334];
              o35_0 = fmaf(eb, g0_4, o35_0);
            }
            { const float eb = bi[335];
              o35_0 = fmaf(eb, g0_2, o35_0);
            }
            { const float eb = bi[336];
              o35_0 = fmaf(eb, g0_5, o35_0);
            }
            { const float eb = bi[337];
              o35_0 = fmaf(eb, g0_11, o35_0);
            }
            { const float eb = bi[338];
              o35_0 = fmaf(eb, g0_6, o35_0);
            }
            { const float eb = bi[339];
              o35_0 = fmaf(eb, g0_12, o35_0);
            }
            { const float eb = bi[340];
              o35_0 = fmaf(eb, g0_22, o35_0);
            }
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
          }
        } break;
        case 1: {  // ket functions [1]
          float o0_1 = 0;
          float o1_1 = 0;
          float o2_1 = 0;
          float o3_1 = 0;
          float o4_1 = 0;
          float o5_1 = 0;
          float o6_1 = 0;
          float o7_1 = 0;
          float o8_1 = 0;
          float o9_1 = 0;
          float o10_1 = 0;
          float o11_1 = 0;
          float o12_1 = 0;
          float o13_1 = 0;
          float o14_1 = 0;
          float o15_1 = 0;
          float o16_1 = 0;
          float o17_1 = 0;
          float o18_1 = 0;
          float o19_1 = 0;
          float o20_1 = 0;
          float o21_1 = 0;
          float o22_1 = 0;
          float o23_1 = 0;
          float o24_1 = 0;
          float o25_1 = 0;
          float o26_1 = 0;
          float o27_1 = 0;
          float o28_1 = 0;
          float o29_1 = 0;
          float o30_1 = 0;
          float o31_1 = 0;
          float o32_1 = 0;
          float o33_1 = 0;
          float o34_1 = 0;
          float o35_1 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            float g1_10 = 0;
            float g1_11 = 0;
            float g1_12 = 0;
            float g1_13 = 0;
            float g1_14 = 0;
            float g1_15 = 0;
            float g1_16 = 0;
            float g1_17 = 0;
            float g1_18 = 0;
            float g1_19 = 0;
            float g1_20 = 0;
            float g1_21 = 0;
            float g1_22 = 0;
            float g1_23 = 0;
            float g1_24 = 0;
            float g1_25 = 0;
            float g1_26 = 0;
            float g1_27 = 0;
            float g1_28 = 0;
            float g1_29 = 0;
            float g1_30 = 0;
            float g1_31 = 0;
            float g1_32 = 0;
            float g1_33 = 0;
            float g1_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek1_0 = kj[7 * kS];
              const float ek1_1 = -kj[8 * kS];
              const float ek1_2 = kj[9 * kS];
              g1_0 = fmaf(ek1_0, b0, g1_0);
              const float r0_0_0_1 = Z * b1;
              g1_1 = fmaf(ek1_0, r0_0_0_1, g1_1);
              const float r0_0_1_0 = Y * b1;
              g1_2 = fmaf(ek1_0, r0_0_1_0, g1_2);
              const float r0_1_0_0 = X * b1;
              g1_3 = fmaf(ek1_0, r0_1_0_0, g1_3);
              g1_0 = fmaf(ek1_1, r0_1_0_0, g1_0);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g1_4 = fmaf(ek1_0, r0_0_0_2, g1_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g1_5 = fmaf(ek1_0, r0_0_1_1, g1_5);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g1_6 = fmaf(ek1_0, r0_0_2_0, g1_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g1_7 = fmaf(ek1_0, r0_1_0_1, g1_7);
              g1_1 = fmaf(ek1_1, r0_1_0_1, g1_1);
              const float r0_1_1_0 = X * r1_0_1_0;
              g1_8 = fmaf(ek1_0, r0_1_1_0, g1_8);
              g1_2 = fmaf(ek1_1, r0_1_1_0, g1_2);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g1_9 = fmaf(ek1_0, r0_2_0_0, g1_9);
              g1_3 = fmaf(ek1_1, r0_2_0_0, g1_3);
              g1_0 = fmaf(ek1_2, r0_2_0_0, g1_0);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g1_10 = fmaf(ek1_0, r0_0_0_3, g1_10);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g1_11 = fmaf(ek1_0, r0_0_1_2, g1_11);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g1_12 = fmaf(ek1_0, r0_0_2_1, g1_12);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g1_13 = fmaf(ek1_0, r0_0_3_0, g1_13);
              const float r0_1_0_2 = X * r1_0_0_2;
              g1_14 = fmaf(ek1_0, r0_1_0_2, g1_14);
              g1_4 = fmaf(ek1_1, r0_1_0_2, g1_4);
              const float r0_1_1_1 = X * r1_0_1_1;
              g1_15 = fmaf(ek1_0, r0_1_1_1, g1_15);
              g1_5 = fmaf(ek1_1, r0_1_1_1, g1_5);
              const float r0_1_2_0 = X * r1_0_2_0;
              g1_16 = fmaf(ek1_0, r0_1_2_0, g1_16);
              g1_6 = fmaf(ek1_1, r0_1_2_0, g1_6);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g1_17 = fmaf(ek1_0, r0_2_0_1, g1_17);
              g1_7 = fmaf(ek1_1, r0_2_0_1, g1_7);
              g1_1 = fmaf(ek1_2, r0_2_0_1, g1_1);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g1_18 = fmaf(ek1_0, r0_2_1_0, g1_18);
              g1_8 = fmaf(ek1_1, r0_2_1_0, g1_8);
              g1_2 = fmaf(ek1_2, r0_2_1_0, g1_2);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g1_19 = fmaf(ek1_0, r0_3_0_0, g1_19);
              g1_9 = fmaf(ek1_1, r0_3_0_0, g1_9);
              g1_3 = fmaf(ek1_2, r0_3_0_0, g1_3);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g1_20 = fmaf(ek1_0, r0_0_0_4, g1_20);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g1_21 = fmaf(ek1_0, r0_0_1_3, g1_21);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g1_22 = fmaf(ek1_0, r0_0_2_2, g1_22);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g1_23 = fmaf(ek1_0, r0_0_3_1, g1_23);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g1_24 = fmaf(ek1_0, r0_0_4_0, g1_24);
              const float r0_1_0_3 = X * r1_0_0_3;
              g1_25 = fmaf(ek1_0, r0_1_0_3, g1_25);
              g1_10 = fmaf(ek1_1, r0_1_0_3, g1_10);
              const float r0_1_1_2 = X * r1_0_1_2;
              g1_26 = fmaf(ek1_0, r0_1_1_2, g1_26);
              g1_11 = fmaf(ek1_1, r0_1_1_2, g1_11);
              const float r0_1_2_1 = X * r1_0_2_1;
              g1_27 = fmaf(ek1_0, r0_1_2_1, g1_27);
              g1_12 = fmaf(ek1_1, r0_1_2_1, g1_12);
              const float r0_1_3_0 = X * r1_0_3_0;
              g1_28 = fmaf(ek1_0, r0_1_3_0, g1_28);
              g1_13 = fmaf(ek1_1, r0_1_3_0, g1_13);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g1_29 = fmaf(ek1_0, r0_2_0_2, g1_29);
              g1_14 = fmaf(ek1_1, r0_2_0_2, g1_14);
              g1_4 = fmaf(ek1_2, r0_2_0_2, g1_4);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g1_30 = fmaf(ek1_0, r0_2_1_1, g1_30);
              g1_15 = fmaf(ek1_1, r0_2_1_1, g1_15);
              g1_5 = fmaf(ek1_2, r0_2_1_1, g1_5);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g1_31 = fmaf(ek1_0, r0_2_2_0, g1_31);
              g1_16 = fmaf(ek1_1, r0_2_2_0, g1_16);
              g1_6 = fmaf(ek1_2, r0_2_2_0, g1_6);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g1_32 = fmaf(ek1_0, r0_3_0_1, g1_32);
              g1_17 = fmaf(ek1_1, r0_3_0_1, g1_17);
              g1_7 = fmaf(ek1_2, r0_3_0_1, g1_7);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g1_33 = fmaf(ek1_0, r0_3_1_0, g1_33);
              g1_18 = fmaf(ek1_1, r0_3_1_0, g1_18);
              g1_8 = fmaf(ek1_2, r0_3_1_0, g1_8);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g1_34 = fmaf(ek1_0, r0_4_0_0, g1_34);
              g1_19 = fmaf(ek1_1, r0_4_0_0, g1_19);
              g1_9 = fmaf(ek1_2, r0_4_0_0, g1_9);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_1_0_4 = X * r1_0_0_4;
              g1_20 = fmaf(ek1_1, r0_1_0_4, g1_20);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_1_1_3 = X * r1_0_1_3;
              g1_21 = fmaf(ek1_1, r0_1_1_3, g1_21);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_1_2_2 = X * r1_0_2_2;
              g1_22 = fmaf(ek1_1, r0_1_2_2, g1_22);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_1_3_1 = X * r1_0_3_1;
              g1_23 = fmaf(ek1_1, r0_1_3_1, g1_23);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_1_4_0 = X * r1_0_4_0;
              g1_24 = fmaf(ek1_1, r0_1_4_0, g1_24);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g1_25 = fmaf(ek1_1, r0_2_0_3, g1_25);
              g1_10 = fmaf(ek1_2, r0_2_0_3, g1_10);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g1_26 = fmaf(ek1_1, r0_2_1_2, g1_26);
              g1_11 = fmaf(ek1_2, r0_2_1_2, g1_11);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g1_27 = fmaf(ek1_1, r0_2_2_1, g1_27);
              g1_12 = fmaf(ek1_2, r0_2_2_1, g1_12);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g1_28 = fmaf(ek1_1, r0_2_3_0, g1_28);
              g1_13 = fmaf(ek1_2, r0_2_3_0, g1_13);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g1_29 = fmaf(ek1_1, r0_3_0_2, g1_29);
              g1_14 = fmaf(ek1_2, r0_3_0_2, g1_14);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g1_30 = fmaf(ek1_1, r0_3_1_1, g1_30);
              g1_15 = fmaf(ek1_2, r0_3_1_1, g1_15);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g1_31 = fmaf(ek1_1, r0_3_2_0, g1_31);
              g1_16 = fmaf(ek1_2, r0_3_2_0, g1_16);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g1_32 = fmaf(ek1_1, r0_4_0_1, g1_32);
              g1_17 = fmaf(ek1_2, r0_4_0_1, g1_17);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g1_33 = fmaf(ek1_1, r0_4_1_0, g1_33);
              g1_18 = fmaf(ek1_2, r0_4_1_0, g1_18);
              const float r4_1_0_0 = X * b5;
              const float r3_2_0_0 = fmaf(X, r4_1_0_0, b4);
              const float r2_3_0_0 = fmaf(X, r3_2_0_0, 2.0f * r3_1_0_0);
              const float r1_4_0_0 = fmaf(X, r2_3_0_0, 3.0f * r2_2_0_0);
              const float r0_5_0_0 = fmaf(X, r1_4_0_0, 4.0f * r1_3_0_0);
              g1_34 = fmaf(ek1_1, r0_5_0_0, g1_34);
              g1_19 = fmaf(ek1_2, r0_5_0_0, g1_19);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_1_0_4 = X * r2_0_0_4;
              const float r0_2_0_4 = fmaf(X, r1_1_0_4, r1_0_0_4);
              g1_20 = fmaf(ek1_2, r0_2_0_4, g1_20);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g1_21 = fmaf(ek1_2, r0_2_1_3, g1_21);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g1_22 = fmaf(ek1_2, r0_2_2_2, g1_22);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g1_23 = fmaf(ek1_2, r0_2_3_1, g1_23);
              const float r5_0_1_0 = Y * b6;
              const float r4_0_2_0 = fmaf(Y, r5_0_1_0, b5);
              const float r3_0_3_0 = fmaf(Y, r4_0_2_0, 2.0f * r4_0_1_0);
              const float r2_0_4_0 = fmaf(Y, r3_0_3_0, 3.0f * r3_0_2_0);
              const float r1_1_4_0 = X * r2_0_4_0;
              const float r0_2_4_0 = fmaf(X, r1_1_4_0, r1_0_4_0);
              g1_24 = fmaf(ek1_2, r0_2_4_0, g1_24);
              const float r2_1_0_3 = X * r3_0_0_3;
              const float r1_2_0_3 = fmaf(X, r2_1_0_3, r2_0_0_3);
              const float r0_3_0_3 = fmaf(X, r1_2_0_3, 2.0f * r1_1_0_3);
              g1_25 = fmaf(ek1_2, r0_3_0_3, g1_25);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g1_26 = fmaf(ek1_2, r0_3_1_2, g1_26);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g1_27 = fmaf(ek1_2, r0_3_2_1, g1_27);
              const float r2_1_3_0 = X * r3_0_3_0;
              const float r1_2_3_0 = fmaf(X, r2_1_3_0, r2_0_3_0);
              const float r0_3_3_0 = fmaf(X, r1_2_3_0, 2.0f * r1_1_3_0);
              g1_28 = fmaf(ek1_2, r0_3_3_0, g1_28);
              const float r3_1_0_2 = X * r4_0_0_2;
              const float r2_2_0_2 = fmaf(X, r3_1_0_2, r3_0_0_2);
              const float r1_3_0_2 = fmaf(X, r2_2_0_2, 2.0f * r2_1_0_2);
              const float r0_4_0_2 = fmaf(X, r1_3_0_2, 3.0f * r1_2_0_2);
              g1_29 = fmaf(ek1_2, r0_4_0_2, g1_29);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g1_30 = fmaf(ek1_2, r0_4_1_1, g1_30);
              const float r3_1_2_0 = X * r4_0_2_0;
              const float r2_2_2_0 = fmaf(X, r3_1_2_0, r3_0_2_0);
              const float r1_3_2_0 = fmaf(X, r2_2_2_0, 2.0f * r2_1_2_0);
              const float r0_4_2_0 = fmaf(X, r1_3_2_0, 3.0f * r1_2_2_0);
              g1_31 = fmaf(ek1_2, r0_4_2_0, g1_31);
              const float r4_1_0_1 = X * r5_0_0_1;
              const float r3_2_0_1 = fmaf(X, r4_1_0_1, r4_0_0_1);
              const float r2_3_0_1 = fmaf(X, r3_2_0_1, 2.0f * r3_1_0_1);
              const float r1_4_0_1 = fmaf(X, r2_3_0_1, 3.0f * r2_2_0_1);
              const float r0_5_0_1 = fmaf(X, r1_4_0_1, 4.0f * r1_3_0_1);
              g1_32 = fmaf(ek1_2, r0_5_0_1, g1_32);
              const float r4_1_1_0 = X * r5_0_1_0;
              const float r3_2_1_0 = fmaf(X, r4_1_1_0, r4_0_1_0);
              const float r2_3_1_0 = fmaf(X, r3_2_1_0, 2.0f * r3_1_1_0);
              const float r1_4_1_0 = fmaf(X, r2_3_1_0, 3.0f * r2_2_1_0);
              const float r0_5_1_0 = fmaf(X, r1_4_1_0, 4.0f * r1_3_1_0);
              g1_33 = fmaf(ek1_2, r0_5_1_0, g1_33);
              const float r5_1_0_0 = X * b6;
              const float r4_2_0_0 = fmaf(X, r5_1_0_0, b5);
              const float r3_3_0_0 = fmaf(X, r4_2_0_0, 2.0f * r4_1_0_0);
              const float r2_4_0_0 = fmaf(X, r3_3_0_0, 3.0f * r3_2_0_0);
              const float r1_5_0_0 = fmaf(X, r2_4_0_0, 4.0f * r2_3_0_0);
              const float r0_6_0_0 = fmaf(X, r1_5_0_0, 5.0f * r1_4_0_0);
              g1_34 = fmaf(ek1_2, r0_6_0_0, g1_34);
            }
            { const float eb = bi[5];
              o0_1 = fmaf(eb, g1_0, o0_1);
            }
            { const float eb = bi[6];
              o0_1 = fmaf(eb, g1_3, o0_1);
            }
            { const float eb = bi[7];
              o0_1 = fmaf(eb, g1_9, o0_1);
            }
            { const float eb = bi[8];
              o0_1 = fmaf(eb, g1_19, o0_1);
            }
            { const float eb = bi[9];
              o0_1 = fmaf(eb, g1_34, o0_1);
            }
            { const float eb = bi[10];
              o1_1 = fmaf(eb, g1_0, o1_1);
            }
            { const float eb = bi[11];
              o1_1 = fmaf(eb, g1_2, o1_1);
            }
            { const float eb = bi[12];
              o1_1 = fmaf(eb, g1_6, o1_1);
            }
            { const float eb = bi[13];
              o1_1 = fmaf(eb, g1_3, o1_1);
            }
            { const float eb = bi[14];
              o1_1 = fmaf(eb, g1_8, o1_1);
            }
            { const float eb = bi[15];
              o1_1 = fmaf(eb, g1_16, o1_1);
            }
            { const float eb = bi[16];
              o1_1 = fmaf(eb, g1_9, o1_1);
            }
            { const float eb = bi[17];
              o1_1 = fmaf(eb, g1_18, o1_1);
            }
            { const float eb = bi[18];
              o1_1 = fmaf(eb, g1_31, o1_1);
            }
            { const float eb = bi[19];
              o2_1 = fmaf(eb, g1_0, o2_1);
            }
            { const float eb = bi[20];
              o2_1 = fmaf(eb, g1_1, o2_1);
            }
            { const float eb = bi[21];
              o2_1 = fmaf(eb, g1_4, o2_1);
            }
            { const float eb = bi[22];
              o2_1 = fmaf(eb, g1_3, o2_1);
            }
            { const float eb = bi[23];
              o2_1 = fmaf(eb, g1_7, o2_1);
            }
            { const float eb = bi[24];
              o2_1 = fmaf(eb, g1_14, o2_1);
            }
            { const float eb = bi[25];
              o2_1 = fmaf(eb, g1_9, o2_1);
            }
            { const float eb = bi[26];
              o2_1 = fmaf(eb, g1_17, o2_1);
            }
            { const float eb = bi[27];
              o2_1 = fmaf(eb, g1_29, o2_1);
            }
            { const float eb = bi[28];
              o3_1 = fmaf(eb, g1_0, o3_1);
            }
            { const float eb = bi[29];
              o3_1 = fmaf(eb, g1_2, o3_1);
            }
            { const float eb = bi[30];
              o3_1 = fmaf(eb, g1_3, o3_1);
            }
            { const float eb = bi[31];
              o3_1 = fmaf(eb, g1_8, o3_1);
            }
            { const float eb = bi[32];
              o3_1 = fmaf(eb, g1_9, o3_1);
            }
            { const float eb = bi[33];
              o3_1 = fmaf(eb, g1_18, o3_1);
            }
            { const float eb = bi[34];
              o3_1 = fmaf(eb, g1_19, o3_1);
            }
            { const float eb = bi[35];
              o3_1 = fmaf(eb, g1_33, o3_1);
            }
            { const float eb = bi[36];
              o4_1 = fmaf(eb, g1_0, o4_1);
            }
            { const float eb = bi[37];
              o4_1 = fmaf(eb, g1_1, o4_1);
            }
            { const float eb = bi[38];
              o4_1 = fmaf(eb, g1_3, o4_1);
            }
            { const float eb = bi[39];
              o4_1 = fmaf(eb, g1_7, o4_1);
            }
            { const float eb = bi[40];
              o4_1 = fmaf(eb, g1_9, o4_1);
            }
            { const float eb = bi[41];
              o4_1 = fmaf(eb, g1_17, o4_1);
            }
            { const float eb = bi[42];
              o4_1 = fmaf(eb, g1_19, o4_1);
            }
            { const float eb = bi[43];
              o4_1 = fmaf(eb, g1_32, o4_1);
            }
            { const float eb = bi[44];
              o5_1 = fmaf(eb, g1_0, o5_1);
            }
            { const float eb = bi[45];
              o5_1 = fmaf(eb, g1_1, o5_1);
            }
            { const float eb = bi[46];
              o5_1 = fmaf(eb, g1_2, o5_1);
            }
            { const float eb = bi[47];
              o5_1 = fmaf(eb, g1_5, o5_1);
            }
            { const float eb = bi[48];
              o5_1 = fmaf(eb, g1_3, o5_1);
            }
            { const float eb = bi[49];
              o5_1 = fmaf(eb, g1_7, o5_1);
            }
            { const float eb = bi[50];
              o5_1 = fmaf(eb, g1_8, o5_1);
            }
            { const float eb = bi[51];
              o5_1 = fmaf(eb, g1_15, o5_1);
            }
            { const float eb = bi[52];
              o5_1 = fmaf(eb, g1_9, o5_1);
            }
            { const float eb = bi[53];
              o5_1 = fmaf(eb, g1_17, o5_1);
            }
            { const float eb = bi[54];
              o5_1 = fmaf(eb, g1_18, o5_1);
            }
            { const float eb = bi[55];
              o5_1 = fmaf(eb, g1_30, o5_1);
            }
            { const float eb = bi[56];
              o6_1 = fmaf(eb, g1_0, o6_1);
            }
            { const float eb = bi[57];
              o6_1 = fmaf(eb, g1_2, o6_1);
            }
            { const float eb = bi[58];
              o6_1 = fmaf(eb, g1_6, o6_1);
            }
            { const float eb = bi[59];
              o6_1 = fmaf(eb, g1_3, o6_1);
            }
            { const float eb = bi[60];
              o6_1 = fmaf(eb, g1_8, o6_1);
            }
            { const float eb = bi[61];
              o6_1 = fmaf(eb, g1_16, o6_1);
            }
            { const float eb = bi[62];
              o6_1 = fmaf(eb, g1_9, o6_1);
            }
            { const float eb = bi[63];
              o6_1 = fmaf(eb, g1_18, o6_1);
            }
            { const float eb = bi[64];
              o6_1 = fmaf(eb, g1_31, o6_1);
            }
            { const float eb = bi[65];
              o7_1 = fmaf(eb, g1_0, o7_1);
            }
            { const float eb = bi[66];
              o7_1 = fmaf(eb, g1_2, o7_1);
            }
            { const float eb = bi[67];
              o7_1 = fmaf(eb, g1_6, o7_1);
            }
            { const float eb = bi[68];
              o7_1 = fmaf(eb, g1_13, o7_1);
            }
            { const float eb = bi[69];
              o7_1 = fmaf(eb, g1_24, o7_1);
            }
            { const float eb = bi[70];
              o8_1 = fmaf(eb, g1_0, o8_1);
            }
            { const float eb = bi[71];
              o8_1 = fmaf(eb, g1_1, o8_1);
            }
            { const float eb = bi[72];
              o8_1 = fmaf(eb, g1_4, o8_1);
            }
            { const float eb = bi[73];
              o8_1 = fmaf(eb, g1_2, o8_1);
            }
            { const float eb = bi[74];
              o8_1 = fmaf(eb, g1_5, o8_1);
            }
            { const float eb = bi[75];
              o8_1 = fmaf(eb, g1_11, o8_1);
            }
            { const float eb = bi[76];
              o8_1 = fmaf(eb, g1_6, o8_1);
            }
            { const float eb = bi[77];
              o8_1 = fmaf(eb, g1_12, o8_1);
            }
            { const float eb = bi[78];
              o8_1 = fmaf(eb, g1_22, o8_1);
            }
            { const float eb = bi[79];
              o9_1 = fmaf(eb, g1_0, o9_1);
            }
            { const float eb = bi[80];
              o9_1 = fmaf(eb, g1_2, o9_1);
            }
            { const float eb = bi[81];
              o9_1 = fmaf(eb, g1_6, o9_1);
            }
            { const float eb = bi[82];
              o9_1 = fmaf(eb, g1_13, o9_1);
            }
            { const float eb = bi[83];
              o9_1 = fmaf(eb, g1_3, o9_1);
            }
            { const float eb = bi[84];
              o9_1 = fmaf(eb, g1_8, o9_1);
            }
            { const float eb = bi[85];
              o9_1 = fmaf(eb, g1_16, o9_1);
            }
            { const float eb = bi[86];
              o9_1 = fmaf(eb, g1_28, o9_1);
            }
            { const float eb = bi[87];
              o10_1 = fmaf(eb, g1_0, o10_1);
            }
            { const float eb = bi[88];
              o10_1 = fmaf(eb, g1_1, o10_1);
            }
            { const float eb = bi[89];
              o10_1 = fmaf(eb, g1_2, o10_1);
            }
            { const float eb = bi[90];
              o10_1 = fmaf(eb, g1_5, o10_1);
            }
            { const float eb = bi[91];
              o10_1 = fmaf(eb, g1_6, o10_1);
            }
            { const float eb = bi[92];
              o10_1 = fmaf(eb, g1_12, o10_1);
            }
            { const float eb = bi[93];
              o10_1 = fmaf(eb, g1_3, o10_1);
            }
            { const float eb = bi[94];
              o10_1 = fmaf(eb, g1_7, o10_1);
            }
            { const float eb = bi[95];
              o10_1 = fmaf(eb, g1_8, o10_1);
            }
            { const float eb = bi[96];
              o10_1 = fmaf(eb, g1_15, o10_1);
            }
            { const float eb = bi[97];
              o10_1 = fmaf(eb, g1_16, o10_1);
            }
            { const float eb = bi[98];
              o10_1 = fmaf(eb, g1_27, o10_1);
            }
            { const float eb = bi[99];
              o11_1 = fmaf(eb, g1_0, o11_1);
            }
            { const float eb = bi[100];
              o11_1 = fmaf(eb, g1_1, o11_1);
            }
            { const float eb = bi[101];
              o11_1 = fmaf(eb, g1_2, o11_1);
            }
            { const float eb = bi[102];
              o11_1 = fmaf(eb, g1_5, o11_1);
            }
            { const float eb = bi[103];
              o11_1 = fmaf(eb, g1_6, o11_1);
            }
            { const float eb = bi[104];
              o11_1 = fmaf(eb, g1_12, o11_1);
            }
            { const float eb = bi[105];
              o11_1 = fmaf(eb, g1_13, o11_1);
            }
            { const float eb = bi[106];
              o11_1 = fmaf(eb, g1_23, o11_1);
            }
            { const float eb = bi[107];
              o12_1 = fmaf(eb, g1_0, o12_1);
            }
            { const float eb = bi[108];
              o12_1 = fmaf(eb, g1_1, o12_1);
            }
            { const float eb = bi[109];
              o12_1 = fmaf(eb, g1_4, o12_1);
            }
            { const float eb = bi[110];
              o12_1 = fmaf(eb, g1_3, o12_1);
            }
            { const float eb = bi[111];
              o12_1 = fmaf(eb, g1_7, o12_1);
            }
            { const float eb = bi[112];
              o12_1 = fmaf(eb, g1_14, o12_1);
            }
            { const float eb = bi[113];
              o12_1 = fmaf(eb, g1_9, o12_1);
            }
            { const float eb = bi[114];
              o12_1 = fmaf(eb, g1_17, o12_1);
            }
            { const float eb = bi[115];
              o12_1 = fmaf(eb, g1_29, o12_1);
            }
            { const float eb = bi[116];
              o13_1 = fmaf(eb, g1_0, o13_1);
            }
            { const float eb = bi[117];
              o13_1 = fmaf(eb, g1_1, o13_1);
            }
            { const float eb = bi[118];
              o13_1 = fmaf(eb, g1_4, o13_1);
            }
            { const float eb = bi[119];
              o13_1 = fmaf(eb, g1_2, o13_1);
            }
            { const float eb = bi[120];
              o13_1 = fmaf(eb, g1_5, o13_1);
            }
            { const float eb = bi[121];
              o13_1 = fmaf(eb, g1_11, o13_1);
            }
            { const float eb = bi[122];
              o13_1 = fmaf(eb, g1_6, o13_1);
            }
            { const float eb = bi[123];
              o13_1 = fmaf(eb, g1_12, o13_1);
            }
            { const float eb = bi[124];
              o13_1 = fmaf(eb, g1_22, o13_1);
            }
            { const float eb = bi[125];
              o14_1 = fmaf(eb, g1_0, o14_1);
            }
            { const float eb = bi[126];
              o14_1 = fmaf(eb, g1_1, o14_1);
            }
            { const float eb = bi[127];
              o14_1 = fmaf(eb, g1_4, o14_1);
            }
            { const float eb = bi[128];
              o14_1 = fmaf(eb, g1_10, o14_1);
            }
            { const float eb = bi[129];
              o14_1 = fmaf(eb, g1_20, o14_1);
            }
            { const float eb = bi[130];
              o15_1 = fmaf(eb, g1_0, o15_1);
            }
            { const float eb = bi[131];
              o15_1 = fmaf(eb, g1_1, o15_1);
            }
            { const float eb = bi[132];
              o15_1 = fmaf(eb, g1_4, o15_1);
            }
            { const float eb = bi[133];
              o15_1 = fmaf(eb, g1_2, o15_1);
            }
            { const float eb = bi[134];
              o15_1 = fmaf(eb, g1_5, o15_1);
            }
            { const float eb = bi[135];
              o15_1 = fmaf(eb, g1_11, o15_1);
            }
            { const float eb = bi[136];
              o15_1 = fmaf(eb, g1_3, o15_1);
            }
            { const float eb = bi[137];
              o15_1 = fmaf(eb, g1_7, o15_1);
            }
            { const float eb = bi[138];
              o15_1 = fmaf(eb, g1_14, o15_1);
            }
            { const float eb = bi[139];
              o15_1 = fmaf(eb, g1_8, o15_1);
            }
            { const float eb = bi[140];
              o15_1 = fmaf(eb, g1_15, o15_1);
            }
            { const float eb = bi[141];
              o15_1 = fmaf(eb, g1_26, o15_1);
            }
            { const float eb = bi[142];
              o16_1 = fmaf(eb, g1_0, o16_1);
            }
            { const float eb = bi[143];
              o16_1 = fmaf(eb, g1_1, o16_1);
            }
            { const float eb = bi[144];
              o16_1 = fmaf(eb, g1_4, o16_1);
            }
            { const float eb = bi[145];
              o16_1 = fmaf(eb, g1_10, o16_1);
            }
            { const float eb = bi[146];
              o16_1 = fmaf(eb, g1_3, o16_1);
            }
            { const float eb = bi[147];
              o16_1 = fmaf(eb, g1_7, o16_1);
            }
            { const float eb = bi[148];
              o16_1 = fmaf(eb, g1_14, o16_1);
            }
            { const float eb = bi[149];
              o16_1 = fmaf(eb, g1_25, o16_1);
            }
            { const float eb = bi[150];
              o17_1 = fmaf(eb, g1_0, o17_1);
            }
            { const float eb = bi[151];
              o17_1 = fmaf(eb, g1_1, o17_1);
            }
            { const float eb = bi[152];
              o17_1 = fmaf(eb, g1_4, o17_1);
            }
            { const float eb = bi[153];
              o17_1 = fmaf(eb, g1_10, o17_1);
            }
            { const float eb = bi[154];
              o17_1 = fmaf(eb, g1_2, o17_1);
            }
            { const float eb = bi[155];
              o17_1 = fmaf(eb, g1_5, o17_1);
            }
            { const float eb = bi[156];
              o17_1 = fmaf(eb, g1_11, o17_1);
            }
            { const float eb = bi[157];
              o17_1 = fmaf(eb, g1_21, o17_1);
            }
            { const float eb = bi[158];
              o18_1 = fmaf(eb, g1_0, o18_1);
            }
            { const float eb = bi[159];
              o18_1 = fmaf(eb, g1_2, o18_1);
            }
            { const float eb = bi[160];
              o18_1 = fmaf(eb, g1_3, o18_1);
            }
            { const float eb = bi[161];
              o18_1 = fmaf(eb, g1_8, o18_1);
            }
            { const float eb = bi[162];
              o18_1 = fmaf(eb, g1_9, o18_1);
            }
            { const float eb = bi[163];
              o18_1 = fmaf(eb, g1_18, o18_1);
            }
            { const float eb = bi[164];
              o18_1 = fmaf(eb, g1_19, o18_1);
            }
            { const float eb = bi[165];
              o18_1 = fmaf(eb, g1_33, o18_1);
            }
            { const float eb = bi[166];
              o19_1 = fmaf(eb, g1_0, o19_1);
            }
            { const float eb = bi[167];
              o19_1 = fmaf(eb, g1_2, o19_1);
            }
            { const float eb = bi[168];
              o19_1 = fmaf(eb, g1_6, o19_1);
            }
            { const float eb = bi[169];
              o19_1 = fmaf(eb, g1_13, o19_1);
            }
            { const float eb = bi[170];
              o19_1 = fmaf(eb, g1_3, o19_1);
            }
            { const float eb = bi[171];
              o19_1 = fmaf(eb, g1_8, o19_1);
            }
            { const float eb = bi[172];
              o19_1 = fmaf(eb, g1_16, o19_1);
            }
            { const float eb = bi[173];
              o19_1 = fmaf(eb, g1_28, o19_1);
            }
            { const float eb = bi[174];
              o20_1 = fmaf(eb, g1_0, o20_1);
            }
            { const float eb = bi[175];
              o20_1 = fmaf(eb, g1_1, o20_1);
            }
            { const float eb = bi[176];
              o20_1 = fmaf(eb, g1_4, o20_1);
            }
            { const float eb = bi[177];
              o20_1 = fmaf(eb, g1_2, o20_1);
            }
            { const float eb = bi[178];
              o20_1 = fmaf(eb, g1_5, o20_1);
            }
            { const float eb = bi[179];
              o20_1 = fmaf(eb, g1_11, o20_1);
            }
            { const float eb = bi[180];
              o20_1 = fmaf(eb, g1_3, o20_1);
            }
            { const float eb = bi[181];
              o20_1 = fmaf(eb, g1_7, o20_1);
            }
            { const float eb = bi[182];
              o20_1 = fmaf(eb, g1_14, o20_1);
            }
            { const float eb = bi[183];
              o20_1 = fmaf(eb, g1_8, o20_1);
            }
            { const float eb = bi[184];
              o20_1 = fmaf(eb, g1_15, o20_1);
            }
            { const float eb = bi[185];
              o20_1 = fmaf(eb, g1_26, o20_1);
            }
            { const float eb = bi[186];
              o21_1 = fmaf(eb, g1_0, o21_1);
            }
            { const float eb = bi[187];
              o21_1 = fmaf(eb, g1_2, o21_1);
            }
            { const float eb = bi[188];
              o21_1 = fmaf(eb, g1_6, o21_1);
            }
            { const float eb = bi[189];
              o21_1 = fmaf(eb, g1_3, o21_1);
            }
            { const float eb = bi[190];
              o21_1 = fmaf(eb, g1_8, o21_1);
            }
            { const float eb = bi[191];
              o21_1 = fmaf(eb, g1_16, o21_1);
            }
            { const float eb = bi[192];
              o21_1 = fmaf(eb, g1_9, o21_1);
            }
            { const float eb = bi[193];
              o21_1 = fmaf(eb, g1_18, o21_1);
            }
            { const float eb = bi[194];
              o21_1 = fmaf(eb, g1_31, o21_1);
            }
            { const float eb = bi[195];
              o22_1 = fmaf(eb, g1_0, o22_1);
            }
            { const float eb = bi[196];
              o22_1 = fmaf(eb, g1_1, o22_1);
            }
            { const float eb = bi[197];
              o22_1 = fmaf(eb, g1_2, o22_1);
            }
            { const float eb = bi[198];
              o22_1 = fmaf(eb, g1_5, o22_1);
            }
            { const float eb = bi[199];
              o22_1 = fmaf(eb, g1_3, o22_1);
            }
            { const float eb = bi[200];
              o22_1 = fmaf(eb, g1_7, o22_1);
            }
            { const float eb = bi[201];
              o22_1 = fmaf(eb, g1_8, o22_1);
            }
            { const float eb = bi[202];
              o22_1 = fmaf(eb, g1_15, o22_1);
            }
            { const float eb = bi[203];
              o22_1 = fmaf(eb, g1_9, o22_1);
            }
            { const float eb = bi[204];
              o22_1 = fmaf(eb, g1_17, o22_1);
            }
            { const float eb = bi[205];
              o22_1 = fmaf(eb, g1_18, o22_1);
            }
            { const float eb = bi[206];
              o22_1 = fmaf(eb, g1_30, o22_1);
            }
            { const float eb = bi[207];
              o23_1 = fmaf(eb, g1_0, o23_1);
            }
            { const float eb = bi[208];
              o23_1 = fmaf(eb, g1_1, o23_1);
            }
            { const float eb = bi[209];
              o23_1 = fmaf(eb, g1_2, o23_1);
            }
            { const float eb = bi[210];
              o23_1 = fmaf(eb, g1_5, o23_1);
            }
            { const float eb = bi[211];
              o23_1 = fmaf(eb, g1_6, o23_1);
            }
            { const float eb = bi[212];
              o23_1 = fmaf(eb, g1_12, o23_1);
            }
            { const float eb = bi[213];
              o23_1 = fmaf(eb, g1_3, o23_1);
            }
            { const float eb = bi[214];
              o23_1 = fmaf(eb, g1_7, o23_1);
            }
            { const float eb = bi[215];
              o23_1 = fmaf(eb, g1_8, o23_1);
            }
            { const float eb = bi[216];
              o23_1 = fmaf(eb, g1_15, o23_1);
            }
            { const float eb = bi[217];
              o23_1 = fmaf(eb, g1_16, o23_1);
            }
            { const float eb = bi[218];
              o23_1 = fmaf(eb, g1_27, o23_1);
            }
            { const float eb = bi[219];
              o24_1 = fmaf(eb, g1_0, o24_1);
            }
            { const float eb = bi[220];
              o24_1 = fmaf(eb, g1_1, o24_1);
            }
            { const float eb = bi[221];
              o24_1 = fmaf(eb, g1_3, o24_1);
            }
            { const float eb = bi[222];
              o24_1 = fmaf(eb, g1_7, o24_1);
            }
            { const float eb = bi[223];
              o24_1 = fmaf(eb, g1_9, o24_1);
            }
            { const float eb = bi[224];
              o24_1 = fmaf(eb, g1_17, o24_1);
            }
            { const float eb = bi[225];
              o24_1 = fmaf(eb, g1_19, o24_1);
            }
            { const float eb = bi[226];
              o24_1 = fmaf(eb, g1_32, o24_1);
            }
            { const float eb = bi[227];
              o25_1 = fmaf(eb, g1_0, o25_1);
            }
            { const float eb = bi[228];
              o25_1 = fmaf(eb, g1_1, o25_1);
            }
            { const float eb = bi[229];
              o25_1 = fmaf(eb, g1_2, o25_1);
            }
            { const float eb = bi[230];
              o25_1 = fmaf(eb, g1_5, o25_1);
            }
            { const float eb = bi[231];
              o25_1 = fmaf(eb, g1_6, o25_1);
            }
            { const float eb = bi[232];
              o25_1 = fmaf(eb, g1_12, o25_1);
            }
            { const float eb = bi[233];
              o25_1 = fmaf(eb, g1_3, o25_1);
            }
            { const float eb = bi[234];
              o25_1 = fmaf(eb, g1_7, o25_1);
            }
            { const float eb = bi[235];
              o25_1 = fmaf(eb, g1_8, o25_1);
            }
            { const float eb = bi[236];
              o25_1 = fmaf(eb, g1_15, o25_1);
            }
            { const float eb = bi[237];
              o25_1 = fmaf(eb, g1_16, o25_1);
            }
            { const float eb = bi[238];
              o25_1 = fmaf(eb, g1_27, o25_1);
            }
            { const float eb = bi[239];
              o26_1 = fmaf(eb, g1_0, o26_1);
            }
            { const float eb = bi[240];
              o26_1 = fmaf(eb, g1_1, o26_1);
            }
            { const float eb = bi[241];
              o26_1 = fmaf(eb, g1_4, o26_1);
            }
            { const float eb = bi[242];
              o26_1 = fmaf(eb, g1_10, o26_1);
            }
            { const float eb = bi[243];
              o26_1 = fmaf(eb, g1_3, o26_1);
            }
            { const float eb = bi[244];
              o26_1 = fmaf(eb, g1_7, o26_1);
            }
            { const float eb = bi[245];
              o26_1 = fmaf(eb, g1_14, o26_1);
            }
            { const float eb = bi[246];
              o26_1 = fmaf(eb, g1_25, o26_1);
            }
            { const float eb = bi[247];
              o27_1 = fmaf(eb, g1_0, o27_1);
            }
            { const float eb = bi[248];
              o27_1 = fmaf(eb, g1_1, o27_1);
            }
            { const float eb = bi[249];
              o27_1 = fmaf(eb, g1_2, o27_1);
            }
            { const float eb = bi[250];
              o27_1 = fmaf(eb, g1_5, o27_1);
            }
            { const float eb = bi[251];
              o27_1 = fmaf(eb, g1_3, o27_1);
            }
            { const float eb = bi[252];
              o27_1 = fmaf(eb, g1_7, o27_1);
            }
            { const float eb = bi[253];
              o27_1 = fmaf(eb, g1_8, o27_1);
            }
            { const float eb = bi[254];
              o27_1 = fmaf(eb, g1_15, o27_1);
            }
            { const float eb = bi[255];
              o27_1 = fmaf(eb, g1_9, o27_1);
            }
            { const float eb = bi[256];
              o27_1 = fmaf(eb, g1_17, o27_1);
            }
            { const float eb = bi[257];
              o27_1 = fmaf(eb, g1_18, o27_1);
            }
            { const float eb = bi[258];
              o27_1 = fmaf(eb, g1_30, o27_1);
            }
            { const float eb = bi[259];
              o28_1 = fmaf(eb, g1_0, o28_1);
            }
            { const float eb = bi[260];
              o28_1 = fmaf(eb, g1_1, o28_1);
            }
            { const float eb = bi[261];
              o28_1 = fmaf(eb, g1_4, o28_1);
            }
            { const float eb = bi[262];
              o28_1 = fmaf(eb, g1_3, o28_1);
            }
            { const float eb = bi[263];
              o28_1 = fmaf(eb, g1_7, o28_1);
            }
            { const float eb = bi[264];
              o28_1 = fmaf(eb, g1_14, o28_1);
            }
            { const float eb = bi[265];
              o28_1 = fmaf(eb, g1_9, o28_1);
            }
            { const float eb = bi[266];
              o28_1 = fmaf(eb, g1_17, o28_1);
            }
            { const float eb = bi[267];
              o28_1 = fmaf(eb, g1_29, o28_1);
            }
            { const float eb = bi[268];
              o29_1 = fmaf(eb, g1_0, o29_1);
            }
            { const float eb = bi[269];
              o29_1 = fmaf(eb, g1_1, o29_1);
            }
            { const float eb = bi[270];
              o29_1 = fmaf(eb, g1_4, o29_1);
            }
            { const float eb = bi[271];
              o29_1 = fmaf(eb, g1_2, o29_1);
            }
            { const float eb = bi[272];
              o29_1 = fmaf(eb, g1_5, o29_1);
            }
            { const float eb = bi[273];
              o29_1 = fmaf(eb, g1_11, o29_1);
            }
            { const float eb = bi[274];
              o29_1 = fmaf(eb, g1_3, o29_1);
            }
            { const float eb = bi[275];
              o29_1 = fmaf(eb, g1_7, o29_1);
            }
            { const float eb = bi[276];
              o29_1 = fmaf(eb, g1_14, o29_1);
            }
            { const float eb = bi[277];
              o29_1 = fmaf(eb, g1_8, o29_1);
            }
            { const float eb = bi[278];
              o29_1 = fmaf(eb, g1_15, o29_1);
            }
            { const float eb = bi[279];
              o29_1 = fmaf(eb, g1_26, o29_1);
            }
            { const float eb = bi[280];
              o30_1 = fmaf(eb, g1_0, o30_1);
            }
            { const float eb = bi[281];
              o30_1 = fmaf(eb, g1_1, o30_1);
            }
            { const float eb = bi[282];
              o30_1 = fmaf(eb, g1_2, o30_1);
            }
            { const float eb = bi[283];
              o30_1 = fmaf(eb, g1_5, o30_1);
            }
            { const float eb = bi[284];
              o30_1 = fmaf(eb, g1_3, o30_1);
            }
            { const float eb = bi[285];
              o30_1 = fmaf(eb, g1_7, o30_1);
            }
            { const float eb = bi[286];
              o30_1 = fmaf(eb, g1_8, o30_1);
            }
            { const float eb = bi[287];
              o30_1 = fmaf(eb, g1_15, o30_1);
            }
            { const float eb = bi[288];
              o30_1 = fmaf(eb, g1_9, o30_1);
            }
            { const float eb = bi[289];
              o30_1 = fmaf(eb, g1_17, o30_1);
            }
            { const float eb = bi[290];
              o30_1 = fmaf(eb, g1_18, o30_1);
            }
            { const float eb = bi[291];
              o30_1 = fmaf(eb, g1_30, o30_1);
            }
            { const float eb = bi[292];
              o31_1 = fmaf(eb, g1_0, o31_1);
            }
            { const float eb = bi[293];
              o31_1 = fmaf(eb, g1_1, o31_1);
            }
            { const float eb = bi[294];
              o31_1 = fmaf(eb, g1_2, o31_1);
            }
            { const float eb = bi[295];
              o31_1 = fmaf(eb, g1_5, o31_1);
            }
            { const float eb = bi[296];
              o31_1 = fmaf(eb, g1_6, o31_1);
            }
            { const float eb = bi[297];
              o31_1 = fmaf(eb, g1_12, o31_1);
            }
            { const float eb = bi[298];
              o31_1 = fmaf(eb, g1_13, o31_1);
            }
            { const float eb = bi[299];
              o31_1 = fmaf(eb, g1_23, o31_1);
            }
            { const float eb = bi[300];
              o32_1 = fmaf(eb, g1_0, o32_1);
            }
            { const float eb = bi[301];
              o32_1 = fmaf(eb, g1_1, o32_1);
            }
            { const float eb = bi[302];
              o32_1 = fmaf(eb, g1_4, o32_1);
            }
            { const float eb = bi[303];
              o32_1 = fmaf(eb, g1_10, o32_1);
            }
            { const float eb = bi[304];
              o32_1 = fmaf(eb, g1_2, o32_1);
            }
            { const float eb = bi[305];
              o32_1 = fmaf(eb, g1_5, o32_1);
            }
            { const float eb = bi[306];
              o32_1 = fmaf(eb, g1_11, o32_1);
            }
            { const float eb = bi[307];
              o32_1 = fmaf(eb, g1_21, o32_1);
            }
            { const float eb = bi[308];
              o33_1 = fmaf(eb, g1_0, o33_1);
            }
            { const float eb = bi[309];
              o33_1 = fmaf(eb, g1_1, o33_1);
            }
            { const float eb = bi[310];
              o33_1 = fmaf(eb, g1_2, o33_1);
            }
            { const float eb = bi[311];
              o33_1 = fmaf(eb, g1_5, o33_1);
            }
            { const float eb = bi[312];
              o33_1 = fmaf(eb, g1_6, o33_1);
            }
            { const float eb = bi[313];
              o33_1 = fmaf(eb, g1_12, o33_1);
            }
            { const float eb = bi[314];
              o33_1 = fmaf(eb, g1_3, o33_1);
            }
            { const float eb = bi[315];
              o33_1 = fmaf(eb, g1_7, o33_1);
            }
            { const float eb = bi[316];
              o33_1 = fmaf(eb, g1_8, o33_1);
            }
            { const float eb = bi[317];
              o33_1 = fmaf(eb, g1_15, o33_1);
            }
            { const float eb = bi[318];
              o33_1 = fmaf(eb, g1_16, o33_1);
            }
            { const float eb = bi[319];
              o33_1 = fmaf(eb, g1_27, o33_1);
            }
            { const float eb = bi[320];
              o34_1 = fmaf(eb, g1_0, o34_1);
            }
            { const float eb = bi[321];
              o34_1 = fmaf(eb, g1_1, o34_1);
            }
            { const float eb = bi[322];
              o34_1 = fmaf(eb, g1_4, o34_1);
            }
            { const float eb = bi[323];
              o34_1 = fmaf(eb, g1_2, o34_1);
            }
            { const float eb = bi[324];
              o34_1 = fmaf(eb, g1_5, o34_1);
            }
            { const float eb = bi[325];
              o34_1 = fmaf(eb, g1_11, o34_1);
            }
            { const float eb = bi[326];
              o34_1 = fmaf(eb, g1_3, o34_1);
            }
            { const float eb = bi[327];
              o34_1 = fmaf(eb, g1_7, o34_1);
            }
            { const float eb = bi[328];
              o34_1 = fmaf(eb, g1_14, o34_1);
            }
            { const float eb = bi[329];
              o34_1 = fmaf(eb, g1_8, o34_1);
            }
            { const float eb = bi[330];
              o34_1 = fmaf(eb, g1_15, o34_1);
            }
            { const float eb = bi[331];
              o34_1 = fmaf(eb, g1_26, o34_1);
            }
            { const float eb = bi[332];
              o35_1 = fmaf(eb, g1_0, o35_1);
            }
            { const float eb = bi[333];
              o35_1 = fmaf(eb, g1_1, o35_1);
            }
            { const float eb = bi[334];
              o35_1 = fmaf(eb, g1_4, o35_1);
            }
            { const float eb = bi[335];
              o35_1 = fmaf(eb, g1_2, o35_1);
            }
            { const float eb = bi[336];
              o35_1 = fmaf(eb, g1_5, o35_1);
            }
            { const float eb = bi[337];
              o35_1 = fmaf(eb, g1_11, o35_1);
            }
            { const float eb = bi[338];
              o35_1 = fmaf(eb, g1_6, o35_1);
            }
            { const float eb = bi[339];
              o35_1 = fmaf(eb, g1_12, o35_1);
            }
            { const float eb = bi[340];
              o35_1 = fmaf(eb, g1_22, o35_1);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk1 = PT[(fI + 0) * N + fJ + 1];
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Abd4_1 = PA[(fQ + 4) * N + fJ + 1];
            const double Abd5_1 = PA[(fQ + 5) * N + fJ + 1];
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
            const double Abc4_0 = PA[(fQ + 4) * N + fI + 0];
            const double Abc5_0 = PA[(fQ + 5) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 1, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5 + o6_1 * ptb6 + o7_1 * ptb7 + o8_1 * ptb8 + o9_1 * ptb9 + o10_1 * ptb10 + o11_1 * ptb11 + o12_1 * ptb12 + o13_1 * ptb13 + o14_1 * ptb14 + o15_1 * ptb15 + o16_1 * ptb16 + o17_1 * ptb17 + o18_1 * ptb18 + o19_1 * ptb19 + o20_1 * ptb20 + o21_1 * ptb21 + o22_1 * ptb22 + o23_1 * ptb23 + o24_1 * ptb24 + o25_1 * ptb25 + o26_1 * ptb26 + o27_1 * ptb27 + o28_1 * ptb28 + o29_1 * ptb29 + o30_1 * ptb30 + o31_1 * ptb31 + o32_1 * ptb32 + o33_1 * ptb33 + o34_1 * ptb34 + o35_1 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_1 * Abd0_1 + o1_1 * Abd1_1 + o2_1 * Abd2_1 + o3_1 * Abd3_1 + o4_1 * Abd4_1 + o5_1 * Abd5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_1 * Aad0_1 + o6_1 * Aad1_1 + o12_1 * Aad2_1 + o18_1 * Aad3_1 + o24_1 * Aad4_1 + o30_1 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_1 * Abc0_0 + o1_1 * Abc1_0 + o2_1 * Abc2_0 + o3_1 * Abc3_0 + o4_1 * Abc4_0 + o5_1 * Abc5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_1 * Aac0_0 + o6_1 * Aac1_0 + o12_1 * Aac2_0 + o18_1 * Aac3_0 + o24_1 * Aac4_0 + o30_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_1 * Aad0_1 + o7_1 * Aad1_1 + o13_1 * Aad2_1 + o19_1 * Aad3_1 + o25_1 * Aad4_1 + o31_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_1 * Aac0_0 + o7_1 * Aac1_0 + o13_1 * Aac2_0 + o19_1 * Aac3_0 + o25_1 * Aac4_0 + o31_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_1 * Aad0_1 + o8_1 * Aad1_1 + o14_1 * Aad2_1 + o20_1 * Aad3_1 + o26_1 * Aad4_1 + o32_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_1 * Aac0_0 + o8_1 * Aac1_0 + o14_1 * Aac2_0 + o20_1 * Aac3_0 + o26_1 * Aac4_0 + o32_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_1 * Aad0_1 + o9_1 * Aad1_1 + o15_1 * Aad2_1 + o21_1 * Aad3_1 + o27_1 * Aad4_1 + o33_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_1 * Aac0_0 + o9_1 * Aac1_0 + o15_1 * Aac2_0 + o21_1 * Aac3_0 + o27_1 * Aac4_0 + o33_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 0, deg * (o4_1 * Aad0_1 + o10_1 * Aad1_1 + o16_1 * Aad2_1 + o22_1 * Aad3_1 + o28_1 * Aad4_1 + o34_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 1, deg * (o4_1 * Aac0_0 + o10_1 * Aac1_0 + o16_1 * Aac2_0 + o22_1 * Aac3_0 + o28_1 * Aac4_0 + o34_1 * Aac5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 0, deg * (o5_1 * Aad0_1 + o11_1 * Aad1_1 + o17_1 * Aad2_1 + o23_1 * Aad3_1 + o29_1 * Aad4_1 + o35_1 * Aad5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 1, deg * (o5_1 * Aac0_0 + o11_1 * Aac1_0 + o17_1 * Aac2_0 + o23_1 * Aac3_0 + o29_1 * Aac4_0 + o35_1 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o6_1 * Abd0_1 + o7_1 * Abd1_1 + o8_1 * Abd2_1 + o9_1 * Abd3_1 + o10_1 * Abd4_1 + o11_1 * Abd5_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o6_1 * Abc0_0 + o7_1 * Abc1_0 + o8_1 * Abc2_0 + o9_1 * Abc3_0 + o10_1 * Abc4_0 + o11_1 * Abc5_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o12_1 * Abd0_1 + o13_1 * Abd1_1 + o14_1 * Abd2_1 + o15_1 * Abd3_1 + o16_1 * Abd4_1 + o17_1 * Abd5_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o12_1 * Abc0_0 + o13_1 * Abc1_0 + o14_1 * Abc2_0 + o15_1 * Abc3_0 + o16_1 * Abc4_0 + o17_1 * Abc5_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o18_1 * Abd0_1 + o19_1 * Abd1_1 + o20_1 * Abd2_1 + o21_1 * Abd3_1 + o22_1 * Abd4_1 + o23_1 * Abd5_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o18_1 * Abc0_0 + o19_1 * Abc1_0 + o20_1 * Abc2_0 + o21_1 * Abc3_0 + o22_1 * Abc4_0 + o23_1 * Abc5_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o24_1 * Abd0_1 + o25_1 * Abd1_1 + o26_1 * Abd2_1 + o27_1 * Abd3_1 + o28_1 * Abd4_1 + o29_1 * Abd5_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o24_1 * Abc0_0 + o25_1 * Abc1_0 + o26_1 * Abc2_0 + o27_1 * Abc3_0 + o28_1 * Abc4_0 + o29_1 * Abc5_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o30_1 * Abd0_1 + o31_1 * Abd1_1 + o32_1 * Abd2_1 + o33_1 * Abd3_1 + o34_1 * Abd4_1 + o35_1 * Abd5_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o30_1 * Abc0_0 + o31_1 * Abc1_0 + o32_1 * Abc2_0 + o33_1 * Abc3_0 + o34_1 * Abc4_0 + o35_1 * Abc5_0));
          }
        } break;
        case 2: {  // ket functions [2]
          float o0_2 = 0;
          float o1_2 = 0;
          float o2_2 = 0;
          float o3_2 = 0;
          float o4_2 = 0;
          float o5_2 = 0;
          float o6_2 = 0;
          float o7_2 = 0;
          float o8_2 = 0;
          float o9_2 = 0;
          float o10_2 = 0;
          float o11_2 = 0;
          float o12_2 = 0;
          float o13_2 = 0;
          float o14_2 = 0;
          float o15_2 = 0;
          float o16_2 = 0;
          float o17_2 = 0;
          float o18_2 = 0;
          float o19_2 = 0;
          float o20_2 = 0;
          float o21_2 = 0;
          float o22_2 = 0;
          float o23_2 = 0;
          float o24_2 = 0;
          float o25_2 = 0;
          float o26_2 = 0;
          float o27_2 = 0;
          float o28_2 = 0;
          float o29_2 = 0;
          float o30_2 = 0;
          float o31_2 = 0;
          float o32_2 = 0;
          float o33_2 = 0;
          float o34_2 = 0;
          float o35_2 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            float g2_10 = 0;
            float g2_11 = 0;
            float g2_12 = 0;
            float g2_13 = 0;
            float g2_14 = 0;
            float g2_15 = 0;
            float g2_16 = 0;
            float g2_17 = 0;
            float g2_18 = 0;
            float g2_19 = 0;
            float g2_20 = 0;
            float g2_21 = 0;
            float g2_22 = 0;
            float g2_23 = 0;
            float g2_24 = 0;
            float g2_25 = 0;
            float g2_26 = 0;
            float g2_27 = 0;
            float g2_28 = 0;
            float g2_29 = 0;
            float g2_30 = 0;
            float g2_31 = 0;
            float g2_32 = 0;
            float g2_33 = 0;
            float g2_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek2_0 = kj[10 * kS];
              const float ek2_1 = -kj[11 * kS];
              const float ek2_2 = -kj[12 * kS];
              const float ek2_3 = kj[13 * kS];
              g2_0 = fmaf(ek2_0, b0, g2_0);
              const float r0_0_0_1 = Z * b1;
              g2_1 = fmaf(ek2_0, r0_0_0_1, g2_1);
              const float r0_0_1_0 = Y * b1;
              g2_2 = fmaf(ek2_0, r0_0_1_0, g2_2);
              g2_0 = fmaf(ek2_1, r0_0_1_0, g2_0);
              const float r0_1_0_0 = X * b1;
              g2_3 = fmaf(ek2_0, r0_1_0_0, g2_3);
              g2_0 = fmaf(ek2_2, r0_1_0_0, g2_0);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g2_4 = fmaf(ek2_0, r0_0_0_2, g2_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g2_5 = fmaf(ek2_0, r0_0_1_1, g2_5);
              g2_1 = fmaf(ek2_1, r0_0_1_1, g2_1);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g2_6 = fmaf(ek2_0, r0_0_2_0, g2_6);
              g2_2 = fmaf(ek2_1, r0_0_2_0, g2_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g2_7 = fmaf(ek2_0, r0_1_0_1, g2_7);
              g2_1 = fmaf(ek2_2, r0_1_0_1, g2_1);
              const float r0_1_1_0 = X * r1_0_1_0;
              g2_8 = fmaf(ek2_0, r0_1_1_0, g2_8);
              g2_3 = fmaf(ek2_1, r0_1_1_0, g2_3);
              g2_2 = fmaf(ek2_2, r0_1_1_0, g2_2);
              g2_0 = fmaf(ek2_3, r0_1_1_0, g2_0);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g2_9 = fmaf(ek2_0, r0_2_0_0, g2_9);
              g2_3 = fmaf(ek2_2, r0_2_0_0, g2_3);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g2_10 = fmaf(ek2_0, r0_0_0_3, g2_10);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g2_11 = fmaf(ek2_0, r0_0_1_2, g2_11);
              g2_4 = fmaf(ek2_1, r0_0_1_2, g2_4);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g2_12 = fmaf(ek2_0, r0_0_2_1, g2_12);
              g2_5 = fmaf(ek2_1, r0_0_2_1, g2_5);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g2_13 = fmaf(ek2_0, r0_0_3_0, g2_13);
              g2_6 = fmaf(ek2_1, r0_0_3_0, g2_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g2_14 = fmaf(ek2_0, r0_1_0_2, g2_14);
              g2_4 = fmaf(ek2_2, r0_1_0_2, g2_4);
              const float r0_1_1_1 = X * r1_0_1_1;
              g2_15 = fmaf(ek2_0, r0_1_1_1, g2_15);
              g2_7 = fmaf(ek2_1, r0_1_1_1, g2_7);
              g2_5 = fmaf(ek2_2, r0_1_1_1, g2_5);
              g2_1 = fmaf(ek2_3, r0_1_1_1, g2_1);
              const float r0_1_2_0 = X * r1_0_2_0;
              g2_16 = fmaf(ek2_0, r0_1_2_0, g2_16);
              g2_8 = fmaf(ek2_1, r0_1_2_0, g2_8);
              g2_6 = fmaf(ek2_2, r0_1_2_0, g2_6);
              g2_2 = fmaf(ek2_3, r0_1_2_0, g2_2);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g2_17 = fmaf(ek2_0, r0_2_0_1, g2_17);
              g2_7 = fmaf(ek2_2, r0_2_0_1, g2_7);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g2_18 = fmaf(ek2_0, r0_2_1_0, g2_18);
              g2_9 = fmaf(ek2_1, r0_2_1_0, g2_9);
              g2_8 = fmaf(ek2_2, r0_2_1_0, g2_8);
              g2_3 = fmaf(ek2_3, r0_2_1_0, g2_3);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g2_19 = fmaf(ek2_0, r0_3_0_0, g2_19);
              g2_9 = fmaf(ek2_2, r0_3_0_0, g2_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g2_20 = fmaf(ek2_0, r0_0_0_4, g2_20);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g2_21 = fmaf(ek2_0, r0_0_1_3, g2_21);
              g2_10 = fmaf(ek2_1, r0_0_1_3, g2_10);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g2_22 = fmaf(ek2_0, r0_0_2_2, g2_22);
              g2_11 = fmaf(ek2_1, r0_0_2_2, g2_11);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g2_23 = fmaf(ek2_0, r0_0_3_1, g2_23);
              g2_12 = fmaf(ek2_1, r0_0_3_1, g2_12);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g2_24 = fmaf(ek2_0, r0_0_4_0, g2_24);
              g2_13 = fmaf(ek2_1, r0_0_4_0, g2_13);
              const float r0_1_0_3 = X * r1_0_0_3;
              g2_25 = fmaf(ek2_0, r0_1_0_3, g2_25);
              g2_10 = fmaf(ek2_2, r0_1_0_3, g2_10);
              const float r0_1_1_2 = X * r1_0_1_2;
              g2_26 = fmaf(ek2_0, r0_1_1_2, g2_26);
              g2_14 = fmaf(ek2_1, r0_1_1_2, g2_14);
              g2_11 = fmaf(ek2_2, r0_1_1_2, g2_11);
              g2_4 = fmaf(ek2_3, r0_1_1_2, g2_4);
              const float r0_1_2_1 = X * r1_0_2_1;
              g2_27 = fmaf(ek2_0, r0_1_2_1, g2_27);
              g2_15 = fmaf(ek2_1, r0_1_2_1, g2_15);
              g2_12 = fmaf(ek2_2, r0_1_2_1, g2_12);
              g2_5 = fmaf(ek2_3, r0_1_2_1, g2_5);
              const float r0_1_3_0 = X * r1_0_3_0;
              g2_28 = fmaf(ek2_0, r0_1_3_0, g2_28);
              g2_16 = fmaf(ek2_1, r0_1_3_0, g2_16);
              g2_13 = fmaf(ek2_2, r0_1_3_0, g2_13);
              g2_6 = fmaf(ek2_3, r0_1_3_0, g2_6);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g2_29 = fmaf(ek2_0, r0_2_0_2, g2_29);
              g2_14 = fmaf(ek2_2, r0_2_0_2, g2_14);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g2_30 = fmaf(ek2_0, r0_2_1_1, g2_30);
              g2_17 = fmaf(ek2_1, r0_2_1_1, g2_17);
              g2_15 = fmaf(ek2_2, r0_2_1_1, g2_15);
              g2_7 = fmaf(ek2_3, r0_2_1_1, g2_7);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g2_31 = fmaf(ek2_0, r0_2_2_0, g2_31);
              g2_18 = fmaf(ek2_1, r0_2_2_0, g2_18);
              g2_16 = fmaf(ek2_2, r0_2_2_0, g2_16);
              g2_8 = fmaf(ek2_3, r0_2_2_0, g2_8);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g2_32 = fmaf(ek2_0, r0_3_0_1, g2_32);
              g2_17 = fmaf(ek2_2, r0_3_0_1, g2_17);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g2_33 = fmaf(ek2_0, r0_3_1_0, g2_33);
              g2_19 = fmaf(ek2_1, r0_3_1_0, g2_19);
              g2_18 = fmaf(ek2_2, r0_3_1_0, g2_18);
              g2_9 = fmaf(ek2_3, r0_3_1_0, g2_9);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g2_34 = fmaf(ek2_0, r0_4_0_0, g2_34);
              g2_19 = fmaf(ek2_2, r0_4_0_0, g2_19);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g2_20 = fmaf(ek2_1, r0_0_1_4, g2_20);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g2_21 = fmaf(ek2_1, r0_0_2_3, g2_21);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g2_22 = fmaf(ek2_1, r0_0_3_2, g2_22);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g2_23 = fmaf(ek2_1, r0_0_4_1, g2_23);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_0_5_0 = fmaf(Y, r1_0_4_0, 4.0f * r1_0_3_0);
              g2_24 = fmaf(ek2_1, r0_0_5_0, g2_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g2_20 = fmaf(ek2_2, r0_1_0_4, g2_20);
              const float r0_1_1_3 = X * r1_0_1_3;
              g2_25 = fmaf(ek2_1, r0_1_1_3, g2_25);
              g2_21 = fmaf(ek2_2, r0_1_1_3, g2_21);
              g2_10 = fmaf(ek2_3, r0_1_1_3, g2_10);
              const float r0_1_2_2 = X * r1_0_2_2;
              g2_26 = fmaf(ek2_1, r0_1_2_2, g2_26);
              g2_22 = fmaf(ek2_2, r0_1_2_2, g2_22);
              g2_11 = fmaf(ek2_3, r0_1_2_2, g2_11);
              const float r0_1_3_1 = X * r1_0_3_1;
              g2_27 = fmaf(ek2_1, r0_1_3_1, g2_27);
              g2_23 = fmaf(ek2_2, r0_1_3_1, g2_23);
              g2_12 = fmaf(ek2_3, r0_1_3_1, g2_12);
              const float r0_1_4_0 = X * r1_0_4_0;
              g2_28 = fmaf(ek2_1, r0_1_4_0, g2_28);
              g2_24 = fmaf(ek2_2, r0_1_4_0, g2_24);
              g2_13 = fmaf(ek2_3, r0_1_4_0, g2_13);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g2_25 = fmaf(ek2_2, r0_2_0_3, g2_25);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g2_29 = fmaf(ek2_1, r0_2_1_2, g2_29);
              g2_26 = fmaf(ek2_2, r0_2_1_2, g2_26);
              g2_14 = fmaf(ek2_3, r0_2_1_2, g2_14);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g2_30 = fmaf(ek2_1, r0_2_2_1, g2_30);
              g2_27 = fmaf(ek2_2, r0_2_2_1, g2_27);
              g2_15 = fmaf(ek2_3, r0_2_2_1, g2_15);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g2_31 = fmaf(ek2_1, r0_2_3_0, g2_31);
              g2_28 = fmaf(ek2_2, r0_2_3_0, g2_28);
              g2_16 = fmaf(ek2_3, r0_2_3_0, g2_16);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g2_29 = fmaf(ek2_2, r0_3_0_2, g2_29);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g2_32 = fmaf(ek2_1, r0_3_1_1, g2_32);
              g2_30 = fmaf(ek2_2, r0_3_1_1, g2_30);
              g2_17 = fmaf(ek2_3, r0_3_1_1, g2_17);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g2_33 = fmaf(ek2_1, r0_3_2_0, g2_33);
              g2_31 = fmaf(ek2_2, r0_3_2_0, g2_31);
              g2_18 = fmaf(ek2_3, r0_3_2_0, g2_18);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g2_32 = fmaf(ek2_2, r0_4_0_1, g2_32);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g2_34 = fmaf(ek2_1, r0_4_1_0, g2_34);
              g2_33 = fmaf(ek2_2, r0_4_1_0, g2_33);
              g2_19 = fmaf(ek2_3, r0_4_1_0, g2_19);
              const float r4_1_0_0 = X * b5;
              const float r3_2_0_0 = fmaf(X, r4_1_0_0, b4);
              const float r2_3_0_0 = fmaf(X, r3_2_0_0, 2.0f * r3_1_0_0);
              const float r1_4_0_0 = fmaf(X, r2_3_0_0, 3.0f * r2_2_0_0);
              const float r0_5_0_0 = fmaf(X, r1_4_0_0, 4.0f * r1_3_0_0);
              g2_34 = fmaf(ek2_2, r0_5_0_0, g2_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_1_1_4 = X * r1_0_1_4;
              g2_20 = fmaf(ek2_3, r0_1_1_4, g2_20);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_1_2_3 = X * r1_0_2_3;
              g2_21 = fmaf(ek2_3, r0_1_2_3, g2_21);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_1_3_2 = X * r1_0_3_2;
              g2_22 = fmaf(ek2_3, r0_1_3_2, g2_22);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_1_4_1 = X * r1_0_4_1;
              g2_23 = fmaf(ek2_3, r0_1_4_1, g2_23);
              const float r5_0_1_0 = Y * b6;
              const float r4_0_2_0 = fmaf(Y, r5_0_1_0, b5);
              const float r3_0_3_0 = fmaf(Y, r4_0_2_0, 2.0f * r4_0_1_0);
              const float r2_0_4_0 = fmaf(Y, r3_0_3_0, 3.0f * r3_0_2_0);
              const float r1_0_5_0 = fmaf(Y, r2_0_4_0, 4.0f * r2_0_3_0);
              const float r0_1_5_0 = X * r1_0_5_0;
              g2_24 = fmaf(ek2_3, r0_1_5_0, g2_24);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g2_25 = fmaf(ek2_3, r0_2_1_3, g2_25);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g2_26 = fmaf(ek2_3, r0_2_2_2, g2_26);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g2_27 = fmaf(ek2_3, r0_2_3_1, g2_27);
              const float r1_1_4_0 = X * r2_0_4_0;
              const float r0_2_4_0 = fmaf(X, r1_1_4_0, r1_0_4_0);
              g2_28 = fmaf(ek2_3, r0_2_4_0, g2_28);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g2_29 = fmaf(ek2_3, r0_3_1_2, g2_29);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g2_30 = fmaf(ek2_3, r0_3_2_1, g2_30);
              const float r2_1_3_0 = X * r3_0_3_0;
              const float r1_2_3_0 = fmaf(X, r2_1_3_0, r2_0_3_0);
              const float r0_3_3_0 = fmaf(X, r1_2_3_0, 2.0f * r1_1_3_0);
              g2_31 = fmaf(ek2_3, r0_3_3_0, g2_31);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g2_32 = fmaf(ek2_3, r0_4_1_1, g2_32);
              const float r3_1_2_0 = X * r4_0_2_0;
              const float r2_2_2_0 = fmaf(X, r3_1_2_0, r3_0_2_0);
              const float r1_3_2_0 = fmaf(X, r2_2_2_0, 2.0f * r2_1_2_0);
              const float r0_4_2_0 = fmaf(X, r1_3_2_0, 3.0f * r1_2_2_0);
              g2_33 = fmaf(ek2_3, r0_4_2_0, g2_33);
              const float r4_1_1_0 = X * r5_0_1_0;
              const float r3_2_1_0 = fmaf(X, r4_1_1_0, r4_0_1_0);
              const float r2_3_1_0 = fmaf(X, r3_2_1_0, 2.0f * r3_1_1_0);
              const float r1_4_1_0 = fmaf(X, r2_3_1_0, 3.0f * r2_2_1_0);
              const float r0_5_1_0 = fmaf(X, r1_4_1_0, 4.0f * r1_3_1_0);
              g2_34 = fmaf(ek2_3, r0_5_1_0, g2_34);
            }
            { const float eb = bi[5];
              o0_2 = fmaf(eb, g2_0, o0_2);
            }
            { const float eb = bi[6];
              o0_2 = fmaf(eb, g2_3, o0_2);
            }
            { const float eb = bi[7];
              o0_2 = fmaf(eb, g2_9, o0_2);
            }
            { const float eb = bi[8];
              o0_2 = fmaf(eb, g2_19, o0_2);
            }
            { const float eb = bi[9];
              o0_2 = fmaf(eb, g2_34, o0_2);
            }
            { const float eb = bi[10];
              o1_2 = fmaf(eb, g2_0, o1_2);
            }
            { const float eb = bi[11];
              o1_2 = fmaf(eb, g2_2, o1_2);
            }
            { const float eb = bi[12];
              o1_2 = fmaf(eb, g2_6, o1_2);
            }
            { const float eb = bi[13];
              o1_2 = fmaf(eb, g2_3, o1_2);
            }
            { const float eb = bi[14];
              o1_2 = fmaf(eb, g2_8, o1_2);
            }
            { const float eb = bi[15];
              o1_2 = fmaf(eb, g2_16, o1_2);
            }
            { const float eb = bi[16];
              o1_2 = fmaf(eb, g2_9, o1_2);
            }
            { const float eb = bi[17];
              o1_2 = fmaf(eb, g2_18, o1_2);
            }
            { const float eb = bi[18];
              o1_2 = fmaf(eb, g2_31, o1_2);
            }
            { const float eb = bi[19];
              o2_2 = fmaf(eb, g2_0, o2_2);
            }
            { const float eb = bi[20];
              o2_2 = fmaf(eb, g2_1, o2_2);
            }
            { const float eb = bi[21];
              o2_2 = fmaf(eb, g2_4, o2_2);
            }
            { const float eb = bi[22];
              o2_2 = fmaf(eb, g2_3, o2_2);
            }
            { const float eb = bi[23];
              o2_2 = fmaf(eb, g2_7, o2_2);
            }
            { const float eb = bi[24];
              o2_2 = fmaf(eb, g2_14, o2_2);
            }
            { const float eb = bi[25];
              o2_2 = fmaf(eb, g2_9, o2_2);
            }
            { const float eb = bi[26];
              o2_2 = fmaf(eb, g2_17, o2_2);
            }
            { const float eb = bi[27];
              o2_2 = fmaf(eb, g2_29, o2_2);
            }
            { const float eb = bi[28];
              o3_2 = fmaf(eb, g2_0, o3_2);
            }
            { const float eb = bi[29];
              o3_2 = fmaf(eb, g2_2, o3_2);
            }
            { const float eb = bi[30];
              o3_2 = fmaf(eb, g2_3, o3_2);
            }
            { const float eb = bi[31];
              o3_2 = fmaf(eb, g2_8, o3_2);
            }
            { const float eb = bi[32];
              o3_2 = fmaf(eb, g2_9, o3_2);
            }
            { const float eb = bi[33];
              o3_2 = fmaf(eb, g2_18, o3_2);
            }
            { const float eb = bi[34];
              o3_2 = fmaf(eb, g2_19, o3_2);
            }
            { const float eb = bi[35];
              o3_2 = fmaf(eb, g2_33, o3_2);
            }
            { const float eb = bi[36];
              o4_2 = fmaf(eb, g2_0, o4_2);
            }
            { const float eb = bi[37];
              o4_2 = fmaf(eb, g2_1, o4_2);
            }
            { const float eb = bi[38];
              o4_2 = fmaf(eb, g2_3, o4_2);
            }
            { const float eb = bi[39];
              o4_2 = fmaf(eb, g2_7, o4_2);
            }
            { const float eb = bi[40];
              o4_2 = fmaf(eb, g2_9, o4_2);
            }
            { const float eb = bi[41];
              o4_2 = fmaf(eb, g2_17, o4_2);
            }
            { const float eb = bi[42];
              o4_2 = fmaf(eb, g2_19, o4_2);
            }
            { const float eb = bi[43];
              o4_2 = fmaf(eb, g2_32, o4_2);
            }
            { const float eb = bi[44];
              o5_2 = fmaf(eb, g2_0, o5_2);
            }
            { const float eb = bi[45];
              o5_2 = fmaf(eb, g2_1, o5_2);
            }
            { const float eb = bi[46];
              o5_2 = fmaf(eb, g2_2, o5_2);
            }
            { const float eb = bi[47];
              o5_2 = fmaf(eb, g2_5, o5_2);
            }
            { const float eb = bi[48];
              o5_2 = fmaf(eb, g2_3, o5_2);
            }
            { const float eb = bi[49];
              o5_2 = fmaf(eb, g2_7, o5_2);
            }
            { const float eb = bi[50];
              o5_2 = fmaf(eb, g2_8, o5_2);
            }
            { const float eb = bi[51];
              o5_2 = fmaf(eb, g2_15, o5_2);
            }
            { const float eb = bi[52];
              o5_2 = fmaf(eb, g2_9, o5_2);
            }
            { const float eb = bi[53];
              o5_2 = fmaf(eb, g2_17, o5_2);
            }
            { const float eb = bi[54];
              o5_2 = fmaf(eb, g2_18, o5_2);
            }
            { const float eb = bi[55];
              o5_2 = fmaf(eb, g2_30, o5_2);
            }
            { const float eb = bi[56];
              o6_2 = fmaf(eb, g2_0, o6_2);
            }
            { const float eb = bi[57];
              o6_2 = fmaf(eb, g2_2, o6_2);
            }
            { const float eb = bi[58];
              o6_2 = fmaf(eb, g2_6, o6_2);
            }
            { const float eb = bi[59];
              o6_2 = fmaf(eb, g2_3, o6_2);
            }
            { const float eb = bi[60];
              o6_2 = fmaf(eb, g2_8, o6_2);
            }
            { const float eb = bi[61];
              o6_2 = fmaf(eb, g2_16, o6_2);
            }
            { const float eb = bi[62];
              o6_2 = fmaf(eb, g2_9, o6_2);
            }
            { const float eb = bi[63];
              o6_2 = fmaf(eb, g2_18, o6_2);
            }
            { const float eb = bi[64];
              o6_2 = fmaf(eb, g2_31, o6_2);
            }
            { const float eb = bi[65];
              o7_2 = fmaf(eb, g2_0, o7_2);
            }
            { const float eb = bi[66];
              o7_2 = fmaf(eb, g2_2, o7_2);
            }
            { const float eb = bi[67];
              o7_2 = fmaf(eb, g2_6, o7_2);
            }
            { const float eb = bi[68];
              o7_2 = fmaf(eb, g2_13, o7_2);
            }
            { const float eb = bi[69];
              o7_2 = fmaf(eb, g2_24, o7_2);
            }
            { const float eb = bi[70];
              o8_2 = fmaf(eb, g2_0, o8_2);
            }
            { const float eb = bi[71];
              o8_2 = fmaf(eb, g2_1, o8_2);
            }
            { const float eb = bi[72];
              o8_2 = fmaf(eb, g2_4, o8_2);
            }
            { const float eb = bi[73];
              o8_2 = fmaf(eb, g2_2, o8_2);
            }
            { const float eb = bi[74];
              o8_2 = fmaf(eb, g2_5, o8_2);
            }
            { const float eb = bi[75];
              o8_2 = fmaf(eb, g2_11, o8_2);
            }
            { const float eb = bi[76];
              o8_2 = fmaf(eb, g2_6, o8_2);
            }
            { const float eb = bi[77];
              o8_2 = fmaf(eb, g2_12, o8_2);
            }
            { const float eb = bi[78];
              o8_2 = fmaf(eb, g2_22, o8_2);
            }
            { const float eb = bi[79];
              o9_2 = fmaf(eb, g2_0, o9_2);
            }
            { const float eb = bi[80];
              o9_2 = fmaf(eb, g2_2, o9_2);
            }
            { const float eb = bi[81];
              o9_2 = fmaf(eb, g2_6, o9_2);
            }
            { const float eb = bi[82];
              o9_2 = fmaf(eb, g2_13, o9_2);
            }
            { const float eb = bi[83];
              o9_2 = fmaf(eb, g2_3, o9_2);
            }
            { const float eb = bi[84];
              o9_2 = fmaf(eb, g2_8, o9_2);
            }
            { const float eb = bi[85];
              o9_2 = fmaf(eb, g2_16, o9_2);
            }
            { const float eb = bi[86];
              o9_2 = fmaf(eb, g2_28, o9_2);
            }
            { const float eb = bi[87];
              o10_2 = fmaf(eb, g2_0, o10_2);
            }
            { const float eb = bi[88];
              o10_2 = fmaf(eb, g2_1, o10_2);
            }
            { const float eb = bi[89];
              o10_2 = fmaf(eb, g2_2, o10_2);
            }
            { const float eb = bi[90];
              o10_2 = fmaf(eb, g2_5, o10_2);
            }
            { const float eb = bi[91];
              o10_2 = fmaf(eb, g2_6, o10_2);
            }
            { const float eb = bi[92];
              o10_2 = fmaf(eb, g2_12, o10_2);
            }
            { const float eb = bi[93];
              o10_2 = fmaf(eb, g2_3, o10_2);
            }
            { const float eb = bi[94];
              o10_2 = fmaf(eb, g2_7, o10_2);
            }
            { const float eb = bi[95];
              o10_2 = fmaf(eb, g2_8, o10_2);
            }
            { const float eb = bi[96];
              o10_2 = fmaf(eb, g2_15, o10_2);
            }
            { const float eb = bi[97];
              o10_2 = fmaf(eb, g2_16, o10_2);
            }
            { const float eb = bi[98];
              o10_2 = fmaf(eb, g2_27, o10_2);
            }
            { const float eb = bi[99];
              o11_2 = fmaf(eb, g2_0, o11_2);
            }
            { const float eb = bi[100];
              o11_2 = fmaf(eb, g2_1, o11_2);
            }
            { const float eb = bi[101];
              o11_2 = fmaf(eb, g2_2, o11_2);
            }
            { const float eb = bi[102];
              o11_2 = fmaf(eb, g2_5, o11_2);
            }
            { const float eb = bi[103];
              o11_2 = fmaf(eb, g2_6, o11_2);
            }
            { const float eb = bi[104];
              o11_2 = fmaf(eb, g2_12, o11_2);
            }
            { const float eb = bi[105];
              o11_2 = fmaf(eb, g2_13, o11_2);
            }
            { const float eb = bi[106];
              o11_2 = fmaf(eb, g2_23, o11_2);
            }
            { const float eb = bi[107];
              o12_2 = fmaf(eb, g2_0, o12_2);
            }
            { const float eb = bi[108];
              o12_2 = fmaf(eb, g2_1, o12_2);
            }
            { const float eb = bi[109];
              o12_2 = fmaf(eb, g2_4, o12_2);
            }
            { const float eb = bi[110];
              o12_2 = fmaf(eb, g2_3, o12_2);
            }
            { const float eb = bi[111];
              o12_2 = fmaf(eb, g2_7, o12_2);
            }
            { const float eb = bi[112];
              o12_2 = fmaf(eb, g2_14, o12_2);
            }
            { const float eb = bi[113];
              o12_2 = fmaf(eb, g2_9, o12_2);
            }
            { const float eb = bi[114];
              o12_2 = fmaf(eb, g2_17, o12_2);
            }
            { const float eb = bi[115];
              o12_2 = fmaf(eb, g2_29, o12_2);
            }
            { const float eb = bi[116];
              o13_2 = fmaf(eb, g2_0, o13_2);
            }
            { const float eb = bi[117];
              o13_2 = fmaf(eb, g2_1, o13_2);
            }
            { const float eb = bi[118];
              o13_2 = fmaf(eb, g2_4, o13_2);
            }
            { const float eb = bi[119];
              o13_2 = fmaf(eb, g2_2, o13_2);
            }
            { const float eb = bi[120];
              o13_2 = fmaf(eb, g2_5, o13_2);
            }
            { const float eb = bi[121];
              o13_2 = fmaf(eb, g2_11, o13_2);
            }
            { const float eb = bi[122];
              o13_2 = fmaf(eb, g2_6, o13_2);
            }
            { const float eb = bi[123];
              o13_2 = fmaf(eb, g2_12, o13_2);
            }
            { const float eb = bi[124];
              o13_2 = fmaf(eb, g2_22, o13_2);
            }
            { const float eb = bi[125];
              o14_2 = fmaf(eb, g2_0, o14_2);
            }
            { const float eb = bi[126];
              o14_2 = fmaf(eb, g2_1, o14_2);
            }
            { const float eb = bi[127];
              o14_2 = fmaf(eb, g2_4, o14_2);
            }
            { const float eb = bi[128];
              o14_2 = fmaf(eb, g2_10, o14_2);
            }
            { const float eb = bi[129];
              o14_2 = fmaf(eb, g2_20, o14_2);
            }
            { const float eb = bi[130];
              o15_2 = fmaf(eb, g2_0, o15_2);
            }
            { const float eb = bi[131];
              o15_2 = fmaf(eb, g2_1, o15_2);
            }
            { const float eb = bi[132];
              o15_2 = fmaf(eb, g2_4, o15_2);
            }
            { const float eb = bi[133];
              o15_2 = fmaf(eb, g2_2, o15_2);
            }
            { const float eb = bi[134];
              o15_2 = fmaf(eb, g2_5, o15_2);
            }
            { const float eb = bi[135];
              o15_2 = fmaf(eb, g2_11, o15_2);
            }
            { const float eb = bi[136];
              o15_2 = fmaf(eb, g2_3, o15_2);
            }
            { const float eb = bi[137];
              o15_2 = fmaf(eb, g2_7, o15_2);
            }
            { const float eb = bi[138];
              o15_2 = fmaf(eb, g2_14, o15_2);
            }
            { const float eb = bi[139];
              o15_2 = fmaf(eb, g2_8, o15_2);
            }
            { const float eb = bi[140];
              o15_2 = fmaf(eb, g2_15, o15_2);
            }
            { const float eb = bi[141];
              o15_2 = fmaf(eb, g2_26, o15_2);
            }
            { const float eb = bi[142];
              o16_2 = fmaf(eb, g2_0, o16_2);
            }
            { const float eb = bi[143];
              o16_2 = fmaf(eb, g2_1, o16_2);
            }
            { const float eb = bi[144];
              o16_2 = fmaf(eb, g2_4, o16_2);
            }
            { const float eb = bi[145];
              o16_2 = fmaf(eb, g2_10, o16_2);
            }
            { const float eb = bi[146];
              o16_2 = fmaf(eb, g2_3, o16_2);
            }
            { const float eb = bi[147];
              o16_2 = fmaf(eb, g2_7, o16_2);
            }
            { const float eb = bi[148];
              o16_2 = fmaf(eb, g2_14, o16_2);
            }
            { const float eb = bi[149];
              o16_2 = fmaf(eb, g2_25, o16_2);
            }
            { const float eb = bi[150];
              o17_2 = fmaf(eb, g2_0, o17_2);
            }
            { const float eb = bi[151];
              o17_2 = fmaf(eb, g2_1, o17_2);
            }
            { const float eb = bi[152];
              o17_2 = fmaf(eb, g2_4, o17_2);
            }
            { const float eb = bi[153];
              o17_2 = fmaf(eb, g2_10, o17_2);
            }
            { const float eb = bi[154];
              o17_2 = fmaf(eb, g2_2, o17_2);
            }
            { const float eb = bi[155];
              o17_2 = fmaf(eb, g2_5, o17_2);
            }
            { const float eb = bi[156];
              o17_2 = fmaf(eb, g2_11, o17_2);
            }
            { const float eb = bi[157];
              o17_2 = fmaf(eb, g2_21, o17_2);
            }
            { const float eb = bi[158];
              o18_2 = fmaf(eb, g2_0, o18_2);
            }
            { const float eb = bi[159];
              o18_2 = fmaf(eb, g2_2, o18_2);
            }
            { const float eb = bi[160];
              o18_2 = fmaf(eb, g2_3, o18_2);
            }
            { const float eb = bi[161];
              o18_2 = fmaf(eb, g2_8, o18_2);
            }
            { const float eb = bi[162];
              o18_2 = fmaf(eb, g2_9, o18_2);
            }
            { const float eb = bi[163];
              o18_2 = fmaf(eb, g2_18, o18_2);
            }
            { const float eb = bi[164];
              o18_2 = fmaf(eb, g2_19, o18_2);
            }
            { const float eb = bi[165];
              o18_2 = fmaf(eb, g2_33, o18_2);
            }
            { const float eb = bi[166];
              o19_2 = fmaf(eb, g2_0, o19_2);
            }
            { const float eb = bi[167];
              o19_2 = fmaf(eb, g2_2, o19_2);
            }
            { const float eb = bi[168];
              o19_2 = fmaf(eb, g2_6, o19_2);
            }
            { const float eb = bi[169];
              o19_2 = fmaf(eb, g2_13, o19_2);
            }
            { const float eb = bi[170];
              o19_2 = fmaf(eb, g2_3, o19_2);
            }
            { const float eb = bi[171];
              o19_2 = fmaf(eb, g2_8, o19_2);
            }
            { const float eb = bi[172];
              o19_2 = fmaf(eb, g2_16, o19_2);
            }
            { const float eb = bi[173];
              o19_2 = fmaf(eb, g2_28, o19_2);
            }
            { const float eb = bi[174];
              o20_2 = fmaf(eb, g2_0, o20_2);
            }
            { const float eb = bi[175];
              o20_2 = fmaf(eb, g2_1, o20_2);
            }
            { const float eb = bi[176];
              o20_2 = fmaf(eb, g2_4, o20_2);
            }
            { const float eb = bi[177];
              o20_2 = fmaf(eb, g2_2, o20_2);
            }
            { const float eb = bi[178];
              o20_2 = fmaf(eb, g2_5, o20_2);
            }
            { const float eb = bi[179];
              o20_2 = fmaf(eb, g2_11, o20_2);
            }
            { const float eb = bi[180];
              o20_2 = fmaf(eb, g2_3, o20_2);
            }
            { const float eb = bi[181];
              o20_2 = fmaf(eb, g2_7, o20_2);
            }
            { const float eb = bi[182];
              o20_2 = fmaf(eb, g2_14, o20_2);
            }
            { const float eb = bi[183];
              o20_2 = fmaf(eb, g2_8, o20_2);
            }
            { const float eb = bi[184];
              o20_2 = fmaf(eb, g2_15, o20_2);
            }
            { const float eb = bi[185];
              o20_2 = fmaf(eb, g2_26, o20_2);
            }
            { const float eb = bi[186];
              o21_2 = fmaf(eb, g2_0, o21_2);
            }
            { const float eb = bi[187];
              o21_2 = fmaf(eb, g2_2, o21_2);
            }
            { const float eb = bi[188];
              o21_2 = fmaf(eb, g2_6, o21_2);
            }
            { const float eb = bi[189];
              o21_2 = fmaf(eb, g2_3, o21_2);
            }
            { const float eb = bi[190];
              o21_2 = fmaf(eb, g2_8, o21_2);
            }
            { const float eb = bi[191];
              o21_2 = fmaf(eb, g2_16, o21_2);
            }
            { const float eb = bi[192];
              o21_2 = fmaf(eb, g2_9, o21_2);
            }
            { const float eb = bi[193];
              o21_2 = fmaf(eb, g2_18, o21_2);
            }
            { const float eb = bi[194];
              o21_2 = fmaf(eb, g2_31, o21_2);
            }
            { const float eb = bi[195];
              o22_2 = fmaf(eb, g2_0, o22_2);
            }
            { const float eb = bi[196];
              o22_2 = fmaf(eb, g2_1, o22_2);
            }
            { const float eb = bi[197];
              o22_2 = fmaf(eb, g2_2, o22_2);
            }
            { const float eb = bi[198];
              o22_2 = fmaf(eb, g2_5, o22_2);
            }
            { const float eb = bi[199];
              o22_2 = fmaf(eb, g2_3, o22_2);
            }
            { const float eb = bi[200];
              o22_2 = fmaf(eb, g2_7, o22_2);
            }
            { const float eb = bi[201];
              o22_2 = fmaf(eb, g2_8, o22_2);
            }
            { const float eb = bi[202];
              o22_2 = fmaf(eb, g2_15, o22_2);
            }
            { const float eb = bi[203];
              o22_2 = fmaf(eb, g2_9, o22_2);
            }
            { const float eb = bi[204];
              o22_2 = fmaf(eb, g2_17, o22_2);
            }
            { const float eb = bi[205];
              o22_2 = fmaf(eb, g2_18, o22_2);
            }
            { const float eb = bi[206];
              o22_2 = fmaf(eb, g2_30, o22_2);
            }
            { const float eb = bi[207];
              o23_2 = fmaf(eb, g2_0, o23_2);
            }
            { const float eb = bi[208];
              o23_2 = fmaf(eb, g2_1, o23_2);
            }
            { const float eb = bi[209];
              o23_2 = fmaf(eb, g2_2, o23_2);
            }
            { const float eb = bi[210];
              o23_2 = fmaf(eb, g2_5, o23_2);
            }
            { const float eb = bi[211];
              o23_2 = fmaf(eb, g2_6, o23_2);
            }
            { const float eb = bi[212];
              o23_2 = fmaf(eb, g2_12, o23_2);
            }
            { const float eb = bi[213];
              o23_2 = fmaf(eb, g2_3, o23_2);
            }
            { const float eb = bi[214];
              o23_2 = fmaf(eb, g2_7, o23_2);
            }
            { const float eb = bi[215];
              o23_2 = fmaf(eb, g2_8, o23_2);
            }
            { const float eb = bi[216];
              o23_2 = fmaf(eb, g2_15, o23_2);
            }
            { const float eb = bi[217];
              o23_2 = fmaf(eb, g2_16, o23_2);
            }
            { const float eb = bi[218];
              o23_2 = fmaf(eb, g2_27, o23_2);
            }
            { const float eb = bi[219];
              o24_2 = fmaf(eb, g2_0, o24_2);
            }
            { const float eb = bi[220];
              o24_2 = fmaf(eb, g2_1, o24_2);
            }
            { const float eb = bi[221];
              o24_2 = fmaf(eb, g2_3, o24_2);
            }
            { const float eb = bi[222];
              o24_2 = fmaf(eb, g2_7, o24_2);
            }
            { const float eb = bi[223];
              o24_2 = fmaf(eb, g2_9, o24_2);
            }
            { const float eb = bi[224];
              o24_2 = fmaf(eb, g2_17, o24_2);
            }
            { const float eb = bi[225];
              o24_2 = fmaf(eb, g2_19, o24_2);
            }
            { const float eb = bi[226];
              o24_2 = fmaf(eb, g2_32, o24_2);
            }
            { const float eb = bi[227];
              o25_2 = fmaf(eb, g2_0, o25_2);
            }
            { const float eb = bi[228];
              o25_2 = fmaf(eb, g2_1, o25_2);
            }
            { const float eb = bi[229];
              o25_2 = fmaf(eb, g2_2, o25_2);
            }
            { const float eb = bi[230];
              o25_2 = fmaf(eb, g2_5, o25_2);
            }
            { const float eb = bi[231];
              o25_2 = fmaf(eb, g2_6, o25_2);
            }
            { const float eb = bi[232];
              o25_2 = fmaf(eb, g2_12, o25_2);
            }
            { const float eb = bi[233];
              o25_2 = fmaf(eb, g2_3, o25_2);
            }
            { const float eb = bi[234];
              o25_2 = fmaf(eb, g2_7, o25_2);
            }
            { const float eb = bi[235];
              o25_2 = fmaf(eb, g2_8, o25_2);
            }
            { const float eb = bi[236];
              o25_2 = fmaf(eb, g2_15, o25_2);
            }
            { const float eb = bi[237];
              o25_2 = fmaf(eb, g2_16, o25_2);
            }
            { const float eb = bi[238];
              o25_2 = fmaf(eb, g2_27, o25_2);
            }
            { const float eb = bi[239];
              o26_2 = fmaf(eb, g2_0, o26_2);
            }
            { const float eb = bi[240];
              o26_2 = fmaf(eb, g2_1, o26_2);
            }
            { const float eb = bi[241];
              o26_2 = fmaf(eb, g2_4, o26_2);
            }
            { const float eb = bi[242];
              o26_2 = fmaf(eb, g2_10, o26_2);
            }
            { const float eb = bi[243];
              o26_2 = fmaf(eb, g2_3, o26_2);
            }
            { const float eb = bi[244];
              o26_2 = fmaf(eb, g2_7, o26_2);
            }
            { const float eb = bi[245];
              o26_2 = fmaf(eb, g2_14, o26_2);
            }
            { const float eb = bi[246];
              o26_2 = fmaf(eb, g2_25, o26_2);
            }
            { const float eb = bi[247];
              o27_2 = fmaf(eb, g2_0, o27_2);
            }
            { const float eb = bi[248];
              o27_2 = fmaf(eb, g2_1, o27_2);
            }
            { const float eb = bi[249];
              o27_2 = fmaf(eb, g2_2, o27_2);
            }
            { const float eb = bi[250];
              o27_2 = fmaf(eb, g2_5, o27_2);
            }
            { const float eb = bi[251];
              o27_2 = fmaf(eb, g2_3, o27_2);
            }
            { const float eb = bi[252];
              o27_2 = fmaf(eb, g2_7, o27_2);
            }
            { const float eb = bi[253];
              o27_2 = fmaf(eb, g2_8, o27_2);
            }
            { const float eb = bi[254];
              o27_2 = fmaf(eb, g2_15, o27_2);
            }
            { const float eb = bi[255];
              o27_2 = fmaf(eb, g2_9, o27_2);
            }
            { const float eb = bi[256];
              o27_2 = fmaf(eb, g2_17, o27_2);
            }
            { const float eb = bi[257];
              o27_2 = fmaf(eb, g2_18, o27_2);
            }
            { const float eb = bi[258];
              o27_2 = fmaf(eb, g2_30, o27_2);
            }
            { const float eb = bi[259];
              o28_2 = fmaf(eb, g2_0, o28_2);
            }
            { const float eb = bi[260];
              o28_2 = fmaf(eb, g2_1, o28_2);
            }
            { const float eb = bi[261];
              o28_2 = fmaf(eb, g2_4, o28_2);
            }
            { const float eb = bi[262];
              o28_2 = fmaf(eb, g2_3, o28_2);
            }
            { const float eb = bi[263];
              o28_2 = fmaf(eb, g2_7, o28_2);
            }
            { const float eb = bi[264];
              o28_2 = fmaf(eb, g2_14, o28_2);
            }
            { const float eb = bi[265];
              o28_2 = fmaf(eb, g2_9, o28_2);
            }
            { const float eb = bi[266];
              o28_2 = fmaf(eb, g2_17, o28_2);
            }
            { const float eb = bi[267];
              o28_2 = fmaf(eb, g2_29, o28_2);
            }
            { const float eb = bi[268];
              o29_2 = fmaf(eb, g2_0, o29_2);
            }
            { const float eb = bi[269];
              o29_2 = fmaf(eb, g2_1, o29_2);
            }
            { const float eb = bi[270];
              o29_2 = fmaf(eb, g2_4, o29_2);
            }
            { const float eb = bi[271];
              o29_2 = fmaf(eb, g2_2, o29_2);
            }
            { const float eb = bi[272];
              o29_2 = fmaf(eb, g2_5, o29_2);
            }
            { const float eb = bi[273];
              o29_2 = fmaf(eb, g2_11, o29_2);
            }
            { const float eb = bi[274];
              o29_2 = fmaf(eb, g2_3, o29_2);
            }
            { const float eb = bi[275];
              o29_2 = fmaf(eb, g2_7, o29_2);
            }
            { const float eb = bi[276];
              o29_2 = fmaf(eb, g2_14, o29_2);
            }
            { const float eb = bi[277];
              o29_2 = fmaf(eb, g2_8, o29_2);
            }
            { const float eb = bi[278];
              o29_2 = fmaf(eb, g2_15, o29_2);
            }
            { const float eb = bi[279];
              o29_2 = fmaf(eb, g2_26, o29_2);
            }
            { const float eb = bi[280];
              o30_2 = fmaf(eb, g2_0, o30_2);
            }
            { const float eb = bi[281];
              o30_2 = fmaf(eb, g2_1, o30_2);
            }
            { const float eb = bi[282];
              o30_2 = fmaf(eb, g2_2, o30_2);
            }
            { const float eb = bi[283];
              o30_2 = fmaf(eb, g2_5, o30_2);
            }
            { const float eb = bi[284];
              o30_2 = fmaf(eb, g2_3, o30_2);
            }
            { const float eb = bi[285];
              o30_2 = fmaf(eb, g2_7, o30_2);
            }
            { const float eb = bi[286];
              o30_2 = fmaf(eb, g2_8, o30_2);
            }
            { const float eb = bi[287];
              o30_2 = fmaf(eb, g2_15, o30_2);
            }
            { const float eb = bi[288];
              o30_2 = fmaf(eb, g2_9, o30_2);
            }
            { const float eb = bi[289];
              o30_2 = fmaf(eb, g2_17, o30_2);
            }
            { const float eb = bi[290];
              o30_2 = fmaf(eb, g2_18, o30_2);
            }
            { const float eb = bi[291];
              o30_2 = fmaf(eb, g2_30, o30_2);
            }
            { const float eb = bi[292];
              o31_2 = fmaf(eb, g2_0, o31_2);
            }
            { const float eb = bi[293];
              o31_2 = fmaf(eb, g2_1, o31_2);
            }
            { const float eb = bi[294];
              o31_2 = fmaf(eb, g2_2, o31_2);
            }
            { const float eb = bi[295];
              o31_2 = fmaf(eb, g2_5, o31_2);
            }
            { const float eb = bi[296];
              o31_2 = fmaf(eb, g2_6, o31_2);
            }
            { const float eb = bi[297];
              o31_2 = fmaf(eb, g2_12, o31_2);
            }
            { const float eb = bi[298];
              o31_2 = fmaf(eb, g2_13, o31_2);
            }
            { const float eb = bi[299];
              o31_2 = fmaf(eb, g2_23, o31_2);
            }
            { const float eb = bi[300];
              o32_2 = fmaf(eb, g2_0, o32_2);
            }
            { const float eb = bi[301];
              o32_2 = fmaf(eb, g2_1, o32_2);
            }
            { const float eb = bi[302];
              o32_2 = fmaf(eb, g2_4, o32_2);
            }
            { const float eb = bi[303];
              o32_2 = fmaf(eb, g2_10, o32_2);
            }
            { const float eb = bi[304];
              o32_2 = fmaf(eb, g2_2, o32_2);
            }
            { const float eb = bi[305];
              o32_2 = fmaf(eb, g2_5, o32_2);
            }
            { const float eb = bi[306];
              o32_2 = fmaf(eb, g2_11, o32_2);
            }
            { const float eb = bi[307];
              o32_2 = fmaf(eb, g2_21, o32_2);
            }
            { const float eb = bi[308];
              o33_2 = fmaf(eb, g2_0, o33_2);
            }
            { const float eb = bi[309];
              o33_2 = fmaf(eb, g2_1, o33_2);
            }
            { const float eb = bi[310];
              o33_2 = fmaf(eb, g2_2, o33_2);
            }
            { const float eb = bi[311];
              o33_2 = fmaf(eb, g2_5, o33_2);
            }
            { const float eb = bi[312];
              o33_2 = fmaf(eb, g2_6, o33_2);
            }
            { const float eb = bi[313];
              o33_2 = fmaf(eb, g2_12, o33_2);
            }
            { const float eb = bi[314];
              o33_2 = fmaf(eb, g2_3, o33_2);
            }
            { const float eb = bi[315];
              o33_2 = fmaf(eb, g2_7, o33_2);
            }
            { const float eb = bi[316];
              o33_2 = fmaf(eb, g2_8, o33_2);
            }
            { const float eb = bi[317];
              o33_2 = fmaf(eb, g2_15, o33_2);
            }
            { const float eb = bi[318];
              o33_2 = fmaf(eb, g2_16, o33_2);
            }
            { const float eb = bi[319];
              o33_2 = fmaf(eb, g2_27, o33_2);
            }
            { const float eb = bi[320];
              o34_2 = fmaf(eb, g2_0, o34_2);
            }
            { const float eb = bi[321];
              o34_2 = fmaf(eb, g2_1, o34_2);
            }
            { const float eb = bi[322];
              o34_2 = fmaf(eb, g2_4, o34_2);
            }
            { const float eb = bi[323];
              o34_2 = fmaf(eb, g2_2, o34_2);
            }
            { const float eb = bi[324];
              o34_2 = fmaf(eb, g2_5, o34_2);
            }
            { const float eb = bi[325];
              o34_2 = fmaf(eb, g2_11, o34_2);
            }
            { const float eb = bi[326];
              o34_2 = fmaf(eb, g2_3, o34_2);
            }
            { const float eb = bi[327];
              o34_2 = fmaf(eb, g2_7, o34_2);
            }
            { const float eb = bi[328];
              o34_2 = fmaf(eb, g2_14, o34_2);
            }
            { const float eb = bi[329];
              o34_2 = fmaf(eb, g2_8, o34_2);
            }
            { const float eb = bi[330];
              o34_2 = fmaf(eb, g2_15, o34_2);
            }
            { const float eb = bi[331];
              o34_2 = fmaf(eb, g2_26, o34_2);
            }
            { const float eb = bi[332];
              o35_2 = fmaf(eb, g2_0, o35_2);
            }
            { const float eb = bi[333];
              o35_2 = fmaf(eb, g2_1, o35_2);
            }
            { const float eb = bi[334];
              o35_2 = fmaf(eb, g2_4, o35_2);
            }
            { const float eb = bi[335];
              o35_2 = fmaf(eb, g2_2, o35_2);
            }
            { const float eb = bi[336];
              o35_2 = fmaf(eb, g2_5, o35_2);
            }
            { const float eb = bi[337];
              o35_2 = fmaf(eb, g2_11, o35_2);
            }
            { const float eb = bi[338];
              o35_2 = fmaf(eb, g2_6, o35_2);
            }
            { const float eb = bi[339];
              o35_2 = fmaf(eb, g2_12, o35_2);
            }
            { const float eb = bi[340];
              o35_2 = fmaf(eb, g2_22, o35_2);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk2 = PT[(fI + 0) * N + fJ + 2];
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
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd4_2 = PA[(fQ + 4) * N + fJ + 2];
            const double Abd5_2 = PA[(fQ + 5) * N + fJ + 2];
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
            const double Abc4_0 = PA[(fQ + 4) * N + fI + 0];
            const double Abc5_0 = PA[(fQ + 5) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 2, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5 + o6_2 * ptb6 + o7_2 * ptb7 + o8_2 * ptb8 + o9_2 * ptb9 + o10_2 * ptb10 + o11_2 * ptb11 + o12_2 * ptb12 + o13_2 * ptb13 + o14_2 * ptb14 + o15_2 * ptb15 + o16_2 * ptb16 + o17_2 * ptb17 + o18_2 * ptb18 + o19_2 * ptb19 + o20_2 * ptb20 + o21_2 * ptb21 + o22_2 * ptb22 + o23_2 * ptb23 + o24_2 * ptb24 + o25_2 * ptb25 + o26_2 * ptb26 + o27_2 * ptb27 + o28_2 * ptb28 + o29_2 * ptb29 + o30_2 * ptb30 + o31_2 * ptb31 + o32_2 * ptb32 + o33_2 * ptb33 + o34_2 * ptb34 + o35_2 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_2 * Abd0_2 + o1_2 * Abd1_2 + o2_2 * Abd2_2 + o3_2 * Abd3_2 + o4_2 * Abd4_2 + o5_2 * Abd5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_2 * Aad0_2 + o6_2 * Aad1_2 + o12_2 * Aad2_2 + o18_2 * Aad3_2 + o24_2 * Aad4_2 + o30_2 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_2 * Abc0_0 + o1_2 * Abc1_0 + o2_2 * Abc2_0 + o3_2 * Abc3_0 + o4_2 * Abc4_0 + o5_2 * Abc5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_2 * Aac0_0 + o6_2 * Aac1_0 + o12_2 * Aac2_0 + o18_2 * Aac3_0 + o24_2 * Aac4_0 + o30_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_2 * Aad0_2 + o7_2 * Aad1_2 + o13_2 * Aad2_2 + o19_2 * Aad3_2 + o25_2 * Aad4_2 + o31_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_2 * Aac0_0 + o7_2 * Aac1_0 + o13_2 * Aac2_0 + o19_2 * Aac3_0 + o25_2 * Aac4_0 + o31_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_2 * Aad0_2 + o8_2 * Aad1_2 + o14_2 * Aad2_2 + o20_2 * Aad3_2 + o26_2 * Aad4_2 + o32_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_2 * Aac0_0 + o8_2 * Aac1_0 + o14_2 * Aac2_0 + o20_2 * Aac3_0 + o26_2 * Aac4_0 + o32_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_2 * Aad0_2 + o9_2 * Aad1_2 + o15_2 * Aad2_2 + o21_2 * Aad3_2 + o27_2 * Aad4_2 + o33_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_2 * Aac0_0 + o9_2 * Aac1_0 + o15_2 * Aac2_0 + o21_2 * Aac3_0 + o27_2 * Aac4_0 + o33_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 0, deg * (o4_2 * Aad0_2 + o10_2 * Aad1_2 + o16_2 * Aad2_2 + o22_2 * Aad3_2 + o28_2 * Aad4_2 + o34_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 2, deg * (o4_2 * Aac0_0 + o10_2 * Aac1_0 + o16_2 * Aac2_0 + o22_2 * Aac3_0 + o28_2 * Aac4_0 + o34_2 * Aac5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 0, deg * (o5_2 * Aad0_2 + o11_2 * Aad1_2 + o17_2 * Aad2_2 + o23_2 * Aad3_2 + o29_2 * Aad4_2 + o35_2 * Aad5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 2, deg * (o5_2 * Aac0_0 + o11_2 * Aac1_0 + o17_2 * Aac2_0 + o23_2 * Aac3_0 + o29_2 * Aac4_0 + o35_2 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o6_2 * Abd0_2 + o7_2 * Abd1_2 + o8_2 * Abd2_2 + o9_2 * Abd3_2 + o10_2 * Abd4_2 + o11_2 * Abd5_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o6_2 * Abc0_0 + o7_2 * Abc1_0 + o8_2 * Abc2_0 + o9_2 * Abc3_0 + o10_2 * Abc4_0 + o11_2 * Abc5_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o12_2 * Abd0_2 + o13_2 * Abd1_2 + o14_2 * Abd2_2 + o15_2 * Abd3_2 + o16_2 * Abd4_2 + o17_2 * Abd5_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o12_2 * Abc0_0 + o13_2 * Abc1_0 + o14_2 * Abc2_0 + o15_2 * Abc3_0 + o16_2 * Abc4_0 + o17_2 * Abc5_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o18_2 * Abd0_2 + o19_2 * Abd1_2 + o20_2 * Abd2_2 + o21_2 * Abd3_2 + o22_2 * Abd4_2 + o23_2 * Abd5_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o18_2 * Abc0_0 + o19_2 * Abc1_0 + o20_2 * Abc2_0 + o21_2 * Abc3_0 + o22_2 * Abc4_0 + o23_2 * Abc5_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o24_2 * Abd0_2 + o25_2 * Abd1_2 + o26_2 * Abd2_2 + o27_2 * Abd3_2 + o28_2 * Abd4_2 + o29_2 * Abd5_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o24_2 * Abc0_0 + o25_2 * Abc1_0 + o26_2 * Abc2_0 + o27_2 * Abc3_0 + o28_2 * Abc4_0 + o29_2 * Abc5_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o30_2 * Abd0_2 + o31_2 * Abd1_2 + o32_2 * Abd2_2 + o33_2 * Abd3_2 + o34_2 * Abd4_2 + o35_2 * Abd5_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o30_2 * Abc0_0 + o31_2 * Abc1_0 + o32_2 * Abc2_0 + o33_2 * Abc3_0 + o34_2 * Abc4_0 + o35_2 * Abc5_0));
          }
        } break;
        case 3: {  // ket functions [3]
          float o0_3 = 0;
          float o1_3 = 0;
          float o2_3 = 0;
          float o3_3 = 0;
          float o4_3 = 0;
          float o5_3 = 0;
          float o6_3 = 0;
          float o7_3 = 0;
          float o8_3 = 0;
          float o9_3 = 0;
          float o10_3 = 0;
          float o11_3 = 0;
          float o12_3 = 0;
          float o13_3 = 0;
          float o14_3 = 0;
          float o15_3 = 0;
          float o16_3 = 0;
          float o17_3 = 0;
          float o18_3 = 0;
          float o19_3 = 0;
          float o20_3 = 0;
          float o21_3 = 0;
          float o22_3 = 0;
          float o23_3 = 0;
          float o24_3 = 0;
          float o25_3 = 0;
          float o26_3 = 0;
          float o27_3 = 0;
          float o28_3 = 0;
          float o29_3 = 0;
          float o30_3 = 0;
          float o31_3 = 0;
          float o32_3 = 0;
          float o33_3 = 0;
          float o34_3 = 0;
          float o35_3 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            float g3_10 = 0;
            float g3_11 = 0;
            float g3_12 = 0;
            float g3_13 = 0;
            float g3_14 = 0;
            float g3_15 = 0;
            float g3_16 = 0;
            float g3_17 = 0;
            float g3_18 = 0;
            float g3_19 = 0;
            float g3_20 = 0;
            float g3_21 = 0;
            float g3_22 = 0;
            float g3_23 = 0;
            float g3_24 = 0;
            float g3_25 = 0;
            float g3_26 = 0;
            float g3_27 = 0;
            float g3_28 = 0;
            float g3_29 = 0;
            float g3_30 = 0;
            float g3_31 = 0;
            float g3_32 = 0;
            float g3_33 = 0;
            float g3_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek3_0 = kj[14 * kS];
              const float ek3_1 = -kj[15 * kS];
              const float ek3_2 = -kj[16 * kS];
              const float ek3_3 = kj[17 * kS];
              g3_0 = fmaf(ek3_0, b0, g3_0);
              const float r0_0_0_1 = Z * b1;
              g3_1 = fmaf(ek3_0, r0_0_0_1, g3_1);
              g3_0 = fmaf(ek3_1, r0_0_0_1, g3_0);
              const float r0_0_1_0 = Y * b1;
              g3_2 = fmaf(ek3_0, r0_0_1_0, g3_2);
              const float r0_1_0_0 = X * b1;
              g3_3 = fmaf(ek3_0, r0_1_0_0, g3_3);
              g3_0 = fmaf(ek3_2, r0_1_0_0, g3_0);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g3_4 = fmaf(ek3_0, r0_0_0_2, g3_4);
              g3_1 = fmaf(ek3_1, r0_0_0_2, g3_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g3_5 = fmaf(ek3_0, r0_0_1_1, g3_5);
              g3_2 = fmaf(ek3_1, r0_0_1_1, g3_2);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g3_6 = fmaf(ek3_0, r0_0_2_0, g3_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g3_7 = fmaf(ek3_0, r0_1_0_1, g3_7);
              g3_3 = fmaf(ek3_1, r0_1_0_1, g3_3);
              g3_1 = fmaf(ek3_2, r0_1_0_1, g3_1);
              g3_0 = fmaf(ek3_3, r0_1_0_1, g3_0);
              const float r0_1_1_0 = X * r1_0_1_0;
              g3_8 = fmaf(ek3_0, r0_1_1_0, g3_8);
              g3_2 = fmaf(ek3_2, r0_1_1_0, g3_2);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g3_9 = fmaf(ek3_0, r0_2_0_0, g3_9);
              g3_3 = fmaf(ek3_2, r0_2_0_0, g3_3);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g3_10 = fmaf(ek3_0, r0_0_0_3, g3_10);
              g3_4 = fmaf(ek3_1, r0_0_0_3, g3_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g3_11 = fmaf(ek3_0, r0_0_1_2, g3_11);
              g3_5 = fmaf(ek3_1, r0_0_1_2, g3_5);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g3_12 = fmaf(ek3_0, r0_0_2_1, g3_12);
              g3_6 = fmaf(ek3_1, r0_0_2_1, g3_6);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g3_13 = fmaf(ek3_0, r0_0_3_0, g3_13);
              const float r0_1_0_2 = X * r1_0_0_2;
              g3_14 = fmaf(ek3_0, r0_1_0_2, g3_14);
              g3_7 = fmaf(ek3_1, r0_1_0_2, g3_7);
              g3_4 = fmaf(ek3_2, r0_1_0_2, g3_4);
              g3_1 = fmaf(ek3_3, r0_1_0_2, g3_1);
              const float r0_1_1_1 = X * r1_0_1_1;
              g3_15 = fmaf(ek3_0, r0_1_1_1, g3_15);
              g3_8 = fmaf(ek3_1, r0_1_1_1, g3_8);
              g3_5 = fmaf(ek3_2, r0_1_1_1, g3_5);
              g3_2 = fmaf(ek3_3, r0_1_1_1, g3_2);
              const float r0_1_2_0 = X * r1_0_2_0;
              g3_16 = fmaf(ek3_0, r0_1_2_0, g3_16);
              g3_6 = fmaf(ek3_2, r0_1_2_0, g3_6);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g3_17 = fmaf(ek3_0, r0_2_0_1, g3_17);
              g3_9 = fmaf(ek3_1, r0_2_0_1, g3_9);
              g3_7 = fmaf(ek3_2, r0_2_0_1, g3_7);
              g3_3 = fmaf(ek3_3, r0_2_0_1, g3_3);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g3_18 = fmaf(ek3_0, r0_2_1_0, g3_18);
              g3_8 = fmaf(ek3_2, r0_2_1_0, g3_8);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g3_19 = fmaf(ek3_0, r0_3_0_0, g3_19);
              g3_9 = fmaf(ek3_2, r0_3_0_0, g3_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g3_20 = fmaf(ek3_0, r0_0_0_4, g3_20);
              g3_10 = fmaf(ek3_1, r0_0_0_4, g3_10);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g3_21 = fmaf(ek3_0, r0_0_1_3, g3_21);
              g3_11 = fmaf(ek3_1, r0_0_1_3, g3_11);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g3_22 = fmaf(ek3_0, r0_0_2_2, g3_22);
              g3_12 = fmaf(ek3_1, r0_0_2_2, g3_12);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g3_23 = fmaf(ek3_0, r0_0_3_1, g3_23);
              g3_13 = fmaf(ek3_1, r0_0_3_1, g3_13);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g3_24 = fmaf(ek3_0, r0_0_4_0, g3_24);
              const float r0_1_0_3 = X * r1_0_0_3;
              g3_25 = fmaf(ek3_0, r0_1_0_3, g3_25);
              g3_14 = fmaf(ek3_1, r0_1_0_3, g3_14);
              g3_10 = fmaf(ek3_2, r0_1_0_3, g3_10);
              g3_4 = fmaf(ek3_3, r0_1_0_3, g3_4);
              const float r0_1_1_2 = X * r1_0_1_2;
              g3_26 = fmaf(ek3_0, r0_1_1_2, g3_26);
              g3_15 = fmaf(ek3_1, r0_1_1_2, g3_15);
              g3_11 = fmaf(ek3_2, r0_1_1_2, g3_11);
              g3_5 = fmaf(ek3_3, r0_1_1_2, g3_5);
              const float r0_1_2_1 = X * r1_0_2_1;
              g3_27 = fmaf(ek3_0, r0_1_2_1, g3_27);
              g3_16 = fmaf(ek3_1, r0_1_2_1, g3_16);
              g3_12 = fmaf(ek3_2, r0_1_2_1, g3_12);
              g3_6 = fmaf(ek3_3, r0_1_2_1, g3_6);
              const float r0_1_3_0 = X * r1_0_3_0;
              g3_28 = fmaf(ek3_0, r0_1_3_0, g3_28);
              g3_13 = fmaf(ek3_2, r0_1_3_0, g3_13);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g3_29 = fmaf(ek3_0, r0_2_0_2, g3_29);
              g3_17 = fmaf(ek3_1, r0_2_0_2, g3_17);
              g3_14 = fmaf(ek3_2, r0_2_0_2, g3_14);
              g3_7 = fmaf(ek3_3, r0_2_0_2, g3_7);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g3_30 = fmaf(ek3_0, r0_2_1_1, g3_30);
              g3_18 = fmaf(ek3_1, r0_2_1_1, g3_18);
              g3_15 = fmaf(ek3_2, r0_2_1_1, g3_15);
              g3_8 = fmaf(ek3_3, r0_2_1_1, g3_8);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g3_31 = fmaf(ek3_0, r0_2_2_0, g3_31);
              g3_16 = fmaf(ek3_2, r0_2_2_0, g3_16);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g3_32 = fmaf(ek3_0, r0_3_0_1, g3_32);
              g3_19 = fmaf(ek3_1, r0_3_0_1, g3_19);
              g3_17 = fmaf(ek3_2, r0_3_0_1, g3_17);
              g3_9 = fmaf(ek3_3, r0_3_0_1, g3_9);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g3_33 = fmaf(ek3_0, r0_3_1_0, g3_33);
              g3_18 = fmaf(ek3_2, r0_3_1_0, g3_18);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g3_34 = fmaf(ek3_0, r0_4_0_0, g3_34);
              g3_19 = fmaf(ek3_2, r0_4_0_0, g3_19);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_0_5 = fmaf(Z, r1_0_0_4, 4.0f * r1_0_0_3);
              g3_20 = fmaf(ek3_1, r0_0_0_5, g3_20);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g3_21 = fmaf(ek3_1, r0_0_1_4, g3_21);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g3_22 = fmaf(ek3_1, r0_0_2_3, g3_22);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g3_23 = fmaf(ek3_1, r0_0_3_2, g3_23);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g3_24 = fmaf(ek3_1, r0_0_4_1, g3_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g3_25 = fmaf(ek3_1, r0_1_0_4, g3_25);
              g3_20 = fmaf(ek3_2, r0_1_0_4, g3_20);
              g3_10 = fmaf(ek3_3, r0_1_0_4, g3_10);
              const float r0_1_1_3 = X * r1_0_1_3;
              g3_26 = fmaf(ek3_1, r0_1_1_3, g3_26);
              g3_21 = fmaf(ek3_2, r0_1_1_3, g3_21);
              g3_11 = fmaf(ek3_3, r0_1_1_3, g3_11);
              const float r0_1_2_2 = X * r1_0_2_2;
              g3_27 = fmaf(ek3_1, r0_1_2_2, g3_27);
              g3_22 = fmaf(ek3_2, r0_1_2_2, g3_22);
              g3_12 = fmaf(ek3_3, r0_1_2_2, g3_12);
              const float r0_1_3_1 = X * r1_0_3_1;
              g3_28 = fmaf(ek3_1, r0_1_3_1, g3_28);
              g3_23 = fmaf(ek3_2, r0_1_3_1, g3_23);
              g3_13 = fmaf(ek3_3, r0_1_3_1, g3_13);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_1_4_0 = X * r1_0_4_0;
              g3_24 = fmaf(ek3_2, r0_1_4_0, g3_24);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g3_29 = fmaf(ek3_1, r0_2_0_3, g3_29);
              g3_25 = fmaf(ek3_2, r0_2_0_3, g3_25);
              g3_14 = fmaf(ek3_3, r0_2_0_3, g3_14);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g3_30 = fmaf(ek3_1, r0_2_1_2, g3_30);
              g3_26 = fmaf(ek3_2, r0_2_1_2, g3_26);
              g3_15 = fmaf(ek3_3, r0_2_1_2, g3_15);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g3_31 = fmaf(ek3_1, r0_2_2_1, g3_31);
              g3_27 = fmaf(ek3_2, r0_2_2_1, g3_27);
              g3_16 = fmaf(ek3_3, r0_2_2_1, g3_16);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g3_28 = fmaf(ek3_2, r0_2_3_0, g3_28);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g3_32 = fmaf(ek3_1, r0_3_0_2, g3_32);
              g3_29 = fmaf(ek3_2, r0_3_0_2, g3_29);
              g3_17 = fmaf(ek3_3, r0_3_0_2, g3_17);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g3_33 = fmaf(ek3_1, r0_3_1_1, g3_33);
              g3_30 = fmaf(ek3_2, r0_3_1_1, g3_30);
              g3_18 = fmaf(ek3_3, r0_3_1_1, g3_18);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g3_31 = fmaf(ek3_2, r0_3_2_0, g3_31);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g3_34 = fmaf(ek3_1, r0_4_0_1, g3_34);
              g3_32 = fmaf(ek3_2, r0_4_0_1, g3_32);
              g3_19 = fmaf(ek3_3, r0_4_0_1, g3_19);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g3_33 = fmaf(ek3_2, r0_4_1_0, g3_33);
              const float r4_1_0_0 = X * b5;
              const float r3_2_0_0 = fmaf(X, r4_1_0_0, b4);
              const float r2_3_0_0 = fmaf(X, r3_2_0_0, 2.0f * r3_1_0_0);
              const float r1_4_0_0 = fmaf(X, r2_3_0_0, 3.0f * r2_2_0_0);
              const float r0_5_0_0 = fmaf(X, r1_4_0_0, 4.0f * r1_3_0_0);
              g3_34 = fmaf(ek3_2, r0_5_0_0, g3_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_0_5 = fmaf(Z, r2_0_0_4, 4.0f * r2_0_0_3);
              const float r0_1_0_5 = X * r1_0_0_5;
              g3_20 = fmaf(ek3_3, r0_1_0_5, g3_20);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_1_1_4 = X * r1_0_1_4;
              g3_21 = fmaf(ek3_3, r0_1_1_4, g3_21);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_1_2_3 = X * r1_0_2_3;
              g3_22 = fmaf(ek3_3, r0_1_2_3, g3_22);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_1_3_2 = X * r1_0_3_2;
              g3_23 = fmaf(ek3_3, r0_1_3_2, g3_23);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_1_4_1 = X * r1_0_4_1;
              g3_24 = fmaf(ek3_3, r0_1_4_1, g3_24);
              const float r1_1_0_4 = X * r2_0_0_4;
              const float r0_2_0_4 = fmaf(X, r1_1_0_4, r1_0_0_4);
              g3_25 = fmaf(ek3_3, r0_2_0_4, g3_25);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g3_26 = fmaf(ek3_3, r0_2_1_3, g3_26);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g3_27 = fmaf(ek3_3, r0_2_2_2, g3_27);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g3_28 = fmaf(ek3_3, r0_2_3_1, g3_28);
              const float r2_1_0_3 = X * r3_0_0_3;
              const float r1_2_0_3 = fmaf(X, r2_1_0_3, r2_0_0_3);
              const float r0_3_0_3 = fmaf(X, r1_2_0_3, 2.0f * r1_1_0_3);
              g3_29 = fmaf(ek3_3, r0_3_0_3, g3_29);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g3_30 = fmaf(ek3_3, r0_3_1_2, g3_30);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g3_31 = fmaf(ek3_3, r0_3_2_1, g3_31);
              const float r3_1_0_2 = X * r4_0_0_2;
              const float r2_2_0_2 = fmaf(X, r3_1_0_2, r3_0_0_2);
              const float r1_3_0_2 = fmaf(X, r2_2_0_2, 2.0f * r2_1_0_2);
              const float r0_4_0_2 = fmaf(X, r1_3_0_2, 3.0f * r1_2_0_2);
              g3_32 = fmaf(ek3_3, r0_4_0_2, g3_32);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g3_33 = fmaf(ek3_3, r0_4_1_1, g3_33);
              const float r4_1_0_1 = X * r5_0_0_1;
              const float r3_2_0_1 = fmaf(X, r4_1_0_1, r4_0_0_1);
              const float r2_3_0_1 = fmaf(X, r3_2_0_1, 2.0f * r3_1_0_1);
              const float r1_4_0_1 = fmaf(X, r2_3_0_1, 3.0f * r2_2_0_1);
              const float r0_5_0_1 = fmaf(X, r1_4_0_1, 4.0f * r1_3_0_1);
              g3_34 = fmaf(ek3_3, r0_5_0_1, g3_34);
            }
            { const float eb = bi[5];
              o0_3 = fmaf(eb, g3_0, o0_3);
            }
            { const float eb = bi[6];
              o0_3 = fmaf(eb, g3_3, o0_3);
            }
            { const float eb = bi[7];
              o0_3 = fmaf(eb, g3_9, o0_3);
            }
            { const float eb = bi[8];
              o0_3 = fmaf(eb, g3_19, o0_3);
            }
            { const float eb = bi[9];
              o0_3 = fmaf(eb, g3_34, o0_3);
            }
            { const float eb = bi[10];
              o1_3 = fmaf(eb, g3_0, o1_3);
            }
            { const float eb = bi[11];
              o1_3 = fmaf(eb, g3_2, o1_3);
            }
            { const float eb = bi[12];
              o1_3 = fmaf(eb, g3_6, o1_3);
            }
            { const float eb = bi[13];
              o1_3 = fmaf(eb, g3_3, o1_3);
            }
            { const float eb = bi[14];
              o1_3 = fmaf(eb, g3_8, o1_3);
            }
            { const float eb = bi[15];
              o1_3 = fmaf(eb, g3_16, o1_3);
            }
            { const float eb = bi[16];
              o1_3 = fmaf(eb, g3_9, o1_3);
            }
            { const float eb = bi[17];
              o1_3 = fmaf(eb, g3_18, o1_3);
            }
            { const float eb = bi[18];
              o1_3 = fmaf(eb, g3_31, o1_3);
            }
            { const float eb = bi[19];
              o2_3 = fmaf(eb, g3_0, o2_3);
            }
            { const float eb = bi[20];
              o2_3 = fmaf(eb, g3_1, o2_3);
            }
            { const float eb = bi[21];
              o2_3 = fmaf(eb, g3_4, o2_3);
            }
            { const float eb = bi[22];
              o2_3 = fmaf(eb, g3_3, o2_3);
            }
            { const float eb = bi[23];
              o2_3 = fmaf(eb, g3_7, o2_3);
            }
            { const float eb = bi[24];
              o2_3 = fmaf(eb, g3_14, o2_3);
            }
            { const float eb = bi[25];
              o2_3 = fmaf(eb, g3_9, o2_3);
            }
            { const float eb = bi[26];
              o2_3 = fmaf(eb, g3_17, o2_3);
            }
            { const float eb = bi[27];
              o2_3 = fmaf(eb, g3_29, o2_3);
            }
            { const float eb = bi[28];
              o3_3 = fmaf(eb, g3_0, o3_3);
            }
            { const float eb = bi[29];
              o3_3 = fmaf(eb, g3_2, o3_3);
            }
            { const float eb = bi[30];
              o3_3 = fmaf(eb, g3_3, o3_3);
            }
            { const float eb = bi[31];
              o3_3 = fmaf(eb, g3_8, o3_3);
            }
            { const float eb = bi[32];
              o3_3 = fmaf(eb, g3_9, o3_3);
            }
            { const float eb = bi[33];
              o3_3 = fmaf(eb, g3_18, o3_3);
            }
            { const float eb = bi[34];
              o3_3 = fmaf(eb, g3_19, o3_3);
            }
            { const float eb = bi[35];
              o3_3 = fmaf(eb, g3_33, o3_3);
            }
            { const float eb = bi[36];
              o4_3 = fmaf(eb, g3_0, o4_3);
            }
            { const float eb = bi[37];
              o4_3 = fmaf(eb, g3_1, o4_3);
            }
            { const float eb = bi[38];
              o4_3 = fmaf(eb, g3_3, o4_3);
            }
            { const float eb = bi[39];
              o4_3 = fmaf(eb, g3_7, o4_3);
            }
            { const float eb = bi[40];
              o4_3 = fmaf(eb, g3_9, o4_3);
            }
            { const float eb = bi[41];
              o4_3 = fmaf(eb, g3_17, o4_3);
            }
            { const float eb = bi[42];
              o4_3 = fmaf(eb, g3_19, o4_3);
            }
            { const float eb = bi[43];
              o4_3 = fmaf(eb, g3_32, o4_3);
            }
            { const float eb = bi[44];
              o5_3 = fmaf(eb, g3_0, o5_3);
            }
            { const float eb = bi[45];
              o5_3 = fmaf(eb, g3_1, o5_3);
            }
            { const float eb = bi[46];
              o5_3 = fmaf(eb, g3_2, o5_3);
            }
            { const float eb = bi[47];
              o5_3 = fmaf(eb, g3_5, o5_3);
            }
            { const float eb = bi[48];
              o5_3 = fmaf(eb, g3_3, o5_3);
            }
            { const float eb = bi[49];
              o5_3 = fmaf(eb, g3_7, o5_3);
            }
            { const float eb = bi[50];
              o5_3 = fmaf(eb, g3_8, o5_3);
            }
            { const float eb = bi[51];
              o5_3 = fmaf(eb, g3_15, o5_3);
            }
            { const float eb = bi[52];
              o5_3 = fmaf(eb, g3_9, o5_3);
            }
            { const float eb = bi[53];
              o5_3 = fmaf(eb, g3_17, o5_3);
            }
            { const float eb = bi[54];
              o5_3 = fmaf(eb, g3_18, o5_3);
            }
            { const float eb = bi[55];
              o5_3 = fmaf(eb, g3_30, o5_3);
            }
            { const float eb = bi[56];
              o6_3 = fmaf(eb, g3_0, o6_3);
            }
            { const float eb = bi[57];
              o6_3 = fmaf(eb, g3_2, o6_3);
            }
            { const float eb = bi[58];
              o6_3 = fmaf(eb, g3_6, o6_3);
            }
            { const float eb = bi[59];
              o6_3 = fmaf(eb, g3_3, o6_3);
            }
            { const float eb = bi[60];
              o6_3 = fmaf(eb, g3_8, o6_3);
            }
            { const float eb = bi[61];
              o6_3 = fmaf(eb, g3_16, o6_3);
            }
            { const float eb = bi[62];
              o6_3 = fmaf(eb, g3_9, o6_3);
            }
            { const float eb = bi[63];
              o6_3 = fmaf(eb, g3_18, o6_3);
            }
            { const float eb = bi[64];
              o6_3 = fmaf(eb, g3_31, o6_3);
            }
            { const float eb = bi[65];
              o7_3 = fmaf(eb, g3_0, o7_3);
            }
            { const float eb = bi[66];
              o7_3 = fmaf(eb, g3_2, o7_3);
            }
            { const float eb = bi[67];
              o7_3 = fmaf(eb, g3_6, o7_3);
            }
            { const float eb = bi[68];
              o7_3 = fmaf(eb, g3_13, o7_3);
            }
            { const float eb = bi[69];
              o7_3 = fmaf(eb, g3_24, o7_3);
            }
            { const float eb = bi[70];
              o8_3 = fmaf(eb, g3_0, o8_3);
            }
            { const float eb = bi[71];
              o8_3 = fmaf(eb, g3_1, o8_3);
            }
            { const float eb = bi[72];
              o8_3 = fmaf(eb, g3_4, o8_3);
            }
            { const float eb = bi[73];
              o8_3 = fmaf(eb, g3_2, o8_3);
            }
            { const float eb = bi[74];
              o8_3 = fmaf(eb, g3_5, o8_3);
            }
            { const float eb = bi[75];
              o8_3 = fmaf(eb, g3_11, o8_3);
            }
            { const float eb = bi[76];
              o8_3 = fmaf(eb, g3_6, o8_3);
            }
            { const float eb = bi[77];
              o8_3 = fmaf(eb, g3_12, o8_3);
            }
            { const float eb = bi[78];
              o8_3 = fmaf(eb, g3_22, o8_3);
            }
            { const float eb = bi[79];
              o9_3 = fmaf(eb, g3_0, o9_3);
            }
            { const float eb = bi[80];
              o9_3 = fmaf(eb, g3_2, o9_3);
            }
            { const float eb = bi[81];
              o9_3 = fmaf(eb, g3_6, o9_3);
            }
            { const float eb = bi[82];
              o9_3 = fmaf(eb, g3_13, o9_3);
            }
            { const float eb = bi[83];
              o9_3 = fmaf(eb, g3_3, o9_3);
            }
            { const float eb = bi[84];
              o9_3 = fmaf(eb, g3_8, o9_3);
            }
            { const float eb = bi[85];
              o9_3 = fmaf(eb, g3_16, o9_3);
            }
            { const float eb = bi[86];
              o9_3 = fmaf(eb, g3_28, o9_3);
            }
            { const float eb = bi[87];
              o10_3 = fmaf(eb, g3_0, o10_3);
            }
            { const float eb = bi[88];
              o10_3 = fmaf(eb, g3_1, o10_3);
            }
            { const float eb = bi[89];
              o10_3 = fmaf(eb, g3_2, o10_3);
            }
            { const float eb = bi[90];
              o10_3 = fmaf(eb, g3_5, o10_3);
            }
            { const float eb = bi[91];
              o10_3 = fmaf(eb, g3_6, o10_3);
            }
            { const float eb = bi[92];
              o10_3 = fmaf(eb, g3_12, o10_3);
            }
            { const float eb = bi[93];
              o10_3 = fmaf(eb, g3_3, o10_3);
            }
            { const float eb = bi[94];
              o10_3 = fmaf(eb, g3_7, o10_3);
            }
            { const float eb = bi[95];
              o10_3 = fmaf(eb, g3_8, o10_3);
            }
            { const float eb = bi[96];
              o10_3 = fmaf(eb, g3_15, o10_3);
            }
            { const float eb = bi[97];
              o10_3 = fmaf(eb, g3_16, o10_3);
            }
            { const float eb = bi[98];
              o10_3 = fmaf(eb, g3_27, o10_3);
            }
            { const float eb = bi[99];
              o11_3 = fmaf(eb, g3_0, o11_3);
            }
            { const float eb = bi[100];
              o11_3 = fmaf(eb, g3_1, o11_3);
            }
            { const float eb = bi[101];
              o11_3 = fmaf(eb, g3_2, o11_3);
            }
            { const float eb = bi[102];
              o11_3 = fmaf(eb, g3_5, o11_3);
            }
            { const float eb = bi[103];
              o11_3 = fmaf(eb, g3_6, o11_3);
            }
            { const float eb = bi[104];
              o11_3 = fmaf(eb, g3_12, o11_3);
            }
            { const float eb = bi[105];
              o11_3 = fmaf(eb, g3_13, o11_3);
            }
            { const float eb = bi[106];
              o11_3 = fmaf(eb, g3_23, o11_3);
            }
            { const float eb = bi[107];
              o12_3 = fmaf(eb, g3_0, o12_3);
            }
            { const float eb = bi[108];
              o12_3 = fmaf(eb, g3_1, o12_3);
            }
            { const float eb = bi[109];
              o12_3 = fmaf(eb, g3_4, o12_3);
            }
            { const float eb = bi[110];
              o12_3 = fmaf(eb, g3_3, o12_3);
            }
            { const float eb = bi[111];
              o12_3 = fmaf(eb, g3_7, o12_3);
            }
            { const float eb = bi[112];
              o12_3 = fmaf(eb, g3_14, o12_3);
            }
            { const float eb = bi[113];
              o12_3 = fmaf(eb, g3_9, o12_3);
            }
            { const float eb = bi[114];
              o12_3 = fmaf(eb, g3_17, o12_3);
            }
            { const float eb = bi[115];
              o12_3 = fmaf(eb, g3_29, o12_3);
            }
            { const float eb = bi[116];
              o13_3 = fmaf(eb, g3_0, o13_3);
            }
            { const float eb = bi[117];
              o13_3 = fmaf(eb, g3_1, o13_3);
            }
            { const float eb = bi[118];
              o13_3 = fmaf(eb, g3_4, o13_3);
            }
            { const float eb = bi[119];
              o13_3 = fmaf(eb, g3_2, o13_3);
            }
            { const float eb = bi[120];
              o13_3 = fmaf(eb, g3_5, o13_3);
            }
            { const float eb = bi[121];
              o13_3 = fmaf(eb, g3_11, o13_3);
            }
            { const float eb = bi[122];
              o13_3 = fmaf(eb, g3_6, o13_3);
            }
            { const float eb = bi[123];
              o13_3 = fmaf(eb, g3_12, o13_3);
            }
            { const float eb = bi[124];
              o13_3 = fmaf(eb, g3_22, o13_3);
            }
            { const float eb = bi[125];
              o14_3 = fmaf(eb, g3_0, o14_3);
            }
            { const float eb = bi[126];
              o14_3 = fmaf(eb, g3_1, o14_3);
            }
            { const float eb = bi[127];
              o14_3 = fmaf(eb, g3_4, o14_3);
            }
            { const float eb = bi[128];
              o14_3 = fmaf(eb, g3_10, o14_3);
            }
            { const float eb = bi[129];
              o14_3 = fmaf(eb, g3_20, o14_3);
            }
            { const float eb = bi[130];
              o15_3 = fmaf(eb, g3_0, o15_3);
            }
            { const float eb = bi[131];
              o15_3 = fmaf(eb, g3_1, o15_3);
            }
            { const float eb = bi[132];
              o15_3 = fmaf(eb, g3_4, o15_3);
            }
            { const float eb = bi[133];
              o15_3 = fmaf(eb, g3_2, o15_3);
            }
            { const float eb = bi[134];
              o15_3 = fmaf(eb, g3_5, o15_3);
            }
            { const float eb = bi[135];
              o15_3 = fmaf(eb, g3_11, o15_3);
            }
            { const float eb = bi[136];
              o15_3 = fmaf(eb, g3_3, o15_3);
            }
            { const float eb = bi[137];
              o15_3 = fmaf(eb, g3_7, o15_3);
            }
            { const float eb = bi[138];
              o15_3 = fmaf(eb, g3_14, o15_3);
            }
            { const float eb = bi[139];
              o15_3 = fmaf(eb, g3_8, o15_3);
            }
            { const float eb = bi[140];
              o15_3 = fmaf(eb, g3_15, o15_3);
            }
            { const float eb = bi[141];
              o15_3 = fmaf(eb, g3_26, o15_3);
            }
            { const float eb = bi[142];
              o16_3 = fmaf(eb, g3_0, o16_3);
            }
            { const float eb = bi[143];
              o16_3 = fmaf(eb, g3_1, o16_3);
            }
            { const float eb = bi[144];
              o16_3 = fmaf(eb, g3_4, o16_3);
            }
            { const float eb = bi[145];
              o16_3 = fmaf(eb, g3_10, o16_3);
            }
            { const float eb = bi[146];
              o16_3 = fmaf(eb, g3_3, o16_3);
            }
            { const float eb = bi[147];
              o16_3 = fmaf(eb, g3_7, o16_3);
            }
            { const float eb = bi[148];
              o16_3 = fmaf(eb, g3_14, o16_3);
            }
            { const float eb = bi[149];
              o16_3 = fmaf(eb, g3_25, o16_3);
            }
            { const float eb = bi[150];
              o17_3 = fmaf(eb, g3_0, o17_3);
            }
            { const float eb = bi[151];
              o17_3 = fmaf(eb, g3_1, o17_3);
            }
            { const float eb = bi[152];
              o17_3 = fmaf(eb, g3_4, o17_3);
            }
            { const float eb = bi[153];
              o17_3 = fmaf(eb, g3_10, o17_3);
            }
            { const float eb = bi[154];
              o17_3 = fmaf(eb, g3_2, o17_3);
            }
            { const float eb = bi[155];
              o17_3 = fmaf(eb, g3_5, o17_3);
            }
            { const float eb = bi[156];
              o17_3 = fmaf(eb, g3_11, o17_3);
            }
            { const float eb = bi[157];
              o17_3 = fmaf(eb, g3_21, o17_3);
            }
            { const float eb = bi[158];
              o18_3 = fmaf(eb, g3_0, o18_3);
            }
            { const float eb = bi[159];
              o18_3 = fmaf(eb, g3_2, o18_3);
            }
            { const float eb = bi[160];
              o18_3 = fmaf(eb, g3_3, o18_3);
            }
            { const float eb = bi[161];
              o18_3 = fmaf(eb, g3_8, o18_3);
            }
            { const float eb = bi[162];
              o18_3 = fmaf(eb, g3_9, o18_3);
            }
            { const float eb = bi[163];
              o18_3 = fmaf(eb, g3_18, o18_3);
            }
            { const float eb = bi[164];
              o18_3 = fmaf(eb, g3_19, o18_3);
            }
            { const float eb = bi[165];
              o18_3 = fmaf(eb, g3_33, o18_3);
            }
            { const float eb = bi[166];
              o19_3 = fmaf(eb, g3_0, o19_3);
            }
            { const float eb = bi[167];
              o19_3 = fmaf(eb, g3_2, o19_3);
            }
            { const float eb = bi[168];
              o19_3 = fmaf(eb, g3_6, o19_3);
            }
            { const float eb = bi[169];
              o19_3 = fmaf(eb, g3_13, o19_3);
            }
            { const float eb = bi[170];
              o19_3 = fmaf(eb, g3_3, o19_3);
            }
            { const float eb = bi[171];
              o19_3 = fmaf(eb, g3_8, o19_3);
            }
            { const float eb = bi[172];
              o19_3 = fmaf(eb, g3_16, o19_3);
            }
            { const float eb = bi[173];
              o19_3 = fmaf(eb, g3_28, o19_3);
            }
            { const float eb = bi[174];
              o20_3 = fmaf(eb, g3_0, o20_3);
            }
            { const float eb = bi[175];
              o20_3 = fmaf(eb, g3_1, o20_3);
            }
            { const float eb = bi[176];
              o20_3 = fmaf(eb, g3_4, o20_3);
            }
            { const float eb = bi[177];
              o20_3 = fmaf(eb, g3_2, o20_3);
            }
            { const float eb = bi[178];
              o20_3 = fmaf(eb, g3_5, o20_3);
            }
            { const float eb = bi[179];
              o20_3 = fmaf(eb, g3_11, o20_3);
            }
            { const float eb = bi[180];
              o20_3 = fmaf(eb, g3_3, o20_3);
            }
            { const float eb = bi[181];
              o20_3 = fmaf(eb, g3_7, o20_3);
            }
            { const float eb = bi[182];
              o20_3 = fmaf(eb, g3_14, o20_3);
            }
            { const float eb = bi[183];
              o20_3 = fmaf(eb, g3_8, o20_3);
            }
            { const float eb = bi[184];
              o20_3 = fmaf(eb, g3_15, o20_3);
            }
            { const float eb = bi[185];
              o20_3 = fmaf(eb, g3_26, o20_3);
            }
            { const float eb = bi[186];
              o21_3 = fmaf(eb, g3_0, o21_3);
            }
            { const float eb = bi[187];
              o21_3 = fmaf(eb, g3_2, o21_3);
            }
            { const float eb = bi[188];
              o21_3 = fmaf(eb, g3_6, o21_3);
            }
            { const float eb = bi[189];
              o21_3 = fmaf(eb, g3_3, o21_3);
            }
            { const float eb = bi[190];
              o21_3 = fmaf(eb, g3_8, o21_3);
            }
            { const float eb = bi[191];
              o21_3 = fmaf(eb, g3_16, o21_3);
            }
            { const float eb = bi[192];
              o21_3 = fmaf(eb, g3_9, o21_3);
            }
            { const float eb = bi[193];
              o21_3 = fmaf(eb, g3_18, o21_3);
            }
            { const float eb = bi[194];
              o21_3 = fmaf(eb, g3_31, o21_3);
            }
            { const float eb = bi[195];
              o22_3 = fmaf(eb, g3_0, o22_3);
            }
            { const float eb = bi[196];
              o22_3 = fmaf(eb, g3_1, o22_3);
            }
            { const float eb = bi[197];
              o22_3 = fmaf(eb, g3_2, o22_3);
            }
            { const float eb = bi[198];
              o22_3 = fmaf(eb, g3_5, o22_3);
            }
            { const float eb = bi[199];
              o22_3 = fmaf(eb, g3_3, o22_3);
            }
            { const float eb = bi[200];
              o22_3 = fmaf(eb, g3_7, o22_3);
            }
            { const float eb = bi[201];
              o22_3 = fmaf(eb, g3_8, o22_3);
            }
            { const float eb = bi[202];
              o22_3 = fmaf(eb, g3_15, o22_3);
            }
            { const float eb = bi[203];
              o22_3 = fmaf(eb, g3_9, o22_3);
            }
            { const float eb = bi[204];
              o22_3 = fmaf(eb, g3_17, o22_3);
            }
            { const float eb = bi[205];
              o22_3 = fmaf(eb, g3_18, o22_3);
            }
            { const float eb = bi[206];
              o22_3 = fmaf(eb, g3_30, o22_3);
            }
            { const float eb = bi[207];
              o23_3 = fmaf(eb, g3_0, o23_3);
            }
            { const float eb = bi[208];
              o23_3 = fmaf(eb, g3_1, o23_3);
            }
            { const float eb = bi[209];
              o23_3 = fmaf(eb, g3_2, o23_3);
            }
            { const float eb = bi[210];
              o23_3 = fmaf(eb, g3_5, o23_3);
            }
            { const float eb = bi[211];
              o23_3 = fmaf(eb, g3_6, o23_3);
            }
            { const float eb = bi[212];
              o23_3 = fmaf(eb, g3_12, o23_3);
            }
            { const float eb = bi[213];
              o23_3 = fmaf(eb, g3_3, o23_3);
            }
            { const float eb = bi[214];
              o23_3 = fmaf(eb, g3_7, o23_3);
            }
            { const float eb = bi[215];
              o23_3 = fmaf(eb, g3_8, o23_3);
            }
            { const float eb = bi[216];
              o23_3 = fmaf(eb, g3_15, o23_3);
            }
            { const float eb = bi[217];
              o23_3 = fmaf(eb, g3_16, o23_3);
            }
            { const float eb = bi[218];
              o23_3 = fmaf(eb, g3_27, o23_3);
            }
            { const float eb = bi[219];
              o24_3 = fmaf(eb, g3_0, o24_3);
            }
            { const float eb = bi[220];
              o24_3 = fmaf(eb, g3_1, o24_3);
            }
            { const float eb = bi[221];
              o24_3 = fmaf(eb, g3_3, o24_3);
            }
            { const float eb = bi[222];
              o24_3 = fmaf(eb, g3_7, o24_3);
            }
            { const float eb = bi[223];
              o24_3 = fmaf(eb, g3_9, o24_3);
            }
            { const float eb = bi[224];
              o24_3 = fmaf(eb, g3_17, o24_3);
            }
            { const float eb = bi[225];
              o24_3 = fmaf(eb, g3_19, o24_3);
            }
            { const float eb = bi[226];
              o24_3 = fmaf(eb, g3_32, o24_3);
            }
            { const float eb = bi[227];
              o25_3 = fmaf(eb, g3_0, o25_3);
            }
            { const float eb = bi[228];
              o25_3 = fmaf(eb, g3_1, o25_3);
            }
            { const float eb = bi[229];
              o25_3 = fmaf(eb, g3_2, o25_3);
            }
            { const float eb = bi[230];
              o25_3 = fmaf(eb, g3_5, o25_3);
            }
            { const float eb = bi[231];
              o25_3 = fmaf(eb, g3_6, o25_3);
            }
            { const float eb = bi[232];
              o25_3 = fmaf(eb, g3_12, o25_3);
            }
            { const float eb = bi[233];
              o25_3 = fmaf(eb, g3_3, o25_3);
            }
            { const float eb = bi[234];
              o25_3 = fmaf(eb, g3_7, o25_3);
            }
            { const float eb = bi[235];
              o25_3 = fmaf(eb, g3_8, o25_3);
            }
            { const float eb = bi[236];
              o25_3 = fmaf(eb, g3_15, o25_3);
            }
            { const float eb = bi[237];
              o25_3 = fmaf(eb, g3_16, o25_3);
            }
            { const float eb = bi[238];
              o25_3 = fmaf(eb, g3_27, o25_3);
            }
            { const float eb = bi[239];
              o26_3 = fmaf(eb, g3_0, o26_3);
            }
            { const float eb = bi[240];
              o26_3 = fmaf(eb, g3_1, o26_3);
            }
            { const float eb = bi[241];
              o26_3 = fmaf(eb, g3_4, o26_3);
            }
            { const float eb = bi[242];
              o26_3 = fmaf(eb, g3_10, o26_3);
            }
            { const float eb = bi[243];
              o26_3 = fmaf(eb, g3_3, o26_3);
            }
            { const float eb = bi[244];
              o26_3 = fmaf(eb, g3_7, o26_3);
            }
            { const float eb = bi[245];
              o26_3 = fmaf(eb, g3_14, o26_3);
            }
            { const float eb = bi[246];
              o26_3 = fmaf(eb, g3_25, o26_3);
            }
            { const float eb = bi[247];
              o27_3 = fmaf(eb, g3_0, o27_3);
            }
            { const float eb = bi[248];
              o27_3 = fmaf(eb, g3_1, o27_3);
            }
            { const float eb = bi[249];
              o27_3 = fmaf(eb, g3_2, o27_3);
            }
            { const float eb = bi[250];
              o27_3 = fmaf(eb, g3_5, o27_3);
            }
            { const float eb = bi[251];
              o27_3 = fmaf(eb, g3_3, o27_3);
            }
            { const float eb = bi[252];
              o27_3 = fmaf(eb, g3_7, o27_3);
            }
            { const float eb = bi[253];
              o27_3 = fmaf(eb, g3_8, o27_3);
            }
            { const float eb = bi[254];
              o27_3 = fmaf(eb, g3_15, o27_3);
            }
            { const float eb = bi[255];
              o27_3 = fmaf(eb, g3_9, o27_3);
            }
            { const float eb = bi[256];
              o27_3 = fmaf(eb, g3_17, o27_3);
            }
            { const float eb = bi[257];
              o27_3 = fmaf(eb, g3_18, o27_3);
            }
            { const float eb = bi[258];
              o27_3 = fmaf(eb, g3_30, o27_3);
            }
            { const float eb = bi[259];
              o28_3 = fmaf(eb, g3_0, o28_3);
            }
            { const float eb = bi[260];
              o28_3 = fmaf(eb, g3_1, o28_3);
            }
            { const float eb = bi[261];
              o28_3 = fmaf(eb, g3_4, o28_3);
            }
            { const float eb = bi[262];
              o28_3 = fmaf(eb, g3_3, o28_3);
            }
            { const float eb = bi[263];
              o28_3 = fmaf(eb, g3_7, o28_3);
            }
            { const float eb = bi[264];
              o28_3 = fmaf(eb, g3_14, o28_3);
            }
            { const float eb = bi[265];
              o28_3 = fmaf(eb, g3_9, o28_3);
            }
            { const float eb = bi[266];
              o28_3 = fmaf(eb, g3_17, o28_3);
            }
            { const float eb = bi[267];
              o28_3 = fmaf(eb, g3_29, o28_3);
            }
            { const float eb = bi[268];
              o29_3 = fmaf(eb, g3_0, o29_3);
            }
            { const float eb = bi[269];
              o29_3 = fmaf(eb, g3_1, o29_3);
            }
            { const float eb = bi[270];
              o29_3 = fmaf(eb, g3_4, o29_3);
            }
            { const float eb = bi[271];
              o29_3 = fmaf(eb, g3_2, o29_3);
            }
            { const float eb = bi[272];
              o29_3 = fmaf(eb, g3_5, o29_3);
            }
            { const float eb = bi[273];
              o29_3 = fmaf(eb, g3_11, o29_3);
            }
            { const float eb = bi[274];
              o29_3 = fmaf(eb, g3_3, o29_3);
            }
            { const float eb = bi[275];
              o29_3 = fmaf(eb, g3_7, o29_3);
            }
            { const float eb = bi[276];
              o29_3 = fmaf(eb, g3_14, o29_3);
            }
            { const float eb = bi[277];
              o29_3 = fmaf(eb, g3_8, o29_3);
            }
            { const float eb = bi[278];
              o29_3 = fmaf(eb, g3_15, o29_3);
            }
            { const float eb = bi[279];
              o29_3 = fmaf(eb, g3_26, o29_3);
            }
            { const float eb = bi[280];
              o30_3 = fmaf(eb, g3_0, o30_3);
            }
            { const float eb = bi[281];
              o30_3 = fmaf(eb, g3_1, o30_3);
            }
            { const float eb = bi[282];
              o30_3 = fmaf(eb, g3_2, o30_3);
            }
            { const float eb = bi[283];
              o30_3 = fmaf(eb, g3_5, o30_3);
            }
            { const float eb = bi[284];
              o30_3 = fmaf(eb, g3_3, o30_3);
            }
            { const float eb = bi[285];
              o30_3 = fmaf(eb, g3_7, o30_3);
            }
            { const float eb = bi[286];
              o30_3 = fmaf(eb, g3_8, o30_3);
            }
            { const float eb = bi[287];
              o30_3 = fmaf(eb, g3_15, o30_3);
            }
            { const float eb = bi[288];
              o30_3 = fmaf(eb, g3_9, o30_3);
            }
            { const float eb = bi[289];
              o30_3 = fmaf(eb, g3_17, o30_3);
            }
            { const float eb = bi[290];
              o30_3 = fmaf(eb, g3_18, o30_3);
            }
            { const float eb = bi[291];
              o30_3 = fmaf(eb, g3_30, o30_3);
            }
            { const float eb = bi[292];
              o31_3 = fmaf(eb, g3_0, o31_3);
            }
            { const float eb = bi[293];
              o31_3 = fmaf(eb, g3_1, o31_3);
            }
            { const float eb = bi[294];
              o31_3 = fmaf(eb, g3_2, o31_3);
            }
            { const float eb = bi[295];
              o31_3 = fmaf(eb, g3_5, o31_3);
            }
            { const float eb = bi[296];
              o31_3 = fmaf(eb, g3_6, o31_3);
            }
            { const float eb = bi[297];
              o31_3 = fmaf(eb, g3_12, o31_3);
            }
            { const float eb = bi[298];
              o31_3 = fmaf(eb, g3_13, o31_3);
            }
            { const float eb = bi[299];
              o31_3 = fmaf(eb, g3_23, o31_3);
            }
            { const float eb = bi[300];
              o32_3 = fmaf(eb, g3_0, o32_3);
            }
            { const float eb = bi[301];
              o32_3 = fmaf(eb, g3_1, o32_3);
            }
            { const float eb = bi[302];
              o32_3 = fmaf(eb, g3_4, o32_3);
            }
            { const float eb = bi[303];
              o32_3 = fmaf(eb, g3_10, o32_3);
            }
            { const float eb = bi[304];
              o32_3 = fmaf(eb, g3_2, o32_3);
            }
            { const float eb = bi[305];
              o32_3 = fmaf(eb, g3_5, o32_3);
            }
            { const float eb = bi[306];
              o32_3 = fmaf(eb, g3_11, o32_3);
            }
            { const float eb = bi[307];
              o32_3 = fmaf(eb, g3_21, o32_3);
            }
            { const float eb = bi[308];
              o33_3 = fmaf(eb, g3_0, o33_3);
            }
            { const float eb = bi[309];
              o33_3 = fmaf(eb, g3_1, o33_3);
            }
            { const float eb = bi[310];
              o33_3 = fmaf(eb, g3_2, o33_3);
            }
            { const float eb = bi[311];
              o33_3 = fmaf(eb, g3_5, o33_3);
            }
            { const float eb = bi[312];
              o33_3 = fmaf(eb, g3_6, o33_3);
            }
            { const float eb = bi[313];
              o33_3 = fmaf(eb, g3_12, o33_3);
            }
            { const float eb = bi[314];
              o33_3 = fmaf(eb, g3_3, o33_3);
            }
            { const float eb = bi[315];
              o33_3 = fmaf(eb, g3_7, o33_3);
            }
            { const float eb = bi[316];
              o33_3 = fmaf(eb, g3_8, o33_3);
            }
            { const float eb = bi[317];
              o33_3 = fmaf(eb, g3_15, o33_3);
            }
            { const float eb = bi[318];
              o33_3 = fmaf(eb, g3_16, o33_3);
            }
            { const float eb = bi[319];
              o33_3 = fmaf(eb, g3_27, o33_3);
            }
            { const float eb = bi[320];
              o34_3 = fmaf(eb, g3_0, o34_3);
            }
            { const float eb = bi[321];
              o34_3 = fmaf(eb, g3_1, o34_3);
            }
            { const float eb = bi[322];
              o34_3 = fmaf(eb, g3_4, o34_3);
            }
            { const float eb = bi[323];
              o34_3 = fmaf(eb, g3_2, o34_3);
            }
            { const float eb = bi[324];
              o34_3 = fmaf(eb, g3_5, o34_3);
            }
            { const float eb = bi[325];
              o34_3 = fmaf(eb, g3_11, o34_3);
            }
            { const float eb = bi[326];
              o34_3 = fmaf(eb, g3_3, o34_3);
            }
            { const float eb = bi[327];
              o34_3 = fmaf(eb, g3_7, o34_3);
            }
            { const float eb = bi[328];
              o34_3 = fmaf(eb, g3_14, o34_3);
            }
            { const float eb = bi[329];
              o34_3 = fmaf(eb, g3_8, o34_3);
            }
            { const float eb = bi[330];
              o34_3 = fmaf(eb, g3_15, o34_3);
            }
            { const float eb = bi[331];
              o34_3 = fmaf(eb, g3_26, o34_3);
            }
            { const float eb = bi[332];
              o35_3 = fmaf(eb, g3_0, o35_3);
            }
            { const float eb = bi[333];
              o35_3 = fmaf(eb, g3_1, o35_3);
            }
            { const float eb = bi[334];
              o35_3 = fmaf(eb, g3_4, o35_3);
            }
            { const float eb = bi[335];
              o35_3 = fmaf(eb, g3_2, o35_3);
            }
            { const float eb = bi[336];
              o35_3 = fmaf(eb, g3_5, o35_3);
            }
            { const float eb = bi[337];
              o35_3 = fmaf(eb, g3_11, o35_3);
            }
            { const float eb = bi[338];
              o35_3 = fmaf(eb, g3_6, o35_3);
            }
            { const float eb = bi[339];
              o35_3 = fmaf(eb, g3_12, o35_3);
            }
            { const float eb = bi[340];
              o35_3 = fmaf(eb, g3_22, o35_3);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk3 = PT[(fI + 0) * N + fJ + 3];
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Abd4_3 = PA[(fQ + 4) * N + fJ + 3];
            const double Abd5_3 = PA[(fQ + 5) * N + fJ + 3];
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
            const double Abc4_0 = PA[(fQ + 4) * N + fI + 0];
            const double Abc5_0 = PA[(fQ + 5) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            const double Aac3_0 = PA[(fP + 3) * N + fI + 0];
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
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
            atomicAdd(Jacc + (fI + 0) * N + fJ + 3, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5 + o6_3 * ptb6 + o7_3 * ptb7 + o8_3 * ptb8 + o9_3 * ptb9 + o10_3 * ptb10 + o11_3 * ptb11 + o12_3 * ptb12 + o13_3 * ptb13 + o14_3 * ptb14 + o15_3 * ptb15 + o16_3 * ptb16 + o17_3 * ptb17 + o18_3 * ptb18 + o19_3 * ptb19 + o20_3 * ptb20 + o21_3 * ptb21 + o22_3 * ptb22 + o23_3 * ptb23 + o24_3 * ptb24 + o25_3 * ptb25 + o26_3 * ptb26 + o27_3 * ptb27 + o28_3 * ptb28 + o29_3 * ptb29 + o30_3 * ptb30 + o31_3 * ptb31 + o32_3 * ptb32 + o33_3 * ptb33 + o34_3 * ptb34 + o35_3 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_3 * Abd0_3 + o1_3 * Abd1_3 + o2_3 * Abd2_3 + o3_3 * Abd3_3 + o4_3 * Abd4_3 + o5_3 * Abd5_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_3 * Aad0_3 + o6_3 * Aad1_3 + o12_3 * Aad2_3 + o18_3 * Aad3_3 + o24_3 * Aad4_3 + o30_3 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_3 * Abc0_0 + o1_3 * Abc1_0 + o2_3 * Abc2_0 + o3_3 * Abc3_0 + o4_3 * Abc4_0 + o5_3 * Abc5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_3 * Aac0_0 + o6_3 * Aac1_0 + o12_3 * Aac2_0 + o18_3 * Aac3_0 + o24_3 * Aac4_0 + o30_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 0, deg * (o1_3 * Aad0_3 + o7_3 * Aad1_3 + o13_3 * Aad2_3 + o19_3 * Aad3_3 + o25_3 * Aad4_3 + o31_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_3 * Aac0_0 + o7_3 * Aac1_0 + o13_3 * Aac2_0 + o19_3 * Aac3_0 + o25_3 * Aac4_0 + o31_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 0, deg * (o2_3 * Aad0_3 + o8_3 * Aad1_3 + o14_3 * Aad2_3 + o20_3 * Aad3_3 + o26_3 * Aad4_3 + o32_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_3 * Aac0_0 + o8_3 * Aac1_0 + o14_3 * Aac2_0 + o20_3 * Aac3_0 + o26_3 * Aac4_0 + o32_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 0, deg * (o3_3 * Aad0_3 + o9_3 * Aad1_3 + o15_3 * Aad2_3 + o21_3 * Aad3_3 + o27_3 * Aad4_3 + o33_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_3 * Aac0_0 + o9_3 * Aac1_0 + o15_3 * Aac2_0 + o21_3 * Aac3_0 + o27_3 * Aac4_0 + o33_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 0, deg * (o4_3 * Aad0_3 + o10_3 * Aad1_3 + o16_3 * Aad2_3 + o22_3 * Aad3_3 + o28_3 * Aad4_3 + o34_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 3, deg * (o4_3 * Aac0_0 + o10_3 * Aac1_0 + o16_3 * Aac2_0 + o22_3 * Aac3_0 + o28_3 * Aac4_0 + o34_3 * Aac5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 0, deg * (o5_3 * Aad0_3 + o11_3 * Aad1_3 + o17_3 * Aad2_3 + o23_3 * Aad3_3 + o29_3 * Aad4_3 + o35_3 * Aad5_3));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 3, deg * (o5_3 * Aac0_0 + o11_3 * Aac1_0 + o17_3 * Aac2_0 + o23_3 * Aac3_0 + o29_3 * Aac4_0 + o35_3 * Aac5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o6_3 * Abd0_3 + o7_3 * Abd1_3 + o8_3 * Abd2_3 + o9_3 * Abd3_3 + o10_3 * Abd4_3 + o11_3 * Abd5_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o6_3 * Abc0_0 + o7_3 * Abc1_0 + o8_3 * Abc2_0 + o9_3 * Abc3_0 + o10_3 * Abc4_0 + o11_3 * Abc5_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o12_3 * Abd0_3 + o13_3 * Abd1_3 + o14_3 * Abd2_3 + o15_3 * Abd3_3 + o16_3 * Abd4_3 + o17_3 * Abd5_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o12_3 * Abc0_0 + o13_3 * Abc1_0 + o14_3 * Abc2_0 + o15_3 * Abc3_0 + o16_3 * Abc4_0 + o17_3 * Abc5_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o18_3 * Abd0_3 + o19_3 * Abd1_3 + o20_3 * Abd2_3 + o21_3 * Abd3_3 + o22_3 * Abd4_3 + o23_3 * Abd5_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o18_3 * Abc0_0 + o19_3 * Abc1_0 + o20_3 * Abc2_0 + o21_3 * Abc3_0 + o22_3 * Abc4_0 + o23_3 * Abc5_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o24_3 * Abd0_3 + o25_3 * Abd1_3 + o26_3 * Abd2_3 + o27_3 * Abd3_3 + o28_3 * Abd4_3 + o29_3 * Abd5_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o24_3 * Abc0_0 + o25_3 * Abc1_0 + o26_3 * Abc2_0 + o27_3 * Abc3_0 + o28_3 * Abc4_0 + o29_3 * Abc5_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o30_3 * Abd0_3 + o31_3 * Abd1_3 + o32_3 * Abd2_3 + o33_3 * Abd3_3 + o34_3 * Abd4_3 + o35_3 * Abd5_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o30_3 * Abc0_0 + o31_3 * Abc1_0 + o32_3 * Abc2_0 + o33_3 * Abc3_0 + o34_3 * Abc4_0 + o35_3 * Abc5_0));
          }
        } break;
        case 4: {  // ket functions [4]
          float o0_4 = 0;
          float o1_4 = 0;
          float o2_4 = 0;
          float o3_4 = 0;
          float o4_4 = 0;
          float o5_4 = 0;
          float o6_4 = 0;
          float o7_4 = 0;
          float o8_4 = 0;
          float o9_4 = 0;
          float o10_4 = 0;
          float o11_4 = 0;
          float o12_4 = 0;
          float o13_4 = 0;
          float o14_4 = 0;
          float o15_4 = 0;
          float o16_4 = 0;
          float o17_4 = 0;
          float o18_4 = 0;
          float o19_4 = 0;
          float o20_4 = 0;
          float o21_4 = 0;
          float o22_4 = 0;
          float o23_4 = 0;
          float o24_4 = 0;
          float o25_4 = 0;
          float o26_4 = 0;
          float o27_4 = 0;
          float o28_4 = 0;
          float o29_4 = 0;
          float o30_4 = 0;
          float o31_4 = 0;
          float o32_4 = 0;
          float o33_4 = 0;
          float o34_4 = 0;
          float o35_4 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
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
            float g4_10 = 0;
            float g4_11 = 0;
            float g4_12 = 0;
            float g4_13 = 0;
            float g4_14 = 0;
            float g4_15 = 0;
            float g4_16 = 0;
            float g4_17 = 0;
            float g4_18 = 0;
            float g4_19 = 0;
            float g4_20 = 0;
            float g4_21 = 0;
            float g4_22 = 0;
            float g4_23 = 0;
            float g4_24 = 0;
            float g4_25 = 0;
            float g4_26 = 0;
            float g4_27 = 0;
            float g4_28 = 0;
            float g4_29 = 0;
            float g4_30 = 0;
            float g4_31 = 0;
            float g4_32 = 0;
            float g4_33 = 0;
            float g4_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[6];
              sqb::boysf<5>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              const float ek4_0 = kj[18 * kS];
              const float ek4_1 = -kj[19 * kS];
              g4_0 = fmaf(ek4_0, b0, g4_0);
              const float r0_0_0_1 = Z * b1;
              g4_1 = fmaf(ek4_0, r0_0_0_1, g4_1);
              const float r0_0_1_0 = Y * b1;
              g4_2 = fmaf(ek4_0, r0_0_1_0, g4_2);
              g4_0 = fmaf(ek4_1, r0_0_1_0, g4_0);
              const float r0_1_0_0 = X * b1;
              g4_3 = fmaf(ek4_0, r0_1_0_0, g4_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g4_4 = fmaf(ek4_0, r0_0_0_2, g4_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g4_5 = fmaf(ek4_0, r0_0_1_1, g4_5);
              g4_1 = fmaf(ek4_1, r0_0_1_1, g4_1);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g4_6 = fmaf(ek4_0, r0_0_2_0, g4_6);
              g4_2 = fmaf(ek4_1, r0_0_2_0, g4_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g4_7 = fmaf(ek4_0, r0_1_0_1, g4_7);
              const float r0_1_1_0 = X * r1_0_1_0;
              g4_8 = fmaf(ek4_0, r0_1_1_0, g4_8);
              g4_3 = fmaf(ek4_1, r0_1_1_0, g4_3);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g4_9 = fmaf(ek4_0, r0_2_0_0, g4_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g4_10 = fmaf(ek4_0, r0_0_0_3, g4_10);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g4_11 = fmaf(ek4_0, r0_0_1_2, g4_11);
              g4_4 = fmaf(ek4_1, r0_0_1_2, g4_4);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g4_12 = fmaf(ek4_0, r0_0_2_1, g4_12);
              g4_5 = fmaf(ek4_1, r0_0_2_1, g4_5);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g4_13 = fmaf(ek4_0, r0_0_3_0, g4_13);
              g4_6 = fmaf(ek4_1, r0_0_3_0, g4_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g4_14 = fmaf(ek4_0, r0_1_0_2, g4_14);
              const float r0_1_1_1 = X * r1_0_1_1;
              g4_15 = fmaf(ek4_0, r0_1_1_1, g4_15);
              g4_7 = fmaf(ek4_1, r0_1_1_1, g4_7);
              const float r0_1_2_0 = X * r1_0_2_0;
              g4_16 = fmaf(ek4_0, r0_1_2_0, g4_16);
              g4_8 = fmaf(ek4_1, r0_1_2_0, g4_8);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g4_17 = fmaf(ek4_0, r0_2_0_1, g4_17);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g4_18 = fmaf(ek4_0, r0_2_1_0, g4_18);
              g4_9 = fmaf(ek4_1, r0_2_1_0, g4_9);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g4_19 = fmaf(ek4_0, r0_3_0_0, g4_19);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g4_20 = fmaf(ek4_0, r0_0_0_4, g4_20);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g4_21 = fmaf(ek4_0, r0_0_1_3, g4_21);
              g4_10 = fmaf(ek4_1, r0_0_1_3, g4_10);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g4_22 = fmaf(ek4_0, r0_0_2_2, g4_22);
              g4_11 = fmaf(ek4_1, r0_0_2_2, g4_11);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g4_23 = fmaf(ek4_0, r0_0_3_1, g4_23);
              g4_12 = fmaf(ek4_1, r0_0_3_1, g4_12);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g4_24 = fmaf(ek4_0, r0_0_4_0, g4_24);
              g4_13 = fmaf(ek4_1, r0_0_4_0, g4_13);
              const float r0_1_0_3 = X * r1_0_0_3;
              g4_25 = fmaf(ek4_0, r0_1_0_3, g4_25);
              const float r0_1_1_2 = X * r1_0_1_2;
              g4_26 = fmaf(ek4_0, r0_1_1_2, g4_26);
              g4_14 = fmaf(ek4_1, r0_1_1_2, g4_14);
              const float r0_1_2_1 = X * r1_0_2_1;
              g4_27 = fmaf(ek4_0, r0_1_2_1, g4_27);
              g4_15 = fmaf(ek4_1, r0_1_2_1, g4_15);
              const float r0_1_3_0 = X * r1_0_3_0;
              g4_28 = fmaf(ek4_0, r0_1_3_0, g4_28);
              g4_16 = fmaf(ek4_1, r0_1_3_0, g4_16);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g4_29 = fmaf(ek4_0, r0_2_0_2, g4_29);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g4_30 = fmaf(ek4_0, r0_2_1_1, g4_30);
              g4_17 = fmaf(ek4_1, r0_2_1_1, g4_17);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g4_31 = fmaf(ek4_0, r0_2_2_0, g4_31);
              g4_18 = fmaf(ek4_1, r0_2_2_0, g4_18);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g4_32 = fmaf(ek4_0, r0_3_0_1, g4_32);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g4_33 = fmaf(ek4_0, r0_3_1_0, g4_33);
              g4_19 = fmaf(ek4_1, r0_3_1_0, g4_19);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g4_34 = fmaf(ek4_0, r0_4_0_0, g4_34);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g4_20 = fmaf(ek4_1, r0_0_1_4, g4_20);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g4_21 = fmaf(ek4_1, r0_0_2_3, g4_21);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g4_22 = fmaf(ek4_1, r0_0_3_2, g4_22);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g4_23 = fmaf(ek4_1, r0_0_4_1, g4_23);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_0_5_0 = fmaf(Y, r1_0_4_0, 4.0f * r1_0_3_0);
              g4_24 = fmaf(ek4_1, r0_0_5_0, g4_24);
              const float r0_1_1_3 = X * r1_0_1_3;
              g4_25 = fmaf(ek4_1, r0_1_1_3, g4_25);
              const float r0_1_2_2 = X * r1_0_2_2;
              g4_26 = fmaf(ek4_1, r0_1_2_2, g4_26);
              const float r0_1_3_1 = X * r1_0_3_1;
              g4_27 = fmaf(ek4_1, r0_1_3_1, g4_27);
              const float r0_1_4_0 = X * r1_0_4_0;
              g4_28 = fmaf(ek4_1, r0_1_4_0, g4_28);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g4_29 = fmaf(ek4_1, r0_2_1_2, g4_29);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g4_30 = fmaf(ek4_1, r0_2_2_1, g4_30);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g4_31 = fmaf(ek4_1, r0_2_3_0, g4_31);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g4_32 = fmaf(ek4_1, r0_3_1_1, g4_32);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g4_33 = fmaf(ek4_1, r0_3_2_0, g4_33);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g4_34 = fmaf(ek4_1, r0_4_1_0, g4_34);
            }
            { const float eb = bi[5];
              o0_4 = fmaf(eb, g4_0, o0_4);
            }
            { const float eb = bi[6];
              o0_4 = fmaf(eb, g4_3, o0_4);
            }
            { const float eb = bi[7];
              o0_4 = fmaf(eb, g4_9, o0_4);
            }
            { const float eb = bi[8];
              o0_4 = fmaf(eb, g4_19, o0_4);
            }
            { const float eb = bi[9];
              o0_4 = fmaf(eb, g4_34, o0_4);
            }
            { const float eb = bi[10];
              o1_4 = fmaf(eb, g4_0, o1_4);
            }
            { const float eb = bi[11];
              o1_4 = fmaf(eb, g4_2, o1_4);
            }
            { const float eb = bi[12];
              o1_4 = fmaf(eb, g4_6, o1_4);
            }
            { const float eb = bi[13];
              o1_4 = fmaf(eb, g4_3, o1_4);
            }
            { const float eb = bi[14];
              o1_4 = fmaf(eb, g4_8, o1_4);
            }
            { const float eb = bi[15];
              o1_4 = fmaf(eb, g4_16, o1_4);
            }
            { const float eb = bi[16];
              o1_4 = fmaf(eb, g4_9, o1_4);
            }
            { const float eb = bi[17];
              o1_4 = fmaf(eb, g4_18, o1_4);
            }
            { const float eb = bi[18];
              o1_4 = fmaf(eb, g4_31, o1_4);
            }
            { const float eb = bi[19];
              o2_4 = fmaf(eb, g4_0, o2_4);
            }
            { const float eb = bi[20];
              o2_4 = fmaf(eb, g4_1, o2_4);
            }
            { const float eb = bi[21];
              o2_4 = fmaf(eb, g4_4, o2_4);
            }
            { const float eb = bi[22];
              o2_4 = fmaf(eb, g4_3, o2_4);
            }
            { const float eb = bi[23];
              o2_4 = fmaf(eb, g4_7, o2_4);
            }
            { const float eb = bi[24];
              o2_4 = fmaf(eb, g4_14, o2_4);
            }
            { const float eb = bi[25];
              o2_4 = fmaf(eb, g4_9, o2_4);
            }
            { const float eb = bi[26];
              o2_4 = fmaf(eb, g4_17, o2_4);
            }
            { const float eb = bi[27];
              o2_4 = fmaf(eb, g4_29, o2_4);
            }
            { const float eb = bi[28];
              o3_4 = fmaf(eb, g4_0, o3_4);
            }
            { const float eb = bi[29];
              o3_4 = fmaf(eb, g4_2, o3_4);
            }
            { const float eb = bi[30];
              o3_4 = fmaf(eb, g4_3, o3_4);
            }
            { const float eb = bi[31];
              o3_4 = fmaf(eb, g4_8, o3_4);
            }
            { const float eb = bi[32];
              o3_4 = fmaf(eb, g4_9, o3_4);
            }
            { const float eb = bi[33];
              o3_4 = fmaf(eb, g4_18, o3_4);
            }
            { const float eb = bi[34];
              o3_4 = fmaf(eb, g4_19, o3_4);
            }
            { const float eb = bi[35];
              o3_4 = fmaf(eb, g4_33, o3_4);
            }
            { const float eb = bi[36];
              o4_4 = fmaf(eb, g4_0, o4_4);
            }
            { const float eb = bi[37];
              o4_4 = fmaf(eb, g4_1, o4_4);
            }
            { const float eb = bi[38];
              o4_4 = fmaf(eb, g4_3, o4_4);
            }
            { const float eb = bi[39];
              o4_4 = fmaf(eb, g4_7, o4_4);
            }
            { const float eb = bi[40];
              o4_4 = fmaf(eb, g4_9, o4_4);
            }
            { const float eb = bi[41];
              o4_4 = fmaf(eb, g4_17, o4_4);
            }
            { const float eb = bi[42];
              o4_4 = fmaf(eb, g4_19, o4_4);
            }
            { const float eb = bi[43];
              o4_4 = fmaf(eb, g4_32, o4_4);
            }
            { const float eb = bi[44];
              o5_4 = fmaf(eb, g4_0, o5_4);
            }
            { const float eb = bi[45];
              o5_4 = fmaf(eb, g4_1, o5_4);
            }
            { const float eb = bi[46];
              o5_4 = fmaf(eb, g4_2, o5_4);
            }
            { const float eb = bi[47];
              o5_4 = fmaf(eb, g4_5, o5_4);
            }
            { const float eb = bi[48];
              o5_4 = fmaf(eb, g4_3, o5_4);
            }
            { const float eb = bi[49];
              o5_4 = fmaf(eb, g4_7, o5_4);
            }
            { const float eb = bi[50];
              o5_4 = fmaf(eb, g4_8, o5_4);
            }
            { const float eb = bi[51];
              o5_4 = fmaf(eb, g4_15, o5_4);
            }
            { const float eb = bi[52];
              o5_4 = fmaf(eb, g4_9, o5_4);
            }
            { const float eb = bi[53];
              o5_4 = fmaf(eb, g4_17, o5_4);
            }
            { const float eb = bi[54];
              o5_4 = fmaf(eb, g4_18, o5_4);
            }
            { const float eb = bi[55];
              o5_4 = fmaf(eb, g4_30, o5_4);
            }
            { const float eb = bi[56];
              o6_4 = fmaf(eb, g4_0, o6_4);
            }
            { const float eb = bi[57];
              o6_4 = fmaf(eb, g4_2, o6_4);
            }
            { const float eb = bi[58];
              o6_4 = fmaf(eb, g4_6, o6_4);
            }
            { const float eb = bi[59];
              o6_4 = fmaf(eb, g4_3, o6_4);
            }
            { const float eb = bi[60];
              o6_4 = fmaf(eb, g4_8, o6_4);
            }
            { const float eb = bi[61];
              o6_4 = fmaf(eb, g4_16, o6_4);
            }
            { const float eb = bi[62];
              o6_4 = fmaf(eb, g4_9, o6_4);
            }
            { const float eb = bi[63];
              o6_4 = fmaf(eb, g4_18, o6_4);
            }
            { const float eb = bi[64];
              o6_4 = fmaf(eb, g4_31, o6_4);
            }
            { const float eb = bi[65];
              o7_4 = fmaf(eb, g4_0, o7_4);
            }
            { const float eb = bi[66];
              o7_4 = fmaf(eb, g4_2, o7_4);
            }
            { const float eb = bi[67];
              o7_4 = fmaf(eb, g4_6, o7_4);
            }
            { const float eb = bi[68];
              o7_4 = fmaf(eb, g4_13, o7_4);
            }
            { const float eb = bi[69];
              o7_4 = fmaf(eb, g4_24, o7_4);
            }
            { const float eb = bi[70];
              o8_4 = fmaf(eb, g4_0, o8_4);
            }
            { const float eb = bi[71];
              o8_4 = fmaf(eb, g4_1, o8_4);
            }
            { const float eb = bi[72];
              o8_4 = fmaf(eb, g4_4, o8_4);
            }
            { const float eb = bi[73];
              o8_4 = fmaf(eb, g4_2, o8_4);
            }
            { const float eb = bi[74];
              o8_4 = fmaf(eb, g4_5, o8_4);
            }
            { const float eb = bi[75];
              o8_4 = fmaf(eb, g4_11, o8_4);
            }
            { const float eb = bi[76];
              o8_4 = fmaf(eb, g4_6, o8_4);
            }
            { const float eb = bi[77];
              o8_4 = fmaf(eb, g4_12, o8_4);
            }
            { const float eb = bi[78];
              o8_4 = fmaf(eb, g4_22, o8_4);
            }
            { const float eb = bi[79];
              o9_4 = fmaf(eb, g4_0, o9_4);
            }
            { const float eb = bi[80];
              o9_4 = fmaf(eb, g4_2, o9_4);
            }
            { const float eb = bi[81];
              o9_4 = fmaf(eb, g4_6, o9_4);
            }
            { const float eb = bi[82];
              o9_4 = fmaf(eb, g4_13, o9_4);
            }
            { const float eb = bi[83];
              o9_4 = fmaf(eb, g4_3, o9_4);
            }
            { const float eb = bi[84];
              o9_4 = fmaf(eb, g4_8, o9_4);
            }
            { const float eb = bi[85];
              o9_4 = fmaf(eb, g4_16, o9_4);
            }
            { const float eb = bi[86];
              o9_4 = fmaf(eb, g4_28, o9_4);
            }
            { const float eb = bi[87];
              o10_4 = fmaf(eb, g4_0, o10_4);
            }
            { const float eb = bi[88];
              o10_4 = fmaf(eb, g4_1, o10_4);
            }
            { const float eb = bi[89];
              o10_4 = fmaf(eb, g4_2, o10_4);
            }
            { const float eb = bi[90];
              o10_4 = fmaf(eb, g4_5, o10_4);
            }
            { const float eb = bi[91];
              o10_4 = fmaf(eb, g4_6, o10_4);
            }
            { const float eb = bi[92];
              o10_4 = fmaf(eb, g4_12, o10_4);
            }
            { const float eb = bi[93];
              o10_4 = fmaf(eb, g4_3, o10_4);
            }
            { const float eb = bi[94];
              o10_4 = fmaf(eb, g4_7, o10_4);
            }
            { const float eb = bi[95];
              o10_4 = fmaf(eb, g4_8, o10_4);
            }
            { const float eb = bi[96];
              o10_4 = fmaf(eb, g4_15, o10_4);
            }
            { const float eb = bi[97];
              o10_4 = fmaf(eb, g4_16, o10_4);
            }
            { const float eb = bi[98];
              o10_4 = fmaf(eb, g4_27, o10_4);
            }
            { const float eb = bi[99];
              o11_4 = fmaf(eb, g4_0, o11_4);
            }
            { const float eb = bi[100];
              o11_4 = fmaf(eb, g4_1, o11_4);
            }
            { const float eb = bi[101];
              o11_4 = fmaf(eb, g4_2, o11_4);
            }
            { const float eb = bi[102];
              o11_4 = fmaf(eb, g4_5, o11_4);
            }
            { const float eb = bi[103];
              o11_4 = fmaf(eb, g4_6, o11_4);
            }
            { const float eb = bi[104];
              o11_4 = fmaf(eb, g4_12, o11_4);
            }
            { const float eb = bi[105];
              o11_4 = fmaf(eb, g4_13, o11_4);
            }
            { const float eb = bi[106];
              o11_4 = fmaf(eb, g4_23, o11_4);
            }
            { const float eb = bi[107];
              o12_4 = fmaf(eb, g4_0, o12_4);
            }
            { const float eb = bi[108];
              o12_4 = fmaf(eb, g4_1, o12_4);
            }
            { const float eb = bi[109];
              o12_4 = fmaf(eb, g4_4, o12_4);
            }
            { const float eb = bi[110];
              o12_4 = fmaf(eb, g4_3, o12_4);
            }
            { const float eb = bi[111];
              o12_4 = fmaf(eb, g4_7, o12_4);
            }
            { const float eb = bi[112];
              o12_4 = fmaf(eb, g4_14, o12_4);
            }
            { const float eb = bi[113];
              o12_4 = fmaf(eb, g4_9, o12_4);
            }
            { const float eb = bi[114];
              o12_4 = fmaf(eb, g4_17, o12_4);
            }
            { const float eb = bi[115];
              o12_4 = fmaf(eb, g4_29, o12_4);
            }
            { const float eb = bi[116];
              o13_4 = fmaf(eb, g4_0, o13_4);
            }
            { const float eb = bi[117];
              o13_4 = fmaf(eb, g4_1, o13_4);
            }
            { const float eb = bi[118];
              o13_4 = fmaf(eb, g4_4, o13_4);
            }
            { const float eb = bi[119];
              o13_4 = fmaf(eb, g4_2, o13_4);
            }
            { const float eb = bi[120];
              o13_4 = fmaf(eb, g4_5, o13_4);
            }
            { const float eb = bi[121];
              o13_4 = fmaf(eb, g4_11, o13_4);
            }
            { const float eb = bi[122];
              o13_4 = fmaf(eb, g4_6, o13_4);
            }
            { const float eb = bi[123];
              o13_4 = fmaf(eb, g4_12, o13_4);
            }
            { const float eb = bi[124];
              o13_4 = fmaf(eb, g4_22, o13_4);
            }
            { const float eb = bi[125];
              o14_4 = fmaf(eb, g4_0, o14_4);
            }
            { const float eb = bi[126];
              o14_4 = fmaf(eb, g4_1, o14_4);
            }
            { const float eb = bi[127];
              o14_4 = fmaf(eb, g4_4, o14_4);
            }
            { const float eb = bi[128];
              o14_4 = fmaf(eb, g4_10, o14_4);
            }
            { const float eb = bi[129];
              o14_4 = fmaf(eb, g4_20, o14_4);
            }
            { const float eb = bi[130];
              o15_4 = fmaf(eb, g4_0, o15_4);
            }
            { const float eb = bi[131];
              o15_4 = fmaf(eb, g4_1, o15_4);
            }
            { const float eb = bi[132];
              o15_4 = fmaf(eb, g4_4, o15_4);
            }
            { const float eb = bi[133];
              o15_4 = fmaf(eb, g4_2, o15_4);
            }
            { const float eb = bi[134];
              o15_4 = fmaf(eb, g4_5, o15_4);
            }
            { const float eb = bi[135];
              o15_4 = fmaf(eb, g4_11, o15_4);
            }
            { const float eb = bi[136];
              o15_4 = fmaf(eb, g4_3, o15_4);
            }
            { const float eb = bi[137];
              o15_4 = fmaf(eb, g4_7, o15_4);
            }
            { const float eb = bi[138];
              o15_4 = fmaf(eb, g4_14, o15_4);
            }
            { const float eb = bi[139];
              o15_4 = fmaf(eb, g4_8, o15_4);
            }
            { const float eb = bi[140];
              o15_4 = fmaf(eb, g4_15, o15_4);
            }
            { const float eb = bi[141];
              o15_4 = fmaf(eb, g4_26, o15_4);
            }
            { const float eb = bi[142];
              o16_4 = fmaf(eb, g4_0, o16_4);
            }
            { const float eb = bi[143];
              o16_4 = fmaf(eb, g4_1, o16_4);
            }
            { const float eb = bi[144];
              o16_4 = fmaf(eb, g4_4, o16_4);
            }
            { const float eb = bi[145];
              o16_4 = fmaf(eb, g4_10, o16_4);
            }
            { const float eb = bi[146];
              o16_4 = fmaf(eb, g4_3, o16_4);
            }
            { const float eb = bi[147];
              o16_4 = fmaf(eb, g4_7, o16_4);
            }
            { const float eb = bi[148];
              o16_4 = fmaf(eb, g4_14, o16_4);
            }
            { const float eb = bi[149];
              o16_4 = fmaf(eb, g4_25, o16_4);
            }
            { const float eb = bi[150];
              o17_4 = fmaf(eb, g4_0, o17_4);
            }
            { const float eb = bi[151];
              o17_4 = fmaf(eb, g4_1, o17_4);
            }
            { const float eb = bi[152];
              o17_4 = fmaf(eb, g4_4, o17_4);
            }
            { const float eb = bi[153];
              o17_4 = fmaf(eb, g4_10, o17_4);
            }
            { const float eb = bi[154];
              o17_4 = fmaf(eb, g4_2, o17_4);
            }
            { const float eb = bi[155];
              o17_4 = fmaf(eb, g4_5, o17_4);
            }
            { const float eb = bi[156];
              o17_4 = fmaf(eb, g4_11, o17_4);
            }
            { const float eb = bi[157];
              o17_4 = fmaf(eb, g4_21, o17_4);
            }
            { const float eb = bi[158];
              o18_4 = fmaf(eb, g4_0, o18_4);
            }
            { const float eb = bi[159];
              o18_4 = fmaf(eb, g4_2, o18_4);
            }
            { const float eb = bi[160];
              o18_4 = fmaf(eb, g4_3, o18_4);
            }
            { const float eb = bi[161];
              o18_4 = fmaf(eb, g4_8, o18_4);
            }
            { const float eb = bi[162];
              o18_4 = fmaf(eb, g4_9, o18_4);
            }
            { const float eb = bi[163];
              o18_4 = fmaf(eb, g4_18, o18_4);
            }
            { const float eb = bi[164];
              o18_4 = fmaf(eb, g4_19, o18_4);
            }
            { const float eb = bi[165];
              o18_4 = fmaf(eb, g4_33, o18_4);
            }
            { const float eb = bi[166];
              o19_4 = fmaf(eb, g4_0, o19_4);
            }
            { const float eb = bi[167];
              o19_4 = fmaf(eb, g4_2, o19_4);
            }
            { const float eb = bi[168];
              o19_4 = fmaf(eb, g4_6, o19_4);
            }
            { const float eb = bi[169];
              o19_4 = fmaf(eb, g4_13, o19_4);
            }
            { const float eb = bi[170];
              o19_4 = fmaf(eb, g4_3, o19_4);
            }
            { const float eb = bi[171];
              o19_4 = fmaf(eb, g4_8, o19_4);
            }
            { const float eb = bi[172];
              o19_4 = fmaf(eb, g4_16, o19_4);
            }
            { const float eb = bi[173];
              o19_4 = fmaf(eb, g4_28, o19_4);
            }
            { const float eb = bi[174];
              o20_4 = fmaf(eb, g4_0, o20_4);
            }
            { const float eb = bi[175];
              o20_4 = fmaf(eb, g4_1, o20_4);
            }
            { const float eb = bi[176];
              o20_4 = fmaf(eb, g4_4, o20_4);
            }
            { const float eb = bi[177];
              o20_4 = fmaf(eb, g4_2, o20_4);
            }
            { const float eb = bi[178];
              o20_4 = fmaf(eb, g4_5, o20_4);
            }
            { const float eb = bi[179];
              o20_4 = fmaf(eb, g4_11, o20_4);
            }
            { const float eb = bi[180];
              o20_4 = fmaf(eb, g4_3, o20_4);
            }
            { const float eb = bi[181];
              o20_4 = fmaf(eb, g4_7, o20_4);
            }
            { const float eb = bi[182];
              o20_4 = fmaf(eb, g4_14, o20_4);
            }
            { const float eb = bi[183];
              o20_4 = fmaf(eb, g4_8, o20_4);
            }
            { const float eb = bi[184];
              o20_4 = fmaf(eb, g4_15, o20_4);
            }
            { const float eb = bi[185];
              o20_4 = fmaf(eb, g4_26, o20_4);
            }
            { const float eb = bi[186];
              o21_4 = fmaf(eb, g4_0, o21_4);
            }
            { const float eb = bi[187];
              o21_4 = fmaf(eb, g4_2, o21_4);
            }
            { const float eb = bi[188];
              o21_4 = fmaf(eb, g4_6, o21_4);
            }
            { const float eb = bi[189];
              o21_4 = fmaf(eb, g4_3, o21_4);
            }
            { const float eb = bi[190];
              o21_4 = fmaf(eb, g4_8, o21_4);
            }
            { const float eb = bi[191];
              o21_4 = fmaf(eb, g4_16, o21_4);
            }
            { const float eb = bi[192];
              o21_4 = fmaf(eb, g4_9, o21_4);
            }
            { const float eb = bi[193];
              o21_4 = fmaf(eb, g4_18, o21_4);
            }
            { const float eb = bi[194];
              o21_4 = fmaf(eb, g4_31, o21_4);
            }
            { const float eb = bi[195];
              o22_4 = fmaf(eb, g4_0, o22_4);
            }
            { const float eb = bi[196];
              o22_4 = fmaf(eb, g4_1, o22_4);
            }
            { const float eb = bi[197];
              o22_4 = fmaf(eb, g4_2, o22_4);
            }
            { const float eb = bi[198];
              o22_4 = fmaf(eb, g4_5, o22_4);
            }
            { const float eb = bi[199];
              o22_4 = fmaf(eb, g4_3, o22_4);
            }
            { const float eb = bi[200];
              o22_4 = fmaf(eb, g4_7, o22_4);
            }
            { const float eb = bi[201];
              o22_4 = fmaf(eb, g4_8, o22_4);
            }
            { const float eb = bi[202];
              o22_4 = fmaf(eb, g4_15, o22_4);
            }
            { const float eb = bi[203];
              o22_4 = fmaf(eb, g4_9, o22_4);
            }
            { const float eb = bi[204];
              o22_4 = fmaf(eb, g4_17, o22_4);
            }
            { const float eb = bi[205];
              o22_4 = fmaf(eb, g4_18, o22_4);
            }
            { const float eb = bi[206];
              o22_4 = fmaf(eb, g4_30, o22_4);
            }
            { const float eb = bi[207];
              o23_4 = fmaf(eb, g4_0, o23_4);
            }
            { const float eb = bi[208];
              o23_4 = fmaf(eb, g4_1, o23_4);
            }
            { const float eb = bi[209];
              o23_4 = fmaf(eb, g4_2, o23_4);
            }
            { const float eb = bi[210];
              o23_4 = fmaf(eb, g4_5, o23_4);
            }
            { const float eb = bi[211];
              o23_4 = fmaf(eb, g4_6, o23_4);
            }
            { const float eb = bi[212];
              o23_4 = fmaf(eb, g4_12, o23_4);
            }
            { const float eb = bi[213];
              o23_4 = fmaf(eb, g4_3, o23_4);
            }
            { const float eb = bi[214];
              o23_4 = fmaf(eb, g4_7, o23_4);
            }
            { const float eb = bi[215];
              o23_4 = fmaf(eb, g4_8, o23_4);
            }
            { const float eb = bi[216];
              o23_4 = fmaf(eb, g4_15, o23_4);
            }
            { const float eb = bi[217];
              o23_4 = fmaf(eb, g4_16, o23_4);
            }
            { const float eb = bi[218];
              o23_4 = fmaf(eb, g4_27, o23_4);
            }
            { const float eb = bi[219];
              o24_4 = fmaf(eb, g4_0, o24_4);
            }
            { const float eb = bi[220];
              o24_4 = fmaf(eb, g4_1, o24_4);
            }
            { const float eb = bi[221];
              o24_4 = fmaf(eb, g4_3, o24_4);
            }
            { const float eb = bi[222];
              o24_4 = fmaf(eb, g4_7, o24_4);
            }
            { const float eb = bi[223];
              o24_4 = fmaf(eb, g4_9, o24_4);
            }
            { const float eb = bi[224];
              o24_4 = fmaf(eb, g4_17, o24_4);
            }
            { const float eb = bi[225];
              o24_4 = fmaf(eb, g4_19, o24_4);
            }
            { const float eb = bi[226];
              o24_4 = fmaf(eb, g4_32, o24_4);
            }
            { const float eb = bi[227];
              o25_4 = fmaf(eb, g4_0, o25_4);
            }
            { const float eb = bi[228];
              o25_4 = fmaf(eb, g4_1, o25_4);
            }
            { const float eb = bi[229];
              o25_4 = fmaf(eb, g4_2, o25_4);
            }
            { const float eb = bi[230];
              o25_4 = fmaf(eb, g4_5, o25_4);
            }
            { const float eb = bi[231];
              o25_4 = fmaf(eb, g4_6, o25_4);
            }
            { const float eb = bi[232];
              o25_4 = fmaf(eb, g4_12, o25_4);
            }
            { const float eb = bi[233];
              o25_4 = fmaf(eb, g4_3, o25_4);
            }
            { const float eb = bi[234];
              o25_4 = fmaf(eb, g4_7, o25_4);
            }
            { const float eb = bi[235];
              o25_4 = fmaf(eb, g4_8, o25_4);
            }
            { const float eb = bi[236];
              o25_4 = fmaf(eb, g4_15, o25_4);
            }
            { const float eb = bi[237];
              o25_4 = fmaf(eb, g4_16, o25_4);
            }
            { const float eb = bi[238];
              o25_4 = fmaf(eb, g4_27, o25_4);
            }
            { const float eb = bi[239];
              o26_4 = fmaf(eb, g4_0, o26_4);
            }
            { const float eb = bi[240];
              o26_4 = fmaf(eb, g4_1, o26_4);
            }
            { const float eb = bi[241];
              o26_4 = fmaf(eb, g4_4, o26_4);
            }
            { const float eb = bi[242];
              o26_4 = fmaf(eb, g4_10, o26_4);
            }
            { const float eb = bi[243];
              o26_4 = fmaf(eb, g4_3, o26_4);
            }
            { const float eb = bi[244];
              o26_4 = fmaf(eb, g4_7, o26_4);
            }
            { const float eb = bi[245];
              o26_4 = fmaf(eb, g4_14, o26_4);
            }
            { const float eb = bi[246];
              o26_4 = fmaf(eb, g4_25, o26_4);
            }
            { const float eb = bi[247];
              o27_4 = fmaf(eb, g4_0, o27_4);
            }
            { const float eb = bi[248];
              o27_4 = fmaf(eb, g4_1, o27_4);
            }
            { const float eb = bi[249];
              o27_4 = fmaf(eb, g4_2, o27_4);
            }
            { const float eb = bi[250];
              o27_4 = fmaf(eb, g4_5, o27_4);
            }
            { const float eb = bi[251];
              o27_4 = fmaf(eb, g4_3, o27_4);
            }
            { const float eb = bi[252];
              o27_4 = fmaf(eb, g4_7, o27_4);
            }
            { const float eb = bi[253];
              o27_4 = fmaf(eb, g4_8, o27_4);
            }
            { const float eb = bi[254];
              o27_4 = fmaf(eb, g4_15, o27_4);
            }
            { const float eb = bi[255];
              o27_4 = fmaf(eb, g4_9, o27_4);
            }
            { const float eb = bi[256];
              o27_4 = fmaf(eb, g4_17, o27_4);
            }
            { const float eb = bi[257];
              o27_4 = fmaf(eb, g4_18, o27_4);
            }
            { const float eb = bi[258];
              o27_4 = fmaf(eb, g4_30, o27_4);
            }
            { const float eb = bi[259];
              o28_4 = fmaf(eb, g4_0, o28_4);
            }
            { const float eb = bi[260];
              o28_4 = fmaf(eb, g4_1, o28_4);
            }
            { const float eb = bi[261];
              o28_4 = fmaf(eb, g4_4, o28_4);
            }
            { const float eb = bi[262];
              o28_4 = fmaf(eb, g4_3, o28_4);
            }
            { const float eb = bi[263];
              o28_4 = fmaf(eb, g4_7, o28_4);
            }
            { const float eb = bi[264];
              o28_4 = fmaf(eb, g4_14, o28_4);
            }
            { const float eb = bi[265];
              o28_4 = fmaf(eb, g4_9, o28_4);
            }
            { const float eb = bi[266];
              o28_4 = fmaf(eb, g4_17, o28_4);
            }
            { const float eb = bi[267];
              o28_4 = fmaf(eb, g4_29, o28_4);
            }
            { const float eb = bi[268];
              o29_4 = fmaf(eb, g4_0, o29_4);
            }
            { const float eb = bi[269];
              o29_4 = fmaf(eb, g4_1, o29_4);
            }
            { const float eb = bi[270];
              o29_4 = fmaf(eb, g4_4, o29_4);
            }
            { const float eb = bi[271];
              o29_4 = fmaf(eb, g4_2, o29_4);
            }
            { const float eb = bi[272];
              o29_4 = fmaf(eb, g4_5, o29_4);
            }
            { const float eb = bi[273];
              o29_4 = fmaf(eb, g4_11, o29_4);
            }
            { const float eb = bi[274];
              o29_4 = fmaf(eb, g4_3, o29_4);
            }
            { const float eb = bi[275];
              o29_4 = fmaf(eb, g4_7, o29_4);
            }
            { const float eb = bi[276];
              o29_4 = fmaf(eb, g4_14, o29_4);
            }
            { const float eb = bi[277];
              o29_4 = fmaf(eb, g4_8, o29_4);
            }
            { const float eb = bi[278];
              o29_4 = fmaf(eb, g4_15, o29_4);
            }
            { const float eb = bi[279];
              o29_4 = fmaf(eb, g4_26, o29_4);
            }
            { const float eb = bi[280];
              o30_4 = fmaf(eb, g4_0, o30_4);
            }
            { const float eb = bi[281];
              o30_4 = fmaf(eb, g4_1, o30_4);
            }
            { const float eb = bi[282];
              o30_4 = fmaf(eb, g4_2, o30_4);
            }
            { const float eb = bi[283];
              o30_4 = fmaf(eb, g4_5, o30_4);
            }
            { const float eb = bi[284];
              o30_4 = fmaf(eb, g4_3, o30_4);
            }
            { const float eb = bi[285];
              o30_4 = fmaf(eb, g4_7, o30_4);
            }
            { const float eb = bi[286];
              o30_4 = fmaf(eb, g4_8, o30_4);
            }
            { const float eb = bi[287];
              o30_4 = fmaf(eb, g4_15, o30_4);
            }
            { const float eb = bi[288];
              o30_4 = fmaf(eb, g4_9, o30_4);
            }
            { const float eb = bi[289];
              o30_4 = fmaf(eb, g4_17, o30_4);
            }
            { const float eb = bi[290];
              o30_4 = fmaf(eb, g4_18, o30_4);
            }
            { const float eb = bi[291];
              o30_4 = fmaf(eb, g4_30, o30_4);
            }
            { const float eb = bi[292];
              o31_4 = fmaf(eb, g4_0, o31_4);
            }
            { const float eb = bi[293];
              o31_4 = fmaf(eb, g4_1, o31_4);
            }
            { const float eb = bi[294];
              o31_4 = fmaf(eb, g4_2, o31_4);
            }
            { const float eb = bi[295];
              o31_4 = fmaf(eb, g4_5, o31_4);
            }
            { const float eb = bi[296];
              o31_4 = fmaf(eb, g4_6, o31_4);
            }
            { const float eb = bi[297];
              o31_4 = fmaf(eb, g4_12, o31_4);
            }
            { const float eb = bi[298];
              o31_4 = fmaf(eb, g4_13, o31_4);
            }
            { const float eb = bi[299];
              o31_4 = fmaf(eb, g4_23, o31_4);
            }
            { const float eb = bi[300];
              o32_4 = fmaf(eb, g4_0, o32_4);
            }
            { const float eb = bi[301];
              o32_4 = fmaf(eb, g4_1, o32_4);
            }
            { const float eb = bi[302];
              o32_4 = fmaf(eb, g4_4, o32_4);
            }
            { const float eb = bi[303];
              o32_4 = fmaf(eb, g4_10, o32_4);
            }
            { const float eb = bi[304];
              o32_4 = fmaf(eb, g4_2, o32_4);
            }
            { const float eb = bi[305];
              o32_4 = fmaf(eb, g4_5, o32_4);
            }
            { const float eb = bi[306];
              o32_4 = fmaf(eb, g4_11, o32_4);
            }
            { const float eb = bi[307];
              o32_4 = fmaf(eb, g4_21, o32_4);
            }
            { const float eb = bi[308];
              o33_4 = fmaf(eb, g4_0, o33_4);
            }
            { const float eb = bi[309];
              o33_4 = fmaf(eb, g4_1, o33_4);
            }
            { const float eb = bi[310];
              o33_4 = fmaf(eb, g4_2, o33_4);
            }
            { const float eb = bi[311];
              o33_4 = fmaf(eb, g4_5, o33_4);
            }
            { const float eb = bi[312];
              o33_4 = fmaf(eb, g4_6, o33_4);
            }
            { const float eb = bi[313];
              o33_4 = fmaf(eb, g4_12, o33_4);
            }
            { const float eb = bi[314];
              o33_4 = fmaf(eb, g4_3, o33_4);
            }
            { const float eb = bi[315];
              o33_4 = fmaf(eb, g4_7, o33_4);
            }
            { const float eb = bi[316];
              o33_4 = fmaf(eb, g4_8, o33_4);
            }
            { const float eb = bi[317];
              o33_4 = fmaf(eb, g4_15, o33_4);
            }
            { const float eb = bi[318];
              o33_4 = fmaf(eb, g4_16, o33_4);
            }
            { const float eb = bi[319];
              o33_4 = fmaf(eb, g4_27, o33_4);
            }
            { const float eb = bi[320];
              o34_4 = fmaf(eb, g4_0, o34_4);
            }
            { const float eb = bi[321];
              o34_4 = fmaf(eb, g4_1, o34_4);
            }
            { const float eb = bi[322];
              o34_4 = fmaf(eb, g4_4, o34_4);
            }
            { const float eb = bi[323];
              o34_4 = fmaf(eb, g4_2, o34_4);
            }
            { const float eb = bi[324];
              o34_4 = fmaf(eb, g4_5, o34_4);
            }
            { const float eb = bi[325];
              o34_4 = fmaf(eb, g4_11, o34_4);
            }
            { const float eb = bi[326];
              o34_4 = fmaf(eb, g4_3, o34_4);
            }
            { const float eb = bi[327];
              o34_4 = fmaf(eb, g4_7, o34_4);
            }
            { const float eb = bi[328];
              o34_4 = fmaf(eb, g4_14, o34_4);
            }
            { const float eb = bi[329];
              o34_4 = fmaf(eb, g4_8, o34_4);
            }
            { const float eb = bi[330];
              o34_4 = fmaf(eb, g4_15, o34_4);
            }
            { const float eb = bi[331];
              o34_4 = fmaf(eb, g4_26, o34_4);
            }
            { const float eb = bi[332];
              o35_4 = fmaf(eb, g4_0, o35_4);
            }
            { const float eb = bi[333];
              o35_4 = fmaf(eb, g4_1, o35_4);
            }
            { const float eb = bi[334];
              o35_4 = fmaf(eb, g4_4, o35_4);
            }
            { const float eb = bi[335];
              o35_4 = fmaf(eb, g4_2, o35_4);
            }
            { const float eb = bi[336];
              o35_4 = fmaf(eb, g4_5, o35_4);
            }
            { const float eb = bi[337];
              o35_4 = fmaf(eb, g4_11, o35_4);
            }
            { const float eb = bi[338];
              o35_4 = fmaf(eb, g4_6, o35_4);
            }
            { const float eb = bi[339];
              o35_4 = fmaf(eb, g4_12, o35_4);
            }
            { const float eb = bi[340];
              o35_4 = fmaf(eb, g4_22, o35_4);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk4 = PT[(fI + 1) * N + fJ + 0];
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
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_4 * ptb0 + o1_4 * ptb1 + o2_4 * ptb2 + o3_4 * ptb3 + o4_4 * ptb4 + o5_4 * ptb5 + o6_4 * ptb6 + o7_4 * ptb7 + o8_4 * ptb8 + o9_4 * ptb9 + o10_4 * ptb10 + o11_4 * ptb11 + o12_4 * ptb12 + o13_4 * ptb13 + o14_4 * ptb14 + o15_4 * ptb15 + o16_4 * ptb16 + o17_4 * ptb17 + o18_4 * ptb18 + o19_4 * ptb19 + o20_4 * ptb20 + o21_4 * ptb21 + o22_4 * ptb22 + o23_4 * ptb23 + o24_4 * ptb24 + o25_4 * ptb25 + o26_4 * ptb26 + o27_4 * ptb27 + o28_4 * ptb28 + o29_4 * ptb29 + o30_4 * ptb30 + o31_4 * ptb31 + o32_4 * ptb32 + o33_4 * ptb33 + o34_4 * ptb34 + o35_4 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_4 * Abd0_0 + o1_4 * Abd1_0 + o2_4 * Abd2_0 + o3_4 * Abd3_0 + o4_4 * Abd4_0 + o5_4 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_4 * Aad0_0 + o6_4 * Aad1_0 + o12_4 * Aad2_0 + o18_4 * Aad3_0 + o24_4 * Aad4_0 + o30_4 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_4 * Abc0_1 + o1_4 * Abc1_1 + o2_4 * Abc2_1 + o3_4 * Abc3_1 + o4_4 * Abc4_1 + o5_4 * Abc5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_4 * Aac0_1 + o6_4 * Aac1_1 + o12_4 * Aac2_1 + o18_4 * Aac3_1 + o24_4 * Aac4_1 + o30_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_4 * Aad0_0 + o7_4 * Aad1_0 + o13_4 * Aad2_0 + o19_4 * Aad3_0 + o25_4 * Aad4_0 + o31_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_4 * Aac0_1 + o7_4 * Aac1_1 + o13_4 * Aac2_1 + o19_4 * Aac3_1 + o25_4 * Aac4_1 + o31_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_4 * Aad0_0 + o8_4 * Aad1_0 + o14_4 * Aad2_0 + o20_4 * Aad3_0 + o26_4 * Aad4_0 + o32_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_4 * Aac0_1 + o8_4 * Aac1_1 + o14_4 * Aac2_1 + o20_4 * Aac3_1 + o26_4 * Aac4_1 + o32_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_4 * Aad0_0 + o9_4 * Aad1_0 + o15_4 * Aad2_0 + o21_4 * Aad3_0 + o27_4 * Aad4_0 + o33_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_4 * Aac0_1 + o9_4 * Aac1_1 + o15_4 * Aac2_1 + o21_4 * Aac3_1 + o27_4 * Aac4_1 + o33_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 1, deg * (o4_4 * Aad0_0 + o10_4 * Aad1_0 + o16_4 * Aad2_0 + o22_4 * Aad3_0 + o28_4 * Aad4_0 + o34_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_4 * Aac0_1 + o10_4 * Aac1_1 + o16_4 * Aac2_1 + o22_4 * Aac3_1 + o28_4 * Aac4_1 + o34_4 * Aac5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 1, deg * (o5_4 * Aad0_0 + o11_4 * Aad1_0 + o17_4 * Aad2_0 + o23_4 * Aad3_0 + o29_4 * Aad4_0 + o35_4 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_4 * Aac0_1 + o11_4 * Aac1_1 + o17_4 * Aac2_1 + o23_4 * Aac3_1 + o29_4 * Aac4_1 + o35_4 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o6_4 * Abd0_0 + o7_4 * Abd1_0 + o8_4 * Abd2_0 + o9_4 * Abd3_0 + o10_4 * Abd4_0 + o11_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_4 * Abc0_1 + o7_4 * Abc1_1 + o8_4 * Abc2_1 + o9_4 * Abc3_1 + o10_4 * Abc4_1 + o11_4 * Abc5_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o12_4 * Abd0_0 + o13_4 * Abd1_0 + o14_4 * Abd2_0 + o15_4 * Abd3_0 + o16_4 * Abd4_0 + o17_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_4 * Abc0_1 + o13_4 * Abc1_1 + o14_4 * Abc2_1 + o15_4 * Abc3_1 + o16_4 * Abc4_1 + o17_4 * Abc5_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o18_4 * Abd0_0 + o19_4 * Abd1_0 + o20_4 * Abd2_0 + o21_4 * Abd3_0 + o22_4 * Abd4_0 + o23_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_4 * Abc0_1 + o19_4 * Abc1_1 + o20_4 * Abc2_1 + o21_4 * Abc3_1 + o22_4 * Abc4_1 + o23_4 * Abc5_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o24_4 * Abd0_0 + o25_4 * Abd1_0 + o26_4 * Abd2_0 + o27_4 * Abd3_0 + o28_4 * Abd4_0 + o29_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_4 * Abc0_1 + o25_4 * Abc1_1 + o26_4 * Abc2_1 + o27_4 * Abc3_1 + o28_4 * Abc4_1 + o29_4 * Abc5_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o30_4 * Abd0_0 + o31_4 * Abd1_0 + o32_4 * Abd2_0 + o33_4 * Abd3_0 + o34_4 * Abd4_0 + o35_4 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_4 * Abc0_1 + o31_4 * Abc1_1 + o32_4 * Abc2_1 + o33_4 * Abc3_1 + o34_4 * Abc4_1 + o35_4 * Abc5_1));
          }
        } break;
        case 5: {  // ket functions [5]
          float o0_5 = 0;
          float o1_5 = 0;
          float o2_5 = 0;
          float o3_5 = 0;
          float o4_5 = 0;
          float o5_5 = 0;
          float o6_5 = 0;
          float o7_5 = 0;
          float o8_5 = 0;
          float o9_5 = 0;
          float o10_5 = 0;
          float o11_5 = 0;
          float o12_5 = 0;
          float o13_5 = 0;
          float o14_5 = 0;
          float o15_5 = 0;
          float o16_5 = 0;
          float o17_5 = 0;
          float o18_5 = 0;
          float o19_5 = 0;
          float o20_5 = 0;
          float o21_5 = 0;
          float o22_5 = 0;
          float o23_5 = 0;
          float o24_5 = 0;
          float o25_5 = 0;
          float o26_5 = 0;
          float o27_5 = 0;
          float o28_5 = 0;
          float o29_5 = 0;
          float o30_5 = 0;
          float o31_5 = 0;
          float o32_5 = 0;
          float o33_5 = 0;
          float o34_5 = 0;
          float o35_5 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
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
            float g5_10 = 0;
            float g5_11 = 0;
            float g5_12 = 0;
            float g5_13 = 0;
            float g5_14 = 0;
            float g5_15 = 0;
            float g5_16 = 0;
            float g5_17 = 0;
            float g5_18 = 0;
            float g5_19 = 0;
            float g5_20 = 0;
            float g5_21 = 0;
            float g5_22 = 0;
            float g5_23 = 0;
            float g5_24 = 0;
            float g5_25 = 0;
            float g5_26 = 0;
            float g5_27 = 0;
            float g5_28 = 0;
            float g5_29 = 0;
            float g5_30 = 0;
            float g5_31 = 0;
            float g5_32 = 0;
            float g5_33 = 0;
            float g5_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek5_0 = kj[20 * kS];
              const float ek5_1 = -kj[21 * kS];
              const float ek5_2 = -kj[22 * kS];
              const float ek5_3 = kj[23 * kS];
              g5_0 = fmaf(ek5_0, b0, g5_0);
              const float r0_0_0_1 = Z * b1;
              g5_1 = fmaf(ek5_0, r0_0_0_1, g5_1);
              const float r0_0_1_0 = Y * b1;
              g5_2 = fmaf(ek5_0, r0_0_1_0, g5_2);
              g5_0 = fmaf(ek5_1, r0_0_1_0, g5_0);
              const float r0_1_0_0 = X * b1;
              g5_3 = fmaf(ek5_0, r0_1_0_0, g5_3);
              g5_0 = fmaf(ek5_2, r0_1_0_0, g5_0);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g5_4 = fmaf(ek5_0, r0_0_0_2, g5_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g5_5 = fmaf(ek5_0, r0_0_1_1, g5_5);
              g5_1 = fmaf(ek5_1, r0_0_1_1, g5_1);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g5_6 = fmaf(ek5_0, r0_0_2_0, g5_6);
              g5_2 = fmaf(ek5_1, r0_0_2_0, g5_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g5_7 = fmaf(ek5_0, r0_1_0_1, g5_7);
              g5_1 = fmaf(ek5_2, r0_1_0_1, g5_1);
              const float r0_1_1_0 = X * r1_0_1_0;
              g5_8 = fmaf(ek5_0, r0_1_1_0, g5_8);
              g5_3 = fmaf(ek5_1, r0_1_1_0, g5_3);
              g5_2 = fmaf(ek5_2, r0_1_1_0, g5_2);
              g5_0 = fmaf(ek5_3, r0_1_1_0, g5_0);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g5_9 = fmaf(ek5_0, r0_2_0_0, g5_9);
              g5_3 = fmaf(ek5_2, r0_2_0_0, g5_3);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g5_10 = fmaf(ek5_0, r0_0_0_3, g5_10);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g5_11 = fmaf(ek5_0, r0_0_1_2, g5_11);
              g5_4 = fmaf(ek5_1, r0_0_1_2, g5_4);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g5_12 = fmaf(ek5_0, r0_0_2_1, g5_12);
              g5_5 = fmaf(ek5_1, r0_0_2_1, g5_5);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g5_13 = fmaf(ek5_0, r0_0_3_0, g5_13);
              g5_6 = fmaf(ek5_1, r0_0_3_0, g5_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g5_14 = fmaf(ek5_0, r0_1_0_2, g5_14);
              g5_4 = fmaf(ek5_2, r0_1_0_2, g5_4);
              const float r0_1_1_1 = X * r1_0_1_1;
              g5_15 = fmaf(ek5_0, r0_1_1_1, g5_15);
              g5_7 = fmaf(ek5_1, r0_1_1_1, g5_7);
              g5_5 = fmaf(ek5_2, r0_1_1_1, g5_5);
              g5_1 = fmaf(ek5_3, r0_1_1_1, g5_1);
              const float r0_1_2_0 = X * r1_0_2_0;
              g5_16 = fmaf(ek5_0, r0_1_2_0, g5_16);
              g5_8 = fmaf(ek5_1, r0_1_2_0, g5_8);
              g5_6 = fmaf(ek5_2, r0_1_2_0, g5_6);
              g5_2 = fmaf(ek5_3, r0_1_2_0, g5_2);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g5_17 = fmaf(ek5_0, r0_2_0_1, g5_17);
              g5_7 = fmaf(ek5_2, r0_2_0_1, g5_7);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g5_18 = fmaf(ek5_0, r0_2_1_0, g5_18);
              g5_9 = fmaf(ek5_1, r0_2_1_0, g5_9);
              g5_8 = fmaf(ek5_2, r0_2_1_0, g5_8);
              g5_3 = fmaf(ek5_3, r0_2_1_0, g5_3);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g5_19 = fmaf(ek5_0, r0_3_0_0, g5_19);
              g5_9 = fmaf(ek5_2, r0_3_0_0, g5_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g5_20 = fmaf(ek5_0, r0_0_0_4, g5_20);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g5_21 = fmaf(ek5_0, r0_0_1_3, g5_21);
              g5_10 = fmaf(ek5_1, r0_0_1_3, g5_10);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g5_22 = fmaf(ek5_0, r0_0_2_2, g5_22);
              g5_11 = fmaf(ek5_1, r0_0_2_2, g5_11);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g5_23 = fmaf(ek5_0, r0_0_3_1, g5_23);
              g5_12 = fmaf(ek5_1, r0_0_3_1, g5_12);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g5_24 = fmaf(ek5_0, r0_0_4_0, g5_24);
              g5_13 = fmaf(ek5_1, r0_0_4_0, g5_13);
              const float r0_1_0_3 = X * r1_0_0_3;
              g5_25 = fmaf(ek5_0, r0_1_0_3, g5_25);
              g5_10 = fmaf(ek5_2, r0_1_0_3, g5_10);
              const float r0_1_1_2 = X * r1_0_1_2;
              g5_26 = fmaf(ek5_0, r0_1_1_2, g5_26);
              g5_14 = fmaf(ek5_1, r0_1_1_2, g5_14);
              g5_11 = fmaf(ek5_2, r0_1_1_2, g5_11);
              g5_4 = fmaf(ek5_3, r0_1_1_2, g5_4);
              const float r0_1_2_1 = X * r1_0_2_1;
              g5_27 = fmaf(ek5_0, r0_1_2_1, g5_27);
              g5_15 = fmaf(ek5_1, r0_1_2_1, g5_15);
              g5_12 = fmaf(ek5_2, r0_1_2_1, g5_12);
              g5_5 = fmaf(ek5_3, r0_1_2_1, g5_5);
              const float r0_1_3_0 = X * r1_0_3_0;
              g5_28 = fmaf(ek5_0, r0_1_3_0, g5_28);
              g5_16 = fmaf(ek5_1, r0_1_3_0, g5_16);
              g5_13 = fmaf(ek5_2, r0_1_3_0, g5_13);
              g5_6 = fmaf(ek5_3, r0_1_3_0, g5_6);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g5_29 = fmaf(ek5_0, r0_2_0_2, g5_29);
              g5_14 = fmaf(ek5_2, r0_2_0_2, g5_14);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g5_30 = fmaf(ek5_0, r0_2_1_1, g5_30);
              g5_17 = fmaf(ek5_1, r0_2_1_1, g5_17);
              g5_15 = fmaf(ek5_2, r0_2_1_1, g5_15);
              g5_7 = fmaf(ek5_3, r0_2_1_1, g5_7);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g5_31 = fmaf(ek5_0, r0_2_2_0, g5_31);
              g5_18 = fmaf(ek5_1, r0_2_2_0, g5_18);
              g5_16 = fmaf(ek5_2, r0_2_2_0, g5_16);
              g5_8 = fmaf(ek5_3, r0_2_2_0, g5_8);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g5_32 = fmaf(ek5_0, r0_3_0_1, g5_32);
              g5_17 = fmaf(ek5_2, r0_3_0_1, g5_17);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g5_33 = fmaf(ek5_0, r0_3_1_0, g5_33);
              g5_19 = fmaf(ek5_1, r0_3_1_0, g5_19);
              g5_18 = fmaf(ek5_2, r0_3_1_0, g5_18);
              g5_9 = fmaf(ek5_3, r0_3_1_0, g5_9);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g5_34 = fmaf(ek5_0, r0_4_0_0, g5_34);
              g5_19 = fmaf(ek5_2, r0_4_0_0, g5_19);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g5_20 = fmaf(ek5_1, r0_0_1_4, g5_20);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g5_21 = fmaf(ek5_1, r0_0_2_3, g5_21);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g5_22 = fmaf(ek5_1, r0_0_3_2, g5_22);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g5_23 = fmaf(ek5_1, r0_0_4_1, g5_23);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_0_5_0 = fmaf(Y, r1_0_4_0, 4.0f * r1_0_3_0);
              g5_24 = fmaf(ek5_1, r0_0_5_0, g5_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g5_20 = fmaf(ek5_2, r0_1_0_4, g5_20);
              const float r0_1_1_3 = X * r1_0_1_3;
              g5_25 = fmaf(ek5_1, r0_1_1_3, g5_25);
              g5_21 = fmaf(ek5_2, r0_1_1_3, g5_21);
              g5_10 = fmaf(ek5_3, r0_1_1_3, g5_10);
              const float r0_1_2_2 = X * r1_0_2_2;
              g5_26 = fmaf(ek5_1, r0_1_2_2, g5_26);
              g5_22 = fmaf(ek5_2, r0_1_2_2, g5_22);
              g5_11 = fmaf(ek5_3, r0_1_2_2, g5_11);
              const float r0_1_3_1 = X * r1_0_3_1;
              g5_27 = fmaf(ek5_1, r0_1_3_1, g5_27);
              g5_23 = fmaf(ek5_2, r0_1_3_1, g5_23);
              g5_12 = fmaf(ek5_3, r0_1_3_1, g5_12);
              const float r0_1_4_0 = X * r1_0_4_0;
              g5_28 = fmaf(ek5_1, r0_1_4_0, g5_28);
              g5_24 = fmaf(ek5_2, r0_1_4_0, g5_24);
              g5_13 = fmaf(ek5_3, r0_1_4_0, g5_13);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g5_25 = fmaf(ek5_2, r0_2_0_3, g5_25);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g5_29 = fmaf(ek5_1, r0_2_1_2, g5_29);
              g5_26 = fmaf(ek5_2, r0_2_1_2, g5_26);
              g5_14 = fmaf(ek5_3, r0_2_1_2, g5_14);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g5_30 = fmaf(ek5_1, r0_2_2_1, g5_30);
              g5_27 = fmaf(ek5_2, r0_2_2_1, g5_27);
              g5_15 = fmaf(ek5_3, r0_2_2_1, g5_15);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g5_31 = fmaf(ek5_1, r0_2_3_0, g5_31);
              g5_28 = fmaf(ek5_2, r0_2_3_0, g5_28);
              g5_16 = fmaf(ek5_3, r0_2_3_0, g5_16);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g5_29 = fmaf(ek5_2, r0_3_0_2, g5_29);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g5_32 = fmaf(ek5_1, r0_3_1_1, g5_32);
              g5_30 = fmaf(ek5_2, r0_3_1_1, g5_30);
              g5_17 = fmaf(ek5_3, r0_3_1_1, g5_17);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g5_33 = fmaf(ek5_1, r0_3_2_0, g5_33);
              g5_31 = fmaf(ek5_2, r0_3_2_0, g5_31);
              g5_18 = fmaf(ek5_3, r0_3_2_0, g5_18);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g5_32 = fmaf(ek5_2, r0_4_0_1, g5_32);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g5_34 = fmaf(ek5_1, r0_4_1_0, g5_34);
              g5_33 = fmaf(ek5_2, r0_4_1_0, g5_33);
              g5_19 = fmaf(ek5_3, r0_4_1_0, g5_19);
              const float r4_1_0_0 = X * b5;
              const float r3_2_0_0 = fmaf(X, r4_1_0_0, b4);
              const float r2_3_0_0 = fmaf(X, r3_2_0_0, 2.0f * r3_1_0_0);
              const float r1_4_0_0 = fmaf(X, r2_3_0_0, 3.0f * r2_2_0_0);
              const float r0_5_0_0 = fmaf(X, r1_4_0_0, 4.0f * r1_3_0_0);
              g5_34 = fmaf(ek5_2, r0_5_0_0, g5_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_1_1_4 = X * r1_0_1_4;
              g5_20 = fmaf(ek5_3, r0_1_1_4, g5_20);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_1_2_3 = X * r1_0_2_3;
              g5_21 = fmaf(ek5_3, r0_1_2_3, g5_21);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_1_3_2 = X * r1_0_3_2;
              g5_22 = fmaf(ek5_3, r0_1_3_2, g5_22);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_1_4_1 = X * r1_0_4_1;
              g5_23 = fmaf(ek5_3, r0_1_4_1, g5_23);
              const float r5_0_1_0 = Y * b6;
              const float r4_0_2_0 = fmaf(Y, r5_0_1_0, b5);
              const float r3_0_3_0 = fmaf(Y, r4_0_2_0, 2.0f * r4_0_1_0);
              const float r2_0_4_0 = fmaf(Y, r3_0_3_0, 3.0f * r3_0_2_0);
              const float r1_0_5_0 = fmaf(Y, r2_0_4_0, 4.0f * r2_0_3_0);
              const float r0_1_5_0 = X * r1_0_5_0;
              g5_24 = fmaf(ek5_3, r0_1_5_0, g5_24);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g5_25 = fmaf(ek5_3, r0_2_1_3, g5_25);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g5_26 = fmaf(ek5_3, r0_2_2_2, g5_26);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g5_27 = fmaf(ek5_3, r0_2_3_1, g5_27);
              const float r1_1_4_0 = X * r2_0_4_0;
              const float r0_2_4_0 = fmaf(X, r1_1_4_0, r1_0_4_0);
              g5_28 = fmaf(ek5_3, r0_2_4_0, g5_28);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g5_29 = fmaf(ek5_3, r0_3_1_2, g5_29);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g5_30 = fmaf(ek5_3, r0_3_2_1, g5_30);
              const float r2_1_3_0 = X * r3_0_3_0;
              const float r1_2_3_0 = fmaf(X, r2_1_3_0, r2_0_3_0);
              const float r0_3_3_0 = fmaf(X, r1_2_3_0, 2.0f * r1_1_3_0);
              g5_31 = fmaf(ek5_3, r0_3_3_0, g5_31);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g5_32 = fmaf(ek5_3, r0_4_1_1, g5_32);
              const float r3_1_2_0 = X * r4_0_2_0;
              const float r2_2_2_0 = fmaf(X, r3_1_2_0, r3_0_2_0);
              const float r1_3_2_0 = fmaf(X, r2_2_2_0, 2.0f * r2_1_2_0);
              const float r0_4_2_0 = fmaf(X, r1_3_2_0, 3.0f * r1_2_2_0);
              g5_33 = fmaf(ek5_3, r0_4_2_0, g5_33);
              const float r4_1_1_0 = X * r5_0_1_0;
              const float r3_2_1_0 = fmaf(X, r4_1_1_0, r4_0_1_0);
              const float r2_3_1_0 = fmaf(X, r3_2_1_0, 2.0f * r3_1_1_0);
              const float r1_4_1_0 = fmaf(X, r2_3_1_0, 3.0f * r2_2_1_0);
              const float r0_5_1_0 = fmaf(X, r1_4_1_0, 4.0f * r1_3_1_0);
              g5_34 = fmaf(ek5_3, r0_5_1_0, g5_34);
            }
            { const float eb = bi[5];
              o0_5 = fmaf(eb, g5_0, o0_5);
            }
            { const float eb = bi[6];
              o0_5 = fmaf(eb, g5_3, o0_5);
            }
            { const float eb = bi[7];
              o0_5 = fmaf(eb, g5_9, o0_5);
            }
            { const float eb = bi[8];
              o0_5 = fmaf(eb, g5_19, o0_5);
            }
            { const float eb = bi[9];
              o0_5 = fmaf(eb, g5_34, o0_5);
            }
            { const float eb = bi[10];
              o1_5 = fmaf(eb, g5_0, o1_5);
            }
            { const float eb = bi[11];
              o1_5 = fmaf(eb, g5_2, o1_5);
            }
            { const float eb = bi[12];
              o1_5 = fmaf(eb, g5_6, o1_5);
            }
            { const float eb = bi[13];
              o1_5 = fmaf(eb, g5_3, o1_5);
            }
            { const float eb = bi[14];
              o1_5 = fmaf(eb, g5_8, o1_5);
            }
            { const float eb = bi[15];
              o1_5 = fmaf(eb, g5_16, o1_5);
            }
            { const float eb = bi[16];
              o1_5 = fmaf(eb, g5_9, o1_5);
            }
            { const float eb = bi[17];
              o1_5 = fmaf(eb, g5_18, o1_5);
            }
            { const float eb = bi[18];
              o1_5 = fmaf(eb, g5_31, o1_5);
            }
            { const float eb = bi[19];
              o2_5 = fmaf(eb, g5_0, o2_5);
            }
            { const float eb = bi[20];
              o2_5 = fmaf(eb, g5_1, o2_5);
            }
            { const float eb = bi[21];
              o2_5 = fmaf(eb, g5_4, o2_5);
            }
            { const float eb = bi[22];
              o2_5 = fmaf(eb, g5_3, o2_5);
            }
            { const float eb = bi[23];
              o2_5 = fmaf(eb, g5_7, o2_5);
            }
            { const float eb = bi[24];
              o2_5 = fmaf(eb, g5_14, o2_5);
            }
            { const float eb = bi[25];
              o2_5 = fmaf(eb, g5_9, o2_5);
            }
            { const float eb = bi[26];
              o2_5 = fmaf(eb, g5_17, o2_5);
            }
            { const float eb = bi[27];
              o2_5 = fmaf(eb, g5_29, o2_5);
            }
            { const float eb = bi[28];
              o3_5 = fmaf(eb, g5_0, o3_5);
            }
            { const float eb = bi[29];
              o3_5 = fmaf(eb, g5_2, o3_5);
            }
            { const float eb = bi[30];
              o3_5 = fmaf(eb, g5_3, o3_5);
            }
            { const float eb = bi[31];
              o3_5 = fmaf(eb, g5_8, o3_5);
            }
            { const float eb = bi[32];
              o3_5 = fmaf(eb, g5_9, o3_5);
            }
            { const float eb = bi[33];
              o3_5 = fmaf(eb, g5_18, o3_5);
            }
            { const float eb = bi[34];
              o3_5 = fmaf(eb, g5_19, o3_5);
            }
            { const float eb = bi[35];
              o3_5 = fmaf(eb, g5_33, o3_5);
            }
            { const float eb = bi[36];
              o4_5 = fmaf(eb, g5_0, o4_5);
            }
            { const float eb = bi[37];
              o4_5 = fmaf(eb, g5_1, o4_5);
            }
            { const float eb = bi[38];
              o4_5 = fmaf(eb, g5_3, o4_5);
            }
            { const float eb = bi[39];
              o4_5 = fmaf(eb, g5_7, o4_5);
            }
            { const float eb = bi[40];
              o4_5 = fmaf(eb, g5_9, o4_5);
            }
            { const float eb = bi[41];
              o4_5 = fmaf(eb, g5_17, o4_5);
            }
            { const float eb = bi[42];
              o4_5 = fmaf(eb, g5_19, o4_5);
            }
            { const float eb = bi[43];
              o4_5 = fmaf(eb, g5_32, o4_5);
            }
            { const float eb = bi[44];
              o5_5 = fmaf(eb, g5_0, o5_5);
            }
            { const float eb = bi[45];
              o5_5 = fmaf(eb, g5_1, o5_5);
            }
            { const float eb = bi[46];
              o5_5 = fmaf(eb, g5_2, o5_5);
            }
            { const float eb = bi[47];
              o5_5 = fmaf(eb, g5_5, o5_5);
            }
            { const float eb = bi[48];
              o5_5 = fmaf(eb, g5_3, o5_5);
            }
            { const float eb = bi[49];
              o5_5 = fmaf(eb, g5_7, o5_5);
            }
            { const float eb = bi[50];
              o5_5 = fmaf(eb, g5_8, o5_5);
            }
            { const float eb = bi[51];
              o5_5 = fmaf(eb, g5_15, o5_5);
            }
            { const float eb = bi[52];
              o5_5 = fmaf(eb, g5_9, o5_5);
            }
            { const float eb = bi[53];
              o5_5 = fmaf(eb, g5_17, o5_5);
            }
            { const float eb = bi[54];
              o5_5 = fmaf(eb, g5_18, o5_5);
            }
            { const float eb = bi[55];
              o5_5 = fmaf(eb, g5_30, o5_5);
            }
            { const float eb = bi[56];
              o6_5 = fmaf(eb, g5_0, o6_5);
            }
            { const float eb = bi[57];
              o6_5 = fmaf(eb, g5_2, o6_5);
            }
            { const float eb = bi[58];
              o6_5 = fmaf(eb, g5_6, o6_5);
            }
            { const float eb = bi[59];
              o6_5 = fmaf(eb, g5_3, o6_5);
            }
            { const float eb = bi[60];
              o6_5 = fmaf(eb, g5_8, o6_5);
            }
            { const float eb = bi[61];
              o6_5 = fmaf(eb, g5_16, o6_5);
            }
            { const float eb = bi[62];
              o6_5 = fmaf(eb, g5_9, o6_5);
            }
            { const float eb = bi[63];
              o6_5 = fmaf(eb, g5_18, o6_5);
            }
            { const float eb = bi[64];
              o6_5 = fmaf(eb, g5_31, o6_5);
            }
            { const float eb = bi[65];
              o7_5 = fmaf(eb, g5_0, o7_5);
            }
            { const float eb = bi[66];
              o7_5 = fmaf(eb, g5_2, o7_5);
            }
            { const float eb = bi[67];
              o7_5 = fmaf(eb, g5_6, o7_5);
            }
            { const float eb = bi[68];
              o7_5 = fmaf(eb, g5_13, o7_5);
            }
            { const float eb = bi[69];
              o7_5 = fmaf(eb, g5_24, o7_5);
            }
            { const float eb = bi[70];
              o8_5 = fmaf(eb, g5_0, o8_5);
            }
            { const float eb = bi[71];
              o8_5 = fmaf(eb, g5_1, o8_5);
            }
            { const float eb = bi[72];
              o8_5 = fmaf(eb, g5_4, o8_5);
            }
            { const float eb = bi[73];
              o8_5 = fmaf(eb, g5_2, o8_5);
            }
            { const float eb = bi[74];
              o8_5 = fmaf(eb, g5_5, o8_5);
            }
            { const float eb = bi[75];
              o8_5 = fmaf(eb, g5_11, o8_5);
            }
            { const float eb = bi[76];
              o8_5 = fmaf(eb, g5_6, o8_5);
            }
            { const float eb = bi[77];
              o8_5 = fmaf(eb, g5_12, o8_5);
            }
            { const float eb = bi[78];
              o8_5 = fmaf(eb, g5_22, o8_5);
            }
            { const float eb = bi[79];
              o9_5 = fmaf(eb, g5_0, o9_5);
            }
            { const float eb = bi[80];
              o9_5 = fmaf(eb, g5_2, o9_5);
            }
            { const float eb = bi[81];
              o9_5 = fmaf(eb, g5_6, o9_5);
            }
            { const float eb = bi[82];
              o9_5 = fmaf(eb, g5_13, o9_5);
            }
            { const float eb = bi[83];
              o9_5 = fmaf(eb, g5_3, o9_5);
            }
            { const float eb = bi[84];
              o9_5 = fmaf(eb, g5_8, o9_5);
            }
            { const float eb = bi[85];
              o9_5 = fmaf(eb, g5_16, o9_5);
            }
            { const float eb = bi[86];
              o9_5 = fmaf(eb, g5_28, o9_5);
            }
            { const float eb = bi[87];
              o10_5 = fmaf(eb, g5_0, o10_5);
            }
            { const float eb = bi[88];
              o10_5 = fmaf(eb, g5_1, o10_5);
            }
            { const float eb = bi[89];
              o10_5 = fmaf(eb, g5_2, o10_5);
            }
            { const float eb = bi[90];
              o10_5 = fmaf(eb, g5_5, o10_5);
            }
            { const float eb = bi[91];
              o10_5 = fmaf(eb, g5_6, o10_5);
            }
            { const float eb = bi[92];
              o10_5 = fmaf(eb, g5_12, o10_5);
            }
            { const float eb = bi[93];
              o10_5 = fmaf(eb, g5_3, o10_5);
            }
            { const float eb = bi[94];
              o10_5 = fmaf(eb, g5_7, o10_5);
            }
            { const float eb = bi[95];
              o10_5 = fmaf(eb, g5_8, o10_5);
            }
            { const float eb = bi[96];
              o10_5 = fmaf(eb, g5_15, o10_5);
            }
            { const float eb = bi[97];
              o10_5 = fmaf(eb, g5_16, o10_5);
            }
            { const float eb = bi[98];
              o10_5 = fmaf(eb, g5_27, o10_5);
            }
            { const float eb = bi[99];
              o11_5 = fmaf(eb, g5_0, o11_5);
            }
            { const float eb = bi[100];
              o11_5 = fmaf(eb, g5_1, o11_5);
            }
            { const float eb = bi[101];
              o11_5 = fmaf(eb, g5_2, o11_5);
            }
            { const float eb = bi[102];
              o11_5 = fmaf(eb, g5_5, o11_5);
            }
            { const float eb = bi[103];
              o11_5 = fmaf(eb, g5_6, o11_5);
            }
            { const float eb = bi[104];
              o11_5 = fmaf(eb, g5_12, o11_5);
            }
            { const float eb = bi[105];
              o11_5 = fmaf(eb, g5_13, o11_5);
            }
            { const float eb = bi[106];
              o11_5 = fmaf(eb, g5_23, o11_5);
            }
            { const float eb = bi[107];
              o12_5 = fmaf(eb, g5_0, o12_5);
            }
            { const float eb = bi[108];
              o12_5 = fmaf(eb, g5_1, o12_5);
            }
            { const float eb = bi[109];
              o12_5 = fmaf(eb, g5_4, o12_5);
            }
            { const float eb = bi[110];
              o12_5 = fmaf(eb, g5_3, o12_5);
            }
            { const float eb = bi[111];
              o12_5 = fmaf(eb, g5_7, o12_5);
            }
            { const float eb = bi[112];
              o12_5 = fmaf(eb, g5_14, o12_5);
            }
            { const float eb = bi[113];
              o12_5 = fmaf(eb, g5_9, o12_5);
            }
            { const float eb = bi[114];
              o12_5 = fmaf(eb, g5_17, o12_5);
            }
            { const float eb = bi[115];
              o12_5 = fmaf(eb, g5_29, o12_5);
            }
            { const float eb = bi[116];
              o13_5 = fmaf(eb, g5_0, o13_5);
            }
            { const float eb = bi[117];
              o13_5 = fmaf(eb, g5_1, o13_5);
            }
            { const float eb = bi[118];
              o13_5 = fmaf(eb, g5_4, o13_5);
            }
            { const float eb = bi[119];
              o13_5 = fmaf(eb, g5_2, o13_5);
            }
            { const float eb = bi[120];
              o13_5 = fmaf(eb, g5_5, o13_5);
            }
            { const float eb = bi[121];
              o13_5 = fmaf(eb, g5_11, o13_5);
            }
            { const float eb = bi[122];
              o13_5 = fmaf(eb, g5_6, o13_5);
            }
            { const float eb = bi[123];
              o13_5 = fmaf(eb, g5_12, o13_5);
            }
            { const float eb = bi[124];
              o13_5 = fmaf(eb, g5_22, o13_5);
            }
            { const float eb = bi[125];
              o14_5 = fmaf(eb, g5_0, o14_5);
            }
            { const float eb = bi[126];
              o14_5 = fmaf(eb, g5_1, o14_5);
            }
            { const float eb = bi[127];
              o14_5 = fmaf(eb, g5_4, o14_5);
            }
            { const float eb = bi[128];
              o14_5 = fmaf(eb, g5_10, o14_5);
            }
            { const float eb = bi[129];
              o14_5 = fmaf(eb, g5_20, o14_5);
            }
            { const float eb = bi[130];
              o15_5 = fmaf(eb, g5_0, o15_5);
            }
            { const float eb = bi[131];
              o15_5 = fmaf(eb, g5_1, o15_5);
            }
            { const float eb = bi[132];
              o15_5 = fmaf(eb, g5_4, o15_5);
            }
            { const float eb = bi[133];
              o15_5 = fmaf(eb, g5_2, o15_5);
            }
            { const float eb = bi[134];
              o15_5 = fmaf(eb, g5_5, o15_5);
            }
            { const float eb = bi[135];
              o15_5 = fmaf(eb, g5_11, o15_5);
            }
            { const float eb = bi[136];
              o15_5 = fmaf(eb, g5_3, o15_5);
            }
            { const float eb = bi[137];
              o15_5 = fmaf(eb, g5_7, o15_5);
            }
            { const float eb = bi[138];
              o15_5 = fmaf(eb, g5_14, o15_5);
            }
            { const float eb = bi[139];
              o15_5 = fmaf(eb, g5_8, o15_5);
            }
            { const float eb = bi[140];
              o15_5 = fmaf(eb, g5_15, o15_5);
            }
            { const float eb = bi[141];
              o15_5 = fmaf(eb, g5_26, o15_5);
            }
            { const float eb = bi[142];
              o16_5 = fmaf(eb, g5_0, o16_5);
            }
            { const float eb = bi[143];
              o16_5 = fmaf(eb, g5_1, o16_5);
            }
            { const float eb = bi[144];
              o16_5 = fmaf(eb, g5_4, o16_5);
            }
            { const float eb = bi[145];
              o16_5 = fmaf(eb, g5_10, o16_5);
            }
            { const float eb = bi[146];
              o16_5 = fmaf(eb, g5_3, o16_5);
            }
            { const float eb = bi[147];
              o16_5 = fmaf(eb, g5_7, o16_5);
            }
            { const float eb = bi[148];
              o16_5 = fmaf(eb, g5_14, o16_5);
            }
            { const float eb = bi[149];
              o16_5 = fmaf(eb, g5_25, o16_5);
            }
            { const float eb = bi[150];
              o17_5 = fmaf(eb, g5_0, o17_5);
            }
            { const float eb = bi[151];
              o17_5 = fmaf(eb, g5_1, o17_5);
            }
            { const float eb = bi[152];
              o17_5 = fmaf(eb, g5_4, o17_5);
            }
            { const float eb = bi[153];
              o17_5 = fmaf(eb, g5_10, o17_5);
            }
            { const float eb = bi[154];
              o17_5 = fmaf(eb, g5_2, o17_5);
            }
            { const float eb = bi[155];
              o17_5 = fmaf(eb, g5_5, o17_5);
            }
            { const float eb = bi[156];
              o17_5 = fmaf(eb, g5_11, o17_5);
            }
            { const float eb = bi[157];
              o17_5 = fmaf(eb, g5_21, o17_5);
            }
            { const float eb = bi[158];
              o18_5 = fmaf(eb, g5_0, o18_5);
            }
            { const float eb = bi[159];
              o18_5 = fmaf(eb, g5_2, o18_5);
            }
            { const float eb = bi[160];
              o18_5 = fmaf(eb, g5_3, o18_5);
            }
            { const float eb = bi[161];
              o18_5 = fmaf(eb, g5_8, o18_5);
            }
            { const float eb = bi[162];
              o18_5 = fmaf(eb, g5_9, o18_5);
            }
            { const float eb = bi[163];
              o18_5 = fmaf(eb, g5_18, o18_5);
            }
            { const float eb = bi[164];
              o18_5 = fmaf(eb, g5_19, o18_5);
            }
            { const float eb = bi[165];
              o18_5 = fmaf(eb, g5_33, o18_5);
            }
            { const float eb = bi[166];
              o19_5 = fmaf(eb, g5_0, o19_5);
            }
            { const float eb = bi[167];
              o19_5 = fmaf(eb, g5_2, o19_5);
            }
            { const float eb = bi[168];
              o19_5 = fmaf(eb, g5_6, o19_5);
            }
            { const float eb = bi[169];
              o19_5 = fmaf(eb, g5_13, o19_5);
            }
            { const float eb = bi[170];
              o19_5 = fmaf(eb, g5_3, o19_5);
            }
            { const float eb = bi[171];
              o19_5 = fmaf(eb, g5_8, o19_5);
            }
            { const float eb = bi[172];
              o19_5 = fmaf(eb, g5_16, o19_5);
            }
            { const float eb = bi[173];
              o19_5 = fmaf(eb, g5_28, o19_5);
            }
            { const float eb = bi[174];
              o20_5 = fmaf(eb, g5_0, o20_5);
            }
            { const float eb = bi[175];
              o20_5 = fmaf(eb, g5_1, o20_5);
            }
            { const float eb = bi[176];
              o20_5 = fmaf(eb, g5_4, o20_5);
            }
            { const float eb = bi[177];
              o20_5 = fmaf(eb, g5_2, o20_5);
            }
            { const float eb = bi[178];
              o20_5 = fmaf(eb, g5_5, o20_5);
            }
            { const float eb = bi[179];
              o20_5 = fmaf(eb, g5_11, o20_5);
            }
            { const float eb = bi[180];
              o20_5 = fmaf(eb, g5_3, o20_5);
            }
            { const float eb = bi[181];
              o20_5 = fmaf(eb, g5_7, o20_5);
            }
            { const float eb = bi[182];
              o20_5 = fmaf(eb, g5_14, o20_5);
            }
            { const float eb = bi[183];
              o20_5 = fmaf(eb, g5_8, o20_5);
            }
            { const float eb = bi[184];
              o20_5 = fmaf(eb, g5_15, o20_5);
            }
            { const float eb = bi[185];
              o20_5 = fmaf(eb, g5_26, o20_5);
            }
            { const float eb = bi[186];
              o21_5 = fmaf(eb, g5_0, o21_5);
            }
            { const float eb = bi[187];
              o21_5 = fmaf(eb, g5_2, o21_5);
            }
            { const float eb = bi[188];
              o21_5 = fmaf(eb, g5_6, o21_5);
            }
            { const float eb = bi[189];
              o21_5 = fmaf(eb, g5_3, o21_5);
            }
            { const float eb = bi[190];
              o21_5 = fmaf(eb, g5_8, o21_5);
            }
            { const float eb = bi[191];
              o21_5 = fmaf(eb, g5_16, o21_5);
            }
            { const float eb = bi[192];
              o21_5 = fmaf(eb, g5_9, o21_5);
            }
            { const float eb = bi[193];
              o21_5 = fmaf(eb, g5_18, o21_5);
            }
            { const float eb = bi[194];
              o21_5 = fmaf(eb, g5_31, o21_5);
            }
            { const float eb = bi[195];
              o22_5 = fmaf(eb, g5_0, o22_5);
            }
            { const float eb = bi[196];
              o22_5 = fmaf(eb, g5_1, o22_5);
            }
            { const float eb = bi[197];
              o22_5 = fmaf(eb, g5_2, o22_5);
            }
            { const float eb = bi[198];
              o22_5 = fmaf(eb, g5_5, o22_5);
            }
            { const float eb = bi[199];
              o22_5 = fmaf(eb, g5_3, o22_5);
            }
            { const float eb = bi[200];
              o22_5 = fmaf(eb, g5_7, o22_5);
            }
            { const float eb = bi[201];
              o22_5 = fmaf(eb, g5_8, o22_5);
            }
            { const float eb = bi[202];
              o22_5 = fmaf(eb, g5_15, o22_5);
            }
            { const float eb = bi[203];
              o22_5 = fmaf(eb, g5_9, o22_5);
            }
            { const float eb = bi[204];
              o22_5 = fmaf(eb, g5_17, o22_5);
            }
            { const float eb = bi[205];
              o22_5 = fmaf(eb, g5_18, o22_5);
            }
            { const float eb = bi[206];
              o22_5 = fmaf(eb, g5_30, o22_5);
            }
            { const float eb = bi[207];
              o23_5 = fmaf(eb, g5_0, o23_5);
            }
            { const float eb = bi[208];
              o23_5 = fmaf(eb, g5_1, o23_5);
            }
            { const float eb = bi[209];
              o23_5 = fmaf(eb, g5_2, o23_5);
            }
            { const float eb = bi[210];
              o23_5 = fmaf(eb, g5_5, o23_5);
            }
            { const float eb = bi[211];
              o23_5 = fmaf(eb, g5_6, o23_5);
            }
            { const float eb = bi[212];
              o23_5 = fmaf(eb, g5_12, o23_5);
            }
            { const float eb = bi[213];
              o23_5 = fmaf(eb, g5_3, o23_5);
            }
            { const float eb = bi[214];
              o23_5 = fmaf(eb, g5_7, o23_5);
            }
            { const float eb = bi[215];
              o23_5 = fmaf(eb, g5_8, o23_5);
            }
            { const float eb = bi[216];
              o23_5 = fmaf(eb, g5_15, o23_5);
            }
            { const float eb = bi[217];
              o23_5 = fmaf(eb, g5_16, o23_5);
            }
            { const float eb = bi[218];
              o23_5 = fmaf(eb, g5_27, o23_5);
            }
            { const float eb = bi[219];
              o24_5 = fmaf(eb, g5_0, o24_5);
            }
            { const float eb = bi[220];
              o24_5 = fmaf(eb, g5_1, o24_5);
            }
            { const float eb = bi[221];
              o24_5 = fmaf(eb, g5_3, o24_5);
            }
            { const float eb = bi[222];
              o24_5 = fmaf(eb, g5_7, o24_5);
            }
            { const float eb = bi[223];
              o24_5 = fmaf(eb, g5_9, o24_5);
            }
            { const float eb = bi[224];
              o24_5 = fmaf(eb, g5_17, o24_5);
            }
            { const float eb = bi[225];
              o24_5 = fmaf(eb, g5_19, o24_5);
            }
            { const float eb = bi[226];
              o24_5 = fmaf(eb, g5_32, o24_5);
            }
            { const float eb = bi[227];
              o25_5 = fmaf(eb, g5_0, o25_5);
            }
            { const float eb = bi[228];
              o25_5 = fmaf(eb, g5_1, o25_5);
            }
            { const float eb = bi[229];
              o25_5 = fmaf(eb, g5_2, o25_5);
            }
            { const float eb = bi[230];
              o25_5 = fmaf(eb, g5_5, o25_5);
            }
            { const float eb = bi[231];
              o25_5 = fmaf(eb, g5_6, o25_5);
            }
            { const float eb = bi[232];
              o25_5 = fmaf(eb, g5_12, o25_5);
            }
            { const float eb = bi[233];
              o25_5 = fmaf(eb, g5_3, o25_5);
            }
            { const float eb = bi[234];
              o25_5 = fmaf(eb, g5_7, o25_5);
            }
            { const float eb = bi[235];
              o25_5 = fmaf(eb, g5_8, o25_5);
            }
            { const float eb = bi[236];
              o25_5 = fmaf(eb, g5_15, o25_5);
            }
            { const float eb = bi[237];
              o25_5 = fmaf(eb, g5_16, o25_5);
            }
            { const float eb = bi[238];
              o25_5 = fmaf(eb, g5_27, o25_5);
            }
            { const float eb = bi[239];
              o26_5 = fmaf(eb, g5_0, o26_5);
            }
            { const float eb = bi[240];
              o26_5 = fmaf(eb, g5_1, o26_5);
            }
            { const float eb = bi[241];
              o26_5 = fmaf(eb, g5_4, o26_5);
            }
            { const float eb = bi[242];
              o26_5 = fmaf(eb, g5_10, o26_5);
            }
            { const float eb = bi[243];
              o26_5 = fmaf(eb, g5_3, o26_5);
            }
            { const float eb = bi[244];
              o26_5 = fmaf(eb, g5_7, o26_5);
            }
            { const float eb = bi[245];
              o26_5 = fmaf(eb, g5_14, o26_5);
            }
            { const float eb = bi[246];
              o26_5 = fmaf(eb, g5_25, o26_5);
            }
            { const float eb = bi[247];
              o27_5 = fmaf(eb, g5_0, o27_5);
            }
            { const float eb = bi[248];
              o27_5 = fmaf(eb, g5_1, o27_5);
            }
            { const float eb = bi[249];
              o27_5 = fmaf(eb, g5_2, o27_5);
            }
            { const float eb = bi[250];
              o27_5 = fmaf(eb, g5_5, o27_5);
            }
            { const float eb = bi[251];
              o27_5 = fmaf(eb, g5_3, o27_5);
            }
            { const float eb = bi[252];
              o27_5 = fmaf(eb, g5_7, o27_5);
            }
            { const float eb = bi[253];
              o27_5 = fmaf(eb, g5_8, o27_5);
            }
            { const float eb = bi[254];
              o27_5 = fmaf(eb, g5_15, o27_5);
            }
            { const float eb = bi[255];
              o27_5 = fmaf(eb, g5_9, o27_5);
            }
            { const float eb = bi[256];
              o27_5 = fmaf(eb, g5_17, o27_5);
            }
            { const float eb = bi[257];
              o27_5 = fmaf(eb, g5_18, o27_5);
            }
            { const float eb = bi[258];
              o27_5 = fmaf(eb, g5_30, o27_5);
            }
            { const float eb = bi[259];
              o28_5 = fmaf(eb, g5_0, o28_5);
            }
            { const float eb = bi[260];
              o28_5 = fmaf(eb, g5_1, o28_5);
            }
            { const float eb = bi[261];
              o28_5 = fmaf(eb, g5_4, o28_5);
            }
            { const float eb = bi[262];
              o28_5 = fmaf(eb, g5_3, o28_5);
            }
            { const float eb = bi[263];
              o28_5 = fmaf(eb, g5_7, o28_5);
            }
            { const float eb = bi[264];
              o28_5 = fmaf(eb, g5_14, o28_5);
            }
            { const float eb = bi[265];
              o28_5 = fmaf(eb, g5_9, o28_5);
            }
            { const float eb = bi[266];
              o28_5 = fmaf(eb, g5_17, o28_5);
            }
            { const float eb = bi[267];
              o28_5 = fmaf(eb, g5_29, o28_5);
            }
            { const float eb = bi[268];
              o29_5 = fmaf(eb, g5_0, o29_5);
            }
            { const float eb = bi[269];
              o29_5 = fmaf(eb, g5_1, o29_5);
            }
            { const float eb = bi[270];
              o29_5 = fmaf(eb, g5_4, o29_5);
            }
            { const float eb = bi[271];
              o29_5 = fmaf(eb, g5_2, o29_5);
            }
            { const float eb = bi[272];
              o29_5 = fmaf(eb, g5_5, o29_5);
            }
            { const float eb = bi[273];
              o29_5 = fmaf(eb, g5_11, o29_5);
            }
            { const float eb = bi[274];
              o29_5 = fmaf(eb, g5_3, o29_5);
            }
            { const float eb = bi[275];
              o29_5 = fmaf(eb, g5_7, o29_5);
            }
            { const float eb = bi[276];
              o29_5 = fmaf(eb, g5_14, o29_5);
            }
            { const float eb = bi[277];
              o29_5 = fmaf(eb, g5_8, o29_5);
            }
            { const float eb = bi[278];
              o29_5 = fmaf(eb, g5_15, o29_5);
            }
            { const float eb = bi[279];
              o29_5 = fmaf(eb, g5_26, o29_5);
            }
            { const float eb = bi[280];
              o30_5 = fmaf(eb, g5_0, o30_5);
            }
            { const float eb = bi[281];
              o30_5 = fmaf(eb, g5_1, o30_5);
            }
            { const float eb = bi[282];
              o30_5 = fmaf(eb, g5_2, o30_5);
            }
            { const float eb = bi[283];
              o30_5 = fmaf(eb, g5_5, o30_5);
            }
            { const float eb = bi[284];
              o30_5 = fmaf(eb, g5_3, o30_5);
            }
            { const float eb = bi[285];
              o30_5 = fmaf(eb, g5_7, o30_5);
            }
            { const float eb = bi[286];
              o30_5 = fmaf(eb, g5_8, o30_5);
            }
            { const float eb = bi[287];
              o30_5 = fmaf(eb, g5_15, o30_5);
            }
            { const float eb = bi[288];
              o30_5 = fmaf(eb, g5_9, o30_5);
            }
            { const float eb = bi[289];
              o30_5 = fmaf(eb, g5_17, o30_5);
            }
            { const float eb = bi[290];
              o30_5 = fmaf(eb, g5_18, o30_5);
            }
            { const float eb = bi[291];
              o30_5 = fmaf(eb, g5_30, o30_5);
            }
            { const float eb = bi[292];
              o31_5 = fmaf(eb, g5_0, o31_5);
            }
            { const float eb = bi[293];
              o31_5 = fmaf(eb, g5_1, o31_5);
            }
            { const float eb = bi[294];
              o31_5 = fmaf(eb, g5_2, o31_5);
            }
            { const float eb = bi[295];
              o31_5 = fmaf(eb, g5_5, o31_5);
            }
            { const float eb = bi[296];
              o31_5 = fmaf(eb, g5_6, o31_5);
            }
            { const float eb = bi[297];
              o31_5 = fmaf(eb, g5_12, o31_5);
            }
            { const float eb = bi[298];
              o31_5 = fmaf(eb, g5_13, o31_5);
            }
            { const float eb = bi[299];
              o31_5 = fmaf(eb, g5_23, o31_5);
            }
            { const float eb = bi[300];
              o32_5 = fmaf(eb, g5_0, o32_5);
            }
            { const float eb = bi[301];
              o32_5 = fmaf(eb, g5_1, o32_5);
            }
            { const float eb = bi[302];
              o32_5 = fmaf(eb, g5_4, o32_5);
            }
            { const float eb = bi[303];
              o32_5 = fmaf(eb, g5_10, o32_5);
            }
            { const float eb = bi[304];
              o32_5 = fmaf(eb, g5_2, o32_5);
            }
            { const float eb = bi[305];
              o32_5 = fmaf(eb, g5_5, o32_5);
            }
            { const float eb = bi[306];
              o32_5 = fmaf(eb, g5_11, o32_5);
            }
            { const float eb = bi[307];
              o32_5 = fmaf(eb, g5_21, o32_5);
            }
            { const float eb = bi[308];
              o33_5 = fmaf(eb, g5_0, o33_5);
            }
            { const float eb = bi[309];
              o33_5 = fmaf(eb, g5_1, o33_5);
            }
            { const float eb = bi[310];
              o33_5 = fmaf(eb, g5_2, o33_5);
            }
            { const float eb = bi[311];
              o33_5 = fmaf(eb, g5_5, o33_5);
            }
            { const float eb = bi[312];
              o33_5 = fmaf(eb, g5_6, o33_5);
            }
            { const float eb = bi[313];
              o33_5 = fmaf(eb, g5_12, o33_5);
            }
            { const float eb = bi[314];
              o33_5 = fmaf(eb, g5_3, o33_5);
            }
            { const float eb = bi[315];
              o33_5 = fmaf(eb, g5_7, o33_5);
            }
            { const float eb = bi[316];
              o33_5 = fmaf(eb, g5_8, o33_5);
            }
            { const float eb = bi[317];
              o33_5 = fmaf(eb, g5_15, o33_5);
            }
            { const float eb = bi[318];
              o33_5 = fmaf(eb, g5_16, o33_5);
            }
            { const float eb = bi[319];
              o33_5 = fmaf(eb, g5_27, o33_5);
            }
            { const float eb = bi[320];
              o34_5 = fmaf(eb, g5_0, o34_5);
            }
            { const float eb = bi[321];
              o34_5 = fmaf(eb, g5_1, o34_5);
            }
            { const float eb = bi[322];
              o34_5 = fmaf(eb, g5_4, o34_5);
            }
            { const float eb = bi[323];
              o34_5 = fmaf(eb, g5_2, o34_5);
            }
            { const float eb = bi[324];
              o34_5 = fmaf(eb, g5_5, o34_5);
            }
            { const float eb = bi[325];
              o34_5 = fmaf(eb, g5_11, o34_5);
            }
            { const float eb = bi[326];
              o34_5 = fmaf(eb, g5_3, o34_5);
            }
            { const float eb = bi[327];
              o34_5 = fmaf(eb, g5_7, o34_5);
            }
            { const float eb = bi[328];
              o34_5 = fmaf(eb, g5_14, o34_5);
            }
            { const float eb = bi[329];
              o34_5 = fmaf(eb, g5_8, o34_5);
            }
            { const float eb = bi[330];
              o34_5 = fmaf(eb, g5_15, o34_5);
            }
            { const float eb = bi[331];
              o34_5 = fmaf(eb, g5_26, o34_5);
            }
            { const float eb = bi[332];
              o35_5 = fmaf(eb, g5_0, o35_5);
            }
            { const float eb = bi[333];
              o35_5 = fmaf(eb, g5_1, o35_5);
            }
            { const float eb = bi[334];
              o35_5 = fmaf(eb, g5_4, o35_5);
            }
            { const float eb = bi[335];
              o35_5 = fmaf(eb, g5_2, o35_5);
            }
            { const float eb = bi[336];
              o35_5 = fmaf(eb, g5_5, o35_5);
            }
            { const float eb = bi[337];
              o35_5 = fmaf(eb, g5_11, o35_5);
            }
            { const float eb = bi[338];
              o35_5 = fmaf(eb, g5_6, o35_5);
            }
            { const float eb = bi[339];
              o35_5 = fmaf(eb, g5_12, o35_5);
            }
            { const float eb = bi[340];
              o35_5 = fmaf(eb, g5_22, o35_5);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk5 = PT[(fI + 1) * N + fJ + 1];
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Abd4_1 = PA[(fQ + 4) * N + fJ + 1];
            const double Abd5_1 = PA[(fQ + 5) * N + fJ + 1];
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
            const double Abc4_1 = PA[(fQ + 4) * N + fI + 1];
            const double Abc5_1 = PA[(fQ + 5) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
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
            atomicAdd(Jacc + (fI + 1) * N + fJ + 1, 2.0 * deg * (o0_5 * ptb0 + o1_5 * ptb1 + o2_5 * ptb2 + o3_5 * ptb3 + o4_5 * ptb4 + o5_5 * ptb5 + o6_5 * ptb6 + o7_5 * ptb7 + o8_5 * ptb8 + o9_5 * ptb9 + o10_5 * ptb10 + o11_5 * ptb11 + o12_5 * ptb12 + o13_5 * ptb13 + o14_5 * ptb14 + o15_5 * ptb15 + o16_5 * ptb16 + o17_5 * ptb17 + o18_5 * ptb18 + o19_5 * ptb19 + o20_5 * ptb20 + o21_5 * ptb21 + o22_5 * ptb22 + o23_5 * ptb23 + o24_5 * ptb24 + o25_5 * ptb25 + o26_5 * ptb26 + o27_5 * ptb27 + o28_5 * ptb28 + o29_5 * ptb29 + o30_5 * ptb30 + o31_5 * ptb31 + o32_5 * ptb32 + o33_5 * ptb33 + o34_5 * ptb34 + o35_5 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_5 * Abd0_1 + o1_5 * Abd1_1 + o2_5 * Abd2_1 + o3_5 * Abd3_1 + o4_5 * Abd4_1 + o5_5 * Abd5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_5 * Aad0_1 + o6_5 * Aad1_1 + o12_5 * Aad2_1 + o18_5 * Aad3_1 + o24_5 * Aad4_1 + o30_5 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_5 * Abc0_1 + o1_5 * Abc1_1 + o2_5 * Abc2_1 + o3_5 * Abc3_1 + o4_5 * Abc4_1 + o5_5 * Abc5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_5 * Aac0_1 + o6_5 * Aac1_1 + o12_5 * Aac2_1 + o18_5 * Aac3_1 + o24_5 * Aac4_1 + o30_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_5 * Aad0_1 + o7_5 * Aad1_1 + o13_5 * Aad2_1 + o19_5 * Aad3_1 + o25_5 * Aad4_1 + o31_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_5 * Aac0_1 + o7_5 * Aac1_1 + o13_5 * Aac2_1 + o19_5 * Aac3_1 + o25_5 * Aac4_1 + o31_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_5 * Aad0_1 + o8_5 * Aad1_1 + o14_5 * Aad2_1 + o20_5 * Aad3_1 + o26_5 * Aad4_1 + o32_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_5 * Aac0_1 + o8_5 * Aac1_1 + o14_5 * Aac2_1 + o20_5 * Aac3_1 + o26_5 * Aac4_1 + o32_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_5 * Aad0_1 + o9_5 * Aad1_1 + o15_5 * Aad2_1 + o21_5 * Aad3_1 + o27_5 * Aad4_1 + o33_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_5 * Aac0_1 + o9_5 * Aac1_1 + o15_5 * Aac2_1 + o21_5 * Aac3_1 + o27_5 * Aac4_1 + o33_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 1, deg * (o4_5 * Aad0_1 + o10_5 * Aad1_1 + o16_5 * Aad2_1 + o22_5 * Aad3_1 + o28_5 * Aad4_1 + o34_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 1, deg * (o4_5 * Aac0_1 + o10_5 * Aac1_1 + o16_5 * Aac2_1 + o22_5 * Aac3_1 + o28_5 * Aac4_1 + o34_5 * Aac5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 1, deg * (o5_5 * Aad0_1 + o11_5 * Aad1_1 + o17_5 * Aad2_1 + o23_5 * Aad3_1 + o29_5 * Aad4_1 + o35_5 * Aad5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 1, deg * (o5_5 * Aac0_1 + o11_5 * Aac1_1 + o17_5 * Aac2_1 + o23_5 * Aac3_1 + o29_5 * Aac4_1 + o35_5 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o6_5 * Abd0_1 + o7_5 * Abd1_1 + o8_5 * Abd2_1 + o9_5 * Abd3_1 + o10_5 * Abd4_1 + o11_5 * Abd5_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o6_5 * Abc0_1 + o7_5 * Abc1_1 + o8_5 * Abc2_1 + o9_5 * Abc3_1 + o10_5 * Abc4_1 + o11_5 * Abc5_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o12_5 * Abd0_1 + o13_5 * Abd1_1 + o14_5 * Abd2_1 + o15_5 * Abd3_1 + o16_5 * Abd4_1 + o17_5 * Abd5_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o12_5 * Abc0_1 + o13_5 * Abc1_1 + o14_5 * Abc2_1 + o15_5 * Abc3_1 + o16_5 * Abc4_1 + o17_5 * Abc5_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o18_5 * Abd0_1 + o19_5 * Abd1_1 + o20_5 * Abd2_1 + o21_5 * Abd3_1 + o22_5 * Abd4_1 + o23_5 * Abd5_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o18_5 * Abc0_1 + o19_5 * Abc1_1 + o20_5 * Abc2_1 + o21_5 * Abc3_1 + o22_5 * Abc4_1 + o23_5 * Abc5_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o24_5 * Abd0_1 + o25_5 * Abd1_1 + o26_5 * Abd2_1 + o27_5 * Abd3_1 + o28_5 * Abd4_1 + o29_5 * Abd5_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o24_5 * Abc0_1 + o25_5 * Abc1_1 + o26_5 * Abc2_1 + o27_5 * Abc3_1 + o28_5 * Abc4_1 + o29_5 * Abc5_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o30_5 * Abd0_1 + o31_5 * Abd1_1 + o32_5 * Abd2_1 + o33_5 * Abd3_1 + o34_5 * Abd4_1 + o35_5 * Abd5_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o30_5 * Abc0_1 + o31_5 * Abc1_1 + o32_5 * Abc2_1 + o33_5 * Abc3_1 + o34_5 * Abc4_1 + o35_5 * Abc5_1));
          }
        } break;
        case 6: {  // ket functions [6]
          float o0_6 = 0;
          float o1_6 = 0;
          float o2_6 = 0;
          float o3_6 = 0;
          float o4_6 = 0;
          float o5_6 = 0;
          float o6_6 = 0;
          float o7_6 = 0;
          float o8_6 = 0;
          float o9_6 = 0;
          float o10_6 = 0;
          float o11_6 = 0;
          float o12_6 = 0;
          float o13_6 = 0;
          float o14_6 = 0;
          float o15_6 = 0;
          float o16_6 = 0;
          float o17_6 = 0;
          float o18_6 = 0;
          float o19_6 = 0;
          float o20_6 = 0;
          float o21_6 = 0;
          float o22_6 = 0;
          float o23_6 = 0;
          float o24_6 = 0;
          float o25_6 = 0;
          float o26_6 = 0;
          float o27_6 = 0;
          float o28_6 = 0;
          float o29_6 = 0;
          float o30_6 = 0;
          float o31_6 = 0;
          float o32_6 = 0;
          float o33_6 = 0;
          float o34_6 = 0;
          float o35_6 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g6_0 = 0;
            float g6_1 = 0;
            float g6_2 = 0;
            float g6_3 = 0;
            float g6_4 = 0;
            float g6_5 = 0;
            float g6_6 = 0;
            float g6_7 = 0;
            float g6_8 = 0;
            float g6_9 = 0;
            float g6_10 = 0;
            float g6_11 = 0;
            float g6_12 = 0;
            float g6_13 = 0;
            float g6_14 = 0;
            float g6_15 = 0;
            float g6_16 = 0;
            float g6_17 = 0;
            float g6_18 = 0;
            float g6_19 = 0;
            float g6_20 = 0;
            float g6_21 = 0;
            float g6_22 = 0;
            float g6_23 = 0;
            float g6_24 = 0;
            float g6_25 = 0;
            float g6_26 = 0;
            float g6_27 = 0;
            float g6_28 = 0;
            float g6_29 = 0;
            float g6_30 = 0;
            float g6_31 = 0;
            float g6_32 = 0;
            float g6_33 = 0;
            float g6_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek6_0 = kj[24 * kS];
              const float ek6_1 = -kj[25 * kS];
              const float ek6_2 = kj[26 * kS];
              g6_0 = fmaf(ek6_0, b0, g6_0);
              const float r0_0_0_1 = Z * b1;
              g6_1 = fmaf(ek6_0, r0_0_0_1, g6_1);
              const float r0_0_1_0 = Y * b1;
              g6_2 = fmaf(ek6_0, r0_0_1_0, g6_2);
              g6_0 = fmaf(ek6_1, r0_0_1_0, g6_0);
              const float r0_1_0_0 = X * b1;
              g6_3 = fmaf(ek6_0, r0_1_0_0, g6_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g6_4 = fmaf(ek6_0, r0_0_0_2, g6_4);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g6_5 = fmaf(ek6_0, r0_0_1_1, g6_5);
              g6_1 = fmaf(ek6_1, r0_0_1_1, g6_1);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g6_6 = fmaf(ek6_0, r0_0_2_0, g6_6);
              g6_2 = fmaf(ek6_1, r0_0_2_0, g6_2);
              g6_0 = fmaf(ek6_2, r0_0_2_0, g6_0);
              const float r0_1_0_1 = X * r1_0_0_1;
              g6_7 = fmaf(ek6_0, r0_1_0_1, g6_7);
              const float r0_1_1_0 = X * r1_0_1_0;
              g6_8 = fmaf(ek6_0, r0_1_1_0, g6_8);
              g6_3 = fmaf(ek6_1, r0_1_1_0, g6_3);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g6_9 = fmaf(ek6_0, r0_2_0_0, g6_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g6_10 = fmaf(ek6_0, r0_0_0_3, g6_10);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g6_11 = fmaf(ek6_0, r0_0_1_2, g6_11);
              g6_4 = fmaf(ek6_1, r0_0_1_2, g6_4);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g6_12 = fmaf(ek6_0, r0_0_2_1, g6_12);
              g6_5 = fmaf(ek6_1, r0_0_2_1, g6_5);
              g6_1 = fmaf(ek6_2, r0_0_2_1, g6_1);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g6_13 = fmaf(ek6_0, r0_0_3_0, g6_13);
              g6_6 = fmaf(ek6_1, r0_0_3_0, g6_6);
              g6_2 = fmaf(ek6_2, r0_0_3_0, g6_2);
              const float r0_1_0_2 = X * r1_0_0_2;
              g6_14 = fmaf(ek6_0, r0_1_0_2, g6_14);
              const float r0_1_1_1 = X * r1_0_1_1;
              g6_15 = fmaf(ek6_0, r0_1_1_1, g6_15);
              g6_7 = fmaf(ek6_1, r0_1_1_1, g6_7);
              const float r0_1_2_0 = X * r1_0_2_0;
              g6_16 = fmaf(ek6_0, r0_1_2_0, g6_16);
              g6_8 = fmaf(ek6_1, r0_1_2_0, g6_8);
              g6_3 = fmaf(ek6_2, r0_1_2_0, g6_3);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g6_17 = fmaf(ek6_0, r0_2_0_1, g6_17);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g6_18 = fmaf(ek6_0, r0_2_1_0, g6_18);
              g6_9 = fmaf(ek6_1, r0_2_1_0, g6_9);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g6_19 = fmaf(ek6_0, r0_3_0_0, g6_19);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g6_20 = fmaf(ek6_0, r0_0_0_4, g6_20);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g6_21 = fmaf(ek6_0, r0_0_1_3, g6_21);
              g6_10 = fmaf(ek6_1, r0_0_1_3, g6_10);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g6_22 = fmaf(ek6_0, r0_0_2_2, g6_22);
              g6_11 = fmaf(ek6_1, r0_0_2_2, g6_11);
              g6_4 = fmaf(ek6_2, r0_0_2_2, g6_4);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g6_23 = fmaf(ek6_0, r0_0_3_1, g6_23);
              g6_12 = fmaf(ek6_1, r0_0_3_1, g6_12);
              g6_5 = fmaf(ek6_2, r0_0_3_1, g6_5);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g6_24 = fmaf(ek6_0, r0_0_4_0, g6_24);
              g6_13 = fmaf(ek6_1, r0_0_4_0, g6_13);
              g6_6 = fmaf(ek6_2, r0_0_4_0, g6_6);
              const float r0_1_0_3 = X * r1_0_0_3;
              g6_25 = fmaf(ek6_0, r0_1_0_3, g6_25);
              const float r0_1_1_2 = X * r1_0_1_2;
              g6_26 = fmaf(ek6_0, r0_1_1_2, g6_26);
              g6_14 = fmaf(ek6_1, r0_1_1_2, g6_14);
              const float r0_1_2_1 = X * r1_0_2_1;
              g6_27 = fmaf(ek6_0, r0_1_2_1, g6_27);
              g6_15 = fmaf(ek6_1, r0_1_2_1, g6_15);
              g6_7 = fmaf(ek6_2, r0_1_2_1, g6_7);
              const float r0_1_3_0 = X * r1_0_3_0;
              g6_28 = fmaf(ek6_0, r0_1_3_0, g6_28);
              g6_16 = fmaf(ek6_1, r0_1_3_0, g6_16);
              g6_8 = fmaf(ek6_2, r0_1_3_0, g6_8);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g6_29 = fmaf(ek6_0, r0_2_0_2, g6_29);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g6_30 = fmaf(ek6_0, r0_2_1_1, g6_30);
              g6_17 = fmaf(ek6_1, r0_2_1_1, g6_17);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g6_31 = fmaf(ek6_0, r0_2_2_0, g6_31);
              g6_18 = fmaf(ek6_1, r0_2_2_0, g6_18);
              g6_9 = fmaf(ek6_2, r0_2_2_0, g6_9);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g6_32 = fmaf(ek6_0, r0_3_0_1, g6_32);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g6_33 = fmaf(ek6_0, r0_3_1_0, g6_33);
              g6_19 = fmaf(ek6_1, r0_3_1_0, g6_19);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g6_34 = fmaf(ek6_0, r0_4_0_0, g6_34);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g6_20 = fmaf(ek6_1, r0_0_1_4, g6_20);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g6_21 = fmaf(ek6_1, r0_0_2_3, g6_21);
              g6_10 = fmaf(ek6_2, r0_0_2_3, g6_10);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g6_22 = fmaf(ek6_1, r0_0_3_2, g6_22);
              g6_11 = fmaf(ek6_2, r0_0_3_2, g6_11);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g6_23 = fmaf(ek6_1, r0_0_4_1, g6_23);
              g6_12 = fmaf(ek6_2, r0_0_4_1, g6_12);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_0_5_0 = fmaf(Y, r1_0_4_0, 4.0f * r1_0_3_0);
              g6_24 = fmaf(ek6_1, r0_0_5_0, g6_24);
              g6_13 = fmaf(ek6_2, r0_0_5_0, g6_13);
              const float r0_1_1_3 = X * r1_0_1_3;
              g6_25 = fmaf(ek6_1, r0_1_1_3, g6_25);
              const float r0_1_2_2 = X * r1_0_2_2;
              g6_26 = fmaf(ek6_1, r0_1_2_2, g6_26);
              g6_14 = fmaf(ek6_2, r0_1_2_2, g6_14);
              const float r0_1_3_1 = X * r1_0_3_1;
              g6_27 = fmaf(ek6_1, r0_1_3_1, g6_27);
              g6_15 = fmaf(ek6_2, r0_1_3_1, g6_15);
              const float r0_1_4_0 = X * r1_0_4_0;
              g6_28 = fmaf(ek6_1, r0_1_4_0, g6_28);
              g6_16 = fmaf(ek6_2, r0_1_4_0, g6_16);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g6_29 = fmaf(ek6_1, r0_2_1_2, g6_29);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g6_30 = fmaf(ek6_1, r0_2_2_1, g6_30);
              g6_17 = fmaf(ek6_2, r0_2_2_1, g6_17);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g6_31 = fmaf(ek6_1, r0_2_3_0, g6_31);
              g6_18 = fmaf(ek6_2, r0_2_3_0, g6_18);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g6_32 = fmaf(ek6_1, r0_3_1_1, g6_32);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g6_33 = fmaf(ek6_1, r0_3_2_0, g6_33);
              g6_19 = fmaf(ek6_2, r0_3_2_0, g6_19);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g6_34 = fmaf(ek6_1, r0_4_1_0, g6_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_0_2_4 = fmaf(Y, r1_0_1_4, r1_0_0_4);
              g6_20 = fmaf(ek6_2, r0_0_2_4, g6_20);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_0_3_3 = fmaf(Y, r1_0_2_3, 2.0f * r1_0_1_3);
              g6_21 = fmaf(ek6_2, r0_0_3_3, g6_21);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_0_4_2 = fmaf(Y, r1_0_3_2, 3.0f * r1_0_2_2);
              g6_22 = fmaf(ek6_2, r0_0_4_2, g6_22);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_0_5_1 = fmaf(Y, r1_0_4_1, 4.0f * r1_0_3_1);
              g6_23 = fmaf(ek6_2, r0_0_5_1, g6_23);
              const float r5_0_1_0 = Y * b6;
              const float r4_0_2_0 = fmaf(Y, r5_0_1_0, b5);
              const float r3_0_3_0 = fmaf(Y, r4_0_2_0, 2.0f * r4_0_1_0);
              const float r2_0_4_0 = fmaf(Y, r3_0_3_0, 3.0f * r3_0_2_0);
              const float r1_0_5_0 = fmaf(Y, r2_0_4_0, 4.0f * r2_0_3_0);
              const float r0_0_6_0 = fmaf(Y, r1_0_5_0, 5.0f * r1_0_4_0);
              g6_24 = fmaf(ek6_2, r0_0_6_0, g6_24);
              const float r0_1_2_3 = X * r1_0_2_3;
              g6_25 = fmaf(ek6_2, r0_1_2_3, g6_25);
              const float r0_1_3_2 = X * r1_0_3_2;
              g6_26 = fmaf(ek6_2, r0_1_3_2, g6_26);
              const float r0_1_4_1 = X * r1_0_4_1;
              g6_27 = fmaf(ek6_2, r0_1_4_1, g6_27);
              const float r0_1_5_0 = X * r1_0_5_0;
              g6_28 = fmaf(ek6_2, r0_1_5_0, g6_28);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g6_29 = fmaf(ek6_2, r0_2_2_2, g6_29);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g6_30 = fmaf(ek6_2, r0_2_3_1, g6_30);
              const float r1_1_4_0 = X * r2_0_4_0;
              const float r0_2_4_0 = fmaf(X, r1_1_4_0, r1_0_4_0);
              g6_31 = fmaf(ek6_2, r0_2_4_0, g6_31);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g6_32 = fmaf(ek6_2, r0_3_2_1, g6_32);
              const float r2_1_3_0 = X * r3_0_3_0;
              const float r1_2_3_0 = fmaf(X, r2_1_3_0, r2_0_3_0);
              const float r0_3_3_0 = fmaf(X, r1_2_3_0, 2.0f * r1_1_3_0);
              g6_33 = fmaf(ek6_2, r0_3_3_0, g6_33);
              const float r3_1_2_0 = X * r4_0_2_0;
              const float r2_2_2_0 = fmaf(X, r3_1_2_0, r3_0_2_0);
              const float r1_3_2_0 = fmaf(X, r2_2_2_0, 2.0f * r2_1_2_0);
              const float r0_4_2_0 = fmaf(X, r1_3_2_0, 3.0f * r1_2_2_0);
              g6_34 = fmaf(ek6_2, r0_4_2_0, g6_34);
            }
            { const float eb = bi[5];
              o0_6 = fmaf(eb, g6_0, o0_6);
            }
            { const float eb = bi[6];
              o0_6 = fmaf(eb, g6_3, o0_6);
            }
            { const float eb = bi[7];
              o0_6 = fmaf(eb, g6_9, o0_6);
            }
            { const float eb = bi[8];
              o0_6 = fmaf(eb, g6_19, o0_6);
            }
            { const float eb = bi[9];
              o0_6 = fmaf(eb, g6_34, o0_6);
            }
            { const float eb = bi[10];
              o1_6 = fmaf(eb, g6_0, o1_6);
            }
            { const float eb = bi[11];
              o1_6 = fmaf(eb, g6_2, o1_6);
            }
            { const float eb = bi[12];
              o1_6 = fmaf(eb, g6_6, o1_6);
            }
            { const float eb = bi[13];
              o1_6 = fmaf(eb, g6_3, o1_6);
            }
            { const float eb = bi[14];
              o1_6 = fmaf(eb, g6_8, o1_6);
            }
            { const float eb = bi[15];
              o1_6 = fmaf(eb, g6_16, o1_6);
            }
            { const float eb = bi[16];
              o1_6 = fmaf(eb, g6_9, o1_6);
            }
            { const float eb = bi[17];
              o1_6 = fmaf(eb, g6_18, o1_6);
            }
            { const float eb = bi[18];
              o1_6 = fmaf(eb, g6_31, o1_6);
            }
            { const float eb = bi[19];
              o2_6 = fmaf(eb, g6_0, o2_6);
            }
            { const float eb = bi[20];
              o2_6 = fmaf(eb, g6_1, o2_6);
            }
            { const float eb = bi[21];
              o2_6 = fmaf(eb, g6_4, o2_6);
            }
            { const float eb = bi[22];
              o2_6 = fmaf(eb, g6_3, o2_6);
            }
            { const float eb = bi[23];
              o2_6 = fmaf(eb, g6_7, o2_6);
            }
            { const float eb = bi[24];
              o2_6 = fmaf(eb, g6_14, o2_6);
            }
            { const float eb = bi[25];
              o2_6 = fmaf(eb, g6_9, o2_6);
            }
            { const float eb = bi[26];
              o2_6 = fmaf(eb, g6_17, o2_6);
            }
            { const float eb = bi[27];
              o2_6 = fmaf(eb, g6_29, o2_6);
            }
            { const float eb = bi[28];
              o3_6 = fmaf(eb, g6_0, o3_6);
            }
            { const float eb = bi[29];
              o3_6 = fmaf(eb, g6_2, o3_6);
            }
            { const float eb = bi[30];
              o3_6 = fmaf(eb, g6_3, o3_6);
            }
            { const float eb = bi[31];
              o3_6 = fmaf(eb, g6_8, o3_6);
            }
            { const float eb = bi[32];
              o3_6 = fmaf(eb, g6_9, o3_6);
            }
            { const float eb = bi[33];
              o3_6 = fmaf(eb, g6_18, o3_6);
            }
            { const float eb = bi[34];
              o3_6 = fmaf(eb, g6_19, o3_6);
            }
            { const float eb = bi[35];
              o3_6 = fmaf(eb, g6_33, o3_6);
            }
            { const float eb = bi[36];
              o4_6 = fmaf(eb, g6_0, o4_6);
            }
            { const float eb = bi[37];
              o4_6 = fmaf(eb, g6_1, o4_6);
            }
            { const float eb = bi[38];
              o4_6 = fmaf(eb, g6_3, o4_6);
            }
            { const float eb = bi[39];
              o4_6 = fmaf(eb, g6_7, o4_6);
            }
            { const float eb = bi[40];
              o4_6 = fmaf(eb, g6_9, o4_6);
            }
            { const float eb = bi[41];
              o4_6 = fmaf(eb, g6_17, o4_6);
            }
            { const float eb = bi[42];
              o4_6 = fmaf(eb, g6_19, o4_6);
            }
            { const float eb = bi[43];
              o4_6 = fmaf(eb, g6_32, o4_6);
            }
            { const float eb = bi[44];
              o5_6 = fmaf(eb, g6_0, o5_6);
            }
            { const float eb = bi[45];
              o5_6 = fmaf(eb, g6_1, o5_6);
            }
            { const float eb = bi[46];
              o5_6 = fmaf(eb, g6_2, o5_6);
            }
            { const float eb = bi[47];
              o5_6 = fmaf(eb, g6_5, o5_6);
            }
            { const float eb = bi[48];
              o5_6 = fmaf(eb, g6_3, o5_6);
            }
            { const float eb = bi[49];
              o5_6 = fmaf(eb, g6_7, o5_6);
            }
            { const float eb = bi[50];
              o5_6 = fmaf(eb, g6_8, o5_6);
            }
            { const float eb = bi[51];
              o5_6 = fmaf(eb, g6_15, o5_6);
            }
            { const float eb = bi[52];
              o5_6 = fmaf(eb, g6_9, o5_6);
            }
            { const float eb = bi[53];
              o5_6 = fmaf(eb, g6_17, o5_6);
            }
            { const float eb = bi[54];
              o5_6 = fmaf(eb, g6_18, o5_6);
            }
            { const float eb = bi[55];
              o5_6 = fmaf(eb, g6_30, o5_6);
            }
            { const float eb = bi[56];
              o6_6 = fmaf(eb, g6_0, o6_6);
            }
            { const float eb = bi[57];
              o6_6 = fmaf(eb, g6_2, o6_6);
            }
            { const float eb = bi[58];
              o6_6 = fmaf(eb, g6_6, o6_6);
            }
            { const float eb = bi[59];
              o6_6 = fmaf(eb, g6_3, o6_6);
            }
            { const float eb = bi[60];
              o6_6 = fmaf(eb, g6_8, o6_6);
            }
            { const float eb = bi[61];
              o6_6 = fmaf(eb, g6_16, o6_6);
            }
            { const float eb = bi[62];
              o6_6 = fmaf(eb, g6_9, o6_6);
            }
            { const float eb = bi[63];
              o6_6 = fmaf(eb, g6_18, o6_6);
            }
            { const float eb = bi[64];
              o6_6 = fmaf(eb, g6_31, o6_6);
            }
            { const float eb = bi[65];
              o7_6 = fmaf(eb, g6_0, o7_6);
            }
            { const float eb = bi[66];
              o7_6 = fmaf(eb, g6_2, o7_6);
            }
            { const float eb = bi[67];
              o7_6 = fmaf(eb, g6_6, o7_6);
            }
            { const float eb = bi[68];
              o7_6 = fmaf(eb, g6_13, o7_6);
            }
            { const float eb = bi[69];
              o7_6 = fmaf(eb, g6_24, o7_6);
            }
            { const float eb = bi[70];
              o8_6 = fmaf(eb, g6_0, o8_6);
            }
            { const float eb = bi[71];
              o8_6 = fmaf(eb, g6_1, o8_6);
            }
            { const float eb = bi[72];
              o8_6 = fmaf(eb, g6_4, o8_6);
            }
            { const float eb = bi[73];
              o8_6 = fmaf(eb, g6_2, o8_6);
            }
            { const float eb = bi[74];
              o8_6 = fmaf(eb, g6_5, o8_6);
            }
            { const float eb = bi[75];
              o8_6 = fmaf(eb, g6_11, o8_6);
            }
            { const float eb = bi[76];
              o8_6 = fmaf(eb, g6_6, o8_6);
            }
            { const float eb = bi[77];
              o8_6 = fmaf(eb, g6_12, o8_6);
            }
            { const float eb = bi[78];
              o8_6 = fmaf(eb, g6_22, o8_6);
            }
            { const float eb = bi[79];
              o9_6 = fmaf(eb, g6_0, o9_6);
            }
            { const float eb = bi[80];
              o9_6 = fmaf(eb, g6_2, o9_6);
            }
            { const float eb = bi[81];
              o9_6 = fmaf(eb, g6_6, o9_6);
            }
            { const float eb = bi[82];
              o9_6 = fmaf(eb, g6_13, o9_6);
            }
            { const float eb = bi[83];
              o9_6 = fmaf(eb, g6_3, o9_6);
            }
            { const float eb = bi[84];
              o9_6 = fmaf(eb, g6_8, o9_6);
            }
            { const float eb = bi[85];
              o9_6 = fmaf(eb, g6_16, o9_6);
            }
            { const float eb = bi[86];
              o9_6 = fmaf(eb, g6_28, o9_6);
            }
            { const float eb = bi[87];
              o10_6 = fmaf(eb, g6_0, o10_6);
            }
            { const float eb = bi[88];
              o10_6 = fmaf(eb, g6_1, o10_6);
            }
            { const float eb = bi[89];
              o10_6 = fmaf(eb, g6_2, o10_6);
            }
            { const float eb = bi[90];
              o10_6 = fmaf(eb, g6_5, o10_6);
            }
            { const float eb = bi[91];
              o10_6 = fmaf(eb, g6_6, o10_6);
            }
            { const float eb = bi[92];
              o10_6 = fmaf(eb, g6_12, o10_6);
            }
            { const float eb = bi[93];
              o10_6 = fmaf(eb, g6_3, o10_6);
            }
            { const float eb = bi[94];
              o10_6 = fmaf(eb, g6_7, o10_6);
            }
            { const float eb = bi[95];
              o10_6 = fmaf(eb, g6_8, o10_6);
            }
            { const float eb = bi[96];
              o10_6 = fmaf(eb, g6_15, o10_6);
            }
            { const float eb = bi[97];
              o10_6 = fmaf(eb, g6_16, o10_6);
            }
            { const float eb = bi[98];
              o10_6 = fmaf(eb, g6_27, o10_6);
            }
            { const float eb = bi[99];
              o11_6 = fmaf(eb, g6_0, o11_6);
            }
            { const float eb = bi[100];
              o11_6 = fmaf(eb, g6_1, o11_6);
            }
            { const float eb = bi[101];
              o11_6 = fmaf(eb, g6_2, o11_6);
            }
            { const float eb = bi[102];
              o11_6 = fmaf(eb, g6_5, o11_6);
            }
            { const float eb = bi[103];
              o11_6 = fmaf(eb, g6_6, o11_6);
            }
            { const float eb = bi[104];
              o11_6 = fmaf(eb, g6_12, o11_6);
            }
            { const float eb = bi[105];
              o11_6 = fmaf(eb, g6_13, o11_6);
            }
            { const float eb = bi[106];
              o11_6 = fmaf(eb, g6_23, o11_6);
            }
            { const float eb = bi[107];
              o12_6 = fmaf(eb, g6_0, o12_6);
            }
            { const float eb = bi[108];
              o12_6 = fmaf(eb, g6_1, o12_6);
            }
            { const float eb = bi[109];
              o12_6 = fmaf(eb, g6_4, o12_6);
            }
            { const float eb = bi[110];
              o12_6 = fmaf(eb, g6_3, o12_6);
            }
            { const float eb = bi[111];
              o12_6 = fmaf(eb, g6_7, o12_6);
            }
            { const float eb = bi[112];
              o12_6 = fmaf(eb, g6_14, o12_6);
            }
            { const float eb = bi[113];
              o12_6 = fmaf(eb, g6_9, o12_6);
            }
            { const float eb = bi[114];
              o12_6 = fmaf(eb, g6_17, o12_6);
            }
            { const float eb = bi[115];
              o12_6 = fmaf(eb, g6_29, o12_6);
            }
            { const float eb = bi[116];
              o13_6 = fmaf(eb, g6_0, o13_6);
            }
            { const float eb = bi[117];
              o13_6 = fmaf(eb, g6_1, o13_6);
            }
            { const float eb = bi[118];
              o13_6 = fmaf(eb, g6_4, o13_6);
            }
            { const float eb = bi[119];
              o13_6 = fmaf(eb, g6_2, o13_6);
            }
            { const float eb = bi[120];
              o13_6 = fmaf(eb, g6_5, o13_6);
            }
            { const float eb = bi[121];
              o13_6 = fmaf(eb, g6_11, o13_6);
            }
            { const float eb = bi[122];
              o13_6 = fmaf(eb, g6_6, o13_6);
            }
            { const float eb = bi[123];
              o13_6 = fmaf(eb, g6_12, o13_6);
            }
            { const float eb = bi[124];
              o13_6 = fmaf(eb, g6_22, o13_6);
            }
            { const float eb = bi[125];
              o14_6 = fmaf(eb, g6_0, o14_6);
            }
            { const float eb = bi[126];
              o14_6 = fmaf(eb, g6_1, o14_6);
            }
            { const float eb = bi[127];
              o14_6 = fmaf(eb, g6_4, o14_6);
            }
            { const float eb = bi[128];
              o14_6 = fmaf(eb, g6_10, o14_6);
            }
            { const float eb = bi[129];
              o14_6 = fmaf(eb, g6_20, o14_6);
            }
            { const float eb = bi[130];
              o15_6 = fmaf(eb, g6_0, o15_6);
            }
            { const float eb = bi[131];
              o15_6 = fmaf(eb, g6_1, o15_6);
            }
            { const float eb = bi[132];
              o15_6 = fmaf(eb, g6_4, o15_6);
            }
            { const float eb = bi[133];
              o15_6 = fmaf(eb, g6_2, o15_6);
            }
            { const float eb = bi[134];
              o15_6 = fmaf(eb, g6_5, o15_6);
            }
            { const float eb = bi[135];
              o15_6 = fmaf(eb, g6_11, o15_6);
            }
            { const float eb = bi[136];
              o15_6 = fmaf(eb, g6_3, o15_6);
            }
            { const float eb = bi[137];
              o15_6 = fmaf(eb, g6_7, o15_6);
            }
            { const float eb = bi[138];
              o15_6 = fmaf(eb, g6_14, o15_6);
            }
            { const float eb = bi[139];
              o15_6 = fmaf(eb, g6_8, o15_6);
            }
            { const float eb = bi[140];
              o15_6 = fmaf(eb, g6_15, o15_6);
            }
            { const float eb = bi[141];
              o15_6 = fmaf(eb, g6_26, o15_6);
            }
            { const float eb = bi[142];
              o16_6 = fmaf(eb, g6_0, o16_6);
            }
            { const float eb = bi[143];
              o16_6 = fmaf(eb, g6_1, o16_6);
            }
            { const float eb = bi[144];
              o16_6 = fmaf(eb, g6_4, o16_6);
            }
            { const float eb = bi[145];
              o16_6 = fmaf(eb, g6_10, o16_6);
            }
            { const float eb = bi[146];
              o16_6 = fmaf(eb, g6_3, o16_6);
            }
            { const float eb = bi[147];
              o16_6 = fmaf(eb, g6_7, o16_6);
            }
            { const float eb = bi[148];
              o16_6 = fmaf(eb, g6_14, o16_6);
            }
            { const float eb = bi[149];
              o16_6 = fmaf(eb, g6_25, o16_6);
            }
            { const float eb = bi[150];
              o17_6 = fmaf(eb, g6_0, o17_6);
            }
            { const float eb = bi[151];
              o17_6 = fmaf(eb, g6_1, o17_6);
            }
            { const float eb = bi[152];
              o17_6 = fmaf(eb, g6_4, o17_6);
            }
            { const float eb = bi[153];
              o17_6 = fmaf(eb, g6_10, o17_6);
            }
            { const float eb = bi[154];
              o17_6 = fmaf(eb, g6_2, o17_6);
            }
            { const float eb = bi[155];
              o17_6 = fmaf(eb, g6_5, o17_6);
            }
            { const float eb = bi[156];
              o17_6 = fmaf(eb, g6_11, o17_6);
            }
            { const float eb = bi[157];
              o17_6 = fmaf(eb, g6_21, o17_6);
            }
            { const float eb = bi[158];
              o18_6 = fmaf(eb, g6_0, o18_6);
            }
            { const float eb = bi[159];
              o18_6 = fmaf(eb, g6_2, o18_6);
            }
            { const float eb = bi[160];
              o18_6 = fmaf(eb, g6_3, o18_6);
            }
            { const float eb = bi[161];
              o18_6 = fmaf(eb, g6_8, o18_6);
            }
            { const float eb = bi[162];
              o18_6 = fmaf(eb, g6_9, o18_6);
            }
            { const float eb = bi[163];
              o18_6 = fmaf(eb, g6_18, o18_6);
            }
            { const float eb = bi[164];
              o18_6 = fmaf(eb, g6_19, o18_6);
            }
            { const float eb = bi[165];
              o18_6 = fmaf(eb, g6_33, o18_6);
            }
            { const float eb = bi[166];
              o19_6 = fmaf(eb, g6_0, o19_6);
            }
            { const float eb = bi[167];
              o19_6 = fmaf(eb, g6_2, o19_6);
            }
            { const float eb = bi[168];
              o19_6 = fmaf(eb, g6_6, o19_6);
            }
            { const float eb = bi[169];
              o19_6 = fmaf(eb, g6_13, o19_6);
            }
            { const float eb = bi[170];
              o19_6 = fmaf(eb, g6_3, o19_6);
            }
            { const float eb = bi[171];
              o19_6 = fmaf(eb, g6_8, o19_6);
            }
            { const float eb = bi[172];
              o19_6 = fmaf(eb, g6_16, o19_6);
            }
            { const float eb = bi[173];
              o19_6 = fmaf(eb, g6_28, o19_6);
            }
            { const float eb = bi[174];
              o20_6 = fmaf(eb, g6_0, o20_6);
            }
            { const float eb = bi[175];
              o20_6 = fmaf(eb, g6_1, o20_6);
            }
            { const float eb = bi[176];
              o20_6 = fmaf(eb, g6_4, o20_6);
            }
            { const float eb = bi[177];
              o20_6 = fmaf(eb, g6_2, o20_6);
            }
            { const float eb = bi[178];
              o20_6 = fmaf(eb, g6_5, o20_6);
            }
            { const float eb = bi[179];
              o20_6 = fmaf(eb, g6_11, o20_6);
            }
            { const float eb = bi[180];
              o20_6 = fmaf(eb, g6_3, o20_6);
            }
            { const float eb = bi[181];
              o20_6 = fmaf(eb, g6_7, o20_6);
            }
            { const float eb = bi[182];
              o20_6 = fmaf(eb, g6_14, o20_6);
            }
            { const float eb = bi[183];
              o20_6 = fmaf(eb, g6_8, o20_6);
            }
            { const float eb = bi[184];
              o20_6 = fmaf(eb, g6_15, o20_6);
            }
            { const float eb = bi[185];
              o20_6 = fmaf(eb, g6_26, o20_6);
            }
            { const float eb = bi[186];
              o21_6 = fmaf(eb, g6_0, o21_6);
            }
            { const float eb = bi[187];
              o21_6 = fmaf(eb, g6_2, o21_6);
            }
            { const float eb = bi[188];
              o21_6 = fmaf(eb, g6_6, o21_6);
            }
            { const float eb = bi[189];
              o21_6 = fmaf(eb, g6_3, o21_6);
            }
            { const float eb = bi[190];
              o21_6 = fmaf(eb, g6_8, o21_6);
            }
            { const float eb = bi[191];
              o21_6 = fmaf(eb, g6_16, o21_6);
            }
            { const float eb = bi[192];
              o21_6 = fmaf(eb, g6_9, o21_6);
            }
            { const float eb = bi[193];
              o21_6 = fmaf(eb, g6_18, o21_6);
            }
            { const float eb = bi[194];
              o21_6 = fmaf(eb, g6_31, o21_6);
            }
            { const float eb = bi[195];
              o22_6 = fmaf(eb, g6_0, o22_6);
            }
            { const float eb = bi[196];
              o22_6 = fmaf(eb, g6_1, o22_6);
            }
            { const float eb = bi[197];
              o22_6 = fmaf(eb, g6_2, o22_6);
            }
            { const float eb = bi[198];
              o22_6 = fmaf(eb, g6_5, o22_6);
            }
            { const float eb = bi[199];
              o22_6 = fmaf(eb, g6_3, o22_6);
            }
            { const float eb = bi[200];
              o22_6 = fmaf(eb, g6_7, o22_6);
            }
            { const float eb = bi[201];
              o22_6 = fmaf(eb, g6_8, o22_6);
            }
            { const float eb = bi[202];
              o22_6 = fmaf(eb, g6_15, o22_6);
            }
            { const float eb = bi[203];
              o22_6 = fmaf(eb, g6_9, o22_6);
            }
            { const float eb = bi[204];
              o22_6 = fmaf(eb, g6_17, o22_6);
            }
            { const float eb = bi[205];
              o22_6 = fmaf(eb, g6_18, o22_6);
            }
            { const float eb = bi[206];
              o22_6 = fmaf(eb, g6_30, o22_6);
            }
            { const float eb = bi[207];
              o23_6 = fmaf(eb, g6_0, o23_6);
            }
            { const float eb = bi[208];
              o23_6 = fmaf(eb, g6_1, o23_6);
            }
            { const float eb = bi[209];
              o23_6 = fmaf(eb, g6_2, o23_6);
            }
            { const float eb = bi[210];
              o23_6 = fmaf(eb, g6_5, o23_6);
            }
            { const float eb = bi[211];
              o23_6 = fmaf(eb, g6_6, o23_6);
            }
            { const float eb = bi[212];
              o23_6 = fmaf(eb, g6_12, o23_6);
            }
            { const float eb = bi[213];
              o23_6 = fmaf(eb, g6_3, o23_6);
            }
            { const float eb = bi[214];
              o23_6 = fmaf(eb, g6_7, o23_6);
            }
            { const float eb = bi[215];
              o23_6 = fmaf(eb, g6_8, o23_6);
            }
            { const float eb = bi[216];
              o23_6 = fmaf(eb, g6_15, o23_6);
            }
            { const float eb = bi[217];
              o23_6 = fmaf(eb, g6_16, o23_6);
            }
            { const float eb = bi[218];
              o23_6 = fmaf(eb, g6_27, o23_6);
            }
            { const float eb = bi[219];
              o24_6 = fmaf(eb, g6_0, o24_6);
            }
            { const float eb = bi[220];
              o24_6 = fmaf(eb, g6_1, o24_6);
            }
            { const float eb = bi[221];
              o24_6 = fmaf(eb, g6_3, o24_6);
            }
            { const float eb = bi[222];
              o24_6 = fmaf(eb, g6_7, o24_6);
            }
            { const float eb = bi[223];
              o24_6 = fmaf(eb, g6_9, o24_6);
            }
            { const float eb = bi[224];
              o24_6 = fmaf(eb, g6_17, o24_6);
            }
            { const float eb = bi[225];
              o24_6 = fmaf(eb, g6_19, o24_6);
            }
            { const float eb = bi[226];
              o24_6 = fmaf(eb, g6_32, o24_6);
            }
            { const float eb = bi[227];
              o25_6 = fmaf(eb, g6_0, o25_6);
            }
            { const float eb = bi[228];
              o25_6 = fmaf(eb, g6_1, o25_6);
            }
            { const float eb = bi[229];
              o25_6 = fmaf(eb, g6_2, o25_6);
            }
            { const float eb = bi[230];
              o25_6 = fmaf(eb, g6_5, o25_6);
            }
            { const float eb = bi[231];
              o25_6 = fmaf(eb, g6_6, o25_6);
            }
            { const float eb = bi[232];
              o25_6 = fmaf(eb, g6_12, o25_6);
            }
            { const float eb = bi[233];
              o25_6 = fmaf(eb, g6_3, o25_6);
            }
            { const float eb = bi[234];
              o25_6 = fmaf(eb, g6_7, o25_6);
            }
            { const float eb = bi[235];
              o25_6 = fmaf(eb, g6_8, o25_6);
            }
            { const float eb = bi[236];
              o25_6 = fmaf(eb, g6_15, o25_6);
            }
            { const float eb = bi[237];
              o25_6 = fmaf(eb, g6_16, o25_6);
            }
            { const float eb = bi[238];
              o25_6 = fmaf(eb, g6_27, o25_6);
            }
            { const float eb = bi[239];
              o26_6 = fmaf(eb, g6_0, o26_6);
            }
            { const float eb = bi[240];
              o26_6 = fmaf(eb, g6_1, o26_6);
            }
            { const float eb = bi[241];
              o26_6 = fmaf(eb, g6_4, o26_6);
            }
            { const float eb = bi[242];
              o26_6 = fmaf(eb, g6_10, o26_6);
            }
            { const float eb = bi[243];
              o26_6 = fmaf(eb, g6_3, o26_6);
            }
            { const float eb = bi[244];
              o26_6 = fmaf(eb, g6_7, o26_6);
            }
            { const float eb = bi[245];
              o26_6 = fmaf(eb, g6_14, o26_6);
            }
            { const float eb = bi[246];
              o26_6 = fmaf(eb, g6_25, o26_6);
            }
            { const float eb = bi[247];
              o27_6 = fmaf(eb, g6_0, o27_6);
            }
            { const float eb = bi[248];
              o27_6 = fmaf(eb, g6_1, o27_6);
            }
            { const float eb = bi[249];
              o27_6 = fmaf(eb, g6_2, o27_6);
            }
            { const float eb = bi[250];
              o27_6 = fmaf(eb, g6_5, o27_6);
            }
            { const float eb = bi[251];
              o27_6 = fmaf(eb, g6_3, o27_6);
            }
            { const float eb = bi[252];
              o27_6 = fmaf(eb, g6_7, o27_6);
            }
            { const float eb = bi[253];
              o27_6 = fmaf(eb, g6_8, o27_6);
            }
            { const float eb = bi[254];
              o27_6 = fmaf(eb, g6_15, o27_6);
            }
            { const float eb = bi[255];
              o27_6 = fmaf(eb, g6_9, o27_6);
            }
            { const float eb = bi[256];
              o27_6 = fmaf(eb, g6_17, o27_6);
            }
            { const float eb = bi[257];
              o27_6 = fmaf(eb, g6_18, o27_6);
            }
            { const float eb = bi[258];
              o27_6 = fmaf(eb, g6_30, o27_6);
            }
            { const float eb = bi[259];
              o28_6 = fmaf(eb, g6_0, o28_6);
            }
            { const float eb = bi[260];
              o28_6 = fmaf(eb, g6_1, o28_6);
            }
            { const float eb = bi[261];
              o28_6 = fmaf(eb, g6_4, o28_6);
            }
            { const float eb = bi[262];
              o28_6 = fmaf(eb, g6_3, o28_6);
            }
            { const float eb = bi[263];
              o28_6 = fmaf(eb, g6_7, o28_6);
            }
            { const float eb = bi[264];
              o28_6 = fmaf(eb, g6_14, o28_6);
            }
            { const float eb = bi[265];
              o28_6 = fmaf(eb, g6_9, o28_6);
            }
            { const float eb = bi[266];
              o28_6 = fmaf(eb, g6_17, o28_6);
            }
            { const float eb = bi[267];
              o28_6 = fmaf(eb, g6_29, o28_6);
            }
            { const float eb = bi[268];
              o29_6 = fmaf(eb, g6_0, o29_6);
            }
            { const float eb = bi[269];
              o29_6 = fmaf(eb, g6_1, o29_6);
            }
            { const float eb = bi[270];
              o29_6 = fmaf(eb, g6_4, o29_6);
            }
            { const float eb = bi[271];
              o29_6 = fmaf(eb, g6_2, o29_6);
            }
            { const float eb = bi[272];
              o29_6 = fmaf(eb, g6_5, o29_6);
            }
            { const float eb = bi[273];
              o29_6 = fmaf(eb, g6_11, o29_6);
            }
            { const float eb = bi[274];
              o29_6 = fmaf(eb, g6_3, o29_6);
            }
            { const float eb = bi[275];
              o29_6 = fmaf(eb, g6_7, o29_6);
            }
            { const float eb = bi[276];
              o29_6 = fmaf(eb, g6_14, o29_6);
            }
            { const float eb = bi[277];
              o29_6 = fmaf(eb, g6_8, o29_6);
            }
            { const float eb = bi[278];
              o29_6 = fmaf(eb, g6_15, o29_6);
            }
            { const float eb = bi[279];
              o29_6 = fmaf(eb, g6_26, o29_6);
            }
            { const float eb = bi[280];
              o30_6 = fmaf(eb, g6_0, o30_6);
            }
            { const float eb = bi[281];
              o30_6 = fmaf(eb, g6_1, o30_6);
            }
            { const float eb = bi[282];
              o30_6 = fmaf(eb, g6_2, o30_6);
            }
            { const float eb = bi[283];
              o30_6 = fmaf(eb, g6_5, o30_6);
            }
            { const float eb = bi[284];
              o30_6 = fmaf(eb, g6_3, o30_6);
            }
            { const float eb = bi[285];
              o30_6 = fmaf(eb, g6_7, o30_6);
            }
            { const float eb = bi[286];
              o30_6 = fmaf(eb, g6_8, o30_6);
            }
            { const float eb = bi[287];
              o30_6 = fmaf(eb, g6_15, o30_6);
            }
            { const float eb = bi[288];
              o30_6 = fmaf(eb, g6_9, o30_6);
            }
            { const float eb = bi[289];
              o30_6 = fmaf(eb, g6_17, o30_6);
            }
            { const float eb = bi[290];
              o30_6 = fmaf(eb, g6_18, o30_6);
            }
            { const float eb = bi[291];
              o30_6 = fmaf(eb, g6_30, o30_6);
            }
            { const float eb = bi[292];
              o31_6 = fmaf(eb, g6_0, o31_6);
            }
            { const float eb = bi[293];
              o31_6 = fmaf(eb, g6_1, o31_6);
            }
            { const float eb = bi[294];
              o31_6 = fmaf(eb, g6_2, o31_6);
            }
            { const float eb = bi[295];
              o31_6 = fmaf(eb, g6_5, o31_6);
            }
            { const float eb = bi[296];
              o31_6 = fmaf(eb, g6_6, o31_6);
            }
            { const float eb = bi[297];
              o31_6 = fmaf(eb, g6_12, o31_6);
            }
            { const float eb = bi[298];
              o31_6 = fmaf(eb, g6_13, o31_6);
            }
            { const float eb = bi[299];
              o31_6 = fmaf(eb, g6_23, o31_6);
            }
            { const float eb = bi[300];
              o32_6 = fmaf(eb, g6_0, o32_6);
            }
            { const float eb = bi[301];
              o32_6 = fmaf(eb, g6_1, o32_6);
            }
            { const float eb = bi[302];
              o32_6 = fmaf(eb, g6_4, o32_6);
            }
            { const float eb = bi[303];
              o32_6 = fmaf(eb, g6_10, o32_6);
            }
            { const float eb = bi[304];
              o32_6 = fmaf(eb, g6_2, o32_6);
            }
            { const float eb = bi[305];
              o32_6 = fmaf(eb, g6_5, o32_6);
            }
            { const float eb = bi[306];
              o32_6 = fmaf(eb, g6_11, o32_6);
            }
            { const float eb = bi[307];
              o32_6 = fmaf(eb, g6_21, o32_6);
            }
            { const float eb = bi[308];
              o33_6 = fmaf(eb, g6_0, o33_6);
            }
            { const float eb = bi[309];
              o33_6 = fmaf(eb, g6_1, o33_6);
            }
            { const float eb = bi[310];
              o33_6 = fmaf(eb, g6_2, o33_6);
            }
            { const float eb = bi[311];
              o33_6 = fmaf(eb, g6_5, o33_6);
            }
            { const float eb = bi[312];
              o33_6 = fmaf(eb, g6_6, o33_6);
            }
            { const float eb = bi[313];
              o33_6 = fmaf(eb, g6_12, o33_6);
            }
            { const float eb = bi[314];
              o33_6 = fmaf(eb, g6_3, o33_6);
            }
            { const float eb = bi[315];
              o33_6 = fmaf(eb, g6_7, o33_6);
            }
            { const float eb = bi[316];
              o33_6 = fmaf(eb, g6_8, o33_6);
            }
            { const float eb = bi[317];
              o33_6 = fmaf(eb, g6_15, o33_6);
            }
            { const float eb = bi[318];
              o33_6 = fmaf(eb, g6_16, o33_6);
            }
            { const float eb = bi[319];
              o33_6 = fmaf(eb, g6_27, o33_6);
            }
            { const float eb = bi[320];
              o34_6 = fmaf(eb, g6_0, o34_6);
            }
            { const float eb = bi[321];
              o34_6 = fmaf(eb, g6_1, o34_6);
            }
            { const float eb = bi[322];
              o34_6 = fmaf(eb, g6_4, o34_6);
            }
            { const float eb = bi[323];
              o34_6 = fmaf(eb, g6_2, o34_6);
            }
            { const float eb = bi[324];
              o34_6 = fmaf(eb, g6_5, o34_6);
            }
            { const float eb = bi[325];
              o34_6 = fmaf(eb, g6_11, o34_6);
            }
            { const float eb = bi[326];
              o34_6 = fmaf(eb, g6_3, o34_6);
            }
            { const float eb = bi[327];
              o34_6 = fmaf(eb, g6_7, o34_6);
            }
            { const float eb = bi[328];
              o34_6 = fmaf(eb, g6_14, o34_6);
            }
            { const float eb = bi[329];
              o34_6 = fmaf(eb, g6_8, o34_6);
            }
            { const float eb = bi[330];
              o34_6 = fmaf(eb, g6_15, o34_6);
            }
            { const float eb = bi[331];
              o34_6 = fmaf(eb, g6_26, o34_6);
            }
            { const float eb = bi[332];
              o35_6 = fmaf(eb, g6_0, o35_6);
            }
            { const float eb = bi[333];
              o35_6 = fmaf(eb, g6_1, o35_6);
            }
            { const float eb = bi[334];
              o35_6 = fmaf(eb, g6_4, o35_6);
            }
            { const float eb = bi[335];
              o35_6 = fmaf(eb, g6_2, o35_6);
            }
            { const float eb = bi[336];
              o35_6 = fmaf(eb, g6_5, o35_6);
            }
            { const float eb = bi[337];
              o35_6 = fmaf(eb, g6_11, o35_6);
            }
            { const float eb = bi[338];
              o35_6 = fmaf(eb, g6_6, o35_6);
            }
            { const float eb = bi[339];
              o35_6 = fmaf(eb, g6_12, o35_6);
            }
            { const float eb = bi[340];
              o35_6 = fmaf(eb, g6_22, o35_6);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk6 = PT[(fI + 1) * N + fJ + 2];
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
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd4_2 = PA[(fQ + 4) * N + fJ + 2];
            const double Abd5_2 = PA[(fQ + 5) * N + fJ + 2];
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
            const double Abc4_1 = PA[(fQ + 4) * N + fI + 1];
            const double Abc5_1 = PA[(fQ + 5) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
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
            jab24 += o24_6 * ptk6;
            jab25 += o25_6 * ptk6;
            jab26 += o26_6 * ptk6;
            jab27 += o27_6 * ptk6;
            jab28 += o28_6 * ptk6;
            jab29 += o29_6 * ptk6;
            jab30 += o30_6 * ptk6;
            jab31 += o31_6 * ptk6;
            jab32 += o32_6 * ptk6;
            jab33 += o33_6 * ptk6;
            jab34 += o34_6 * ptk6;
            jab35 += o35_6 * ptk6;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 2, 2.0 * deg * (o0_6 * ptb0 + o1_6 * ptb1 + o2_6 * ptb2 + o3_6 * ptb3 + o4_6 * ptb4 + o5_6 * ptb5 + o6_6 * ptb6 + o7_6 * ptb7 + o8_6 * ptb8 + o9_6 * ptb9 + o10_6 * ptb10 + o11_6 * ptb11 + o12_6 * ptb12 + o13_6 * ptb13 + o14_6 * ptb14 + o15_6 * ptb15 + o16_6 * ptb16 + o17_6 * ptb17 + o18_6 * ptb18 + o19_6 * ptb19 + o20_6 * ptb20 + o21_6 * ptb21 + o22_6 * ptb22 + o23_6 * ptb23 + o24_6 * ptb24 + o25_6 * ptb25 + o26_6 * ptb26 + o27_6 * ptb27 + o28_6 * ptb28 + o29_6 * ptb29 + o30_6 * ptb30 + o31_6 * ptb31 + o32_6 * ptb32 + o33_6 * ptb33 + o34_6 * ptb34 + o35_6 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_6 * Abd0_2 + o1_6 * Abd1_2 + o2_6 * Abd2_2 + o3_6 * Abd3_2 + o4_6 * Abd4_2 + o5_6 * Abd5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_6 * Aad0_2 + o6_6 * Aad1_2 + o12_6 * Aad2_2 + o18_6 * Aad3_2 + o24_6 * Aad4_2 + o30_6 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_6 * Abc0_1 + o1_6 * Abc1_1 + o2_6 * Abc2_1 + o3_6 * Abc3_1 + o4_6 * Abc4_1 + o5_6 * Abc5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_6 * Aac0_1 + o6_6 * Aac1_1 + o12_6 * Aac2_1 + o18_6 * Aac3_1 + o24_6 * Aac4_1 + o30_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_6 * Aad0_2 + o7_6 * Aad1_2 + o13_6 * Aad2_2 + o19_6 * Aad3_2 + o25_6 * Aad4_2 + o31_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_6 * Aac0_1 + o7_6 * Aac1_1 + o13_6 * Aac2_1 + o19_6 * Aac3_1 + o25_6 * Aac4_1 + o31_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_6 * Aad0_2 + o8_6 * Aad1_2 + o14_6 * Aad2_2 + o20_6 * Aad3_2 + o26_6 * Aad4_2 + o32_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_6 * Aac0_1 + o8_6 * Aac1_1 + o14_6 * Aac2_1 + o20_6 * Aac3_1 + o26_6 * Aac4_1 + o32_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_6 * Aad0_2 + o9_6 * Aad1_2 + o15_6 * Aad2_2 + o21_6 * Aad3_2 + o27_6 * Aad4_2 + o33_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_6 * Aac0_1 + o9_6 * Aac1_1 + o15_6 * Aac2_1 + o21_6 * Aac3_1 + o27_6 * Aac4_1 + o33_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 1, deg * (o4_6 * Aad0_2 + o10_6 * Aad1_2 + o16_6 * Aad2_2 + o22_6 * Aad3_2 + o28_6 * Aad4_2 + o34_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 2, deg * (o4_6 * Aac0_1 + o10_6 * Aac1_1 + o16_6 * Aac2_1 + o22_6 * Aac3_1 + o28_6 * Aac4_1 + o34_6 * Aac5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 1, deg * (o5_6 * Aad0_2 + o11_6 * Aad1_2 + o17_6 * Aad2_2 + o23_6 * Aad3_2 + o29_6 * Aad4_2 + o35_6 * Aad5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 2, deg * (o5_6 * Aac0_1 + o11_6 * Aac1_1 + o17_6 * Aac2_1 + o23_6 * Aac3_1 + o29_6 * Aac4_1 + o35_6 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o6_6 * Abd0_2 + o7_6 * Abd1_2 + o8_6 * Abd2_2 + o9_6 * Abd3_2 + o10_6 * Abd4_2 + o11_6 * Abd5_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o6_6 * Abc0_1 + o7_6 * Abc1_1 + o8_6 * Abc2_1 + o9_6 * Abc3_1 + o10_6 * Abc4_1 + o11_6 * Abc5_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o12_6 * Abd0_2 + o13_6 * Abd1_2 + o14_6 * Abd2_2 + o15_6 * Abd3_2 + o16_6 * Abd4_2 + o17_6 * Abd5_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o12_6 * Abc0_1 + o13_6 * Abc1_1 + o14_6 * Abc2_1 + o15_6 * Abc3_1 + o16_6 * Abc4_1 + o17_6 * Abc5_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o18_6 * Abd0_2 + o19_6 * Abd1_2 + o20_6 * Abd2_2 + o21_6 * Abd3_2 + o22_6 * Abd4_2 + o23_6 * Abd5_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o18_6 * Abc0_1 + o19_6 * Abc1_1 + o20_6 * Abc2_1 + o21_6 * Abc3_1 + o22_6 * Abc4_1 + o23_6 * Abc5_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o24_6 * Abd0_2 + o25_6 * Abd1_2 + o26_6 * Abd2_2 + o27_6 * Abd3_2 + o28_6 * Abd4_2 + o29_6 * Abd5_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o24_6 * Abc0_1 + o25_6 * Abc1_1 + o26_6 * Abc2_1 + o27_6 * Abc3_1 + o28_6 * Abc4_1 + o29_6 * Abc5_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o30_6 * Abd0_2 + o31_6 * Abd1_2 + o32_6 * Abd2_2 + o33_6 * Abd3_2 + o34_6 * Abd4_2 + o35_6 * Abd5_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o30_6 * Abc0_1 + o31_6 * Abc1_1 + o32_6 * Abc2_1 + o33_6 * Abc3_1 + o34_6 * Abc4_1 + o35_6 * Abc5_1));
          }
        } break;
        case 7: {  // ket functions [7]
          float o0_7 = 0;
          float o1_7 = 0;
          float o2_7 = 0;
          float o3_7 = 0;
          float o4_7 = 0;
          float o5_7 = 0;
          float o6_7 = 0;
          float o7_7 = 0;
          float o8_7 = 0;
          float o9_7 = 0;
          float o10_7 = 0;
          float o11_7 = 0;
          float o12_7 = 0;
          float o13_7 = 0;
          float o14_7 = 0;
          float o15_7 = 0;
          float o16_7 = 0;
          float o17_7 = 0;
          float o18_7 = 0;
          float o19_7 = 0;
          float o20_7 = 0;
          float o21_7 = 0;
          float o22_7 = 0;
          float o23_7 = 0;
          float o24_7 = 0;
          float o25_7 = 0;
          float o26_7 = 0;
          float o27_7 = 0;
          float o28_7 = 0;
          float o29_7 = 0;
          float o30_7 = 0;
          float o31_7 = 0;
          float o32_7 = 0;
          float o33_7 = 0;
          float o34_7 = 0;
          float o35_7 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g7_0 = 0;
            float g7_1 = 0;
            float g7_2 = 0;
            float g7_3 = 0;
            float g7_4 = 0;
            float g7_5 = 0;
            float g7_6 = 0;
            float g7_7 = 0;
            float g7_8 = 0;
            float g7_9 = 0;
            float g7_10 = 0;
            float g7_11 = 0;
            float g7_12 = 0;
            float g7_13 = 0;
            float g7_14 = 0;
            float g7_15 = 0;
            float g7_16 = 0;
            float g7_17 = 0;
            float g7_18 = 0;
            float g7_19 = 0;
            float g7_20 = 0;
            float g7_21 = 0;
            float g7_22 = 0;
            float g7_23 = 0;
            float g7_24 = 0;
            float g7_25 = 0;
            float g7_26 = 0;
            float g7_27 = 0;
            float g7_28 = 0;
            float g7_29 = 0;
            float g7_30 = 0;
            float g7_31 = 0;
            float g7_32 = 0;
            float g7_33 = 0;
            float g7_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek7_0 = kj[27 * kS];
              const float ek7_1 = -kj[28 * kS];
              const float ek7_2 = -kj[29 * kS];
              const float ek7_3 = kj[30 * kS];
              g7_0 = fmaf(ek7_0, b0, g7_0);
              const float r0_0_0_1 = Z * b1;
              g7_1 = fmaf(ek7_0, r0_0_0_1, g7_1);
              g7_0 = fmaf(ek7_1, r0_0_0_1, g7_0);
              const float r0_0_1_0 = Y * b1;
              g7_2 = fmaf(ek7_0, r0_0_1_0, g7_2);
              g7_0 = fmaf(ek7_2, r0_0_1_0, g7_0);
              const float r0_1_0_0 = X * b1;
              g7_3 = fmaf(ek7_0, r0_1_0_0, g7_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g7_4 = fmaf(ek7_0, r0_0_0_2, g7_4);
              g7_1 = fmaf(ek7_1, r0_0_0_2, g7_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g7_5 = fmaf(ek7_0, r0_0_1_1, g7_5);
              g7_2 = fmaf(ek7_1, r0_0_1_1, g7_2);
              g7_1 = fmaf(ek7_2, r0_0_1_1, g7_1);
              g7_0 = fmaf(ek7_3, r0_0_1_1, g7_0);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g7_6 = fmaf(ek7_0, r0_0_2_0, g7_6);
              g7_2 = fmaf(ek7_2, r0_0_2_0, g7_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g7_7 = fmaf(ek7_0, r0_1_0_1, g7_7);
              g7_3 = fmaf(ek7_1, r0_1_0_1, g7_3);
              const float r0_1_1_0 = X * r1_0_1_0;
              g7_8 = fmaf(ek7_0, r0_1_1_0, g7_8);
              g7_3 = fmaf(ek7_2, r0_1_1_0, g7_3);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g7_9 = fmaf(ek7_0, r0_2_0_0, g7_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g7_10 = fmaf(ek7_0, r0_0_0_3, g7_10);
              g7_4 = fmaf(ek7_1, r0_0_0_3, g7_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g7_11 = fmaf(ek7_0, r0_0_1_2, g7_11);
              g7_5 = fmaf(ek7_1, r0_0_1_2, g7_5);
              g7_4 = fmaf(ek7_2, r0_0_1_2, g7_4);
              g7_1 = fmaf(ek7_3, r0_0_1_2, g7_1);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g7_12 = fmaf(ek7_0, r0_0_2_1, g7_12);
              g7_6 = fmaf(ek7_1, r0_0_2_1, g7_6);
              g7_5 = fmaf(ek7_2, r0_0_2_1, g7_5);
              g7_2 = fmaf(ek7_3, r0_0_2_1, g7_2);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g7_13 = fmaf(ek7_0, r0_0_3_0, g7_13);
              g7_6 = fmaf(ek7_2, r0_0_3_0, g7_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g7_14 = fmaf(ek7_0, r0_1_0_2, g7_14);
              g7_7 = fmaf(ek7_1, r0_1_0_2, g7_7);
              const float r0_1_1_1 = X * r1_0_1_1;
              g7_15 = fmaf(ek7_0, r0_1_1_1, g7_15);
              g7_8 = fmaf(ek7_1, r0_1_1_1, g7_8);
              g7_7 = fmaf(ek7_2, r0_1_1_1, g7_7);
              g7_3 = fmaf(ek7_3, r0_1_1_1, g7_3);
              const float r0_1_2_0 = X * r1_0_2_0;
              g7_16 = fmaf(ek7_0, r0_1_2_0, g7_16);
              g7_8 = fmaf(ek7_2, r0_1_2_0, g7_8);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g7_17 = fmaf(ek7_0, r0_2_0_1, g7_17);
              g7_9 = fmaf(ek7_1, r0_2_0_1, g7_9);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g7_18 = fmaf(ek7_0, r0_2_1_0, g7_18);
              g7_9 = fmaf(ek7_2, r0_2_1_0, g7_9);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g7_19 = fmaf(ek7_0, r0_3_0_0, g7_19);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g7_20 = fmaf(ek7_0, r0_0_0_4, g7_20);
              g7_10 = fmaf(ek7_1, r0_0_0_4, g7_10);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g7_21 = fmaf(ek7_0, r0_0_1_3, g7_21);
              g7_11 = fmaf(ek7_1, r0_0_1_3, g7_11);
              g7_10 = fmaf(ek7_2, r0_0_1_3, g7_10);
              g7_4 = fmaf(ek7_3, r0_0_1_3, g7_4);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g7_22 = fmaf(ek7_0, r0_0_2_2, g7_22);
              g7_12 = fmaf(ek7_1, r0_0_2_2, g7_12);
              g7_11 = fmaf(ek7_2, r0_0_2_2, g7_11);
              g7_5 = fmaf(ek7_3, r0_0_2_2, g7_5);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g7_23 = fmaf(ek7_0, r0_0_3_1, g7_23);
              g7_13 = fmaf(ek7_1, r0_0_3_1, g7_13);
              g7_12 = fmaf(ek7_2, r0_0_3_1, g7_12);
              g7_6 = fmaf(ek7_3, r0_0_3_1, g7_6);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g7_24 = fmaf(ek7_0, r0_0_4_0, g7_24);
              g7_13 = fmaf(ek7_2, r0_0_4_0, g7_13);
              const float r0_1_0_3 = X * r1_0_0_3;
              g7_25 = fmaf(ek7_0, r0_1_0_3, g7_25);
              g7_14 = fmaf(ek7_1, r0_1_0_3, g7_14);
              const float r0_1_1_2 = X * r1_0_1_2;
              g7_26 = fmaf(ek7_0, r0_1_1_2, g7_26);
              g7_15 = fmaf(ek7_1, r0_1_1_2, g7_15);
              g7_14 = fmaf(ek7_2, r0_1_1_2, g7_14);
              g7_7 = fmaf(ek7_3, r0_1_1_2, g7_7);
              const float r0_1_2_1 = X * r1_0_2_1;
              g7_27 = fmaf(ek7_0, r0_1_2_1, g7_27);
              g7_16 = fmaf(ek7_1, r0_1_2_1, g7_16);
              g7_15 = fmaf(ek7_2, r0_1_2_1, g7_15);
              g7_8 = fmaf(ek7_3, r0_1_2_1, g7_8);
              const float r0_1_3_0 = X * r1_0_3_0;
              g7_28 = fmaf(ek7_0, r0_1_3_0, g7_28);
              g7_16 = fmaf(ek7_2, r0_1_3_0, g7_16);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g7_29 = fmaf(ek7_0, r0_2_0_2, g7_29);
              g7_17 = fmaf(ek7_1, r0_2_0_2, g7_17);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g7_30 = fmaf(ek7_0, r0_2_1_1, g7_30);
              g7_18 = fmaf(ek7_1, r0_2_1_1, g7_18);
              g7_17 = fmaf(ek7_2, r0_2_1_1, g7_17);
              g7_9 = fmaf(ek7_3, r0_2_1_1, g7_9);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g7_31 = fmaf(ek7_0, r0_2_2_0, g7_31);
              g7_18 = fmaf(ek7_2, r0_2_2_0, g7_18);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g7_32 = fmaf(ek7_0, r0_3_0_1, g7_32);
              g7_19 = fmaf(ek7_1, r0_3_0_1, g7_19);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g7_33 = fmaf(ek7_0, r0_3_1_0, g7_33);
              g7_19 = fmaf(ek7_2, r0_3_1_0, g7_19);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g7_34 = fmaf(ek7_0, r0_4_0_0, g7_34);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_0_5 = fmaf(Z, r1_0_0_4, 4.0f * r1_0_0_3);
              g7_20 = fmaf(ek7_1, r0_0_0_5, g7_20);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g7_21 = fmaf(ek7_1, r0_0_1_4, g7_21);
              g7_20 = fmaf(ek7_2, r0_0_1_4, g7_20);
              g7_10 = fmaf(ek7_3, r0_0_1_4, g7_10);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g7_22 = fmaf(ek7_1, r0_0_2_3, g7_22);
              g7_21 = fmaf(ek7_2, r0_0_2_3, g7_21);
              g7_11 = fmaf(ek7_3, r0_0_2_3, g7_11);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g7_23 = fmaf(ek7_1, r0_0_3_2, g7_23);
              g7_22 = fmaf(ek7_2, r0_0_3_2, g7_22);
              g7_12 = fmaf(ek7_3, r0_0_3_2, g7_12);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g7_24 = fmaf(ek7_1, r0_0_4_1, g7_24);
              g7_23 = fmaf(ek7_2, r0_0_4_1, g7_23);
              g7_13 = fmaf(ek7_3, r0_0_4_1, g7_13);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_0_5_0 = fmaf(Y, r1_0_4_0, 4.0f * r1_0_3_0);
              g7_24 = fmaf(ek7_2, r0_0_5_0, g7_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g7_25 = fmaf(ek7_1, r0_1_0_4, g7_25);
              const float r0_1_1_3 = X * r1_0_1_3;
              g7_26 = fmaf(ek7_1, r0_1_1_3, g7_26);
              g7_25 = fmaf(ek7_2, r0_1_1_3, g7_25);
              g7_14 = fmaf(ek7_3, r0_1_1_3, g7_14);
              const float r0_1_2_2 = X * r1_0_2_2;
              g7_27 = fmaf(ek7_1, r0_1_2_2, g7_27);
              g7_26 = fmaf(ek7_2, r0_1_2_2, g7_26);
              g7_15 = fmaf(ek7_3, r0_1_2_2, g7_15);
              const float r0_1_3_1 = X * r1_0_3_1;
              g7_28 = fmaf(ek7_1, r0_1_3_1, g7_28);
              g7_27 = fmaf(ek7_2, r0_1_3_1, g7_27);
              g7_16 = fmaf(ek7_3, r0_1_3_1, g7_16);
              const float r0_1_4_0 = X * r1_0_4_0;
              g7_28 = fmaf(ek7_2, r0_1_4_0, g7_28);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g7_29 = fmaf(ek7_1, r0_2_0_3, g7_29);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g7_30 = fmaf(ek7_1, r0_2_1_2, g7_30);
              g7_29 = fmaf(ek7_2, r0_2_1_2, g7_29);
              g7_17 = fmaf(ek7_3, r0_2_1_2, g7_17);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g7_31 = fmaf(ek7_1, r0_2_2_1, g7_31);
              g7_30 = fmaf(ek7_2, r0_2_2_1, g7_30);
              g7_18 = fmaf(ek7_3, r0_2_2_1, g7_18);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g7_31 = fmaf(ek7_2, r0_2_3_0, g7_31);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g7_32 = fmaf(ek7_1, r0_3_0_2, g7_32);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g7_33 = fmaf(ek7_1, r0_3_1_1, g7_33);
              g7_32 = fmaf(ek7_2, r0_3_1_1, g7_32);
              g7_19 = fmaf(ek7_3, r0_3_1_1, g7_19);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g7_33 = fmaf(ek7_2, r0_3_2_0, g7_33);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g7_34 = fmaf(ek7_1, r0_4_0_1, g7_34);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g7_34 = fmaf(ek7_2, r0_4_1_0, g7_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_0_5 = fmaf(Z, r2_0_0_4, 4.0f * r2_0_0_3);
              const float r0_0_1_5 = Y * r1_0_0_5;
              g7_20 = fmaf(ek7_3, r0_0_1_5, g7_20);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_0_2_4 = fmaf(Y, r1_0_1_4, r1_0_0_4);
              g7_21 = fmaf(ek7_3, r0_0_2_4, g7_21);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_0_3_3 = fmaf(Y, r1_0_2_3, 2.0f * r1_0_1_3);
              g7_22 = fmaf(ek7_3, r0_0_3_3, g7_22);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_0_4_2 = fmaf(Y, r1_0_3_2, 3.0f * r1_0_2_2);
              g7_23 = fmaf(ek7_3, r0_0_4_2, g7_23);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_0_5_1 = fmaf(Y, r1_0_4_1, 4.0f * r1_0_3_1);
              g7_24 = fmaf(ek7_3, r0_0_5_1, g7_24);
              const float r0_1_1_4 = X * r1_0_1_4;
              g7_25 = fmaf(ek7_3, r0_1_1_4, g7_25);
              const float r0_1_2_3 = X * r1_0_2_3;
              g7_26 = fmaf(ek7_3, r0_1_2_3, g7_26);
              const float r0_1_3_2 = X * r1_0_3_2;
              g7_27 = fmaf(ek7_3, r0_1_3_2, g7_27);
              const float r0_1_4_1 = X * r1_0_4_1;
              g7_28 = fmaf(ek7_3, r0_1_4_1, g7_28);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g7_29 = fmaf(ek7_3, r0_2_1_3, g7_29);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g7_30 = fmaf(ek7_3, r0_2_2_2, g7_30);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g7_31 = fmaf(ek7_3, r0_2_3_1, g7_31);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g7_32 = fmaf(ek7_3, r0_3_1_2, g7_32);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g7_33 = fmaf(ek7_3, r0_3_2_1, g7_33);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g7_34 = fmaf(ek7_3, r0_4_1_1, g7_34);
            }
            { const float eb = bi[5];
              o0_7 = fmaf(eb, g7_0, o0_7);
            }
            { const float eb = bi[6];
              o0_7 = fmaf(eb, g7_3, o0_7);
            }
            { const float eb = bi[7];
              o0_7 = fmaf(eb, g7_9, o0_7);
            }
            { const float eb = bi[8];
              o0_7 = fmaf(eb, g7_19, o0_7);
            }
            { const float eb = bi[9];
              o0_7 = fmaf(eb, g7_34, o0_7);
            }
            { const float eb = bi[10];
              o1_7 = fmaf(eb, g7_0, o1_7);
            }
            { const float eb = bi[11];
              o1_7 = fmaf(eb, g7_2, o1_7);
            }
            { const float eb = bi[12];
              o1_7 = fmaf(eb, g7_6, o1_7);
            }
            { const float eb = bi[13];
              o1_7 = fmaf(eb, g7_3, o1_7);
            }
            { const float eb = bi[14];
              o1_7 = fmaf(eb, g7_8, o1_7);
            }
            { const float eb = bi[15];
              o1_7 = fmaf(eb, g7_16, o1_7);
            }
            { const float eb = bi[16];
              o1_7 = fmaf(eb, g7_9, o1_7);
            }
            { const float eb = bi[17];
              o1_7 = fmaf(eb, g7_18, o1_7);
            }
            { const float eb = bi[18];
              o1_7 = fmaf(eb, g7_31, o1_7);
            }
            { const float eb = bi[19];
              o2_7 = fmaf(eb, g7_0, o2_7);
            }
            { const float eb = bi[20];
              o2_7 = fmaf(eb, g7_1, o2_7);
            }
            { const float eb = bi[21];
              o2_7 = fmaf(eb, g7_4, o2_7);
            }
            { const float eb = bi[22];
              o2_7 = fmaf(eb, g7_3, o2_7);
            }
            { const float eb = bi[23];
              o2_7 = fmaf(eb, g7_7, o2_7);
            }
            { const float eb = bi[24];
              o2_7 = fmaf(eb, g7_14, o2_7);
            }
            { const float eb = bi[25];
              o2_7 = fmaf(eb, g7_9, o2_7);
            }
            { const float eb = bi[26];
              o2_7 = fmaf(eb, g7_17, o2_7);
            }
            { const float eb = bi[27];
              o2_7 = fmaf(eb, g7_29, o2_7);
            }
            { const float eb = bi[28];
              o3_7 = fmaf(eb, g7_0, o3_7);
            }
            { const float eb = bi[29];
              o3_7 = fmaf(eb, g7_2, o3_7);
            }
            { const float eb = bi[30];
              o3_7 = fmaf(eb, g7_3, o3_7);
            }
            { const float eb = bi[31];
              o3_7 = fmaf(eb, g7_8, o3_7);
            }
            { const float eb = bi[32];
              o3_7 = fmaf(eb, g7_9, o3_7);
            }
            { const float eb = bi[33];
              o3_7 = fmaf(eb, g7_18, o3_7);
            }
            { const float eb = bi[34];
              o3_7 = fmaf(eb, g7_19, o3_7);
            }
            { const float eb = bi[35];
              o3_7 = fmaf(eb, g7_33, o3_7);
            }
            { const float eb = bi[36];
              o4_7 = fmaf(eb, g7_0, o4_7);
            }
            { const float eb = bi[37];
              o4_7 = fmaf(eb, g7_1, o4_7);
            }
            { const float eb = bi[38];
              o4_7 = fmaf(eb, g7_3, o4_7);
            }
            { const float eb = bi[39];
              o4_7 = fmaf(eb, g7_7, o4_7);
            }
            { const float eb = bi[40];
              o4_7 = fmaf(eb, g7_9, o4_7);
            }
            { const float eb = bi[41];
              o4_7 = fmaf(eb, g7_17, o4_7);
            }
            { const float eb = bi[42];
              o4_7 = fmaf(eb, g7_19, o4_7);
            }
            { const float eb = bi[43];
              o4_7 = fmaf(eb, g7_32, o4_7);
            }
            { const float eb = bi[44];
              o5_7 = fmaf(eb, g7_0, o5_7);
            }
            { const float eb = bi[45];
              o5_7 = fmaf(eb, g7_1, o5_7);
            }
            { const float eb = bi[46];
              o5_7 = fmaf(eb, g7_2, o5_7);
            }
            { const float eb = bi[47];
              o5_7 = fmaf(eb, g7_5, o5_7);
            }
            { const float eb = bi[48];
              o5_7 = fmaf(eb, g7_3, o5_7);
            }
            { const float eb = bi[49];
              o5_7 = fmaf(eb, g7_7, o5_7);
            }
            { const float eb = bi[50];
              o5_7 = fmaf(eb, g7_8, o5_7);
            }
            { const float eb = bi[51];
              o5_7 = fmaf(eb, g7_15, o5_7);
            }
            { const float eb = bi[52];
              o5_7 = fmaf(eb, g7_9, o5_7);
            }
            { const float eb = bi[53];
              o5_7 = fmaf(eb, g7_17, o5_7);
            }
            { const float eb = bi[54];
              o5_7 = fmaf(eb, g7_18, o5_7);
            }
            { const float eb = bi[55];
              o5_7 = fmaf(eb, g7_30, o5_7);
            }
            { const float eb = bi[56];
              o6_7 = fmaf(eb, g7_0, o6_7);
            }
            { const float eb = bi[57];
              o6_7 = fmaf(eb, g7_2, o6_7);
            }
            { const float eb = bi[58];
              o6_7 = fmaf(eb, g7_6, o6_7);
            }
            { const float eb = bi[59];
              o6_7 = fmaf(eb, g7_3, o6_7);
            }
            { const float eb = bi[60];
              o6_7 = fmaf(eb, g7_8, o6_7);
            }
            { const float eb = bi[61];
              o6_7 = fmaf(eb, g7_16, o6_7);
            }
            { const float eb = bi[62];
              o6_7 = fmaf(eb, g7_9, o6_7);
            }
            { const float eb = bi[63];
              o6_7 = fmaf(eb, g7_18, o6_7);
            }
            { const float eb = bi[64];
              o6_7 = fmaf(eb, g7_31, o6_7);
            }
            { const float eb = bi[65];
              o7_7 = fmaf(eb, g7_0, o7_7);
            }
            { const float eb = bi[66];
              o7_7 = fmaf(eb, g7_2, o7_7);
            }
            { const float eb = bi[67];
              o7_7 = fmaf(eb, g7_6, o7_7);
            }
            { const float eb = bi[68];
              o7_7 = fmaf(eb, g7_13, o7_7);
            }
            { const float eb = bi[69];
              o7_7 = fmaf(eb, g7_24, o7_7);
            }
            { const float eb = bi[70];
              o8_7 = fmaf(eb, g7_0, o8_7);
            }
            { const float eb = bi[71];
              o8_7 = fmaf(eb, g7_1, o8_7);
            }
            { const float eb = bi[72];
              o8_7 = fmaf(eb, g7_4, o8_7);
            }
            { const float eb = bi[73];
              o8_7 = fmaf(eb, g7_2, o8_7);
            }
            { const float eb = bi[74];
              o8_7 = fmaf(eb, g7_5, o8_7);
            }
            { const float eb = bi[75];
              o8_7 = fmaf(eb, g7_11, o8_7);
            }
            { const float eb = bi[76];
              o8_7 = fmaf(eb, g7_6, o8_7);
            }
            { const float eb = bi[77];
              o8_7 = fmaf(eb, g7_12, o8_7);
            }
            { const float eb = bi[78];
              o8_7 = fmaf(eb, g7_22, o8_7);
            }
            { const float eb = bi[79];
              o9_7 = fmaf(eb, g7_0, o9_7);
            }
            { const float eb = bi[80];
              o9_7 = fmaf(eb, g7_2, o9_7);
            }
            { const float eb = bi[81];
              o9_7 = fmaf(eb, g7_6, o9_7);
            }
            { const float eb = bi[82];
              o9_7 = fmaf(eb, g7_13, o9_7);
            }
            { const float eb = bi[83];
              o9_7 = fmaf(eb, g7_3, o9_7);
            }
            { const float eb = bi[84];
              o9_7 = fmaf(eb, g7_8, o9_7);
            }
            { const float eb = bi[85];
              o9_7 = fmaf(eb, g7_16, o9_7);
            }
            { const float eb = bi[86];
              o9_7 = fmaf(eb, g7_28, o9_7);
            }
            { const float eb = bi[87];
              o10_7 = fmaf(eb, g7_0, o10_7);
            }
            { const float eb = bi[88];
              o10_7 = fmaf(eb, g7_1, o10_7);
            }
            { const float eb = bi[89];
              o10_7 = fmaf(eb, g7_2, o10_7);
            }
            { const float eb = bi[90];
              o10_7 = fmaf(eb, g7_5, o10_7);
            }
            { const float eb = bi[91];
              o10_7 = fmaf(eb, g7_6, o10_7);
            }
            { const float eb = bi[92];
              o10_7 = fmaf(eb, g7_12, o10_7);
            }
            { const float eb = bi[93];
              o10_7 = fmaf(eb, g7_3, o10_7);
            }
            { const float eb = bi[94];
              o10_7 = fmaf(eb, g7_7, o10_7);
            }
            { const float eb = bi[95];
              o10_7 = fmaf(eb, g7_8, o10_7);
            }
            { const float eb = bi[96];
              o10_7 = fmaf(eb, g7_15, o10_7);
            }
            { const float eb = bi[97];
              o10_7 = fmaf(eb, g7_16, o10_7);
            }
            { const float eb = bi[98];
              o10_7 = fmaf(eb, g7_27, o10_7);
            }
            { const float eb = bi[99];
              o11_7 = fmaf(eb, g7_0, o11_7);
            }
            { const float eb = bi[100];
              o11_7 = fmaf(eb, g7_1, o11_7);
            }
            { const float eb = bi[101];
              o11_7 = fmaf(eb, g7_2, o11_7);
            }
            { const float eb = bi[102];
              o11_7 = fmaf(eb, g7_5, o11_7);
            }
            { const float eb = bi[103];
              o11_7 = fmaf(eb, g7_6, o11_7);
            }
            { const float eb = bi[104];
              o11_7 = fmaf(eb, g7_12, o11_7);
            }
            { const float eb = bi[105];
              o11_7 = fmaf(eb, g7_13, o11_7);
            }
            { const float eb = bi[106];
              o11_7 = fmaf(eb, g7_23, o11_7);
            }
            { const float eb = bi[107];
              o12_7 = fmaf(eb, g7_0, o12_7);
            }
            { const float eb = bi[108];
              o12_7 = fmaf(eb, g7_1, o12_7);
            }
            { const float eb = bi[109];
              o12_7 = fmaf(eb, g7_4, o12_7);
            }
            { const float eb = bi[110];
              o12_7 = fmaf(eb, g7_3, o12_7);
            }
            { const float eb = bi[111];
              o12_7 = fmaf(eb, g7_7, o12_7);
            }
            { const float eb = bi[112];
              o12_7 = fmaf(eb, g7_14, o12_7);
            }
            { const float eb = bi[113];
              o12_7 = fmaf(eb, g7_9, o12_7);
            }
            { const float eb = bi[114];
              o12_7 = fmaf(eb, g7_17, o12_7);
            }
            { const float eb = bi[115];
              o12_7 = fmaf(eb, g7_29, o12_7);
            }
            { const float eb = bi[116];
              o13_7 = fmaf(eb, g7_0, o13_7);
            }
            { const float eb = bi[117];
              o13_7 = fmaf(eb, g7_1, o13_7);
            }
            { const float eb = bi[118];
              o13_7 = fmaf(eb, g7_4, o13_7);
            }
            { const float eb = bi[119];
              o13_7 = fmaf(eb, g7_2, o13_7);
            }
            { const float eb = bi[120];
              o13_7 = fmaf(eb, g7_5, o13_7);
            }
            { const float eb = bi[121];
              o13_7 = fmaf(eb, g7_11, o13_7);
            }
            { const float eb = bi[122];
              o13_7 = fmaf(eb, g7_6, o13_7);
            }
            { const float eb = bi[123];
              o13_7 = fmaf(eb, g7_12, o13_7);
            }
            { const float eb = bi[124];
              o13_7 = fmaf(eb, g7_22, o13_7);
            }
            { const float eb = bi[125];
              o14_7 = fmaf(eb, g7_0, o14_7);
            }
            { const float eb = bi[126];
              o14_7 = fmaf(eb, g7_1, o14_7);
            }
            { const float eb = bi[127];
              o14_7 = fmaf(eb, g7_4, o14_7);
            }
            { const float eb = bi[128];
              o14_7 = fmaf(eb, g7_10, o14_7);
            }
            { const float eb = bi[129];
              o14_7 = fmaf(eb, g7_20, o14_7);
            }
            { const float eb = bi[130];
              o15_7 = fmaf(eb, g7_0, o15_7);
            }
            { const float eb = bi[131];
              o15_7 = fmaf(eb, g7_1, o15_7);
            }
            { const float eb = bi[132];
              o15_7 = fmaf(eb, g7_4, o15_7);
            }
            { const float eb = bi[133];
              o15_7 = fmaf(eb, g7_2, o15_7);
            }
            { const float eb = bi[134];
              o15_7 = fmaf(eb, g7_5, o15_7);
            }
            { const float eb = bi[135];
              o15_7 = fmaf(eb, g7_11, o15_7);
            }
            { const float eb = bi[136];
              o15_7 = fmaf(eb, g7_3, o15_7);
            }
            { const float eb = bi[137];
              o15_7 = fmaf(eb, g7_7, o15_7);
            }
            { const float eb = bi[138];
              o15_7 = fmaf(eb, g7_14, o15_7);
            }
            { const float eb = bi[139];
              o15_7 = fmaf(eb, g7_8, o15_7);
            }
            { const float eb = bi[140];
              o15_7 = fmaf(eb, g7_15, o15_7);
            }
            { const float eb = bi[141];
              o15_7 = fmaf(eb, g7_26, o15_7);
            }
            { const float eb = bi[142];
              o16_7 = fmaf(eb, g7_0, o16_7);
            }
            { const float eb = bi[143];
              o16_7 = fmaf(eb, g7_1, o16_7);
            }
            { const float eb = bi[144];
              o16_7 = fmaf(eb, g7_4, o16_7);
            }
            { const float eb = bi[145];
              o16_7 = fmaf(eb, g7_10, o16_7);
            }
            { const float eb = bi[146];
              o16_7 = fmaf(eb, g7_3, o16_7);
            }
            { const float eb = bi[147];
              o16_7 = fmaf(eb, g7_7, o16_7);
            }
            { const float eb = bi[148];
              o16_7 = fmaf(eb, g7_14, o16_7);
            }
            { const float eb = bi[149];
              o16_7 = fmaf(eb, g7_25, o16_7);
            }
            { const float eb = bi[150];
              o17_7 = fmaf(eb, g7_0, o17_7);
            }
            { const float eb = bi[151];
              o17_7 = fmaf(eb, g7_1, o17_7);
            }
            { const float eb = bi[152];
              o17_7 = fmaf(eb, g7_4, o17_7);
            }
            { const float eb = bi[153];
              o17_7 = fmaf(eb, g7_10, o17_7);
            }
            { const float eb = bi[154];
              o17_7 = fmaf(eb, g7_2, o17_7);
            }
            { const float eb = bi[155];
              o17_7 = fmaf(eb, g7_5, o17_7);
            }
            { const float eb = bi[156];
              o17_7 = fmaf(eb, g7_11, o17_7);
            }
            { const float eb = bi[157];
              o17_7 = fmaf(eb, g7_21, o17_7);
            }
            { const float eb = bi[158];
              o18_7 = fmaf(eb, g7_0, o18_7);
            }
            { const float eb = bi[159];
              o18_7 = fmaf(eb, g7_2, o18_7);
            }
            { const float eb = bi[160];
              o18_7 = fmaf(eb, g7_3, o18_7);
            }
            { const float eb = bi[161];
              o18_7 = fmaf(eb, g7_8, o18_7);
            }
            { const float eb = bi[162];
              o18_7 = fmaf(eb, g7_9, o18_7);
            }
            { const float eb = bi[163];
              o18_7 = fmaf(eb, g7_18, o18_7);
            }
            { const float eb = bi[164];
              o18_7 = fmaf(eb, g7_19, o18_7);
            }
            { const float eb = bi[165];
              o18_7 = fmaf(eb, g7_33, o18_7);
            }
            { const float eb = bi[166];
              o19_7 = fmaf(eb, g7_0, o19_7);
            }
            { const float eb = bi[167];
              o19_7 = fmaf(eb, g7_2, o19_7);
            }
            { const float eb = bi[168];
              o19_7 = fmaf(eb, g7_6, o19_7);
            }
            { const float eb = bi[169];
              o19_7 = fmaf(eb, g7_13, o19_7);
            }
            { const float eb = bi[170];
              o19_7 = fmaf(eb, g7_3, o19_7);
            }
            { const float eb = bi[171];
              o19_7 = fmaf(eb, g7_8, o19_7);
            }
            { const float eb = bi[172];
              o19_7 = fmaf(eb, g7_16, o19_7);
            }
            { const float eb = bi[173];
              o19_7 = fmaf(eb, g7_28, o19_7);
            }
            { const float eb = bi[174];
              o20_7 = fmaf(eb, g7_0, o20_7);
            }
            { const float eb = bi[175];
              o20_7 = fmaf(eb, g7_1, o20_7);
            }
            { const float eb = bi[176];
              o20_7 = fmaf(eb, g7_4, o20_7);
            }
            { const float eb = bi[177];
              o20_7 = fmaf(eb, g7_2, o20_7);
            }
            { const float eb = bi[178];
              o20_7 = fmaf(eb, g7_5, o20_7);
            }
            { const float eb = bi[179];
              o20_7 = fmaf(eb, g7_11, o20_7);
            }
            { const float eb = bi[180];
              o20_7 = fmaf(eb, g7_3, o20_7);
            }
            { const float eb = bi[181];
              o20_7 = fmaf(eb, g7_7, o20_7);
            }
            { const float eb = bi[182];
              o20_7 = fmaf(eb, g7_14, o20_7);
            }
            { const float eb = bi[183];
              o20_7 = fmaf(eb, g7_8, o20_7);
            }
            { const float eb = bi[184];
              o20_7 = fmaf(eb, g7_15, o20_7);
            }
            { const float eb = bi[185];
              o20_7 = fmaf(eb, g7_26, o20_7);
            }
            { const float eb = bi[186];
              o21_7 = fmaf(eb, g7_0, o21_7);
            }
            { const float eb = bi[187];
              o21_7 = fmaf(eb, g7_2, o21_7);
            }
            { const float eb = bi[188];
              o21_7 = fmaf(eb, g7_6, o21_7);
            }
            { const float eb = bi[189];
              o21_7 = fmaf(eb, g7_3, o21_7);
            }
            { const float eb = bi[190];
              o21_7 = fmaf(eb, g7_8, o21_7);
            }
            { const float eb = bi[191];
              o21_7 = fmaf(eb, g7_16, o21_7);
            }
            { const float eb = bi[192];
              o21_7 = fmaf(eb, g7_9, o21_7);
            }
            { const float eb = bi[193];
              o21_7 = fmaf(eb, g7_18, o21_7);
            }
            { const float eb = bi[194];
              o21_7 = fmaf(eb, g7_31, o21_7);
            }
            { const float eb = bi[195];
              o22_7 = fmaf(eb, g7_0, o22_7);
            }
            { const float eb = bi[196];
              o22_7 = fmaf(eb, g7_1, o22_7);
            }
            { const float eb = bi[197];
              o22_7 = fmaf(eb, g7_2, o22_7);
            }
            { const float eb = bi[198];
              o22_7 = fmaf(eb, g7_5, o22_7);
            }
            { const float eb = bi[199];
              o22_7 = fmaf(eb, g7_3, o22_7);
            }
            { const float eb = bi[200];
              o22_7 = fmaf(eb, g7_7, o22_7);
            }
            { const float eb = bi[201];
              o22_7 = fmaf(eb, g7_8, o22_7);
            }
            { const float eb = bi[202];
              o22_7 = fmaf(eb, g7_15, o22_7);
            }
            { const float eb = bi[203];
              o22_7 = fmaf(eb, g7_9, o22_7);
            }
            { const float eb = bi[204];
              o22_7 = fmaf(eb, g7_17, o22_7);
            }
            { const float eb = bi[205];
              o22_7 = fmaf(eb, g7_18, o22_7);
            }
            { const float eb = bi[206];
              o22_7 = fmaf(eb, g7_30, o22_7);
            }
            { const float eb = bi[207];
              o23_7 = fmaf(eb, g7_0, o23_7);
            }
            { const float eb = bi[208];
              o23_7 = fmaf(eb, g7_1, o23_7);
            }
            { const float eb = bi[209];
              o23_7 = fmaf(eb, g7_2, o23_7);
            }
            { const float eb = bi[210];
              o23_7 = fmaf(eb, g7_5, o23_7);
            }
            { const float eb = bi[211];
              o23_7 = fmaf(eb, g7_6, o23_7);
            }
            { const float eb = bi[212];
              o23_7 = fmaf(eb, g7_12, o23_7);
            }
            { const float eb = bi[213];
              o23_7 = fmaf(eb, g7_3, o23_7);
            }
            { const float eb = bi[214];
              o23_7 = fmaf(eb, g7_7, o23_7);
            }
            { const float eb = bi[215];
              o23_7 = fmaf(eb, g7_8, o23_7);
            }
            { const float eb = bi[216];
              o23_7 = fmaf(eb, g7_15, o23_7);
            }
            { const float eb = bi[217];
              o23_7 = fmaf(eb, g7_16, o23_7);
            }
            { const float eb = bi[218];
              o23_7 = fmaf(eb, g7_27, o23_7);
            }
            { const float eb = bi[219];
              o24_7 = fmaf(eb, g7_0, o24_7);
            }
            { const float eb = bi[220];
              o24_7 = fmaf(eb, g7_1, o24_7);
            }
            { const float eb = bi[221];
              o24_7 = fmaf(eb, g7_3, o24_7);
            }
            { const float eb = bi[222];
              o24_7 = fmaf(eb, g7_7, o24_7);
            }
            { const float eb = bi[223];
              o24_7 = fmaf(eb, g7_9, o24_7);
            }
            { const float eb = bi[224];
              o24_7 = fmaf(eb, g7_17, o24_7);
            }
            { const float eb = bi[225];
              o24_7 = fmaf(eb, g7_19, o24_7);
            }
            { const float eb = bi[226];
              o24_7 = fmaf(eb, g7_32, o24_7);
            }
            { const float eb = bi[227];
              o25_7 = fmaf(eb, g7_0, o25_7);
            }
            { const float eb = bi[228];
              o25_7 = fmaf(eb, g7_1, o25_7);
            }
            { const float eb = bi[229];
              o25_7 = fmaf(eb, g7_2, o25_7);
            }
            { const float eb = bi[230];
              o25_7 = fmaf(eb, g7_5, o25_7);
            }
            { const float eb = bi[231];
              o25_7 = fmaf(eb, g7_6, o25_7);
            }
            { const float eb = bi[232];
              o25_7 = fmaf(eb, g7_12, o25_7);
            }
            { const float eb = bi[233];
              o25_7 = fmaf(eb, g7_3, o25_7);
            }
            { const float eb = bi[234];
              o25_7 = fmaf(eb, g7_7, o25_7);
            }
            { const float eb = bi[235];
              o25_7 = fmaf(eb, g7_8, o25_7);
            }
            { const float eb = bi[236];
              o25_7 = fmaf(eb, g7_15, o25_7);
            }
            { const float eb = bi[237];
              o25_7 = fmaf(eb, g7_16, o25_7);
            }
            { const float eb = bi[238];
              o25_7 = fmaf(eb, g7_27, o25_7);
            }
            { const float eb = bi[239];
              o26_7 = fmaf(eb, g7_0, o26_7);
            }
            { const float eb = bi[240];
              o26_7 = fmaf(eb, g7_1, o26_7);
            }
            { const float eb = bi[241];
              o26_7 = fmaf(eb, g7_4, o26_7);
            }
            { const float eb = bi[242];
              o26_7 = fmaf(eb, g7_10, o26_7);
            }
            { const float eb = bi[243];
              o26_7 = fmaf(eb, g7_3, o26_7);
            }
            { const float eb = bi[244];
              o26_7 = fmaf(eb, g7_7, o26_7);
            }
            { const float eb = bi[245];
              o26_7 = fmaf(eb, g7_14, o26_7);
            }
            { const float eb = bi[246];
              o26_7 = fmaf(eb, g7_25, o26_7);
            }
            { const float eb = bi[247];
              o27_7 = fmaf(eb, g7_0, o27_7);
            }
            { const float eb = bi[248];
              o27_7 = fmaf(eb, g7_1, o27_7);
            }
            { const float eb = bi[249];
              o27_7 = fmaf(eb, g7_2, o27_7);
            }
            { const float eb = bi[250];
              o27_7 = fmaf(eb, g7_5, o27_7);
            }
            { const float eb = bi[251];
              o27_7 = fmaf(eb, g7_3, o27_7);
            }
            { const float eb = bi[252];
              o27_7 = fmaf(eb, g7_7, o27_7);
            }
            { const float eb = bi[253];
              o27_7 = fmaf(eb, g7_8, o27_7);
            }
            { const float eb = bi[254];
              o27_7 = fmaf(eb, g7_15, o27_7);
            }
            { const float eb = bi[255];
              o27_7 = fmaf(eb, g7_9, o27_7);
            }
            { const float eb = bi[256];
              o27_7 = fmaf(eb, g7_17, o27_7);
            }
            { const float eb = bi[257];
              o27_7 = fmaf(eb, g7_18, o27_7);
            }
            { const float eb = bi[258];
              o27_7 = fmaf(eb, g7_30, o27_7);
            }
            { const float eb = bi[259];
              o28_7 = fmaf(eb, g7_0, o28_7);
            }
            { const float eb = bi[260];
              o28_7 = fmaf(eb, g7_1, o28_7);
            }
            { const float eb = bi[261];
              o28_7 = fmaf(eb, g7_4, o28_7);
            }
            { const float eb = bi[262];
              o28_7 = fmaf(eb, g7_3, o28_7);
            }
            { const float eb = bi[263];
              o28_7 = fmaf(eb, g7_7, o28_7);
            }
            { const float eb = bi[264];
              o28_7 = fmaf(eb, g7_14, o28_7);
            }
            { const float eb = bi[265];
              o28_7 = fmaf(eb, g7_9, o28_7);
            }
            { const float eb = bi[266];
              o28_7 = fmaf(eb, g7_17, o28_7);
            }
            { const float eb = bi[267];
              o28_7 = fmaf(eb, g7_29, o28_7);
            }
            { const float eb = bi[268];
              o29_7 = fmaf(eb, g7_0, o29_7);
            }
            { const float eb = bi[269];
              o29_7 = fmaf(eb, g7_1, o29_7);
            }
            { const float eb = bi[270];
              o29_7 = fmaf(eb, g7_4, o29_7);
            }
            { const float eb = bi[271];
              o29_7 = fmaf(eb, g7_2, o29_7);
            }
            { const float eb = bi[272];
              o29_7 = fmaf(eb, g7_5, o29_7);
            }
            { const float eb = bi[273];
              o29_7 = fmaf(eb, g7_11, o29_7);
            }
            { const float eb = bi[274];
              o29_7 = fmaf(eb, g7_3, o29_7);
            }
            { const float eb = bi[275];
              o29_7 = fmaf(eb, g7_7, o29_7);
            }
            { const float eb = bi[276];
              o29_7 = fmaf(eb, g7_14, o29_7);
            }
            { const float eb = bi[277];
              o29_7 = fmaf(eb, g7_8, o29_7);
            }
            { const float eb = bi[278];
              o29_7 = fmaf(eb, g7_15, o29_7);
            }
            { const float eb = bi[279];
              o29_7 = fmaf(eb, g7_26, o29_7);
            }
            { const float eb = bi[280];
              o30_7 = fmaf(eb, g7_0, o30_7);
            }
            { const float eb = bi[281];
              o30_7 = fmaf(eb, g7_1, o30_7);
            }
            { const float eb = bi[282];
              o30_7 = fmaf(eb, g7_2, o30_7);
            }
            { const float eb = bi[283];
              o30_7 = fmaf(eb, g7_5, o30_7);
            }
            { const float eb = bi[284];
              o30_7 = fmaf(eb, g7_3, o30_7);
            }
            { const float eb = bi[285];
              o30_7 = fmaf(eb, g7_7, o30_7);
            }
            { const float eb = bi[286];
              o30_7 = fmaf(eb, g7_8, o30_7);
            }
            { const float eb = bi[287];
              o30_7 = fmaf(eb, g7_15, o30_7);
            }
            { const float eb = bi[288];
              o30_7 = fmaf(eb, g7_9, o30_7);
            }
            { const float eb = bi[289];
              o30_7 = fmaf(eb, g7_17, o30_7);
            }
            { const float eb = bi[290];
              o30_7 = fmaf(eb, g7_18, o30_7);
            }
            { const float eb = bi[291];
              o30_7 = fmaf(eb, g7_30, o30_7);
            }
            { const float eb = bi[292];
              o31_7 = fmaf(eb, g7_0, o31_7);
            }
            { const float eb = bi[293];
              o31_7 = fmaf(eb, g7_1, o31_7);
            }
            { const float eb = bi[294];
              o31_7 = fmaf(eb, g7_2, o31_7);
            }
            { const float eb = bi[295];
              o31_7 = fmaf(eb, g7_5, o31_7);
            }
            { const float eb = bi[296];
              o31_7 = fmaf(eb, g7_6, o31_7);
            }
            { const float eb = bi[297];
              o31_7 = fmaf(eb, g7_12, o31_7);
            }
            { const float eb = bi[298];
              o31_7 = fmaf(eb, g7_13, o31_7);
            }
            { const float eb = bi[299];
              o31_7 = fmaf(eb, g7_23, o31_7);
            }
            { const float eb = bi[300];
              o32_7 = fmaf(eb, g7_0, o32_7);
            }
            { const float eb = bi[301];
              o32_7 = fmaf(eb, g7_1, o32_7);
            }
            { const float eb = bi[302];
              o32_7 = fmaf(eb, g7_4, o32_7);
            }
            { const float eb = bi[303];
              o32_7 = fmaf(eb, g7_10, o32_7);
            }
            { const float eb = bi[304];
              o32_7 = fmaf(eb, g7_2, o32_7);
            }
            { const float eb = bi[305];
              o32_7 = fmaf(eb, g7_5, o32_7);
            }
            { const float eb = bi[306];
              o32_7 = fmaf(eb, g7_11, o32_7);
            }
            { const float eb = bi[307];
              o32_7 = fmaf(eb, g7_21, o32_7);
            }
            { const float eb = bi[308];
              o33_7 = fmaf(eb, g7_0, o33_7);
            }
            { const float eb = bi[309];
              o33_7 = fmaf(eb, g7_1, o33_7);
            }
            { const float eb = bi[310];
              o33_7 = fmaf(eb, g7_2, o33_7);
            }
            { const float eb = bi[311];
              o33_7 = fmaf(eb, g7_5, o33_7);
            }
            { const float eb = bi[312];
              o33_7 = fmaf(eb, g7_6, o33_7);
            }
            { const float eb = bi[313];
              o33_7 = fmaf(eb, g7_12, o33_7);
            }
            { const float eb = bi[314];
              o33_7 = fmaf(eb, g7_3, o33_7);
            }
            { const float eb = bi[315];
              o33_7 = fmaf(eb, g7_7, o33_7);
            }
            { const float eb = bi[316];
              o33_7 = fmaf(eb, g7_8, o33_7);
            }
            { const float eb = bi[317];
              o33_7 = fmaf(eb, g7_15, o33_7);
            }
            { const float eb = bi[318];
              o33_7 = fmaf(eb, g7_16, o33_7);
            }
            { const float eb = bi[319];
              o33_7 = fmaf(eb, g7_27, o33_7);
            }
            { const float eb = bi[320];
              o34_7 = fmaf(eb, g7_0, o34_7);
            }
            { const float eb = bi[321];
              o34_7 = fmaf(eb, g7_1, o34_7);
            }
            { const float eb = bi[322];
              o34_7 = fmaf(eb, g7_4, o34_7);
            }
            { const float eb = bi[323];
              o34_7 = fmaf(eb, g7_2, o34_7);
            }
            { const float eb = bi[324];
              o34_7 = fmaf(eb, g7_5, o34_7);
            }
            { const float eb = bi[325];
              o34_7 = fmaf(eb, g7_11, o34_7);
            }
            { const float eb = bi[326];
              o34_7 = fmaf(eb, g7_3, o34_7);
            }
            { const float eb = bi[327];
              o34_7 = fmaf(eb, g7_7, o34_7);
            }
            { const float eb = bi[328];
              o34_7 = fmaf(eb, g7_14, o34_7);
            }
            { const float eb = bi[329];
              o34_7 = fmaf(eb, g7_8, o34_7);
            }
            { const float eb = bi[330];
              o34_7 = fmaf(eb, g7_15, o34_7);
            }
            { const float eb = bi[331];
              o34_7 = fmaf(eb, g7_26, o34_7);
            }
            { const float eb = bi[332];
              o35_7 = fmaf(eb, g7_0, o35_7);
            }
            { const float eb = bi[333];
              o35_7 = fmaf(eb, g7_1, o35_7);
            }
            { const float eb = bi[334];
              o35_7 = fmaf(eb, g7_4, o35_7);
            }
            { const float eb = bi[335];
              o35_7 = fmaf(eb, g7_2, o35_7);
            }
            { const float eb = bi[336];
              o35_7 = fmaf(eb, g7_5, o35_7);
            }
            { const float eb = bi[337];
              o35_7 = fmaf(eb, g7_11, o35_7);
            }
            { const float eb = bi[338];
              o35_7 = fmaf(eb, g7_6, o35_7);
            }
            { const float eb = bi[339];
              o35_7 = fmaf(eb, g7_12, o35_7);
            }
            { const float eb = bi[340];
              o35_7 = fmaf(eb, g7_22, o35_7);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk7 = PT[(fI + 1) * N + fJ + 3];
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Abd4_3 = PA[(fQ + 4) * N + fJ + 3];
            const double Abd5_3 = PA[(fQ + 5) * N + fJ + 3];
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
            const double Abc4_1 = PA[(fQ + 4) * N + fI + 1];
            const double Abc5_1 = PA[(fQ + 5) * N + fI + 1];
            const double Aac0_1 = PA[(fP + 0) * N + fI + 1];
            const double Aac1_1 = PA[(fP + 1) * N + fI + 1];
            const double Aac2_1 = PA[(fP + 2) * N + fI + 1];
            const double Aac3_1 = PA[(fP + 3) * N + fI + 1];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
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
            jab24 += o24_7 * ptk7;
            jab25 += o25_7 * ptk7;
            jab26 += o26_7 * ptk7;
            jab27 += o27_7 * ptk7;
            jab28 += o28_7 * ptk7;
            jab29 += o29_7 * ptk7;
            jab30 += o30_7 * ptk7;
            jab31 += o31_7 * ptk7;
            jab32 += o32_7 * ptk7;
            jab33 += o33_7 * ptk7;
            jab34 += o34_7 * ptk7;
            jab35 += o35_7 * ptk7;
            atomicAdd(Jacc + (fI + 1) * N + fJ + 3, 2.0 * deg * (o0_7 * ptb0 + o1_7 * ptb1 + o2_7 * ptb2 + o3_7 * ptb3 + o4_7 * ptb4 + o5_7 * ptb5 + o6_7 * ptb6 + o7_7 * ptb7 + o8_7 * ptb8 + o9_7 * ptb9 + o10_7 * ptb10 + o11_7 * ptb11 + o12_7 * ptb12 + o13_7 * ptb13 + o14_7 * ptb14 + o15_7 * ptb15 + o16_7 * ptb16 + o17_7 * ptb17 + o18_7 * ptb18 + o19_7 * ptb19 + o20_7 * ptb20 + o21_7 * ptb21 + o22_7 * ptb22 + o23_7 * ptb23 + o24_7 * ptb24 + o25_7 * ptb25 + o26_7 * ptb26 + o27_7 * ptb27 + o28_7 * ptb28 + o29_7 * ptb29 + o30_7 * ptb30 + o31_7 * ptb31 + o32_7 * ptb32 + o33_7 * ptb33 + o34_7 * ptb34 + o35_7 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_7 * Abd0_3 + o1_7 * Abd1_3 + o2_7 * Abd2_3 + o3_7 * Abd3_3 + o4_7 * Abd4_3 + o5_7 * Abd5_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_7 * Aad0_3 + o6_7 * Aad1_3 + o12_7 * Aad2_3 + o18_7 * Aad3_3 + o24_7 * Aad4_3 + o30_7 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_7 * Abc0_1 + o1_7 * Abc1_1 + o2_7 * Abc2_1 + o3_7 * Abc3_1 + o4_7 * Abc4_1 + o5_7 * Abc5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_7 * Aac0_1 + o6_7 * Aac1_1 + o12_7 * Aac2_1 + o18_7 * Aac3_1 + o24_7 * Aac4_1 + o30_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 1, deg * (o1_7 * Aad0_3 + o7_7 * Aad1_3 + o13_7 * Aad2_3 + o19_7 * Aad3_3 + o25_7 * Aad4_3 + o31_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_7 * Aac0_1 + o7_7 * Aac1_1 + o13_7 * Aac2_1 + o19_7 * Aac3_1 + o25_7 * Aac4_1 + o31_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 1, deg * (o2_7 * Aad0_3 + o8_7 * Aad1_3 + o14_7 * Aad2_3 + o20_7 * Aad3_3 + o26_7 * Aad4_3 + o32_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_7 * Aac0_1 + o8_7 * Aac1_1 + o14_7 * Aac2_1 + o20_7 * Aac3_1 + o26_7 * Aac4_1 + o32_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 1, deg * (o3_7 * Aad0_3 + o9_7 * Aad1_3 + o15_7 * Aad2_3 + o21_7 * Aad3_3 + o27_7 * Aad4_3 + o33_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_7 * Aac0_1 + o9_7 * Aac1_1 + o15_7 * Aac2_1 + o21_7 * Aac3_1 + o27_7 * Aac4_1 + o33_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 1, deg * (o4_7 * Aad0_3 + o10_7 * Aad1_3 + o16_7 * Aad2_3 + o22_7 * Aad3_3 + o28_7 * Aad4_3 + o34_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 3, deg * (o4_7 * Aac0_1 + o10_7 * Aac1_1 + o16_7 * Aac2_1 + o22_7 * Aac3_1 + o28_7 * Aac4_1 + o34_7 * Aac5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 1, deg * (o5_7 * Aad0_3 + o11_7 * Aad1_3 + o17_7 * Aad2_3 + o23_7 * Aad3_3 + o29_7 * Aad4_3 + o35_7 * Aad5_3));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 3, deg * (o5_7 * Aac0_1 + o11_7 * Aac1_1 + o17_7 * Aac2_1 + o23_7 * Aac3_1 + o29_7 * Aac4_1 + o35_7 * Aac5_1));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o6_7 * Abd0_3 + o7_7 * Abd1_3 + o8_7 * Abd2_3 + o9_7 * Abd3_3 + o10_7 * Abd4_3 + o11_7 * Abd5_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o6_7 * Abc0_1 + o7_7 * Abc1_1 + o8_7 * Abc2_1 + o9_7 * Abc3_1 + o10_7 * Abc4_1 + o11_7 * Abc5_1));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o12_7 * Abd0_3 + o13_7 * Abd1_3 + o14_7 * Abd2_3 + o15_7 * Abd3_3 + o16_7 * Abd4_3 + o17_7 * Abd5_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o12_7 * Abc0_1 + o13_7 * Abc1_1 + o14_7 * Abc2_1 + o15_7 * Abc3_1 + o16_7 * Abc4_1 + o17_7 * Abc5_1));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o18_7 * Abd0_3 + o19_7 * Abd1_3 + o20_7 * Abd2_3 + o21_7 * Abd3_3 + o22_7 * Abd4_3 + o23_7 * Abd5_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o18_7 * Abc0_1 + o19_7 * Abc1_1 + o20_7 * Abc2_1 + o21_7 * Abc3_1 + o22_7 * Abc4_1 + o23_7 * Abc5_1));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o24_7 * Abd0_3 + o25_7 * Abd1_3 + o26_7 * Abd2_3 + o27_7 * Abd3_3 + o28_7 * Abd4_3 + o29_7 * Abd5_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o24_7 * Abc0_1 + o25_7 * Abc1_1 + o26_7 * Abc2_1 + o27_7 * Abc3_1 + o28_7 * Abc4_1 + o29_7 * Abc5_1));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o30_7 * Abd0_3 + o31_7 * Abd1_3 + o32_7 * Abd2_3 + o33_7 * Abd3_3 + o34_7 * Abd4_3 + o35_7 * Abd5_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o30_7 * Abc0_1 + o31_7 * Abc1_1 + o32_7 * Abc2_1 + o33_7 * Abc3_1 + o34_7 * Abc4_1 + o35_7 * Abc5_1));
          }
        } break;
        case 8: {  // ket functions [8]
          float o0_8 = 0;
          float o1_8 = 0;
          float o2_8 = 0;
          float o3_8 = 0;
          float o4_8 = 0;
          float o5_8 = 0;
          float o6_8 = 0;
          float o7_8 = 0;
          float o8_8 = 0;
          float o9_8 = 0;
          float o10_8 = 0;
          float o11_8 = 0;
          float o12_8 = 0;
          float o13_8 = 0;
          float o14_8 = 0;
          float o15_8 = 0;
          float o16_8 = 0;
          float o17_8 = 0;
          float o18_8 = 0;
          float o19_8 = 0;
          float o20_8 = 0;
          float o21_8 = 0;
          float o22_8 = 0;
          float o23_8 = 0;
          float o24_8 = 0;
          float o25_8 = 0;
          float o26_8 = 0;
          float o27_8 = 0;
          float o28_8 = 0;
          float o29_8 = 0;
          float o30_8 = 0;
          float o31_8 = 0;
          float o32_8 = 0;
          float o33_8 = 0;
          float o34_8 = 0;
          float o35_8 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g8_0 = 0;
            float g8_1 = 0;
            float g8_2 = 0;
            float g8_3 = 0;
            float g8_4 = 0;
            float g8_5 = 0;
            float g8_6 = 0;
            float g8_7 = 0;
            float g8_8 = 0;
            float g8_9 = 0;
            float g8_10 = 0;
            float g8_11 = 0;
            float g8_12 = 0;
            float g8_13 = 0;
            float g8_14 = 0;
            float g8_15 = 0;
            float g8_16 = 0;
            float g8_17 = 0;
            float g8_18 = 0;
            float g8_19 = 0;
            float g8_20 = 0;
            float g8_21 = 0;
            float g8_22 = 0;
            float g8_23 = 0;
            float g8_24 = 0;
            float g8_25 = 0;
            float g8_26 = 0;
            float g8_27 = 0;
            float g8_28 = 0;
            float g8_29 = 0;
            float g8_30 = 0;
            float g8_31 = 0;
            float g8_32 = 0;
            float g8_33 = 0;
            float g8_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[6];
              sqb::boysf<5>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              const float ek8_0 = kj[31 * kS];
              const float ek8_1 = -kj[32 * kS];
              g8_0 = fmaf(ek8_0, b0, g8_0);
              const float r0_0_0_1 = Z * b1;
              g8_1 = fmaf(ek8_0, r0_0_0_1, g8_1);
              g8_0 = fmaf(ek8_1, r0_0_0_1, g8_0);
              const float r0_0_1_0 = Y * b1;
              g8_2 = fmaf(ek8_0, r0_0_1_0, g8_2);
              const float r0_1_0_0 = X * b1;
              g8_3 = fmaf(ek8_0, r0_1_0_0, g8_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g8_4 = fmaf(ek8_0, r0_0_0_2, g8_4);
              g8_1 = fmaf(ek8_1, r0_0_0_2, g8_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g8_5 = fmaf(ek8_0, r0_0_1_1, g8_5);
              g8_2 = fmaf(ek8_1, r0_0_1_1, g8_2);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g8_6 = fmaf(ek8_0, r0_0_2_0, g8_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g8_7 = fmaf(ek8_0, r0_1_0_1, g8_7);
              g8_3 = fmaf(ek8_1, r0_1_0_1, g8_3);
              const float r0_1_1_0 = X * r1_0_1_0;
              g8_8 = fmaf(ek8_0, r0_1_1_0, g8_8);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g8_9 = fmaf(ek8_0, r0_2_0_0, g8_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g8_10 = fmaf(ek8_0, r0_0_0_3, g8_10);
              g8_4 = fmaf(ek8_1, r0_0_0_3, g8_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g8_11 = fmaf(ek8_0, r0_0_1_2, g8_11);
              g8_5 = fmaf(ek8_1, r0_0_1_2, g8_5);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g8_12 = fmaf(ek8_0, r0_0_2_1, g8_12);
              g8_6 = fmaf(ek8_1, r0_0_2_1, g8_6);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g8_13 = fmaf(ek8_0, r0_0_3_0, g8_13);
              const float r0_1_0_2 = X * r1_0_0_2;
              g8_14 = fmaf(ek8_0, r0_1_0_2, g8_14);
              g8_7 = fmaf(ek8_1, r0_1_0_2, g8_7);
              const float r0_1_1_1 = X * r1_0_1_1;
              g8_15 = fmaf(ek8_0, r0_1_1_1, g8_15);
              g8_8 = fmaf(ek8_1, r0_1_1_1, g8_8);
              const float r0_1_2_0 = X * r1_0_2_0;
              g8_16 = fmaf(ek8_0, r0_1_2_0, g8_16);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g8_17 = fmaf(ek8_0, r0_2_0_1, g8_17);
              g8_9 = fmaf(ek8_1, r0_2_0_1, g8_9);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g8_18 = fmaf(ek8_0, r0_2_1_0, g8_18);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g8_19 = fmaf(ek8_0, r0_3_0_0, g8_19);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g8_20 = fmaf(ek8_0, r0_0_0_4, g8_20);
              g8_10 = fmaf(ek8_1, r0_0_0_4, g8_10);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g8_21 = fmaf(ek8_0, r0_0_1_3, g8_21);
              g8_11 = fmaf(ek8_1, r0_0_1_3, g8_11);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g8_22 = fmaf(ek8_0, r0_0_2_2, g8_22);
              g8_12 = fmaf(ek8_1, r0_0_2_2, g8_12);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g8_23 = fmaf(ek8_0, r0_0_3_1, g8_23);
              g8_13 = fmaf(ek8_1, r0_0_3_1, g8_13);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g8_24 = fmaf(ek8_0, r0_0_4_0, g8_24);
              const float r0_1_0_3 = X * r1_0_0_3;
              g8_25 = fmaf(ek8_0, r0_1_0_3, g8_25);
              g8_14 = fmaf(ek8_1, r0_1_0_3, g8_14);
              const float r0_1_1_2 = X * r1_0_1_2;
              g8_26 = fmaf(ek8_0, r0_1_1_2, g8_26);
              g8_15 = fmaf(ek8_1, r0_1_1_2, g8_15);
              const float r0_1_2_1 = X * r1_0_2_1;
              g8_27 = fmaf(ek8_0, r0_1_2_1, g8_27);
              g8_16 = fmaf(ek8_1, r0_1_2_1, g8_16);
              const float r0_1_3_0 = X * r1_0_3_0;
              g8_28 = fmaf(ek8_0, r0_1_3_0, g8_28);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g8_29 = fmaf(ek8_0, r0_2_0_2, g8_29);
              g8_17 = fmaf(ek8_1, r0_2_0_2, g8_17);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g8_30 = fmaf(ek8_0, r0_2_1_1, g8_30);
              g8_18 = fmaf(ek8_1, r0_2_1_1, g8_18);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g8_31 = fmaf(ek8_0, r0_2_2_0, g8_31);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g8_32 = fmaf(ek8_0, r0_3_0_1, g8_32);
              g8_19 = fmaf(ek8_1, r0_3_0_1, g8_19);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g8_33 = fmaf(ek8_0, r0_3_1_0, g8_33);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g8_34 = fmaf(ek8_0, r0_4_0_0, g8_34);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_0_5 = fmaf(Z, r1_0_0_4, 4.0f * r1_0_0_3);
              g8_20 = fmaf(ek8_1, r0_0_0_5, g8_20);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g8_21 = fmaf(ek8_1, r0_0_1_4, g8_21);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g8_22 = fmaf(ek8_1, r0_0_2_3, g8_22);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g8_23 = fmaf(ek8_1, r0_0_3_2, g8_23);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g8_24 = fmaf(ek8_1, r0_0_4_1, g8_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g8_25 = fmaf(ek8_1, r0_1_0_4, g8_25);
              const float r0_1_1_3 = X * r1_0_1_3;
              g8_26 = fmaf(ek8_1, r0_1_1_3, g8_26);
              const float r0_1_2_2 = X * r1_0_2_2;
              g8_27 = fmaf(ek8_1, r0_1_2_2, g8_27);
              const float r0_1_3_1 = X * r1_0_3_1;
              g8_28 = fmaf(ek8_1, r0_1_3_1, g8_28);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g8_29 = fmaf(ek8_1, r0_2_0_3, g8_29);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g8_30 = fmaf(ek8_1, r0_2_1_2, g8_30);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g8_31 = fmaf(ek8_1, r0_2_2_1, g8_31);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g8_32 = fmaf(ek8_1, r0_3_0_2, g8_32);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g8_33 = fmaf(ek8_1, r0_3_1_1, g8_33);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g8_34 = fmaf(ek8_1, r0_4_0_1, g8_34);
            }
            { const float eb = bi[5];
              o0_8 = fmaf(eb, g8_0, o0_8);
            }
            { const float eb = bi[6];
              o0_8 = fmaf(eb, g8_3, o0_8);
            }
            { const float eb = bi[7];
              o0_8 = fmaf(eb, g8_9, o0_8);
            }
            { const float eb = bi[8];
              o0_8 = fmaf(eb, g8_19, o0_8);
            }
            { const float eb = bi[9];
              o0_8 = fmaf(eb, g8_34, o0_8);
            }
            { const float eb = bi[10];
              o1_8 = fmaf(eb, g8_0, o1_8);
            }
            { const float eb = bi[11];
              o1_8 = fmaf(eb, g8_2, o1_8);
            }
            { const float eb = bi[12];
              o1_8 = fmaf(eb, g8_6, o1_8);
            }
            { const float eb = bi[13];
              o1_8 = fmaf(eb, g8_3, o1_8);
            }
            { const float eb = bi[14];
              o1_8 = fmaf(eb, g8_8, o1_8);
            }
            { const float eb = bi[15];
              o1_8 = fmaf(eb, g8_16, o1_8);
            }
            { const float eb = bi[16];
              o1_8 = fmaf(eb, g8_9, o1_8);
            }
            { const float eb = bi[17];
              o1_8 = fmaf(eb, g8_18, o1_8);
            }
            { const float eb = bi[18];
              o1_8 = fmaf(eb, g8_31, o1_8);
            }
            { const float eb = bi[19];
              o2_8 = fmaf(eb, g8_0, o2_8);
            }
            { const float eb = bi[20];
              o2_8 = fmaf(eb, g8_1, o2_8);
            }
            { const float eb = bi[21];
              o2_8 = fmaf(eb, g8_4, o2_8);
            }
            { const float eb = bi[22];
              o2_8 = fmaf(eb, g8_3, o2_8);
            }
            { const float eb = bi[23];
              o2_8 = fmaf(eb, g8_7, o2_8);
            }
            { const float eb = bi[24];
              o2_8 = fmaf(eb, g8_14, o2_8);
            }
            { const float eb = bi[25];
              o2_8 = fmaf(eb, g8_9, o2_8);
            }
            { const float eb = bi[26];
              o2_8 = fmaf(eb, g8_17, o2_8);
            }
            { const float eb = bi[27];
              o2_8 = fmaf(eb, g8_29, o2_8);
            }
            { const float eb = bi[28];
              o3_8 = fmaf(eb, g8_0, o3_8);
            }
            { const float eb = bi[29];
              o3_8 = fmaf(eb, g8_2, o3_8);
            }
            { const float eb = bi[30];
              o3_8 = fmaf(eb, g8_3, o3_8);
            }
            { const float eb = bi[31];
              o3_8 = fmaf(eb, g8_8, o3_8);
            }
            { const float eb = bi[32];
              o3_8 = fmaf(eb, g8_9, o3_8);
            }
            { const float eb = bi[33];
              o3_8 = fmaf(eb, g8_18, o3_8);
            }
            { const float eb = bi[34];
              o3_8 = fmaf(eb, g8_19, o3_8);
            }
            { const float eb = bi[35];
              o3_8 = fmaf(eb, g8_33, o3_8);
            }
            { const float eb = bi[36];
              o4_8 = fmaf(eb, g8_0, o4_8);
            }
            { const float eb = bi[37];
              o4_8 = fmaf(eb, g8_1, o4_8);
            }
            { const float eb = bi[38];
              o4_8 = fmaf(eb, g8_3, o4_8);
            }
            { const float eb = bi[39];
              o4_8 = fmaf(eb, g8_7, o4_8);
            }
            { const float eb = bi[40];
              o4_8 = fmaf(eb, g8_9, o4_8);
            }
            { const float eb = bi[41];
              o4_8 = fmaf(eb, g8_17, o4_8);
            }
            { const float eb = bi[42];
              o4_8 = fmaf(eb, g8_19, o4_8);
            }
            { const float eb = bi[43];
              o4_8 = fmaf(eb, g8_32, o4_8);
            }
            { const float eb = bi[44];
              o5_8 = fmaf(eb, g8_0, o5_8);
            }
            { const float eb = bi[45];
              o5_8 = fmaf(eb, g8_1, o5_8);
            }
            { const float eb = bi[46];
              o5_8 = fmaf(eb, g8_2, o5_8);
            }
            { const float eb = bi[47];
              o5_8 = fmaf(eb, g8_5, o5_8);
            }
            { const float eb = bi[48];
              o5_8 = fmaf(eb, g8_3, o5_8);
            }
            { const float eb = bi[49];
              o5_8 = fmaf(eb, g8_7, o5_8);
            }
            { const float eb = bi[50];
              o5_8 = fmaf(eb, g8_8, o5_8);
            }
            { const float eb = bi[51];
              o5_8 = fmaf(eb, g8_15, o5_8);
            }
            { const float eb = bi[52];
              o5_8 = fmaf(eb, g8_9, o5_8);
            }
            { const float eb = bi[53];
              o5_8 = fmaf(eb, g8_17, o5_8);
            }
            { const float eb = bi[54];
              o5_8 = fmaf(eb, g8_18, o5_8);
            }
            { const float eb = bi[55];
              o5_8 = fmaf(eb, g8_30, o5_8);
            }
            { const float eb = bi[56];
              o6_8 = fmaf(eb, g8_0, o6_8);
            }
            { const float eb = bi[57];
              o6_8 = fmaf(eb, g8_2, o6_8);
            }
            { const float eb = bi[58];
              o6_8 = fmaf(eb, g8_6, o6_8);
            }
            { const float eb = bi[59];
              o6_8 = fmaf(eb, g8_3, o6_8);
            }
            { const float eb = bi[60];
              o6_8 = fmaf(eb, g8_8, o6_8);
            }
            { const float eb = bi[61];
              o6_8 = fmaf(eb, g8_16, o6_8);
            }
            { const float eb = bi[62];
              o6_8 = fmaf(eb, g8_9, o6_8);
            }
            { const float eb = bi[63];
              o6_8 = fmaf(eb, g8_18, o6_8);
            }
            { const float eb = bi[64];
              o6_8 = fmaf(eb, g8_31, o6_8);
            }
            { const float eb = bi[65];
              o7_8 = fmaf(eb, g8_0, o7_8);
            }
            { const float eb = bi[66];
              o7_8 = fmaf(eb, g8_2, o7_8);
            }
            { const float eb = bi[67];
              o7_8 = fmaf(eb, g8_6, o7_8);
            }
            { const float eb = bi[68];
              o7_8 = fmaf(eb, g8_13, o7_8);
            }
            { const float eb = bi[69];
              o7_8 = fmaf(eb, g8_24, o7_8);
            }
            { const float eb = bi[70];
              o8_8 = fmaf(eb, g8_0, o8_8);
            }
            { const float eb = bi[71];
              o8_8 = fmaf(eb, g8_1, o8_8);
            }
            { const float eb = bi[72];
              o8_8 = fmaf(eb, g8_4, o8_8);
            }
            { const float eb = bi[73];
              o8_8 = fmaf(eb, g8_2, o8_8);
            }
            { const float eb = bi[74];
              o8_8 = fmaf(eb, g8_5, o8_8);
            }
            { const float eb = bi[75];
              o8_8 = fmaf(eb, g8_11, o8_8);
            }
            { const float eb = bi[76];
              o8_8 = fmaf(eb, g8_6, o8_8);
            }
            { const float eb = bi[77];
              o8_8 = fmaf(eb, g8_12, o8_8);
            }
            { const float eb = bi[78];
              o8_8 = fmaf(eb, g8_22, o8_8);
            }
            { const float eb = bi[79];
              o9_8 = fmaf(eb, g8_0, o9_8);
            }
            { const float eb = bi[80];
              o9_8 = fmaf(eb, g8_2, o9_8);
            }
            { const float eb = bi[81];
              o9_8 = fmaf(eb, g8_6, o9_8);
            }
            { const float eb = bi[82];
              o9_8 = fmaf(eb, g8_13, o9_8);
            }
            { const float eb = bi[83];
              o9_8 = fmaf(eb, g8_3, o9_8);
            }
            { const float eb = bi[84];
              o9_8 = fmaf(eb, g8_8, o9_8);
            }
            { const float eb = bi[85];
              o9_8 = fmaf(eb, g8_16, o9_8);
            }
            { const float eb = bi[86];
              o9_8 = fmaf(eb, g8_28, o9_8);
            }
            { const float eb = bi[87];
              o10_8 = fmaf(eb, g8_0, o10_8);
            }
            { const float eb = bi[88];
              o10_8 = fmaf(eb, g8_1, o10_8);
            }
            { const float eb = bi[89];
              o10_8 = fmaf(eb, g8_2, o10_8);
            }
            { const float eb = bi[90];
              o10_8 = fmaf(eb, g8_5, o10_8);
            }
            { const float eb = bi[91];
              o10_8 = fmaf(eb, g8_6, o10_8);
            }
            { const float eb = bi[92];
              o10_8 = fmaf(eb, g8_12, o10_8);
            }
            { const float eb = bi[93];
              o10_8 = fmaf(eb, g8_3, o10_8);
            }
            { const float eb = bi[94];
              o10_8 = fmaf(eb, g8_7, o10_8);
            }
            { const float eb = bi[95];
              o10_8 = fmaf(eb, g8_8, o10_8);
            }
            { const float eb = bi[96];
              o10_8 = fmaf(eb, g8_15, o10_8);
            }
            { const float eb = bi[97];
              o10_8 = fmaf(eb, g8_16, o10_8);
            }
            { const float eb = bi[98];
              o10_8 = fmaf(eb, g8_27, o10_8);
            }
            { const float eb = bi[99];
              o11_8 = fmaf(eb, g8_0, o11_8);
            }
            { const float eb = bi[100];
              o11_8 = fmaf(eb, g8_1, o11_8);
            }
            { const float eb = bi[101];
              o11_8 = fmaf(eb, g8_2, o11_8);
            }
            { const float eb = bi[102];
              o11_8 = fmaf(eb, g8_5, o11_8);
            }
            { const float eb = bi[103];
              o11_8 = fmaf(eb, g8_6, o11_8);
            }
            { const float eb = bi[104];
              o11_8 = fmaf(eb, g8_12, o11_8);
            }
            { const float eb = bi[105];
              o11_8 = fmaf(eb, g8_13, o11_8);
            }
            { const float eb = bi[106];
              o11_8 = fmaf(eb, g8_23, o11_8);
            }
            { const float eb = bi[107];
              o12_8 = fmaf(eb, g8_0, o12_8);
            }
            { const float eb = bi[108];
              o12_8 = fmaf(eb, g8_1, o12_8);
            }
            { const float eb = bi[109];
              o12_8 = fmaf(eb, g8_4, o12_8);
            }
            { const float eb = bi[110];
              o12_8 = fmaf(eb, g8_3, o12_8);
            }
            { const float eb = bi[111];
              o12_8 = fmaf(eb, g8_7, o12_8);
            }
            { const float eb = bi[112];
              o12_8 = fmaf(eb, g8_14, o12_8);
            }
            { const float eb = bi[113];
              o12_8 = fmaf(eb, g8_9, o12_8);
            }
            { const float eb = bi[114];
              o12_8 = fmaf(eb, g8_17, o12_8);
            }
            { const float eb = bi[115];
              o12_8 = fmaf(eb, g8_29, o12_8);
            }
            { const float eb = bi[116];
              o13_8 = fmaf(eb, g8_0, o13_8);
            }
            { const float eb = bi[117];
              o13_8 = fmaf(eb, g8_1, o13_8);
            }
            { const float eb = bi[118];
              o13_8 = fmaf(eb, g8_4, o13_8);
            }
            { const float eb = bi[119];
              o13_8 = fmaf(eb, g8_2, o13_8);
            }
            { const float eb = bi[120];
              o13_8 = fmaf(eb, g8_5, o13_8);
            }
            { const float eb = bi[121];
              o13_8 = fmaf(eb, g8_11, o13_8);
            }
            { const float eb = bi[122];
              o13_8 = fmaf(eb, g8_6, o13_8);
            }
            { const float eb = bi[123];
              o13_8 = fmaf(eb, g8_12, o13_8);
            }
            { const float eb = bi[124];
              o13_8 = fmaf(eb, g8_22, o13_8);
            }
            { const float eb = bi[125];
              o14_8 = fmaf(eb, g8_0, o14_8);
            }
            { const float eb = bi[126];
              o14_8 = fmaf(eb, g8_1, o14_8);
            }
            { const float eb = bi[127];
              o14_8 = fmaf(eb, g8_4, o14_8);
            }
            { const float eb = bi[128];
              o14_8 = fmaf(eb, g8_10, o14_8);
            }
            { const float eb = bi[129];
              o14_8 = fmaf(eb, g8_20, o14_8);
            }
            { const float eb = bi[130];
              o15_8 = fmaf(eb, g8_0, o15_8);
            }
            { const float eb = bi[131];
              o15_8 = fmaf(eb, g8_1, o15_8);
            }
            { const float eb = bi[132];
              o15_8 = fmaf(eb, g8_4, o15_8);
            }
            { const float eb = bi[133];
              o15_8 = fmaf(eb, g8_2, o15_8);
            }
            { const float eb = bi[134];
              o15_8 = fmaf(eb, g8_5, o15_8);
            }
            { const float eb = bi[135];
              o15_8 = fmaf(eb, g8_11, o15_8);
            }
            { const float eb = bi[136];
              o15_8 = fmaf(eb, g8_3, o15_8);
            }
            { const float eb = bi[137];
              o15_8 = fmaf(eb, g8_7, o15_8);
            }
            { const float eb = bi[138];
              o15_8 = fmaf(eb, g8_14, o15_8);
            }
            { const float eb = bi[139];
              o15_8 = fmaf(eb, g8_8, o15_8);
            }
            { const float eb = bi[140];
              o15_8 = fmaf(eb, g8_15, o15_8);
            }
            { const float eb = bi[141];
              o15_8 = fmaf(eb, g8_26, o15_8);
            }
            { const float eb = bi[142];
              o16_8 = fmaf(eb, g8_0, o16_8);
            }
            { const float eb = bi[143];
              o16_8 = fmaf(eb, g8_1, o16_8);
            }
            { const float eb = bi[144];
              o16_8 = fmaf(eb, g8_4, o16_8);
            }
            { const float eb = bi[145];
              o16_8 = fmaf(eb, g8_10, o16_8);
            }
            { const float eb = bi[146];
              o16_8 = fmaf(eb, g8_3, o16_8);
            }
            { const float eb = bi[147];
              o16_8 = fmaf(eb, g8_7, o16_8);
            }
            { const float eb = bi[148];
              o16_8 = fmaf(eb, g8_14, o16_8);
            }
            { const float eb = bi[149];
              o16_8 = fmaf(eb, g8_25, o16_8);
            }
            { const float eb = bi[150];
              o17_8 = fmaf(eb, g8_0, o17_8);
            }
            { const float eb = bi[151];
              o17_8 = fmaf(eb, g8_1, o17_8);
            }
            { const float eb = bi[152];
              o17_8 = fmaf(eb, g8_4, o17_8);
            }
            { const float eb = bi[153];
              o17_8 = fmaf(eb, g8_10, o17_8);
            }
            { const float eb = bi[154];
              o17_8 = fmaf(eb, g8_2, o17_8);
            }
            { const float eb = bi[155];
              o17_8 = fmaf(eb, g8_5, o17_8);
            }
            { const float eb = bi[156];
              o17_8 = fmaf(eb, g8_11, o17_8);
            }
            { const float eb = bi[157];
              o17_8 = fmaf(eb, g8_21, o17_8);
            }
            { const float eb = bi[158];
              o18_8 = fmaf(eb, g8_0, o18_8);
            }
            { const float eb = bi[159];
              o18_8 = fmaf(eb, g8_2, o18_8);
            }
            { const float eb = bi[160];
              o18_8 = fmaf(eb, g8_3, o18_8);
            }
            { const float eb = bi[161];
              o18_8 = fmaf(eb, g8_8, o18_8);
            }
            { const float eb = bi[162];
              o18_8 = fmaf(eb, g8_9, o18_8);
            }
            { const float eb = bi[163];
              o18_8 = fmaf(eb, g8_18, o18_8);
            }
            { const float eb = bi[164];
              o18_8 = fmaf(eb, g8_19, o18_8);
            }
            { const float eb = bi[165];
              o18_8 = fmaf(eb, g8_33, o18_8);
            }
            { const float eb = bi[166];
              o19_8 = fmaf(eb, g8_0, o19_8);
            }
            { const float eb = bi[167];
              o19_8 = fmaf(eb, g8_2, o19_8);
            }
            { const float eb = bi[168];
              o19_8 = fmaf(eb, g8_6, o19_8);
            }
            { const float eb = bi[169];
              o19_8 = fmaf(eb, g8_13, o19_8);
            }
            { const float eb = bi[170];
              o19_8 = fmaf(eb, g8_3, o19_8);
            }
            { const float eb = bi[171];
              o19_8 = fmaf(eb, g8_8, o19_8);
            }
            { const float eb = bi[172];
              o19_8 = fmaf(eb, g8_16, o19_8);
            }
            { const float eb = bi[173];
              o19_8 = fmaf(eb, g8_28, o19_8);
            }
            { const float eb = bi[174];
              o20_8 = fmaf(eb, g8_0, o20_8);
            }
            { const float eb = bi[175];
              o20_8 = fmaf(eb, g8_1, o20_8);
            }
            { const float eb = bi[176];
              o20_8 = fmaf(eb, g8_4, o20_8);
            }
            { const float eb = bi[177];
              o20_8 = fmaf(eb, g8_2, o20_8);
            }
            { const float eb = bi[178];
              o20_8 = fmaf(eb, g8_5, o20_8);
            }
            { const float eb = bi[179];
              o20_8 = fmaf(eb, g8_11, o20_8);
            }
            { const float eb = bi[180];
              o20_8 = fmaf(eb, g8_3, o20_8);
            }
            { const float eb = bi[181];
              o20_8 = fmaf(eb, g8_7, o20_8);
            }
            { const float eb = bi[182];
              o20_8 = fmaf(eb, g8_14, o20_8);
            }
            { const float eb = bi[183];
              o20_8 = fmaf(eb, g8_8, o20_8);
            }
            { const float eb = bi[184];
              o20_8 = fmaf(eb, g8_15, o20_8);
            }
            { const float eb = bi[185];
              o20_8 = fmaf(eb, g8_26, o20_8);
            }
            { const float eb = bi[186];
              o21_8 = fmaf(eb, g8_0, o21_8);
            }
            { const float eb = bi[187];
              o21_8 = fmaf(eb, g8_2, o21_8);
            }
            { const float eb = bi[188];
              o21_8 = fmaf(eb, g8_6, o21_8);
            }
            { const float eb = bi[189];
              o21_8 = fmaf(eb, g8_3, o21_8);
            }
            { const float eb = bi[190];
              o21_8 = fmaf(eb, g8_8, o21_8);
            }
            { const float eb = bi[191];
              o21_8 = fmaf(eb, g8_16, o21_8);
            }
            { const float eb = bi[192];
              o21_8 = fmaf(eb, g8_9, o21_8);
            }
            { const float eb = bi[193];
              o21_8 = fmaf(eb, g8_18, o21_8);
            }
            { const float eb = bi[194];
              o21_8 = fmaf(eb, g8_31, o21_8);
            }
            { const float eb = bi[195];
              o22_8 = fmaf(eb, g8_0, o22_8);
            }
            { const float eb = bi[196];
              o22_8 = fmaf(eb, g8_1, o22_8);
            }
            { const float eb = bi[197];
              o22_8 = fmaf(eb, g8_2, o22_8);
            }
            { const float eb = bi[198];
              o22_8 = fmaf(eb, g8_5, o22_8);
            }
            { const float eb = bi[199];
              o22_8 = fmaf(eb, g8_3, o22_8);
            }
            { const float eb = bi[200];
              o22_8 = fmaf(eb, g8_7, o22_8);
            }
            { const float eb = bi[201];
              o22_8 = fmaf(eb, g8_8, o22_8);
            }
            { const float eb = bi[202];
              o22_8 = fmaf(eb, g8_15, o22_8);
            }
            { const float eb = bi[203];
              o22_8 = fmaf(eb, g8_9, o22_8);
            }
            { const float eb = bi[204];
              o22_8 = fmaf(eb, g8_17, o22_8);
            }
            { const float eb = bi[205];
              o22_8 = fmaf(eb, g8_18, o22_8);
            }
            { const float eb = bi[206];
              o22_8 = fmaf(eb, g8_30, o22_8);
            }
            { const float eb = bi[207];
              o23_8 = fmaf(eb, g8_0, o23_8);
            }
            { const float eb = bi[208];
              o23_8 = fmaf(eb, g8_1, o23_8);
            }
            { const float eb = bi[209];
              o23_8 = fmaf(eb, g8_2, o23_8);
            }
            { const float eb = bi[210];
              o23_8 = fmaf(eb, g8_5, o23_8);
            }
            { const float eb = bi[211];
              o23_8 = fmaf(eb, g8_6, o23_8);
            }
            { const float eb = bi[212];
              o23_8 = fmaf(eb, g8_12, o23_8);
            }
            { const float eb = bi[213];
              o23_8 = fmaf(eb, g8_3, o23_8);
            }
            { const float eb = bi[214];
              o23_8 = fmaf(eb, g8_7, o23_8);
            }
            { const float eb = bi[215];
              o23_8 = fmaf(eb, g8_8, o23_8);
            }
            { const float eb = bi[216];
              o23_8 = fmaf(eb, g8_15, o23_8);
            }
            { const float eb = bi[217];
              o23_8 = fmaf(eb, g8_16, o23_8);
            }
            { const float eb = bi[218];
              o23_8 = fmaf(eb, g8_27, o23_8);
            }
            { const float eb = bi[219];
              o24_8 = fmaf(eb, g8_0, o24_8);
            }
            { const float eb = bi[220];
              o24_8 = fmaf(eb, g8_1, o24_8);
            }
            { const float eb = bi[221];
              o24_8 = fmaf(eb, g8_3, o24_8);
            }
            { const float eb = bi[222];
              o24_8 = fmaf(eb, g8_7, o24_8);
            }
            { const float eb = bi[223];
              o24_8 = fmaf(eb, g8_9, o24_8);
            }
            { const float eb = bi[224];
              o24_8 = fmaf(eb, g8_17, o24_8);
            }
            { const float eb = bi[225];
              o24_8 = fmaf(eb, g8_19, o24_8);
            }
            { const float eb = bi[226];
              o24_8 = fmaf(eb, g8_32, o24_8);
            }
            { const float eb = bi[227];
              o25_8 = fmaf(eb, g8_0, o25_8);
            }
            { const float eb = bi[228];
              o25_8 = fmaf(eb, g8_1, o25_8);
            }
            { const float eb = bi[229];
              o25_8 = fmaf(eb, g8_2, o25_8);
            }
            { const float eb = bi[230];
              o25_8 = fmaf(eb, g8_5, o25_8);
            }
            { const float eb = bi[231];
              o25_8 = fmaf(eb, g8_6, o25_8);
            }
            { const float eb = bi[232];
              o25_8 = fmaf(eb, g8_12, o25_8);
            }
            { const float eb = bi[233];
              o25_8 = fmaf(eb, g8_3, o25_8);
            }
            { const float eb = bi[234];
              o25_8 = fmaf(eb, g8_7, o25_8);
            }
            { const float eb = bi[235];
              o25_8 = fmaf(eb, g8_8, o25_8);
            }
            { const float eb = bi[236];
              o25_8 = fmaf(eb, g8_15, o25_8);
            }
            { const float eb = bi[237];
              o25_8 = fmaf(eb, g8_16, o25_8);
            }
            { const float eb = bi[238];
              o25_8 = fmaf(eb, g8_27, o25_8);
            }
            { const float eb = bi[239];
              o26_8 = fmaf(eb, g8_0, o26_8);
            }
            { const float eb = bi[240];
              o26_8 = fmaf(eb, g8_1, o26_8);
            }
            { const float eb = bi[241];
              o26_8 = fmaf(eb, g8_4, o26_8);
            }
            { const float eb = bi[242];
              o26_8 = fmaf(eb, g8_10, o26_8);
            }
            { const float eb = bi[243];
              o26_8 = fmaf(eb, g8_3, o26_8);
            }
            { const float eb = bi[244];
              o26_8 = fmaf(eb, g8_7, o26_8);
            }
            { const float eb = bi[245];
              o26_8 = fmaf(eb, g8_14, o26_8);
            }
            { const float eb = bi[246];
              o26_8 = fmaf(eb, g8_25, o26_8);
            }
            { const float eb = bi[247];
              o27_8 = fmaf(eb, g8_0, o27_8);
            }
            { const float eb = bi[248];
              o27_8 = fmaf(eb, g8_1, o27_8);
            }
            { const float eb = bi[249];
              o27_8 = fmaf(eb, g8_2, o27_8);
            }
            { const float eb = bi[250];
              o27_8 = fmaf(eb, g8_5, o27_8);
            }
            { const float eb = bi[251];
              o27_8 = fmaf(eb, g8_3, o27_8);
            }
            { const float eb = bi[252];
              o27_8 = fmaf(eb, g8_7, o27_8);
            }
            { const float eb = bi[253];
              o27_8 = fmaf(eb, g8_8, o27_8);
            }
            { const float eb = bi[254];
              o27_8 = fmaf(eb, g8_15, o27_8);
            }
            { const float eb = bi[255];
              o27_8 = fmaf(eb, g8_9, o27_8);
            }
            { const float eb = bi[256];
              o27_8 = fmaf(eb, g8_17, o27_8);
            }
            { const float eb = bi[257];
              o27_8 = fmaf(eb, g8_18, o27_8);
            }
            { const float eb = bi[258];
              o27_8 = fmaf(eb, g8_30, o27_8);
            }
            { const float eb = bi[259];
              o28_8 = fmaf(eb, g8_0, o28_8);
            }
            { const float eb = bi[260];
              o28_8 = fmaf(eb, g8_1, o28_8);
            }
            { const float eb = bi[261];
              o28_8 = fmaf(eb, g8_4, o28_8);
            }
            { const float eb = bi[262];
              o28_8 = fmaf(eb, g8_3, o28_8);
            }
            { const float eb = bi[263];
              o28_8 = fmaf(eb, g8_7, o28_8);
            }
            { const float eb = bi[264];
              o28_8 = fmaf(eb, g8_14, o28_8);
            }
            { const float eb = bi[265];
              o28_8 = fmaf(eb, g8_9, o28_8);
            }
            { const float eb = bi[266];
              o28_8 = fmaf(eb, g8_17, o28_8);
            }
            { const float eb = bi[267];
              o28_8 = fmaf(eb, g8_29, o28_8);
            }
            { const float eb = bi[268];
              o29_8 = fmaf(eb, g8_0, o29_8);
            }
            { const float eb = bi[269];
              o29_8 = fmaf(eb, g8_1, o29_8);
            }
            { const float eb = bi[270];
              o29_8 = fmaf(eb, g8_4, o29_8);
            }
            { const float eb = bi[271];
              o29_8 = fmaf(eb, g8_2, o29_8);
            }
            { const float eb = bi[272];
              o29_8 = fmaf(eb, g8_5, o29_8);
            }
            { const float eb = bi[273];
              o29_8 = fmaf(eb, g8_11, o29_8);
            }
            { const float eb = bi[274];
              o29_8 = fmaf(eb, g8_3, o29_8);
            }
            { const float eb = bi[275];
              o29_8 = fmaf(eb, g8_7, o29_8);
            }
            { const float eb = bi[276];
              o29_8 = fmaf(eb, g8_14, o29_8);
            }
            { const float eb = bi[277];
              o29_8 = fmaf(eb, g8_8, o29_8);
            }
            { const float eb = bi[278];
              o29_8 = fmaf(eb, g8_15, o29_8);
            }
            { const float eb = bi[279];
              o29_8 = fmaf(eb, g8_26, o29_8);
            }
            { const float eb = bi[280];
              o30_8 = fmaf(eb, g8_0, o30_8);
            }
            { const float eb = bi[281];
              o30_8 = fmaf(eb, g8_1, o30_8);
            }
            { const float eb = bi[282];
              o30_8 = fmaf(eb, g8_2, o30_8);
            }
            { const float eb = bi[283];
              o30_8 = fmaf(eb, g8_5, o30_8);
            }
            { const float eb = bi[284];
              o30_8 = fmaf(eb, g8_3, o30_8);
            }
            { const float eb = bi[285];
              o30_8 = fmaf(eb, g8_7, o30_8);
            }
            { const float eb = bi[286];
              o30_8 = fmaf(eb, g8_8, o30_8);
            }
            { const float eb = bi[287];
              o30_8 = fmaf(eb, g8_15, o30_8);
            }
            { const float eb = bi[288];
              o30_8 = fmaf(eb, g8_9, o30_8);
            }
            { const float eb = bi[289];
              o30_8 = fmaf(eb, g8_17, o30_8);
            }
            { const float eb = bi[290];
              o30_8 = fmaf(eb, g8_18, o30_8);
            }
            { const float eb = bi[291];
              o30_8 = fmaf(eb, g8_30, o30_8);
            }
            { const float eb = bi[292];
              o31_8 = fmaf(eb, g8_0, o31_8);
            }
            { const float eb = bi[293];
              o31_8 = fmaf(eb, g8_1, o31_8);
            }
            { const float eb = bi[294];
              o31_8 = fmaf(eb, g8_2, o31_8);
            }
            { const float eb = bi[295];
              o31_8 = fmaf(eb, g8_5, o31_8);
            }
            { const float eb = bi[296];
              o31_8 = fmaf(eb, g8_6, o31_8);
            }
            { const float eb = bi[297];
              o31_8 = fmaf(eb, g8_12, o31_8);
            }
            { const float eb = bi[298];
              o31_8 = fmaf(eb, g8_13, o31_8);
            }
            { const float eb = bi[299];
              o31_8 = fmaf(eb, g8_23, o31_8);
            }
            { const float eb = bi[300];
              o32_8 = fmaf(eb, g8_0, o32_8);
            }
            { const float eb = bi[301];
              o32_8 = fmaf(eb, g8_1, o32_8);
            }
            { const float eb = bi[302];
              o32_8 = fmaf(eb, g8_4, o32_8);
            }
            { const float eb = bi[303];
              o32_8 = fmaf(eb, g8_10, o32_8);
            }
            { const float eb = bi[304];
              o32_8 = fmaf(eb, g8_2, o32_8);
            }
            { const float eb = bi[305];
              o32_8 = fmaf(eb, g8_5, o32_8);
            }
            { const float eb = bi[306];
              o32_8 = fmaf(eb, g8_11, o32_8);
            }
            { const float eb = bi[307];
              o32_8 = fmaf(eb, g8_21, o32_8);
            }
            { const float eb = bi[308];
              o33_8 = fmaf(eb, g8_0, o33_8);
            }
            { const float eb = bi[309];
              o33_8 = fmaf(eb, g8_1, o33_8);
            }
            { const float eb = bi[310];
              o33_8 = fmaf(eb, g8_2, o33_8);
            }
            { const float eb = bi[311];
              o33_8 = fmaf(eb, g8_5, o33_8);
            }
            { const float eb = bi[312];
              o33_8 = fmaf(eb, g8_6, o33_8);
            }
            { const float eb = bi[313];
              o33_8 = fmaf(eb, g8_12, o33_8);
            }
            { const float eb = bi[314];
              o33_8 = fmaf(eb, g8_3, o33_8);
            }
            { const float eb = bi[315];
              o33_8 = fmaf(eb, g8_7, o33_8);
            }
            { const float eb = bi[316];
              o33_8 = fmaf(eb, g8_8, o33_8);
            }
            { const float eb = bi[317];
              o33_8 = fmaf(eb, g8_15, o33_8);
            }
            { const float eb = bi[318];
              o33_8 = fmaf(eb, g8_16, o33_8);
            }
            { const float eb = bi[319];
              o33_8 = fmaf(eb, g8_27, o33_8);
            }
            { const float eb = bi[320];
              o34_8 = fmaf(eb, g8_0, o34_8);
            }
            { const float eb = bi[321];
              o34_8 = fmaf(eb, g8_1, o34_8);
            }
            { const float eb = bi[322];
              o34_8 = fmaf(eb, g8_4, o34_8);
            }
            { const float eb = bi[323];
              o34_8 = fmaf(eb, g8_2, o34_8);
            }
            { const float eb = bi[324];
              o34_8 = fmaf(eb, g8_5, o34_8);
            }
            { const float eb = bi[325];
              o34_8 = fmaf(eb, g8_11, o34_8);
            }
            { const float eb = bi[326];
              o34_8 = fmaf(eb, g8_3, o34_8);
            }
            { const float eb = bi[327];
              o34_8 = fmaf(eb, g8_7, o34_8);
            }
            { const float eb = bi[328];
              o34_8 = fmaf(eb, g8_14, o34_8);
            }
            { const float eb = bi[329];
              o34_8 = fmaf(eb, g8_8, o34_8);
            }
            { const float eb = bi[330];
              o34_8 = fmaf(eb, g8_15, o34_8);
            }
            { const float eb = bi[331];
              o34_8 = fmaf(eb, g8_26, o34_8);
            }
            { const float eb = bi[332];
              o35_8 = fmaf(eb, g8_0, o35_8);
            }
            { const float eb = bi[333];
              o35_8 = fmaf(eb, g8_1, o35_8);
            }
            { const float eb = bi[334];
              o35_8 = fmaf(eb, g8_4, o35_8);
            }
            { const float eb = bi[335];
              o35_8 = fmaf(eb, g8_2, o35_8);
            }
            { const float eb = bi[336];
              o35_8 = fmaf(eb, g8_5, o35_8);
            }
            { const float eb = bi[337];
              o35_8 = fmaf(eb, g8_11, o35_8);
            }
            { const float eb = bi[338];
              o35_8 = fmaf(eb, g8_6, o35_8);
            }
            { const float eb = bi[339];
              o35_8 = fmaf(eb, g8_12, o35_8);
            }
            { const float eb = bi[340];
              o35_8 = fmaf(eb, g8_22, o35_8);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk8 = PT[(fI + 2) * N + fJ + 0];
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
            jab24 += o24_8 * ptk8;
            jab25 += o25_8 * ptk8;
            jab26 += o26_8 * ptk8;
            jab27 += o27_8 * ptk8;
            jab28 += o28_8 * ptk8;
            jab29 += o29_8 * ptk8;
            jab30 += o30_8 * ptk8;
            jab31 += o31_8 * ptk8;
            jab32 += o32_8 * ptk8;
            jab33 += o33_8 * ptk8;
            jab34 += o34_8 * ptk8;
            jab35 += o35_8 * ptk8;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_8 * ptb0 + o1_8 * ptb1 + o2_8 * ptb2 + o3_8 * ptb3 + o4_8 * ptb4 + o5_8 * ptb5 + o6_8 * ptb6 + o7_8 * ptb7 + o8_8 * ptb8 + o9_8 * ptb9 + o10_8 * ptb10 + o11_8 * ptb11 + o12_8 * ptb12 + o13_8 * ptb13 + o14_8 * ptb14 + o15_8 * ptb15 + o16_8 * ptb16 + o17_8 * ptb17 + o18_8 * ptb18 + o19_8 * ptb19 + o20_8 * ptb20 + o21_8 * ptb21 + o22_8 * ptb22 + o23_8 * ptb23 + o24_8 * ptb24 + o25_8 * ptb25 + o26_8 * ptb26 + o27_8 * ptb27 + o28_8 * ptb28 + o29_8 * ptb29 + o30_8 * ptb30 + o31_8 * ptb31 + o32_8 * ptb32 + o33_8 * ptb33 + o34_8 * ptb34 + o35_8 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_8 * Abd0_0 + o1_8 * Abd1_0 + o2_8 * Abd2_0 + o3_8 * Abd3_0 + o4_8 * Abd4_0 + o5_8 * Abd5_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_8 * Aad0_0 + o6_8 * Aad1_0 + o12_8 * Aad2_0 + o18_8 * Aad3_0 + o24_8 * Aad4_0 + o30_8 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_8 * Abc0_2 + o1_8 * Abc1_2 + o2_8 * Abc2_2 + o3_8 * Abc3_2 + o4_8 * Abc4_2 + o5_8 * Abc5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_8 * Aac0_2 + o6_8 * Aac1_2 + o12_8 * Aac2_2 + o18_8 * Aac3_2 + o24_8 * Aac4_2 + o30_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_8 * Aad0_0 + o7_8 * Aad1_0 + o13_8 * Aad2_0 + o19_8 * Aad3_0 + o25_8 * Aad4_0 + o31_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 0, deg * (o1_8 * Aac0_2 + o7_8 * Aac1_2 + o13_8 * Aac2_2 + o19_8 * Aac3_2 + o25_8 * Aac4_2 + o31_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_8 * Aad0_0 + o8_8 * Aad1_0 + o14_8 * Aad2_0 + o20_8 * Aad3_0 + o26_8 * Aad4_0 + o32_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 0, deg * (o2_8 * Aac0_2 + o8_8 * Aac1_2 + o14_8 * Aac2_2 + o20_8 * Aac3_2 + o26_8 * Aac4_2 + o32_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_8 * Aad0_0 + o9_8 * Aad1_0 + o15_8 * Aad2_0 + o21_8 * Aad3_0 + o27_8 * Aad4_0 + o33_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 0, deg * (o3_8 * Aac0_2 + o9_8 * Aac1_2 + o15_8 * Aac2_2 + o21_8 * Aac3_2 + o27_8 * Aac4_2 + o33_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 2, deg * (o4_8 * Aad0_0 + o10_8 * Aad1_0 + o16_8 * Aad2_0 + o22_8 * Aad3_0 + o28_8 * Aad4_0 + o34_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 0, deg * (o4_8 * Aac0_2 + o10_8 * Aac1_2 + o16_8 * Aac2_2 + o22_8 * Aac3_2 + o28_8 * Aac4_2 + o34_8 * Aac5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 2, deg * (o5_8 * Aad0_0 + o11_8 * Aad1_0 + o17_8 * Aad2_0 + o23_8 * Aad3_0 + o29_8 * Aad4_0 + o35_8 * Aad5_0));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 0, deg * (o5_8 * Aac0_2 + o11_8 * Aac1_2 + o17_8 * Aac2_2 + o23_8 * Aac3_2 + o29_8 * Aac4_2 + o35_8 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o6_8 * Abd0_0 + o7_8 * Abd1_0 + o8_8 * Abd2_0 + o9_8 * Abd3_0 + o10_8 * Abd4_0 + o11_8 * Abd5_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o6_8 * Abc0_2 + o7_8 * Abc1_2 + o8_8 * Abc2_2 + o9_8 * Abc3_2 + o10_8 * Abc4_2 + o11_8 * Abc5_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o12_8 * Abd0_0 + o13_8 * Abd1_0 + o14_8 * Abd2_0 + o15_8 * Abd3_0 + o16_8 * Abd4_0 + o17_8 * Abd5_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o12_8 * Abc0_2 + o13_8 * Abc1_2 + o14_8 * Abc2_2 + o15_8 * Abc3_2 + o16_8 * Abc4_2 + o17_8 * Abc5_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o18_8 * Abd0_0 + o19_8 * Abd1_0 + o20_8 * Abd2_0 + o21_8 * Abd3_0 + o22_8 * Abd4_0 + o23_8 * Abd5_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o18_8 * Abc0_2 + o19_8 * Abc1_2 + o20_8 * Abc2_2 + o21_8 * Abc3_2 + o22_8 * Abc4_2 + o23_8 * Abc5_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o24_8 * Abd0_0 + o25_8 * Abd1_0 + o26_8 * Abd2_0 + o27_8 * Abd3_0 + o28_8 * Abd4_0 + o29_8 * Abd5_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o24_8 * Abc0_2 + o25_8 * Abc1_2 + o26_8 * Abc2_2 + o27_8 * Abc3_2 + o28_8 * Abc4_2 + o29_8 * Abc5_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o30_8 * Abd0_0 + o31_8 * Abd1_0 + o32_8 * Abd2_0 + o33_8 * Abd3_0 + o34_8 * Abd4_0 + o35_8 * Abd5_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o30_8 * Abc0_2 + o31_8 * Abc1_2 + o32_8 * Abc2_2 + o33_8 * Abc3_2 + o34_8 * Abc4_2 + o35_8 * Abc5_2));
          }
        } break;
        case 9: {  // ket functions [9]
          float o0_9 = 0;
          float o1_9 = 0;
          float o2_9 = 0;
          float o3_9 = 0;
          float o4_9 = 0;
          float o5_9 = 0;
          float o6_9 = 0;
          float o7_9 = 0;
          float o8_9 = 0;
          float o9_9 = 0;
          float o10_9 = 0;
          float o11_9 = 0;
          float o12_9 = 0;
          float o13_9 = 0;
          float o14_9 = 0;
          float o15_9 = 0;
          float o16_9 = 0;
          float o17_9 = 0;
          float o18_9 = 0;
          float o19_9 = 0;
          float o20_9 = 0;
          float o21_9 = 0;
          float o22_9 = 0;
          float o23_9 = 0;
          float o24_9 = 0;
          float o25_9 = 0;
          float o26_9 = 0;
          float o27_9 = 0;
          float o28_9 = 0;
          float o29_9 = 0;
          float o30_9 = 0;
          float o31_9 = 0;
          float o32_9 = 0;
          float o33_9 = 0;
          float o34_9 = 0;
          float o35_9 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g9_0 = 0;
            float g9_1 = 0;
            float g9_2 = 0;
            float g9_3 = 0;
            float g9_4 = 0;
            float g9_5 = 0;
            float g9_6 = 0;
            float g9_7 = 0;
            float g9_8 = 0;
            float g9_9 = 0;
            float g9_10 = 0;
            float g9_11 = 0;
            float g9_12 = 0;
            float g9_13 = 0;
            float g9_14 = 0;
            float g9_15 = 0;
            float g9_16 = 0;
            float g9_17 = 0;
            float g9_18 = 0;
            float g9_19 = 0;
            float g9_20 = 0;
            float g9_21 = 0;
            float g9_22 = 0;
            float g9_23 = 0;
            float g9_24 = 0;
            float g9_25 = 0;
            float g9_26 = 0;
            float g9_27 = 0;
            float g9_28 = 0;
            float g9_29 = 0;
            float g9_30 = 0;
            float g9_31 = 0;
            float g9_32 = 0;
            float g9_33 = 0;
            float g9_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek9_0 = kj[33 * kS];
              const float ek9_1 = -kj[34 * kS];
              const float ek9_2 = -kj[35 * kS];
              const float ek9_3 = kj[36 * kS];
              g9_0 = fmaf(ek9_0, b0, g9_0);
              const float r0_0_0_1 = Z * b1;
              g9_1 = fmaf(ek9_0, r0_0_0_1, g9_1);
              g9_0 = fmaf(ek9_1, r0_0_0_1, g9_0);
              const float r0_0_1_0 = Y * b1;
              g9_2 = fmaf(ek9_0, r0_0_1_0, g9_2);
              const float r0_1_0_0 = X * b1;
              g9_3 = fmaf(ek9_0, r0_1_0_0, g9_3);
              g9_0 = fmaf(ek9_2, r0_1_0_0, g9_0);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g9_4 = fmaf(ek9_0, r0_0_0_2, g9_4);
              g9_1 = fmaf(ek9_1, r0_0_0_2, g9_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g9_5 = fmaf(ek9_0, r0_0_1_1, g9_5);
              g9_2 = fmaf(ek9_1, r0_0_1_1, g9_2);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g9_6 = fmaf(ek9_0, r0_0_2_0, g9_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g9_7 = fmaf(ek9_0, r0_1_0_1, g9_7);
              g9_3 = fmaf(ek9_1, r0_1_0_1, g9_3);
              g9_1 = fmaf(ek9_2, r0_1_0_1, g9_1);
              g9_0 = fmaf(ek9_3, r0_1_0_1, g9_0);
              const float r0_1_1_0 = X * r1_0_1_0;
              g9_8 = fmaf(ek9_0, r0_1_1_0, g9_8);
              g9_2 = fmaf(ek9_2, r0_1_1_0, g9_2);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g9_9 = fmaf(ek9_0, r0_2_0_0, g9_9);
              g9_3 = fmaf(ek9_2, r0_2_0_0, g9_3);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g9_10 = fmaf(ek9_0, r0_0_0_3, g9_10);
              g9_4 = fmaf(ek9_1, r0_0_0_3, g9_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g9_11 = fmaf(ek9_0, r0_0_1_2, g9_11);
              g9_5 = fmaf(ek9_1, r0_0_1_2, g9_5);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g9_12 = fmaf(ek9_0, r0_0_2_1, g9_12);
              g9_6 = fmaf(ek9_1, r0_0_2_1, g9_6);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g9_13 = fmaf(ek9_0, r0_0_3_0, g9_13);
              const float r0_1_0_2 = X * r1_0_0_2;
              g9_14 = fmaf(ek9_0, r0_1_0_2, g9_14);
              g9_7 = fmaf(ek9_1, r0_1_0_2, g9_7);
              g9_4 = fmaf(ek9_2, r0_1_0_2, g9_4);
              g9_1 = fmaf(ek9_3, r0_1_0_2, g9_1);
              const float r0_1_1_1 = X * r1_0_1_1;
              g9_15 = fmaf(ek9_0, r0_1_1_1, g9_15);
              g9_8 = fmaf(ek9_1, r0_1_1_1, g9_8);
              g9_5 = fmaf(ek9_2, r0_1_1_1, g9_5);
              g9_2 = fmaf(ek9_3, r0_1_1_1, g9_2);
              const float r0_1_2_0 = X * r1_0_2_0;
              g9_16 = fmaf(ek9_0, r0_1_2_0, g9_16);
              g9_6 = fmaf(ek9_2, r0_1_2_0, g9_6);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g9_17 = fmaf(ek9_0, r0_2_0_1, g9_17);
              g9_9 = fmaf(ek9_1, r0_2_0_1, g9_9);
              g9_7 = fmaf(ek9_2, r0_2_0_1, g9_7);
              g9_3 = fmaf(ek9_3, r0_2_0_1, g9_3);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g9_18 = fmaf(ek9_0, r0_2_1_0, g9_18);
              g9_8 = fmaf(ek9_2, r0_2_1_0, g9_8);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g9_19 = fmaf(ek9_0, r0_3_0_0, g9_19);
              g9_9 = fmaf(ek9_2, r0_3_0_0, g9_9);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g9_20 = fmaf(ek9_0, r0_0_0_4, g9_20);
              g9_10 = fmaf(ek9_1, r0_0_0_4, g9_10);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g9_21 = fmaf(ek9_0, r0_0_1_3, g9_21);
              g9_11 = fmaf(ek9_1, r0_0_1_3, g9_11);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g9_22 = fmaf(ek9_0, r0_0_2_2, g9_22);
              g9_12 = fmaf(ek9_1, r0_0_2_2, g9_12);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g9_23 = fmaf(ek9_0, r0_0_3_1, g9_23);
              g9_13 = fmaf(ek9_1, r0_0_3_1, g9_13);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g9_24 = fmaf(ek9_0, r0_0_4_0, g9_24);
              const float r0_1_0_3 = X * r1_0_0_3;
              g9_25 = fmaf(ek9_0, r0_1_0_3, g9_25);
              g9_14 = fmaf(ek9_1, r0_1_0_3, g9_14);
              g9_10 = fmaf(ek9_2, r0_1_0_3, g9_10);
              g9_4 = fmaf(ek9_3, r0_1_0_3, g9_4);
              const float r0_1_1_2 = X * r1_0_1_2;
              g9_26 = fmaf(ek9_0, r0_1_1_2, g9_26);
              g9_15 = fmaf(ek9_1, r0_1_1_2, g9_15);
              g9_11 = fmaf(ek9_2, r0_1_1_2, g9_11);
              g9_5 = fmaf(ek9_3, r0_1_1_2, g9_5);
              const float r0_1_2_1 = X * r1_0_2_1;
              g9_27 = fmaf(ek9_0, r0_1_2_1, g9_27);
              g9_16 = fmaf(ek9_1, r0_1_2_1, g9_16);
              g9_12 = fmaf(ek9_2, r0_1_2_1, g9_12);
              g9_6 = fmaf(ek9_3, r0_1_2_1, g9_6);
              const float r0_1_3_0 = X * r1_0_3_0;
              g9_28 = fmaf(ek9_0, r0_1_3_0, g9_28);
              g9_13 = fmaf(ek9_2, r0_1_3_0, g9_13);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g9_29 = fmaf(ek9_0, r0_2_0_2, g9_29);
              g9_17 = fmaf(ek9_1, r0_2_0_2, g9_17);
              g9_14 = fmaf(ek9_2, r0_2_0_2, g9_14);
              g9_7 = fmaf(ek9_3, r0_2_0_2, g9_7);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g9_30 = fmaf(ek9_0, r0_2_1_1, g9_30);
              g9_18 = fmaf(ek9_1, r0_2_1_1, g9_18);
              g9_15 = fmaf(ek9_2, r0_2_1_1, g9_15);
              g9_8 = fmaf(ek9_3, r0_2_1_1, g9_8);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g9_31 = fmaf(ek9_0, r0_2_2_0, g9_31);
              g9_16 = fmaf(ek9_2, r0_2_2_0, g9_16);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g9_32 = fmaf(ek9_0, r0_3_0_1, g9_32);
              g9_19 = fmaf(ek9_1, r0_3_0_1, g9_19);
              g9_17 = fmaf(ek9_2, r0_3_0_1, g9_17);
              g9_9 = fmaf(ek9_3, r0_3_0_1, g9_9);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g9_33 = fmaf(ek9_0, r0_3_1_0, g9_33);
              g9_18 = fmaf(ek9_2, r0_3_1_0, g9_18);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g9_34 = fmaf(ek9_0, r0_4_0_0, g9_34);
              g9_19 = fmaf(ek9_2, r0_4_0_0, g9_19);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_0_5 = fmaf(Z, r1_0_0_4, 4.0f * r1_0_0_3);
              g9_20 = fmaf(ek9_1, r0_0_0_5, g9_20);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g9_21 = fmaf(ek9_1, r0_0_1_4, g9_21);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g9_22 = fmaf(ek9_1, r0_0_2_3, g9_22);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g9_23 = fmaf(ek9_1, r0_0_3_2, g9_23);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g9_24 = fmaf(ek9_1, r0_0_4_1, g9_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g9_25 = fmaf(ek9_1, r0_1_0_4, g9_25);
              g9_20 = fmaf(ek9_2, r0_1_0_4, g9_20);
              g9_10 = fmaf(ek9_3, r0_1_0_4, g9_10);
              const float r0_1_1_3 = X * r1_0_1_3;
              g9_26 = fmaf(ek9_1, r0_1_1_3, g9_26);
              g9_21 = fmaf(ek9_2, r0_1_1_3, g9_21);
              g9_11 = fmaf(ek9_3, r0_1_1_3, g9_11);
              const float r0_1_2_2 = X * r1_0_2_2;
              g9_27 = fmaf(ek9_1, r0_1_2_2, g9_27);
              g9_22 = fmaf(ek9_2, r0_1_2_2, g9_22);
              g9_12 = fmaf(ek9_3, r0_1_2_2, g9_12);
              const float r0_1_3_1 = X * r1_0_3_1;
              g9_28 = fmaf(ek9_1, r0_1_3_1, g9_28);
              g9_23 = fmaf(ek9_2, r0_1_3_1, g9_23);
              g9_13 = fmaf(ek9_3, r0_1_3_1, g9_13);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_1_4_0 = X * r1_0_4_0;
              g9_24 = fmaf(ek9_2, r0_1_4_0, g9_24);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g9_29 = fmaf(ek9_1, r0_2_0_3, g9_29);
              g9_25 = fmaf(ek9_2, r0_2_0_3, g9_25);
              g9_14 = fmaf(ek9_3, r0_2_0_3, g9_14);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g9_30 = fmaf(ek9_1, r0_2_1_2, g9_30);
              g9_26 = fmaf(ek9_2, r0_2_1_2, g9_26);
              g9_15 = fmaf(ek9_3, r0_2_1_2, g9_15);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g9_31 = fmaf(ek9_1, r0_2_2_1, g9_31);
              g9_27 = fmaf(ek9_2, r0_2_2_1, g9_27);
              g9_16 = fmaf(ek9_3, r0_2_2_1, g9_16);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g9_28 = fmaf(ek9_2, r0_2_3_0, g9_28);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g9_32 = fmaf(ek9_1, r0_3_0_2, g9_32);
              g9_29 = fmaf(ek9_2, r0_3_0_2, g9_29);
              g9_17 = fmaf(ek9_3, r0_3_0_2, g9_17);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g9_33 = fmaf(ek9_1, r0_3_1_1, g9_33);
              g9_30 = fmaf(ek9_2, r0_3_1_1, g9_30);
              g9_18 = fmaf(ek9_3, r0_3_1_1, g9_18);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g9_31 = fmaf(ek9_2, r0_3_2_0, g9_31);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g9_34 = fmaf(ek9_1, r0_4_0_1, g9_34);
              g9_32 = fmaf(ek9_2, r0_4_0_1, g9_32);
              g9_19 = fmaf(ek9_3, r0_4_0_1, g9_19);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g9_33 = fmaf(ek9_2, r0_4_1_0, g9_33);
              const float r4_1_0_0 = X * b5;
              const float r3_2_0_0 = fmaf(X, r4_1_0_0, b4);
              const float r2_3_0_0 = fmaf(X, r3_2_0_0, 2.0f * r3_1_0_0);
              const float r1_4_0_0 = fmaf(X, r2_3_0_0, 3.0f * r2_2_0_0);
              const float r0_5_0_0 = fmaf(X, r1_4_0_0, 4.0f * r1_3_0_0);
              g9_34 = fmaf(ek9_2, r0_5_0_0, g9_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_0_5 = fmaf(Z, r2_0_0_4, 4.0f * r2_0_0_3);
              const float r0_1_0_5 = X * r1_0_0_5;
              g9_20 = fmaf(ek9_3, r0_1_0_5, g9_20);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_1_1_4 = X * r1_0_1_4;
              g9_21 = fmaf(ek9_3, r0_1_1_4, g9_21);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_1_2_3 = X * r1_0_2_3;
              g9_22 = fmaf(ek9_3, r0_1_2_3, g9_22);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_1_3_2 = X * r1_0_3_2;
              g9_23 = fmaf(ek9_3, r0_1_3_2, g9_23);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_1_4_1 = X * r1_0_4_1;
              g9_24 = fmaf(ek9_3, r0_1_4_1, g9_24);
              const float r1_1_0_4 = X * r2_0_0_4;
              const float r0_2_0_4 = fmaf(X, r1_1_0_4, r1_0_0_4);
              g9_25 = fmaf(ek9_3, r0_2_0_4, g9_25);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g9_26 = fmaf(ek9_3, r0_2_1_3, g9_26);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g9_27 = fmaf(ek9_3, r0_2_2_2, g9_27);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g9_28 = fmaf(ek9_3, r0_2_3_1, g9_28);
              const float r2_1_0_3 = X * r3_0_0_3;
              const float r1_2_0_3 = fmaf(X, r2_1_0_3, r2_0_0_3);
              const float r0_3_0_3 = fmaf(X, r1_2_0_3, 2.0f * r1_1_0_3);
              g9_29 = fmaf(ek9_3, r0_3_0_3, g9_29);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g9_30 = fmaf(ek9_3, r0_3_1_2, g9_30);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g9_31 = fmaf(ek9_3, r0_3_2_1, g9_31);
              const float r3_1_0_2 = X * r4_0_0_2;
              const float r2_2_0_2 = fmaf(X, r3_1_0_2, r3_0_0_2);
              const float r1_3_0_2 = fmaf(X, r2_2_0_2, 2.0f * r2_1_0_2);
              const float r0_4_0_2 = fmaf(X, r1_3_0_2, 3.0f * r1_2_0_2);
              g9_32 = fmaf(ek9_3, r0_4_0_2, g9_32);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g9_33 = fmaf(ek9_3, r0_4_1_1, g9_33);
              const float r4_1_0_1 = X * r5_0_0_1;
              const float r3_2_0_1 = fmaf(X, r4_1_0_1, r4_0_0_1);
              const float r2_3_0_1 = fmaf(X, r3_2_0_1, 2.0f * r3_1_0_1);
              const float r1_4_0_1 = fmaf(X, r2_3_0_1, 3.0f * r2_2_0_1);
              const float r0_5_0_1 = fmaf(X, r1_4_0_1, 4.0f * r1_3_0_1);
              g9_34 = fmaf(ek9_3, r0_5_0_1, g9_34);
            }
            { const float eb = bi[5];
              o0_9 = fmaf(eb, g9_0, o0_9);
            }
            { const float eb = bi[6];
              o0_9 = fmaf(eb, g9_3, o0_9);
            }
            { const float eb = bi[7];
              o0_9 = fmaf(eb, g9_9, o0_9);
            }
            { const float eb = bi[8];
              o0_9 = fmaf(eb, g9_19, o0_9);
            }
            { const float eb = bi[9];
              o0_9 = fmaf(eb, g9_34, o0_9);
            }
            { const float eb = bi[10];
              o1_9 = fmaf(eb, g9_0, o1_9);
            }
            { const float eb = bi[11];
              o1_9 = fmaf(eb, g9_2, o1_9);
            }
            { const float eb = bi[12];
              o1_9 = fmaf(eb, g9_6, o1_9);
            }
            { const float eb = bi[13];
              o1_9 = fmaf(eb, g9_3, o1_9);
            }
            { const float eb = bi[14];
              o1_9 = fmaf(eb, g9_8, o1_9);
            }
            { const float eb = bi[15];
              o1_9 = fmaf(eb, g9_16, o1_9);
            }
            { const float eb = bi[16];
              o1_9 = fmaf(eb, g9_9, o1_9);
            }
            { const float eb = bi[17];
              o1_9 = fmaf(eb, g9_18, o1_9);
            }
            { const float eb = bi[18];
              o1_9 = fmaf(eb, g9_31, o1_9);
            }
            { const float eb = bi[19];
              o2_9 = fmaf(eb, g9_0, o2_9);
            }
            { const float eb = bi[20];
              o2_9 = fmaf(eb, g9_1, o2_9);
            }
            { const float eb = bi[21];
              o2_9 = fmaf(eb, g9_4, o2_9);
            }
            { const float eb = bi[22];
              o2_9 = fmaf(eb, g9_3, o2_9);
            }
            { const float eb = bi[23];
              o2_9 = fmaf(eb, g9_7, o2_9);
            }
            { const float eb = bi[24];
              o2_9 = fmaf(eb, g9_14, o2_9);
            }
            { const float eb = bi[25];
              o2_9 = fmaf(eb, g9_9, o2_9);
            }
            { const float eb = bi[26];
              o2_9 = fmaf(eb, g9_17, o2_9);
            }
            { const float eb = bi[27];
              o2_9 = fmaf(eb, g9_29, o2_9);
            }
            { const float eb = bi[28];
              o3_9 = fmaf(eb, g9_0, o3_9);
            }
            { const float eb = bi[29];
              o3_9 = fmaf(eb, g9_2, o3_9);
            }
            { const float eb = bi[30];
              o3_9 = fmaf(eb, g9_3, o3_9);
            }
            { const float eb = bi[31];
              o3_9 = fmaf(eb, g9_8, o3_9);
            }
            { const float eb = bi[32];
              o3_9 = fmaf(eb, g9_9, o3_9);
            }
            { const float eb = bi[33];
              o3_9 = fmaf(eb, g9_18, o3_9);
            }
            { const float eb = bi[34];
              o3_9 = fmaf(eb, g9_19, o3_9);
            }
            { const float eb = bi[35];
              o3_9 = fmaf(eb, g9_33, o3_9);
            }
            { const float eb = bi[36];
              o4_9 = fmaf(eb, g9_0, o4_9);
            }
            { const float eb = bi[37];
              o4_9 = fmaf(eb, g9_1, o4_9);
            }
            { const float eb = bi[38];
              o4_9 = fmaf(eb, g9_3, o4_9);
            }
            { const float eb = bi[39];
              o4_9 = fmaf(eb, g9_7, o4_9);
            }
            { const float eb = bi[40];
              o4_9 = fmaf(eb, g9_9, o4_9);
            }
            { const float eb = bi[41];
              o4_9 = fmaf(eb, g9_17, o4_9);
            }
            { const float eb = bi[42];
              o4_9 = fmaf(eb, g9_19, o4_9);
            }
            { const float eb = bi[43];
              o4_9 = fmaf(eb, g9_32, o4_9);
            }
            { const float eb = bi[44];
              o5_9 = fmaf(eb, g9_0, o5_9);
            }
            { const float eb = bi[45];
              o5_9 = fmaf(eb, g9_1, o5_9);
            }
            { const float eb = bi[46];
              o5_9 = fmaf(eb, g9_2, o5_9);
            }
            { const float eb = bi[47];
              o5_9 = fmaf(eb, g9_5, o5_9);
            }
            { const float eb = bi[48];
              o5_9 = fmaf(eb, g9_3, o5_9);
            }
            { const float eb = bi[49];
              o5_9 = fmaf(eb, g9_7, o5_9);
            }
            { const float eb = bi[50];
              o5_9 = fmaf(eb, g9_8, o5_9);
            }
            { const float eb = bi[51];
              o5_9 = fmaf(eb, g9_15, o5_9);
            }
            { const float eb = bi[52];
              o5_9 = fmaf(eb, g9_9, o5_9);
            }
            { const float eb = bi[53];
              o5_9 = fmaf(eb, g9_17, o5_9);
            }
            { const float eb = bi[54];
              o5_9 = fmaf(eb, g9_18, o5_9);
            }
            { const float eb = bi[55];
              o5_9 = fmaf(eb, g9_30, o5_9);
            }
            { const float eb = bi[56];
              o6_9 = fmaf(eb, g9_0, o6_9);
            }
            { const float eb = bi[57];
              o6_9 = fmaf(eb, g9_2, o6_9);
            }
            { const float eb = bi[58];
              o6_9 = fmaf(eb, g9_6, o6_9);
            }
            { const float eb = bi[59];
              o6_9 = fmaf(eb, g9_3, o6_9);
            }
            { const float eb = bi[60];
              o6_9 = fmaf(eb, g9_8, o6_9);
            }
            { const float eb = bi[61];
              o6_9 = fmaf(eb, g9_16, o6_9);
            }
            { const float eb = bi[62];
              o6_9 = fmaf(eb, g9_9, o6_9);
            }
            { const float eb = bi[63];
              o6_9 = fmaf(eb, g9_18, o6_9);
            }
            { const float eb = bi[64];
              o6_9 = fmaf(eb, g9_31, o6_9);
            }
            { const float eb = bi[65];
              o7_9 = fmaf(eb, g9_0, o7_9);
            }
            { const float eb = bi[66];
              o7_9 = fmaf(eb, g9_2, o7_9);
            }
            { const float eb = bi[67];
              o7_9 = fmaf(eb, g9_6, o7_9);
            }
            { const float eb = bi[68];
              o7_9 = fmaf(eb, g9_13, o7_9);
            }
            { const float eb = bi[69];
              o7_9 = fmaf(eb, g9_24, o7_9);
            }
            { const float eb = bi[70];
              o8_9 = fmaf(eb, g9_0, o8_9);
            }
            { const float eb = bi[71];
              o8_9 = fmaf(eb, g9_1, o8_9);
            }
            { const float eb = bi[72];
              o8_9 = fmaf(eb, g9_4, o8_9);
            }
            { const float eb = bi[73];
              o8_9 = fmaf(eb, g9_2, o8_9);
            }
            { const float eb = bi[74];
              o8_9 = fmaf(eb, g9_5, o8_9);
            }
            { const float eb = bi[75];
              o8_9 = fmaf(eb, g9_11, o8_9);
            }
            { const float eb = bi[76];
              o8_9 = fmaf(eb, g9_6, o8_9);
            }
            { const float eb = bi[77];
              o8_9 = fmaf(eb, g9_12, o8_9);
            }
            { const float eb = bi[78];
              o8_9 = fmaf(eb, g9_22, o8_9);
            }
            { const float eb = bi[79];
              o9_9 = fmaf(eb, g9_0, o9_9);
            }
            { const float eb = bi[80];
              o9_9 = fmaf(eb, g9_2, o9_9);
            }
            { const float eb = bi[81];
              o9_9 = fmaf(eb, g9_6, o9_9);
            }
            { const float eb = bi[82];
              o9_9 = fmaf(eb, g9_13, o9_9);
            }
            { const float eb = bi[83];
              o9_9 = fmaf(eb, g9_3, o9_9);
            }
            { const float eb = bi[84];
              o9_9 = fmaf(eb, g9_8, o9_9);
            }
            { const float eb = bi[85];
              o9_9 = fmaf(eb, g9_16, o9_9);
            }
            { const float eb = bi[86];
              o9_9 = fmaf(eb, g9_28, o9_9);
            }
            { const float eb = bi[87];
              o10_9 = fmaf(eb, g9_0, o10_9);
            }
            { const float eb = bi[88];
              o10_9 = fmaf(eb, g9_1, o10_9);
            }
            { const float eb = bi[89];
              o10_9 = fmaf(eb, g9_2, o10_9);
            }
            { const float eb = bi[90];
              o10_9 = fmaf(eb, g9_5, o10_9);
            }
            { const float eb = bi[91];
              o10_9 = fmaf(eb, g9_6, o10_9);
            }
            { const float eb = bi[92];
              o10_9 = fmaf(eb, g9_12, o10_9);
            }
            { const float eb = bi[93];
              o10_9 = fmaf(eb, g9_3, o10_9);
            }
            { const float eb = bi[94];
              o10_9 = fmaf(eb, g9_7, o10_9);
            }
            { const float eb = bi[95];
              o10_9 = fmaf(eb, g9_8, o10_9);
            }
            { const float eb = bi[96];
              o10_9 = fmaf(eb, g9_15, o10_9);
            }
            { const float eb = bi[97];
              o10_9 = fmaf(eb, g9_16, o10_9);
            }
            { const float eb = bi[98];
              o10_9 = fmaf(eb, g9_27, o10_9);
            }
            { const float eb = bi[99];
              o11_9 = fmaf(eb, g9_0, o11_9);
            }
            { const float eb = bi[100];
              o11_9 = fmaf(eb, g9_1, o11_9);
            }
            { const float eb = bi[101];
              o11_9 = fmaf(eb, g9_2, o11_9);
            }
            { const float eb = bi[102];
              o11_9 = fmaf(eb, g9_5, o11_9);
            }
            { const float eb = bi[103];
              o11_9 = fmaf(eb, g9_6, o11_9);
            }
            { const float eb = bi[104];
              o11_9 = fmaf(eb, g9_12, o11_9);
            }
            { const float eb = bi[105];
              o11_9 = fmaf(eb, g9_13, o11_9);
            }
            { const float eb = bi[106];
              o11_9 = fmaf(eb, g9_23, o11_9);
            }
            { const float eb = bi[107];
              o12_9 = fmaf(eb, g9_0, o12_9);
            }
            { const float eb = bi[108];
              o12_9 = fmaf(eb, g9_1, o12_9);
            }
            { const float eb = bi[109];
              o12_9 = fmaf(eb, g9_4, o12_9);
            }
            { const float eb = bi[110];
              o12_9 = fmaf(eb, g9_3, o12_9);
            }
            { const float eb = bi[111];
              o12_9 = fmaf(eb, g9_7, o12_9);
            }
            { const float eb = bi[112];
              o12_9 = fmaf(eb, g9_14, o12_9);
            }
            { const float eb = bi[113];
              o12_9 = fmaf(eb, g9_9, o12_9);
            }
            { const float eb = bi[114];
              o12_9 = fmaf(eb, g9_17, o12_9);
            }
            { const float eb = bi[115];
              o12_9 = fmaf(eb, g9_29, o12_9);
            }
            { const float eb = bi[116];
              o13_9 = fmaf(eb, g9_0, o13_9);
            }
            { const float eb = bi[117];
              o13_9 = fmaf(eb, g9_1, o13_9);
            }
            { const float eb = bi[118];
              o13_9 = fmaf(eb, g9_4, o13_9);
            }
            { const float eb = bi[119];
              o13_9 = fmaf(eb, g9_2, o13_9);
            }
            { const float eb = bi[120];
              o13_9 = fmaf(eb, g9_5, o13_9);
            }
            { const float eb = bi[121];
              o13_9 = fmaf(eb, g9_11, o13_9);
            }
            { const float eb = bi[122];
              o13_9 = fmaf(eb, g9_6, o13_9);
            }
            { const float eb = bi[123];
              o13_9 = fmaf(eb, g9_12, o13_9);
            }
            { const float eb = bi[124];
              o13_9 = fmaf(eb, g9_22, o13_9);
            }
            { const float eb = bi[125];
              o14_9 = fmaf(eb, g9_0, o14_9);
            }
            { const float eb = bi[126];
              o14_9 = fmaf(eb, g9_1, o14_9);
            }
            { const float eb = bi[127];
              o14_9 = fmaf(eb, g9_4, o14_9);
            }
            { const float eb = bi[128];
              o14_9 = fmaf(eb, g9_10, o14_9);
            }
            { const float eb = bi[129];
              o14_9 = fmaf(eb, g9_20, o14_9);
            }
            { const float eb = bi[130];
              o15_9 = fmaf(eb, g9_0, o15_9);
            }
            { const float eb = bi[131];
              o15_9 = fmaf(eb, g9_1, o15_9);
            }
            { const float eb = bi[132];
              o15_9 = fmaf(eb, g9_4, o15_9);
            }
            { const float eb = bi[133];
              o15_9 = fmaf(eb, g9_2, o15_9);
            }
            { const float eb = bi[134];
              o15_9 = fmaf(eb, g9_5, o15_9);
            }
            { const float eb = bi[135];
              o15_9 = fmaf(eb, g9_11, o15_9);
            }
            { const float eb = bi[136];
              o15_9 = fmaf(eb, g9_3, o15_9);
            }
            { const float eb = bi[137];
              o15_9 = fmaf(eb, g9_7, o15_9);
            }
            { const float eb = bi[138];
              o15_9 = fmaf(eb, g9_14, o15_9);
            }
            { const float eb = bi[139];
              o15_9 = fmaf(eb, g9_8, o15_9);
            }
            { const float eb = bi[140];
              o15_9 = fmaf(eb, g9_15, o15_9);
            }
            { const float eb = bi[141];
              o15_9 = fmaf(eb, g9_26, o15_9);
            }
            { const float eb = bi[142];
              o16_9 = fmaf(eb, g9_0, o16_9);
            }
            { const float eb = bi[143];
              o16_9 = fmaf(eb, g9_1, o16_9);
            }
            { const float eb = bi[144];
              o16_9 = fmaf(eb, g9_4, o16_9);
            }
            { const float eb = bi[145];
              o16_9 = fmaf(eb, g9_10, o16_9);
            }
            { const float eb = bi[146];
              o16_9 = fmaf(eb, g9_3, o16_9);
            }
            { const float eb = bi[147];
              o16_9 = fmaf(eb, g9_7, o16_9);
            }
            { const float eb = bi[148];
              o16_9 = fmaf(eb, g9_14, o16_9);
            }
            { const float eb = bi[149];
              o16_9 = fmaf(eb, g9_25, o16_9);
            }
            { const float eb = bi[150];
              o17_9 = fmaf(eb, g9_0, o17_9);
            }
            { const float eb = bi[151];
              o17_9 = fmaf(eb, g9_1, o17_9);
            }
            { const float eb = bi[152];
              o17_9 = fmaf(eb, g9_4, o17_9);
            }
            { const float eb = bi[153];
              o17_9 = fmaf(eb, g9_10, o17_9);
            }
            { const float eb = bi[154];
              o17_9 = fmaf(eb, g9_2, o17_9);
            }
            { const float eb = bi[155];
              o17_9 = fmaf(eb, g9_5, o17_9);
            }
            { const float eb = bi[156];
              o17_9 = fmaf(eb, g9_11, o17_9);
            }
            { const float eb = bi[157];
              o17_9 = fmaf(eb, g9_21, o17_9);
            }
            { const float eb = bi[158];
              o18_9 = fmaf(eb, g9_0, o18_9);
            }
            { const float eb = bi[159];
              o18_9 = fmaf(eb, g9_2, o18_9);
            }
            { const float eb = bi[160];
              o18_9 = fmaf(eb, g9_3, o18_9);
            }
            { const float eb = bi[161];
              o18_9 = fmaf(eb, g9_8, o18_9);
            }
            { const float eb = bi[162];
              o18_9 = fmaf(eb, g9_9, o18_9);
            }
            { const float eb = bi[163];
              o18_9 = fmaf(eb, g9_18, o18_9);
            }
            { const float eb = bi[164];
              o18_9 = fmaf(eb, g9_19, o18_9);
            }
            { const float eb = bi[165];
              o18_9 = fmaf(eb, g9_33, o18_9);
            }
            { const float eb = bi[166];
              o19_9 = fmaf(eb, g9_0, o19_9);
            }
            { const float eb = bi[167];
              o19_9 = fmaf(eb, g9_2, o19_9);
            }
            { const float eb = bi[168];
              o19_9 = fmaf(eb, g9_6, o19_9);
            }
            { const float eb = bi[169];
              o19_9 = fmaf(eb, g9_13, o19_9);
            }
            { const float eb = bi[170];
              o19_9 = fmaf(eb, g9_3, o19_9);
            }
            { const float eb = bi[171];
              o19_9 = fmaf(eb, g9_8, o19_9);
            }
            { const float eb = bi[172];
              o19_9 = fmaf(eb, g9_16, o19_9);
            }
            { const float eb = bi[173];
              o19_9 = fmaf(eb, g9_28, o19_9);
            }
            { const float eb = bi[174];
              o20_9 = fmaf(eb, g9_0, o20_9);
            }
            { const float eb = bi[175];
              o20_9 = fmaf(eb, g9_1, o20_9);
            }
            { const float eb = bi[176];
              o20_9 = fmaf(eb, g9_4, o20_9);
            }
            { const float eb = bi[177];
              o20_9 = fmaf(eb, g9_2, o20_9);
            }
            { const float eb = bi[178];
              o20_9 = fmaf(eb, g9_5, o20_9);
            }
            { const float eb = bi[179];
              o20_9 = fmaf(eb, g9_11, o20_9);
            }
            { const float eb = bi[180];
              o20_9 = fmaf(eb, g9_3, o20_9);
            }
            { const float eb = bi[181];
              o20_9 = fmaf(eb, g9_7, o20_9);
            }
            { const float eb = bi[182];
              o20_9 = fmaf(eb, g9_14, o20_9);
            }
            { const float eb = bi[183];
              o20_9 = fmaf(eb, g9_8, o20_9);
            }
            { const float eb = bi[184];
              o20_9 = fmaf(eb, g9_15, o20_9);
            }
            { const float eb = bi[185];
              o20_9 = fmaf(eb, g9_26, o20_9);
            }
            { const float eb = bi[186];
              o21_9 = fmaf(eb, g9_0, o21_9);
            }
            { const float eb = bi[187];
              o21_9 = fmaf(eb, g9_2, o21_9);
            }
            { const float eb = bi[188];
              o21_9 = fmaf(eb, g9_6, o21_9);
            }
            { const float eb = bi[189];
              o21_9 = fmaf(eb, g9_3, o21_9);
            }
            { const float eb = bi[190];
              o21_9 = fmaf(eb, g9_8, o21_9);
            }
            { const float eb = bi[191];
              o21_9 = fmaf(eb, g9_16, o21_9);
            }
            { const float eb = bi[192];
              o21_9 = fmaf(eb, g9_9, o21_9);
            }
            { const float eb = bi[193];
              o21_9 = fmaf(eb, g9_18, o21_9);
            }
            { const float eb = bi[194];
              o21_9 = fmaf(eb, g9_31, o21_9);
            }
            { const float eb = bi[195];
              o22_9 = fmaf(eb, g9_0, o22_9);
            }
            { const float eb = bi[196];
              o22_9 = fmaf(eb, g9_1, o22_9);
            }
            { const float eb = bi[197];
              o22_9 = fmaf(eb, g9_2, o22_9);
            }
            { const float eb = bi[198];
              o22_9 = fmaf(eb, g9_5, o22_9);
            }
            { const float eb = bi[199];
              o22_9 = fmaf(eb, g9_3, o22_9);
            }
            { const float eb = bi[200];
              o22_9 = fmaf(eb, g9_7, o22_9);
            }
            { const float eb = bi[201];
              o22_9 = fmaf(eb, g9_8, o22_9);
            }
            { const float eb = bi[202];
              o22_9 = fmaf(eb, g9_15, o22_9);
            }
            { const float eb = bi[203];
              o22_9 = fmaf(eb, g9_9, o22_9);
            }
            { const float eb = bi[204];
              o22_9 = fmaf(eb, g9_17, o22_9);
            }
            { const float eb = bi[205];
              o22_9 = fmaf(eb, g9_18, o22_9);
            }
            { const float eb = bi[206];
              o22_9 = fmaf(eb, g9_30, o22_9);
            }
            { const float eb = bi[207];
              o23_9 = fmaf(eb, g9_0, o23_9);
            }
            { const float eb = bi[208];
              o23_9 = fmaf(eb, g9_1, o23_9);
            }
            { const float eb = bi[209];
              o23_9 = fmaf(eb, g9_2, o23_9);
            }
            { const float eb = bi[210];
              o23_9 = fmaf(eb, g9_5, o23_9);
            }
            { const float eb = bi[211];
              o23_9 = fmaf(eb, g9_6, o23_9);
            }
            { const float eb = bi[212];
              o23_9 = fmaf(eb, g9_12, o23_9);
            }
            { const float eb = bi[213];
              o23_9 = fmaf(eb, g9_3, o23_9);
            }
            { const float eb = bi[214];
              o23_9 = fmaf(eb, g9_7, o23_9);
            }
            { const float eb = bi[215];
              o23_9 = fmaf(eb, g9_8, o23_9);
            }
            { const float eb = bi[216];
              o23_9 = fmaf(eb, g9_15, o23_9);
            }
            { const float eb = bi[217];
              o23_9 = fmaf(eb, g9_16, o23_9);
            }
            { const float eb = bi[218];
              o23_9 = fmaf(eb, g9_27, o23_9);
            }
            { const float eb = bi[219];
              o24_9 = fmaf(eb, g9_0, o24_9);
            }
            { const float eb = bi[220];
              o24_9 = fmaf(eb, g9_1, o24_9);
            }
            { const float eb = bi[221];
              o24_9 = fmaf(eb, g9_3, o24_9);
            }
            { const float eb = bi[222];
              o24_9 = fmaf(eb, g9_7, o24_9);
            }
            { const float eb = bi[223];
              o24_9 = fmaf(eb, g9_9, o24_9);
            }
            { const float eb = bi[224];
              o24_9 = fmaf(eb, g9_17, o24_9);
            }
            { const float eb = bi[225];
              o24_9 = fmaf(eb, g9_19, o24_9);
            }
            { const float eb = bi[226];
              o24_9 = fmaf(eb, g9_32, o24_9);
            }
            { const float eb = bi[227];
              o25_9 = fmaf(eb, g9_0, o25_9);
            }
            { const float eb = bi[228];
              o25_9 = fmaf(eb, g9_1, o25_9);
            }
            { const float eb = bi[229];
              o25_9 = fmaf(eb, g9_2, o25_9);
            }
            { const float eb = bi[230];
              o25_9 = fmaf(eb, g9_5, o25_9);
            }
            { const float eb = bi[231];
              o25_9 = fmaf(eb, g9_6, o25_9);
            }
            { const float eb = bi[232];
              o25_9 = fmaf(eb, g9_12, o25_9);
            }
            { const float eb = bi[233];
              o25_9 = fmaf(eb, g9_3, o25_9);
            }
            { const float eb = bi[234];
              o25_9 = fmaf(eb, g9_7, o25_9);
            }
            { const float eb = bi[235];
              o25_9 = fmaf(eb, g9_8, o25_9);
            }
            { const float eb = bi[236];
              o25_9 = fmaf(eb, g9_15, o25_9);
            }
            { const float eb = bi[237];
              o25_9 = fmaf(eb, g9_16, o25_9);
            }
            { const float eb = bi[238];
              o25_9 = fmaf(eb, g9_27, o25_9);
            }
            { const float eb = bi[239];
              o26_9 = fmaf(eb, g9_0, o26_9);
            }
            { const float eb = bi[240];
              o26_9 = fmaf(eb, g9_1, o26_9);
            }
            { const float eb = bi[241];
              o26_9 = fmaf(eb, g9_4, o26_9);
            }
            { const float eb = bi[242];
              o26_9 = fmaf(eb, g9_10, o26_9);
            }
            { const float eb = bi[243];
              o26_9 = fmaf(eb, g9_3, o26_9);
            }
            { const float eb = bi[244];
              o26_9 = fmaf(eb, g9_7, o26_9);
            }
            { const float eb = bi[245];
              o26_9 = fmaf(eb, g9_14, o26_9);
            }
            { const float eb = bi[246];
              o26_9 = fmaf(eb, g9_25, o26_9);
            }
            { const float eb = bi[247];
              o27_9 = fmaf(eb, g9_0, o27_9);
            }
            { const float eb = bi[248];
              o27_9 = fmaf(eb, g9_1, o27_9);
            }
            { const float eb = bi[249];
              o27_9 = fmaf(eb, g9_2, o27_9);
            }
            { const float eb = bi[250];
              o27_9 = fmaf(eb, g9_5, o27_9);
            }
            { const float eb = bi[251];
              o27_9 = fmaf(eb, g9_3, o27_9);
            }
            { const float eb = bi[252];
              o27_9 = fmaf(eb, g9_7, o27_9);
            }
            { const float eb = bi[253];
              o27_9 = fmaf(eb, g9_8, o27_9);
            }
            { const float eb = bi[254];
              o27_9 = fmaf(eb, g9_15, o27_9);
            }
            { const float eb = bi[255];
              o27_9 = fmaf(eb, g9_9, o27_9);
            }
            { const float eb = bi[256];
              o27_9 = fmaf(eb, g9_17, o27_9);
            }
            { const float eb = bi[257];
              o27_9 = fmaf(eb, g9_18, o27_9);
            }
            { const float eb = bi[258];
              o27_9 = fmaf(eb, g9_30, o27_9);
            }
            { const float eb = bi[259];
              o28_9 = fmaf(eb, g9_0, o28_9);
            }
            { const float eb = bi[260];
              o28_9 = fmaf(eb, g9_1, o28_9);
            }
            { const float eb = bi[261];
              o28_9 = fmaf(eb, g9_4, o28_9);
            }
            { const float eb = bi[262];
              o28_9 = fmaf(eb, g9_3, o28_9);
            }
            { const float eb = bi[263];
              o28_9 = fmaf(eb, g9_7, o28_9);
            }
            { const float eb = bi[264];
              o28_9 = fmaf(eb, g9_14, o28_9);
            }
            { const float eb = bi[265];
              o28_9 = fmaf(eb, g9_9, o28_9);
            }
            { const float eb = bi[266];
              o28_9 = fmaf(eb, g9_17, o28_9);
            }
            { const float eb = bi[267];
              o28_9 = fmaf(eb, g9_29, o28_9);
            }
            { const float eb = bi[268];
              o29_9 = fmaf(eb, g9_0, o29_9);
            }
            { const float eb = bi[269];
              o29_9 = fmaf(eb, g9_1, o29_9);
            }
            { const float eb = bi[270];
              o29_9 = fmaf(eb, g9_4, o29_9);
            }
            { const float eb = bi[271];
              o29_9 = fmaf(eb, g9_2, o29_9);
            }
            { const float eb = bi[272];
              o29_9 = fmaf(eb, g9_5, o29_9);
            }
            { const float eb = bi[273];
              o29_9 = fmaf(eb, g9_11, o29_9);
            }
            { const float eb = bi[274];
              o29_9 = fmaf(eb, g9_3, o29_9);
            }
            { const float eb = bi[275];
              o29_9 = fmaf(eb, g9_7, o29_9);
            }
            { const float eb = bi[276];
              o29_9 = fmaf(eb, g9_14, o29_9);
            }
            { const float eb = bi[277];
              o29_9 = fmaf(eb, g9_8, o29_9);
            }
            { const float eb = bi[278];
              o29_9 = fmaf(eb, g9_15, o29_9);
            }
            { const float eb = bi[279];
              o29_9 = fmaf(eb, g9_26, o29_9);
            }
            { const float eb = bi[280];
              o30_9 = fmaf(eb, g9_0, o30_9);
            }
            { const float eb = bi[281];
              o30_9 = fmaf(eb, g9_1, o30_9);
            }
            { const float eb = bi[282];
              o30_9 = fmaf(eb, g9_2, o30_9);
            }
            { const float eb = bi[283];
              o30_9 = fmaf(eb, g9_5, o30_9);
            }
            { const float eb = bi[284];
              o30_9 = fmaf(eb, g9_3, o30_9);
            }
            { const float eb = bi[285];
              o30_9 = fmaf(eb, g9_7, o30_9);
            }
            { const float eb = bi[286];
              o30_9 = fmaf(eb, g9_8, o30_9);
            }
            { const float eb = bi[287];
              o30_9 = fmaf(eb, g9_15, o30_9);
            }
            { const float eb = bi[288];
              o30_9 = fmaf(eb, g9_9, o30_9);
            }
            { const float eb = bi[289];
              o30_9 = fmaf(eb, g9_17, o30_9);
            }
            { const float eb = bi[290];
              o30_9 = fmaf(eb, g9_18, o30_9);
            }
            { const float eb = bi[291];
              o30_9 = fmaf(eb, g9_30, o30_9);
            }
            { const float eb = bi[292];
              o31_9 = fmaf(eb, g9_0, o31_9);
            }
            { const float eb = bi[293];
              o31_9 = fmaf(eb, g9_1, o31_9);
            }
            { const float eb = bi[294];
              o31_9 = fmaf(eb, g9_2, o31_9);
            }
            { const float eb = bi[295];
              o31_9 = fmaf(eb, g9_5, o31_9);
            }
            { const float eb = bi[296];
              o31_9 = fmaf(eb, g9_6, o31_9);
            }
            { const float eb = bi[297];
              o31_9 = fmaf(eb, g9_12, o31_9);
            }
            { const float eb = bi[298];
              o31_9 = fmaf(eb, g9_13, o31_9);
            }
            { const float eb = bi[299];
              o31_9 = fmaf(eb, g9_23, o31_9);
            }
            { const float eb = bi[300];
              o32_9 = fmaf(eb, g9_0, o32_9);
            }
            { const float eb = bi[301];
              o32_9 = fmaf(eb, g9_1, o32_9);
            }
            { const float eb = bi[302];
              o32_9 = fmaf(eb, g9_4, o32_9);
            }
            { const float eb = bi[303];
              o32_9 = fmaf(eb, g9_10, o32_9);
            }
            { const float eb = bi[304];
              o32_9 = fmaf(eb, g9_2, o32_9);
            }
            { const float eb = bi[305];
              o32_9 = fmaf(eb, g9_5, o32_9);
            }
            { const float eb = bi[306];
              o32_9 = fmaf(eb, g9_11, o32_9);
            }
            { const float eb = bi[307];
              o32_9 = fmaf(eb, g9_21, o32_9);
            }
            { const float eb = bi[308];
              o33_9 = fmaf(eb, g9_0, o33_9);
            }
            { const float eb = bi[309];
              o33_9 = fmaf(eb, g9_1, o33_9);
            }
            { const float eb = bi[310];
              o33_9 = fmaf(eb, g9_2, o33_9);
            }
            { const float eb = bi[311];
              o33_9 = fmaf(eb, g9_5, o33_9);
            }
            { const float eb = bi[312];
              o33_9 = fmaf(eb, g9_6, o33_9);
            }
            { const float eb = bi[313];
              o33_9 = fmaf(eb, g9_12, o33_9);
            }
            { const float eb = bi[314];
              o33_9 = fmaf(eb, g9_3, o33_9);
            }
            { const float eb = bi[315];
              o33_9 = fmaf(eb, g9_7, o33_9);
            }
            { const float eb = bi[316];
              o33_9 = fmaf(eb, g9_8, o33_9);
            }
            { const float eb = bi[317];
              o33_9 = fmaf(eb, g9_15, o33_9);
            }
            { const float eb = bi[318];
              o33_9 = fmaf(eb, g9_16, o33_9);
            }
            { const float eb = bi[319];
              o33_9 = fmaf(eb, g9_27, o33_9);
            }
            { const float eb = bi[320];
              o34_9 = fmaf(eb, g9_0, o34_9);
            }
            { const float eb = bi[321];
              o34_9 = fmaf(eb, g9_1, o34_9);
            }
            { const float eb = bi[322];
              o34_9 = fmaf(eb, g9_4, o34_9);
            }
            { const float eb = bi[323];
              o34_9 = fmaf(eb, g9_2, o34_9);
            }
            { const float eb = bi[324];
              o34_9 = fmaf(eb, g9_5, o34_9);
            }
            { const float eb = bi[325];
              o34_9 = fmaf(eb, g9_11, o34_9);
            }
            { const float eb = bi[326];
              o34_9 = fmaf(eb, g9_3, o34_9);
            }
            { const float eb = bi[327];
              o34_9 = fmaf(eb, g9_7, o34_9);
            }
            { const float eb = bi[328];
              o34_9 = fmaf(eb, g9_14, o34_9);
            }
            { const float eb = bi[329];
              o34_9 = fmaf(eb, g9_8, o34_9);
            }
            { const float eb = bi[330];
              o34_9 = fmaf(eb, g9_15, o34_9);
            }
            { const float eb = bi[331];
              o34_9 = fmaf(eb, g9_26, o34_9);
            }
            { const float eb = bi[332];
              o35_9 = fmaf(eb, g9_0, o35_9);
            }
            { const float eb = bi[333];
              o35_9 = fmaf(eb, g9_1, o35_9);
            }
            { const float eb = bi[334];
              o35_9 = fmaf(eb, g9_4, o35_9);
            }
            { const float eb = bi[335];
              o35_9 = fmaf(eb, g9_2, o35_9);
            }
            { const float eb = bi[336];
              o35_9 = fmaf(eb, g9_5, o35_9);
            }
            { const float eb = bi[337];
              o35_9 = fmaf(eb, g9_11, o35_9);
            }
            { const float eb = bi[338];
              o35_9 = fmaf(eb, g9_6, o35_9);
            }
            { const float eb = bi[339];
              o35_9 = fmaf(eb, g9_12, o35_9);
            }
            { const float eb = bi[340];
              o35_9 = fmaf(eb, g9_22, o35_9);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk9 = PT[(fI + 2) * N + fJ + 1];
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
            const double Abd0_1 = PA[(fQ + 0) * N + fJ + 1];
            const double Abd1_1 = PA[(fQ + 1) * N + fJ + 1];
            const double Abd2_1 = PA[(fQ + 2) * N + fJ + 1];
            const double Abd3_1 = PA[(fQ + 3) * N + fJ + 1];
            const double Abd4_1 = PA[(fQ + 4) * N + fJ + 1];
            const double Abd5_1 = PA[(fQ + 5) * N + fJ + 1];
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
            const double Abc4_2 = PA[(fQ + 4) * N + fI + 2];
            const double Abc5_2 = PA[(fQ + 5) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
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
            jab24 += o24_9 * ptk9;
            jab25 += o25_9 * ptk9;
            jab26 += o26_9 * ptk9;
            jab27 += o27_9 * ptk9;
            jab28 += o28_9 * ptk9;
            jab29 += o29_9 * ptk9;
            jab30 += o30_9 * ptk9;
            jab31 += o31_9 * ptk9;
            jab32 += o32_9 * ptk9;
            jab33 += o33_9 * ptk9;
            jab34 += o34_9 * ptk9;
            jab35 += o35_9 * ptk9;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 1, 2.0 * deg * (o0_9 * ptb0 + o1_9 * ptb1 + o2_9 * ptb2 + o3_9 * ptb3 + o4_9 * ptb4 + o5_9 * ptb5 + o6_9 * ptb6 + o7_9 * ptb7 + o8_9 * ptb8 + o9_9 * ptb9 + o10_9 * ptb10 + o11_9 * ptb11 + o12_9 * ptb12 + o13_9 * ptb13 + o14_9 * ptb14 + o15_9 * ptb15 + o16_9 * ptb16 + o17_9 * ptb17 + o18_9 * ptb18 + o19_9 * ptb19 + o20_9 * ptb20 + o21_9 * ptb21 + o22_9 * ptb22 + o23_9 * ptb23 + o24_9 * ptb24 + o25_9 * ptb25 + o26_9 * ptb26 + o27_9 * ptb27 + o28_9 * ptb28 + o29_9 * ptb29 + o30_9 * ptb30 + o31_9 * ptb31 + o32_9 * ptb32 + o33_9 * ptb33 + o34_9 * ptb34 + o35_9 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_9 * Abd0_1 + o1_9 * Abd1_1 + o2_9 * Abd2_1 + o3_9 * Abd3_1 + o4_9 * Abd4_1 + o5_9 * Abd5_1));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_9 * Aad0_1 + o6_9 * Aad1_1 + o12_9 * Aad2_1 + o18_9 * Aad3_1 + o24_9 * Aad4_1 + o30_9 * Aad5_1));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 1, deg * (o0_9 * Abc0_2 + o1_9 * Abc1_2 + o2_9 * Abc2_2 + o3_9 * Abc3_2 + o4_9 * Abc4_2 + o5_9 * Abc5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 1, deg * (o0_9 * Aac0_2 + o6_9 * Aac1_2 + o12_9 * Aac2_2 + o18_9 * Aac3_2 + o24_9 * Aac4_2 + o30_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_9 * Aad0_1 + o7_9 * Aad1_1 + o13_9 * Aad2_1 + o19_9 * Aad3_1 + o25_9 * Aad4_1 + o31_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 1, deg * (o1_9 * Aac0_2 + o7_9 * Aac1_2 + o13_9 * Aac2_2 + o19_9 * Aac3_2 + o25_9 * Aac4_2 + o31_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_9 * Aad0_1 + o8_9 * Aad1_1 + o14_9 * Aad2_1 + o20_9 * Aad3_1 + o26_9 * Aad4_1 + o32_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 1, deg * (o2_9 * Aac0_2 + o8_9 * Aac1_2 + o14_9 * Aac2_2 + o20_9 * Aac3_2 + o26_9 * Aac4_2 + o32_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_9 * Aad0_1 + o9_9 * Aad1_1 + o15_9 * Aad2_1 + o21_9 * Aad3_1 + o27_9 * Aad4_1 + o33_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 1, deg * (o3_9 * Aac0_2 + o9_9 * Aac1_2 + o15_9 * Aac2_2 + o21_9 * Aac3_2 + o27_9 * Aac4_2 + o33_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 2, deg * (o4_9 * Aad0_1 + o10_9 * Aad1_1 + o16_9 * Aad2_1 + o22_9 * Aad3_1 + o28_9 * Aad4_1 + o34_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 1, deg * (o4_9 * Aac0_2 + o10_9 * Aac1_2 + o16_9 * Aac2_2 + o22_9 * Aac3_2 + o28_9 * Aac4_2 + o34_9 * Aac5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 2, deg * (o5_9 * Aad0_1 + o11_9 * Aad1_1 + o17_9 * Aad2_1 + o23_9 * Aad3_1 + o29_9 * Aad4_1 + o35_9 * Aad5_1));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 1, deg * (o5_9 * Aac0_2 + o11_9 * Aac1_2 + o17_9 * Aac2_2 + o23_9 * Aac3_2 + o29_9 * Aac4_2 + o35_9 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o6_9 * Abd0_1 + o7_9 * Abd1_1 + o8_9 * Abd2_1 + o9_9 * Abd3_1 + o10_9 * Abd4_1 + o11_9 * Abd5_1));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 1, deg * (o6_9 * Abc0_2 + o7_9 * Abc1_2 + o8_9 * Abc2_2 + o9_9 * Abc3_2 + o10_9 * Abc4_2 + o11_9 * Abc5_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o12_9 * Abd0_1 + o13_9 * Abd1_1 + o14_9 * Abd2_1 + o15_9 * Abd3_1 + o16_9 * Abd4_1 + o17_9 * Abd5_1));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 1, deg * (o12_9 * Abc0_2 + o13_9 * Abc1_2 + o14_9 * Abc2_2 + o15_9 * Abc3_2 + o16_9 * Abc4_2 + o17_9 * Abc5_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o18_9 * Abd0_1 + o19_9 * Abd1_1 + o20_9 * Abd2_1 + o21_9 * Abd3_1 + o22_9 * Abd4_1 + o23_9 * Abd5_1));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 1, deg * (o18_9 * Abc0_2 + o19_9 * Abc1_2 + o20_9 * Abc2_2 + o21_9 * Abc3_2 + o22_9 * Abc4_2 + o23_9 * Abc5_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o24_9 * Abd0_1 + o25_9 * Abd1_1 + o26_9 * Abd2_1 + o27_9 * Abd3_1 + o28_9 * Abd4_1 + o29_9 * Abd5_1));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 1, deg * (o24_9 * Abc0_2 + o25_9 * Abc1_2 + o26_9 * Abc2_2 + o27_9 * Abc3_2 + o28_9 * Abc4_2 + o29_9 * Abc5_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o30_9 * Abd0_1 + o31_9 * Abd1_1 + o32_9 * Abd2_1 + o33_9 * Abd3_1 + o34_9 * Abd4_1 + o35_9 * Abd5_1));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 1, deg * (o30_9 * Abc0_2 + o31_9 * Abc1_2 + o32_9 * Abc2_2 + o33_9 * Abc3_2 + o34_9 * Abc4_2 + o35_9 * Abc5_2));
          }
        } break;
        case 10: {  // ket functions [10]
          float o0_10 = 0;
          float o1_10 = 0;
          float o2_10 = 0;
          float o3_10 = 0;
          float o4_10 = 0;
          float o5_10 = 0;
          float o6_10 = 0;
          float o7_10 = 0;
          float o8_10 = 0;
          float o9_10 = 0;
          float o10_10 = 0;
          float o11_10 = 0;
          float o12_10 = 0;
          float o13_10 = 0;
          float o14_10 = 0;
          float o15_10 = 0;
          float o16_10 = 0;
          float o17_10 = 0;
          float o18_10 = 0;
          float o19_10 = 0;
          float o20_10 = 0;
          float o21_10 = 0;
          float o22_10 = 0;
          float o23_10 = 0;
          float o24_10 = 0;
          float o25_10 = 0;
          float o26_10 = 0;
          float o27_10 = 0;
          float o28_10 = 0;
          float o29_10 = 0;
          float o30_10 = 0;
          float o31_10 = 0;
          float o32_10 = 0;
          float o33_10 = 0;
          float o34_10 = 0;
          float o35_10 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g10_0 = 0;
            float g10_1 = 0;
            float g10_2 = 0;
            float g10_3 = 0;
            float g10_4 = 0;
            float g10_5 = 0;
            float g10_6 = 0;
            float g10_7 = 0;
            float g10_8 = 0;
            float g10_9 = 0;
            float g10_10 = 0;
            float g10_11 = 0;
            float g10_12 = 0;
            float g10_13 = 0;
            float g10_14 = 0;
            float g10_15 = 0;
            float g10_16 = 0;
            float g10_17 = 0;
            float g10_18 = 0;
            float g10_19 = 0;
            float g10_20 = 0;
            float g10_21 = 0;
            float g10_22 = 0;
            float g10_23 = 0;
            float g10_24 = 0;
            float g10_25 = 0;
            float g10_26 = 0;
            float g10_27 = 0;
            float g10_28 = 0;
            float g10_29 = 0;
            float g10_30 = 0;
            float g10_31 = 0;
            float g10_32 = 0;
            float g10_33 = 0;
            float g10_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek10_0 = kj[37 * kS];
              const float ek10_1 = -kj[38 * kS];
              const float ek10_2 = -kj[39 * kS];
              const float ek10_3 = kj[40 * kS];
              g10_0 = fmaf(ek10_0, b0, g10_0);
              const float r0_0_0_1 = Z * b1;
              g10_1 = fmaf(ek10_0, r0_0_0_1, g10_1);
              g10_0 = fmaf(ek10_1, r0_0_0_1, g10_0);
              const float r0_0_1_0 = Y * b1;
              g10_2 = fmaf(ek10_0, r0_0_1_0, g10_2);
              g10_0 = fmaf(ek10_2, r0_0_1_0, g10_0);
              const float r0_1_0_0 = X * b1;
              g10_3 = fmaf(ek10_0, r0_1_0_0, g10_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g10_4 = fmaf(ek10_0, r0_0_0_2, g10_4);
              g10_1 = fmaf(ek10_1, r0_0_0_2, g10_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g10_5 = fmaf(ek10_0, r0_0_1_1, g10_5);
              g10_2 = fmaf(ek10_1, r0_0_1_1, g10_2);
              g10_1 = fmaf(ek10_2, r0_0_1_1, g10_1);
              g10_0 = fmaf(ek10_3, r0_0_1_1, g10_0);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g10_6 = fmaf(ek10_0, r0_0_2_0, g10_6);
              g10_2 = fmaf(ek10_2, r0_0_2_0, g10_2);
              const float r0_1_0_1 = X * r1_0_0_1;
              g10_7 = fmaf(ek10_0, r0_1_0_1, g10_7);
              g10_3 = fmaf(ek10_1, r0_1_0_1, g10_3);
              const float r0_1_1_0 = X * r1_0_1_0;
              g10_8 = fmaf(ek10_0, r0_1_1_0, g10_8);
              g10_3 = fmaf(ek10_2, r0_1_1_0, g10_3);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g10_9 = fmaf(ek10_0, r0_2_0_0, g10_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g10_10 = fmaf(ek10_0, r0_0_0_3, g10_10);
              g10_4 = fmaf(ek10_1, r0_0_0_3, g10_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g10_11 = fmaf(ek10_0, r0_0_1_2, g10_11);
              g10_5 = fmaf(ek10_1, r0_0_1_2, g10_5);
              g10_4 = fmaf(ek10_2, r0_0_1_2, g10_4);
              g10_1 = fmaf(ek10_3, r0_0_1_2, g10_1);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g10_12 = fmaf(ek10_0, r0_0_2_1, g10_12);
              g10_6 = fmaf(ek10_1, r0_0_2_1, g10_6);
              g10_5 = fmaf(ek10_2, r0_0_2_1, g10_5);
              g10_2 = fmaf(ek10_3, r0_0_2_1, g10_2);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g10_13 = fmaf(ek10_0, r0_0_3_0, g10_13);
              g10_6 = fmaf(ek10_2, r0_0_3_0, g10_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g10_14 = fmaf(ek10_0, r0_1_0_2, g10_14);
              g10_7 = fmaf(ek10_1, r0_1_0_2, g10_7);
              const float r0_1_1_1 = X * r1_0_1_1;
              g10_15 = fmaf(ek10_0, r0_1_1_1, g10_15);
              g10_8 = fmaf(ek10_1, r0_1_1_1, g10_8);
              g10_7 = fmaf(ek10_2, r0_1_1_1, g10_7);
              g10_3 = fmaf(ek10_3, r0_1_1_1, g10_3);
              const float r0_1_2_0 = X * r1_0_2_0;
              g10_16 = fmaf(ek10_0, r0_1_2_0, g10_16);
              g10_8 = fmaf(ek10_2, r0_1_2_0, g10_8);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g10_17 = fmaf(ek10_0, r0_2_0_1, g10_17);
              g10_9 = fmaf(ek10_1, r0_2_0_1, g10_9);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g10_18 = fmaf(ek10_0, r0_2_1_0, g10_18);
              g10_9 = fmaf(ek10_2, r0_2_1_0, g10_9);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g10_19 = fmaf(ek10_0, r0_3_0_0, g10_19);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g10_20 = fmaf(ek10_0, r0_0_0_4, g10_20);
              g10_10 = fmaf(ek10_1, r0_0_0_4, g10_10);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g10_21 = fmaf(ek10_0, r0_0_1_3, g10_21);
              g10_11 = fmaf(ek10_1, r0_0_1_3, g10_11);
              g10_10 = fmaf(ek10_2, r0_0_1_3, g10_10);
              g10_4 = fmaf(ek10_3, r0_0_1_3, g10_4);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g10_22 = fmaf(ek10_0, r0_0_2_2, g10_22);
              g10_12 = fmaf(ek10_1, r0_0_2_2, g10_12);
              g10_11 = fmaf(ek10_2, r0_0_2_2, g10_11);
              g10_5 = fmaf(ek10_3, r0_0_2_2, g10_5);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g10_23 = fmaf(ek10_0, r0_0_3_1, g10_23);
              g10_13 = fmaf(ek10_1, r0_0_3_1, g10_13);
              g10_12 = fmaf(ek10_2, r0_0_3_1, g10_12);
              g10_6 = fmaf(ek10_3, r0_0_3_1, g10_6);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g10_24 = fmaf(ek10_0, r0_0_4_0, g10_24);
              g10_13 = fmaf(ek10_2, r0_0_4_0, g10_13);
              const float r0_1_0_3 = X * r1_0_0_3;
              g10_25 = fmaf(ek10_0, r0_1_0_3, g10_25);
              g10_14 = fmaf(ek10_1, r0_1_0_3, g10_14);
              const float r0_1_1_2 = X * r1_0_1_2;
              g10_26 = fmaf(ek10_0, r0_1_1_2, g10_26);
              g10_15 = fmaf(ek10_1, r0_1_1_2, g10_15);
              g10_14 = fmaf(ek10_2, r0_1_1_2, g10_14);
              g10_7 = fmaf(ek10_3, r0_1_1_2, g10_7);
              const float r0_1_2_1 = X * r1_0_2_1;
              g10_27 = fmaf(ek10_0, r0_1_2_1, g10_27);
              g10_16 = fmaf(ek10_1, r0_1_2_1, g10_16);
              g10_15 = fmaf(ek10_2, r0_1_2_1, g10_15);
              g10_8 = fmaf(ek10_3, r0_1_2_1, g10_8);
              const float r0_1_3_0 = X * r1_0_3_0;
              g10_28 = fmaf(ek10_0, r0_1_3_0, g10_28);
              g10_16 = fmaf(ek10_2, r0_1_3_0, g10_16);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g10_29 = fmaf(ek10_0, r0_2_0_2, g10_29);
              g10_17 = fmaf(ek10_1, r0_2_0_2, g10_17);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g10_30 = fmaf(ek10_0, r0_2_1_1, g10_30);
              g10_18 = fmaf(ek10_1, r0_2_1_1, g10_18);
              g10_17 = fmaf(ek10_2, r0_2_1_1, g10_17);
              g10_9 = fmaf(ek10_3, r0_2_1_1, g10_9);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g10_31 = fmaf(ek10_0, r0_2_2_0, g10_31);
              g10_18 = fmaf(ek10_2, r0_2_2_0, g10_18);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g10_32 = fmaf(ek10_0, r0_3_0_1, g10_32);
              g10_19 = fmaf(ek10_1, r0_3_0_1, g10_19);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g10_33 = fmaf(ek10_0, r0_3_1_0, g10_33);
              g10_19 = fmaf(ek10_2, r0_3_1_0, g10_19);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g10_34 = fmaf(ek10_0, r0_4_0_0, g10_34);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_0_5 = fmaf(Z, r1_0_0_4, 4.0f * r1_0_0_3);
              g10_20 = fmaf(ek10_1, r0_0_0_5, g10_20);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g10_21 = fmaf(ek10_1, r0_0_1_4, g10_21);
              g10_20 = fmaf(ek10_2, r0_0_1_4, g10_20);
              g10_10 = fmaf(ek10_3, r0_0_1_4, g10_10);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g10_22 = fmaf(ek10_1, r0_0_2_3, g10_22);
              g10_21 = fmaf(ek10_2, r0_0_2_3, g10_21);
              g10_11 = fmaf(ek10_3, r0_0_2_3, g10_11);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g10_23 = fmaf(ek10_1, r0_0_3_2, g10_23);
              g10_22 = fmaf(ek10_2, r0_0_3_2, g10_22);
              g10_12 = fmaf(ek10_3, r0_0_3_2, g10_12);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g10_24 = fmaf(ek10_1, r0_0_4_1, g10_24);
              g10_23 = fmaf(ek10_2, r0_0_4_1, g10_23);
              g10_13 = fmaf(ek10_3, r0_0_4_1, g10_13);
              const float r4_0_1_0 = Y * b5;
              const float r3_0_2_0 = fmaf(Y, r4_0_1_0, b4);
              const float r2_0_3_0 = fmaf(Y, r3_0_2_0, 2.0f * r3_0_1_0);
              const float r1_0_4_0 = fmaf(Y, r2_0_3_0, 3.0f * r2_0_2_0);
              const float r0_0_5_0 = fmaf(Y, r1_0_4_0, 4.0f * r1_0_3_0);
              g10_24 = fmaf(ek10_2, r0_0_5_0, g10_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g10_25 = fmaf(ek10_1, r0_1_0_4, g10_25);
              const float r0_1_1_3 = X * r1_0_1_3;
              g10_26 = fmaf(ek10_1, r0_1_1_3, g10_26);
              g10_25 = fmaf(ek10_2, r0_1_1_3, g10_25);
              g10_14 = fmaf(ek10_3, r0_1_1_3, g10_14);
              const float r0_1_2_2 = X * r1_0_2_2;
              g10_27 = fmaf(ek10_1, r0_1_2_2, g10_27);
              g10_26 = fmaf(ek10_2, r0_1_2_2, g10_26);
              g10_15 = fmaf(ek10_3, r0_1_2_2, g10_15);
              const float r0_1_3_1 = X * r1_0_3_1;
              g10_28 = fmaf(ek10_1, r0_1_3_1, g10_28);
              g10_27 = fmaf(ek10_2, r0_1_3_1, g10_27);
              g10_16 = fmaf(ek10_3, r0_1_3_1, g10_16);
              const float r0_1_4_0 = X * r1_0_4_0;
              g10_28 = fmaf(ek10_2, r0_1_4_0, g10_28);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g10_29 = fmaf(ek10_1, r0_2_0_3, g10_29);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g10_30 = fmaf(ek10_1, r0_2_1_2, g10_30);
              g10_29 = fmaf(ek10_2, r0_2_1_2, g10_29);
              g10_17 = fmaf(ek10_3, r0_2_1_2, g10_17);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g10_31 = fmaf(ek10_1, r0_2_2_1, g10_31);
              g10_30 = fmaf(ek10_2, r0_2_2_1, g10_30);
              g10_18 = fmaf(ek10_3, r0_2_2_1, g10_18);
              const float r1_1_3_0 = X * r2_0_3_0;
              const float r0_2_3_0 = fmaf(X, r1_1_3_0, r1_0_3_0);
              g10_31 = fmaf(ek10_2, r0_2_3_0, g10_31);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g10_32 = fmaf(ek10_1, r0_3_0_2, g10_32);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g10_33 = fmaf(ek10_1, r0_3_1_1, g10_33);
              g10_32 = fmaf(ek10_2, r0_3_1_1, g10_32);
              g10_19 = fmaf(ek10_3, r0_3_1_1, g10_19);
              const float r2_1_2_0 = X * r3_0_2_0;
              const float r1_2_2_0 = fmaf(X, r2_1_2_0, r2_0_2_0);
              const float r0_3_2_0 = fmaf(X, r1_2_2_0, 2.0f * r1_1_2_0);
              g10_33 = fmaf(ek10_2, r0_3_2_0, g10_33);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g10_34 = fmaf(ek10_1, r0_4_0_1, g10_34);
              const float r3_1_1_0 = X * r4_0_1_0;
              const float r2_2_1_0 = fmaf(X, r3_1_1_0, r3_0_1_0);
              const float r1_3_1_0 = fmaf(X, r2_2_1_0, 2.0f * r2_1_1_0);
              const float r0_4_1_0 = fmaf(X, r1_3_1_0, 3.0f * r1_2_1_0);
              g10_34 = fmaf(ek10_2, r0_4_1_0, g10_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_0_5 = fmaf(Z, r2_0_0_4, 4.0f * r2_0_0_3);
              const float r0_0_1_5 = Y * r1_0_0_5;
              g10_20 = fmaf(ek10_3, r0_0_1_5, g10_20);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_0_2_4 = fmaf(Y, r1_0_1_4, r1_0_0_4);
              g10_21 = fmaf(ek10_3, r0_0_2_4, g10_21);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_0_3_3 = fmaf(Y, r1_0_2_3, 2.0f * r1_0_1_3);
              g10_22 = fmaf(ek10_3, r0_0_3_3, g10_22);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_0_4_2 = fmaf(Y, r1_0_3_2, 3.0f * r1_0_2_2);
              g10_23 = fmaf(ek10_3, r0_0_4_2, g10_23);
              const float r4_0_1_1 = Y * r5_0_0_1;
              const float r3_0_2_1 = fmaf(Y, r4_0_1_1, r4_0_0_1);
              const float r2_0_3_1 = fmaf(Y, r3_0_2_1, 2.0f * r3_0_1_1);
              const float r1_0_4_1 = fmaf(Y, r2_0_3_1, 3.0f * r2_0_2_1);
              const float r0_0_5_1 = fmaf(Y, r1_0_4_1, 4.0f * r1_0_3_1);
              g10_24 = fmaf(ek10_3, r0_0_5_1, g10_24);
              const float r0_1_1_4 = X * r1_0_1_4;
              g10_25 = fmaf(ek10_3, r0_1_1_4, g10_25);
              const float r0_1_2_3 = X * r1_0_2_3;
              g10_26 = fmaf(ek10_3, r0_1_2_3, g10_26);
              const float r0_1_3_2 = X * r1_0_3_2;
              g10_27 = fmaf(ek10_3, r0_1_3_2, g10_27);
              const float r0_1_4_1 = X * r1_0_4_1;
              g10_28 = fmaf(ek10_3, r0_1_4_1, g10_28);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g10_29 = fmaf(ek10_3, r0_2_1_3, g10_29);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g10_30 = fmaf(ek10_3, r0_2_2_2, g10_30);
              const float r1_1_3_1 = X * r2_0_3_1;
              const float r0_2_3_1 = fmaf(X, r1_1_3_1, r1_0_3_1);
              g10_31 = fmaf(ek10_3, r0_2_3_1, g10_31);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g10_32 = fmaf(ek10_3, r0_3_1_2, g10_32);
              const float r2_1_2_1 = X * r3_0_2_1;
              const float r1_2_2_1 = fmaf(X, r2_1_2_1, r2_0_2_1);
              const float r0_3_2_1 = fmaf(X, r1_2_2_1, 2.0f * r1_1_2_1);
              g10_33 = fmaf(ek10_3, r0_3_2_1, g10_33);
              const float r3_1_1_1 = X * r4_0_1_1;
              const float r2_2_1_1 = fmaf(X, r3_1_1_1, r3_0_1_1);
              const float r1_3_1_1 = fmaf(X, r2_2_1_1, 2.0f * r2_1_1_1);
              const float r0_4_1_1 = fmaf(X, r1_3_1_1, 3.0f * r1_2_1_1);
              g10_34 = fmaf(ek10_3, r0_4_1_1, g10_34);
            }
            { const float eb = bi[5];
              o0_10 = fmaf(eb, g10_0, o0_10);
            }
            { const float eb = bi[6];
              o0_10 = fmaf(eb, g10_3, o0_10);
            }
            { const float eb = bi[7];
              o0_10 = fmaf(eb, g10_9, o0_10);
            }
            { const float eb = bi[8];
              o0_10 = fmaf(eb, g10_19, o0_10);
            }
            { const float eb = bi[9];
              o0_10 = fmaf(eb, g10_34, o0_10);
            }
            { const float eb = bi[10];
              o1_10 = fmaf(eb, g10_0, o1_10);
            }
            { const float eb = bi[11];
              o1_10 = fmaf(eb, g10_2, o1_10);
            }
            { const float eb = bi[12];
              o1_10 = fmaf(eb, g10_6, o1_10);
            }
            { const float eb = bi[13];
              o1_10 = fmaf(eb, g10_3, o1_10);
            }
            { const float eb = bi[14];
              o1_10 = fmaf(eb, g10_8, o1_10);
            }
            { const float eb = bi[15];
              o1_10 = fmaf(eb, g10_16, o1_10);
            }
            { const float eb = bi[16];
              o1_10 = fmaf(eb, g10_9, o1_10);
            }
            { const float eb = bi[17];
              o1_10 = fmaf(eb, g10_18, o1_10);
            }
            { const float eb = bi[18];
              o1_10 = fmaf(eb, g10_31, o1_10);
            }
            { const float eb = bi[19];
              o2_10 = fmaf(eb, g10_0, o2_10);
            }
            { const float eb = bi[20];
              o2_10 = fmaf(eb, g10_1, o2_10);
            }
            { const float eb = bi[21];
              o2_10 = fmaf(eb, g10_4, o2_10);
            }
            { const float eb = bi[22];
              o2_10 = fmaf(eb, g10_3, o2_10);
            }
            { const float eb = bi[23];
              o2_10 = fmaf(eb, g10_7, o2_10);
            }
            { const float eb = bi[24];
              o2_10 = fmaf(eb, g10_14, o2_10);
            }
            { const float eb = bi[25];
              o2_10 = fmaf(eb, g10_9, o2_10);
            }
            { const float eb = bi[26];
              o2_10 = fmaf(eb, g10_17, o2_10);
            }
            { const float eb = bi[27];
              o2_10 = fmaf(eb, g10_29, o2_10);
            }
            { const float eb = bi[28];
              o3_10 = fmaf(eb, g10_0, o3_10);
            }
            { const float eb = bi[29];
              o3_10 = fmaf(eb, g10_2, o3_10);
            }
            { const float eb = bi[30];
              o3_10 = fmaf(eb, g10_3, o3_10);
            }
            { const float eb = bi[31];
              o3_10 = fmaf(eb, g10_8, o3_10);
            }
            { const float eb = bi[32];
              o3_10 = fmaf(eb, g10_9, o3_10);
            }
            { const float eb = bi[33];
              o3_10 = fmaf(eb, g10_18, o3_10);
            }
            { const float eb = bi[34];
              o3_10 = fmaf(eb, g10_19, o3_10);
            }
            { const float eb = bi[35];
              o3_10 = fmaf(eb, g10_33, o3_10);
            }
            { const float eb = bi[36];
              o4_10 = fmaf(eb, g10_0, o4_10);
            }
            { const float eb = bi[37];
              o4_10 = fmaf(eb, g10_1, o4_10);
            }
            { const float eb = bi[38];
              o4_10 = fmaf(eb, g10_3, o4_10);
            }
            { const float eb = bi[39];
              o4_10 = fmaf(eb, g10_7, o4_10);
            }
            { const float eb = bi[40];
              o4_10 = fmaf(eb, g10_9, o4_10);
            }
            { const float eb = bi[41];
              o4_10 = fmaf(eb, g10_17, o4_10);
            }
            { const float eb = bi[42];
              o4_10 = fmaf(eb, g10_19, o4_10);
            }
            { const float eb = bi[43];
              o4_10 = fmaf(eb, g10_32, o4_10);
            }
            { const float eb = bi[44];
              o5_10 = fmaf(eb, g10_0, o5_10);
            }
            { const float eb = bi[45];
              o5_10 = fmaf(eb, g10_1, o5_10);
            }
            { const float eb = bi[46];
              o5_10 = fmaf(eb, g10_2, o5_10);
            }
            { const float eb = bi[47];
              o5_10 = fmaf(eb, g10_5, o5_10);
            }
            { const float eb = bi[48];
              o5_10 = fmaf(eb, g10_3, o5_10);
            }
            { const float eb = bi[49];
              o5_10 = fmaf(eb, g10_7, o5_10);
            }
            { const float eb = bi[50];
              o5_10 = fmaf(eb, g10_8, o5_10);
            }
            { const float eb = bi[51];
              o5_10 = fmaf(eb, g10_15, o5_10);
            }
            { const float eb = bi[52];
              o5_10 = fmaf(eb, g10_9, o5_10);
            }
            { const float eb = bi[53];
              o5_10 = fmaf(eb, g10_17, o5_10);
            }
            { const float eb = bi[54];
              o5_10 = fmaf(eb, g10_18, o5_10);
            }
            { const float eb = bi[55];
              o5_10 = fmaf(eb, g10_30, o5_10);
            }
            { const float eb = bi[56];
              o6_10 = fmaf(eb, g10_0, o6_10);
            }
            { const float eb = bi[57];
              o6_10 = fmaf(eb, g10_2, o6_10);
            }
            { const float eb = bi[58];
              o6_10 = fmaf(eb, g10_6, o6_10);
            }
            { const float eb = bi[59];
              o6_10 = fmaf(eb, g10_3, o6_10);
            }
            { const float eb = bi[60];
              o6_10 = fmaf(eb, g10_8, o6_10);
            }
            { const float eb = bi[61];
              o6_10 = fmaf(eb, g10_16, o6_10);
            }
            { const float eb = bi[62];
              o6_10 = fmaf(eb, g10_9, o6_10);
            }
            { const float eb = bi[63];
              o6_10 = fmaf(eb, g10_18, o6_10);
            }
            { const float eb = bi[64];
              o6_10 = fmaf(eb, g10_31, o6_10);
            }
            { const float eb = bi[65];
              o7_10 = fmaf(eb, g10_0, o7_10);
            }
            { const float eb = bi[66];
              o7_10 = fmaf(eb, g10_2, o7_10);
            }
            { const float eb = bi[67];
              o7_10 = fmaf(eb, g10_6, o7_10);
            }
            { const float eb = bi[68];
              o7_10 = fmaf(eb, g10_13, o7_10);
            }
            { const float eb = bi[69];
              o7_10 = fmaf(eb, g10_24, o7_10);
            }
            { const float eb = bi[70];
              o8_10 = fmaf(eb, g10_0, o8_10);
            }
            { const float eb = bi[71];
              o8_10 = fmaf(eb, g10_1, o8_10);
            }
            { const float eb = bi[72];
              o8_10 = fmaf(eb, g10_4, o8_10);
            }
            { const float eb = bi[73];
              o8_10 = fmaf(eb, g10_2, o8_10);
            }
            { const float eb = bi[74];
              o8_10 = fmaf(eb, g10_5, o8_10);
            }
            { const float eb = bi[75];
              o8_10 = fmaf(eb, g10_11, o8_10);
            }
            { const float eb = bi[76];
              o8_10 = fmaf(eb, g10_6, o8_10);
            }
            { const float eb = bi[77];
              o8_10 = fmaf(eb, g10_12, o8_10);
            }
            { const float eb = bi[78];
              o8_10 = fmaf(eb, g10_22, o8_10);
            }
            { const float eb = bi[79];
              o9_10 = fmaf(eb, g10_0, o9_10);
            }
            { const float eb = bi[80];
              o9_10 = fmaf(eb, g10_2, o9_10);
            }
            { const float eb = bi[81];
              o9_10 = fmaf(eb, g10_6, o9_10);
            }
            { const float eb = bi[82];
              o9_10 = fmaf(eb, g10_13, o9_10);
            }
            { const float eb = bi[83];
              o9_10 = fmaf(eb, g10_3, o9_10);
            }
            { const float eb = bi[84];
              o9_10 = fmaf(eb, g10_8, o9_10);
            }
            { const float eb = bi[85];
              o9_10 = fmaf(eb, g10_16, o9_10);
            }
            { const float eb = bi[86];
              o9_10 = fmaf(eb, g10_28, o9_10);
            }
            { const float eb = bi[87];
              o10_10 = fmaf(eb, g10_0, o10_10);
            }
            { const float eb = bi[88];
              o10_10 = fmaf(eb, g10_1, o10_10);
            }
            { const float eb = bi[89];
              o10_10 = fmaf(eb, g10_2, o10_10);
            }
            { const float eb = bi[90];
              o10_10 = fmaf(eb, g10_5, o10_10);
            }
            { const float eb = bi[91];
              o10_10 = fmaf(eb, g10_6, o10_10);
            }
            { const float eb = bi[92];
              o10_10 = fmaf(eb, g10_12, o10_10);
            }
            { const float eb = bi[93];
              o10_10 = fmaf(eb, g10_3, o10_10);
            }
            { const float eb = bi[94];
              o10_10 = fmaf(eb, g10_7, o10_10);
            }
            { const float eb = bi[95];
              o10_10 = fmaf(eb, g10_8, o10_10);
            }
            { const float eb = bi[96];
              o10_10 = fmaf(eb, g10_15, o10_10);
            }
            { const float eb = bi[97];
              o10_10 = fmaf(eb, g10_16, o10_10);
            }
            { const float eb = bi[98];
              o10_10 = fmaf(eb, g10_27, o10_10);
            }
            { const float eb = bi[99];
              o11_10 = fmaf(eb, g10_0, o11_10);
            }
            { const float eb = bi[100];
              o11_10 = fmaf(eb, g10_1, o11_10);
            }
            { const float eb = bi[101];
              o11_10 = fmaf(eb, g10_2, o11_10);
            }
            { const float eb = bi[102];
              o11_10 = fmaf(eb, g10_5, o11_10);
            }
            { const float eb = bi[103];
              o11_10 = fmaf(eb, g10_6, o11_10);
            }
            { const float eb = bi[104];
              o11_10 = fmaf(eb, g10_12, o11_10);
            }
            { const float eb = bi[105];
              o11_10 = fmaf(eb, g10_13, o11_10);
            }
            { const float eb = bi[106];
              o11_10 = fmaf(eb, g10_23, o11_10);
            }
            { const float eb = bi[107];
              o12_10 = fmaf(eb, g10_0, o12_10);
            }
            { const float eb = bi[108];
              o12_10 = fmaf(eb, g10_1, o12_10);
            }
            { const float eb = bi[109];
              o12_10 = fmaf(eb, g10_4, o12_10);
            }
            { const float eb = bi[110];
              o12_10 = fmaf(eb, g10_3, o12_10);
            }
            { const float eb = bi[111];
              o12_10 = fmaf(eb, g10_7, o12_10);
            }
            { const float eb = bi[112];
              o12_10 = fmaf(eb, g10_14, o12_10);
            }
            { const float eb = bi[113];
              o12_10 = fmaf(eb, g10_9, o12_10);
            }
            { const float eb = bi[114];
              o12_10 = fmaf(eb, g10_17, o12_10);
            }
            { const float eb = bi[115];
              o12_10 = fmaf(eb, g10_29, o12_10);
            }
            { const float eb = bi[116];
              o13_10 = fmaf(eb, g10_0, o13_10);
            }
            { const float eb = bi[117];
              o13_10 = fmaf(eb, g10_1, o13_10);
            }
            { const float eb = bi[118];
              o13_10 = fmaf(eb, g10_4, o13_10);
            }
            { const float eb = bi[119];
              o13_10 = fmaf(eb, g10_2, o13_10);
            }
            { const float eb = bi[120];
              o13_10 = fmaf(eb, g10_5, o13_10);
            }
            { const float eb = bi[121];
              o13_10 = fmaf(eb, g10_11, o13_10);
            }
            { const float eb = bi[122];
              o13_10 = fmaf(eb, g10_6, o13_10);
            }
            { const float eb = bi[123];
              o13_10 = fmaf(eb, g10_12, o13_10);
            }
            { const float eb = bi[124];
              o13_10 = fmaf(eb, g10_22, o13_10);
            }
            { const float eb = bi[125];
              o14_10 = fmaf(eb, g10_0, o14_10);
            }
            { const float eb = bi[126];
              o14_10 = fmaf(eb, g10_1, o14_10);
            }
            { const float eb = bi[127];
              o14_10 = fmaf(eb, g10_4, o14_10);
            }
            { const float eb = bi[128];
              o14_10 = fmaf(eb, g10_10, o14_10);
            }
            { const float eb = bi[129];
              o14_10 = fmaf(eb, g10_20, o14_10);
            }
            { const float eb = bi[130];
              o15_10 = fmaf(eb, g10_0, o15_10);
            }
            { const float eb = bi[131];
              o15_10 = fmaf(eb, g10_1, o15_10);
            }
            { const float eb = bi[132];
              o15_10 = fmaf(eb, g10_4, o15_10);
            }
            { const float eb = bi[133];
              o15_10 = fmaf(eb, g10_2, o15_10);
            }
            { const float eb = bi[134];
              o15_10 = fmaf(eb, g10_5, o15_10);
            }
            { const float eb = bi[135];
              o15_10 = fmaf(eb, g10_11, o15_10);
            }
            { const float eb = bi[136];
              o15_10 = fmaf(eb, g10_3, o15_10);
            }
            { const float eb = bi[137];
              o15_10 = fmaf(eb, g10_7, o15_10);
            }
            { const float eb = bi[138];
              o15_10 = fmaf(eb, g10_14, o15_10);
            }
            { const float eb = bi[139];
              o15_10 = fmaf(eb, g10_8, o15_10);
            }
            { const float eb = bi[140];
              o15_10 = fmaf(eb, g10_15, o15_10);
            }
            { const float eb = bi[141];
              o15_10 = fmaf(eb, g10_26, o15_10);
            }
            { const float eb = bi[142];
              o16_10 = fmaf(eb, g10_0, o16_10);
            }
            { const float eb = bi[143];
              o16_10 = fmaf(eb, g10_1, o16_10);
            }
            { const float eb = bi[144];
              o16_10 = fmaf(eb, g10_4, o16_10);
            }
            { const float eb = bi[145];
              o16_10 = fmaf(eb, g10_10, o16_10);
            }
            { const float eb = bi[146];
              o16_10 = fmaf(eb, g10_3, o16_10);
            }
            { const float eb = bi[147];
              o16_10 = fmaf(eb, g10_7, o16_10);
            }
            { const float eb = bi[148];
              o16_10 = fmaf(eb, g10_14, o16_10);
            }
            { const float eb = bi[149];
              o16_10 = fmaf(eb, g10_25, o16_10);
            }
            { const float eb = bi[150];
              o17_10 = fmaf(eb, g10_0, o17_10);
            }
            { const float eb = bi[151];
              o17_10 = fmaf(eb, g10_1, o17_10);
            }
            { const float eb = bi[152];
              o17_10 = fmaf(eb, g10_4, o17_10);
            }
            { const float eb = bi[153];
              o17_10 = fmaf(eb, g10_10, o17_10);
            }
            { const float eb = bi[154];
              o17_10 = fmaf(eb, g10_2, o17_10);
            }
            { const float eb = bi[155];
              o17_10 = fmaf(eb, g10_5, o17_10);
            }
            { const float eb = bi[156];
              o17_10 = fmaf(eb, g10_11, o17_10);
            }
            { const float eb = bi[157];
              o17_10 = fmaf(eb, g10_21, o17_10);
            }
            { const float eb = bi[158];
              o18_10 = fmaf(eb, g10_0, o18_10);
            }
            { const float eb = bi[159];
              o18_10 = fmaf(eb, g10_2, o18_10);
            }
            { const float eb = bi[160];
              o18_10 = fmaf(eb, g10_3, o18_10);
            }
            { const float eb = bi[161];
              o18_10 = fmaf(eb, g10_8, o18_10);
            }
            { const float eb = bi[162];
              o18_10 = fmaf(eb, g10_9, o18_10);
            }
            { const float eb = bi[163];
              o18_10 = fmaf(eb, g10_18, o18_10);
            }
            { const float eb = bi[164];
              o18_10 = fmaf(eb, g10_19, o18_10);
            }
            { const float eb = bi[165];
              o18_10 = fmaf(eb, g10_33, o18_10);
            }
            { const float eb = bi[166];
              o19_10 = fmaf(eb, g10_0, o19_10);
            }
            { const float eb = bi[167];
              o19_10 = fmaf(eb, g10_2, o19_10);
            }
            { const float eb = bi[168];
              o19_10 = fmaf(eb, g10_6, o19_10);
            }
            { const float eb = bi[169];
              o19_10 = fmaf(eb, g10_13, o19_10);
            }
            { const float eb = bi[170];
              o19_10 = fmaf(eb, g10_3, o19_10);
            }
            { const float eb = bi[171];
              o19_10 = fmaf(eb, g10_8, o19_10);
            }
            { const float eb = bi[172];
              o19_10 = fmaf(eb, g10_16, o19_10);
            }
            { const float eb = bi[173];
              o19_10 = fmaf(eb, g10_28, o19_10);
            }
            { const float eb = bi[174];
              o20_10 = fmaf(eb, g10_0, o20_10);
            }
            { const float eb = bi[175];
              o20_10 = fmaf(eb, g10_1, o20_10);
            }
            { const float eb = bi[176];
              o20_10 = fmaf(eb, g10_4, o20_10);
            }
            { const float eb = bi[177];
              o20_10 = fmaf(eb, g10_2, o20_10);
            }
            { const float eb = bi[178];
              o20_10 = fmaf(eb, g10_5, o20_10);
            }
            { const float eb = bi[179];
              o20_10 = fmaf(eb, g10_11, o20_10);
            }
            { const float eb = bi[180];
              o20_10 = fmaf(eb, g10_3, o20_10);
            }
            { const float eb = bi[181];
              o20_10 = fmaf(eb, g10_7, o20_10);
            }
            { const float eb = bi[182];
              o20_10 = fmaf(eb, g10_14, o20_10);
            }
            { const float eb = bi[183];
              o20_10 = fmaf(eb, g10_8, o20_10);
            }
            { const float eb = bi[184];
              o20_10 = fmaf(eb, g10_15, o20_10);
            }
            { const float eb = bi[185];
              o20_10 = fmaf(eb, g10_26, o20_10);
            }
            { const float eb = bi[186];
              o21_10 = fmaf(eb, g10_0, o21_10);
            }
            { const float eb = bi[187];
              o21_10 = fmaf(eb, g10_2, o21_10);
            }
            { const float eb = bi[188];
              o21_10 = fmaf(eb, g10_6, o21_10);
            }
            { const float eb = bi[189];
              o21_10 = fmaf(eb, g10_3, o21_10);
            }
            { const float eb = bi[190];
              o21_10 = fmaf(eb, g10_8, o21_10);
            }
            { const float eb = bi[191];
              o21_10 = fmaf(eb, g10_16, o21_10);
            }
            { const float eb = bi[192];
              o21_10 = fmaf(eb, g10_9, o21_10);
            }
            { const float eb = bi[193];
              o21_10 = fmaf(eb, g10_18, o21_10);
            }
            { const float eb = bi[194];
              o21_10 = fmaf(eb, g10_31, o21_10);
            }
            { const float eb = bi[195];
              o22_10 = fmaf(eb, g10_0, o22_10);
            }
            { const float eb = bi[196];
              o22_10 = fmaf(eb, g10_1, o22_10);
            }
            { const float eb = bi[197];
              o22_10 = fmaf(eb, g10_2, o22_10);
            }
            { const float eb = bi[198];
              o22_10 = fmaf(eb, g10_5, o22_10);
            }
            { const float eb = bi[199];
              o22_10 = fmaf(eb, g10_3, o22_10);
            }
            { const float eb = bi[200];
              o22_10 = fmaf(eb, g10_7, o22_10);
            }
            { const float eb = bi[201];
              o22_10 = fmaf(eb, g10_8, o22_10);
            }
            { const float eb = bi[202];
              o22_10 = fmaf(eb, g10_15, o22_10);
            }
            { const float eb = bi[203];
              o22_10 = fmaf(eb, g10_9, o22_10);
            }
            { const float eb = bi[204];
              o22_10 = fmaf(eb, g10_17, o22_10);
            }
            { const float eb = bi[205];
              o22_10 = fmaf(eb, g10_18, o22_10);
            }
            { const float eb = bi[206];
              o22_10 = fmaf(eb, g10_30, o22_10);
            }
            { const float eb = bi[207];
              o23_10 = fmaf(eb, g10_0, o23_10);
            }
            { const float eb = bi[208];
              o23_10 = fmaf(eb, g10_1, o23_10);
            }
            { const float eb = bi[209];
              o23_10 = fmaf(eb, g10_2, o23_10);
            }
            { const float eb = bi[210];
              o23_10 = fmaf(eb, g10_5, o23_10);
            }
            { const float eb = bi[211];
              o23_10 = fmaf(eb, g10_6, o23_10);
            }
            { const float eb = bi[212];
              o23_10 = fmaf(eb, g10_12, o23_10);
            }
            { const float eb = bi[213];
              o23_10 = fmaf(eb, g10_3, o23_10);
            }
            { const float eb = bi[214];
              o23_10 = fmaf(eb, g10_7, o23_10);
            }
            { const float eb = bi[215];
              o23_10 = fmaf(eb, g10_8, o23_10);
            }
            { const float eb = bi[216];
              o23_10 = fmaf(eb, g10_15, o23_10);
            }
            { const float eb = bi[217];
              o23_10 = fmaf(eb, g10_16, o23_10);
            }
            { const float eb = bi[218];
              o23_10 = fmaf(eb, g10_27, o23_10);
            }
            { const float eb = bi[219];
              o24_10 = fmaf(eb, g10_0, o24_10);
            }
            { const float eb = bi[220];
              o24_10 = fmaf(eb, g10_1, o24_10);
            }
            { const float eb = bi[221];
              o24_10 = fmaf(eb, g10_3, o24_10);
            }
            { const float eb = bi[222];
              o24_10 = fmaf(eb, g10_7, o24_10);
            }
            { const float eb = bi[223];
              o24_10 = fmaf(eb, g10_9, o24_10);
            }
            { const float eb = bi[224];
              o24_10 = fmaf(eb, g10_17, o24_10);
            }
            { const float eb = bi[225];
              o24_10 = fmaf(eb, g10_19, o24_10);
            }
            { const float eb = bi[226];
              o24_10 = fmaf(eb, g10_32, o24_10);
            }
            { const float eb = bi[227];
              o25_10 = fmaf(eb, g10_0, o25_10);
            }
            { const float eb = bi[228];
              o25_10 = fmaf(eb, g10_1, o25_10);
            }
            { const float eb = bi[229];
              o25_10 = fmaf(eb, g10_2, o25_10);
            }
            { const float eb = bi[230];
              o25_10 = fmaf(eb, g10_5, o25_10);
            }
            { const float eb = bi[231];
              o25_10 = fmaf(eb, g10_6, o25_10);
            }
            { const float eb = bi[232];
              o25_10 = fmaf(eb, g10_12, o25_10);
            }
            { const float eb = bi[233];
              o25_10 = fmaf(eb, g10_3, o25_10);
            }
            { const float eb = bi[234];
              o25_10 = fmaf(eb, g10_7, o25_10);
            }
            { const float eb = bi[235];
              o25_10 = fmaf(eb, g10_8, o25_10);
            }
            { const float eb = bi[236];
              o25_10 = fmaf(eb, g10_15, o25_10);
            }
            { const float eb = bi[237];
              o25_10 = fmaf(eb, g10_16, o25_10);
            }
            { const float eb = bi[238];
              o25_10 = fmaf(eb, g10_27, o25_10);
            }
            { const float eb = bi[239];
              o26_10 = fmaf(eb, g10_0, o26_10);
            }
            { const float eb = bi[240];
              o26_10 = fmaf(eb, g10_1, o26_10);
            }
            { const float eb = bi[241];
              o26_10 = fmaf(eb, g10_4, o26_10);
            }
            { const float eb = bi[242];
              o26_10 = fmaf(eb, g10_10, o26_10);
            }
            { const float eb = bi[243];
              o26_10 = fmaf(eb, g10_3, o26_10);
            }
            { const float eb = bi[244];
              o26_10 = fmaf(eb, g10_7, o26_10);
            }
            { const float eb = bi[245];
              o26_10 = fmaf(eb, g10_14, o26_10);
            }
            { const float eb = bi[246];
              o26_10 = fmaf(eb, g10_25, o26_10);
            }
            { const float eb = bi[247];
              o27_10 = fmaf(eb, g10_0, o27_10);
            }
            { const float eb = bi[248];
              o27_10 = fmaf(eb, g10_1, o27_10);
            }
            { const float eb = bi[249];
              o27_10 = fmaf(eb, g10_2, o27_10);
            }
            { const float eb = bi[250];
              o27_10 = fmaf(eb, g10_5, o27_10);
            }
            { const float eb = bi[251];
              o27_10 = fmaf(eb, g10_3, o27_10);
            }
            { const float eb = bi[252];
              o27_10 = fmaf(eb, g10_7, o27_10);
            }
            { const float eb = bi[253];
              o27_10 = fmaf(eb, g10_8, o27_10);
            }
            { const float eb = bi[254];
              o27_10 = fmaf(eb, g10_15, o27_10);
            }
            { const float eb = bi[255];
              o27_10 = fmaf(eb, g10_9, o27_10);
            }
            { const float eb = bi[256];
              o27_10 = fmaf(eb, g10_17, o27_10);
            }
            { const float eb = bi[257];
              o27_10 = fmaf(eb, g10_18, o27_10);
            }
            { const float eb = bi[258];
              o27_10 = fmaf(eb, g10_30, o27_10);
            }
            { const float eb = bi[259];
              o28_10 = fmaf(eb, g10_0, o28_10);
            }
            { const float eb = bi[260];
              o28_10 = fmaf(eb, g10_1, o28_10);
            }
            { const float eb = bi[261];
              o28_10 = fmaf(eb, g10_4, o28_10);
            }
            { const float eb = bi[262];
              o28_10 = fmaf(eb, g10_3, o28_10);
            }
            { const float eb = bi[263];
              o28_10 = fmaf(eb, g10_7, o28_10);
            }
            { const float eb = bi[264];
              o28_10 = fmaf(eb, g10_14, o28_10);
            }
            { const float eb = bi[265];
              o28_10 = fmaf(eb, g10_9, o28_10);
            }
            { const float eb = bi[266];
              o28_10 = fmaf(eb, g10_17, o28_10);
            }
            { const float eb = bi[267];
              o28_10 = fmaf(eb, g10_29, o28_10);
            }
            { const float eb = bi[268];
              o29_10 = fmaf(eb, g10_0, o29_10);
            }
            { const float eb = bi[269];
              o29_10 = fmaf(eb, g10_1, o29_10);
            }
            { const float eb = bi[270];
              o29_10 = fmaf(eb, g10_4, o29_10);
            }
            { const float eb = bi[271];
              o29_10 = fmaf(eb, g10_2, o29_10);
            }
            { const float eb = bi[272];
              o29_10 = fmaf(eb, g10_5, o29_10);
            }
            { const float eb = bi[273];
              o29_10 = fmaf(eb, g10_11, o29_10);
            }
            { const float eb = bi[274];
              o29_10 = fmaf(eb, g10_3, o29_10);
            }
            { const float eb = bi[275];
              o29_10 = fmaf(eb, g10_7, o29_10);
            }
            { const float eb = bi[276];
              o29_10 = fmaf(eb, g10_14, o29_10);
            }
            { const float eb = bi[277];
              o29_10 = fmaf(eb, g10_8, o29_10);
            }
            { const float eb = bi[278];
              o29_10 = fmaf(eb, g10_15, o29_10);
            }
            { const float eb = bi[279];
              o29_10 = fmaf(eb, g10_26, o29_10);
            }
            { const float eb = bi[280];
              o30_10 = fmaf(eb, g10_0, o30_10);
            }
            { const float eb = bi[281];
              o30_10 = fmaf(eb, g10_1, o30_10);
            }
            { const float eb = bi[282];
              o30_10 = fmaf(eb, g10_2, o30_10);
            }
            { const float eb = bi[283];
              o30_10 = fmaf(eb, g10_5, o30_10);
            }
            { const float eb = bi[284];
              o30_10 = fmaf(eb, g10_3, o30_10);
            }
            { const float eb = bi[285];
              o30_10 = fmaf(eb, g10_7, o30_10);
            }
            { const float eb = bi[286];
              o30_10 = fmaf(eb, g10_8, o30_10);
            }
            { const float eb = bi[287];
              o30_10 = fmaf(eb, g10_15, o30_10);
            }
            { const float eb = bi[288];
              o30_10 = fmaf(eb, g10_9, o30_10);
            }
            { const float eb = bi[289];
              o30_10 = fmaf(eb, g10_17, o30_10);
            }
            { const float eb = bi[290];
              o30_10 = fmaf(eb, g10_18, o30_10);
            }
            { const float eb = bi[291];
              o30_10 = fmaf(eb, g10_30, o30_10);
            }
            { const float eb = bi[292];
              o31_10 = fmaf(eb, g10_0, o31_10);
            }
            { const float eb = bi[293];
              o31_10 = fmaf(eb, g10_1, o31_10);
            }
            { const float eb = bi[294];
              o31_10 = fmaf(eb, g10_2, o31_10);
            }
            { const float eb = bi[295];
              o31_10 = fmaf(eb, g10_5, o31_10);
            }
            { const float eb = bi[296];
              o31_10 = fmaf(eb, g10_6, o31_10);
            }
            { const float eb = bi[297];
              o31_10 = fmaf(eb, g10_12, o31_10);
            }
            { const float eb = bi[298];
              o31_10 = fmaf(eb, g10_13, o31_10);
            }
            { const float eb = bi[299];
              o31_10 = fmaf(eb, g10_23, o31_10);
            }
            { const float eb = bi[300];
              o32_10 = fmaf(eb, g10_0, o32_10);
            }
            { const float eb = bi[301];
              o32_10 = fmaf(eb, g10_1, o32_10);
            }
            { const float eb = bi[302];
              o32_10 = fmaf(eb, g10_4, o32_10);
            }
            { const float eb = bi[303];
              o32_10 = fmaf(eb, g10_10, o32_10);
            }
            { const float eb = bi[304];
              o32_10 = fmaf(eb, g10_2, o32_10);
            }
            { const float eb = bi[305];
              o32_10 = fmaf(eb, g10_5, o32_10);
            }
            { const float eb = bi[306];
              o32_10 = fmaf(eb, g10_11, o32_10);
            }
            { const float eb = bi[307];
              o32_10 = fmaf(eb, g10_21, o32_10);
            }
            { const float eb = bi[308];
              o33_10 = fmaf(eb, g10_0, o33_10);
            }
            { const float eb = bi[309];
              o33_10 = fmaf(eb, g10_1, o33_10);
            }
            { const float eb = bi[310];
              o33_10 = fmaf(eb, g10_2, o33_10);
            }
            { const float eb = bi[311];
              o33_10 = fmaf(eb, g10_5, o33_10);
            }
            { const float eb = bi[312];
              o33_10 = fmaf(eb, g10_6, o33_10);
            }
            { const float eb = bi[313];
              o33_10 = fmaf(eb, g10_12, o33_10);
            }
            { const float eb = bi[314];
              o33_10 = fmaf(eb, g10_3, o33_10);
            }
            { const float eb = bi[315];
              o33_10 = fmaf(eb, g10_7, o33_10);
            }
            { const float eb = bi[316];
              o33_10 = fmaf(eb, g10_8, o33_10);
            }
            { const float eb = bi[317];
              o33_10 = fmaf(eb, g10_15, o33_10);
            }
            { const float eb = bi[318];
              o33_10 = fmaf(eb, g10_16, o33_10);
            }
            { const float eb = bi[319];
              o33_10 = fmaf(eb, g10_27, o33_10);
            }
            { const float eb = bi[320];
              o34_10 = fmaf(eb, g10_0, o34_10);
            }
            { const float eb = bi[321];
              o34_10 = fmaf(eb, g10_1, o34_10);
            }
            { const float eb = bi[322];
              o34_10 = fmaf(eb, g10_4, o34_10);
            }
            { const float eb = bi[323];
              o34_10 = fmaf(eb, g10_2, o34_10);
            }
            { const float eb = bi[324];
              o34_10 = fmaf(eb, g10_5, o34_10);
            }
            { const float eb = bi[325];
              o34_10 = fmaf(eb, g10_11, o34_10);
            }
            { const float eb = bi[326];
              o34_10 = fmaf(eb, g10_3, o34_10);
            }
            { const float eb = bi[327];
              o34_10 = fmaf(eb, g10_7, o34_10);
            }
            { const float eb = bi[328];
              o34_10 = fmaf(eb, g10_14, o34_10);
            }
            { const float eb = bi[329];
              o34_10 = fmaf(eb, g10_8, o34_10);
            }
            { const float eb = bi[330];
              o34_10 = fmaf(eb, g10_15, o34_10);
            }
            { const float eb = bi[331];
              o34_10 = fmaf(eb, g10_26, o34_10);
            }
            { const float eb = bi[332];
              o35_10 = fmaf(eb, g10_0, o35_10);
            }
            { const float eb = bi[333];
              o35_10 = fmaf(eb, g10_1, o35_10);
            }
            { const float eb = bi[334];
              o35_10 = fmaf(eb, g10_4, o35_10);
            }
            { const float eb = bi[335];
              o35_10 = fmaf(eb, g10_2, o35_10);
            }
            { const float eb = bi[336];
              o35_10 = fmaf(eb, g10_5, o35_10);
            }
            { const float eb = bi[337];
              o35_10 = fmaf(eb, g10_11, o35_10);
            }
            { const float eb = bi[338];
              o35_10 = fmaf(eb, g10_6, o35_10);
            }
            { const float eb = bi[339];
              o35_10 = fmaf(eb, g10_12, o35_10);
            }
            { const float eb = bi[340];
              o35_10 = fmaf(eb, g10_22, o35_10);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk10 = PT[(fI + 2) * N + fJ + 2];
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
            const double Abd0_2 = PA[(fQ + 0) * N + fJ + 2];
            const double Abd1_2 = PA[(fQ + 1) * N + fJ + 2];
            const double Abd2_2 = PA[(fQ + 2) * N + fJ + 2];
            const double Abd3_2 = PA[(fQ + 3) * N + fJ + 2];
            const double Abd4_2 = PA[(fQ + 4) * N + fJ + 2];
            const double Abd5_2 = PA[(fQ + 5) * N + fJ + 2];
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
            const double Abc4_2 = PA[(fQ + 4) * N + fI + 2];
            const double Abc5_2 = PA[(fQ + 5) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
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
            jab24 += o24_10 * ptk10;
            jab25 += o25_10 * ptk10;
            jab26 += o26_10 * ptk10;
            jab27 += o27_10 * ptk10;
            jab28 += o28_10 * ptk10;
            jab29 += o29_10 * ptk10;
            jab30 += o30_10 * ptk10;
            jab31 += o31_10 * ptk10;
            jab32 += o32_10 * ptk10;
            jab33 += o33_10 * ptk10;
            jab34 += o34_10 * ptk10;
            jab35 += o35_10 * ptk10;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 2, 2.0 * deg * (o0_10 * ptb0 + o1_10 * ptb1 + o2_10 * ptb2 + o3_10 * ptb3 + o4_10 * ptb4 + o5_10 * ptb5 + o6_10 * ptb6 + o7_10 * ptb7 + o8_10 * ptb8 + o9_10 * ptb9 + o10_10 * ptb10 + o11_10 * ptb11 + o12_10 * ptb12 + o13_10 * ptb13 + o14_10 * ptb14 + o15_10 * ptb15 + o16_10 * ptb16 + o17_10 * ptb17 + o18_10 * ptb18 + o19_10 * ptb19 + o20_10 * ptb20 + o21_10 * ptb21 + o22_10 * ptb22 + o23_10 * ptb23 + o24_10 * ptb24 + o25_10 * ptb25 + o26_10 * ptb26 + o27_10 * ptb27 + o28_10 * ptb28 + o29_10 * ptb29 + o30_10 * ptb30 + o31_10 * ptb31 + o32_10 * ptb32 + o33_10 * ptb33 + o34_10 * ptb34 + o35_10 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_10 * Abd0_2 + o1_10 * Abd1_2 + o2_10 * Abd2_2 + o3_10 * Abd3_2 + o4_10 * Abd4_2 + o5_10 * Abd5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_10 * Aad0_2 + o6_10 * Aad1_2 + o12_10 * Aad2_2 + o18_10 * Aad3_2 + o24_10 * Aad4_2 + o30_10 * Aad5_2));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 2, deg * (o0_10 * Abc0_2 + o1_10 * Abc1_2 + o2_10 * Abc2_2 + o3_10 * Abc3_2 + o4_10 * Abc4_2 + o5_10 * Abc5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 2, deg * (o0_10 * Aac0_2 + o6_10 * Aac1_2 + o12_10 * Aac2_2 + o18_10 * Aac3_2 + o24_10 * Aac4_2 + o30_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_10 * Aad0_2 + o7_10 * Aad1_2 + o13_10 * Aad2_2 + o19_10 * Aad3_2 + o25_10 * Aad4_2 + o31_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 2, deg * (o1_10 * Aac0_2 + o7_10 * Aac1_2 + o13_10 * Aac2_2 + o19_10 * Aac3_2 + o25_10 * Aac4_2 + o31_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_10 * Aad0_2 + o8_10 * Aad1_2 + o14_10 * Aad2_2 + o20_10 * Aad3_2 + o26_10 * Aad4_2 + o32_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 2, deg * (o2_10 * Aac0_2 + o8_10 * Aac1_2 + o14_10 * Aac2_2 + o20_10 * Aac3_2 + o26_10 * Aac4_2 + o32_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_10 * Aad0_2 + o9_10 * Aad1_2 + o15_10 * Aad2_2 + o21_10 * Aad3_2 + o27_10 * Aad4_2 + o33_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 2, deg * (o3_10 * Aac0_2 + o9_10 * Aac1_2 + o15_10 * Aac2_2 + o21_10 * Aac3_2 + o27_10 * Aac4_2 + o33_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 2, deg * (o4_10 * Aad0_2 + o10_10 * Aad1_2 + o16_10 * Aad2_2 + o22_10 * Aad3_2 + o28_10 * Aad4_2 + o34_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 2, deg * (o4_10 * Aac0_2 + o10_10 * Aac1_2 + o16_10 * Aac2_2 + o22_10 * Aac3_2 + o28_10 * Aac4_2 + o34_10 * Aac5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 2, deg * (o5_10 * Aad0_2 + o11_10 * Aad1_2 + o17_10 * Aad2_2 + o23_10 * Aad3_2 + o29_10 * Aad4_2 + o35_10 * Aad5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 2, deg * (o5_10 * Aac0_2 + o11_10 * Aac1_2 + o17_10 * Aac2_2 + o23_10 * Aac3_2 + o29_10 * Aac4_2 + o35_10 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o6_10 * Abd0_2 + o7_10 * Abd1_2 + o8_10 * Abd2_2 + o9_10 * Abd3_2 + o10_10 * Abd4_2 + o11_10 * Abd5_2));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 2, deg * (o6_10 * Abc0_2 + o7_10 * Abc1_2 + o8_10 * Abc2_2 + o9_10 * Abc3_2 + o10_10 * Abc4_2 + o11_10 * Abc5_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o12_10 * Abd0_2 + o13_10 * Abd1_2 + o14_10 * Abd2_2 + o15_10 * Abd3_2 + o16_10 * Abd4_2 + o17_10 * Abd5_2));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 2, deg * (o12_10 * Abc0_2 + o13_10 * Abc1_2 + o14_10 * Abc2_2 + o15_10 * Abc3_2 + o16_10 * Abc4_2 + o17_10 * Abc5_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o18_10 * Abd0_2 + o19_10 * Abd1_2 + o20_10 * Abd2_2 + o21_10 * Abd3_2 + o22_10 * Abd4_2 + o23_10 * Abd5_2));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 2, deg * (o18_10 * Abc0_2 + o19_10 * Abc1_2 + o20_10 * Abc2_2 + o21_10 * Abc3_2 + o22_10 * Abc4_2 + o23_10 * Abc5_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o24_10 * Abd0_2 + o25_10 * Abd1_2 + o26_10 * Abd2_2 + o27_10 * Abd3_2 + o28_10 * Abd4_2 + o29_10 * Abd5_2));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 2, deg * (o24_10 * Abc0_2 + o25_10 * Abc1_2 + o26_10 * Abc2_2 + o27_10 * Abc3_2 + o28_10 * Abc4_2 + o29_10 * Abc5_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o30_10 * Abd0_2 + o31_10 * Abd1_2 + o32_10 * Abd2_2 + o33_10 * Abd3_2 + o34_10 * Abd4_2 + o35_10 * Abd5_2));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 2, deg * (o30_10 * Abc0_2 + o31_10 * Abc1_2 + o32_10 * Abc2_2 + o33_10 * Abc3_2 + o34_10 * Abc4_2 + o35_10 * Abc5_2));
          }
        } break;
        case 11: {  // ket functions [11]
          float o0_11 = 0;
          float o1_11 = 0;
          float o2_11 = 0;
          float o3_11 = 0;
          float o4_11 = 0;
          float o5_11 = 0;
          float o6_11 = 0;
          float o7_11 = 0;
          float o8_11 = 0;
          float o9_11 = 0;
          float o10_11 = 0;
          float o11_11 = 0;
          float o12_11 = 0;
          float o13_11 = 0;
          float o14_11 = 0;
          float o15_11 = 0;
          float o16_11 = 0;
          float o17_11 = 0;
          float o18_11 = 0;
          float o19_11 = 0;
          float o20_11 = 0;
          float o21_11 = 0;
          float o22_11 = 0;
          float o23_11 = 0;
          float o24_11 = 0;
          float o25_11 = 0;
          float o26_11 = 0;
          float o27_11 = 0;
          float o28_11 = 0;
          float o29_11 = 0;
          float o30_11 = 0;
          float o31_11 = 0;
          float o32_11 = 0;
          float o33_11 = 0;
          float o34_11 = 0;
          float o35_11 = 0;
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 341;
            const float p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            float g11_0 = 0;
            float g11_1 = 0;
            float g11_2 = 0;
            float g11_3 = 0;
            float g11_4 = 0;
            float g11_5 = 0;
            float g11_6 = 0;
            float g11_7 = 0;
            float g11_8 = 0;
            float g11_9 = 0;
            float g11_10 = 0;
            float g11_11 = 0;
            float g11_12 = 0;
            float g11_13 = 0;
            float g11_14 = 0;
            float g11_15 = 0;
            float g11_16 = 0;
            float g11_17 = 0;
            float g11_18 = 0;
            float g11_19 = 0;
            float g11_20 = 0;
            float g11_21 = 0;
            float g11_22 = 0;
            float g11_23 = 0;
            float g11_24 = 0;
            float g11_25 = 0;
            float g11_26 = 0;
            float g11_27 = 0;
            float g11_28 = 0;
            float g11_29 = 0;
            float g11_30 = 0;
            float g11_31 = 0;
            float g11_32 = 0;
            float g11_33 = 0;
            float g11_34 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const float* __restrict__ kj = kprim + (long long)j * 44 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[7];
              sqb::boysf<6>(T, a.boys_tab_f, F);
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
              w *= m2a;
              const float b5 = w * F[5];
              w *= m2a;
              const float b6 = w * F[6];
              const float ek11_0 = kj[41 * kS];
              const float ek11_1 = -kj[42 * kS];
              const float ek11_2 = kj[43 * kS];
              g11_0 = fmaf(ek11_0, b0, g11_0);
              const float r0_0_0_1 = Z * b1;
              g11_1 = fmaf(ek11_0, r0_0_0_1, g11_1);
              g11_0 = fmaf(ek11_1, r0_0_0_1, g11_0);
              const float r0_0_1_0 = Y * b1;
              g11_2 = fmaf(ek11_0, r0_0_1_0, g11_2);
              const float r0_1_0_0 = X * b1;
              g11_3 = fmaf(ek11_0, r0_1_0_0, g11_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g11_4 = fmaf(ek11_0, r0_0_0_2, g11_4);
              g11_1 = fmaf(ek11_1, r0_0_0_2, g11_1);
              g11_0 = fmaf(ek11_2, r0_0_0_2, g11_0);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g11_5 = fmaf(ek11_0, r0_0_1_1, g11_5);
              g11_2 = fmaf(ek11_1, r0_0_1_1, g11_2);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g11_6 = fmaf(ek11_0, r0_0_2_0, g11_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g11_7 = fmaf(ek11_0, r0_1_0_1, g11_7);
              g11_3 = fmaf(ek11_1, r0_1_0_1, g11_3);
              const float r0_1_1_0 = X * r1_0_1_0;
              g11_8 = fmaf(ek11_0, r0_1_1_0, g11_8);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g11_9 = fmaf(ek11_0, r0_2_0_0, g11_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g11_10 = fmaf(ek11_0, r0_0_0_3, g11_10);
              g11_4 = fmaf(ek11_1, r0_0_0_3, g11_4);
              g11_1 = fmaf(ek11_2, r0_0_0_3, g11_1);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g11_11 = fmaf(ek11_0, r0_0_1_2, g11_11);
              g11_5 = fmaf(ek11_1, r0_0_1_2, g11_5);
              g11_2 = fmaf(ek11_2, r0_0_1_2, g11_2);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g11_12 = fmaf(ek11_0, r0_0_2_1, g11_12);
              g11_6 = fmaf(ek11_1, r0_0_2_1, g11_6);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g11_13 = fmaf(ek11_0, r0_0_3_0, g11_13);
              const float r0_1_0_2 = X * r1_0_0_2;
              g11_14 = fmaf(ek11_0, r0_1_0_2, g11_14);
              g11_7 = fmaf(ek11_1, r0_1_0_2, g11_7);
              g11_3 = fmaf(ek11_2, r0_1_0_2, g11_3);
              const float r0_1_1_1 = X * r1_0_1_1;
              g11_15 = fmaf(ek11_0, r0_1_1_1, g11_15);
              g11_8 = fmaf(ek11_1, r0_1_1_1, g11_8);
              const float r0_1_2_0 = X * r1_0_2_0;
              g11_16 = fmaf(ek11_0, r0_1_2_0, g11_16);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g11_17 = fmaf(ek11_0, r0_2_0_1, g11_17);
              g11_9 = fmaf(ek11_1, r0_2_0_1, g11_9);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g11_18 = fmaf(ek11_0, r0_2_1_0, g11_18);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g11_19 = fmaf(ek11_0, r0_3_0_0, g11_19);
              const float r3_0_0_1 = Z * b4;
              const float r2_0_0_2 = fmaf(Z, r3_0_0_1, b3);
              const float r1_0_0_3 = fmaf(Z, r2_0_0_2, 2.0f * r2_0_0_1);
              const float r0_0_0_4 = fmaf(Z, r1_0_0_3, 3.0f * r1_0_0_2);
              g11_20 = fmaf(ek11_0, r0_0_0_4, g11_20);
              g11_10 = fmaf(ek11_1, r0_0_0_4, g11_10);
              g11_4 = fmaf(ek11_2, r0_0_0_4, g11_4);
              const float r0_0_1_3 = Y * r1_0_0_3;
              g11_21 = fmaf(ek11_0, r0_0_1_3, g11_21);
              g11_11 = fmaf(ek11_1, r0_0_1_3, g11_11);
              g11_5 = fmaf(ek11_2, r0_0_1_3, g11_5);
              const float r1_0_1_2 = Y * r2_0_0_2;
              const float r0_0_2_2 = fmaf(Y, r1_0_1_2, r1_0_0_2);
              g11_22 = fmaf(ek11_0, r0_0_2_2, g11_22);
              g11_12 = fmaf(ek11_1, r0_0_2_2, g11_12);
              g11_6 = fmaf(ek11_2, r0_0_2_2, g11_6);
              const float r2_0_1_1 = Y * r3_0_0_1;
              const float r1_0_2_1 = fmaf(Y, r2_0_1_1, r2_0_0_1);
              const float r0_0_3_1 = fmaf(Y, r1_0_2_1, 2.0f * r1_0_1_1);
              g11_23 = fmaf(ek11_0, r0_0_3_1, g11_23);
              g11_13 = fmaf(ek11_1, r0_0_3_1, g11_13);
              const float r3_0_1_0 = Y * b4;
              const float r2_0_2_0 = fmaf(Y, r3_0_1_0, b3);
              const float r1_0_3_0 = fmaf(Y, r2_0_2_0, 2.0f * r2_0_1_0);
              const float r0_0_4_0 = fmaf(Y, r1_0_3_0, 3.0f * r1_0_2_0);
              g11_24 = fmaf(ek11_0, r0_0_4_0, g11_24);
              const float r0_1_0_3 = X * r1_0_0_3;
              g11_25 = fmaf(ek11_0, r0_1_0_3, g11_25);
              g11_14 = fmaf(ek11_1, r0_1_0_3, g11_14);
              g11_7 = fmaf(ek11_2, r0_1_0_3, g11_7);
              const float r0_1_1_2 = X * r1_0_1_2;
              g11_26 = fmaf(ek11_0, r0_1_1_2, g11_26);
              g11_15 = fmaf(ek11_1, r0_1_1_2, g11_15);
              g11_8 = fmaf(ek11_2, r0_1_1_2, g11_8);
              const float r0_1_2_1 = X * r1_0_2_1;
              g11_27 = fmaf(ek11_0, r0_1_2_1, g11_27);
              g11_16 = fmaf(ek11_1, r0_1_2_1, g11_16);
              const float r0_1_3_0 = X * r1_0_3_0;
              g11_28 = fmaf(ek11_0, r0_1_3_0, g11_28);
              const float r1_1_0_2 = X * r2_0_0_2;
              const float r0_2_0_2 = fmaf(X, r1_1_0_2, r1_0_0_2);
              g11_29 = fmaf(ek11_0, r0_2_0_2, g11_29);
              g11_17 = fmaf(ek11_1, r0_2_0_2, g11_17);
              g11_9 = fmaf(ek11_2, r0_2_0_2, g11_9);
              const float r1_1_1_1 = X * r2_0_1_1;
              const float r0_2_1_1 = fmaf(X, r1_1_1_1, r1_0_1_1);
              g11_30 = fmaf(ek11_0, r0_2_1_1, g11_30);
              g11_18 = fmaf(ek11_1, r0_2_1_1, g11_18);
              const float r1_1_2_0 = X * r2_0_2_0;
              const float r0_2_2_0 = fmaf(X, r1_1_2_0, r1_0_2_0);
              g11_31 = fmaf(ek11_0, r0_2_2_0, g11_31);
              const float r2_1_0_1 = X * r3_0_0_1;
              const float r1_2_0_1 = fmaf(X, r2_1_0_1, r2_0_0_1);
              const float r0_3_0_1 = fmaf(X, r1_2_0_1, 2.0f * r1_1_0_1);
              g11_32 = fmaf(ek11_0, r0_3_0_1, g11_32);
              g11_19 = fmaf(ek11_1, r0_3_0_1, g11_19);
              const float r2_1_1_0 = X * r3_0_1_0;
              const float r1_2_1_0 = fmaf(X, r2_1_1_0, r2_0_1_0);
              const float r0_3_1_0 = fmaf(X, r1_2_1_0, 2.0f * r1_1_1_0);
              g11_33 = fmaf(ek11_0, r0_3_1_0, g11_33);
              const float r3_1_0_0 = X * b4;
              const float r2_2_0_0 = fmaf(X, r3_1_0_0, b3);
              const float r1_3_0_0 = fmaf(X, r2_2_0_0, 2.0f * r2_1_0_0);
              const float r0_4_0_0 = fmaf(X, r1_3_0_0, 3.0f * r1_2_0_0);
              g11_34 = fmaf(ek11_0, r0_4_0_0, g11_34);
              const float r4_0_0_1 = Z * b5;
              const float r3_0_0_2 = fmaf(Z, r4_0_0_1, b4);
              const float r2_0_0_3 = fmaf(Z, r3_0_0_2, 2.0f * r3_0_0_1);
              const float r1_0_0_4 = fmaf(Z, r2_0_0_3, 3.0f * r2_0_0_2);
              const float r0_0_0_5 = fmaf(Z, r1_0_0_4, 4.0f * r1_0_0_3);
              g11_20 = fmaf(ek11_1, r0_0_0_5, g11_20);
              g11_10 = fmaf(ek11_2, r0_0_0_5, g11_10);
              const float r0_0_1_4 = Y * r1_0_0_4;
              g11_21 = fmaf(ek11_1, r0_0_1_4, g11_21);
              g11_11 = fmaf(ek11_2, r0_0_1_4, g11_11);
              const float r1_0_1_3 = Y * r2_0_0_3;
              const float r0_0_2_3 = fmaf(Y, r1_0_1_3, r1_0_0_3);
              g11_22 = fmaf(ek11_1, r0_0_2_3, g11_22);
              g11_12 = fmaf(ek11_2, r0_0_2_3, g11_12);
              const float r2_0_1_2 = Y * r3_0_0_2;
              const float r1_0_2_2 = fmaf(Y, r2_0_1_2, r2_0_0_2);
              const float r0_0_3_2 = fmaf(Y, r1_0_2_2, 2.0f * r1_0_1_2);
              g11_23 = fmaf(ek11_1, r0_0_3_2, g11_23);
              g11_13 = fmaf(ek11_2, r0_0_3_2, g11_13);
              const float r3_0_1_1 = Y * r4_0_0_1;
              const float r2_0_2_1 = fmaf(Y, r3_0_1_1, r3_0_0_1);
              const float r1_0_3_1 = fmaf(Y, r2_0_2_1, 2.0f * r2_0_1_1);
              const float r0_0_4_1 = fmaf(Y, r1_0_3_1, 3.0f * r1_0_2_1);
              g11_24 = fmaf(ek11_1, r0_0_4_1, g11_24);
              const float r0_1_0_4 = X * r1_0_0_4;
              g11_25 = fmaf(ek11_1, r0_1_0_4, g11_25);
              g11_14 = fmaf(ek11_2, r0_1_0_4, g11_14);
              const float r0_1_1_3 = X * r1_0_1_3;
              g11_26 = fmaf(ek11_1, r0_1_1_3, g11_26);
              g11_15 = fmaf(ek11_2, r0_1_1_3, g11_15);
              const float r0_1_2_2 = X * r1_0_2_2;
              g11_27 = fmaf(ek11_1, r0_1_2_2, g11_27);
              g11_16 = fmaf(ek11_2, r0_1_2_2, g11_16);
              const float r0_1_3_1 = X * r1_0_3_1;
              g11_28 = fmaf(ek11_1, r0_1_3_1, g11_28);
              const float r1_1_0_3 = X * r2_0_0_3;
              const float r0_2_0_3 = fmaf(X, r1_1_0_3, r1_0_0_3);
              g11_29 = fmaf(ek11_1, r0_2_0_3, g11_29);
              g11_17 = fmaf(ek11_2, r0_2_0_3, g11_17);
              const float r1_1_1_2 = X * r2_0_1_2;
              const float r0_2_1_2 = fmaf(X, r1_1_1_2, r1_0_1_2);
              g11_30 = fmaf(ek11_1, r0_2_1_2, g11_30);
              g11_18 = fmaf(ek11_2, r0_2_1_2, g11_18);
              const float r1_1_2_1 = X * r2_0_2_1;
              const float r0_2_2_1 = fmaf(X, r1_1_2_1, r1_0_2_1);
              g11_31 = fmaf(ek11_1, r0_2_2_1, g11_31);
              const float r2_1_0_2 = X * r3_0_0_2;
              const float r1_2_0_2 = fmaf(X, r2_1_0_2, r2_0_0_2);
              const float r0_3_0_2 = fmaf(X, r1_2_0_2, 2.0f * r1_1_0_2);
              g11_32 = fmaf(ek11_1, r0_3_0_2, g11_32);
              g11_19 = fmaf(ek11_2, r0_3_0_2, g11_19);
              const float r2_1_1_1 = X * r3_0_1_1;
              const float r1_2_1_1 = fmaf(X, r2_1_1_1, r2_0_1_1);
              const float r0_3_1_1 = fmaf(X, r1_2_1_1, 2.0f * r1_1_1_1);
              g11_33 = fmaf(ek11_1, r0_3_1_1, g11_33);
              const float r3_1_0_1 = X * r4_0_0_1;
              const float r2_2_0_1 = fmaf(X, r3_1_0_1, r3_0_0_1);
              const float r1_3_0_1 = fmaf(X, r2_2_0_1, 2.0f * r2_1_0_1);
              const float r0_4_0_1 = fmaf(X, r1_3_0_1, 3.0f * r1_2_0_1);
              g11_34 = fmaf(ek11_1, r0_4_0_1, g11_34);
              const float r5_0_0_1 = Z * b6;
              const float r4_0_0_2 = fmaf(Z, r5_0_0_1, b5);
              const float r3_0_0_3 = fmaf(Z, r4_0_0_2, 2.0f * r4_0_0_1);
              const float r2_0_0_4 = fmaf(Z, r3_0_0_3, 3.0f * r3_0_0_2);
              const float r1_0_0_5 = fmaf(Z, r2_0_0_4, 4.0f * r2_0_0_3);
              const float r0_0_0_6 = fmaf(Z, r1_0_0_5, 5.0f * r1_0_0_4);
              g11_20 = fmaf(ek11_2, r0_0_0_6, g11_20);
              const float r0_0_1_5 = Y * r1_0_0_5;
              g11_21 = fmaf(ek11_2, r0_0_1_5, g11_21);
              const float r1_0_1_4 = Y * r2_0_0_4;
              const float r0_0_2_4 = fmaf(Y, r1_0_1_4, r1_0_0_4);
              g11_22 = fmaf(ek11_2, r0_0_2_4, g11_22);
              const float r2_0_1_3 = Y * r3_0_0_3;
              const float r1_0_2_3 = fmaf(Y, r2_0_1_3, r2_0_0_3);
              const float r0_0_3_3 = fmaf(Y, r1_0_2_3, 2.0f * r1_0_1_3);
              g11_23 = fmaf(ek11_2, r0_0_3_3, g11_23);
              const float r3_0_1_2 = Y * r4_0_0_2;
              const float r2_0_2_2 = fmaf(Y, r3_0_1_2, r3_0_0_2);
              const float r1_0_3_2 = fmaf(Y, r2_0_2_2, 2.0f * r2_0_1_2);
              const float r0_0_4_2 = fmaf(Y, r1_0_3_2, 3.0f * r1_0_2_2);
              g11_24 = fmaf(ek11_2, r0_0_4_2, g11_24);
              const float r0_1_0_5 = X * r1_0_0_5;
              g11_25 = fmaf(ek11_2, r0_1_0_5, g11_25);
              const float r0_1_1_4 = X * r1_0_1_4;
              g11_26 = fmaf(ek11_2, r0_1_1_4, g11_26);
              const float r0_1_2_3 = X * r1_0_2_3;
              g11_27 = fmaf(ek11_2, r0_1_2_3, g11_27);
              const float r0_1_3_2 = X * r1_0_3_2;
              g11_28 = fmaf(ek11_2, r0_1_3_2, g11_28);
              const float r1_1_0_4 = X * r2_0_0_4;
              const float r0_2_0_4 = fmaf(X, r1_1_0_4, r1_0_0_4);
              g11_29 = fmaf(ek11_2, r0_2_0_4, g11_29);
              const float r1_1_1_3 = X * r2_0_1_3;
              const float r0_2_1_3 = fmaf(X, r1_1_1_3, r1_0_1_3);
              g11_30 = fmaf(ek11_2, r0_2_1_3, g11_30);
              const float r1_1_2_2 = X * r2_0_2_2;
              const float r0_2_2_2 = fmaf(X, r1_1_2_2, r1_0_2_2);
              g11_31 = fmaf(ek11_2, r0_2_2_2, g11_31);
              const float r2_1_0_3 = X * r3_0_0_3;
              const float r1_2_0_3 = fmaf(X, r2_1_0_3, r2_0_0_3);
              const float r0_3_0_3 = fmaf(X, r1_2_0_3, 2.0f * r1_1_0_3);
              g11_32 = fmaf(ek11_2, r0_3_0_3, g11_32);
              const float r2_1_1_2 = X * r3_0_1_2;
              const float r1_2_1_2 = fmaf(X, r2_1_1_2, r2_0_1_2);
              const float r0_3_1_2 = fmaf(X, r1_2_1_2, 2.0f * r1_1_1_2);
              g11_33 = fmaf(ek11_2, r0_3_1_2, g11_33);
              const float r3_1_0_2 = X * r4_0_0_2;
              const float r2_2_0_2 = fmaf(X, r3_1_0_2, r3_0_0_2);
              const float r1_3_0_2 = fmaf(X, r2_2_0_2, 2.0f * r2_1_0_2);
              const float r0_4_0_2 = fmaf(X, r1_3_0_2, 3.0f * r1_2_0_2);
              g11_34 = fmaf(ek11_2, r0_4_0_2, g11_34);
            }
            { const float eb = bi[5];
              o0_11 = fmaf(eb, g11_0, o0_11);
            }
            { const float eb = bi[6];
              o0_11 = fmaf(eb, g11_3, o0_11);
            }
            { const float eb = bi[7];
              o0_11 = fmaf(eb, g11_9, o0_11);
            }
            { const float eb = bi[8];
              o0_11 = fmaf(eb, g11_19, o0_11);
            }
            { const float eb = bi[9];
              o0_11 = fmaf(eb, g11_34, o0_11);
            }
            { const float eb = bi[10];
              o1_11 = fmaf(eb, g11_0, o1_11);
            }
            { const float eb = bi[11];
              o1_11 = fmaf(eb, g11_2, o1_11);
            }
            { const float eb = bi[12];
              o1_11 = fmaf(eb, g11_6, o1_11);
            }
            { const float eb = bi[13];
              o1_11 = fmaf(eb, g11_3, o1_11);
            }
            { const float eb = bi[14];
              o1_11 = fmaf(eb, g11_8, o1_11);
            }
            { const float eb = bi[15];
              o1_11 = fmaf(eb, g11_16, o1_11);
            }
            { const float eb = bi[16];
              o1_11 = fmaf(eb, g11_9, o1_11);
            }
            { const float eb = bi[17];
              o1_11 = fmaf(eb, g11_18, o1_11);
            }
            { const float eb = bi[18];
              o1_11 = fmaf(eb, g11_31, o1_11);
            }
            { const float eb = bi[19];
              o2_11 = fmaf(eb, g11_0, o2_11);
            }
            { const float eb = bi[20];
              o2_11 = fmaf(eb, g11_1, o2_11);
            }
            { const float eb = bi[21];
              o2_11 = fmaf(eb, g11_4, o2_11);
            }
            { const float eb = bi[22];
              o2_11 = fmaf(eb, g11_3, o2_11);
            }
            { const float eb = bi[23];
              o2_11 = fmaf(eb, g11_7, o2_11);
            }
            { const float eb = bi[24];
              o2_11 = fmaf(eb, g11_14, o2_11);
            }
            { const float eb = bi[25];
              o2_11 = fmaf(eb, g11_9, o2_11);
            }
            { const float eb = bi[26];
              o2_11 = fmaf(eb, g11_17, o2_11);
            }
            { const float eb = bi[27];
              o2_11 = fmaf(eb, g11_29, o2_11);
            }
            { const float eb = bi[28];
              o3_11 = fmaf(eb, g11_0, o3_11);
            }
            { const float eb = bi[29];
              o3_11 = fmaf(eb, g11_2, o3_11);
            }
            { const float eb = bi[30];
              o3_11 = fmaf(eb, g11_3, o3_11);
            }
            { const float eb = bi[31];
              o3_11 = fmaf(eb, g11_8, o3_11);
            }
            { const float eb = bi[32];
              o3_11 = fmaf(eb, g11_9, o3_11);
            }
            { const float eb = bi[33];
              o3_11 = fmaf(eb, g11_18, o3_11);
            }
            { const float eb = bi[34];
              o3_11 = fmaf(eb, g11_19, o3_11);
            }
            { const float eb = bi[35];
              o3_11 = fmaf(eb, g11_33, o3_11);
            }
            { const float eb = bi[36];
              o4_11 = fmaf(eb, g11_0, o4_11);
            }
            { const float eb = bi[37];
              o4_11 = fmaf(eb, g11_1, o4_11);
            }
            { const float eb = bi[38];
              o4_11 = fmaf(eb, g11_3, o4_11);
            }
            { const float eb = bi[39];
              o4_11 = fmaf(eb, g11_7, o4_11);
            }
            { const float eb = bi[40];
              o4_11 = fmaf(eb, g11_9, o4_11);
            }
            { const float eb = bi[41];
              o4_11 = fmaf(eb, g11_17, o4_11);
            }
            { const float eb = bi[42];
              o4_11 = fmaf(eb, g11_19, o4_11);
            }
            { const float eb = bi[43];
              o4_11 = fmaf(eb, g11_32, o4_11);
            }
            { const float eb = bi[44];
              o5_11 = fmaf(eb, g11_0, o5_11);
            }
            { const float eb = bi[45];
              o5_11 = fmaf(eb, g11_1, o5_11);
            }
            { const float eb = bi[46];
              o5_11 = fmaf(eb, g11_2, o5_11);
            }
            { const float eb = bi[47];
              o5_11 = fmaf(eb, g11_5, o5_11);
            }
            { const float eb = bi[48];
              o5_11 = fmaf(eb, g11_3, o5_11);
            }
            { const float eb = bi[49];
              o5_11 = fmaf(eb, g11_7, o5_11);
            }
            { const float eb = bi[50];
              o5_11 = fmaf(eb, g11_8, o5_11);
            }
            { const float eb = bi[51];
              o5_11 = fmaf(eb, g11_15, o5_11);
            }
            { const float eb = bi[52];
              o5_11 = fmaf(eb, g11_9, o5_11);
            }
            { const float eb = bi[53];
              o5_11 = fmaf(eb, g11_17, o5_11);
            }
            { const float eb = bi[54];
              o5_11 = fmaf(eb, g11_18, o5_11);
            }
            { const float eb = bi[55];
              o5_11 = fmaf(eb, g11_30, o5_11);
            }
            { const float eb = bi[56];
              o6_11 = fmaf(eb, g11_0, o6_11);
            }
            { const float eb = bi[57];
              o6_11 = fmaf(eb, g11_2, o6_11);
            }
            { const float eb = bi[58];
              o6_11 = fmaf(eb, g11_6, o6_11);
            }
            { const float eb = bi[59];
              o6_11 = fmaf(eb, g11_3, o6_11);
            }
            { const float eb = bi[60];
              o6_11 = fmaf(eb, g11_8, o6_11);
            }
            { const float eb = bi[61];
              o6_11 = fmaf(eb, g11_16, o6_11);
            }
            { const float eb = bi[62];
              o6_11 = fmaf(eb, g11_9, o6_11);
            }
            { const float eb = bi[63];
              o6_11 = fmaf(eb, g11_18, o6_11);
            }
            { const float eb = bi[64];
              o6_11 = fmaf(eb, g11_31, o6_11);
            }
            { const float eb = bi[65];
              o7_11 = fmaf(eb, g11_0, o7_11);
            }
            { const float eb = bi[66];
              o7_11 = fmaf(eb, g11_2, o7_11);
            }
            { const float eb = bi[67];
              o7_11 = fmaf(eb, g11_6, o7_11);
            }
            { const float eb = bi[68];
              o7_11 = fmaf(eb, g11_13, o7_11);
            }
            { const float eb = bi[69];
              o7_11 = fmaf(eb, g11_24, o7_11);
            }
            { const float eb = bi[70];
              o8_11 = fmaf(eb, g11_0, o8_11);
            }
            { const float eb = bi[71];
              o8_11 = fmaf(eb, g11_1, o8_11);
            }
            { const float eb = bi[72];
              o8_11 = fmaf(eb, g11_4, o8_11);
            }
            { const float eb = bi[73];
              o8_11 = fmaf(eb, g11_2, o8_11);
            }
            { const float eb = bi[74];
              o8_11 = fmaf(eb, g11_5, o8_11);
            }
            { const float eb = bi[75];
              o8_11 = fmaf(eb, g11_11, o8_11);
            }
            { const float eb = bi[76];
              o8_11 = fmaf(eb, g11_6, o8_11);
            }
            { const float eb = bi[77];
              o8_11 = fmaf(eb, g11_12, o8_11);
            }
            { const float eb = bi[78];
              o8_11 = fmaf(eb, g11_22, o8_11);
            }
            { const float eb = bi[79];
              o9_11 = fmaf(eb, g11_0, o9_11);
            }
            { const float eb = bi[80];
              o9_11 = fmaf(eb, g11_2, o9_11);
            }
            { const float eb = bi[81];
              o9_11 = fmaf(eb, g11_6, o9_11);
            }
            { const float eb = bi[82];
              o9_11 = fmaf(eb, g11_13, o9_11);
            }
            { const float eb = bi[83];
              o9_11 = fmaf(eb, g11_3, o9_11);
            }
            { const float eb = bi[84];
              o9_11 = fmaf(eb, g11_8, o9_11);
            }
            { const float eb = bi[85];
              o9_11 = fmaf(eb, g11_16, o9_11);
            }
            { const float eb = bi[86];
              o9_11 = fmaf(eb, g11_28, o9_11);
            }
            { const float eb = bi[87];
              o10_11 = fmaf(eb, g11_0, o10_11);
            }
            { const float eb = bi[88];
              o10_11 = fmaf(eb, g11_1, o10_11);
            }
            { const float eb = bi[89];
              o10_11 = fmaf(eb, g11_2, o10_11);
            }
            { const float eb = bi[90];
              o10_11 = fmaf(eb, g11_5, o10_11);
            }
            { const float eb = bi[91];
              o10_11 = fmaf(eb, g11_6, o10_11);
            }
            { const float eb = bi[92];
              o10_11 = fmaf(eb, g11_12, o10_11);
            }
            { const float eb = bi[93];
              o10_11 = fmaf(eb, g11_3, o10_11);
            }
            { const float eb = bi[94];
              o10_11 = fmaf(eb, g11_7, o10_11);
            }
            { const float eb = bi[95];
              o10_11 = fmaf(eb, g11_8, o10_11);
            }
            { const float eb = bi[96];
              o10_11 = fmaf(eb, g11_15, o10_11);
            }
            { const float eb = bi[97];
              o10_11 = fmaf(eb, g11_16, o10_11);
            }
            { const float eb = bi[98];
              o10_11 = fmaf(eb, g11_27, o10_11);
            }
            { const float eb = bi[99];
              o11_11 = fmaf(eb, g11_0, o11_11);
            }
            { const float eb = bi[100];
              o11_11 = fmaf(eb, g11_1, o11_11);
            }
            { const float eb = bi[101];
              o11_11 = fmaf(eb, g11_2, o11_11);
            }
            { const float eb = bi[102];
              o11_11 = fmaf(eb, g11_5, o11_11);
            }
            { const float eb = bi[103];
              o11_11 = fmaf(eb, g11_6, o11_11);
            }
            { const float eb = bi[104];
              o11_11 = fmaf(eb, g11_12, o11_11);
            }
            { const float eb = bi[105];
              o11_11 = fmaf(eb, g11_13, o11_11);
            }
            { const float eb = bi[106];
              o11_11 = fmaf(eb, g11_23, o11_11);
            }
            { const float eb = bi[107];
              o12_11 = fmaf(eb, g11_0, o12_11);
            }
            { const float eb = bi[108];
              o12_11 = fmaf(eb, g11_1, o12_11);
            }
            { const float eb = bi[109];
              o12_11 = fmaf(eb, g11_4, o12_11);
            }
            { const float eb = bi[110];
              o12_11 = fmaf(eb, g11_3, o12_11);
            }
            { const float eb = bi[111];
              o12_11 = fmaf(eb, g11_7, o12_11);
            }
            { const float eb = bi[112];
              o12_11 = fmaf(eb, g11_14, o12_11);
            }
            { const float eb = bi[113];
              o12_11 = fmaf(eb, g11_9, o12_11);
            }
            { const float eb = bi[114];
              o12_11 = fmaf(eb, g11_17, o12_11);
            }
            { const float eb = bi[115];
              o12_11 = fmaf(eb, g11_29, o12_11);
            }
            { const float eb = bi[116];
              o13_11 = fmaf(eb, g11_0, o13_11);
            }
            { const float eb = bi[117];
              o13_11 = fmaf(eb, g11_1, o13_11);
            }
            { const float eb = bi[118];
              o13_11 = fmaf(eb, g11_4, o13_11);
            }
            { const float eb = bi[119];
              o13_11 = fmaf(eb, g11_2, o13_11);
            }
            { const float eb = bi[120];
              o13_11 = fmaf(eb, g11_5, o13_11);
            }
            { const float eb = bi[121];
              o13_11 = fmaf(eb, g11_11, o13_11);
            }
            { const float eb = bi[122];
              o13_11 = fmaf(eb, g11_6, o13_11);
            }
            { const float eb = bi[123];
              o13_11 = fmaf(eb, g11_12, o13_11);
            }
            { const float eb = bi[124];
              o13_11 = fmaf(eb, g11_22, o13_11);
            }
            { const float eb = bi[125];
              o14_11 = fmaf(eb, g11_0, o14_11);
            }
            { const float eb = bi[126];
              o14_11 = fmaf(eb, g11_1, o14_11);
            }
            { const float eb = bi[127];
              o14_11 = fmaf(eb, g11_4, o14_11);
            }
            { const float eb = bi[128];
              o14_11 = fmaf(eb, g11_10, o14_11);
            }
            { const float eb = bi[129];
              o14_11 = fmaf(eb, g11_20, o14_11);
            }
            { const float eb = bi[130];
              o15_11 = fmaf(eb, g11_0, o15_11);
            }
            { const float eb = bi[131];
              o15_11 = fmaf(eb, g11_1, o15_11);
            }
            { const float eb = bi[132];
              o15_11 = fmaf(eb, g11_4, o15_11);
            }
            { const float eb = bi[133];
              o15_11 = fmaf(eb, g11_2, o15_11);
            }
            { const float eb = bi[134];
              o15_11 = fmaf(eb, g11_5, o15_11);
            }
            { const float eb = bi[135];
              o15_11 = fmaf(eb, g11_11, o15_11);
            }
            { const float eb = bi[136];
              o15_11 = fmaf(eb, g11_3, o15_11);
            }
            { const float eb = bi[137];
              o15_11 = fmaf(eb, g11_7, o15_11);
            }
            { const float eb = bi[138];
              o15_11 = fmaf(eb, g11_14, o15_11);
            }
            { const float eb = bi[139];
              o15_11 = fmaf(eb, g11_8, o15_11);
            }
            { const float eb = bi[140];
              o15_11 = fmaf(eb, g11_15, o15_11);
            }
            { const float eb = bi[141];
              o15_11 = fmaf(eb, g11_26, o15_11);
            }
            { const float eb = bi[142];
              o16_11 = fmaf(eb, g11_0, o16_11);
            }
            { const float eb = bi[143];
              o16_11 = fmaf(eb, g11_1, o16_11);
            }
            { const float eb = bi[144];
              o16_11 = fmaf(eb, g11_4, o16_11);
            }
            { const float eb = bi[145];
              o16_11 = fmaf(eb, g11_10, o16_11);
            }
            { const float eb = bi[146];
              o16_11 = fmaf(eb, g11_3, o16_11);
            }
            { const float eb = bi[147];
              o16_11 = fmaf(eb, g11_7, o16_11);
            }
            { const float eb = bi[148];
              o16_11 = fmaf(eb, g11_14, o16_11);
            }
            { const float eb = bi[149];
              o16_11 = fmaf(eb, g11_25, o16_11);
            }
            { const float eb = bi[150];
              o17_11 = fmaf(eb, g11_0, o17_11);
            }
            { const float eb = bi[151];
              o17_11 = fmaf(eb, g11_1, o17_11);
            }
            { const float eb = bi[152];
              o17_11 = fmaf(eb, g11_4, o17_11);
            }
            { const float eb = bi[153];
              o17_11 = fmaf(eb, g11_10, o17_11);
            }
            { const float eb = bi[154];
              o17_11 = fmaf(eb, g11_2, o17_11);
            }
            { const float eb = bi[155];
              o17_11 = fmaf(eb, g11_5, o17_11);
            }
            { const float eb = bi[156];
              o17_11 = fmaf(eb, g11_11, o17_11);
            }
            { const float eb = bi[157];
              o17_11 = fmaf(eb, g11_21, o17_11);
            }
            { const float eb = bi[158];
              o18_11 = fmaf(eb, g11_0, o18_11);
            }
            { const float eb = bi[159];
              o18_11 = fmaf(eb, g11_2, o18_11);
            }
            { const float eb = bi[160];
              o18_11 = fmaf(eb, g11_3, o18_11);
            }
            { const float eb = bi[161];
              o18_11 = fmaf(eb, g11_8, o18_11);
            }
            { const float eb = bi[162];
              o18_11 = fmaf(eb, g11_9, o18_11);
            }
            { const float eb = bi[163];
              o18_11 = fmaf(eb, g11_18, o18_11);
            }
            { const float eb = bi[164];
              o18_11 = fmaf(eb, g11_19, o18_11);
            }
            { const float eb = bi[165];
              o18_11 = fmaf(eb, g11_33, o18_11);
            }
            { const float eb = bi[166];
              o19_11 = fmaf(eb, g11_0, o19_11);
            }
            { const float eb = bi[167];
              o19_11 = fmaf(eb, g11_2, o19_11);
            }
            { const float eb = bi[168];
              o19_11 = fmaf(eb, g11_6, o19_11);
            }
            { const float eb = bi[169];
              o19_11 = fmaf(eb, g11_13, o19_11);
            }
            { const float eb = bi[170];
              o19_11 = fmaf(eb, g11_3, o19_11);
            }
            { const float eb = bi[171];
              o19_11 = fmaf(eb, g11_8, o19_11);
            }
            { const float eb = bi[172];
              o19_11 = fmaf(eb, g11_16, o19_11);
            }
            { const float eb = bi[173];
              o19_11 = fmaf(eb, g11_28, o19_11);
            }
            { const float eb = bi[174];
              o20_11 = fmaf(eb, g11_0, o20_11);
            }
            { const float eb = bi[175];
              o20_11 = fmaf(eb, g11_1, o20_11);
            }
            { const float eb = bi[176];
              o20_11 = fmaf(eb, g11_4, o20_11);
            }
            { const float eb = bi[177];
              o20_11 = fmaf(eb, g11_2, o20_11);
            }
            { const float eb = bi[178];
              o20_11 = fmaf(eb, g11_5, o20_11);
            }
            { const float eb = bi[179];
              o20_11 = fmaf(eb, g11_11, o20_11);
            }
            { const float eb = bi[180];
              o20_11 = fmaf(eb, g11_3, o20_11);
            }
            { const float eb = bi[181];
              o20_11 = fmaf(eb, g11_7, o20_11);
            }
            { const float eb = bi[182];
              o20_11 = fmaf(eb, g11_14, o20_11);
            }
            { const float eb = bi[183];
              o20_11 = fmaf(eb, g11_8, o20_11);
            }
            { const float eb = bi[184];
              o20_11 = fmaf(eb, g11_15, o20_11);
            }
            { const float eb = bi[185];
              o20_11 = fmaf(eb, g11_26, o20_11);
            }
            { const float eb = bi[186];
              o21_11 = fmaf(eb, g11_0, o21_11);
            }
            { const float eb = bi[187];
              o21_11 = fmaf(eb, g11_2, o21_11);
            }
            { const float eb = bi[188];
              o21_11 = fmaf(eb, g11_6, o21_11);
            }
            { const float eb = bi[189];
              o21_11 = fmaf(eb, g11_3, o21_11);
            }
            { const float eb = bi[190];
              o21_11 = fmaf(eb, g11_8, o21_11);
            }
            { const float eb = bi[191];
              o21_11 = fmaf(eb, g11_16, o21_11);
            }
            { const float eb = bi[192];
              o21_11 = fmaf(eb, g11_9, o21_11);
            }
            { const float eb = bi[193];
              o21_11 = fmaf(eb, g11_18, o21_11);
            }
            { const float eb = bi[194];
              o21_11 = fmaf(eb, g11_31, o21_11);
            }
            { const float eb = bi[195];
              o22_11 = fmaf(eb, g11_0, o22_11);
            }
            { const float eb = bi[196];
              o22_11 = fmaf(eb, g11_1, o22_11);
            }
            { const float eb = bi[197];
              o22_11 = fmaf(eb, g11_2, o22_11);
            }
            { const float eb = bi[198];
              o22_11 = fmaf(eb, g11_5, o22_11);
            }
            { const float eb = bi[199];
              o22_11 = fmaf(eb, g11_3, o22_11);
            }
            { const float eb = bi[200];
              o22_11 = fmaf(eb, g11_7, o22_11);
            }
            { const float eb = bi[201];
              o22_11 = fmaf(eb, g11_8, o22_11);
            }
            { const float eb = bi[202];
              o22_11 = fmaf(eb, g11_15, o22_11);
            }
            { const float eb = bi[203];
              o22_11 = fmaf(eb, g11_9, o22_11);
            }
            { const float eb = bi[204];
              o22_11 = fmaf(eb, g11_17, o22_11);
            }
            { const float eb = bi[205];
              o22_11 = fmaf(eb, g11_18, o22_11);
            }
            { const float eb = bi[206];
              o22_11 = fmaf(eb, g11_30, o22_11);
            }
            { const float eb = bi[207];
              o23_11 = fmaf(eb, g11_0, o23_11);
            }
            { const float eb = bi[208];
              o23_11 = fmaf(eb, g11_1, o23_11);
            }
            { const float eb = bi[209];
              o23_11 = fmaf(eb, g11_2, o23_11);
            }
            { const float eb = bi[210];
              o23_11 = fmaf(eb, g11_5, o23_11);
            }
            { const float eb = bi[211];
              o23_11 = fmaf(eb, g11_6, o23_11);
            }
            { const float eb = bi[212];
              o23_11 = fmaf(eb, g11_12, o23_11);
            }
            { const float eb = bi[213];
              o23_11 = fmaf(eb, g11_3, o23_11);
            }
            { const float eb = bi[214];
              o23_11 = fmaf(eb, g11_7, o23_11);
            }
            { const float eb = bi[215];
              o23_11 = fmaf(eb, g11_8, o23_11);
            }
            { const float eb = bi[216];
              o23_11 = fmaf(eb, g11_15, o23_11);
            }
            { const float eb = bi[217];
              o23_11 = fmaf(eb, g11_16, o23_11);
            }
            { const float eb = bi[218];
              o23_11 = fmaf(eb, g11_27, o23_11);
            }
            { const float eb = bi[219];
              o24_11 = fmaf(eb, g11_0, o24_11);
            }
            { const float eb = bi[220];
              o24_11 = fmaf(eb, g11_1, o24_11);
            }
            { const float eb = bi[221];
              o24_11 = fmaf(eb, g11_3, o24_11);
            }
            { const float eb = bi[222];
              o24_11 = fmaf(eb, g11_7, o24_11);
            }
            { const float eb = bi[223];
              o24_11 = fmaf(eb, g11_9, o24_11);
            }
            { const float eb = bi[224];
              o24_11 = fmaf(eb, g11_17, o24_11);
            }
            { const float eb = bi[225];
              o24_11 = fmaf(eb, g11_19, o24_11);
            }
            { const float eb = bi[226];
              o24_11 = fmaf(eb, g11_32, o24_11);
            }
            { const float eb = bi[227];
              o25_11 = fmaf(eb, g11_0, o25_11);
            }
            { const float eb = bi[228];
              o25_11 = fmaf(eb, g11_1, o25_11);
            }
            { const float eb = bi[229];
              o25_11 = fmaf(eb, g11_2, o25_11);
            }
            { const float eb = bi[230];
              o25_11 = fmaf(eb, g11_5, o25_11);
            }
            { const float eb = bi[231];
              o25_11 = fmaf(eb, g11_6, o25_11);
            }
            { const float eb = bi[232];
              o25_11 = fmaf(eb, g11_12, o25_11);
            }
            { const float eb = bi[233];
              o25_11 = fmaf(eb, g11_3, o25_11);
            }
            { const float eb = bi[234];
              o25_11 = fmaf(eb, g11_7, o25_11);
            }
            { const float eb = bi[235];
              o25_11 = fmaf(eb, g11_8, o25_11);
            }
            { const float eb = bi[236];
              o25_11 = fmaf(eb, g11_15, o25_11);
            }
            { const float eb = bi[237];
              o25_11 = fmaf(eb, g11_16, o25_11);
            }
            { const float eb = bi[238];
              o25_11 = fmaf(eb, g11_27, o25_11);
            }
            { const float eb = bi[239];
              o26_11 = fmaf(eb, g11_0, o26_11);
            }
            { const float eb = bi[240];
              o26_11 = fmaf(eb, g11_1, o26_11);
            }
            { const float eb = bi[241];
              o26_11 = fmaf(eb, g11_4, o26_11);
            }
            { const float eb = bi[242];
              o26_11 = fmaf(eb, g11_10, o26_11);
            }
            { const float eb = bi[243];
              o26_11 = fmaf(eb, g11_3, o26_11);
            }
            { const float eb = bi[244];
              o26_11 = fmaf(eb, g11_7, o26_11);
            }
            { const float eb = bi[245];
              o26_11 = fmaf(eb, g11_14, o26_11);
            }
            { const float eb = bi[246];
              o26_11 = fmaf(eb, g11_25, o26_11);
            }
            { const float eb = bi[247];
              o27_11 = fmaf(eb, g11_0, o27_11);
            }
            { const float eb = bi[248];
              o27_11 = fmaf(eb, g11_1, o27_11);
            }
            { const float eb = bi[249];
              o27_11 = fmaf(eb, g11_2, o27_11);
            }
            { const float eb = bi[250];
              o27_11 = fmaf(eb, g11_5, o27_11);
            }
            { const float eb = bi[251];
              o27_11 = fmaf(eb, g11_3, o27_11);
            }
            { const float eb = bi[252];
              o27_11 = fmaf(eb, g11_7, o27_11);
            }
            { const float eb = bi[253];
              o27_11 = fmaf(eb, g11_8, o27_11);
            }
            { const float eb = bi[254];
              o27_11 = fmaf(eb, g11_15, o27_11);
            }
            { const float eb = bi[255];
              o27_11 = fmaf(eb, g11_9, o27_11);
            }
            { const float eb = bi[256];
              o27_11 = fmaf(eb, g11_17, o27_11);
            }
            { const float eb = bi[257];
              o27_11 = fmaf(eb, g11_18, o27_11);
            }
            { const float eb = bi[258];
              o27_11 = fmaf(eb, g11_30, o27_11);
            }
            { const float eb = bi[259];
              o28_11 = fmaf(eb, g11_0, o28_11);
            }
            { const float eb = bi[260];
              o28_11 = fmaf(eb, g11_1, o28_11);
            }
            { const float eb = bi[261];
              o28_11 = fmaf(eb, g11_4, o28_11);
            }
            { const float eb = bi[262];
              o28_11 = fmaf(eb, g11_3, o28_11);
            }
            { const float eb = bi[263];
              o28_11 = fmaf(eb, g11_7, o28_11);
            }
            { const float eb = bi[264];
              o28_11 = fmaf(eb, g11_14, o28_11);
            }
            { const float eb = bi[265];
              o28_11 = fmaf(eb, g11_9, o28_11);
            }
            { const float eb = bi[266];
              o28_11 = fmaf(eb, g11_17, o28_11);
            }
            { const float eb = bi[267];
              o28_11 = fmaf(eb, g11_29, o28_11);
            }
            { const float eb = bi[268];
              o29_11 = fmaf(eb, g11_0, o29_11);
            }
            { const float eb = bi[269];
              o29_11 = fmaf(eb, g11_1, o29_11);
            }
            { const float eb = bi[270];
              o29_11 = fmaf(eb, g11_4, o29_11);
            }
            { const float eb = bi[271];
              o29_11 = fmaf(eb, g11_2, o29_11);
            }
            { const float eb = bi[272];
              o29_11 = fmaf(eb, g11_5, o29_11);
            }
            { const float eb = bi[273];
              o29_11 = fmaf(eb, g11_11, o29_11);
            }
            { const float eb = bi[274];
              o29_11 = fmaf(eb, g11_3, o29_11);
            }
            { const float eb = bi[275];
              o29_11 = fmaf(eb, g11_7, o29_11);
            }
            { const float eb = bi[276];
              o29_11 = fmaf(eb, g11_14, o29_11);
            }
            { const float eb = bi[277];
              o29_11 = fmaf(eb, g11_8, o29_11);
            }
            { const float eb = bi[278];
              o29_11 = fmaf(eb, g11_15, o29_11);
            }
            { const float eb = bi[279];
              o29_11 = fmaf(eb, g11_26, o29_11);
            }
            { const float eb = bi[280];
              o30_11 = fmaf(eb, g11_0, o30_11);
            }
            { const float eb = bi[281];
              o30_11 = fmaf(eb, g11_1, o30_11);
            }
            { const float eb = bi[282];
              o30_11 = fmaf(eb, g11_2, o30_11);
            }
            { const float eb = bi[283];
              o30_11 = fmaf(eb, g11_5, o30_11);
            }
            { const float eb = bi[284];
              o30_11 = fmaf(eb, g11_3, o30_11);
            }
            { const float eb = bi[285];
              o30_11 = fmaf(eb, g11_7, o30_11);
            }
            { const float eb = bi[286];
              o30_11 = fmaf(eb, g11_8, o30_11);
            }
            { const float eb = bi[287];
              o30_11 = fmaf(eb, g11_15, o30_11);
            }
            { const float eb = bi[288];
              o30_11 = fmaf(eb, g11_9, o30_11);
            }
            { const float eb = bi[289];
              o30_11 = fmaf(eb, g11_17, o30_11);
            }
            { const float eb = bi[290];
              o30_11 = fmaf(eb, g11_18, o30_11);
            }
            { const float eb = bi[291];
              o30_11 = fmaf(eb, g11_30, o30_11);
            }
            { const float eb = bi[292];
              o31_11 = fmaf(eb, g11_0, o31_11);
            }
            { const float eb = bi[293];
              o31_11 = fmaf(eb, g11_1, o31_11);
            }
            { const float eb = bi[294];
              o31_11 = fmaf(eb, g11_2, o31_11);
            }
            { const float eb = bi[295];
              o31_11 = fmaf(eb, g11_5, o31_11);
            }
            { const float eb = bi[296];
              o31_11 = fmaf(eb, g11_6, o31_11);
            }
            { const float eb = bi[297];
              o31_11 = fmaf(eb, g11_12, o31_11);
            }
            { const float eb = bi[298];
              o31_11 = fmaf(eb, g11_13, o31_11);
            }
            { const float eb = bi[299];
              o31_11 = fmaf(eb, g11_23, o31_11);
            }
            { const float eb = bi[300];
              o32_11 = fmaf(eb, g11_0, o32_11);
            }
            { const float eb = bi[301];
              o32_11 = fmaf(eb, g11_1, o32_11);
            }
            { const float eb = bi[302];
              o32_11 = fmaf(eb, g11_4, o32_11);
            }
            { const float eb = bi[303];
              o32_11 = fmaf(eb, g11_10, o32_11);
            }
            { const float eb = bi[304];
              o32_11 = fmaf(eb, g11_2, o32_11);
            }
            { const float eb = bi[305];
              o32_11 = fmaf(eb, g11_5, o32_11);
            }
            { const float eb = bi[306];
              o32_11 = fmaf(eb, g11_11, o32_11);
            }
            { const float eb = bi[307];
              o32_11 = fmaf(eb, g11_21, o32_11);
            }
            { const float eb = bi[308];
              o33_11 = fmaf(eb, g11_0, o33_11);
            }
            { const float eb = bi[309];
              o33_11 = fmaf(eb, g11_1, o33_11);
            }
            { const float eb = bi[310];
              o33_11 = fmaf(eb, g11_2, o33_11);
            }
            { const float eb = bi[311];
              o33_11 = fmaf(eb, g11_5, o33_11);
            }
            { const float eb = bi[312];
              o33_11 = fmaf(eb, g11_6, o33_11);
            }
            { const float eb = bi[313];
              o33_11 = fmaf(eb, g11_12, o33_11);
            }
            { const float eb = bi[314];
              o33_11 = fmaf(eb, g11_3, o33_11);
            }
            { const float eb = bi[315];
              o33_11 = fmaf(eb, g11_7, o33_11);
            }
            { const float eb = bi[316];
              o33_11 = fmaf(eb, g11_8, o33_11);
            }
            { const float eb = bi[317];
              o33_11 = fmaf(eb, g11_15, o33_11);
            }
            { const float eb = bi[318];
              o33_11 = fmaf(eb, g11_16, o33_11);
            }
            { const float eb = bi[319];
              o33_11 = fmaf(eb, g11_27, o33_11);
            }
            { const float eb = bi[320];
              o34_11 = fmaf(eb, g11_0, o34_11);
            }
            { const float eb = bi[321];
              o34_11 = fmaf(eb, g11_1, o34_11);
            }
            { const float eb = bi[322];
              o34_11 = fmaf(eb, g11_4, o34_11);
            }
            { const float eb = bi[323];
              o34_11 = fmaf(eb, g11_2, o34_11);
            }
            { const float eb = bi[324];
              o34_11 = fmaf(eb, g11_5, o34_11);
            }
            { const float eb = bi[325];
              o34_11 = fmaf(eb, g11_11, o34_11);
            }
            { const float eb = bi[326];
              o34_11 = fmaf(eb, g11_3, o34_11);
            }
            { const float eb = bi[327];
              o34_11 = fmaf(eb, g11_7, o34_11);
            }
            { const float eb = bi[328];
              o34_11 = fmaf(eb, g11_14, o34_11);
            }
            { const float eb = bi[329];
              o34_11 = fmaf(eb, g11_8, o34_11);
            }
            { const float eb = bi[330];
              o34_11 = fmaf(eb, g11_15, o34_11);
            }
            { const float eb = bi[331];
              o34_11 = fmaf(eb, g11_26, o34_11);
            }
            { const float eb = bi[332];
              o35_11 = fmaf(eb, g11_0, o35_11);
            }
            { const float eb = bi[333];
              o35_11 = fmaf(eb, g11_1, o35_11);
            }
            { const float eb = bi[334];
              o35_11 = fmaf(eb, g11_4, o35_11);
            }
            { const float eb = bi[335];
              o35_11 = fmaf(eb, g11_2, o35_11);
            }
            { const float eb = bi[336];
              o35_11 = fmaf(eb, g11_5, o35_11);
            }
            { const float eb = bi[337];
              o35_11 = fmaf(eb, g11_11, o35_11);
            }
            { const float eb = bi[338];
              o35_11 = fmaf(eb, g11_6, o35_11);
            }
            { const float eb = bi[339];
              o35_11 = fmaf(eb, g11_12, o35_11);
            }
            { const float eb = bi[340];
              o35_11 = fmaf(eb, g11_22, o35_11);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk11 = PT[(fI + 2) * N + fJ + 3];
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
            const double Abd0_3 = PA[(fQ + 0) * N + fJ + 3];
            const double Abd1_3 = PA[(fQ + 1) * N + fJ + 3];
            const double Abd2_3 = PA[(fQ + 2) * N + fJ + 3];
            const double Abd3_3 = PA[(fQ + 3) * N + fJ + 3];
            const double Abd4_3 = PA[(fQ + 4) * N + fJ + 3];
            const double Abd5_3 = PA[(fQ + 5) * N + fJ + 3];
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
            const double Abc4_2 = PA[(fQ + 4) * N + fI + 2];
            const double Abc5_2 = PA[(fQ + 5) * N + fI + 2];
            const double Aac0_2 = PA[(fP + 0) * N + fI + 2];
            const double Aac1_2 = PA[(fP + 1) * N + fI + 2];
            const double Aac2_2 = PA[(fP + 2) * N + fI + 2];
            const double Aac3_2 = PA[(fP + 3) * N + fI + 2];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
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
            jab24 += o24_11 * ptk11;
            jab25 += o25_11 * ptk11;
            jab26 += o26_11 * ptk11;
            jab27 += o27_11 * ptk11;
            jab28 += o28_11 * ptk11;
            jab29 += o29_11 * ptk11;
            jab30 += o30_11 * ptk11;
            jab31 += o31_11 * ptk11;
            jab32 += o32_11 * ptk11;
            jab33 += o33_11 * ptk11;
            jab34 += o34_11 * ptk11;
            jab35 += o35_11 * ptk11;
            atomicAdd(Jacc + (fI + 2) * N + fJ + 3, 2.0 * deg * (o0_11 * ptb0 + o1_11 * ptb1 + o2_11 * ptb2 + o3_11 * ptb3 + o4_11 * ptb4 + o5_11 * ptb5 + o6_11 * ptb6 + o7_11 * ptb7 + o8_11 * ptb8 + o9_11 * ptb9 + o10_11 * ptb10 + o11_11 * ptb11 + o12_11 * ptb12 + o13_11 * ptb13 + o14_11 * ptb14 + o15_11 * ptb15 + o16_11 * ptb16 + o17_11 * ptb17 + o18_11 * ptb18 + o19_11 * ptb19 + o20_11 * ptb20 + o21_11 * ptb21 + o22_11 * ptb22 + o23_11 * ptb23 + o24_11 * ptb24 + o25_11 * ptb25 + o26_11 * ptb26 + o27_11 * ptb27 + o28_11 * ptb28 + o29_11 * ptb29 + o30_11 * ptb30 + o31_11 * ptb31 + o32_11 * ptb32 + o33_11 * ptb33 + o34_11 * ptb34 + o35_11 * ptb35));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_11 * Abd0_3 + o1_11 * Abd1_3 + o2_11 * Abd2_3 + o3_11 * Abd3_3 + o4_11 * Abd4_3 + o5_11 * Abd5_3));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_11 * Aad0_3 + o6_11 * Aad1_3 + o12_11 * Aad2_3 + o18_11 * Aad3_3 + o24_11 * Aad4_3 + o30_11 * Aad5_3));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 3, deg * (o0_11 * Abc0_2 + o1_11 * Abc1_2 + o2_11 * Abc2_2 + o3_11 * Abc3_2 + o4_11 * Abc4_2 + o5_11 * Abc5_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 3, deg * (o0_11 * Aac0_2 + o6_11 * Aac1_2 + o12_11 * Aac2_2 + o18_11 * Aac3_2 + o24_11 * Aac4_2 + o30_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 1) * N + fI + 2, deg * (o1_11 * Aad0_3 + o7_11 * Aad1_3 + o13_11 * Aad2_3 + o19_11 * Aad3_3 + o25_11 * Aad4_3 + o31_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 1) * N + fJ + 3, deg * (o1_11 * Aac0_2 + o7_11 * Aac1_2 + o13_11 * Aac2_2 + o19_11 * Aac3_2 + o25_11 * Aac4_2 + o31_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 2) * N + fI + 2, deg * (o2_11 * Aad0_3 + o8_11 * Aad1_3 + o14_11 * Aad2_3 + o20_11 * Aad3_3 + o26_11 * Aad4_3 + o32_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 2) * N + fJ + 3, deg * (o2_11 * Aac0_2 + o8_11 * Aac1_2 + o14_11 * Aac2_2 + o20_11 * Aac3_2 + o26_11 * Aac4_2 + o32_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 3) * N + fI + 2, deg * (o3_11 * Aad0_3 + o9_11 * Aad1_3 + o15_11 * Aad2_3 + o21_11 * Aad3_3 + o27_11 * Aad4_3 + o33_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 3) * N + fJ + 3, deg * (o3_11 * Aac0_2 + o9_11 * Aac1_2 + o15_11 * Aac2_2 + o21_11 * Aac3_2 + o27_11 * Aac4_2 + o33_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 4) * N + fI + 2, deg * (o4_11 * Aad0_3 + o10_11 * Aad1_3 + o16_11 * Aad2_3 + o22_11 * Aad3_3 + o28_11 * Aad4_3 + o34_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 4) * N + fJ + 3, deg * (o4_11 * Aac0_2 + o10_11 * Aac1_2 + o16_11 * Aac2_2 + o22_11 * Aac3_2 + o28_11 * Aac4_2 + o34_11 * Aac5_2));
            atomicAdd(KAacc + (fQ + 5) * N + fI + 2, deg * (o5_11 * Aad0_3 + o11_11 * Aad1_3 + o17_11 * Aad2_3 + o23_11 * Aad3_3 + o29_11 * Aad4_3 + o35_11 * Aad5_3));
            atomicAdd(KAacc + (fQ + 5) * N + fJ + 3, deg * (o5_11 * Aac0_2 + o11_11 * Aac1_2 + o17_11 * Aac2_2 + o23_11 * Aac3_2 + o29_11 * Aac4_2 + o35_11 * Aac5_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o6_11 * Abd0_3 + o7_11 * Abd1_3 + o8_11 * Abd2_3 + o9_11 * Abd3_3 + o10_11 * Abd4_3 + o11_11 * Abd5_3));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 3, deg * (o6_11 * Abc0_2 + o7_11 * Abc1_2 + o8_11 * Abc2_2 + o9_11 * Abc3_2 + o10_11 * Abc4_2 + o11_11 * Abc5_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o12_11 * Abd0_3 + o13_11 * Abd1_3 + o14_11 * Abd2_3 + o15_11 * Abd3_3 + o16_11 * Abd4_3 + o17_11 * Abd5_3));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 3, deg * (o12_11 * Abc0_2 + o13_11 * Abc1_2 + o14_11 * Abc2_2 + o15_11 * Abc3_2 + o16_11 * Abc4_2 + o17_11 * Abc5_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o18_11 * Abd0_3 + o19_11 * Abd1_3 + o20_11 * Abd2_3 + o21_11 * Abd3_3 + o22_11 * Abd4_3 + o23_11 * Abd5_3));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 3, deg * (o18_11 * Abc0_2 + o19_11 * Abc1_2 + o20_11 * Abc2_2 + o21_11 * Abc3_2 + o22_11 * Abc4_2 + o23_11 * Abc5_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o24_11 * Abd0_3 + o25_11 * Abd1_3 + o26_11 * Abd2_3 + o27_11 * Abd3_3 + o28_11 * Abd4_3 + o29_11 * Abd5_3));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 3, deg * (o24_11 * Abc0_2 + o25_11 * Abc1_2 + o26_11 * Abc2_2 + o27_11 * Abc3_2 + o28_11 * Abc4_2 + o29_11 * Abc5_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o30_11 * Abd0_3 + o31_11 * Abd1_3 + o32_11 * Abd2_3 + o33_11 * Abd3_3 + o34_11 * Abd4_3 + o35_11 * Abd5_3));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 3, deg * (o30_11 * Abc0_2 + o31_11 * Abc1_2 + o32_11 * Abc2_2 + o33_11 * Abc3_2 + o34_11 * Abc4_2 + o35_11 * Abc5_2));
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
