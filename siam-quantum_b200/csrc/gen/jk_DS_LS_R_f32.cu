// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DS_LS_R_f32(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 26; x += blockDim.x) sbra[x] = a.bra_prims_f[bp.poff + (long long)x * bp.kstride];
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
          for (int i = gi; i < nbp; i += si) {
            const float* __restrict__ bi = sbra + i * 26;
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
              const float* __restrict__ kj = kprim + (long long)j * 12 * kS;
              const float q = kj[0];
              const float pq = p + q;
              const float rs = rsqrtf(pq);
              if (TWO_PI_2_5F * kpb * kj[4 * kS] * rs < PRIM_CUTOFF_F) continue;
              ++nprimq;
              const float alpha = p * q * (rs * rs);
              const float X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const float T = alpha * fmaf(X, X, fmaf(Y, Y, Z * Z));
              float F[4];
              sqb::boysf<3>(T, a.boys_tab_f, F);
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
              const float ek0_0 = kj[5 * kS];
              const float ek1_0 = kj[6 * kS];
              const float ek1_1 = -kj[7 * kS];
              const float ek2_0 = kj[8 * kS];
              const float ek2_1 = -kj[9 * kS];
              const float ek3_0 = kj[10 * kS];
              const float ek3_1 = -kj[11 * kS];
              g0_0 = fmaf(ek0_0, b0, g0_0);
              g1_0 = fmaf(ek1_0, b0, g1_0);
              g2_0 = fmaf(ek2_0, b0, g2_0);
              g3_0 = fmaf(ek3_0, b0, g3_0);
              const float r0_0_0_1 = Z * b1;
              g0_1 = fmaf(ek0_0, r0_0_0_1, g0_1);
              g1_1 = fmaf(ek1_0, r0_0_0_1, g1_1);
              g2_1 = fmaf(ek2_0, r0_0_0_1, g2_1);
              g3_1 = fmaf(ek3_0, r0_0_0_1, g3_1);
              g3_0 = fmaf(ek3_1, r0_0_0_1, g3_0);
              const float r0_0_1_0 = Y * b1;
              g0_2 = fmaf(ek0_0, r0_0_1_0, g0_2);
              g1_2 = fmaf(ek1_0, r0_0_1_0, g1_2);
              g2_2 = fmaf(ek2_0, r0_0_1_0, g2_2);
              g2_0 = fmaf(ek2_1, r0_0_1_0, g2_0);
              g3_2 = fmaf(ek3_0, r0_0_1_0, g3_2);
              const float r0_1_0_0 = X * b1;
              g0_3 = fmaf(ek0_0, r0_1_0_0, g0_3);
              g1_3 = fmaf(ek1_0, r0_1_0_0, g1_3);
              g1_0 = fmaf(ek1_1, r0_1_0_0, g1_0);
              g2_3 = fmaf(ek2_0, r0_1_0_0, g2_3);
              g3_3 = fmaf(ek3_0, r0_1_0_0, g3_3);
              const float r1_0_0_1 = Z * b2;
              const float r0_0_0_2 = fmaf(Z, r1_0_0_1, b1);
              g0_4 = fmaf(ek0_0, r0_0_0_2, g0_4);
              g1_4 = fmaf(ek1_0, r0_0_0_2, g1_4);
              g2_4 = fmaf(ek2_0, r0_0_0_2, g2_4);
              g3_4 = fmaf(ek3_0, r0_0_0_2, g3_4);
              g3_1 = fmaf(ek3_1, r0_0_0_2, g3_1);
              const float r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fmaf(ek0_0, r0_0_1_1, g0_5);
              g1_5 = fmaf(ek1_0, r0_0_1_1, g1_5);
              g2_5 = fmaf(ek2_0, r0_0_1_1, g2_5);
              g2_1 = fmaf(ek2_1, r0_0_1_1, g2_1);
              g3_5 = fmaf(ek3_0, r0_0_1_1, g3_5);
              g3_2 = fmaf(ek3_1, r0_0_1_1, g3_2);
              const float r1_0_1_0 = Y * b2;
              const float r0_0_2_0 = fmaf(Y, r1_0_1_0, b1);
              g0_6 = fmaf(ek0_0, r0_0_2_0, g0_6);
              g1_6 = fmaf(ek1_0, r0_0_2_0, g1_6);
              g2_6 = fmaf(ek2_0, r0_0_2_0, g2_6);
              g2_2 = fmaf(ek2_1, r0_0_2_0, g2_2);
              g3_6 = fmaf(ek3_0, r0_0_2_0, g3_6);
              const float r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fmaf(ek0_0, r0_1_0_1, g0_7);
              g1_7 = fmaf(ek1_0, r0_1_0_1, g1_7);
              g1_1 = fmaf(ek1_1, r0_1_0_1, g1_1);
              g2_7 = fmaf(ek2_0, r0_1_0_1, g2_7);
              g3_7 = fmaf(ek3_0, r0_1_0_1, g3_7);
              g3_3 = fmaf(ek3_1, r0_1_0_1, g3_3);
              const float r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fmaf(ek0_0, r0_1_1_0, g0_8);
              g1_8 = fmaf(ek1_0, r0_1_1_0, g1_8);
              g1_2 = fmaf(ek1_1, r0_1_1_0, g1_2);
              g2_8 = fmaf(ek2_0, r0_1_1_0, g2_8);
              g2_3 = fmaf(ek2_1, r0_1_1_0, g2_3);
              g3_8 = fmaf(ek3_0, r0_1_1_0, g3_8);
              const float r1_1_0_0 = X * b2;
              const float r0_2_0_0 = fmaf(X, r1_1_0_0, b1);
              g0_9 = fmaf(ek0_0, r0_2_0_0, g0_9);
              g1_9 = fmaf(ek1_0, r0_2_0_0, g1_9);
              g1_3 = fmaf(ek1_1, r0_2_0_0, g1_3);
              g2_9 = fmaf(ek2_0, r0_2_0_0, g2_9);
              g3_9 = fmaf(ek3_0, r0_2_0_0, g3_9);
              const float r2_0_0_1 = Z * b3;
              const float r1_0_0_2 = fmaf(Z, r2_0_0_1, b2);
              const float r0_0_0_3 = fmaf(Z, r1_0_0_2, 2.0f * r1_0_0_1);
              g3_4 = fmaf(ek3_1, r0_0_0_3, g3_4);
              const float r0_0_1_2 = Y * r1_0_0_2;
              g2_4 = fmaf(ek2_1, r0_0_1_2, g2_4);
              g3_5 = fmaf(ek3_1, r0_0_1_2, g3_5);
              const float r1_0_1_1 = Y * r2_0_0_1;
              const float r0_0_2_1 = fmaf(Y, r1_0_1_1, r1_0_0_1);
              g2_5 = fmaf(ek2_1, r0_0_2_1, g2_5);
              g3_6 = fmaf(ek3_1, r0_0_2_1, g3_6);
              const float r2_0_1_0 = Y * b3;
              const float r1_0_2_0 = fmaf(Y, r2_0_1_0, b2);
              const float r0_0_3_0 = fmaf(Y, r1_0_2_0, 2.0f * r1_0_1_0);
              g2_6 = fmaf(ek2_1, r0_0_3_0, g2_6);
              const float r0_1_0_2 = X * r1_0_0_2;
              g1_4 = fmaf(ek1_1, r0_1_0_2, g1_4);
              g3_7 = fmaf(ek3_1, r0_1_0_2, g3_7);
              const float r0_1_1_1 = X * r1_0_1_1;
              g1_5 = fmaf(ek1_1, r0_1_1_1, g1_5);
              g2_7 = fmaf(ek2_1, r0_1_1_1, g2_7);
              g3_8 = fmaf(ek3_1, r0_1_1_1, g3_8);
              const float r0_1_2_0 = X * r1_0_2_0;
              g1_6 = fmaf(ek1_1, r0_1_2_0, g1_6);
              g2_8 = fmaf(ek2_1, r0_1_2_0, g2_8);
              const float r1_1_0_1 = X * r2_0_0_1;
              const float r0_2_0_1 = fmaf(X, r1_1_0_1, r1_0_0_1);
              g1_7 = fmaf(ek1_1, r0_2_0_1, g1_7);
              g3_9 = fmaf(ek3_1, r0_2_0_1, g3_9);
              const float r1_1_1_0 = X * r2_0_1_0;
              const float r0_2_1_0 = fmaf(X, r1_1_1_0, r1_0_1_0);
              g1_8 = fmaf(ek1_1, r0_2_1_0, g1_8);
              g2_9 = fmaf(ek2_1, r0_2_1_0, g2_9);
              const float r2_1_0_0 = X * b3;
              const float r1_2_0_0 = fmaf(X, r2_1_0_0, b2);
              const float r0_3_0_0 = fmaf(X, r1_2_0_0, 2.0f * r1_1_0_0);
              g1_9 = fmaf(ek1_1, r0_3_0_0, g1_9);
            }
            { const float eb = bi[5];
              o0_0 = fmaf(eb, g0_0, o0_0);
              o0_1 = fmaf(eb, g1_0, o0_1);
              o0_2 = fmaf(eb, g2_0, o0_2);
              o0_3 = fmaf(eb, g3_0, o0_3);
            }
            { const float eb = bi[6];
              o0_0 = fmaf(eb, g0_3, o0_0);
              o0_1 = fmaf(eb, g1_3, o0_1);
              o0_2 = fmaf(eb, g2_3, o0_2);
              o0_3 = fmaf(eb, g3_3, o0_3);
            }
            { const float eb = bi[7];
              o0_0 = fmaf(eb, g0_9, o0_0);
              o0_1 = fmaf(eb, g1_9, o0_1);
              o0_2 = fmaf(eb, g2_9, o0_2);
              o0_3 = fmaf(eb, g3_9, o0_3);
            }
            { const float eb = bi[8];
              o1_0 = fmaf(eb, g0_0, o1_0);
              o1_1 = fmaf(eb, g1_0, o1_1);
              o1_2 = fmaf(eb, g2_0, o1_2);
              o1_3 = fmaf(eb, g3_0, o1_3);
            }
            { const float eb = bi[9];
              o1_0 = fmaf(eb, g0_2, o1_0);
              o1_1 = fmaf(eb, g1_2, o1_1);
              o1_2 = fmaf(eb, g2_2, o1_2);
              o1_3 = fmaf(eb, g3_2, o1_3);
            }
            { const float eb = bi[10];
              o1_0 = fmaf(eb, g0_6, o1_0);
              o1_1 = fmaf(eb, g1_6, o1_1);
              o1_2 = fmaf(eb, g2_6, o1_2);
              o1_3 = fmaf(eb, g3_6, o1_3);
            }
            { const float eb = bi[11];
              o2_0 = fmaf(eb, g0_0, o2_0);
              o2_1 = fmaf(eb, g1_0, o2_1);
              o2_2 = fmaf(eb, g2_0, o2_2);
              o2_3 = fmaf(eb, g3_0, o2_3);
            }
            { const float eb = bi[12];
              o2_0 = fmaf(eb, g0_1, o2_0);
              o2_1 = fmaf(eb, g1_1, o2_1);
              o2_2 = fmaf(eb, g2_1, o2_2);
              o2_3 = fmaf(eb, g3_1, o2_3);
            }
            { const float eb = bi[13];
              o2_0 = fmaf(eb, g0_4, o2_0);
              o2_1 = fmaf(eb, g1_4, o2_1);
              o2_2 = fmaf(eb, g2_4, o2_2);
              o2_3 = fmaf(eb, g3_4, o2_3);
            }
            { const float eb = bi[14];
              o3_0 = fmaf(eb, g0_0, o3_0);
              o3_1 = fmaf(eb, g1_0, o3_1);
              o3_2 = fmaf(eb, g2_0, o3_2);
              o3_3 = fmaf(eb, g3_0, o3_3);
            }
            { const float eb = bi[15];
              o3_0 = fmaf(eb, g0_2, o3_0);
              o3_1 = fmaf(eb, g1_2, o3_1);
              o3_2 = fmaf(eb, g2_2, o3_2);
              o3_3 = fmaf(eb, g3_2, o3_3);
            }
            { const float eb = bi[16];
              o3_0 = fmaf(eb, g0_3, o3_0);
              o3_1 = fmaf(eb, g1_3, o3_1);
              o3_2 = fmaf(eb, g2_3, o3_2);
              o3_3 = fmaf(eb, g3_3, o3_3);
            }
            { const float eb = bi[17];
              o3_0 = fmaf(eb, g0_8, o3_0);
              o3_1 = fmaf(eb, g1_8, o3_1);
              o3_2 = fmaf(eb, g2_8, o3_2);
              o3_3 = fmaf(eb, g3_8, o3_3);
            }
            { const float eb = bi[18];
              o4_0 = fmaf(eb, g0_0, o4_0);
              o4_1 = fmaf(eb, g1_0, o4_1);
              o4_2 = fmaf(eb, g2_0, o4_2);
              o4_3 = fmaf(eb, g3_0, o4_3);
            }
            { const float eb = bi[19];
              o4_0 = fmaf(eb, g0_1, o4_0);
              o4_1 = fmaf(eb, g1_1, o4_1);
              o4_2 = fmaf(eb, g2_1, o4_2);
              o4_3 = fmaf(eb, g3_1, o4_3);
            }
            { const float eb = bi[20];
              o4_0 = fmaf(eb, g0_3, o4_0);
              o4_1 = fmaf(eb, g1_3, o4_1);
              o4_2 = fmaf(eb, g2_3, o4_2);
              o4_3 = fmaf(eb, g3_3, o4_3);
            }
            { const float eb = bi[21];
              o4_0 = fmaf(eb, g0_7, o4_0);
              o4_1 = fmaf(eb, g1_7, o4_1);
              o4_2 = fmaf(eb, g2_7, o4_2);
              o4_3 = fmaf(eb, g3_7, o4_3);
            }
            { const float eb = bi[22];
              o5_0 = fmaf(eb, g0_0, o5_0);
              o5_1 = fmaf(eb, g1_0, o5_1);
              o5_2 = fmaf(eb, g2_0, o5_2);
              o5_3 = fmaf(eb, g3_0, o5_3);
            }
            { const float eb = bi[23];
              o5_0 = fmaf(eb, g0_1, o5_0);
              o5_1 = fmaf(eb, g1_1, o5_1);
              o5_2 = fmaf(eb, g2_1, o5_2);
              o5_3 = fmaf(eb, g3_1, o5_3);
            }
            { const float eb = bi[24];
              o5_0 = fmaf(eb, g0_2, o5_0);
              o5_1 = fmaf(eb, g1_2, o5_1);
              o5_2 = fmaf(eb, g2_2, o5_2);
              o5_3 = fmaf(eb, g3_2, o5_3);
            }
            { const float eb = bi[25];
              o5_0 = fmaf(eb, g0_5, o5_0);
              o5_1 = fmaf(eb, g1_5, o5_1);
              o5_2 = fmaf(eb, g2_5, o5_2);
              o5_3 = fmaf(eb, g3_5, o5_3);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptk1 = PT[(fI + 1) * N + fJ + 0];
            const double ptk2 = PT[(fI + 2) * N + fJ + 0];
            const double ptk3 = PT[(fI + 3) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 1) * N + fQ + 0];
            const double ptb2 = PT[(fP + 2) * N + fQ + 0];
            const double ptb3 = PT[(fP + 3) * N + fQ + 0];
            const double ptb4 = PT[(fP + 4) * N + fQ + 0];
            const double ptb5 = PT[(fP + 5) * N + fQ + 0];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Aad3_0 = PA[(fP + 3) * N + fJ + 0];
            const double Aad4_0 = PA[(fP + 4) * N + fJ + 0];
            const double Aad5_0 = PA[(fP + 5) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Abc0_1 = PA[(fQ + 0) * N + fI + 1];
            const double Abc0_2 = PA[(fQ + 0) * N + fI + 2];
            const double Abc0_3 = PA[(fQ + 0) * N + fI + 3];
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
            const double Aac4_0 = PA[(fP + 4) * N + fI + 0];
            const double Aac4_1 = PA[(fP + 4) * N + fI + 1];
            const double Aac4_2 = PA[(fP + 4) * N + fI + 2];
            const double Aac4_3 = PA[(fP + 4) * N + fI + 3];
            const double Aac5_0 = PA[(fP + 5) * N + fI + 0];
            const double Aac5_1 = PA[(fP + 5) * N + fI + 1];
            const double Aac5_2 = PA[(fP + 5) * N + fI + 2];
            const double Aac5_3 = PA[(fP + 5) * N + fI + 3];
            jab0 += o0_0 * ptk0 + o0_1 * ptk1 + o0_2 * ptk2 + o0_3 * ptk3;
            jab1 += o1_0 * ptk0 + o1_1 * ptk1 + o1_2 * ptk2 + o1_3 * ptk3;
            jab2 += o2_0 * ptk0 + o2_1 * ptk1 + o2_2 * ptk2 + o2_3 * ptk3;
            jab3 += o3_0 * ptk0 + o3_1 * ptk1 + o3_2 * ptk2 + o3_3 * ptk3;
            jab4 += o4_0 * ptk0 + o4_1 * ptk1 + o4_2 * ptk2 + o4_3 * ptk3;
            jab5 += o5_0 * ptk0 + o5_1 * ptk1 + o5_2 * ptk2 + o5_3 * ptk3;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5));
            atomicAdd(Jacc + (fI + 3) * N + fJ + 0, 2.0 * deg * (o0_3 * ptb0 + o1_3 * ptb1 + o2_3 * ptb2 + o3_3 * ptb3 + o4_3 * ptb4 + o5_3 * ptb5));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o1_0 * Aad1_0 + o2_0 * Aad2_0 + o3_0 * Aad3_0 + o4_0 * Aad4_0 + o5_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o0_1 * Abc0_1 + o0_2 * Abc0_2 + o0_3 * Abc0_3));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o0_1 * Aac0_1 + o0_2 * Aac0_2 + o0_3 * Aac0_3 + o1_0 * Aac1_0 + o1_1 * Aac1_1 + o1_2 * Aac1_2 + o1_3 * Aac1_3 + o2_0 * Aac2_0 + o2_1 * Aac2_1 + o2_2 * Aac2_2 + o2_3 * Aac2_3 + o3_0 * Aac3_0 + o3_1 * Aac3_1 + o3_2 * Aac3_2 + o3_3 * Aac3_3 + o4_0 * Aac4_0 + o4_1 * Aac4_1 + o4_2 * Aac4_2 + o4_3 * Aac4_3 + o5_0 * Aac5_0 + o5_1 * Aac5_1 + o5_2 * Aac5_2 + o5_3 * Aac5_3));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Aad0_0 + o1_1 * Aad1_0 + o2_1 * Aad2_0 + o3_1 * Aad3_0 + o4_1 * Aad4_0 + o5_1 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Aad0_0 + o1_2 * Aad1_0 + o2_2 * Aad2_0 + o3_2 * Aad3_0 + o4_2 * Aad4_0 + o5_2 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fI + 3, deg * (o0_3 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 3, deg * (o0_3 * Aad0_0 + o1_3 * Aad1_0 + o2_3 * Aad2_0 + o3_3 * Aad3_0 + o4_3 * Aad4_0 + o5_3 * Aad5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o1_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o1_0 * Abc0_0 + o1_1 * Abc0_1 + o1_2 * Abc0_2 + o1_3 * Abc0_3));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o1_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o1_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 3, deg * (o1_3 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o2_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o2_0 * Abc0_0 + o2_1 * Abc0_1 + o2_2 * Abc0_2 + o2_3 * Abc0_3));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o2_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o2_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 3, deg * (o2_3 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o3_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o3_0 * Abc0_0 + o3_1 * Abc0_1 + o3_2 * Abc0_2 + o3_3 * Abc0_3));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o3_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o3_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 3, deg * (o3_3 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o4_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o4_1 * Abc0_1 + o4_2 * Abc0_2 + o4_3 * Abc0_3));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o4_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o4_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 3, deg * (o4_3 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o5_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o5_0 * Abc0_0 + o5_1 * Abc0_1 + o5_2 * Abc0_2 + o5_3 * Abc0_3));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o5_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o5_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 3, deg * (o5_3 * Abd0_0));
          }
        } break;
        }
      }
      {
        const double s2 = 2.0 * deg;
        double v[8] = {s2 * jab0, s2 * jab1, s2 * jab2, s2 * jab3, s2 * jab4, s2 * jab5, 0.0, 0.0};
        const double s = sqb::warp_sum_scatter<8>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 6 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 1) * N + bp.fQ + ab % 1, s);
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
