// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_DS_PS_U(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 26; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];
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
        case 0: {  // ket functions [0, 1, 2]
          double o0_0 = 0;
          double o0_1 = 0;
          double o0_2 = 0;
          double o1_0 = 0;
          double o1_1 = 0;
          double o1_2 = 0;
          double o2_0 = 0;
          double o2_1 = 0;
          double o2_2 = 0;
          double o3_0 = 0;
          double o3_1 = 0;
          double o3_2 = 0;
          double o4_0 = 0;
          double o4_1 = 0;
          double o4_2 = 0;
          double o5_0 = 0;
          double o5_1 = 0;
          double o5_2 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 26;
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
              const double ek0_1 = -kj[6 * kS];
              const double ek1_0 = kj[7 * kS];
              const double ek1_1 = -kj[8 * kS];
              const double ek2_0 = kj[9 * kS];
              const double ek2_1 = -kj[10 * kS];
              g0_0 = fma(ek0_0, b0, g0_0);
              g1_0 = fma(ek1_0, b0, g1_0);
              g2_0 = fma(ek2_0, b0, g2_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              g1_1 = fma(ek1_0, r0_0_0_1, g1_1);
              g2_1 = fma(ek2_0, r0_0_0_1, g2_1);
              g2_0 = fma(ek2_1, r0_0_0_1, g2_0);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              g1_2 = fma(ek1_0, r0_0_1_0, g1_2);
              g1_0 = fma(ek1_1, r0_0_1_0, g1_0);
              g2_2 = fma(ek2_0, r0_0_1_0, g2_2);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
              g0_0 = fma(ek0_1, r0_1_0_0, g0_0);
              g1_3 = fma(ek1_0, r0_1_0_0, g1_3);
              g2_3 = fma(ek2_0, r0_1_0_0, g2_3);
              const double r1_0_0_1 = Z * b2;
              const double r0_0_0_2 = fma(Z, r1_0_0_1, b1);
              g0_4 = fma(ek0_0, r0_0_0_2, g0_4);
              g1_4 = fma(ek1_0, r0_0_0_2, g1_4);
              g2_4 = fma(ek2_0, r0_0_0_2, g2_4);
              g2_1 = fma(ek2_1, r0_0_0_2, g2_1);
              const double r0_0_1_1 = Y * r1_0_0_1;
              g0_5 = fma(ek0_0, r0_0_1_1, g0_5);
              g1_5 = fma(ek1_0, r0_0_1_1, g1_5);
              g1_1 = fma(ek1_1, r0_0_1_1, g1_1);
              g2_5 = fma(ek2_0, r0_0_1_1, g2_5);
              g2_2 = fma(ek2_1, r0_0_1_1, g2_2);
              const double r1_0_1_0 = Y * b2;
              const double r0_0_2_0 = fma(Y, r1_0_1_0, b1);
              g0_6 = fma(ek0_0, r0_0_2_0, g0_6);
              g1_6 = fma(ek1_0, r0_0_2_0, g1_6);
              g1_2 = fma(ek1_1, r0_0_2_0, g1_2);
              g2_6 = fma(ek2_0, r0_0_2_0, g2_6);
              const double r0_1_0_1 = X * r1_0_0_1;
              g0_7 = fma(ek0_0, r0_1_0_1, g0_7);
              g0_1 = fma(ek0_1, r0_1_0_1, g0_1);
              g1_7 = fma(ek1_0, r0_1_0_1, g1_7);
              g2_7 = fma(ek2_0, r0_1_0_1, g2_7);
              g2_3 = fma(ek2_1, r0_1_0_1, g2_3);
              const double r0_1_1_0 = X * r1_0_1_0;
              g0_8 = fma(ek0_0, r0_1_1_0, g0_8);
              g0_2 = fma(ek0_1, r0_1_1_0, g0_2);
              g1_8 = fma(ek1_0, r0_1_1_0, g1_8);
              g1_3 = fma(ek1_1, r0_1_1_0, g1_3);
              g2_8 = fma(ek2_0, r0_1_1_0, g2_8);
              const double r1_1_0_0 = X * b2;
              const double r0_2_0_0 = fma(X, r1_1_0_0, b1);
              g0_9 = fma(ek0_0, r0_2_0_0, g0_9);
              g0_3 = fma(ek0_1, r0_2_0_0, g0_3);
              g1_9 = fma(ek1_0, r0_2_0_0, g1_9);
              g2_9 = fma(ek2_0, r0_2_0_0, g2_9);
              const double r2_0_0_1 = Z * b3;
              const double r1_0_0_2 = fma(Z, r2_0_0_1, b2);
              const double r0_0_0_3 = fma(Z, r1_0_0_2, 2.0 * r1_0_0_1);
              g2_4 = fma(ek2_1, r0_0_0_3, g2_4);
              const double r0_0_1_2 = Y * r1_0_0_2;
              g1_4 = fma(ek1_1, r0_0_1_2, g1_4);
              g2_5 = fma(ek2_1, r0_0_1_2, g2_5);
              const double r1_0_1_1 = Y * r2_0_0_1;
              const double r0_0_2_1 = fma(Y, r1_0_1_1, r1_0_0_1);
              g1_5 = fma(ek1_1, r0_0_2_1, g1_5);
              g2_6 = fma(ek2_1, r0_0_2_1, g2_6);
              const double r2_0_1_0 = Y * b3;
              const double r1_0_2_0 = fma(Y, r2_0_1_0, b2);
              const double r0_0_3_0 = fma(Y, r1_0_2_0, 2.0 * r1_0_1_0);
              g1_6 = fma(ek1_1, r0_0_3_0, g1_6);
              const double r0_1_0_2 = X * r1_0_0_2;
              g0_4 = fma(ek0_1, r0_1_0_2, g0_4);
              g2_7 = fma(ek2_1, r0_1_0_2, g2_7);
              const double r0_1_1_1 = X * r1_0_1_1;
              g0_5 = fma(ek0_1, r0_1_1_1, g0_5);
              g1_7 = fma(ek1_1, r0_1_1_1, g1_7);
              g2_8 = fma(ek2_1, r0_1_1_1, g2_8);
              const double r0_1_2_0 = X * r1_0_2_0;
              g0_6 = fma(ek0_1, r0_1_2_0, g0_6);
              g1_8 = fma(ek1_1, r0_1_2_0, g1_8);
              const double r1_1_0_1 = X * r2_0_0_1;
              const double r0_2_0_1 = fma(X, r1_1_0_1, r1_0_0_1);
              g0_7 = fma(ek0_1, r0_2_0_1, g0_7);
              g2_9 = fma(ek2_1, r0_2_0_1, g2_9);
              const double r1_1_1_0 = X * r2_0_1_0;
              const double r0_2_1_0 = fma(X, r1_1_1_0, r1_0_1_0);
              g0_8 = fma(ek0_1, r0_2_1_0, g0_8);
              g1_9 = fma(ek1_1, r0_2_1_0, g1_9);
              const double r2_1_0_0 = X * b3;
              const double r1_2_0_0 = fma(X, r2_1_0_0, b2);
              const double r0_3_0_0 = fma(X, r1_2_0_0, 2.0 * r1_1_0_0);
              g0_9 = fma(ek0_1, r0_3_0_0, g0_9);
            }
            { const double eb = bi[5];
              o0_0 = fma(eb, g0_0, o0_0);
              o0_1 = fma(eb, g1_0, o0_1);
              o0_2 = fma(eb, g2_0, o0_2);
            }
            { const double eb = bi[6];
              o0_0 = fma(eb, g0_3, o0_0);
              o0_1 = fma(eb, g1_3, o0_1);
              o0_2 = fma(eb, g2_3, o0_2);
            }
            { const double eb = bi[7];
              o0_0 = fma(eb, g0_9, o0_0);
              o0_1 = fma(eb, g1_9, o0_1);
              o0_2 = fma(eb, g2_9, o0_2);
            }
            { const double eb = bi[8];
              o1_0 = fma(eb, g0_0, o1_0);
              o1_1 = fma(eb, g1_0, o1_1);
              o1_2 = fma(eb, g2_0, o1_2);
            }
            { const double eb = bi[9];
              o1_0 = fma(eb, g0_2, o1_0);
              o1_1 = fma(eb, g1_2, o1_1);
              o1_2 = fma(eb, g2_2, o1_2);
            }
            { const double eb = bi[10];
              o1_0 = fma(eb, g0_6, o1_0);
              o1_1 = fma(eb, g1_6, o1_1);
              o1_2 = fma(eb, g2_6, o1_2);
            }
            { const double eb = bi[11];
              o2_0 = fma(eb, g0_0, o2_0);
              o2_1 = fma(eb, g1_0, o2_1);
              o2_2 = fma(eb, g2_0, o2_2);
            }
            { const double eb = bi[12];
              o2_0 = fma(eb, g0_1, o2_0);
              o2_1 = fma(eb, g1_1, o2_1);
              o2_2 = fma(eb, g2_1, o2_2);
            }
            { const double eb = bi[13];
              o2_0 = fma(eb, g0_4, o2_0);
              o2_1 = fma(eb, g1_4, o2_1);
              o2_2 = fma(eb, g2_4, o2_2);
            }
            { const double eb = bi[14];
              o3_0 = fma(eb, g0_0, o3_0);
              o3_1 = fma(eb, g1_0, o3_1);
              o3_2 = fma(eb, g2_0, o3_2);
            }
            { const double eb = bi[15];
              o3_0 = fma(eb, g0_2, o3_0);
              o3_1 = fma(eb, g1_2, o3_1);
              o3_2 = fma(eb, g2_2, o3_2);
            }
            { const double eb = bi[16];
              o3_0 = fma(eb, g0_3, o3_0);
              o3_1 = fma(eb, g1_3, o3_1);
              o3_2 = fma(eb, g2_3, o3_2);
            }
            { const double eb = bi[17];
              o3_0 = fma(eb, g0_8, o3_0);
              o3_1 = fma(eb, g1_8, o3_1);
              o3_2 = fma(eb, g2_8, o3_2);
            }
            { const double eb = bi[18];
              o4_0 = fma(eb, g0_0, o4_0);
              o4_1 = fma(eb, g1_0, o4_1);
              o4_2 = fma(eb, g2_0, o4_2);
            }
            { const double eb = bi[19];
              o4_0 = fma(eb, g0_1, o4_0);
              o4_1 = fma(eb, g1_1, o4_1);
              o4_2 = fma(eb, g2_1, o4_2);
            }
            { const double eb = bi[20];
              o4_0 = fma(eb, g0_3, o4_0);
              o4_1 = fma(eb, g1_3, o4_1);
              o4_2 = fma(eb, g2_3, o4_2);
            }
            { const double eb = bi[21];
              o4_0 = fma(eb, g0_7, o4_0);
              o4_1 = fma(eb, g1_7, o4_1);
              o4_2 = fma(eb, g2_7, o4_2);
            }
            { const double eb = bi[22];
              o5_0 = fma(eb, g0_0, o5_0);
              o5_1 = fma(eb, g1_0, o5_1);
              o5_2 = fma(eb, g2_0, o5_2);
            }
            { const double eb = bi[23];
              o5_0 = fma(eb, g0_1, o5_0);
              o5_1 = fma(eb, g1_1, o5_1);
              o5_2 = fma(eb, g2_1, o5_2);
            }
            { const double eb = bi[24];
              o5_0 = fma(eb, g0_2, o5_0);
              o5_1 = fma(eb, g1_2, o5_1);
              o5_2 = fma(eb, g2_2, o5_2);
            }
            { const double eb = bi[25];
              o5_0 = fma(eb, g0_5, o5_0);
              o5_1 = fma(eb, g1_5, o5_1);
              o5_2 = fma(eb, g2_5, o5_2);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0);
            o0_1 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0);
            o0_2 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0);
            o1_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0);
            o1_1 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0);
            o1_2 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0);
            o2_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0);
            o2_1 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0);
            o2_2 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0);
            o3_0 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0);
            o3_1 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0);
            o3_2 = sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0);
            o4_0 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0);
            o4_1 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0);
            o4_2 = sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0);
            o5_0 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0);
            o5_1 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0);
            o5_2 = sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o0_1 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o0_2 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o1_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o1_1 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o1_2 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o2_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o2_1 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o2_2 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o3_0 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o3_1 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o3_2 - sqb::mpole_value(a.mpole, N, fP + 3, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o4_0 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o4_1 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o4_2 - sqb::mpole_value(a.mpole, N, fP + 4, fQ + 0, fI + 2, fJ + 0)));
            e = fmax(e, fabs(o5_0 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o5_1 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 1, fJ + 0)));
            e = fmax(e, fabs(o5_2 - sqb::mpole_value(a.mpole, N, fP + 5, fQ + 0, fI + 2, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptk1 = PT[(fI + 1) * N + fJ + 0];
            const double ptk2 = PT[(fI + 2) * N + fJ + 0];
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
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bad1_0 = PB[(fP + 1) * N + fJ + 0];
            const double Bad2_0 = PB[(fP + 2) * N + fJ + 0];
            const double Bad3_0 = PB[(fP + 3) * N + fJ + 0];
            const double Bad4_0 = PB[(fP + 4) * N + fJ + 0];
            const double Bad5_0 = PB[(fP + 5) * N + fJ + 0];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bbc0_1 = PB[(fQ + 0) * N + fI + 1];
            const double Bbc0_2 = PB[(fQ + 0) * N + fI + 2];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            const double Bac0_1 = PB[(fP + 0) * N + fI + 1];
            const double Bac0_2 = PB[(fP + 0) * N + fI + 2];
            const double Bac1_0 = PB[(fP + 1) * N + fI + 0];
            const double Bac1_1 = PB[(fP + 1) * N + fI + 1];
            const double Bac1_2 = PB[(fP + 1) * N + fI + 2];
            const double Bac2_0 = PB[(fP + 2) * N + fI + 0];
            const double Bac2_1 = PB[(fP + 2) * N + fI + 1];
            const double Bac2_2 = PB[(fP + 2) * N + fI + 2];
            const double Bac3_0 = PB[(fP + 3) * N + fI + 0];
            const double Bac3_1 = PB[(fP + 3) * N + fI + 1];
            const double Bac3_2 = PB[(fP + 3) * N + fI + 2];
            const double Bac4_0 = PB[(fP + 4) * N + fI + 0];
            const double Bac4_1 = PB[(fP + 4) * N + fI + 1];
            const double Bac4_2 = PB[(fP + 4) * N + fI + 2];
            const double Bac5_0 = PB[(fP + 5) * N + fI + 0];
            const double Bac5_1 = PB[(fP + 5) * N + fI + 1];
            const double Bac5_2 = PB[(fP + 5) * N + fI + 2];
            jab0 += o0_0 * ptk0 + o0_1 * ptk1 + o0_2 * ptk2;
            jab1 += o1_0 * ptk0 + o1_1 * ptk1 + o1_2 * ptk2;
            jab2 += o2_0 * ptk0 + o2_1 * ptk1 + o2_2 * ptk2;
            jab3 += o3_0 * ptk0 + o3_1 * ptk1 + o3_2 * ptk2;
            jab4 += o4_0 * ptk0 + o4_1 * ptk1 + o4_2 * ptk2;
            jab5 += o5_0 * ptk0 + o5_1 * ptk1 + o5_2 * ptk2;
            atomicAdd(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2 + o3_0 * ptb3 + o4_0 * ptb4 + o5_0 * ptb5));
            atomicAdd(Jacc + (fI + 1) * N + fJ + 0, 2.0 * deg * (o0_1 * ptb0 + o1_1 * ptb1 + o2_1 * ptb2 + o3_1 * ptb3 + o4_1 * ptb4 + o5_1 * ptb5));
            atomicAdd(Jacc + (fI + 2) * N + fJ + 0, 2.0 * deg * (o0_2 * ptb0 + o1_2 * ptb1 + o2_2 * ptb2 + o3_2 * ptb3 + o4_2 * ptb4 + o5_2 * ptb5));
            atomicAdd(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o1_0 * Aad1_0 + o2_0 * Aad2_0 + o3_0 * Aad3_0 + o4_0 * Aad4_0 + o5_0 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0 + o0_1 * Abc0_1 + o0_2 * Abc0_2));
            atomicAdd(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o0_1 * Aac0_1 + o0_2 * Aac0_2 + o1_0 * Aac1_0 + o1_1 * Aac1_1 + o1_2 * Aac1_2 + o2_0 * Aac2_0 + o2_1 * Aac2_1 + o2_2 * Aac2_2 + o3_0 * Aac3_0 + o3_1 * Aac3_1 + o3_2 * Aac3_2 + o4_0 * Aac4_0 + o4_1 * Aac4_1 + o4_2 * Aac4_2 + o5_0 * Aac5_0 + o5_1 * Aac5_1 + o5_2 * Aac5_2));
            atomicAdd(KAacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Aad0_0 + o1_1 * Aad1_0 + o2_1 * Aad2_0 + o3_1 * Aad3_0 + o4_1 * Aad4_0 + o5_1 * Aad5_0));
            atomicAdd(KAacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Abd0_0));
            atomicAdd(KAacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Aad0_0 + o1_2 * Aad1_0 + o2_2 * Aad2_0 + o3_2 * Aad3_0 + o4_2 * Aad4_0 + o5_2 * Aad5_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 0, deg * (o1_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 1) * N + fJ + 0, deg * (o1_0 * Abc0_0 + o1_1 * Abc0_1 + o1_2 * Abc0_2));
            atomicAdd(KAacc + (fP + 1) * N + fI + 1, deg * (o1_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 1) * N + fI + 2, deg * (o1_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 0, deg * (o2_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fJ + 0, deg * (o2_0 * Abc0_0 + o2_1 * Abc0_1 + o2_2 * Abc0_2));
            atomicAdd(KAacc + (fP + 2) * N + fI + 1, deg * (o2_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 2) * N + fI + 2, deg * (o2_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 0, deg * (o3_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fJ + 0, deg * (o3_0 * Abc0_0 + o3_1 * Abc0_1 + o3_2 * Abc0_2));
            atomicAdd(KAacc + (fP + 3) * N + fI + 1, deg * (o3_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 3) * N + fI + 2, deg * (o3_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 0, deg * (o4_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fJ + 0, deg * (o4_0 * Abc0_0 + o4_1 * Abc0_1 + o4_2 * Abc0_2));
            atomicAdd(KAacc + (fP + 4) * N + fI + 1, deg * (o4_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 4) * N + fI + 2, deg * (o4_2 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 0, deg * (o5_0 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fJ + 0, deg * (o5_0 * Abc0_0 + o5_1 * Abc0_1 + o5_2 * Abc0_2));
            atomicAdd(KAacc + (fP + 5) * N + fI + 1, deg * (o5_1 * Abd0_0));
            atomicAdd(KAacc + (fP + 5) * N + fI + 2, deg * (o5_2 * Abd0_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Bbd0_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Bad0_0 + o1_0 * Bad1_0 + o2_0 * Bad2_0 + o3_0 * Bad3_0 + o4_0 * Bad4_0 + o5_0 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Bbc0_0 + o0_1 * Bbc0_1 + o0_2 * Bbc0_2));
            atomicAdd(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Bac0_0 + o0_1 * Bac0_1 + o0_2 * Bac0_2 + o1_0 * Bac1_0 + o1_1 * Bac1_1 + o1_2 * Bac1_2 + o2_0 * Bac2_0 + o2_1 * Bac2_1 + o2_2 * Bac2_2 + o3_0 * Bac3_0 + o3_1 * Bac3_1 + o3_2 * Bac3_2 + o4_0 * Bac4_0 + o4_1 * Bac4_1 + o4_2 * Bac4_2 + o5_0 * Bac5_0 + o5_1 * Bac5_1 + o5_2 * Bac5_2));
            atomicAdd(KBacc + (fP + 0) * N + fI + 1, deg * (o0_1 * Bbd0_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 1, deg * (o0_1 * Bad0_0 + o1_1 * Bad1_0 + o2_1 * Bad2_0 + o3_1 * Bad3_0 + o4_1 * Bad4_0 + o5_1 * Bad5_0));
            atomicAdd(KBacc + (fP + 0) * N + fI + 2, deg * (o0_2 * Bbd0_0));
            atomicAdd(KBacc + (fQ + 0) * N + fI + 2, deg * (o0_2 * Bad0_0 + o1_2 * Bad1_0 + o2_2 * Bad2_0 + o3_2 * Bad3_0 + o4_2 * Bad4_0 + o5_2 * Bad5_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 0, deg * (o1_0 * Bbd0_0));
            atomicAdd(KBacc + (fP + 1) * N + fJ + 0, deg * (o1_0 * Bbc0_0 + o1_1 * Bbc0_1 + o1_2 * Bbc0_2));
            atomicAdd(KBacc + (fP + 1) * N + fI + 1, deg * (o1_1 * Bbd0_0));
            atomicAdd(KBacc + (fP + 1) * N + fI + 2, deg * (o1_2 * Bbd0_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 0, deg * (o2_0 * Bbd0_0));
            atomicAdd(KBacc + (fP + 2) * N + fJ + 0, deg * (o2_0 * Bbc0_0 + o2_1 * Bbc0_1 + o2_2 * Bbc0_2));
            atomicAdd(KBacc + (fP + 2) * N + fI + 1, deg * (o2_1 * Bbd0_0));
            atomicAdd(KBacc + (fP + 2) * N + fI + 2, deg * (o2_2 * Bbd0_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 0, deg * (o3_0 * Bbd0_0));
            atomicAdd(KBacc + (fP + 3) * N + fJ + 0, deg * (o3_0 * Bbc0_0 + o3_1 * Bbc0_1 + o3_2 * Bbc0_2));
            atomicAdd(KBacc + (fP + 3) * N + fI + 1, deg * (o3_1 * Bbd0_0));
            atomicAdd(KBacc + (fP + 3) * N + fI + 2, deg * (o3_2 * Bbd0_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 0, deg * (o4_0 * Bbd0_0));
            atomicAdd(KBacc + (fP + 4) * N + fJ + 0, deg * (o4_0 * Bbc0_0 + o4_1 * Bbc0_1 + o4_2 * Bbc0_2));
            atomicAdd(KBacc + (fP + 4) * N + fI + 1, deg * (o4_1 * Bbd0_0));
            atomicAdd(KBacc + (fP + 4) * N + fI + 2, deg * (o4_2 * Bbd0_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 0, deg * (o5_0 * Bbd0_0));
            atomicAdd(KBacc + (fP + 5) * N + fJ + 0, deg * (o5_0 * Bbc0_0 + o5_1 * Bbc0_1 + o5_2 * Bbc0_2));
            atomicAdd(KBacc + (fP + 5) * N + fI + 1, deg * (o5_1 * Bbd0_0));
            atomicAdd(KBacc + (fP + 5) * N + fI + 2, deg * (o5_2 * Bbd0_0));
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
