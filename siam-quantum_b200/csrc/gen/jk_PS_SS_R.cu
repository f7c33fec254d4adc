// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_PS_SS_R(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 11; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];
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
      unsigned long long nprimq = 0, nflush = 0;
      if (ok) {
        const double* __restrict__ kprim = a.ket_prims + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = mpq ? 0 : bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gi < nbp ? (unsigned long long)((nbp - gi + si - 1) / si) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // ket functions [0]
          double o0_0 = 0;
          double o1_0 = 0;
          double o2_0 = 0;
          for (int i = gi; i < nbp; i += si) {
            const double* __restrict__ bi = sbra + i * 11;
            const double p = bi[0], Px = bi[1], Py = bi[2], Pz = bi[3], kpb = bi[4];
            double g0_0 = 0;
            double g0_1 = 0;
            double g0_2 = 0;
            double g0_3 = 0;
            for (int j = gj; j < nkp; j += sj) {
              const double* __restrict__ kj = kprim + (long long)j * 6 * kS;
              const double q = kj[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * kpb * kj[4 * kS] * rs < PRIM_CUTOFF) continue;
              ++nprimq;
              const double alpha = p * q * (rs * rs);
              const double X = Px - kj[kS], Y = Py - kj[2 * kS], Z = Pz - kj[3 * kS];
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[2];
              sqb::boys<1>(T, a.boys_tab, F);
              const double s0 = TWO_PI_2_5 * rs;
              const double m2a = -2.0 * alpha;
              double w = s0;
              const double b0 = w * F[0];
              w *= m2a;
              const double b1 = w * F[1];
              const double ek0_0 = kj[5 * kS];
              g0_0 = fma(ek0_0, b0, g0_0);
              const double r0_0_0_1 = Z * b1;
              g0_1 = fma(ek0_0, r0_0_0_1, g0_1);
              const double r0_0_1_0 = Y * b1;
              g0_2 = fma(ek0_0, r0_0_1_0, g0_2);
              const double r0_1_0_0 = X * b1;
              g0_3 = fma(ek0_0, r0_1_0_0, g0_3);
            }
            { const double eb = bi[5];
              o0_0 = fma(eb, g0_0, o0_0);
            }
            { const double eb = bi[6];
              o0_0 = fma(eb, g0_3, o0_0);
            }
            { const double eb = bi[7];
              o1_0 = fma(eb, g0_0, o1_0);
            }
            { const double eb = bi[8];
              o1_0 = fma(eb, g0_2, o1_0);
            }
            { const double eb = bi[9];
              o2_0 = fma(eb, g0_0, o2_0);
            }
            { const double eb = bi[10];
              o2_0 = fma(eb, g0_1, o2_0);
            }
          }
          if (mpq) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            o0_0 = sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0);
            o1_0 = sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0);
            o2_0 = sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0);
          } else if (erexp == sqb::ERR_UNKNOWN && a.erbank) {
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            double e = 0.0;
            e = fmax(e, fabs(o0_0 - sqb::mpole_value(a.mpole, N, fP + 0, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o1_0 - sqb::mpole_value(a.mpole, N, fP + 1, fQ + 0, fI + 0, fJ + 0)));
            e = fmax(e, fabs(o2_0 - sqb::mpole_value(a.mpole, N, fP + 2, fQ + 0, fI + 0, fJ + 0)));
            atomicMax(a.erscr + erx, (unsigned long long)__double_as_longlong(e) | (1ull << 63));
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double ptb1 = PT[(fP + 1) * N + fQ + 0];
            const double ptb2 = PT[(fP + 2) * N + fQ + 0];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Aad1_0 = PA[(fP + 1) * N + fJ + 0];
            const double Aad2_0 = PA[(fP + 2) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Aac1_0 = PA[(fP + 1) * N + fI + 0];
            const double Aac2_0 = PA[(fP + 2) * N + fI + 0];
            jab0 += o0_0 * ptk0;
            jab1 += o1_0 * ptk0;
            jab2 += o2_0 * ptk0;
            sqb::group_add(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0 + o1_0 * ptb1 + o2_0 * ptb2), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0 + o1_0 * Aad1_0 + o2_0 * Aad2_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0 + o1_0 * Aac1_0 + o2_0 * Aac2_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 1) * N + fI + 0, deg * (o1_0 * Abd0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 1) * N + fJ + 0, deg * (o1_0 * Abc0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 2) * N + fI + 0, deg * (o2_0 * Abd0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 2) * N + fJ + 0, deg * (o2_0 * Abc0_0), isplit, gmask, grp == 0);
          }
        } break;
        }
      }
      {
        const double s2 = 2.0 * deg;
        double v[4] = {s2 * jab0, s2 * jab1, s2 * jab2, 0.0};
        const double s = sqb::warp_sum_scatter<4>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 3 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 1) * N + bp.fQ + ab % 1, s);
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
