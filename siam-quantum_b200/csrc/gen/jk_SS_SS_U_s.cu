// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"

extern "C" __global__ void __launch_bounds__(128)
jk_SS_SS_U_s(const sqb::JKArgs a, const sqb::WorkItem* __restrict__ items) {
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
      for (int x = threadIdx.x; x < bp.nprim * 6; x += blockDim.x) sbra[x] = a.bra_prims[bp.poff + (long long)x * bp.kstride];
      __syncthreads();
      // threads sharing one quartet: si strides over the bra primitives x sj over the ket primitives
      const int si = it.split & 0xffff, sj = it.split >> 16, isplit = si * sj;
      const int kl = threadIdx.x / isplit, grp = threadIdx.x - kl * isplit;
      const int gj = grp / si, gi = grp - gj * si;
      const unsigned gmask = isplit >= 32 ? 0xffffffffu : ((1u << isplit) - 1u) << ((threadIdx.x & 31) & ~(isplit - 1));
      const int pass = qp_;                   // block of bra functions handled by this CTA
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
      unsigned long long nprimq = 0, nflush = 0;
      if (ok) {
        const double* __restrict__ kprim = a.ket_prims + kp.poff;
        const int kS = kp.kstride;                   // distance between the fields of one ket record
        const int nbp = bp.nprim, nkp = kp.nprim;
        nflush = pass == 0 && gj < nkp ? (unsigned long long)((nkp - gj + sj - 1) / sj) : 0ull;
        const double* __restrict__ PA = a.PA + mr.moff;
        const double* __restrict__ PB = a.PB + mr.moff;
        const double* __restrict__ PT = a.PT + mr.moff;
        switch (pass) {
        case 0: {  // bra functions [0]
          double o0_0 = 0;
          for (int j = gj; j < nkp; j += sj) {
            const double* __restrict__ kj = kprim + (long long)j * 6 * kS;
            const double q = kj[0], Qx = kj[kS], Qy = kj[2 * kS], Qz = kj[3 * kS], kq = kj[4 * kS];
            double g0_0 = 0;
            for (int i = gi; i < nbp; i += si) {
              const double* __restrict__ bi = sbra + i * 6;
              const double p = bi[0];
              const double pq = p + q;
              const double rs = rsqrt(pq);
              if (TWO_PI_2_5 * bi[4] * kq * rs < PRIM_CUTOFF) continue;
              ++nprimq;
              const double alpha = p * q * (rs * rs);
              const double X = bi[1] - Qx, Y = bi[2] - Qy, Z = bi[3] - Qz;
              const double T = alpha * fma(X, X, fma(Y, Y, Z * Z));
              double F[1];
              sqb::boys<0>(T, a.boys_tab, F);
              const double s0 = TWO_PI_2_5 * rs;
              const double m2a = -2.0 * alpha;
              double w = s0;
              const double b0 = w * F[0];
              const double eb0_0 = bi[5];
              g0_0 = fma(eb0_0, b0, g0_0);
            }
            { const double ek = kj[5 * kS];
              o0_0 = fma(ek, g0_0, o0_0);
            }
          }
          {  // digest
            const int fP = bp.fP, fQ = bp.fQ, fI = kp.fP, fJ = kp.fQ;
            const double ptk0 = PT[(fI + 0) * N + fJ + 0];
            const double ptb0 = PT[(fP + 0) * N + fQ + 0];
            const double Abd0_0 = PA[(fQ + 0) * N + fJ + 0];
            const double Aad0_0 = PA[(fP + 0) * N + fJ + 0];
            const double Abc0_0 = PA[(fQ + 0) * N + fI + 0];
            const double Aac0_0 = PA[(fP + 0) * N + fI + 0];
            const double Bbd0_0 = PB[(fQ + 0) * N + fJ + 0];
            const double Bad0_0 = PB[(fP + 0) * N + fJ + 0];
            const double Bbc0_0 = PB[(fQ + 0) * N + fI + 0];
            const double Bac0_0 = PB[(fP + 0) * N + fI + 0];
            jab0 += o0_0 * ptk0;
            sqb::group_add(Jacc + (fI + 0) * N + fJ + 0, 2.0 * deg * (o0_0 * ptb0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Abd0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Aad0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Abc0_0), isplit, gmask, grp == 0);
            sqb::group_add(KAacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Aac0_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 0) * N + fI + 0, deg * (o0_0 * Bbd0_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 0) * N + fI + 0, deg * (o0_0 * Bad0_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fP + 0) * N + fJ + 0, deg * (o0_0 * Bbc0_0), isplit, gmask, grp == 0);
            sqb::group_add(KBacc + (fQ + 0) * N + fJ + 0, deg * (o0_0 * Bac0_0), isplit, gmask, grp == 0);
          }
        } break;
        }
      }
      switch (pass) {
      case 0:
      {
        const double s2 = 2.0 * deg;
        double v[1] = {s2 * jab0};
        const double s = sqb::warp_sum_scatter<1>(v);
        const int l = threadIdx.x & 31, ab = l + 0;
        if (l < 1 && s != 0.0) atomicAdd(Jacc + (bp.fP + ab / 1) * N + bp.fQ + ab % 1, s);
      }
      break;
      }
      sqb::count_add(a.counters + 0, (ok && grp == 0 && pass == 0) ? 1ull : 0ull);
      sqb::count_add(a.counters + 1, nprimq);
      sqb::count_add(a.counters + 2, nflush);
      sqb::count_add(a.counters + 3, (ok && pass == 0) ? 1ull : 0ull);
    }
  }
}
