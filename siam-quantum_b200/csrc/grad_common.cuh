// Records of the generated gradient class kernels (gen_grad_kernels.py) and their table.
#pragma once
#include "jk_common.cuh"

namespace sqb {

// One shell pair of a class, in the gradient's order (primitive count, then falling bound).
struct GradPair {
  int P, Q, fP, fQ;        // sorted shell indices; first functions
  int nprim, poff, kstride;// primitive pairs; field f of record j at poff + (j * fields + f) * kstride
  int atP, atQ;            // atoms of the two shells
  int pad_;
  double sch, pm;          // block maxima of the Schwarz matrix and of |PT|
};

struct GradArgs {
  const GradPair* bra_pairs;
  const double* bra_prims;
  const GradPair* ket_pairs;
  const double* ket_prims;
  const double* PT;        // PA + PB, PA - PB
  const double* PS;
  const double* boys_tab;  // row table of boys<M>
  double* grad;            // ncopy copies of the 3 natom components, `stride` doubles apart
  double screen;
  int nbf, same_class, chunk, ncopy, stride;
};

struct GradKernel {
  int bra_cls, ket_cls;
  const void* fn;
  int passes;              // ket function pairs = grid.y
  int nb;                  // doubles of one bra primitive record in shared memory
  int ops;                 // operations of one primitive step of one pass (estimate: split and order)
};

extern const GradKernel kGradKernels[];
extern const int kNumGradKernels;

}  // namespace sqb
