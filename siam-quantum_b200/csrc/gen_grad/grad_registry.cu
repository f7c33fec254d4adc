// generated by gen_grad_kernels.py -- do not edit
#include "../grad_common.cuh"

extern "C" __global__ void grad_SS_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PS_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PS_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LS_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LS_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LS_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DS_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DS_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DS_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DS_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_PP(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_PP(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_PL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_PP(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_PL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_LL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_PP(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_PL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_LL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_DP(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DL_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DL_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DL_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DL_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_DL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_DL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_DL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_DL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DL_DL(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_SS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_PS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_LS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DS(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PP_DD(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_PL_DD(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_LL_DD(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DP_DD(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DL_DD(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_0(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_1(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_2(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_3(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_4(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_5(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_6(const sqb::GradArgs, const sqb::WorkItem*);
extern "C" __global__ void grad_DD_DD_7(const sqb::GradArgs, const sqb::WorkItem*);

namespace sqb {
const GradKernel kGradKernels[62] = {
  {0, 0, (const void*)grad_SS_SS, 1, 15, 90},
  {3, 0, (const void*)grad_PS_SS, 1, 26, 156},
  {3, 3, (const void*)grad_PS_PS, 3, 26, 192},
  {1, 0, (const void*)grad_LS_SS, 1, 27, 174},
  {1, 3, (const void*)grad_LS_PS, 3, 27, 210},
  {1, 1, (const void*)grad_LS_LS, 4, 27, 210},
  {6, 0, (const void*)grad_DS_SS, 1, 44, 318},
  {6, 3, (const void*)grad_DS_PS, 3, 44, 369},
  {6, 1, (const void*)grad_DS_LS, 4, 44, 369},
  {6, 6, (const void*)grad_DS_DS, 6, 44, 438},
  {5, 0, (const void*)grad_PP_SS, 1, 52, 408},
  {5, 3, (const void*)grad_PP_PS, 3, 52, 459},
  {5, 1, (const void*)grad_PP_LS, 4, 52, 459},
  {5, 6, (const void*)grad_PP_DS, 6, 52, 528},
  {5, 5, (const void*)grad_PP_PP, 9, 52, 528},
  {4, 0, (const void*)grad_PL_SS, 1, 53, 498},
  {4, 3, (const void*)grad_PL_PS, 3, 53, 549},
  {4, 1, (const void*)grad_PL_LS, 4, 53, 549},
  {4, 6, (const void*)grad_PL_DS, 6, 53, 618},
  {4, 5, (const void*)grad_PL_PP, 9, 53, 618},
  {4, 4, (const void*)grad_PL_PL, 12, 53, 618},
  {2, 0, (const void*)grad_LL_SS, 1, 54, 618},
  {2, 3, (const void*)grad_LL_PS, 3, 54, 669},
  {2, 1, (const void*)grad_LL_LS, 4, 54, 669},
  {2, 6, (const void*)grad_LL_DS, 6, 54, 738},
  {2, 5, (const void*)grad_LL_PP, 9, 54, 738},
  {2, 4, (const void*)grad_LL_PL, 12, 54, 738},
  {2, 2, (const void*)grad_LL_LL, 16, 54, 738},
  {8, 0, (const void*)grad_DP_SS, 1, 91, 1089},
  {8, 3, (const void*)grad_DP_PS, 3, 91, 1158},
  {8, 1, (const void*)grad_DP_LS, 4, 91, 1158},
  {8, 6, (const void*)grad_DP_DS, 6, 91, 1248},
  {8, 5, (const void*)grad_DP_PP, 9, 91, 1248},
  {8, 4, (const void*)grad_DP_PL, 12, 91, 1248},
  {8, 2, (const void*)grad_DP_LL, 16, 91, 1248},
  {8, 8, (const void*)grad_DP_DP, 18, 91, 1362},
  {7, 0, (const void*)grad_DL_SS, 1, 92, 1389},
  {7, 3, (const void*)grad_DL_PS, 3, 92, 1458},
  {7, 1, (const void*)grad_DL_LS, 4, 92, 1458},
  {7, 6, (const void*)grad_DL_DS, 6, 92, 1548},
  {5, 7, (const void*)grad_PP_DL, 24, 52, 618},
  {4, 7, (const void*)grad_PL_DL, 24, 53, 708},
  {2, 7, (const void*)grad_LL_DL, 24, 54, 828},
  {8, 7, (const void*)grad_DP_DL, 24, 91, 1362},
  {7, 7, (const void*)grad_DL_DL, 24, 92, 1662},
  {9, 0, (const void*)grad_DD_SS, 1, 157, 3138},
  {9, 3, (const void*)grad_DD_PS, 3, 157, 3228},
  {9, 1, (const void*)grad_DD_LS, 4, 157, 3228},
  {9, 6, (const void*)grad_DD_DS, 6, 157, 3342},
  {5, 9, (const void*)grad_PP_DD, 36, 52, 732},
  {4, 9, (const void*)grad_PL_DD, 36, 53, 822},
  {2, 9, (const void*)grad_LL_DD, 36, 54, 942},
  {8, 9, (const void*)grad_DP_DD, 36, 91, 1503},
  {7, 9, (const void*)grad_DL_DD, 36, 92, 1803},
  {9, 9, (const void*)grad_DD_DD_0, 3, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_1, 6, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_2, 6, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_3, 3, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_4, 6, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_5, 3, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_6, 3, 157, 3654},
  {9, 9, (const void*)grad_DD_DD_7, 6, 157, 3654},
};
const int kNumGradKernels = 62;
}  // namespace sqb
