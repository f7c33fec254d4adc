// generated by gen_jk_kernels.py -- do not edit
#include "../jk_common.cuh"
#include "../jk_registry.h"

extern "C" __global__ void jk_SS_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_SS_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_SS_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_SS_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_SS_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_SS_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PS_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LS_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DS_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PP_PP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_PL_PL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_PL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_LL_LL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_PL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_LL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DP_DP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_PL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_LL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DL_R_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DL_DL_U_w(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_SS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_SS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_SS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_SS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_SS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_SS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DS_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DS_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DS_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DS_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DS_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DS_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PP_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PP_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PP_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PP_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PL_R_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_PL_U_s(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LL_R_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_LL_U_f32(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DP_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DP_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DL_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DL_U(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DD_R(const sqb::JKArgs, const sqb::WorkItem*);
extern "C" __global__ void jk_DD_DD_U(const sqb::JKArgs, const sqb::WorkItem*);

namespace sqb {
const char* const kPairClassNames[10] = {"SS", "LS", "LL", "PS", "PL", "PP", "DS", "DL", "DP", "DD"};
const ClassKernel kClassKernels[55] = {
  {0, 0, 1, 1, 1, 1, 0, 1, (const void*)jk_SS_SS_R, (const void*)jk_SS_SS_U, 48, 2, 18,
   1, (const void*)jk_SS_SS_R_f32, (const void*)jk_SS_SS_U_f32, 48, 2, 18,
   48,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_SS_SS_R_s, (const void*)jk_SS_SS_U_s, 48, 2, 18,
   2, 1},
  {3, 0, 3, 1, 6, 1, 1, 1, (const void*)jk_PS_SS_R, (const void*)jk_PS_SS_U, 62, 12, 46,
   1, (const void*)jk_PS_SS_R_f32, (const void*)jk_PS_SS_U_f32, 62, 12, 46,
   62,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_PS_SS_R_s, (const void*)jk_PS_SS_U_s, 66, 6, 46,
   2, 1},
  {3, 3, 3, 3, 6, 6, 2, 1, (const void*)jk_PS_PS_R, (const void*)jk_PS_PS_U, 119, 36, 130,
   1, (const void*)jk_PS_PS_R_f32, (const void*)jk_PS_PS_U_f32, 119, 36, 130,
   119,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_PS_PS_R_s, (const void*)jk_PS_PS_U_s, 119, 36, 130,
   2, 1},
  {1, 0, 4, 1, 7, 1, 1, 1, (const void*)jk_LS_SS_R, (const void*)jk_LS_SS_U, 62, 14, 60,
   1, (const void*)jk_LS_SS_R_f32, (const void*)jk_LS_SS_U_f32, 62, 14, 60,
   62,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_LS_SS_R_s, (const void*)jk_LS_SS_U_s, 68, 8, 60,
   2, 1},
  {1, 3, 4, 3, 7, 6, 2, 1, (const void*)jk_LS_PS_R, (const void*)jk_LS_PS_U, 119, 42, 170,
   1, (const void*)jk_LS_PS_R_f32, (const void*)jk_LS_PS_U_f32, 119, 42, 170,
   119,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_LS_PS_R_s, (const void*)jk_LS_PS_U_s, 127, 48, 170,
   2, 1},
  {1, 1, 4, 4, 7, 7, 2, 1, (const void*)jk_LS_LS_R, (const void*)jk_LS_LS_U, 127, 56, 225,
   1, (const void*)jk_LS_LS_R_f32, (const void*)jk_LS_LS_U_f32, 127, 56, 225,
   127,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_LS_LS_R_s, (const void*)jk_LS_LS_U_s, 127, 56, 225,
   2, 1},
  {6, 0, 6, 1, 21, 1, 2, 1, (const void*)jk_DS_SS_R, (const void*)jk_DS_SS_U, 91, 42, 88,
   1, (const void*)jk_DS_SS_R_f32, (const void*)jk_DS_SS_U_f32, 91, 42, 88,
   91,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_DS_SS_R_s, (const void*)jk_DS_SS_U_s, 113, 12, 88,
   2, 1},
  {6, 3, 6, 3, 21, 6, 3, 1, (const void*)jk_DS_PS_R, (const void*)jk_DS_PS_U, 227, 126, 250,
   1, (const void*)jk_DS_PS_R_f32, (const void*)jk_DS_PS_U_f32, 227, 126, 250,
   227,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_DS_PS_R_s, (const void*)jk_DS_PS_U_s, 275, 72, 250,
   2, 0},
  {6, 1, 6, 4, 21, 7, 3, 1, (const void*)jk_DS_LS_R, (const void*)jk_DS_LS_U, 247, 168, 331,
   1, (const void*)jk_DS_LS_R_f32, (const void*)jk_DS_LS_U_f32, 247, 168, 331,
   247,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_DS_LS_R_s, (const void*)jk_DS_LS_U_s, 275, 84, 331,
   2, 0},
  {6, 6, 6, 6, 21, 21, 4, 2, (const void*)jk_DS_DS_R, (const void*)jk_DS_DS_U, 737, 252, 500,
   1, (const void*)jk_DS_DS_R_f32, (const void*)jk_DS_DS_U_f32, 594, 252, 493,
   594,
   1, (const void*)jk_DS_DS_R_w, (const void*)jk_DS_DS_U_w, 594, 252, 493,
   1, (const void*)jk_DS_DS_R_s, (const void*)jk_DS_DS_U_s, 594, 252, 493,
   0, 0},
  {5, 0, 9, 1, 33, 1, 2, 1, (const void*)jk_PP_SS_R, (const void*)jk_PP_SS_U, 91, 66, 122,
   1, (const void*)jk_PP_SS_R_f32, (const void*)jk_PP_SS_U_f32, 91, 66, 122,
   91,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_PP_SS_R_s, (const void*)jk_PP_SS_U_s, 137, 18, 122,
   2, 1},
  {5, 3, 9, 3, 33, 6, 3, 1, (const void*)jk_PP_PS_R, (const void*)jk_PP_PS_U, 227, 198, 354,
   1, (const void*)jk_PP_PS_R_f32, (const void*)jk_PP_PS_U_f32, 227, 198, 354,
   227,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_PP_PS_R_s, (const void*)jk_PP_PS_U_s, 371, 108, 354,
   2, 0},
  {5, 1, 9, 4, 33, 7, 3, 2, (const void*)jk_PP_LS_R, (const void*)jk_PP_LS_U, 335, 264, 476,
   1, (const void*)jk_PP_LS_R_f32, (const void*)jk_PP_LS_U_f32, 247, 264, 470,
   247,
   1, (const void*)jk_PP_LS_R_w, (const void*)jk_PP_LS_U_w, 247, 264, 470,
   1, (const void*)jk_PP_LS_R_s, (const void*)jk_PP_LS_U_s, 371, 126, 470,
   2, 0},
  {5, 6, 9, 6, 33, 21, 4, 2, (const void*)jk_PP_DS_R, (const void*)jk_PP_DS_U, 753, 396, 708,
   1, (const void*)jk_PP_DS_R_f32, (const void*)jk_PP_DS_U_f32, 594, 396, 702,
   594,
   1, (const void*)jk_PP_DS_R_w, (const void*)jk_PP_DS_U_w, 594, 396, 702,
   2, (const void*)jk_PP_DS_R_s, (const void*)jk_PP_DS_U_s, 945, 378, 728,
   1, 0},
  {5, 5, 9, 9, 33, 33, 4, 3, (const void*)jk_PP_PP_R, (const void*)jk_PP_PP_U, 1120, 594, 1062,
   2, (const void*)jk_PP_PP_R_f32, (const void*)jk_PP_PP_U_f32, 977, 594, 1044,
   834,
   2, (const void*)jk_PP_PP_R_w, (const void*)jk_PP_PP_U_w, 977, 594, 1044,
   2, (const void*)jk_PP_PP_R_s, (const void*)jk_PP_PP_U_s, 977, 594, 1062,
   1, 0},
  {4, 0, 12, 1, 39, 1, 2, 1, (const void*)jk_PL_SS_R, (const void*)jk_PL_SS_U, 91, 78, 160,
   1, (const void*)jk_PL_SS_R_f32, (const void*)jk_PL_SS_U_f32, 91, 78, 160,
   91,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_PL_SS_R_s, (const void*)jk_PL_SS_U_s, 149, 24, 160,
   2, 1},
  {4, 3, 12, 3, 39, 6, 3, 2, (const void*)jk_PL_PS_R, (const void*)jk_PL_PS_U, 315, 234, 473,
   1, (const void*)jk_PL_PS_R_f32, (const void*)jk_PL_PS_U_f32, 227, 234, 466,
   227,
   1, (const void*)jk_PL_PS_R_w, (const void*)jk_PL_PS_U_w, 227, 234, 466,
   1, (const void*)jk_PL_PS_R_s, (const void*)jk_PL_PS_U_s, 419, 144, 466,
   2, 0},
  {4, 1, 12, 4, 39, 7, 3, 2, (const void*)jk_PL_LS_R, (const void*)jk_PL_LS_U, 339, 312, 626,
   1, (const void*)jk_PL_LS_R_f32, (const void*)jk_PL_LS_U_f32, 247, 312, 619,
   247,
   1, (const void*)jk_PL_LS_R_w, (const void*)jk_PL_LS_U_w, 247, 312, 619,
   1, (const void*)jk_PL_LS_R_s, (const void*)jk_PL_LS_U_s, 419, 168, 619,
   2, 0},
  {4, 6, 12, 6, 39, 21, 4, 3, (const void*)jk_PL_DS_R, (const void*)jk_PL_DS_U, 878, 468, 939,
   2, (const void*)jk_PL_DS_R_f32, (const void*)jk_PL_DS_U_f32, 721, 468, 932,
   594,
   2, (const void*)jk_PL_DS_R_w, (const void*)jk_PL_DS_U_w, 721, 468, 932,
   2, (const void*)jk_PL_DS_R_s, (const void*)jk_PL_DS_U_s, 1097, 504, 965,
   1, 0},
  {4, 5, 12, 9, 39, 33, 4, 5, (const void*)jk_PL_PP_R, (const void*)jk_PL_PP_U, 1365, 702, 1419,
   2, (const void*)jk_PL_PP_R_f32, (const void*)jk_PL_PP_U_f32, 976, 702, 1384,
   834,
   2, (const void*)jk_PL_PP_R_w, (const void*)jk_PL_PP_U_w, 976, 702, 1384,
   2, (const void*)jk_PL_PP_R_s, (const void*)jk_PL_PP_U_s, 1101, 792, 1404,
   1, 0},
  {4, 4, 12, 12, 39, 39, 4, 6, (const void*)jk_PL_PL_R, (const void*)jk_PL_PL_U, 1618, 936, 1878,
   3, (const void*)jk_PL_PL_R_f32, (const void*)jk_PL_PL_U_f32, 1240, 936, 1857,
   954,
   3, (const void*)jk_PL_PL_R_w, (const void*)jk_PL_PL_U_w, 1240, 936, 1857,
   3, (const void*)jk_PL_PL_R_s, (const void*)jk_PL_PL_U_s, 1238, 936, 1905,
   1, 0},
  {2, 0, 16, 1, 46, 1, 2, 1, (const void*)jk_LL_SS_R, (const void*)jk_LL_SS_U, 91, 92, 210,
   1, (const void*)jk_LL_SS_R_f32, (const void*)jk_LL_SS_U_f32, 91, 92, 210,
   91,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_LL_SS_R_s, (const void*)jk_LL_SS_U_s, 163, 32, 210,
   2, 1},
  {2, 3, 16, 3, 46, 6, 3, 2, (const void*)jk_LL_PS_R, (const void*)jk_LL_PS_U, 315, 276, 622,
   1, (const void*)jk_LL_PS_R_f32, (const void*)jk_LL_PS_U_f32, 227, 276, 614,
   227,
   1, (const void*)jk_LL_PS_R_w, (const void*)jk_LL_PS_U_w, 227, 276, 614,
   1, (const void*)jk_LL_PS_R_s, (const void*)jk_LL_PS_U_s, 475, 192, 614,
   2, 0},
  {2, 1, 16, 4, 46, 7, 3, 2, (const void*)jk_LL_LS_R, (const void*)jk_LL_LS_U, 339, 368, 824,
   1, (const void*)jk_LL_LS_R_f32, (const void*)jk_LL_LS_U_f32, 247, 368, 816,
   247,
   1, (const void*)jk_LL_LS_R_w, (const void*)jk_LL_LS_U_w, 247, 368, 816,
   1, (const void*)jk_LL_LS_R_s, (const void*)jk_LL_LS_U_s, 475, 224, 816,
   2, 0},
  {2, 6, 16, 6, 46, 21, 4, 3, (const void*)jk_LL_DS_R, (const void*)jk_LL_DS_U, 878, 552, 1236,
   2, (const void*)jk_LL_DS_R_f32, (const void*)jk_LL_DS_U_f32, 737, 552, 1228,
   594,
   2, (const void*)jk_LL_DS_R_w, (const void*)jk_LL_DS_U_w, 737, 552, 1228,
   2, (const void*)jk_LL_DS_R_s, (const void*)jk_LL_DS_U_s, 1247, 672, 1260,
   1, 0},
  {2, 5, 16, 9, 46, 33, 4, 5, (const void*)jk_LL_PP_R, (const void*)jk_LL_PP_U, 1365, 828, 1866,
   3, (const void*)jk_LL_PP_R_f32, (const void*)jk_LL_PP_U_f32, 1120, 828, 1842,
   834,
   3, (const void*)jk_LL_PP_R_w, (const void*)jk_LL_PP_U_w, 1120, 828, 1842,
   3, (const void*)jk_LL_PP_R_s, (const void*)jk_LL_PP_U_s, 1377, 1056, 1884,
   1, 0},
  {2, 4, 16, 12, 46, 39, 4, 6, (const void*)jk_LL_PL_R, (const void*)jk_LL_PL_U, 1618, 1104, 2472,
   3, (const void*)jk_LL_PL_R_f32, (const void*)jk_LL_PL_U_f32, 1240, 1104, 2448,
   954,
   3, (const void*)jk_LL_PL_R_w, (const void*)jk_LL_PL_U_w, 1240, 1104, 2448,
   4, (const void*)jk_LL_PL_R_s, (const void*)jk_LL_PL_U_s, 1459, 1248, 2540,
   1, 0},
  {2, 2, 16, 16, 46, 46, 4, 8, (const void*)jk_LL_LL_R, (const void*)jk_LL_LL_U, 1957, 1472, 3296,
   4, (const void*)jk_LL_LL_R_f32, (const void*)jk_LL_LL_U_f32, 1513, 1472, 3232,
   1094,
   4, (const void*)jk_LL_LL_R_w, (const void*)jk_LL_LL_U_w, 1513, 1472, 3232,
   4, (const void*)jk_LL_LL_R_s, (const void*)jk_LL_LL_U_s, 1487, 1472, 3360,
   1, 0},
  {8, 0, 18, 1, 108, 1, 3, 1, (const void*)jk_DP_SS_R, (const void*)jk_DP_SS_U, 147, 216, 236,
   1, (const void*)jk_DP_SS_R_f32, (const void*)jk_DP_SS_U_f32, 147, 216, 236,
   147,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_DP_SS_R_s, (const void*)jk_DP_SS_U_s, 323, 36, 236,
   0, 0},
  {8, 3, 18, 3, 108, 6, 4, 3, (const void*)jk_DP_PS_R, (const void*)jk_DP_PS_U, 700, 648, 708,
   1, (const void*)jk_DP_PS_R_f32, (const void*)jk_DP_PS_U_f32, 414, 648, 690,
   414,
   1, (const void*)jk_DP_PS_R_w, (const void*)jk_DP_PS_U_w, 414, 648, 690,
   1, (const void*)jk_DP_PS_R_s, (const void*)jk_DP_PS_U_s, 1038, 216, 690,
   1, 0},
  {8, 1, 18, 4, 108, 7, 4, 4, (const void*)jk_DP_LS_R, (const void*)jk_DP_LS_U, 847, 864, 944,
   2, (const void*)jk_DP_LS_R_f32, (const void*)jk_DP_LS_U_f32, 597, 864, 926,
   454,
   2, (const void*)jk_DP_LS_R_w, (const void*)jk_DP_LS_U_w, 597, 864, 926,
   2, (const void*)jk_DP_LS_R_s, (const void*)jk_DP_LS_U_s, 1153, 252, 940,
   1, 0},
  {8, 6, 18, 6, 108, 21, 5, 6, (const void*)jk_DP_DS_R, (const void*)jk_DP_DS_U, 2156, 1296, 1416,
   2, (const void*)jk_DP_DS_R_f32, (const void*)jk_DP_DS_U_f32, 1396, 1296, 1380,
   1127,
   2, (const void*)jk_DP_DS_R_w, (const void*)jk_DP_DS_U_w, 1396, 1296, 1380,
   3, (const void*)jk_DP_DS_R_s, (const void*)jk_DP_DS_U_s, 2899, 756, 1444,
   1, 0},
  {8, 5, 18, 9, 108, 33, 5, 9, (const void*)jk_DP_PP_R, (const void*)jk_DP_PP_U, 3313, 1944, 2124,
   3, (const void*)jk_DP_PP_R_f32, (const void*)jk_DP_PP_U_f32, 2089, 1944, 2070,
   1607,
   3, (const void*)jk_DP_PP_R_w, (const void*)jk_DP_PP_U_w, 2089, 1944, 2070,
   3, (const void*)jk_DP_PP_R_s, (const void*)jk_DP_PP_U_s, 2936, 1188, 2088,
   1, 0},
  {8, 4, 18, 12, 108, 39, 5, 12, (const void*)jk_DP_PL_R, (const void*)jk_DP_PL_U, 4013, 2592, 2832,
   4, (const void*)jk_DP_PL_R_f32, (const void*)jk_DP_PL_U_f32, 2503, 2592, 2760,
   1847,
   4, (const void*)jk_DP_PL_R_w, (const void*)jk_DP_PL_U_w, 2503, 2592, 2760,
   4, (const void*)jk_DP_PL_R_s, (const void*)jk_DP_PL_U_s, 3154, 1404, 2828,
   1, 0},
  {8, 2, 18, 16, 108, 46, 5, 16, (const void*)jk_DP_LL_R, (const void*)jk_DP_LL_U, 4860, 3456, 3776,
   6, (const void*)jk_DP_LL_R_f32, (const void*)jk_DP_LL_U_f32, 3205, 3456, 3704,
   2127,
   6, (const void*)jk_DP_LL_R_w, (const void*)jk_DP_LL_U_w, 3205, 3456, 3704,
   5, (const void*)jk_DP_LL_R_s, (const void*)jk_DP_LL_U_s, 3318, 1656, 3800,
   1, 0},
  {8, 8, 18, 18, 108, 108, 6, 18, (const void*)jk_DP_DP_R, (const void*)jk_DP_DP_U, 9981, 3888, 4248,
   6, (const void*)jk_DP_DP_R_f32, (const void*)jk_DP_DP_U_f32, 6529, 3888, 4140,
   4784,
   6, (const void*)jk_DP_DP_R_w, (const void*)jk_DP_DP_U_w, 6529, 3888, 4140,
   6, (const void*)jk_DP_DP_R_s, (const void*)jk_DP_DP_U_s, 6529, 3888, 4320,
   1, 0},
  {7, 0, 24, 1, 129, 1, 3, 1, (const void*)jk_DL_SS_R, (const void*)jk_DL_SS_U, 147, 258, 310,
   1, (const void*)jk_DL_SS_R_f32, (const void*)jk_DL_SS_U_f32, 147, 258, 310,
   147,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_DL_SS_R_s, (const void*)jk_DL_SS_U_s, 365, 48, 310,
   2, 0},
  {7, 3, 24, 3, 129, 6, 4, 3, (const void*)jk_DL_PS_R, (const void*)jk_DL_PS_U, 700, 774, 930,
   2, (const void*)jk_DL_PS_R_f32, (const void*)jk_DL_PS_U_f32, 557, 774, 920,
   414,
   2, (const void*)jk_DL_PS_R_w, (const void*)jk_DL_PS_U_w, 557, 774, 920,
   2, (const void*)jk_DL_PS_R_s, (const void*)jk_DL_PS_U_s, 1337, 288, 936,
   1, 0},
  {7, 1, 24, 4, 129, 7, 4, 4, (const void*)jk_DL_LS_R, (const void*)jk_DL_LS_U, 847, 1032, 1240,
   2, (const void*)jk_DL_LS_R_f32, (const void*)jk_DL_LS_U_f32, 607, 1032, 1220,
   454,
   2, (const void*)jk_DL_LS_R_w, (const void*)jk_DL_LS_U_w, 607, 1032, 1220,
   2, (const void*)jk_DL_LS_R_s, (const void*)jk_DL_LS_U_s, 1349, 336, 1238,
   1, 0},
  {7, 6, 24, 6, 129, 21, 5, 6, (const void*)jk_DL_DS_R, (const void*)jk_DL_DS_U, 2156, 1548, 1860,
   3, (const void*)jk_DL_DS_R_f32, (const void*)jk_DL_DS_U_f32, 1616, 1548, 1830,
   1127,
   3, (const void*)jk_DL_DS_R_w, (const void*)jk_DL_DS_U_w, 1616, 1548, 1830,
   3, (const void*)jk_DL_DS_R_s, (const void*)jk_DL_DS_U_s, 3356, 1008, 1890,
   1, 0},
  {7, 5, 24, 9, 129, 33, 5, 9, (const void*)jk_DL_PP_R, (const void*)jk_DL_PP_U, 3313, 2322, 2790,
   5, (const void*)jk_DL_PP_R_f32, (const void*)jk_DL_PP_U_f32, 2509, 2322, 2760,
   1607,
   5, (const void*)jk_DL_PP_R_w, (const void*)jk_DL_PP_U_w, 2509, 2322, 2760,
   4, (const void*)jk_DL_PP_R_s, (const void*)jk_DL_PP_U_s, 3548, 1584, 2808,
   1, 0},
  {7, 4, 24, 12, 129, 39, 5, 12, (const void*)jk_DL_PL_R, (const void*)jk_DL_PL_U, 4013, 3096, 3720,
   6, (const void*)jk_DL_PL_R_f32, (const void*)jk_DL_PL_U_f32, 2988, 3096, 3660,
   1847,
   6, (const void*)jk_DL_PL_R_w, (const void*)jk_DL_PL_U_w, 2988, 3096, 3660,
   5, (const void*)jk_DL_PL_R_s, (const void*)jk_DL_PL_U_s, 3765, 1872, 3779,
   1, 0},
  {7, 2, 24, 16, 129, 46, 5, 16, (const void*)jk_DL_LL_R, (const void*)jk_DL_LL_U, 4860, 4128, 4960,
   8, (const void*)jk_DL_LL_R_f32, (const void*)jk_DL_LL_U_f32, 3595, 4128, 4880,
   2127,
   8, (const void*)jk_DL_LL_R_w, (const void*)jk_DL_LL_U_w, 3595, 4128, 4880,
   6, (const void*)jk_DL_LL_R_s, (const void*)jk_DL_LL_U_s, 3896, 2208, 5040,
   1, 0},
  {7, 8, 24, 18, 129, 108, 6, 18, (const void*)jk_DL_DP_R, (const void*)jk_DL_DP_U, 9981, 4644, 5580,
   9, (const void*)jk_DL_DP_R_f32, (const void*)jk_DL_DP_U_f32, 7698, 4644, 5490,
   4784,
   9, (const void*)jk_DL_DP_R_w, (const void*)jk_DL_DP_U_w, 7698, 4644, 5490,
   8, (const void*)jk_DL_DP_R_s, (const void*)jk_DL_DP_U_s, 8092, 5184, 5796,
   1, 0},
  {7, 7, 24, 24, 129, 129, 6, 24, (const void*)jk_DL_DL_R, (const void*)jk_DL_DL_U, 12137, 6192, 7440,
   12, (const void*)jk_DL_DL_R_f32, (const void*)jk_DL_DL_U_f32, 9230, 6192, 7320,
   5624,
   12, (const void*)jk_DL_DL_R_w, (const void*)jk_DL_DL_U_w, 9230, 6192, 7320,
   0, nullptr, nullptr, 0, 0, 0,
   1, 0},
  {9, 0, 36, 1, 336, 1, 4, 1, (const void*)jk_DD_SS_R, (const void*)jk_DD_SS_U, 244, 672, 458,
   1, (const void*)jk_DD_SS_R_f32, (const void*)jk_DD_SS_U_f32, 244, 672, 458,
   244,
   0, nullptr, nullptr, 0, 0, 0,
   1, (const void*)jk_DD_SS_R_s, (const void*)jk_DD_SS_U_s, 846, 72, 458,
   0, 0},
  {9, 3, 36, 3, 336, 6, 5, 3, (const void*)jk_DD_PS_R, (const void*)jk_DD_PS_U, 1189, 2016, 1374,
   3, (const void*)jk_DD_PS_R_f32, (const void*)jk_DD_PS_U_f32, 1189, 2016, 1374,
   707,
   0, nullptr, nullptr, 0, 0, 0,
   2, (const void*)jk_DD_PS_R_s, (const void*)jk_DD_PS_U_s, 3244, 432, 1380,
   0, 0},
  {9, 1, 36, 4, 336, 7, 5, 4, (const void*)jk_DD_LS_R, (const void*)jk_DD_LS_U, 1433, 2688, 1832,
   4, (const void*)jk_DD_LS_R_f32, (const void*)jk_DD_LS_U_f32, 1433, 2688, 1832,
   777,
   0, nullptr, nullptr, 0, 0, 0,
   3, (const void*)jk_DD_LS_R_s, (const void*)jk_DD_LS_U_s, 3427, 504, 1872,
   0, 0},
  {9, 6, 36, 6, 336, 21, 6, 6, (const void*)jk_DD_DS_R, (const void*)jk_DD_DS_U, 3679, 4032, 2748,
   6, (const void*)jk_DD_DS_R_f32, (const void*)jk_DD_DS_U_f32, 3679, 4032, 2748,
   1934,
   0, nullptr, nullptr, 0, 0, 0,
   5, (const void*)jk_DD_DS_R_s, (const void*)jk_DD_DS_U_s, 8670, 1512, 2911,
   0, 0},
  {9, 5, 36, 9, 336, 33, 6, 9, (const void*)jk_DD_PP_R, (const void*)jk_DD_PP_U, 5655, 6048, 4122,
   9, (const void*)jk_DD_PP_R_f32, (const void*)jk_DD_PP_U_f32, 5655, 6048, 4122,
   2774,
   0, nullptr, nullptr, 0, 0, 0,
   6, (const void*)jk_DD_PP_R_s, (const void*)jk_DD_PP_U_s, 8929, 2376, 4248,
   0, 0},
  {9, 4, 36, 12, 336, 39, 6, 12, (const void*)jk_DD_PL_R, (const void*)jk_DD_PL_U, 6844, 8064, 5496,
   12, (const void*)jk_DD_PL_R_f32, (const void*)jk_DD_PL_U_f32, 6844, 8064, 5496,
   3194,
   0, nullptr, nullptr, 0, 0, 0,
   8, (const void*)jk_DD_PL_R_s, (const void*)jk_DD_PL_U_s, 9635, 2808, 5712,
   0, 0},
  {9, 2, 36, 16, 336, 46, 6, 16, (const void*)jk_DD_LL_R, (const void*)jk_DD_LL_U, 8277, 10752, 7328,
   16, (const void*)jk_DD_LL_R_f32, (const void*)jk_DD_LL_U_f32, 8277, 10752, 7328,
   3684,
   0, nullptr, nullptr, 0, 0, 0,
   0, nullptr, nullptr, 0, 0, 0,
   0, 0},
  {9, 8, 36, 18, 336, 108, 7, 18, (const void*)jk_DD_DP_R, (const void*)jk_DD_DP_U, 16974, 12096, 8244,
   0, nullptr, nullptr, 0, 0, 0,
   8286,
   0, nullptr, nullptr, 0, 0, 0,
   0, nullptr, nullptr, 0, 0, 0,
   0, 0},
  {9, 7, 36, 24, 336, 129, 7, 24, (const void*)jk_DD_DL_R, (const void*)jk_DD_DL_U, 20653, 16128, 10992,
   0, nullptr, nullptr, 0, 0, 0,
   9756,
   0, nullptr, nullptr, 0, 0, 0,
   0, nullptr, nullptr, 0, 0, 0,
   0, 0},
  {9, 9, 36, 36, 336, 336, 8, 36, (const void*)jk_DD_DD_R, (const void*)jk_DD_DD_U, 49460, 24192, 16488,
   0, nullptr, nullptr, 0, 0, 0,
   24617,
   0, nullptr, nullptr, 0, 0, 0,
   0, nullptr, nullptr, 0, 0, 0,
   0, 0},
};
const int kNumClassKernels = 55;
}  // namespace sqb
