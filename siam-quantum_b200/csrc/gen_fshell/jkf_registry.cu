// generated by gen_fshell_kernels.py -- do not edit
#include "../jk_generic_dev.cuh"

extern "C" __global__ void jkf_FS_0(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FL_0(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FL_1(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FP_0(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FD_0(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FD_1(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FF_0(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FF_1(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FF_2(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FF_3(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);
extern "C" __global__ void jkf_FF_4(const sqb::FArgs, const sqb::FRun*, const long long*, int, long long, long long);

namespace sqb {
const FKernel kFKernels[11] = {
  {0, (const void*)jkf_FS_0},
  {1, (const void*)jkf_FL_0},
  {1, (const void*)jkf_FL_1},
  {2, (const void*)jkf_FP_0},
  {3, (const void*)jkf_FD_0},
  {3, (const void*)jkf_FD_1},
  {4, (const void*)jkf_FF_0},
  {4, (const void*)jkf_FF_1},
  {4, (const void*)jkf_FF_2},
  {4, (const void*)jkf_FF_3},
  {4, (const void*)jkf_FF_4},
};
const int kNumFKernels = 11;
}  // namespace sqb
