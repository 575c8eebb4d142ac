// Plain FP64 form: small CTAs of the fused cell step, and the factored step
// (instantiations; a unit of its own so that it compiles in parallel with the
// larger ones).
#include "bx_launch.cuh"
#include "bx_plain.cuh"
namespace bx {
BX_DEFINE_CELL_STEP_LAUNCHER(double, 32)
BX_DEFINE_CELL_STEP_LAUNCHER(double, 64)

namespace {
using PlainKernel = void (*)(PlainGeom, StepPtrs, StepConst, PlainRun);
PlainKernel plain_kernel(bool six, bool gated, bool res) {
  if (res) return six ? (gated ? k_plain_step<1, true, true> : k_plain_step<1, false, true>)
                      : (gated ? k_plain_step<0, true, true> : k_plain_step<0, false, true>);
  return six ? (gated ? k_plain_step<1, true, false> : k_plain_step<1, false, false>)
             : (gated ? k_plain_step<0, true, false> : k_plain_step<0, false, false>);
}
size_t plain_smem(const StepConst& k, const PlainRun& r, bool gated) {
  return sizeof(double) * (size_t)PlainSmem(r.nc_max, r.ne_max, r.nm_max, k.I, gated).total;
}
}  // namespace

cudaError_t launch_plain_step(bool six, bool gated, cudaStream_t s, const PlainGeom& g, const StepPtrs& p,
                              const StepConst& k, const PlainRun& r) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)g.ntile);
  cfg.blockDim = dim3(kPlainT);
  cfg.dynamicSmemBytes = plain_smem(k, r, gated);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, plain_kernel(six, gated, false), g, p, k, r);
}

cudaError_t launch_plain_resident(bool six, bool gated, cudaStream_t s, const PlainGeom& g, const StepPtrs& p,
                                  const StepConst& k, const PlainRun& r) {
  cudaError_t e = cudaMemsetAsync(r.ctl, 0, sizeof(unsigned), s);   // the barrier counter
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<PlainGeom*>(&g), const_cast<StepPtrs*>(&p), const_cast<StepConst*>(&k),
                  const_cast<PlainRun*>(&r)};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(plain_kernel(six, gated, true)),
                                     dim3((unsigned)g.ntile), dim3(kPlainT), args, plain_smem(k, r, gated), s);
}

cudaError_t plain_resident_per_sm(bool six, bool gated, size_t smem, int* per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, plain_kernel(six, gated, true), kPlainT, smem);
}

cudaError_t plain_smem_attr(bool six, bool gated, size_t smem) {
  for (int res = 0; res < 2; ++res) {
    const cudaError_t e = cudaFuncSetAttribute(plain_kernel(six, gated, res != 0),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace bx
