// Plain FP64 form: small CTAs of the fused cell step, and the factored step
// (instantiations; a unit of its own so that it compiles in parallel with the
// larger ones).
#include "bx_launch.cuh"
#include "bx_plain.cuh"
namespace bx {
BX_DEFINE_CELL_STEP_LAUNCHER(double, 32)
BX_DEFINE_CELL_STEP_LAUNCHER(double, 64)

namespace {
using PlainKernel = void (*)(PlainGeom, StepPtrs, StepConst, PlainRun, EnvNp);
enum PlainForm { PF_STREAM, PF_RES, PF_ECM };
template <bool RES, bool ECM>
PlainKernel pick(bool six, bool gated) {
  return six ? (gated ? k_plain_step<1, true, RES, ECM> : k_plain_step<1, false, RES, ECM>)
             : (gated ? k_plain_step<0, true, RES, ECM> : k_plain_step<0, false, RES, ECM>);
}
PlainKernel plain_kernel(bool six, bool gated, PlainForm f) {
  return f == PF_RES ? pick<true, false>(six, gated) : f == PF_ECM ? pick<false, true>(six, gated)
                                                                   : pick<false, false>(six, gated);
}
size_t plain_smem(const StepConst& k, const PlainRun& r, bool gated, bool ecm) {
  return sizeof(double) * (size_t)PlainSmem(r.nc_max, r.ne_max, r.nm_max, k.I, gated, ecm).total;
}
}  // namespace

cudaError_t launch_plain_step(bool six, bool gated, bool ecm, cudaStream_t s, const PlainGeom& g, const StepPtrs& p,
                              const StepConst& k, const PlainRun& r, const EnvNp& en) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(g.ntile + en.nblk));
  cfg.blockDim = dim3(kPlainT);
  cfg.dynamicSmemBytes = plain_smem(k, r, gated, ecm);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, plain_kernel(six, gated, ecm ? PF_ECM : PF_STREAM), g, p, k, r, en);
}

cudaError_t launch_plain_resident(bool six, bool gated, cudaStream_t s, const PlainGeom& g, const StepPtrs& p,
                                  const StepConst& k, const PlainRun& r, int counter) {
  cudaError_t e = cudaMemsetAsync(r.ctl, counter, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  EnvNp en{};
  void* args[] = {const_cast<PlainGeom*>(&g), const_cast<StepPtrs*>(&p), const_cast<StepConst*>(&k),
                  const_cast<PlainRun*>(&r), &en};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(plain_kernel(six, gated, PF_RES)),
                                     dim3((unsigned)g.ntile), dim3(kPlainT), args, plain_smem(k, r, gated, false), s);
}

cudaError_t plain_resident_per_sm(bool six, bool gated, size_t smem, int* per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, plain_kernel(six, gated, PF_RES), kPlainT, smem);
}

cudaError_t plain_smem_attr(bool six, bool gated, bool ecm, size_t smem) {
  for (PlainForm f : {PF_STREAM, PF_RES, PF_ECM}) {
    if ((f == PF_ECM) != ecm) continue;
    const cudaError_t e = cudaFuncSetAttribute(plain_kernel(six, gated, f),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace bx
