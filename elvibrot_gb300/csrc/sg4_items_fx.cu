// sg4_items_fx.cu -- the persistent H.psi kernel in block fixed point, one
// parameter-block size per translation unit: EVR_KIND = 0 the small block, 1
// the large one.
#include "sg4_fixed.cuh"

#ifndef EVR_KIND
#error "compile with -DEVR_KIND=0 (small parameter block) or 1 (large)"
#endif

namespace evr {

#define EVR_K_CAP (EVR_KIND == 1 ? EVR_PB_LARGE : EVR_PB_SMALL)

// the kernel's `it`, `fs` and `next`
static_assert(sizeof(ItemShared) + sizeof(FxShared) + sizeof(int) <= EVR_FX_STATIC_SMEM, "static shared memory of the items");

// The same item loop as hpsi_items_kernel.
template <int CAP>
__global__ void __launch_bounds__(EVR_FX_THREADS, EVR_FX_CTAS) hpsi_fixed_kernel(const __grid_constant__ ParamBlock<CAP> P,
                                                              const MItem* __restrict__ items, int n_items,
                                                              int item_base, unsigned int* counter) {
  __shared__ ItemShared it;
  __shared__ FxShared fs;
  __shared__ int next;
  for (int round = 0;; ++round) {
    if (threadIdx.x == 0) next = counter ? (int)atomicAdd(counter, 1u) : (round == 0 ? item_base + (int)blockIdx.x : n_items);
    __syncthreads();
    const int idx = next;
    __syncthreads();
    if (idx >= n_items) break;
    const MItem m = items[idx];
    run_item_fx(P.p[m.ctx], it, fs, m.term, m.rhs0, m.r);
  }
}

static void k_launch(unsigned grid, size_t smem, cudaStream_t s, const ParamBlock<EVR_K_CAP>& P, const MItem* items,
                     int n_items, int item_base, unsigned int* counter) {
  hpsi_fixed_kernel<EVR_K_CAP><<<grid, EVR_FX_THREADS, smem, s>>>(P, items, n_items, item_base, counter);
}

static cudaError_t k_static_smem(size_t* bytes) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, hpsi_fixed_kernel<EVR_K_CAP>);
  if (e == cudaSuccess) *bytes = a.sharedSizeBytes;
  return e;
}

static cudaError_t k_set_smem(int bytes) {
  return cudaFuncSetAttribute(hpsi_fixed_kernel<EVR_K_CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

#if EVR_KIND == 0
const MultiEntry<EVR_PB_SMALL> multi_fxsmall = {k_launch, k_static_smem, k_set_smem};
#else
const MultiEntry<EVR_PB_LARGE> multi_fxlarge = {k_launch, k_static_smem, k_set_smem};
#endif

}  // namespace evr
