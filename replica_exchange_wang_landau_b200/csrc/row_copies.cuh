// row_copies.cuh — what the sweeps share that copy rows of couplings to shared memory ahead of the walker
// (sweep.cu, sweep_split.cu).
#pragma once
#include "common.cuh"

namespace wlg {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

template <int kPrec> struct CouplingType;
template <> struct CouplingType<WLG_PRECISION_FP64> { using T = double; };
template <> struct CouplingType<WLG_PRECISION_FP32> { using T = float; };
template <> struct CouplingType<WLG_PRECISION_BF16> { using T = __nv_bfloat16; };

}  // namespace wlg
