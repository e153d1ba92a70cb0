// tma.cuh -- bulk tensor copies into shared memory: the mbarrier helpers, the
// descriptor of a float32 tensor, and the word a context's kernels set when one
// of their bounded waits runs out.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "cuda_util.cuh"

namespace ctbb {

// Descriptor of a float32 tensor (dims and box innermost first, strides of
// dims 1 .. rank - 1 in bytes); samples outside it read as zeros.
int tensor_map_f32(CUtensorMap *map, const float *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                   const cuuint32_t *box);
// The word that the kernels of one context set when a bounded wait on a copy
// runs out, in pinned host memory so that it is read without a copy.  Such a
// kernel also writes NaN in place of the results it could not form.  Every
// stage call of the context looks at the word before its own launches, every
// synchronising call after its last; the first to find it set clears it and
// fails.
struct CopyError {
    int *word = nullptr;
    int ensure();  // CTBB_ERR_ALLOC if there is no pinned memory
    bool set() const { return word && *const_cast<volatile int *>(word); }
    void clear() { if (word) *const_cast<volatile int *>(word) = 0; }
    void release();
};
// The library-wide context's word (allocated if need be).
int *copy_error_word();

namespace {

constexpr uint32_t kWaitTries = 100000, kSuspendNs = 20000;

__device__ __forceinline__ uint32_t smem_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void barrier_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void barrier_arrive_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Waits for the phase of the given parity, in at most kWaitTries tries that
// may each sleep kSuspendNs (about two seconds); false when they ran out.
__device__ __forceinline__ bool barrier_wait(uint32_t bar, uint32_t parity)
{
    uint32_t left;
    asm volatile(
        "{\n .reg .pred p, q;\n"
        " mov.u32 %0, %3;\n"
        "WAIT_%=:\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %4;\n"
        " @p bra DONE_%=;\n"
        " sub.u32 %0, %0, 1;\n"
        " setp.ne.u32 q, %0, 0;\n"
        " @q bra WAIT_%=;\n"
        "DONE_%=:\n}\n"
        : "=&r"(left)
        : "r"(bar), "r"(parity), "n"(kWaitTries), "n"(kSuspendNs)
        : "memory");
    return left != 0;
}

// After a wait that ran out: give copies in flight time to land in this CTA's
// shared memory before it is left (two milliseconds).
__device__ __forceinline__ void wait_for_stray_copies()
{
    uint64_t t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (int n = 0; n < (1 << 20); ++n) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 2000000ull) break;
    }
}

}  // namespace

}  // namespace ctbb
