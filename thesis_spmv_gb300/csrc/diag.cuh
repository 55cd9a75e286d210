// diag.cuh -- the diagonal-slice group routine shared by the single-matrix
// kernel (diag.cu, which describes the layout) and the batched service's
// kernel (batch_diag.cu).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace pwmgpu {

// 4 CTAs of 256 threads per SM: 64 registers hold the ten x loads a lane has
// in flight without a spill, and 160 KB of stages leave 68 KB of L1 for x.
// (48 registers spill: 0.35 ms on the 4096^2 stencil; 3 CTAs 0.173 ms.)
constexpr int kDiagNT = 256;
constexpr int kDiagOcc = 4;
constexpr int kDiagR = 2;           // rows per lane
constexpr int kDiagRows = 32 * kDiagR;
constexpr int kDiagU = 5;           // slots per group (staged, and x loaded, together)
constexpr int kDiagStages = 2;      // groups staged: the one in use and the next
constexpr int kDiagMaxSlots = 256;  // per slice: more is no diagonal matrix
constexpr int kDiagMaxCtas = 8;     // per SM (room for the shares of ||y||^2)

// The rows of a slot that hold an element: bit l of word r for row 32 r + l.
struct __align__(4 * kDiagR) SlotMask {
    unsigned w[kDiagR];
};

// The lane's values of one slot, global -> shared, asynchronously (read once
// per pass: evict-first).
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src, uint64_t pol) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src),
                     "l"(pol)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src),
                     "n"(BYTES), "l"(pol)
                     : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Stage m slots (at most kDiagU) of the lane's own values: src / dst are the
// lane's first element of the group in global / shared memory.
template <typename VT>
__device__ __forceinline__ void stage_group(VT* dst, const VT* src, int m, uint64_t pol) {
#pragma unroll
    for (int u = 0; u < kDiagU; ++u)
        if (u < m) copy_async<kDiagR * (int)sizeof(VT)>(dst + u * kDiagRows, src + u * kDiagRows, pol);
}

template <typename VT>
constexpr int diag_smem() {
    return (kDiagNT / 32) * kDiagStages * kDiagU * kDiagRows * (int)sizeof(VT);
}

// A group: the next kDiagU (or fewer) slots of a warp's slice c.  offl and
// ml: the group's offsets and (where some slot lacks rows) mask words, one
// per lane, loaded when the group is staged.
struct DiagGroup {
    int c, slot;
    int left;  // 2 * slots of the slice from `slot` on + (some slot lacks rows)
    int offl;
    unsigned ml;
};

// At most kDiagU slots: acc[r] += value * x[row + 32 r + offset], in slot
// order.  All x loads go out together, then the wait for the values.
template <bool PART, typename VT, typename XT>
__device__ __forceinline__ void group_fma(const XT* __restrict__ xr, const VT* st, const DiagGroup& q, int lane,
                                          XT (&acc)[kDiagR]) {
    XT g[kDiagU][kDiagR];
    const int m = q.left >> 1;
    unsigned on = ~0u;  // bit u R + r: the lane's row r has an element in slot u
    if (PART) {
        on = 0u;
#pragma unroll
        for (int i = 0; i < kDiagU * kDiagR; ++i) on |= ((__shfl_sync(0xffffffffu, q.ml, i) >> lane) & 1u) << i;
    }
#pragma unroll
    for (int u = 0; u < kDiagU; ++u) {
        const XT* xd = xr + __shfl_sync(0xffffffffu, q.offl, u);
#pragma unroll
        for (int r = 0; r < kDiagR; ++r)
            g[u][r] = u < m && (!PART || ((on >> (u * kDiagR + r)) & 1u)) ? __ldg(xd + 32 * r) : XT(0);
    }
    copy_wait<kDiagStages - 1>();
#pragma unroll
    for (int u = 0; u < kDiagU; ++u) {
        if (u < m) {
#pragma unroll
            for (int r = 0; r < kDiagR; ++r)
                if (!PART || ((on >> (u * kDiagR + r)) & 1u))
                    acc[r] = fma((XT)st[u * kDiagRows + r], g[u][r], acc[r]);
        }
    }
}

}  // namespace pwmgpu
