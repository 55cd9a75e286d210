// batch_diag.cu -- a power step of every live solve of a diagonal-slice class
// (the serving loop's stencils; diag.cu describes the layout, batch.h the
// tables).
//
// The slots' slices form one list; a warp takes a run of consecutive slices,
// so its slot advances by a comparison, and stages the next group of values
// ahead as the single-matrix kernel does.  A step of the batch is a few
// microseconds of work, so what bounds it is the chain of dependent loads at
// its start (slice -> slot -> record -> offsets -> x) and the launches around
// it: the chain up to the values runs before the wait for the step before
// (programmatic dependent launch), and a key step is one kernel.  For that
// the slot state holds three key words in rotation: step `it` of a round
// reads the key of v_k from word it % 3, folds v_{k+1}'s into word
// (it + 1) % 3 and clears word (it + 2) % 3, last read by the step before;
// the iteration count advances once, in the round's norm passes.  Measured
// on 16 grids of 38^2 .. 512^2 (0.9 M rows), a round of 8 steps with BF16
// values: 0.234 -> 0.100 ms against the SELL-32 classes (with every class's
// kernels in the graph), with FP64 values 0.356 -> 0.168 ms.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "batch.h"
#include "diag.cuh"
#include "internal.h"
#include "merge.cuh"

namespace pwmgpu {

namespace {

// KEYS: a key step (see above); else the rows only.  from_key: the rescale of
// this step comes from key word it % 3 (the step before was a key step), else
// from ||v_k||^2 (none on a solve's first step).
// 3 CTAs per SM: the slots' pointers beside the x loads need 80 registers
// (4 per SM, with a few spills: 4 % slower on the 16 grids, 6 % faster on
// 128 of them; 5: 30 and 19 % slower).
template <typename VT, typename XT, bool KEYS>
__global__ void __launch_bounds__(kDiagNT, 3) k_batch_diag(const BatchTable* __restrict__ Tp, int it,
                                                                  int from_key) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * kDiagNT + threadIdx.x) >> 5), tw = (int)((gridDim.x * kDiagNT) >> 5);
    const int ntiles = Tp->ntiles;
    const int K = (ntiles + tw - 1) / tw;
    const long long first = (long long)gw * K;
    if (first >= ntiles) {
        pdl_wait();
        return;
    }
    const int g1 = (int)(first + K < ntiles ? first + K : ntiles);
    const BatchSlot* __restrict__ slots = Tp->slots;
    VT* const ring = reinterpret_cast<VT*>(smem_raw) +
                     (threadIdx.x >> 5) * (kDiagStages * kDiagU * kDiagRows) + lane * kDiagR;
    const uint64_t pol = policy_evict_first();
    // the next group to stage: slice pg (of slot pj) from plan slot ps on
    int pg = (int)first, pj = Tp->tile_slot[first];
    const int2* prec;
    const int32_t* poffs;
    const unsigned* pmasks;
    const VT* pval;
    int pend, ps, pl;
    auto enter = [&]() {  // slot pj's plan, at slice pg
        const BatchSlot* d = slots + pj;
        prec = d->drec - d->tile0;
        poffs = d->doffs;
        pmasks = d->dmasks;
        pval = static_cast<const VT*>(d->valp) + lane * kDiagR;
        pend = d->tile0 + d->nsub;
    };
    auto slice = [&]() {
        const int2 q = __ldg(prec + pg);
        ps = q.x;
        pl = q.y;
    };
    enter();
    slice();
    struct Item {
        DiagGroup q;
        int j;
    };
    auto stage_next = [&](int stage) {
        Item x{{pg, ps, pl, 0, 0u}, pj};
        if (pg < g1) {
            const int m = pl >> 1;
            stage_group(ring + stage * (kDiagU * kDiagRows), pval + (size_t)ps * kDiagRows, m, pol);
            if (lane < m) x.q.offl = __ldg(poffs + ps + lane);
            if ((pl & 1) && lane < m * kDiagR) x.q.ml = __ldg(pmasks + (size_t)ps * kDiagR + lane);
            ps += kDiagU;
            pl -= 2 * kDiagU;
            if (pl < 2 && ++pg < g1) {
                if (pg >= pend) {  // slots own consecutive slices
                    ++pj;
                    enter();
                }
                slice();
            }
        }
        copy_commit();
        return x;
    };
    Item cur = stage_next(0);
    pdl_wait();
    SlotState* const states = Tp->states;
    int jc = -1, stage = 0, tile0 = 0, nor = 0, e = 0;
    const XT* in = nullptr;
    XT* out = nullptr;
    SlotState* st = nullptr;
    unsigned mx = 0u;
    XT acc[kDiagR] = {};
    while (cur.q.c < g1) {
        const Item nxt = stage_next(stage ^ 1);
        if (cur.j != jc) {
            if (KEYS && jc >= 0) {
                warp_max_out(mx, &st->mxr[(it + 1) % 3]);
                mx = 0u;
            }
            jc = cur.j;
            const BatchSlot* d = slots + jc;
            st = states + d->state;
            tile0 = d->tile0;
            nor = d->nor;
            const int k = st->k + (from_key ? it : 0);
            in = static_cast<const XT*>((k & 1) ? d->Y : d->X);
            out = static_cast<XT*>((k & 1) ? d->X : d->Y);
            e = k == 0 ? 0
                : from_key ? pow2_rescale_exponent_key<XT>(st->mxr[it % 3])
                           : pow2_rescale_exponent(st->nsq, rescale_window<XT>());
        }
        const int c = cur.q.c - tile0;
        if (KEYS && c == 0 && lane == 0 && cur.q.left < 2 * (kDiagU + 1)) st->mxr[(it + 2) % 3] = 0u;
        const int row = c * kDiagRows + lane;
        const VT* sv = ring + stage * (kDiagU * kDiagRows);
        if (cur.q.left & 1) group_fma<true, VT, XT>(in + row, sv, cur.q, lane, acc);
        else group_fma<false, VT, XT>(in + row, sv, cur.q, lane, acc);
        if (cur.q.left < 2 * (kDiagU + 1)) {  // the slice's last group
#pragma unroll
            for (int r = 0; r < kDiagR; ++r) {
                if (row + 32 * r < nor) {
                    XT o = acc[r];
                    if (e != 0) o = scale_pow2(o, e);
                    out[row + 32 * r] = o;
                    if (KEYS) mx = max(mx, mag_key(o));
                }
                acc[r] = XT(0);
            }
        }
        cur = nxt;
        stage ^= 1;
    }
    if (KEYS) warp_max_out(mx, &st->mxr[(it + 1) % 3]);
}

template <typename VT, typename XT, bool KEYS>
int batch_diag_grid(int sm_count) {
    static int occ = 0;
    if (occ == 0) {
        int o = 0;
        cudaFuncSetAttribute(k_batch_diag<VT, XT, KEYS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             diag_smem<VT>());
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_batch_diag<VT, XT, KEYS>, kDiagNT, diag_smem<VT>()) !=
                cudaSuccess ||
            o < 1)
            o = 1;
        occ = o;
    }
    return occ * sm_count;
}

template <typename VT, typename XT, bool KEYS>
cudaError_t launch(const BatchTable* T, int it, int from_key, int sm_count, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(batch_diag_grid<VT, XT, KEYS>(sm_count));
    cfg.blockDim = dim3(kDiagNT);
    cfg.dynamicSmemBytes = diag_smem<VT>();
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_batch_diag<VT, XT, KEYS>, T, it, from_key);
}

template <typename VT, typename XT>
cudaError_t step(const BatchTable* T, int it, bool keys, int from_key, int sm_count, cudaStream_t st) {
    return keys ? launch<VT, XT, true>(T, it, from_key, sm_count, st)
                : launch<VT, XT, false>(T, it, from_key, sm_count, st);
}

}  // namespace

void batch_diag_prepare(int sm_count) {
    batch_diag_grid<double, double, true>(sm_count);
    batch_diag_grid<double, double, false>(sm_count);
    batch_diag_grid<float, float, true>(sm_count);
    batch_diag_grid<float, float, false>(sm_count);
    batch_diag_grid<__nv_bfloat16, float, true>(sm_count);
    batch_diag_grid<__nv_bfloat16, float, false>(sm_count);
}

cudaError_t launch_batch_diag(int cfg, const BatchTable* T, int it, bool keys, bool from_key, int sm_count,
                              cudaStream_t st) {
    switch (cfg) {
        case kCfgF32: return step<float, float>(T, it, keys, from_key, sm_count, st);
        case kCfgBF16: return step<__nv_bfloat16, float>(T, it, keys, from_key, sm_count, st);
        default: return step<double, double>(T, it, keys, from_key, sm_count, st);
    }
}

}  // namespace pwmgpu
