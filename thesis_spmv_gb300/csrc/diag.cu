// diag.cu -- diagonal slices: storage and SpMV for stencils and other
// matrices whose entries lie on few diagonals.
//
// Rows are cut into slices of 64.  A slice's slots are the distinct
// column - row offsets of its rows, merged in CRS order: slot j holds, for
// each of the 64 rows, the row's element at column row + offset_j, or
// nothing (a bit per row in the slot's mask; a slice whose slots are all
// full reads no masks).  A nonzero costs its value and 1/64 of a 4-byte
// offset: 8.06 bytes in FP64, 4.06 in FP32, where the merge layout streams
// 10 (16-bit columns) to 12 and SELL-32 6, and there are no row ends, carries
// or fix-up kernel.  Lane l of a warp sums rows l and l + 32 of its slice,
// each left to right in CRS order (as CRS::mv, Matrix/CRS.hpp:99-109), one
// FMA per element; x[row + offset] is a coalesced load with no index to wait
// for.
//
// What bounds it: HBM and, in FP64, the FP64 pipe (2 FMAs per clock per SM),
// close to each other on a 5-point stencil (4096^2: 0.140 ms for 8 bytes per
// nonzero and two vectors, 0.133 ms of FMAs).  Both want the loads far ahead
// of their use, so a lane copies its own values of the warp's next group of
// up to 5 slots into shared memory (cp.async, 16 bytes per slot; read back by
// the same lane, so nothing is synchronised) while the current group's ten x
// loads are in flight.  One group ahead suffices: with values loaded straight
// into registers the 4096^2 product took 0.187 ms (long-scoreboard stalls on
// DRAM latency), with an L2 prefetch of the next slice 0.175 ms, with the
// stages 0.160 ms; two groups ahead cost resident CTAs (0.183 ms).  Slices of
// 64 rows rather than 128: twice the warps on small matrices, and a shorter
// last round.
//
// Measured against the layouts it replaced, y = A x (GB300): FP64 4096^2
// 5-point 0.208 -> 0.160 ms, 3001 x 2777 5-point 0.105 -> 0.080, 1999 x 1501
// 9-point 0.073 -> 0.061, 512^2 9.4 -> 4.9 us; FP32 4096^2 0.151 -> 0.091 ms,
// 1999 x 1501 9-point 0.046 -> 0.025; power step 4096^2 0.217 -> 0.164 ms,
// 512^2 11.1 -> 6.2 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "diag.cuh"
#include "internal.h"
#include "merge.cuh"

namespace pwmgpu {

namespace {

// The rows of a slice walked together: head() is the smallest column - row
// offset among the rows' next elements (INT_MAX: none left); the walk's user
// takes the elements at that offset and loads the rows' next ones.  Every
// row's elements come in CRS order, whatever that order is.
struct SliceWalk {
    int row, cur[kDiagR], end[kDiagR], off[kDiagR];
    __device__ __forceinline__ void load(const int32_t* __restrict__ col, int r) {
        off[r] = cur[r] < end[r] ? __ldg(col + cur[r]) - (row + 32 * r) : INT_MAX;
    }
    __device__ __forceinline__ SliceWalk(const int32_t* __restrict__ row_start, const int32_t* __restrict__ col,
                                         int nor, int c, int lane) {
        row = c * kDiagRows + lane;
#pragma unroll
        for (int r = 0; r < kDiagR; ++r) {
            const int i = row + 32 * r;
            cur[r] = i < nor ? __ldg(row_start + i) : 0;
            end[r] = i < nor ? __ldg(row_start + i + 1) : 0;
            load(col, r);
        }
    }
    __device__ __forceinline__ int head() const {
        int d = off[0];
#pragma unroll
        for (int r = 1; r < kDiagR; ++r) d = min(d, off[r]);
        return __reduce_min_sync(0xffffffffu, d);
    }
};

// Slots per slice (ptr[c + 1], scanned afterwards), their sum in 64 bits, and
// flag = 1 once a slice exceeds kDiagMaxSlots or the sum exceeds `most` (the
// rest then stops early).  A CTA adds its slots to the sum 512 at a time -- an
// addition per warp takes half a millisecond on 4 M rows -- and 64 at a time
// where there are few, so that a small matrix stops in time (1024 irregular
// rows: 25 us sooner).
__global__ void __launch_bounds__(256) k_diag_count(const int32_t* __restrict__ row_start,
                                                    const int32_t* __restrict__ col, int nor, int nslices,
                                                    unsigned long long most, int32_t* __restrict__ ptr,
                                                    unsigned long long* total, int* flag) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const int step = nslices <= 4096 ? 6 : 9;
    __shared__ unsigned slots;  // of the CTA's slices
    unsigned sum = 0;           // of the warp's
    if (threadIdx.x == 0) slots = 0u;
    __syncthreads();
    // n more slots; whether the sum of all is known to exceed `most`
    auto add = [&](unsigned n) {
        const unsigned before = atomicAdd(&slots, n);
        const unsigned long long whole = ((before + n) >> step) - (before >> step);
        return whole && atomicAdd(total, whole << step) + (whole << step) > most;
    };
    for (int c = blockIdx.x * wpb + (threadIdx.x >> 5); c < nslices; c += gridDim.x * wpb) {
        if (__any_sync(0xffffffffu, *(volatile int*)flag)) break;
        SliceWalk w(row_start, col, nor, c, lane);
        int n = 0;
        for (int d; n <= kDiagMaxSlots && (d = w.head()) != INT_MAX; ++n) {
#pragma unroll
            for (int r = 0; r < kDiagR; ++r)
                if (w.off[r] == d) {
                    ++w.cur[r];
                    w.load(col, r);
                }
            if ((++sum & 63) == 0) {
                const bool over = lane == 0 && add(64u);
                if (over) *(volatile int*)flag = 1;
                if (__any_sync(0xffffffffu, over)) break;
            }
        }
        if (lane == 0) {
            ptr[c + 1] = n;
            if (n > kDiagMaxSlots) *(volatile int*)flag = 1;
        }
    }
    if (lane == 0) (void)add(sum & 63);
    __syncthreads();
    const unsigned left = slots & ((1u << step) - 1u);
    if (threadIdx.x == 0 && left) atomicAdd(total, (unsigned long long)left);
}

// The slots' offsets, masks and FP64 values, and the slices' records.
__global__ void __launch_bounds__(256) k_diag_fill(const int32_t* __restrict__ row_start,
                                                   const int32_t* __restrict__ col, const double* __restrict__ val,
                                                   int nor, int nslices, const int32_t* __restrict__ ptr,
                                                   int2* __restrict__ rec, int32_t* __restrict__ offs,
                                                   SlotMask* __restrict__ masks, double* __restrict__ out) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int c = blockIdx.x * wpb + (threadIdx.x >> 5); c < nslices; c += gridDim.x * wpb) {
        const int s0 = ptr[c], n = ptr[c + 1] - s0;
        SliceWalk w(row_start, col, nor, c, lane);
        bool part = false;
        for (int j = 0; j < n; ++j) {
            const int d = w.head();
            double v[kDiagR];
            unsigned m[kDiagR];
#pragma unroll
            for (int r = 0; r < kDiagR; ++r) {
                const bool here = w.off[r] == d;
                m[r] = __ballot_sync(0xffffffffu, here);
                part |= m[r] != 0xffffffffu;
                v[r] = 0.0;
                if (here) {
                    v[r] = __ldg(val + w.cur[r]);
                    ++w.cur[r];
                    w.load(col, r);
                }
            }
            double* o = out + ((size_t)(s0 + j) * 32 + lane) * kDiagR;
            SlotMask q;
#pragma unroll
            for (int r = 0; r < kDiagR; ++r) {
                o[r] = v[r];
                q.w[r] = m[r];
            }
            if (lane == 0) {
                offs[s0 + j] = d;
                masks[s0 + j] = q;
            }
        }
        if (lane == 0) rec[c] = make_int2(s0, (n << 1) | (part ? 1 : 0));
    }
}

// out[p] = the largest column that slices [0, ns (p + 1) / K) may read (by
// slice and offset: up to kDiagRows - 1 columns too many where the last rows lack it).
__global__ void __launch_bounds__(256) k_diag_maxcol(const int2* __restrict__ rec, const int32_t* __restrict__ offs,
                                                     int nslices, int nor, int noc, int K, int* __restrict__ out) {
    __shared__ int red[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c0 = (int)((long long)nslices * blockIdx.x / K), c1 = (int)((long long)nslices * (blockIdx.x + 1) / K);
    int mx = -1;
    for (int c = c0 + (int)threadIdx.x; c < c1; c += 256) {
        const int2 q = rec[c];
        const int last = (int)min((long long)nor, (c + 1LL) * kDiagRows) - 1;
        for (int j = 0; j < (q.y >> 1); ++j)
            mx = max(mx, (int)min((long long)noc - 1, (long long)last + offs[q.x + j]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) red[w] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) mx = max(mx, red[i]);
        for (int p = blockIdx.x; p < K; ++p) atomicMax(out + p, mx);
    }
}

template <typename VT>
__global__ void k_diag_convert(const double* __restrict__ in, VT* __restrict__ out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (VT)in[i];
}

template <typename VT, typename XT>
struct DiagArgs {
    const int2* rec;
    const int32_t* offs;
    const unsigned* masks;  // kDiagR words per slot
    const VT* val;
    int nor, c0, c1;  // slices [c0, c1)
    const XT* x;
    XT* y;
    const unsigned int* mx_in;  // MODE_POWER / MODE_SCALE: the rescale's source (or nsq_in, or neither: e = 0)
    const double* nsq_in;
    unsigned int* mx_out;  // MODE_SCALE
    double* npart;         // MODE_POWER: per-CTA shares of ||y||^2, summed in order by the last CTA
    unsigned int* counter;
    double* nsq_out;
};

template <int MODE, typename VT, typename XT>
__global__ void __launch_bounds__(kDiagNT, kDiagOcc) k_diag_spmv(DiagArgs<VT, XT> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int tw = (gridDim.x * kDiagNT) >> 5;
    // the lane's own values only: no other thread reads what it stages
    VT* const ring = reinterpret_cast<VT*>(smem_raw) +
                     (threadIdx.x >> 5) * (kDiagStages * kDiagU * kDiagRows) + lane * kDiagR;
    const uint64_t pol = policy_evict_first();
    // the next group to stage: slice pc's slots from ps on; prec: the record
    // of the slice after it
    int pc = a.c0 + (int)((blockIdx.x * kDiagNT + threadIdx.x) >> 5);
    int2 prec = pc < a.c1 ? __ldg(a.rec + pc) : make_int2(0, 0);
    int ps = prec.x, pl = prec.y;
    prec = pc + tw < a.c1 ? __ldg(a.rec + pc + tw) : make_int2(0, 0);
    auto stage_next = [&](int stage) {
        DiagGroup q{pc, ps, pl, 0, 0u};
        if (pc < a.c1) {
            const int m = pl >> 1;
            const VT* src = a.val + ((size_t)ps * kDiagRows + lane * kDiagR);
            stage_group(ring + stage * (kDiagU * kDiagRows), src, m, pol);
            if (lane < m) q.offl = __ldg(a.offs + ps + lane);
            if ((pl & 1) && lane < m * kDiagR) q.ml = __ldg(a.masks + (size_t)ps * kDiagR + lane);
            ps += kDiagU;
            pl -= 2 * kDiagU;
            if (pl < 2) {
                pc += tw;
                ps = prec.x;
                pl = prec.y;
                prec = pc + tw < a.c1 ? __ldg(a.rec + pc + tw) : make_int2(0, 0);
            }
        }
        copy_commit();
        return q;
    };
    // Plan data, loaded before the kernel before on the stream has ended: what
    // stage_next reads (records, offsets, masks, values) was complete, its
    // stream synchronised, before this launch was made.
    DiagGroup cur = stage_next(0);
    pdl_wait();
    int e = 0;
    if (MODE != MODE_SPMV)
        e = a.mx_in ? pow2_rescale_exponent_key<XT>(*a.mx_in)
                    : (a.nsq_in ? pow2_rescale_exponent(*a.nsq_in, rescale_window<XT>()) : 0);
    double ss = 0.0;
    unsigned mx = 0u;
    int stage = 0;
    XT acc[kDiagR] = {};
    while (cur.c < a.c1) {
        const DiagGroup nxt = stage_next(stage ^ 1);
        const int row = cur.c * kDiagRows + lane;
        const VT* st = ring + stage * (kDiagU * kDiagRows);
        if (cur.left & 1) group_fma<true, VT, XT>(a.x + row, st, cur, lane, acc);
        else group_fma<false, VT, XT>(a.x + row, st, cur, lane, acc);
        if (cur.left < 2 * (kDiagU + 1)) {  // the slice's last group
#pragma unroll
            for (int r = 0; r < kDiagR; ++r) {
                if (row + 32 * r < a.nor) {
                    XT o = acc[r];
                    if (MODE != MODE_SPMV && e != 0) o = scale_pow2(o, e);
                    a.y[row + 32 * r] = o;
                    if (MODE == MODE_POWER) ss = fma((double)o, (double)o, ss);
                    if (MODE == MODE_SCALE) mx = max(mx, mag_key(o));
                }
                acc[r] = XT(0);
            }
        }
        cur = nxt;
        stage ^= 1;
    }
    if (MODE == MODE_SCALE && a.mx_out) block_max_out<kDiagNT>(mx, a.mx_out);
    if (MODE != MODE_POWER || !a.npart) return;
    __shared__ double red[kDiagNT / 32];
    __shared__ bool am_last;
    const double t = block_sum<kDiagNT>(ss, red);
    if (threadIdx.x == 0) {
        a.npart[blockIdx.x] = t;
        __threadfence();
        am_last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (am_last && threadIdx.x < 32) {
        __threadfence();
        double s = 0.0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) s += __ldcg(a.npart + i);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) {
            *a.nsq_out = s;
            *a.counter = 0u;
        }
    }
}

template <int MODE, typename VT, typename XT>
int diag_occ() {
    static int occ = 0;
    if (occ == 0) {
        int o = 0;
        cudaFuncSetAttribute(k_diag_spmv<MODE, VT, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, diag_smem<VT>());
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_diag_spmv<MODE, VT, XT>, kDiagNT, diag_smem<VT>()) !=
                cudaSuccess ||
            o < 1)
            o = 1;
        occ = std::min(o, kDiagMaxCtas);
    }
    return occ;
}

template <int MODE, typename VT, typename XT>
cudaError_t diag_launch(const DiagArgs<VT, XT>& a, int sm_count, bool pdl, cudaStream_t st) {
    const long long ctas = ((long long)(a.c1 - a.c0) + kDiagNT / 32 - 1) / (kDiagNT / 32);
    if (ctas <= 0) return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::min<long long>(ctas, (long long)diag_occ<MODE, VT, XT>() * sm_count));
    cfg.blockDim = dim3(kDiagNT);
    cfg.dynamicSmemBytes = diag_smem<VT>();
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k_diag_spmv<MODE, VT, XT>, a);
    return cudaGetLastError();
}

template <typename VT, typename XT>
cudaError_t diag_mode(int mode, const DiagArgs<VT, XT>& a, int sm_count, bool pdl, cudaStream_t st) {
    switch (mode) {
        case kModePower: return diag_launch<MODE_POWER, VT, XT>(a, sm_count, pdl, st);
        case kModeScale: return diag_launch<MODE_SCALE, VT, XT>(a, sm_count, pdl, st);
        default: return diag_launch<MODE_SPMV, VT, XT>(a, sm_count, pdl, st);
    }
}

}  // namespace

void DiagPlan::release() {
    dev_free(mem);
    dev_free(val32);
    dev_free(valbf);
    *this = DiagPlan();
}

// One allocation of scratch (DiagFound, slots per slice, the scan's), one of
// the plan: on a small matrix the allocations and waits are the build's cost.
namespace {
// Stored elements within 1.25 of the nonzeros: at that line the layout
// streams 10.1 bytes per nonzero, as much as the merge layout at its
// best (10, plus a fix-up kernel).  (128 slots more: a few slices,
// where either is one launch's latency.)
unsigned long long most_slots(long long nnz) {
    return (unsigned long long)((1.25 * (double)nnz + 128.0 * kDiagRows) / kDiagRows);
}
int* slot_ptr(const DiagBuild& B) { return reinterpret_cast<int32_t*>(B.tmp + sizeof(DiagFound)); }
int fill_blocks(int nslices, int sm_count) {
    return (int)std::min<long long>(((long long)nslices + 7) / 8, 32LL * sm_count);
}
}  // namespace

int diag_count(DiagBuild& B, const int32_t* row_start, const int32_t* col, int nor, long long nnz, int sm_count,
               Scratch& scratch, DiagFound* found, cudaStream_t st) {
    B = DiagBuild();
    if (nor <= 0 || nnz <= 0) return 1;
    const int ns = (nor + kDiagRows - 1) / kDiagRows;
    const size_t heads = sizeof(DiagFound) + sizeof(int32_t);
    cudaError_t e = scratch.alloc(&B.tmp, heads + sizeof(int32_t) * ((size_t)ns + (size_t)scan_scratch_elems(ns)));
    if (e == cudaSuccess) e = cudaMemsetAsync(B.tmp, 0, heads, st);
    if (e == cudaSuccess) {
        DiagFound* d = reinterpret_cast<DiagFound*>(B.tmp);
        k_diag_count<<<fill_blocks(ns, sm_count), 256, 0, st>>>(row_start, col, nor, ns, most_slots(nnz), slot_ptr(B),
                                                                &d->total, &d->flag);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(found, B.tmp, sizeof *found, cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return 2;
    }
    B.nslices = ns;
    return 0;
}

int diag_fill(DiagPlan& D, const DiagBuild& B, const DiagFound& found, const int32_t* row_start, const int32_t* col,
              const double* val, int nor, long long nnz, int sm_count, cudaStream_t st) {
    D.release();
    if (found.flag || found.total > most_slots(nnz)) return 1;
    const int ns = B.nslices;
    const size_t slots = (size_t)found.total, elems = slots * kDiagRows;
    auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
    const size_t vb = up(sizeof(double) * (elems + 1)), rb = up(sizeof(int2) * (size_t)ns),
                 mb = up(sizeof(SlotMask) * (slots + 1)), ob = up(sizeof(int32_t) * (slots + 1)),
                 nb = sizeof(double) * kDiagMaxCtas * (size_t)sm_count;
    int32_t* ptr = slot_ptr(B);
    cudaError_t e = dev_alloc(&D.mem, vb + rb + mb + ob + nb);
    if (e == cudaSuccess) e = launch_inclusive_scan(ptr + 1, ns, ptr + 1 + ns, st);
    if (e == cudaSuccess) {
        unsigned char* p = static_cast<unsigned char*>(D.mem);
        D.val64 = reinterpret_cast<double*>(p);
        D.rec = reinterpret_cast<int2*>(p + vb);
        D.masks = p + vb + rb;
        D.offs = reinterpret_cast<int32_t*>(p + vb + rb + mb);
        D.npart = reinterpret_cast<double*>(p + vb + rb + mb + ob);
        k_diag_fill<<<fill_blocks(ns, sm_count), 256, 0, st>>>(row_start, col, val, nor, ns, ptr, D.rec, D.offs,
                                                               (SlotMask*)D.masks, D.val64);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        if (D.mem) (void)cudaStreamSynchronize(st);
        D.release();
        return 2;
    }
    D.nslices = ns;
    D.elems = (long long)elems;
    return 0;
}

int diag_low_values(DiagPlan& D, bool bf16, int sm_count, cudaStream_t st) {
    void** dst = bf16 ? &D.valbf : (void**)&D.val32;
    if (*dst) return 0;
    if (dev_alloc(dst, (bf16 ? sizeof(__nv_bfloat16) : sizeof(float)) * ((size_t)D.elems + 8)) != cudaSuccess) {
        (void)cudaGetLastError();
        *dst = nullptr;
        return 2;
    }
    if (bf16)
        k_diag_convert<__nv_bfloat16><<<8 * sm_count, 256, 0, st>>>(D.val64, (__nv_bfloat16*)D.valbf, (size_t)D.elems);
    else
        k_diag_convert<float><<<8 * sm_count, 256, 0, st>>>(D.val64, D.val32, (size_t)D.elems);
    // k_diag_spmv stages its first values before it waits for the kernel
    // before it, so they are complete before a product can be launched
    if (cudaGetLastError() == cudaSuccess && cudaStreamSynchronize(st) == cudaSuccess) return 0;
    (void)cudaGetLastError();
    dev_free(*dst);
    *dst = nullptr;
    return 2;
}

cudaError_t launch_diag_maxcol(const DiagPlan& D, int nor, int noc, int K, int* out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0xFF, sizeof(int) * (size_t)K, st);  // -1 everywhere
    if (e != cudaSuccess) return e;
    k_diag_maxcol<<<K, 256, 0, st>>>(D.rec, D.offs, D.nslices, nor, noc, K, out);
    return cudaGetLastError();
}

cudaError_t launch_diag_spmv(const DiagPlan& D, int cfg, int mode, int nor, const void* x, void* y,
                             const SliceStep& s, int sm_count, cudaStream_t st) {
    const int c1 = s.c1 < 0 ? D.nslices : s.c1;
    double* np = s.nsq_out ? D.npart : nullptr;
    const unsigned* masks = (const unsigned*)D.masks;
    if (cfg == kCfgF64)
        return diag_mode(mode,
                         DiagArgs<double, double>{D.rec, D.offs, masks, D.val64, nor, s.c0, c1, (const double*)x,
                                                  (double*)y, s.mx_in, s.nsq_in, s.mx_out, np, s.counter, s.nsq_out},
                         sm_count, s.pdl, st);
    if (cfg == kCfgBF16)
        return diag_mode(mode,
                         DiagArgs<__nv_bfloat16, float>{D.rec, D.offs, masks, (const __nv_bfloat16*)D.valbf, nor, s.c0,
                                                        c1, (const float*)x, (float*)y, s.mx_in, s.nsq_in, s.mx_out,
                                                        np, s.counter, s.nsq_out},
                         sm_count, s.pdl, st);
    return diag_mode(mode,
                     DiagArgs<float, float>{D.rec, D.offs, masks, D.val32, nor, s.c0, c1, (const float*)x, (float*)y,
                                            s.mx_in, s.nsq_in, s.mx_out, np, s.counter, s.nsq_out},
                     sm_count, s.pdl, st);
}

int diag_slice_rows() { return kDiagRows; }

void diag_warm_launch_caches() {
    (void)diag_occ<MODE_SPMV, double, double>();
    (void)diag_occ<MODE_POWER, double, double>();
    (void)diag_occ<MODE_SCALE, double, double>();
    (void)diag_occ<MODE_SPMV, float, float>();
    (void)diag_occ<MODE_POWER, float, float>();
    (void)diag_occ<MODE_SCALE, float, float>();
    (void)diag_occ<MODE_SPMV, __nv_bfloat16, float>();
    (void)diag_occ<MODE_POWER, __nv_bfloat16, float>();
    (void)diag_occ<MODE_SCALE, __nv_bfloat16, float>();
}

}  // namespace pwmgpu
