// rows.cu -- sorted rows: storage and SpMV for matrices whose columns go
// anywhere.
//
// Rows are sorted by length (longest first, equal lengths in row order;
// within each of up to 16 windows of consecutive rows, a late window's longest
// rows in an earlier one) and cut into items, a
// warp's work: 32 rows with a lane each, 8 rows with four lanes each, or one
// row with the whole warp, by length.  An item is a run of units of 64
// (column, value) pairs: in unit j a lane with G lanes to its row holds the
// row's elements 2 (j G + q) and the next, q its place among the G.  A warp
// loads its lanes' pairs of kRowsU units together, gathers x and adds, one FMA
// per element; a lane with a row of its own sums it left to right in CRS order
// (as CRS::mv, Matrix/CRS.hpp:99-109), else the lanes' sums meet in a fixed
// shuffle tree.  Absent elements have column -1 and read nothing.  There are
// no row ends inside an item, no carries and no fix-up.
//
// Bound: the gathers of x.  A GB300 serves 295 G random 8-byte gathers a
// second (0.94 per clock and SM, whatever the size of x), so 67 M elements
// take 227 us, and 264 us with the 12 bytes per element streamed beside them.
// The merge path needs its shared memory for row ends and products: fewer
// warps, fewer gathers in flight, and a fix-up per launch.  FP64 SpMV, merge
// path -> here: 4.19 M rows / 67 M elements (lengths from a power law) 343 ->
// 266 us; 2 M / 32 M 171 -> 122; 0.3 M / 4.8 M 50.7 -> 27.5; 30 K / 0.24 M
// 9.4 -> 5.1 us.  Twenty power steps on 1 M rows: 2.14 -> 1.60 ms.
//
// Windows keep a chunk of rows (and the y they store) together: a host-array
// product sends a window's rows home while the next one runs.  (A row that
// moved to an earlier window is stored before it is sent.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "internal.h"
#include "merge.cuh"

namespace pwmgpu {

namespace {

constexpr int kRowsNT = 128;
constexpr int kRowsOcc = 10;        // 48 registers
constexpr int kRowsU = 3;           // units whose loads are issued together
constexpr int kRowsWindows = 16;    // at most

// The windows of a matrix, the lengths from which a row gets four lanes (t4)
// and a warp (t32 <= 254) and goes before the other rows of its window (first
// >= t32), and the elements by which a row beyond kRowsLate moves one window up.
struct RowsCut {
    int windows, wrows, t4, t32, first, up;
};
constexpr int kRowsLate = 512;  // elements of a row that may start last
// Rows of each window by class (0: a warp, 1: four lanes, 2: a lane each), the
// first item of each (window, class), the longest row, and the units of all
// items.
struct RowsHead {
    int rows[3 * kRowsWindows];
    int item[3 * kRowsWindows + 1];
    int longest;
    unsigned long long units;
};
__host__ __device__ constexpr int class_shift(int cls) { return cls == 0 ? 5 : cls == 1 ? 2 : 0; }  // log2 of G

// The window in whose items a row runs: its own, or an earlier one where the
// work from its own window on is over before a warp has done the row.
__device__ __forceinline__ int row_window(int r, int len, const RowsCut& cut) {
    const int back = len > kRowsLate ? (len - kRowsLate) / cut.up : 0;
    return min(r / cut.wrows, max(cut.windows - 1 - back, 0));
}

// Sort key of a row: its window above a byte that puts long rows first (0: from
// cut.first on; lengths below 254 each have a value of their own).
__global__ void __launch_bounds__(256) k_rows_keys(const int32_t* __restrict__ row_start, int nor, RowsCut cut,
                                                   unsigned long long* __restrict__ key, int32_t* __restrict__ row,
                                                   RowsHead* head) {
    __shared__ int cnt[kRowsWindows * 3];
    for (int i = threadIdx.x; i < kRowsWindows * 3; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    int longest = 0;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nor; r += gridDim.x * blockDim.x) {
        const int len = row_start[r + 1] - row_start[r], w = row_window(r, len, cut);
        key[r] = (unsigned long long)w << 8 | (unsigned long long)(len >= cut.first ? 0 : 255 - min(len, 254));
        row[r] = r;
        atomicAdd(&cnt[3 * w + (len >= cut.t32 ? 0 : len >= cut.t4 ? 1 : 2)], 1);
        longest = max(longest, len);
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if ((threadIdx.x & 31) == 0) atomicMax(&head->longest, longest);
    __syncthreads();
    for (int i = threadIdx.x; i < kRowsWindows * 3; i += blockDim.x)
        if (cnt[i]) atomicAdd(&head->rows[i], cnt[i]);
}

// Items: where each (window, class) starts among them, their rows, and the
// units of each (off[i + 1], zero before and scanned afterwards).
__global__ void __launch_bounds__(256) k_rows_items(const int32_t* __restrict__ row_start,
                                                    const int32_t* __restrict__ perm, RowsHead* head,
                                                    int4* __restrict__ rec, int32_t* __restrict__ off) {
    constexpr int classes = 3 * kRowsWindows;
    __shared__ struct {
        int rows[classes], item[classes + 1], row[classes];
    } h;
    if (threadIdx.x < classes) h.rows[threadIdx.x] = head->rows[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        int items = 0, rows = 0;
        for (int k = 0; k < classes; ++k) {
            const int per = 32 >> class_shift(k % 3);
            h.item[k] = items;
            h.row[k] = rows;
            items += (h.rows[k] + per - 1) / per;
            rows += h.rows[k];
        }
        h.item[classes] = items;
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x <= classes) head->item[threadIdx.x] = h.item[threadIdx.x];
    unsigned long long sum = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < h.item[classes]; i += gridDim.x * blockDim.x) {
        int k = 0;
        while (i >= h.item[k + 1]) ++k;
        const int gs = class_shift(k % 3), per = 32 >> gs;
        const int first = (i - h.item[k]) * per, at = h.row[k] + first;
        const int r = perm[at];  // the item's longest row
        const int len = row_start[r + 1] - row_start[r];
        const int n = (len + (2 << gs) - 1) >> (gs + 1);
        rec[i] = make_int4(0, n, at, gs << 8 | min(h.rows[k] - first, per));
        off[i + 1] = n;
        sum += (unsigned long long)n;
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&head->units, sum);
}

__global__ void __launch_bounds__(256) k_rows_fill(const int32_t* __restrict__ row_start,
                                                   const int32_t* __restrict__ col, const double* __restrict__ val,
                                                   const int32_t* __restrict__ perm, int nitems,
                                                   const int32_t* __restrict__ off, int4* __restrict__ rec,
                                                   int32_t* __restrict__ ocol, double* __restrict__ oval) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int i = blockIdx.x * wpb + (threadIdx.x >> 5); i < nitems; i += gridDim.x * wpb) {
        const int4 q = rec[i];
        const int gs = q.w >> 8, sub = lane >> gs, place = lane & ((1 << gs) - 1);
        const int r = sub < (q.w & 255) ? perm[q.z + sub] : -1;
        const int k0 = r >= 0 ? row_start[r] : 0, len = r >= 0 ? row_start[r + 1] - k0 : 0;
        int2* oc = reinterpret_cast<int2*>(ocol + (size_t)off[i] * 64) + lane;
        double2* ov = reinterpret_cast<double2*>(oval + (size_t)off[i] * 64) + lane;
        for (int j = 0; j < q.y; ++j) {
            const int e = 2 * ((j << gs) + place);
            const bool a = e < len, b = e + 1 < len;
            oc[32 * (size_t)j] = make_int2(a ? col[k0 + e] : -1, b ? col[k0 + e + 1] : -1);
            ov[32 * (size_t)j] = make_double2(a ? val[k0 + e] : 0.0, b ? val[k0 + e + 1] : 0.0);
        }
        if (lane == 0) rec[i].x = off[i];
    }
}

// out[w] = the largest column of windows 0 .. w (kMaxcolCtas CTAs per window).
constexpr int kMaxcolCtas = 32;
struct RowsWins {
    int item[kRowsWindows + 1], n;
};
__global__ void __launch_bounds__(256) k_rows_maxcol(const int4* __restrict__ rec, const int32_t* __restrict__ col,
                                                     RowsWins g, long long units, int windows, int* __restrict__ out) {
    const int w = blockIdx.x / kMaxcolCtas, part = blockIdx.x % kMaxcolCtas;
    const long long lo = g.item[w] < g.n ? rec[g.item[w]].x : units, hi = g.item[w + 1] < g.n ? rec[g.item[w + 1]].x : units;
    const long long len = (hi - lo) * 64, p0 = lo * 64 + len * part / kMaxcolCtas, p1 = lo * 64 + len * (part + 1) / kMaxcolCtas;
    int mx = -1;
    for (long long k = p0 + threadIdx.x; k < p1; k += 256) mx = max(mx, __ldg(col + k));
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0)
        for (int p = w; p < windows; ++p) atomicMax(out + p, mx);
}

template <typename VT>
__global__ void k_rows_convert(const double* __restrict__ in, VT* __restrict__ out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (VT)in[i];
}

__device__ __forceinline__ void load_pair(const double* p, double (&v)[2]) {
    const double2 q = __ldcs(reinterpret_cast<const double2*>(p));
    v[0] = q.x;
    v[1] = q.y;
}
__device__ __forceinline__ void load_pair(const float* p, float (&v)[2]) {
    const float2 q = __ldcs(reinterpret_cast<const float2*>(p));
    v[0] = q.x;
    v[1] = q.y;
}
__device__ __forceinline__ void load_pair(const __nv_bfloat16* p, float (&v)[2]) {
    const unsigned q = __ldcs(reinterpret_cast<const unsigned*>(p));
    v[0] = __uint_as_float(q << 16);
    v[1] = __uint_as_float(q & 0xffff0000u);
}

template <typename VT, typename XT>
struct RowsArgs {
    const int4* rec;
    const int32_t* perm;
    const int32_t* col;
    const VT* val;
    int i0, i1;  // items [i0, i1)
    const XT* x;
    XT* y;
    const unsigned int* mx_in;
    const double* nsq_in;
    unsigned int* mx_out;
    double* npart;
    unsigned int* counter;
    double* nsq_out;
};

// A warp per item, the items in list order: the block scheduler hands the next
// ones to the SMs that are free, so the long items at a window's start balance
// themselves (a resident grid that strides over the items took 0.30 ms instead
// of 0.267 on the 4M-row irregular matrix, and warps with four items each 0.29).
template <int MODE, typename VT, typename XT>
__global__ void __launch_bounds__(kRowsNT, kRowsOcc) k_rows_spmv(RowsArgs<VT, XT> a) {
    const int lane = threadIdx.x & 31;
    const int i = a.i0 + (int)((blockIdx.x * kRowsNT + threadIdx.x) >> 5);
    const int4 q = i < a.i1 ? __ldg(a.rec + i) : make_int4(0, 0, 0, 0);
    const int gs = q.w >> 8, n = q.y;
    const int sub = lane >> gs;
    const bool mine = sub < (q.w & 255) && (lane & ((1 << gs) - 1)) == 0;
    const int row = mine ? __ldg(a.perm + q.z + sub) : 0;
    const int32_t* cp = a.col + (size_t)q.x * 64 + 2 * lane;
    const VT* vp = a.val + (size_t)q.x * 64 + 2 * lane;
    pdl_wait();
    int e = 0;
    if (MODE != MODE_SPMV)
        e = a.mx_in ? pow2_rescale_exponent_key<XT>(*a.mx_in)
                    : (a.nsq_in ? pow2_rescale_exponent(*a.nsq_in, rescale_window<XT>()) : 0);
    XT acc = XT(0);
#pragma unroll 1
    for (int j = 0; j < n; j += kRowsU) {
        int2 c[kRowsU];
        XT v[kRowsU][2], g[kRowsU][2];
#pragma unroll
        for (int u = 0; u < kRowsU; ++u)
            c[u] = j + u < n ? __ldcs(reinterpret_cast<const int2*>(cp + 64 * (size_t)(j + u))) : make_int2(-1, -1);
#pragma unroll
        for (int u = 0; u < kRowsU; ++u)
            if (j + u < n) load_pair(vp + 64 * (size_t)(j + u), v[u]);
#pragma unroll
        for (int u = 0; u < kRowsU; ++u) {
            g[u][0] = c[u].x >= 0 ? __ldg(a.x + c[u].x) : XT(0);
            g[u][1] = c[u].y >= 0 ? __ldg(a.x + c[u].y) : XT(0);
        }
#pragma unroll
        for (int u = 0; u < kRowsU; ++u) {
            if (c[u].x >= 0) acc = fma(v[u][0], g[u][0], acc);
            if (c[u].y >= 0) acc = fma(v[u][1], g[u][1], acc);
        }
    }
    for (int o = (1 << gs) >> 1; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    XT o = acc;
    if (MODE != MODE_SPMV && e != 0) o = scale_pow2(o, e);
    if (mine) a.y[row] = o;
    if (MODE == MODE_SCALE && a.mx_out) {
        __shared__ unsigned wmax[kRowsNT / 32];
        const unsigned m = __reduce_max_sync(0xffffffffu, mine ? mag_key(o) : 0u);
        if (lane == 0) wmax[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned t = wmax[0];
            for (int w = 1; w < kRowsNT / 32; ++w) t = max(t, wmax[w]);
            if (t > __ldcg(a.mx_out)) atomicMax(a.mx_out, t);  // (most CTAs are below the largest so far)
        }
    }
    if (MODE != MODE_POWER || !a.npart) return;
    __shared__ double red[kRowsNT / 32];
    __shared__ bool am_last;
    const double t = block_sum<kRowsNT>(mine ? (double)o * (double)o : 0.0, red);
    if (threadIdx.x == 0) {
        a.npart[blockIdx.x] = t;
        __threadfence();
        am_last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    double s = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kRowsNT) s += __ldcg(a.npart + k);
    s = block_sum<kRowsNT>(s, red);
    if (threadIdx.x == 0) {
        *a.nsq_out = s;
        *a.counter = 0u;
    }
}

template <int MODE, typename VT, typename XT>
cudaError_t rows_launch(const RowsArgs<VT, XT>& a, bool pdl, cudaStream_t st) {
    if (a.i1 <= a.i0) return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((a.i1 - a.i0 + kRowsNT / 32 - 1) / (kRowsNT / 32)));
    cfg.blockDim = dim3(kRowsNT);
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k_rows_spmv<MODE, VT, XT>, a);
    return cudaGetLastError();
}

template <typename VT, typename XT>
cudaError_t rows_mode(int mode, const RowsArgs<VT, XT>& a, bool pdl, cudaStream_t st) {
    switch (mode) {
        case kModePower: return rows_launch<MODE_POWER, VT, XT>(a, pdl, st);
        case kModeScale: return rows_launch<MODE_SCALE, VT, XT>(a, pdl, st);
        default: return rows_launch<MODE_SPMV, VT, XT>(a, pdl, st);
    }
}

}  // namespace

void RowsPlan::release() {
    dev_free(mem);
    dev_free(val32);
    dev_free(valbf);
    *this = RowsPlan();
}

int rows_build(RowsPlan& R, const int32_t* row_start, const int32_t* col, const double* val, int nor, long long nnz,
               bool narrow, int sm_count, Scratch& keep, void* pinned, cudaStream_t st) {
    R.release();
    if (nor <= 0 || nnz <= 0) return 1;
    // Lengths from which a row gets four lanes and a warp.  An item takes a
    // batch of loads per 6 elements of a lane, about 0.8 us, so a small
    // matrix (little work beside its longest items) cuts earlier.  64 / 255
    // and 16 / 64: 30.5 and 27.5 us on 4.8 M nonzeros, 9.8 and 5.1 us on
    // 0.24 M; on 67 M nonzeros 64 / 255 beat 128 / 255 and 32 / 255 by 3 %.
    RowsCut cut{1, nor, 64, 254, 0, 0};
    if (nnz < (1LL << 23)) {
        cut.t4 = 16;
        cut.t32 = 64;
    }
    if (nor >= kRowsWindows * 16384) {
        cut.windows = kRowsWindows;
        cut.wrows = (nor + kRowsWindows - 1) / kRowsWindows;
    }
    // A warp does 2000 elements of a row while the matrix does a million (7.5 ns
    // and 4 ps an element): what a row has beyond kRowsLate runs beside the
    // windows from its own on, or moves up to a window with as much behind it.
    cut.up = (int)std::max(1LL, nnz / (2000LL * cut.windows));
    cut.first = kRowsLate + (int)(nnz / 32000);
    static_assert(sizeof(RowsHead) <= kPinnedBlock, "the pinned block");
    RowsHead& h = *static_cast<RowsHead*>(pinned);
    auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
    const long long most = (long long)nor + 3 * kRowsWindows;  // items at most
    const long long tabn = triplet_sort_table_elems(nor);
    const size_t hb = up(sizeof h), ob = up(sizeof(int32_t) * ((size_t)most + 1)),
                 kb = up(sizeof(unsigned long long) * (size_t)nor), sb = up(sizeof(int32_t) * (size_t)nor),
                 tb = up(sizeof(int32_t) * (size_t)tabn),
                 cb = up(sizeof(int32_t) * (size_t)scan_scratch_elems(std::max(tabn, most))),
                 ib = sizeof(int4) * (size_t)most;
    const int blocks = std::min(16 * sm_count, (nor + 255) / 256);
    // past this the longest row is too long (see below)
    const double longest = 1024.0 + std::min((double)nnz / 1000.0, 4096.0 + (double)nnz / 4000.0);
    unsigned char* tmp = nullptr;
    int rc = 2;
    do {
        if (keep.alloc(&tmp, hb + ob + 2 * kb + 2 * sb + tb + cb + ib) != cudaSuccess) break;
        unsigned char* p = tmp;
        RowsHead* dh = reinterpret_cast<RowsHead*>(p);
        auto* off = reinterpret_cast<int32_t*>(p += hb);
        auto* ka = reinterpret_cast<unsigned long long*>(p += ob);
        auto* kbuf = reinterpret_cast<unsigned long long*>(p += kb);
        auto* perm = reinterpret_cast<int32_t*>(p += kb);
        auto* other = reinterpret_cast<int32_t*>(p += sb);
        auto* tab = reinterpret_cast<int32_t*>(p += sb);
        auto* scratch = reinterpret_cast<int32_t*>(p += tb);
        auto* rec = reinterpret_cast<int4*>(p += cb);
        if (cudaMemsetAsync(tmp, 0, hb + ob, st) != cudaSuccess) break;
        if (cut.windows > 1) std::swap(perm, other);
        k_rows_keys<<<blocks, 256, 0, st>>>(row_start, nor, cut, ka, other, dh);
        if (cut.windows > 1) {
            // (many rows: no sort of a matrix that a long row rules out, 1 ms on 4 M rows)
            if (cudaMemcpyAsync(&h.longest, &dh->longest, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                break;
            if ((double)h.longest > longest) {
                rc = 1;
                break;
            }
        }
        if (launch_radix_pass(ka, other, nor, 0, tab, scratch, kbuf, perm, st) != cudaSuccess) break;
        if (cut.windows > 1) {
            if (launch_radix_pass(kbuf, perm, nor, 8, tab, scratch, ka, other, st) != cudaSuccess) break;
            std::swap(perm, other);
        }
        k_rows_items<<<std::min(4 * sm_count, (nor + 255) / 256), 256, 0, st>>>(row_start, perm, dh, rec, off);
        if (launch_inclusive_scan(off + 1, most, scratch, st) != cudaSuccess) break;
        if (cudaMemcpyAsync(&h, dh, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess) break;
        if (cudaStreamSynchronize(st) != cudaSuccess) break;
        // A row is one warp's work, 4.2 ns an element where L2 holds the matrix
        // and 7.5 where it does not: 1024 elements take as long as a small
        // matrix does on the merge path, a thousandth of the nonzeros as long as
        // the rest of one in L2 (4.8 M, longest row 2400: 28 us, merge path 50),
        // and a quarter of that is half of the rest of a large one.  (Longer
        // ones: 60 000 elements in 67 M 450 us, 560 where the row came last,
        // merge path 351; 17 000 in 16.7 M 134 and 102; eight of 10 000 in 9.5 M
        // 85 and 66.)  Padding: as the merge layout's extra.
        if ((double)h.longest > longest || h.units >= (1ull << 31) ||
            (double)h.units * 64.0 > 1.25 * (double)nnz + 16384.0) {
            rc = 1;
            break;
        }
        const int items = h.item[3 * kRowsWindows];
        // Short items in great number: a warp's launch outweighs its loads,
        // and the merge path with 16-bit columns reads 2 bytes less per
        // element.  SPMV time here and there: 4 M rows of 8 in a band of 30
        // 95 us, 92 (ten power steps 1.22 ms, 1.06), of 6 85 and 70, 16 in a
        // band of 300 66 and 93; columns anywhere: 4 M rows of 2 77 and 55,
        // of 4 109 and 103, of 6 102 and 147; 2 M rows of 2 25 and 42, of 4
        // 37 and 55 us.
        if (items > (narrow ? 8192 : 65536) && (double)h.units < (narrow ? 6.0 : 3.0) * (double)items) {
            rc = 1;
            break;
        }
        const size_t elems = (size_t)h.units * 64, vb = up(sizeof(double) * (elems + 64)),
                     nb = up(sizeof(int32_t) * (elems + 64)), rb = up(sizeof(int4) * (size_t)items),
                     gb = sizeof(double) * ((size_t)items / (kRowsNT / 32) + 1);
        if (dev_alloc(&R.mem, vb + nb + rb + sb + gb) != cudaSuccess) {
            R.mem = nullptr;
            break;
        }
        p = static_cast<unsigned char*>(R.mem);
        R.val64 = reinterpret_cast<double*>(p);
        R.col = reinterpret_cast<int32_t*>(p += vb);
        R.rec = reinterpret_cast<int4*>(p += nb);
        R.perm = reinterpret_cast<int32_t*>(p += rb);
        R.npart = reinterpret_cast<double*>(p += sb);
        if (cudaMemcpyAsync(R.perm, perm, sizeof(int32_t) * (size_t)nor, cudaMemcpyDeviceToDevice, st) !=
                cudaSuccess ||
            cudaMemcpyAsync(R.rec, rec, sizeof(int4) * (size_t)items, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            break;
        k_rows_fill<<<std::min(32 * sm_count, (items + 7) / 8), 256, 0, st>>>(row_start, col, val, R.perm, items, off,
                                                                              R.rec, R.col, R.val64);
        if (cudaGetLastError() != cudaSuccess) break;
        R.nitems = items;
        R.windows = cut.windows;
        R.wrows = cut.wrows;
        R.elems = (long long)elems;
        for (int w = 0; w <= kRowsWindows; ++w) R.win[w] = h.item[3 * w];
        rc = 0;
    } while (0);
    if (rc) {
        (void)cudaGetLastError();
        if (R.mem) (void)cudaStreamSynchronize(st);
        R.release();
    }
    return rc;
}

int rows_low_values(RowsPlan& R, bool bf16, int sm_count, cudaStream_t st) {
    void** dst = bf16 ? &R.valbf : (void**)&R.val32;
    if (*dst) return 0;
    if (dev_alloc(dst, (bf16 ? sizeof(__nv_bfloat16) : sizeof(float)) * ((size_t)R.elems + 64)) != cudaSuccess) {
        (void)cudaGetLastError();
        *dst = nullptr;
        return 2;
    }
    if (bf16)
        k_rows_convert<__nv_bfloat16><<<8 * sm_count, 256, 0, st>>>(R.val64, (__nv_bfloat16*)R.valbf, (size_t)R.elems);
    else
        k_rows_convert<float><<<8 * sm_count, 256, 0, st>>>(R.val64, R.val32, (size_t)R.elems);
    if (cudaGetLastError() == cudaSuccess && cudaStreamSynchronize(st) == cudaSuccess) return 0;
    (void)cudaGetLastError();
    dev_free(*dst);
    *dst = nullptr;
    return 2;
}

cudaError_t launch_rows_maxcol(const RowsPlan& R, int* out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0xFF, sizeof(int) * (size_t)R.windows, st);  // -1 everywhere
    if (e != cudaSuccess) return e;
    RowsWins g{};
    for (int w = 0; w <= R.windows; ++w) g.item[w] = w < R.windows ? R.win[w] : R.nitems;
    g.n = R.nitems;
    k_rows_maxcol<<<R.windows * kMaxcolCtas, 256, 0, st>>>(R.rec, R.col, g, R.elems / 64, R.windows, out);
    return cudaGetLastError();
}

cudaError_t launch_rows_spmv(const RowsPlan& R, int cfg, int mode, const void* x, void* y, const SliceStep& s,
                             cudaStream_t st) {
    const int i1 = s.c1 < 0 ? R.nitems : s.c1;
    double* np = s.nsq_out ? R.npart : nullptr;
    if (cfg == kCfgF64)
        return rows_mode(mode,
                         RowsArgs<double, double>{R.rec, R.perm, R.col, R.val64, s.c0, i1, (const double*)x, (double*)y,
                                                  s.mx_in, s.nsq_in, s.mx_out, np, s.counter, s.nsq_out},
                         s.pdl, st);
    if (cfg == kCfgBF16)
        return rows_mode(mode,
                         RowsArgs<__nv_bfloat16, float>{R.rec, R.perm, R.col, (const __nv_bfloat16*)R.valbf, s.c0, i1,
                                                        (const float*)x, (float*)y, s.mx_in, s.nsq_in, s.mx_out, np,
                                                        s.counter, s.nsq_out},
                         s.pdl, st);
    return rows_mode(mode,
                     RowsArgs<float, float>{R.rec, R.perm, R.col, R.val32, s.c0, i1, (const float*)x, (float*)y, s.mx_in,
                                            s.nsq_in, s.mx_out, np, s.counter, s.nsq_out},
                     s.pdl, st);
}

}  // namespace pwmgpu
