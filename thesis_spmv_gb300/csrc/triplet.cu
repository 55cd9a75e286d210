// triplet.cu -- triplet (COO) -> CRS on the device, in the order of
// Util/TripletToCRS.hpp:135-172: rows ascending, columns ascending within a
// row.  For unique coordinates that order is unique; entries with the same
// (row, column) keep their input order (a stable sort), which is also what the
// host counting sort of the previous loader gave.
//
// Plan:
//   1. k_trip_scan: one read of rows / cols.  Range check (the first bad entry
//      by atomicMin), per-row counts (warp-aggregated atomics; their scan is
//      row_start), each entry's arrival number in its row (what the atomic
//      returned), the longest row, and two order flags: "not sorted by (row,
//      col)" and "not sorted by column".
//   2. Already sorted by (row, col): col / val are the input, copied.
//   3. Rows of at most kRowSortMax entries, where that pays (triplet_rows_fit):
//      k_trip_bucket writes each entry's index to row_start + arrival number,
//      k_trip_rows sorts every row in shared memory by (column, index) -- an
//      element's place is the number of smaller keys in its row, so the order
//      of the arrivals does not matter -- and k_trip_vals gathers the values.  Bound by the row atomics, the
//      scattered stores and the two gathers; every other access is a stream.
//      Scattered stores of 4 bytes run at 196 G/s, of 16 bytes at 31 G/s (67
//      and 268 MB), gathers at 260 G/s from what L2 holds and 117 G/s from 134
//      MB: so the index alone is scattered, and columns and values are
//      gathered one after the other.  Load of 21 M shuffled entries of a
//      2048^2 stencil: 7.9 ms with the radix sort, 3.15 with scattered {column,
//      index, value} records, 2.80 so (scan 0.24 ms, bucket 0.26, rows 0.26,
//      values 0.27); sorted by column 2.40 -> 2.23 ms; 8 M entries of a random
//      matrix 1.34 -> 1.20.
//   4. Otherwise: a stable LSD radix sort of the packed key row << 32 | col
//      with 8-bit digits: first the column digits (skipped when the input is
//      already sorted by column -- a stable sort by a key that is already in
//      order is the identity), then the row digits.  Per pass: k_radix_hist
//      counts digits per 4096-item tile into a digit-major table (one
//      inclusive scan makes it the exclusive offsets of every (digit, tile)),
//      and k_radix_scatter ranks each tile's items stably (warp match on the
//      digit, per-warp digit counters in shared memory) and writes key and
//      source index to their places; k_trip_gather then takes col = low word
//      of the sorted key and val = vals[source].
#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

namespace pwmgpu {

namespace {

constexpr int kRadixBins = 256;
constexpr int kSortWarps = 8;
constexpr int kSortThreads = kSortWarps * 32;
constexpr int kSortRounds = 16;                           // rounds of 32 items per warp
constexpr int kSortTile = kSortThreads * kSortRounds;     // 4096 items per CTA
constexpr int kWarpItems = 32 * kSortRounds;              // 512 consecutive items per warp

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Pass 1.  cnt has nor + 1 zeroed entries; the count of row r goes to
// cnt[r + 1] so that an inclusive scan of cnt + 1 leaves row_start in cnt.
__global__ void k_trip_scan(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols, long long nnz,
                            int32_t nor, int32_t noc, int32_t* __restrict__ cnt, int32_t* __restrict__ pos,
                            TripletScan* flags) {
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    bool unsorted_rc = false, unsorted_c = false;
    int longest = 0;
    // whole warps walk the array so that the neighbour exchange stays in-warp
    const long long start = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long span = (nnz + 31) / 32 * 32;
    for (long long k = start; k < span; k += stride) {
        const bool in = k < nnz;
        const int32_t r = in ? rows[k] : 0;
        const int32_t c = in ? cols[k] : 0;
        int32_t pr = __shfl_up_sync(0xffffffffu, r, 1);
        int32_t pc = __shfl_up_sync(0xffffffffu, c, 1);
        if (lane == 0 && in && k > 0) {
            pr = rows[k - 1];
            pc = cols[k - 1];
        }
        if (in && k > 0) {
            unsorted_rc |= r < pr || (r == pr && c < pc);
            unsorted_c |= c < pc;
        }
        const bool ok = in && r >= 0 && r < nor && c >= 0 && c < noc;
        if (in && !ok) atomicMin(&flags->bad, (unsigned long long)k);
        // rows of a warp are often equal (sorted input): one atomic per row
        const int key = ok ? r : -1 - lane;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        int first = 0;
        if (ok && lane == leader) first = atomicAdd(&cnt[r + 1], __popc(peers));
        first = __shfl_sync(0xffffffffu, first, leader);
        if (ok) {
            const int at = first + __popc(peers & lanemask_lt());
            pos[k] = at;
            longest = max(longest, at + 1);
        }
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if (lane == 0) atomicMax(&flags->longest, longest);
    if (__any_sync(0xffffffffu, unsorted_rc) && lane == 0) atomicOr(&flags->unsorted_rc, 1u);
    if (__any_sync(0xffffffffu, unsorted_c) && lane == 0) atomicOr(&flags->unsorted_c, 1u);
}

constexpr int kRowSortMax = 4096;  // entries of a row k_trip_rows sorts (32 KB of keys)
constexpr int kRowSortRows = 512;  // rows per CTA
// Threads per CTA: the keys of four CTAs leave L1 room for the gathers in
// flight (256 threads, six CTAs: 0.54 ms on 21 M entries; so 0.26).
constexpr int kRowSortNT = 512;
constexpr int kTripU = 4;  // entries per thread whose loads go together

// src[row_start[r] + arrival number] = the entry's index.  Four entries per
// thread with their loads together: the row_start gathers hide behind each
// other.
__global__ void __launch_bounds__(256) k_trip_bucket(const int32_t* __restrict__ rows, const int32_t* __restrict__ pos,
                                                     long long nnz, const int32_t* __restrict__ row_start,
                                                     int32_t* __restrict__ src) {
    constexpr int U = kTripU;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long k0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; k0 < nnz; k0 += U * step) {
        int32_t at[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = k0 + u * step;
            if (k < nnz) at[u] = __ldcs(rows + k);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = k0 + u * step;
            if (k < nnz) at[u] = __ldg(row_start + at[u]) + __ldcs(pos + k);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = k0 + u * step;
            if (k < nnz) src[at[u]] = (int32_t)k;
        }
    }
}

// Compares k_trip_rows makes, a row's length squared each, from the row counts:
// the sum, and the most of any kRowSortRows rows a CTA takes at a time.
__global__ void __launch_bounds__(256) k_trip_work(const int32_t* __restrict__ cnt, int32_t nor, TripletWork* out) {
    const int lane = threadIdx.x & 31;
    unsigned long long sum = 0, most = 0;
    const long long blocks = ((long long)nor + kRowSortRows - 1) / kRowSortRows;
    for (long long b = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); b < blocks; b += (long long)gridDim.x * 8) {
        const long long r1 = min((long long)nor, (b + 1) * kRowSortRows);
        unsigned long long t = 0;
        for (long long r = b * kRowSortRows + lane; r < r1; r += 32) {
            const unsigned long long n = (unsigned long long)__ldg(cnt + r);
            t += n * n;
        }
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        sum += t;
        most = most > t ? most : t;
    }
    if (lane == 0 && most) {
        atomicAdd(&out->sum, sum);
        atomicMax(&out->most, most);
    }
}

// Sort each row's records by (column, index).  A CTA takes kRowSortRows rows,
// as many consecutive ones at a time as fit kRowSortMax keys.
__global__ void __launch_bounds__(kRowSortNT) k_trip_rows(int32_t* __restrict__ src,
                                                          const int32_t* __restrict__ cols,
                                                          const int32_t* __restrict__ row_start, int32_t nor,
                                                          int32_t* __restrict__ col, int32_t* __restrict__ rows_out) {
    constexpr int U = kTripU;
    __shared__ unsigned long long key[kRowSortMax];
    __shared__ int start[kRowSortRows + 1];
    const int tid = threadIdx.x;
    for (long long r0 = (long long)blockIdx.x * kRowSortRows; r0 < nor; r0 += (long long)gridDim.x * kRowSortRows) {
        const int n = (int)(nor - r0 < kRowSortRows ? nor - r0 : kRowSortRows);
        for (int i = tid; i <= n; i += kRowSortNT) start[i] = __ldg(row_start + r0 + i);
        __syncthreads();
        for (int a = 0; a < n;) {
            // rows [a, b): the most that fit (every row alone fits)
            int b = a + 1, hi = n;
            while (b < hi) {
                const int mid = (b + hi + 1) >> 1;
                if (start[mid] - start[a] <= kRowSortMax) b = mid;
                else hi = mid - 1;
            }
            const int base = start[a], m = start[b] - base;
            for (int i0 = tid; i0 < m; i0 += U * kRowSortNT) {
                uint32_t k[U];
                int32_t c[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (i0 + u * kRowSortNT < m) k[u] = (uint32_t)__ldcs(src + base + i0 + u * kRowSortNT);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (i0 + u * kRowSortNT < m) c[u] = __ldg(cols + k[u]);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (i0 + u * kRowSortNT < m)
                        key[i0 + u * kRowSortNT] = (unsigned long long)(uint32_t)c[u] << 32 | k[u];
            }
            __syncthreads();
            for (int i = tid; i < m; i += kRowSortNT) {
                int lo = a, up = b - 1;  // the row of element i
                while (lo < up) {
                    const int mid = (lo + up + 1) >> 1;
                    if (start[mid] - base <= i) lo = mid;
                    else up = mid - 1;
                }
                const int s = start[lo] - base, t = start[lo + 1] - base;
                const unsigned long long mine = key[i];
                int at = s;
                for (int j = s; j < t; ++j) at += key[j] < mine;
                __stcs(col + base + at, (int32_t)(uint32_t)(mine >> 32));
                __stcs(src + base + at, (int32_t)(uint32_t)mine);
                if (rows_out) __stcs(rows_out + base + at, (int32_t)(r0 + lo));
            }
            __syncthreads();
            a = b;
        }
    }
}

// val[i] = vals[src[i]].  After k_trip_rows and not in it: there the gathers
// of the columns and of the values would evict each other from L2.
__global__ void __launch_bounds__(256) k_trip_vals(const int32_t* __restrict__ src, const double* __restrict__ vals,
                                                   long long nnz, double* __restrict__ val) {
    constexpr int U = kTripU;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long k0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; k0 < nnz; k0 += U * step) {
        uint32_t at[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u * step < nnz) at[u] = (uint32_t)__ldcs(src + k0 + u * step);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u * step < nnz) v[u] = __ldg(vals + at[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u * step < nnz) __stcs(val + k0 + u * step, v[u]);
    }
}

__global__ void k_trip_pack(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols, long long nnz,
                            unsigned long long* __restrict__ keys, int32_t* __restrict__ src) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += stride) {
        keys[k] = ((unsigned long long)(uint32_t)rows[k] << 32) | (uint32_t)cols[k];
        src[k] = (int32_t)k;
    }
}

__device__ __forceinline__ int digit_of(unsigned long long key, int shift) { return (int)(key >> shift) & 0xff; }

// Digit counts of one tile: tab[1 + d * tiles + tile] (tab[0] = 0 is the
// leading zero of the exclusive offsets).
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const unsigned long long* __restrict__ keys, long long n,
                                                             int shift, int32_t* __restrict__ tab, int tiles) {
    __shared__ int h[kRadixBins];
    const int lane = threadIdx.x & 31;
    h[threadIdx.x] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int r = 0; r < kSortRounds; ++r) {
        const long long k = base + (long long)r * kSortThreads + threadIdx.x;
        const bool in = k < n;
        const int d = in ? digit_of(keys[k], shift) : 0x100 | lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (in && lane == __ffs(peers) - 1) atomicAdd(&h[d & (kRadixBins - 1)], __popc(peers));
    }
    __syncthreads();
    tab[1 + (long long)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x == 0) tab[0] = 0;
}

// Stable scatter of one tile.  Warp w owns items [base + 512 w, base + 512 (w+1))
// in rounds of 32 consecutive items, so (warp, round, lane) order is the
// items' order; an item's place is the (digit, tile) offset + the same-digit
// items of earlier warps + of earlier rounds of its warp + of lower lanes.
__global__ void __launch_bounds__(kSortThreads, 3) k_radix_scatter(const unsigned long long* __restrict__ keys_in,
                                                                const int32_t* __restrict__ src_in, long long n,
                                                                int shift, const int32_t* __restrict__ tab, int tiles,
                                                                unsigned long long* __restrict__ keys_out,
                                                                int32_t* __restrict__ src_out) {
    __shared__ int wc[kSortWarps][kRadixBins];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < kSortWarps; ++i) wc[i][threadIdx.x] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kSortTile + (long long)w * kWarpItems;
    unsigned long long key[kSortRounds];
    int32_t src[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const long long k = base + r * 32 + lane;
        const bool in = k < n;
        key[r] = in ? keys_in[k] : 0ull;
        src[r] = in ? src_in[k] : 0;
        const int d = in ? digit_of(key[r], shift) : 0x100 | lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (in && lane == __ffs(peers) - 1) wc[w][d & (kRadixBins - 1)] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        const int d = threadIdx.x;
        int run = tab[(long long)d * tiles + blockIdx.x];
#pragma unroll
        for (int i = 0; i < kSortWarps; ++i) {
            const int c = wc[i][d];
            wc[i][d] = run;
            run += c;
        }
    }
    __syncthreads();
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const long long k = base + r * 32 + lane;
        const bool in = k < n;
        const int d = in ? digit_of(key[r], shift) : 0x100 | lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int dd = d & (kRadixBins - 1);  // == d for items in range
        const int at = in ? wc[w][dd] + __popc(peers & lt) : 0;
        __syncwarp();
        if (in && lane == __ffs(peers) - 1) wc[w][dd] += __popc(peers);
        __syncwarp();
        if (in) {
            keys_out[at] = key[r];
            src_out[at] = src[r];
        }
    }
}

__global__ void k_trip_gather(const unsigned long long* __restrict__ keys, const int32_t* src, const double* vals,
                              long long nnz, int32_t* __restrict__ col, double* __restrict__ val, int32_t* rows_out) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += stride) {
        const unsigned long long key = keys[k];
        const int32_t s = src[k];
        col[k] = (int32_t)(uint32_t)key;
        val[k] = vals[s];
        if (rows_out) rows_out[k] = (int32_t)(key >> 32);  // may alias src: same k, read above
    }
}

int bits_for(long long extent) {
    int b = 0;
    while (b < 32 && (1LL << b) < extent) ++b;
    return b;
}

int stream_grid(long long n, int sm_count) {
    long long b = (n + 255) / 256;
    const long long cap = (long long)sm_count * 8;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

}  // namespace

cudaError_t launch_triplet_scan(const int32_t* rows, const int32_t* cols, long long nnz, int32_t nor, int32_t noc,
                                int32_t* cnt, int32_t* pos, TripletScan* flags, int sm_count, cudaStream_t st) {
    if (nnz <= 0) return cudaSuccess;
    k_trip_scan<<<stream_grid(nnz, sm_count), 256, 0, st>>>(rows, cols, nnz, nor, noc, cnt, pos, flags);
    return cudaGetLastError();
}

// k_trip_rows ranks an element against every key of its row, and a CTA takes
// kRowSortRows rows: measured 33 ps per compare of one CTA, where the radix sort
// takes some 40 us and 0.2 (row digits only) to 0.37 ns per entry.  So a CTA's
// compares are held to what the radix sort does meanwhile, and all of them to
// 1024 per entry (0.1 ns with the SMs busy).  Loads with rows
// of up to 4096 entries always here, and by this rule: 512 x 4096 entries 288
// and 1.0 ms, 2000 x 1000 18.6 and 0.88, 4096 x 4096 290 and 3.4, 1 M rows of 4
// around 512 of 1000 11.0 and 1.5; 100 000 x 300 stays here (6.1 ms).
bool triplet_rows_fit(int longest, const TripletWork* w, long long nnz) {
    const unsigned long long limit = (1ull << 20) + 4ull * (unsigned long long)nnz,
                             row = (unsigned long long)longest * (unsigned long long)longest;
    if (longest > kRowSortMax || row > limit) return false;
    if (!w) return row * kRowSortRows <= limit && longest <= 1024;
    return w->most <= limit && w->sum <= 1024ull * (unsigned long long)nnz;
}

cudaError_t launch_triplet_work(const int32_t* cnt, int32_t nor, TripletWork* out, int sm_count, cudaStream_t st) {
    const cudaError_t e = cudaMemsetAsync(out, 0, sizeof(TripletWork), st);
    if (e != cudaSuccess) return e;
    const long long ctas = ((long long)nor + 8 * kRowSortRows - 1) / (8 * kRowSortRows);
    k_trip_work<<<(int)(ctas < 4LL * sm_count ? ctas : 4LL * sm_count), 256, 0, st>>>(cnt, nor, out);
    return cudaGetLastError();
}

cudaError_t launch_triplet_rows(const int32_t* rows, const int32_t* cols, const double* vals, int32_t* pos,
                                long long nnz, const int32_t* row_start, int32_t nor, int32_t* src, int32_t* col,
                                double* val, bool rows_out, int sm_count, cudaStream_t st) {
    if (nnz <= 0) return cudaSuccess;
    k_trip_bucket<<<stream_grid((nnz + kTripU - 1) / kTripU, sm_count), 256, 0, st>>>(rows, pos, nnz, row_start, src);
    const long long ctas = ((long long)nor + kRowSortRows - 1) / kRowSortRows;
    // (the arrival numbers are done with: pos takes the sorted rows)
    k_trip_rows<<<(int)(ctas < 16LL * sm_count ? ctas : 16LL * sm_count), kRowSortNT, 0, st>>>(
        src, cols, row_start, nor, col, rows_out ? pos : nullptr);
    k_trip_vals<<<stream_grid((nnz + kTripU - 1) / kTripU, sm_count), 256, 0, st>>>(src, vals, nnz, val);
    return cudaGetLastError();
}

long long triplet_sort_table_elems(long long nnz) {
    const long long tiles = (nnz + kSortTile - 1) / kSortTile;
    return tiles * kRadixBins + 1;
}

int triplet_sort_passes(int32_t nor, int32_t noc, bool col_passes) {
    return (col_passes ? (bits_for(noc) + 7) / 8 : 0) + (bits_for(nor) + 7) / 8;
}

cudaError_t launch_triplet_sort(const int32_t* rows, const int32_t* cols, long long nnz, int32_t nor, int32_t noc,
                                bool col_passes, unsigned long long* keys_a, int32_t* src_a,
                                unsigned long long* keys_b, int32_t* src_b, int32_t* tab, int32_t* scan_scratch,
                                unsigned long long** keys_sorted, int32_t** src_sorted, int sm_count,
                                cudaStream_t st) {
    *keys_sorted = keys_a;
    *src_sorted = src_a;
    if (nnz <= 0) return cudaSuccess;
    k_trip_pack<<<stream_grid(nnz, sm_count), 256, 0, st>>>(rows, cols, nnz, keys_a, src_a);
    int shifts[8], np = 0;
    if (col_passes)
        for (int s = 0; s < bits_for(noc); s += 8) shifts[np++] = s;
    for (int s = 0; s < bits_for(nor); s += 8) shifts[np++] = 32 + s;
    unsigned long long *ki = keys_a, *ko = keys_b;
    int32_t *si = src_a, *so = src_b;
    for (int p = 0; p < np; ++p) {
        const cudaError_t e = launch_radix_pass(ki, si, nnz, shifts[p], tab, scan_scratch, ko, so, st);
        if (e != cudaSuccess) return e;
        unsigned long long* kt = ki;
        ki = ko;
        ko = kt;
        int32_t* t = si;
        si = so;
        so = t;
    }
    *keys_sorted = ki;
    *src_sorted = si;
    return cudaGetLastError();
}

cudaError_t launch_radix_pass(const unsigned long long* keys, const int32_t* src, long long n, int shift,
                              int32_t* tab, int32_t* scan_scratch, unsigned long long* keys_out, int32_t* src_out,
                              cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const long long tiles = (n + kSortTile - 1) / kSortTile;
    k_radix_hist<<<(unsigned)tiles, kSortThreads, 0, st>>>(keys, n, shift, tab, (int)tiles);
    const cudaError_t e = launch_inclusive_scan(tab + 1, tiles * kRadixBins, scan_scratch, st);
    if (e != cudaSuccess) return e;
    k_radix_scatter<<<(unsigned)tiles, kSortThreads, 0, st>>>(keys, src, n, shift, tab, (int)tiles, keys_out, src_out);
    return cudaGetLastError();
}

cudaError_t launch_triplet_gather(const unsigned long long* keys, const int32_t* src, const double* vals,
                                  long long nnz, int32_t* col, double* val, int32_t* rows_out, int sm_count,
                                  cudaStream_t st) {
    if (nnz <= 0) return cudaSuccess;
    k_trip_gather<<<stream_grid(nnz, sm_count), 256, 0, st>>>(keys, src, vals, nnz, col, val, rows_out);
    return cudaGetLastError();
}

}  // namespace pwmgpu
