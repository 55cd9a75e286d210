// internal.h -- declarations shared by the host side (pwmgpu.cpp) and the
// kernel translation units.  Not part of the public ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "pwmgpu.h"

namespace pwmgpu {

// Device CRS view (row_start[nor+1], col[nnz], val[nnz]; each array padded by
// kArrayPad elements past its end).
struct DevMatrix {
    int32_t nor = 0, noc = 0;
    long long nnz = 0;
    int32_t* row_start = nullptr;
    int32_t* col = nullptr;
    double* val = nullptr;
};

// Merge kernel modes (merge.cuh MergeMode): plain SpMV; a power step with its
// squared norm; a power step tracking only the largest magnitude key.
enum { kModeSpmv = 0, kModePower = 1, kModeScale = 2 };

// Largest clock64 interval any spin-wait may take before it reports
// PWMGPU_ERR_TIMEOUT (about 2 s at the 2.07 GHz maximum SM clock).
constexpr long long kWaitCycles = 4000000000LL;

// merge.cu
// Items per lane of a merge-path sub-tile (a sub-tile is 32 * kMliIpt merge
// items, one warp); the lane-interleaved storage is laid out for this size.
constexpr int kMliIpt = 12;

// Merge-path kernel configurations (value / vector / accumulation types).
enum { kCfgF64 = 0, kCfgF32 = 2, kCfgBF16 = 3 };
struct MergeGeom {
    int wm;    // merge items per sub-tile (one warp)
    int w;     // warps per CTA
    int smem;  // dynamic shared memory per CTA
    int occ;   // resident CTAs per SM
    int nt;    // threads per CTA
};

// Per-matrix plan of the merge-path kernel: sub-tile boundaries, metadata,
// row-end masks and the lane-interleaved column / FP64 value arrays.
// devmem.cpp: device blocks from the device's pool.  A block is ready on every
// stream when dev_alloc returns; dev_free waits for nothing, so the work that
// used the block has been synchronised before.
cudaError_t dev_alloc(void** out, size_t bytes);
void dev_free(void* p);
// Waits for all work on `device` (as cudaFree does), so that blocks whose users
// are not all known can be freed inside the scope.  Where the wait is refused
// (a stream is being captured, not relaxed), the scope's dev_free calls keep their blocks
// until a later scope's wait succeeds.
class DevIdle {
public:
    explicit DevIdle(int device);
    ~DevIdle();
    DevIdle(const DevIdle&) = delete;
    DevIdle& operator=(const DevIdle&) = delete;

private:
    bool refused_ = false;
};
// Bytes the current device's pool holds without using them.
size_t dev_idle_bytes();
// Device blocks of a build whose kernels may still be under way: they go back
// after a wait for the stream, one for all of them.
class Scratch {
public:
    explicit Scratch(cudaStream_t st) : st_(st) {}
    ~Scratch() { release(); }
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    template <typename T>
    cudaError_t alloc(T** p, size_t bytes) {
        *p = nullptr;
        if (n_ == kMost) return cudaErrorMemoryAllocation;
        const cudaError_t e = dev_alloc((void**)p, bytes);
        if (e == cudaSuccess) blocks_[n_++] = *p;
        else *p = nullptr;
        return e;
    }
    void release() {
        if (n_ == 0) return;
        (void)cudaStreamSynchronize(st_);
        while (n_ > 0) dev_free(blocks_[--n_]);
    }

private:
    static constexpr int kMost = 8;
    void* blocks_[kMost];
    int n_ = 0;
    cudaStream_t st_;
};
// A pinned host block: what a handle reads back from the device (a copy into
// pageable memory would wait for the stream by itself, some 8 us each).
constexpr size_t kPinnedBlock = 1024;
cudaError_t pinned_alloc(void** out);
void pinned_free(void* p);

struct MliPlan {
    int nsub = 0;
    int2* subc = nullptr;       // nsub + 1 merge coordinates (row, nonzero)
    int4* rec = nullptr;        // 2 x nsub: {rw0, kw0, rw1, kw1}, {first row, flags, base, nkw}
    uint16_t* masks = nullptr;  // nsub x 32 row-end masks
    int32_t* colp = nullptr;    // lane-interleaved column indices
    double* valp = nullptr;     // lane-interleaved FP64 values
    uint16_t* colp16 = nullptr; // or null: the same columns as offsets from the sub-tile's base (rec0.w)
    // fix-up runs with a carry to add: {first sub-tile t, completing sub-tile n, row r, 0},
    // ordered by t; run_pre[t] = runs whose first sub-tile is < t (nsub + 1 entries)
    int4* runs = nullptr;
    int* run_pre = nullptr;
    int nruns = 0;
};
long long mli_storage_elems(long long nnz, long long nsub);

// sell.cu: SELL-32 copy of a matrix for the FP32 / BF16 iterations (slices
// of 32 rows, column-major in the slice, 16-bit column offsets from
// 32 s - 32768, padding skipped); built when every column fits and the
// padding is within a quarter of the nonzeros.
struct SellPlan {
    int state = 0;  // 0: not built, 1: built, -1: the matrix does not fit the format
    int nslices = 0;
    long long stored = 0;        // padded elements
    int32_t* soff = nullptr;     // nslices + 1 element offsets
    uint16_t* col16 = nullptr;   // column - (32 s - 32768)
    float* val32 = nullptr;      // FP32 values (built on first use)
    void* valbf = nullptr;       // BF16 values (built on first use)
    double* npart = nullptr;     // per-CTA shares of ||y||^2
    void release();
};
int sell_grid(int nslices, int sm_count);
// Fill the launch-geometry caches (occupancies) of the merge and SELL kernels
// once, so that matrix builds on several host threads only read them.
void warm_launch_caches(int sm_count);
// Build the slices (first call) and the value array of the requested type
// from CRS arrays; 0 = built, 1 = the matrix does not fit (state -1), 2 = a
// CUDA error or no memory (state 0).
int sell_build(SellPlan& S, const int32_t* row_start, const int32_t* col, const double* val, int nor, long long nnz,
               bool bf16, int sm_count, cudaStream_t st);
// y = 2^e A x (e from nsq_in, or 0 when null) on FP32 vectors; with nsq_out,
// also *nsq_out = ||y||^2 (deterministic; counter zero between launches).
cudaError_t launch_sell_spmv(const SellPlan& S, bool bf16, const int32_t* row_start, int nor, const float* x, float* y,
                             const double* nsq_in, double* nsq_out, unsigned int* counter, int sm_count,
                             cudaStream_t st);

// diag.cu: diagonal slices (64 rows; per slot one column - row offset, a row
// mask and the rows' values) of a matrix whose entries lie on few diagonals;
// the FP64 SpMV and power steps, and the FP32 / BF16 ones, of stencils.
struct DiagPlan {
    int nslices = 0;             // 0: the matrix does not fit the layout
    long long elems = 0;         // stored elements (64 per slot)
    void* mem = nullptr;         // the allocation that rec .. val64 and npart lie in
    int2* rec = nullptr;         // per slice: {first slot, slots << 1 | some slot lacks rows}
    int32_t* offs = nullptr;     // per slot: column - row
    void* masks = nullptr;       // per slot: the rows of the slice that have an element
    double* val64 = nullptr;     // value of row 32 r + l of the slice at (slot * 32 + l) * 2 + r
    float* val32 = nullptr;      // the same in FP32 (made on first use)
    void* valbf = nullptr;       // the same in BF16 (made on first use)
    double* npart = nullptr;     // per-CTA shares of ||y||^2
    void release();
};
// The slices of a CRS matrix, in two steps with a wait for the stream between
// them and, before the CRS arrays or the scratch go, after them: the kernels of
// diag_count leave what they find in `found`, pinned host memory.  0 = on the
// way, 1 = the matrix does not fit (D stays empty), 2 = a CUDA error or no
// memory (D stays empty).
struct DiagFound {
    unsigned long long total;  // slots
    int flag, pad;             // flag: a slice has more than it may
};
struct DiagBuild {
    unsigned char* tmp = nullptr;
    int nslices = 0;
};
int diag_count(DiagBuild& B, const int32_t* row_start, const int32_t* col, int nor, long long nnz, int sm_count,
               Scratch& scratch, DiagFound* found, cudaStream_t st);
int diag_fill(DiagPlan& D, const DiagBuild& B, const DiagFound& found, const int32_t* row_start, const int32_t* col,
              const double* val, int nor, long long nnz, int sm_count, cudaStream_t st);
// The values in FP32 / BF16, made on first use and complete on return (the
// stream is synchronised: not inside a capture).  0, or 2 as diag_fill.
int diag_low_values(DiagPlan& D, bool bf16, int sm_count, cudaStream_t st);
// One pass over slices [c0, c1) (c1 < 0: all).  mode kModeSpmv: y = A x;
// kModePower: y = 2^e A x and *nsq_out = ||y||^2 (when given; counter zero
// between launches); kModeScale: y = 2^e A x and atomicMax(*mx_out) of y's
// magnitude keys.  e from *mx_in, else *nsq_in, else 0.
struct SliceStep {
    const unsigned int* mx_in = nullptr;
    const double* nsq_in = nullptr;
    unsigned int* mx_out = nullptr;
    unsigned int* counter = nullptr;
    double* nsq_out = nullptr;
    int c0 = 0, c1 = -1;
    bool pdl = true;
};
cudaError_t launch_diag_spmv(const DiagPlan& D, int cfg, int mode, int nor, const void* x, void* y,
                             const SliceStep& s, int sm_count, cudaStream_t st);
// Pipelined host-array SpMV: out[p] = the largest column the slices of chunks
// 0..p read (slices [0, nslices (p + 1) / K)).
cudaError_t launch_diag_maxcol(const DiagPlan& D, int nor, int noc, int K, int* out, cudaStream_t st);
int diag_slice_rows();
void diag_warm_launch_caches();

// rows.cu: rows sorted by length within windows of consecutive rows, in items
// of 32, 8 or 1 rows (a warp each); no carries.
struct RowsPlan {
    int nitems = 0;              // 0: the matrix does not fit the layout
    int windows = 0, wrows = 0;  // windows of wrows rows
    int win[17] = {};            // first item of each window (then nitems)
    long long elems = 0;         // stored elements (64 per unit)
    void* mem = nullptr;         // the allocation that rec .. val64 and npart lie in
    int4* rec = nullptr;         // per item: {first unit, units, first row in perm, log2 lanes per row << 8 | rows}
    int32_t* perm = nullptr;     // the rows in item order
    int32_t* col = nullptr;      // columns, -1: absent
    double* val64 = nullptr;
    float* val32 = nullptr;      // the same in FP32 (made on first use)
    void* valbf = nullptr;       // the same in BF16 (made on first use)
    double* npart = nullptr;     // per-CTA shares of ||y||^2
    void release();
};
// pinned: kPinnedBlock bytes.  0 = on the way (the CRS arrays and the scratch
// are in use until the stream has been waited for), 1 = the matrix does not fit, 2 = a CUDA error or no
// memory (R stays empty).
int rows_build(RowsPlan& R, const int32_t* row_start, const int32_t* col, const double* val, int nor, long long nnz,
               bool narrow, int sm_count, Scratch& keep, void* pinned, cudaStream_t st);
// As diag_low_values.
int rows_low_values(RowsPlan& R, bool bf16, int sm_count, cudaStream_t st);
// Pipelined host-array SpMV: out[w] = the largest column of windows 0 .. w.
cudaError_t launch_rows_maxcol(const RowsPlan& R, int* out, cudaStream_t st);
// As launch_diag_spmv, over items [s.c0, s.c1).
cudaError_t launch_rows_spmv(const RowsPlan& R, int cfg, int mode, const void* x, void* y, const SliceStep& s,
                             cudaStream_t st);

// l1: launch variant of the merge kernels.  Bit 0: 0 = most resident CTAs,
// 1 = a smaller shared-memory carveout, more L1 for irregular gathers; bit 1:
// stream the plan's 16-bit column offsets (set only when the plan has them);
// bit 2: the FP64 SpMV's x gathers bypass L1 (the persistent and the
// low-precision kernels ignore it).
MergeGeom merge_geometry(int cfg, int l1 = 0);
int merge_grid(int cfg, int nsub, int sm_count, int l1 = 0);
int fixup_grid(int num_tiles, int sm_count);
int dot_grid(long long n, int sm_count);
// Persistent power-method kernel (cooperative launch): grid size for a
// matrix with nsub sub-tiles, 0 if the kernel cannot be made co-resident.
int power_persistent_grid(int cfg, int nsub, int sm_count, int l1 = 0);
// Iterations k0 .. k0+nk-1 on X/Y (ping-pong; v_k in X for even k), nsq[k]
// = ||v_k||^2 (nsq[k0] read when k0 > 0), result (5 doubles, or null):
// {lambda, residual^2, ||v_k||^2, v_k.v_{k+1}, e_k} of the last iteration.
// partials: 2 doubles per CTA; barrier: 2 words (zeroed here).
// wait: the grid barrier's budget (clock64 cycles) before it records
// PWMGPU_ERR_TIMEOUT, and extra arrivals it waits for beyond the grid (0;
// pwmgpu_test_grid_wait sets 1 to make every barrier run out of budget).
struct GridWait {
    long long cycles;
    unsigned int extra;
};
// mxk: k0 + nk + 1 zeroed words (or null): iterations before the last two
// of the launch track only the iterate's largest magnitude key (mxk[k+1]) for
// the rescale instead of summing ||v||^2 (nsq[k+1] is then not written).
cudaError_t launch_power_persistent(int cfg, const DevMatrix& M, const void* valp, const MliPlan& P, int grid,
                                    void* X, void* Y, void* carries, int k0, int nk, double* nsq, double* result,
                                    double* partials, unsigned int* barrier, int* status, cudaStream_t st,
                                    int l1, GridWait wait, unsigned int* mxk = nullptr);
cudaError_t launch_merge_partition(const int32_t* row_start, int nor, long long nnz, long long ipt, int parts,
                                   int2* out, cudaStream_t st);
cudaError_t launch_mli_plan(const int32_t* row_start, const int32_t* col, const double* val, const MliPlan& P,
                            int sm_count, cudaStream_t st);
cudaError_t launch_mli_convert(const MliPlan& P, int cfg, void* out, int sm_count, cudaStream_t st);
// the separate-kernel form of a solve chunk: FP32 norm pass and the result pass
cudaError_t launch_power_norm_f32(const float* y, const float* x, int n, double* partials, unsigned int* counter,
                                  double* out, int grid, cudaStream_t st);
cudaError_t launch_solve_result(bool f32, const void* in, const void* out, int n, const double* nsq_k,
                                const double* nd, double* nsq_next, double* result, double* partials,
                                unsigned int* counter, int grid, cudaStream_t st);
// fix-up run descriptors of a plan (P.runs, P.run_pre, P.nruns), counted and
// filled with a wait for the stream between (`found`: pinned) and before the
// scratch goes; 0, or 1 where they cannot be made
int fix_runs_count(MliPlan& P, const int32_t* row_start, int nor, int4** desc, Scratch& scratch, int* found,
                   cudaStream_t st);
int fix_runs_fill(MliPlan& P, const int4* desc, int found, cudaStream_t st);
// and the fix-up over descriptors [k0, k1)
cudaError_t launch_fix_runs_f64(int mode, const MliPlan& P, int k0, int k1, double* y, const double* carries,
                                const double* nsq_in, cudaStream_t st);
cudaError_t launch_fix_runs_f32(int mode, const MliPlan& P, int k0, int k1, float* y, const float* carries,
                                const double* nsq_in, cudaStream_t st);
// ||y||^2 of a power step inside its kernels: the MODE_POWER SpMV launched
// with `npart` writes one share per CTA (spmv_grid of them), this fix-up over
// all runs adds one per CTA after them and its last CTA writes the ordered
// total to *nsq_out.  npart holds power_norm_parts(P, spmv_grid) doubles;
// counter is zero between launches.
int power_norm_parts(const MliPlan& P, int spmv_grid);
// mx_in (optional): the step's rescale from its input's largest magnitude key
// instead of nsq_in.
cudaError_t launch_fix_runs_norm(bool f32, const MliPlan& P, void* y, const void* carries, const double* nsq_in,
                                 double* npart, int spmv_grid, unsigned int* counter, double* nsq_out,
                                 cudaStream_t st, const unsigned int* mx_in = nullptr);
// The fix-up of a MODE_SCALE step: carries times 2^e (e from *mx_in, else
// from *nsq_in, else 0 -- the same source as the step's SpMV), and atomicMax
// of the fixed rows' magnitude keys into *mx_out.
cudaError_t launch_fix_runs_scale(bool f32, const MliPlan& P, void* y, const void* carries, const double* nsq_in,
                                  const unsigned int* mx_in, unsigned int* mx_out, cudaStream_t st);
cudaError_t launch_mli_colspan(const MliPlan& P, int* cbase, int* flag, int sm_count, cudaStream_t st);
cudaError_t launch_mli_col16(const MliPlan& P, const int* cbase, int sm_count, cudaStream_t st);
cudaError_t launch_mli_unpermute(const MliPlan& P, int32_t* col, double* val, int sm_count, cudaStream_t st);
// mode kModeScale: mx_in (or nsq_in, or neither: e = 0) sets the rescale,
// the stored rows' magnitude keys go to atomicMax(*mx_out); kModePower may
// take its rescale from mx_in as well.
cudaError_t launch_merge_spmv(int cfg, int mode, const DevMatrix& M, const void* valp, const MliPlan& P, int grid,
                              const void* x, void* y, void* carries, const double* nsq_in, int* status,
                              cudaStream_t st, int l1 = 0, double* npart = nullptr,
                              const unsigned int* mx_in = nullptr, unsigned int* mx_out = nullptr);
// Carries of the merge SpMV into y (MODE_POWER: times the rescale factor of
// nsq_in).
cudaError_t launch_merge_fixup_f64(int mode, const DevMatrix& M, const int2* tiles, int num_tiles, double* y,
                                   const double* carries, const double* nsq_in, int fix_grid, cudaStream_t st);
cudaError_t launch_merge_fixup_f32(int mode, const DevMatrix& M, const int2* tiles, int num_tiles, float* y,
                                   const float* carries, const double* nsq_in, int fix_grid, cudaStream_t st);
// out[0] = ||y||^2 and, when x is given, out[1] = x . y (deterministic;
// partials: 2 per CTA of `grid`; counter zero between launches).
cudaError_t launch_power_norm_f64(const double* y, const double* x, int n, double* partials, unsigned int* counter,
                                  double* out, int grid, cudaStream_t st);
cudaError_t launch_power_finalize_f64(double* last, const double* nsq_last, double* prev, const double* nsq_prev,
                                      int n, int sm_count, cudaStream_t st);
// Rows [first_row, last_row) of the Poisson matrix (last_row < 0: all m*n).
cudaError_t launch_poisson_crs(int m, int n, int32_t* row_start, int32_t* col, double* val, int sm_count,
                               cudaStream_t st, int first_row = 0, int last_row = -1);
long long poisson_rows_nnz(int m, int n, int first_row, int last_row);
cudaError_t launch_dot2_f64(const double* a, const double* b, int n, double* partials, unsigned int* counter,
                            double* out, int grid, cudaStream_t st);
cudaError_t launch_dot2_f32(const float* a, const float* b, int n, double* partials, unsigned int* counter,
                            double* out, int grid, cudaStream_t st);
cudaError_t launch_resid_f64(const double* a, double sa, const double* b, double sb, int n, double* partials,
                             unsigned int* counter, double* out, int grid, cudaStream_t st);
cudaError_t launch_resid_f32(const float* a, double sa, const float* b, double sb, int n, double* partials,
                             unsigned int* counter, double* out, int grid, cudaStream_t st);
cudaError_t launch_convert_f64_f32(const double* s, float* d, long long n, int sm_count, cudaStream_t st);
cudaError_t launch_convert_f32_f64(const float* s, double* d, long long n, int sm_count, cudaStream_t st);
cudaError_t launch_convert_f64_bf16(const double* s, void* d, long long n, int sm_count, cudaStream_t st);
cudaError_t launch_bf16_exact(const double* v, long long n, int* flag, int sm_count, cudaStream_t st);

// gen.cu: seeded random sparse matrices and an in-place int32 inclusive scan
void random_length_table(int kind, double mean, double sigma, int max_len, std::vector<uint64_t>& thr);
cudaError_t launch_random_count(const uint64_t* thr, int max_len, int n, uint64_t seed, int band_permille,
                                int band_half, int32_t* row_start, unsigned long long* total, int sm_count,
                                cudaStream_t st);
cudaError_t launch_random_fill(const uint64_t* thr, int max_len, int n, uint64_t seed, int band_permille,
                               int band_half, const int32_t* row_start, int32_t* col, double* val, int sm_count,
                               cudaStream_t st);
long long scan_scratch_elems(long long n);
cudaError_t launch_inclusive_scan(int32_t* a, long long n, int32_t* scratch, cudaStream_t st);

// triplet.cu: triplet -> CRS on the device (rows bucketed and sorted in shared
// memory, or a stable LSD radix sort by (row, col))
struct TripletScan {
    unsigned long long bad;   // first entry with a row or column out of range (~0 when none)
    unsigned int unsorted_rc; // input not sorted by (row, col)
    unsigned int unsorted_c;  // input not sorted by column
    int longest;              // entries of the longest row
    int pad;
};
cudaError_t launch_triplet_scan(const int32_t* rows, const int32_t* cols, long long nnz, int32_t nor, int32_t noc,
                                int32_t* cnt, int32_t* pos, TripletScan* flags, int sm_count, cudaStream_t st);
// The work of launch_triplet_rows on rows of these lengths.
struct TripletWork {
    unsigned long long sum, most;  // sums of squared row lengths: all rows', and the largest of a CTA's rows
};
// cnt: the row lengths.
cudaError_t launch_triplet_work(const int32_t* cnt, int32_t nor, TripletWork* out, int sm_count, cudaStream_t st);
// Whether launch_triplet_rows sorts the rows no slower than the radix sort (w
// null: from the longest row alone; false then means perhaps).
bool triplet_rows_fit(int longest, const TripletWork* w, long long nnz);
// CRS from the row starts and the scan's arrival numbers pos (which receive the
// sorted rows with rows_out); src: nnz words of scratch.
cudaError_t launch_triplet_rows(const int32_t* rows, const int32_t* cols, const double* vals, int32_t* pos,
                                long long nnz, const int32_t* row_start, int32_t nor, int32_t* src, int32_t* col,
                                double* val, bool rows_out, int sm_count, cudaStream_t st);
// One stable pass of the radix sort by the keys' byte at `shift` (tab:
// triplet_sort_table_elems(n) words, scan_scratch for as many).
cudaError_t launch_radix_pass(const unsigned long long* keys, const int32_t* src, long long n, int shift,
                              int32_t* tab, int32_t* scan_scratch, unsigned long long* keys_out, int32_t* src_out,
                              cudaStream_t st);
long long triplet_sort_table_elems(long long nnz);
int triplet_sort_passes(int32_t nor, int32_t noc, bool col_passes);
cudaError_t launch_triplet_sort(const int32_t* rows, const int32_t* cols, long long nnz, int32_t nor, int32_t noc,
                                bool col_passes, unsigned long long* keys_a, int32_t* src_a,
                                unsigned long long* keys_b, int32_t* src_b, int32_t* tab, int32_t* scan_scratch,
                                unsigned long long** keys_sorted, int32_t** src_sorted, int sm_count,
                                cudaStream_t st);
cudaError_t launch_triplet_gather(const unsigned long long* keys, const int32_t* src, const double* vals,
                                  long long nnz, int32_t* col, double* val, int32_t* rows_out, int sm_count,
                                  cudaStream_t st);

// stats.cu: Util_Scripts/calc_stats.cpp figures on the device
struct StatsDev {
    double rows_var, block_avg, block_var;
    int max_row_nnz, balanced;
};
int stats_row_ctas(int n);
cudaError_t launch_matrix_stats(const int32_t* row_start, const int32_t* col, int n, double avg, int bits, int nbw,
                                unsigned int* blocks, long long* brow, double* row_partials, double* blk_partials,
                                StatsDev* out, cudaStream_t st);

// hostcopy.cu: SM-driven copy between pageable host memory and the device
// (only where the device reaches pageable memory)
cudaError_t launch_host_copy(const double* src, double* dst, long long n, cudaStream_t st);

// batch.cu: one round (`steps` power steps + the residual pass) of every slot
// of a class table; seeded uniform start vectors
struct BatchTable;
void batch_prepare(int sm_count);
// layout of the class's slots: merge path, SELL-32 copies (FP32 / BF16
// values) or diagonal slices.
enum { kBatchMerge = 0, kBatchSell = 1, kBatchDiag = 2 };
cudaError_t launch_batch_round(int cfg, const BatchTable* T, int steps, int sm_count, cudaStream_t st, int layout);
// batch_diag.cu: step `it` of a round of a diagonal-slice class
void batch_diag_prepare(int sm_count);
cudaError_t launch_batch_diag(int cfg, const BatchTable* T, int it, bool keys, bool from_key, int sm_count,
                              cudaStream_t st);
cudaError_t launch_tile_slots(const BatchTable* T, int nslots, cudaStream_t st);
cudaError_t launch_fill_uniform(double* x, int n, uint64_t seed, int sm_count, cudaStream_t st);

// The tile kernel (k_csb_spmv) runs both blocked formats: rows in windows of
// S, each window's tiles ("units", elements of one block in an S-column
// window) from a list; tiles of at least kTileDenseUnit elements stage their
// x window in shared memory, the rest are merged into one gathered unit.
constexpr int kTileDenseUnit = 256;

// csb.cu: CSB (CSB.hpp) parameters, host build and SpMV
void csb_params(int nor, int noc, int* beta, int* bits);
int csb_window(int nor, int beta, int sm_count);
int csb_build_host(int nor, int noc, long long nnz, const int32_t* row_start, const int32_t* col, const double* val,
                   int beta, int bits, std::vector<uint32_t>& ind, std::vector<double>& data,
                   std::vector<int32_t>& blk_ptr, int S, std::vector<int>& win_ptr, std::vector<int>& unit_data);
bool csb_kernel_layout(const std::vector<uint32_t>& ind, const std::vector<double>& data, int S,
                       std::vector<int>& win_ptr, std::vector<int>& units, std::vector<uint32_t>& kind,
                       std::vector<double>& kdata, std::vector<int32_t>& kcol);
cudaError_t launch_csb_spmv(const uint32_t* ind, const int32_t* kcol, const double* data, const int* win_ptr, const int* units, int nwin,
                            int S, int nor, int noc, const double* x, double* y, const double* nsq_in, int* status,
                            int sm_count, cudaStream_t st, int variant = 0);
constexpr int kCsbVariants = 4;

// coh.cu: CO-H (BlockCOH.hpp) host build and SpMV
int coh_build_host(int nor, int noc, long long nnz, const int32_t* row_start, const int32_t* col, const double* val,
                   int threads, std::vector<int32_t>& part_info, std::vector<uint16_t>& row_jump,
                   std::vector<uint16_t>& col_jump, std::vector<double>& data, std::vector<int32_t>& block_nnz,
                   std::vector<int16_t>& row_jump_block, std::vector<int16_t>& col_jump_block,
                   std::vector<int>& parts, std::vector<int>& blocks);
// The CO-H matrix as tiles for the tile kernel: per window of S rows, the
// tiles of its rows' CO-H blocks -- partitions in row order, each
// partition's blocks in its Hilbert order, a block's tiles by column window
// -- with elements row-major inside a tile (columns ascending per row, as
// in the block's ICRS order).  Outputs as csb_build_host's (ind = local row
// << 16 | column - tile column, win_ptr: sparse tiles then dense ones).
// parts: 8 ints per partition as coh_build_host writes them.
void coh_tile_units(int nor, int noc, long long nnz, const int32_t* row_start, const int32_t* col, const double* val,
                    const std::vector<int>& parts, int S, std::vector<uint32_t>& ind, std::vector<double>& data,
                    std::vector<int>& win_ptr, std::vector<int>& unit_data);

// Pipelined host-array SpMV: chunk records (4 ints per chunk: first
// sub-tile, its first row, row-split flag, largest column read), and the
// SpMV / fix-up over sub-tile ranges.
cudaError_t launch_pipeline_plan(const int32_t* row_start, const MliPlan& P, int K, int* out, cudaStream_t st);
cudaError_t launch_merge_spmv_range(const DevMatrix& M, const MliPlan& P, int t0, int t1, int grid, const double* x,
                                    double* y, double* carries, int* status, cudaStream_t st, int l1);
cudaError_t launch_merge_fixup_range(const DevMatrix& M, const int2* tiles, int num_tiles, int f0, int f1, double* y,
                                     const double* carries, cudaStream_t st, int sm_count);

// Record the calling thread's last error message (pwmgpu_last_error).
void record_error(const char* msg);

// Poisson row start closed form (shared with the host checker of the
// device generator).
long long poisson_row_start_host(long long row, long long m, long long n);

}  // namespace pwmgpu
