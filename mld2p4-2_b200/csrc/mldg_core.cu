// mldg_core.cu -- handle, upload, finalize, V-cycle recorder, apply, Krylov.
//
// The V-cycle follows mld_d_inner_mult (mlprec/impl/mld_dmlprec_aply.f90:590-809,
// ml_cycle = VCYCLE) level by level; smoothers follow
// mld_d_jac_smoother_apply_vect.f90:107-177 with the diag solver (:102 of
// mld_d_diag_solver_apply_vect.f90) or the ILU solver
// (mld_d_ilu_solver_apply_vect.f90:130-142).  All device memory is allocated
// in mldg_finalize; an apply only launches kernels (optionally replayed from a
// CUDA graph captured on first use).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <chrono>
#include <cmath>
#include <map>
#include <set>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include <omp.h>

#include "mldg.h"
#include "mldg_kernels.cuh"
#include "mldg_multi.cuh"
#include "mldg_tri.h"
#include "mldg_trigrp.h"
#include "mldg_trsv_win.cuh"
#include "mldg_trsv_rep.cuh"
#include "mldg_trsv_blk.cuh"
#include "mldg_trsv_grp.cuh"
#include "mldg_ilu0.cuh"
#include "mldg_spgemm.cuh"
#include "mldg_spmv_stg.cuh"

namespace mldg {

// ---------------------------------------------------------------------------
struct Error {
  int code;
  std::string msg;
};

#define MLDG_CUDA(call)                                                              \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess)                                                           \
      throw Error{MLDG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)}; \
  } while (0)

static void fail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  throw Error{code, buf};
}

struct HostCSR {
  int nr = 0, nc = 0;
  std::vector<int> irp, ja;
  std::vector<double> val;
  bool present() const { return !irp.empty(); }
  int64_t nnz() const { return irp.empty() ? 0 : irp[nr]; }
};

static HostCSR copy_csr(const mldg_csr &c, int base, const char *what, int lev) {
  HostCSR h;
  if (!c.irp) return h;
  if (c.nrows < 0 || c.ncols < 0) fail(MLDG_ERR_ARG, "level %d %s: negative size", lev, what);
  h.nr = c.nrows;
  h.nc = c.ncols;
  h.irp.resize((size_t)h.nr + 1);
  for (int i = 0; i <= h.nr; ++i) h.irp[i] = c.irp[i] - base;
  if (h.irp[0] != 0) fail(MLDG_ERR_ARG, "level %d %s: irp[0] != base", lev, what);
  for (int i = 0; i < h.nr; ++i)
    if (h.irp[i + 1] < h.irp[i]) fail(MLDG_ERR_ARG, "level %d %s: irp not monotone", lev, what);
  const int64_t nnz = h.irp[h.nr];
  if (nnz > 0 && (!c.ja || !c.val)) fail(MLDG_ERR_ARG, "level %d %s: missing ja/val", lev, what);
  h.ja.resize((size_t)nnz);
  h.val.assign(c.val, c.val + nnz);
  for (int64_t k = 0; k < nnz; ++k) {
    const int j = c.ja[k] - base;
    if (j < 0 || j >= h.nc) fail(MLDG_ERR_ARG, "level %d %s: column %d out of range", lev, what, j);
    h.ja[k] = j;
  }
  return h;
}

static HostCSR transpose(const HostCSR &a) {
  HostCSR t;
  t.nr = a.nc;
  t.nc = a.nr;
  t.irp.assign((size_t)t.nr + 1, 0);
  const int64_t nnz = a.nnz();
  t.ja.resize((size_t)nnz);
  t.val.resize((size_t)nnz);
  for (int64_t k = 0; k < nnz; ++k) t.irp[a.ja[k] + 1]++;
  for (int j = 0; j < t.nr; ++j) t.irp[j + 1] += t.irp[j];
  // rows of the transpose in source-row order (sorted columns): each thread
  // owns a contiguous block of source rows and fills from per-thread
  // starting offsets computed by a column-count prefix over the blocks
  const int nt = std::max(1, std::min(omp_get_max_threads(), a.nr / 4096 + 1));
  std::vector<std::vector<int>> cnt((size_t)nt);
#pragma omp parallel num_threads(nt)
  {
    const int tid = omp_get_thread_num();
    const int i0 = (int)((int64_t)a.nr * tid / nt), i1 = (int)((int64_t)a.nr * (tid + 1) / nt);
    std::vector<int> &c = cnt[(size_t)tid];
    c.assign((size_t)t.nr, 0);
    for (int i = i0; i < i1; ++i)
      for (int k = a.irp[i]; k < a.irp[i + 1]; ++k) c[a.ja[k]]++;
#pragma omp barrier
#pragma omp for schedule(static)
    for (int j = 0; j < t.nr; ++j) {
      int off = t.irp[j];
      for (int q = 0; q < nt; ++q) {
        const int v = cnt[(size_t)q][j];
        cnt[(size_t)q][j] = off;
        off += v;
      }
    }
    for (int i = i0; i < i1; ++i)
      for (int k = a.irp[i]; k < a.irp[i + 1]; ++k) {
        const int p = c[a.ja[k]]++;
        t.ja[p] = i;
        t.val[p] = a.val[k];
      }
  }
  return t;
}

struct HostLevel {
  bool uploaded = false;
  HostCSR A, P, R, ND, L, U;
  std::vector<double> d;
  int kind = MLDG_SMOOTHER_BJAC, sweeps_pre = 1, sweeps_post = 1;
  double damp = 1.0;
};

// Allocations of this thread until one fails on purpose, negative: none does
// (mldg_test_set_alloc_failure).
static thread_local int g_alloc_failure = -1;

// ---------------------------------------------------------------------------
// Device memory arena: everything lives until mldg_destroy.
struct Arena {
  std::vector<void *> ptrs;
  size_t bytes = 0;
  template <typename T>
  T *alloc(size_t n) {
    void *p = nullptr;
    if (n == 0) n = 1;
    // 64 bytes of slack past the end: the staged kernels' bulk copies widen
    // each slice to 16-byte boundaries (mldg_spmv_stg.cuh)
    const bool on_purpose = g_alloc_failure >= 0 && g_alloc_failure-- == 0;
    const cudaError_t e = on_purpose ? cudaErrorMemoryAllocation : cudaMalloc(&p, n * sizeof(T) + 64);
    if (e != cudaSuccess) {
      cudaGetLastError();  // the call reports it; the next call on the handle starts clean
      fail(MLDG_ERR_ALLOC, "cudaMalloc(%zu bytes): %s", n * sizeof(T), cudaGetErrorString(e));
    }
    ptrs.push_back(p);
    bytes += n * sizeof(T);
    return (T *)p;
  }
  template <typename T>
  T *upload(const T *v, size_t n) {
    T *p = alloc<T>(n);
    if (n) MLDG_CUDA(cudaMemcpy(p, v, n * sizeof(T), cudaMemcpyHostToDevice));
    return p;
  }
  template <typename T>
  T *upload(const std::vector<T> &v) {
    return upload(v.data(), v.size());
  }
  void release() { release_to({0, 0}); }
  // what is allocated after mark() is given back by release_to
  typedef std::pair<size_t, size_t> Mark;
  Mark mark() const { return {ptrs.size(), bytes}; }
  void release_to(Mark m) {
    for (size_t k = m.first; k < ptrs.size(); ++k) cudaFree(ptrs[k]);
    ptrs.resize(m.first);
    bytes = m.second;
  }
};

// Staged kernels (mldg_spmv_stg.cuh): dynamic shared memory opted in once
// per kernel (to the most a CTA may have) and the resident CTAs per SM
// cached per (kernel, size).  The engine fills
// the cache for every (kernel, size) its operators can launch before any
// stream capture (stg_prepare); a launch that misses it while its stream is
// being captured fails instead of configuring a kernel under capture.
template <typename K>
static int stg_occ(K kern, size_t smem, cudaStream_t st = nullptr) {
  static std::mutex mu;
  static std::map<std::pair<const void *, size_t>, int> occ;
  std::lock_guard<std::mutex> lk(mu);
  auto key = std::make_pair((const void *)kern, smem);
  auto it = occ.find(key);
  if (it != occ.end()) return it->second;
  if (st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    MLDG_CUDA(cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone) fail(MLDG_ERR_INTERNAL, "staged kernel not prepared before capture");
  }
  // the opt-in is one value per kernel: the largest any launch may ask for
  static std::set<const void *> opted;
  if (opted.insert((const void *)kern).second)
    MLDG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStgSmemMax));
  int per_sm = 0;
  MLDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kStgThreads, smem));
  occ[key] = per_sm;
  return per_sm;
}
// a persistent grid of (resident CTAs per SM) x SMs, at most one warp per tile
template <typename K, typename... Args>
static void stg_launch(K kern, size_t smem, int ntiles, int nsm, cudaStream_t st, Args... args) {
  const int per_sm = stg_occ(kern, smem, st);
  if (per_sm < 1) fail(MLDG_ERR_INTERNAL, "staged kernel does not fit (%zu bytes of shared memory)", smem);
  const int grid = std::max(1, std::min((ntiles + kStgWarps - 1) / kStgWarps, per_sm * nsm));
  kern<<<grid, kStgThreads, smem, st>>>(args...);
}

// Launch of a streaming kernel, with programmatic dependent launch when pdl
// is set: the kernel (which calls pdl_enter first) may be scheduled while
// the previous kernel in the stream finishes, so the gap between dependent
// launches of a V-cycle or a Krylov iteration shrinks.
template <typename... KArgs, typename... Args>
static void launch_k(bool pdl, void (*kern)(KArgs...), int grid, int block, cudaStream_t st, Args... args) {
  if (!pdl) {
    kern<<<grid, block, 0, st>>>(args...);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  MLDG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}

// Launch-shape choices kept in a file (MLDG_TUNE_FILE): finalize reads the
// choice of every operator (and of the Krylov SpMV) found there instead of
// timing it, and appends the ones it timed, so a later process (a profiler
// run, whose own timings are distorted) launches exactly the same kernels.
// One line per operator: "spmv <value bytes> <fp16 form> <level> <operator>
// <rows> <entries> <lanes per row> <format> <16-diagonal passes>", or "kry
// <rows> <entries> <lanes per row> <format>".
static std::map<std::string, std::array<int, 3>> tune_file_read() {
  std::map<std::string, std::array<int, 3>> m;
  const char *fn = std::getenv("MLDG_TUNE_FILE");
  if (!fn) return m;
  std::FILE *f = std::fopen(fn, "r");
  if (!f) return m;
  char line[256];
  while (std::fgets(line, sizeof line, f)) {
    char kind[8] = {};
    long long a[6] = {};
    int c[3] = {0, 0, 0};
    if (std::sscanf(line, "%7s", kind) != 1) continue;
    if (!std::strcmp(kind, "spmv") &&
        std::sscanf(line, "%*s %lld %lld %lld %lld %lld %lld %d %d %d", &a[0], &a[1], &a[2], &a[3], &a[4], &a[5], &c[0],
                    &c[1], &c[2]) == 9) {
      char key[128];
      std::snprintf(key, sizeof key, "spmv %lld %lld %lld %lld %lld %lld", a[0], a[1], a[2], a[3], a[4], a[5]);
      m[key] = {c[0], c[1], c[2]};
    } else if (!std::strcmp(kind, "kry") &&
               std::sscanf(line, "%*s %lld %lld %d %d", &a[0], &a[1], &c[0], &c[1]) == 4) {
      char key[128];
      std::snprintf(key, sizeof key, "kry %lld %lld", a[0], a[1]);
      m[key] = {c[0], c[1], 0};
    }
  }
  std::fclose(f);
  return m;
}
static void tune_file_append(const std::string &line) {
  const char *fn = std::getenv("MLDG_TUNE_FILE");
  if (!fn) return;
  if (std::FILE *f = std::fopen(fn, "a")) {
    std::fputs(line.c_str(), f);
    std::fputc('\n', f);
    std::fclose(f);
  }
}

template <typename T>
struct DCSR {
  int nr = 0, nc = 0;
  int64_t nnz = 0;
  int *irp = nullptr, *ja = nullptr;
  short *jd = nullptr;  // int16 column offsets from the row (square, |j - i| <= 32767), or null
  T *val = nullptr;
  int tpr = 1;
  // sliced-ELL copy (SELL-32, see k_spmv_sell): slice offsets, values and
  // column indices (int16 offsets from the row when jd is set, else int32),
  // built when the padding stays small; used when the autotuner finds it faster
  int *soff = nullptr;
  T *sval = nullptr;
  short *sjd = nullptr;
  int *sja = nullptr;
  int64_t slots = 0;
  // 0: CSR kernels; 1 or 2: SELL kernels with that many slices per warp
  // iteration; 3: the software-pipelined SELL kernels (k_spmv_sellp,
  // k_jacobi_sellp); 4: the staged SELL kernels (k_spmv_stg, k_jacobi_stg);
  // 5: the HDIA kernels (k_spmv_hdia, k_jacobi_hdia)
  int sell = 0;
  // hacked-diagonal copy (HDIA-32, see k_spmv_hdia) of a square operator:
  // per slice of 32 rows its ascending column offsets (hdoff from
  // hdptr[s]) and one value per (offset, row); values of type T, or FP16
  // row-scaled (hdhval) in the FP16 operator form; built when the slices
  // share few diagonals, used when the autotuner finds it faster
  int *hdptr = nullptr, *hdoff = nullptr;
  T *hdval = nullptr;
  __half *hdhval = nullptr;
  int64_t hdslots = 0;
  bool hdia() const { return sell == 5 && hdptr != nullptr; }
  bool hd16 = false;  // HDIA kernels with 16 diagonals' loads per pass (long rows) instead of 4
  int hd_nslice() const { return nslice(); }
  // staged SELL tiles (k_spmv_stg, k_jacobi_stg): packed blocks of
  // consecutive slices and their descriptors, the largest block tblock
  // bytes; used when sell == 4
  int4 *tiles = nullptr;
  uint4 *pk = nullptr;
  int ntiles = 0, tblock = 0;
  // FP16 operator form (float engines only): FP16 copies of val and sval
  // scaled by rows, a_ij = rs_i * h_ij with rs_i = max_j |a_ij| in FP32;
  // the single-vector SpMV and Jacobi kernels read these instead of val/sval
  __half *hval = nullptr, *shval = nullptr;
  float *rs = nullptr;
  bool present() const { return irp != nullptr; }
  bool h16() const { return rs != nullptr; }
  int64_t idx_bytes() const { return jd ? 2 : 4; }
  int64_t val_bytes() const { return h16() ? 2 : (int64_t)sizeof(T); }
  int64_t scale_bytes() const { return h16() ? 4 * (int64_t)nr : 0; }
  int nslice() const { return (nr + 31) / 32; }
  // bytes of the matrix as the chosen kernel reads it
  int64_t mat_bytes() const {
    if (hdia())
      return hdslots * val_bytes() + 4 * ((int64_t)hd_nslice() + 1) + 4 * (hdslots / 32) +
             scale_bytes();
    return ((sell >= 1 && sell <= 3) ? slots * (val_bytes() + idx_bytes()) + 4 * ((int64_t)nslice() + 1)
                 : nnz * (val_bytes() + idx_bytes()) + 4 * ((int64_t)nr + 1)) +
           scale_bytes();
  }
  // algorithmic bytes: CSR nnz*(value + index) + 4*(rows + 1) (+ the row
  // scales), or, for an operator that also has its HDIA copy, that copy's
  // compulsory bytes when fewer: one value per entry (no padding), the slice
  // pointers and offsets (+ the row scales)
  int64_t csr_bytes() const { return nnz * (val_bytes() + idx_bytes()) + 4 * ((int64_t)nr + 1) + scale_bytes(); }
  int64_t alg_bytes() const {
    const int64_t csr = csr_bytes();
    if (!hdptr) return csr;
    return std::min(csr, nnz * val_bytes() + 4 * ((int64_t)hd_nslice() + 1) +
                             4 * (hdslots / 32) + scale_bytes());
  }
};

template <typename T>
struct DTri {
  int n = 0, rev = 0, nlevels = 0;
  int64_t nnz = 0;
  int *lvl_ptr = nullptr, *prow = nullptr, *pirp = nullptr, *pja = nullptr;
  T *pval = nullptr;
  int *counters = nullptr;
  int nblk = 0;
  int2 *blk = nullptr;
  int tpr = 1, e = 4;
  int mode = 0;     // 0: staged single CTA, 1: single CTA, 2: sync-free
  StageCfg stg{};
  int4 *desc = nullptr;
  bool cta = true;  // single-CTA kernel (solution in shared memory) vs sync-free
  int threads = 512, grid = 1;
  size_t smem = 0;
  // host copy of the level schedule (transformed index space)
  std::vector<int> h_lvl, h_prow, h_pirp, h_pja;
  std::vector<double> h_pval;
  // multi-RHS sync-free solve (k_trsv_sf_m): level-aligned blocks of 32/K rows, per log2(K)
  int2 *blkm[6] = {};
  int nblkm[6] = {}, gridm[6] = {};
  // its ELL form (k_trsv_ell), per log2(K); ok = false falls back to k_trsv_sf_m
  struct Ell {
    bool ok = false, pf = false;
    int ntask = 0, npad = 0, E = 0, S = 1, grid = 0, backoff = 0;
    int *prow = nullptr, *ej = nullptr, *ovp = nullptr, *ovj = nullptr, *ctr = nullptr;
    int2 *toff = nullptr;
    T *ev = nullptr, *ovv = nullptr;
    int64_t slots = 0;  // entry slots stored (sum over tasks of slots per row x rows per task)
    unsigned long long *trace = nullptr;  // MLDG_ELL_TRACE: per-task timestamps
    std::vector<int> h_task_level;
  } ell[6];
  bool present() const { return prow != nullptr; }
};

// Plan of the windowed cluster solve (k_trsv_win) for one triangular factor.
template <typename T>
struct DWin {
  int n = 0, nsteps = 0, W = 0, wshift = 0, C = 1, D = 4, capR = 0, capE = 0, tpr = 1;
  int off_win = 0, off_desc = 0, off_bar = 0, off_ring = 0, stage_bytes = 0;
  size_t smem = 0;
  int64_t nnz = 0;
  WinDesc *desc = nullptr;
  int *orig = nullptr, *pirp = nullptr, *pja = nullptr;
  T *pval = nullptr;
  int *nextpos = nullptr;  // feed of the following solve of the pair
  T *nextscale = nullptr;
  unsigned long long *trace = nullptr;  // MLDG_WIN_TRACE: per-phase cycle counters
  std::vector<int> h_orig, h_pos;  // position -> original row, original row -> position
  std::vector<WinDesc> h_desc;
  bool ok = false;
};

// Plan of the replicated-window cluster solve (k_trsv_rep) for one triangular
// factor: per CTA and step one block (row descriptors, ring slots and values of
// the entries, far entries), its descriptor, and the position maps.
template <typename T>
struct DRep {
  bool ok = false, linked = false;
  int n = 0, nsteps = 0, C = 8, R = 0, capB = 0, stage_bytes = 0, ring_bytes = 0;
  size_t smem = 0;
  int64_t nnz = 0, nfar = 0, block_bytes = 0;
  int4 *desc = nullptr;
  uint4 *blocks = nullptr;
  T *xp = nullptr;    // position-ordered solution for far readers
  int *orig = nullptr;
  unsigned long long *trace = nullptr;  // MLDG_REP_TRACE: per-phase cycle counters
  std::vector<int> h_orig, h_pos;  // position -> original row, original row -> position
  std::vector<int> h_tail_ptr, h_tail;
  // host schedule, released once the blocks are built
  std::vector<int> step_ptr;       // nsteps + 1 first positions
  std::vector<int> pirp, dep;      // entries in position order, dependency positions
  std::vector<double> val;
  std::vector<unsigned char> cls;  // per entry: 0 previous step, 3 two to kRepG steps back, 1 older (ring), 2 far
  int *vbytes = nullptr;           // per step: bytes of its values (every row, one T each)
  int *tail_ptr = nullptr, *tail = nullptr;  // far-copy positions reset after the last step, per CTA
  std::vector<int> rst_step;       // per position read by a far entry: the step that resets its copy
  std::vector<unsigned char> feeds;  // per position: read by a far entry
};
constexpr int kRepTPR = 4;

// Plan of the partitioned solve (k_trsv_blk) for one triangular factor.
template <typename T>
struct DBlk {
  bool ok = false;
  int n = 0, nblocks = 0, nsteps = 0, W = 0, stage_bytes = 0, aux_cap = 0;
  size_t smem = 0;
  int64_t nnz = 0, plan_bytes = 0;
  int *bstep = nullptr;
  int2 *sdesc = nullptr;
  uint4 *plan = nullptr;
  int *ticket = nullptr;
};

// Grouped solve: entries of V and W per group, entries of a row, the bound on a
// row of W, and the widest block of columns of a narrow level.  A group's
// entries should stream in about the time of its hand-off, which takes longer
// the more warps take part: n/5 entries between these limits (solve pair at idim=40, 64,000 rows:
// 86 us with 50,000 and 100,000, 98 us with 200,000; idim=101, 1,030,301 rows:
// 333 us with 200,000, 408 us with 100,000).  Blocks above eight columns
// move 16 or 32 values an entry, so a group holds fewer entries, and levels of
// short rows (at most kGrpWide entries) keep the ELL solve (32 columns at
// idim=64: level 0, 3 entries a row: 250 us a solve, ELL 178; level 1, 14 entries:
// 304 us, ELL 345).
constexpr int64_t kGrpBudgetMin = 50000, kGrpBudgetMax = 200000;
constexpr int kGrpRow = 512;
constexpr double kGrpGrowth = 64.0;
constexpr int kGrpCols = 8, kGrpWide = 8;
// The grouped solves of a batch share by their rows the blocks that the device
// has room for, of kGrpBatchThreads threads (20 warps an SM in FP64, 28 in FP32;
// 16 and 24 in blocks of 256): with fewer the SMs idle, with more some solves'
// blocks keep out others that they do not wait for.  A system has at least
// kGrpBatchLeast: a small one of many, left with two blocks of 256, was slower
// than its level-by-level solve.  Measured in FP32, ms for 64, 48, 24 and 8 systems
// of idim 24..96 and 64 of idim 24..44: 134, 109, 77, 51 and 29.4; with 6/7 of the
// room 137, 107, 76, 51, 29.1, with 8/7 143, 112, 80, 55, 30.1; in blocks of 256
// with 2/3 of their room 167, 129, 85, 55, 34.0, with all of it 141, 109, 77, 51,
// 29.8, with twice it 159, 130, 98, 75, 35.4; by level 150, 131, 105, 91, 31.7;
// with no bound 620 for the 64.  FP64: 176, 135, 85, 51 and 37.9; by level 157,
// 137, -, 96 and 34.2: many systems of 64-bit values are the one case where the
// entries that the groups add cost more than their hand-offs save.
constexpr int kGrpBatchThreads = 128, kGrpBatchLeast = 12;
// Solves that run at once without a batch divide half of the room equally
// (g_grp_running), each with at least this many blocks.
constexpr double kGrpShare = 0.5;
constexpr int kGrpShareLeast = 6;
static int64_t grp_budget(int n, int K) {
  return K > kGrpCols ? kGrpBudgetMin / 2 : K > 1 ? kGrpBudgetMin : std::max(kGrpBudgetMin, std::min<int64_t>(kGrpBudgetMax, n / 5));
}
// columns of one task: a 32-byte sector of a row's K values
template <typename T>
constexpr int grp_cols(int K) {
  return K < (int)(32 / sizeof(T)) ? K : (int)(32 / sizeof(T));
}

// original row of every position, and the dependencies as positions
static void grp_positions(int n, bool rev, const std::vector<int> &prow, const std::vector<int> &pja,
                          std::vector<int> &orig, std::vector<int> &dep) {
  std::vector<int> pos((size_t)n);
  orig.resize((size_t)n);
  dep.resize(pja.size());
  for (int p = 0; p < n; ++p) {
    pos[prow[p]] = p;
    orig[p] = rev ? n - 1 - prow[p] : prow[p];
  }
#pragma omp parallel for schedule(static, 4096)
  for (int64_t k = 0; k < (int64_t)dep.size(); ++k) dep[k] = pos[pja[k]];
}

// Warp tasks of a grouped plan (layout: mldg_trsv_grp.cuh).
template <typename T>
struct GrpTasks {
  std::vector<int4> desc;
  std::unique_ptr<int4[]> idx;  // left uninitialised until the threads that fill it touch it
  std::unique_ptr<T[]> val;
  int64_t slots = 0;  // entries stored, padding included
};
// wcol(c), wscale(c): index in b and factor of W's column position c; false
// when the slots outgrow the descriptors
template <typename T, typename FC, typename FS>
static bool grp_tasks(const TriGroups &g, int KC, FC wcol, FS wscale, GrpTasks<T> &out) {
  const int R = 32 / KC, ng = (int)g.gptr.size() - 1;
  auto len = [&](int p) { return (int64_t)std::max(g.row[p].nv, g.row[p].nw); };
  int64_t at = 0;  // slot groups (one int4 of indices each)
  for (int b = 0; b < ng; ++b)
    for (int p = g.gptr[b]; p < g.gptr[b + 1];) {
      // lanes per (row, column) so that every row of the task is one pass of
      // eight entries a lane; rows lengthen along a group, so a longer row
      // ahead widens the task's lanes and narrows the task
      int lt = 0, rows = 1;
      auto fits = [&](int64_t l) { return l <= (8 << lt) || (2 << lt) > R; };
      while (!fits(len(p))) ++lt;
      while (rows < (R >> lt) && p + rows < g.gptr[b + 1]) {
        const int keep = lt;
        while (!fits(len(p + rows))) ++lt;
        if (rows + 1 > (R >> lt)) {
          lt = keep;
          break;
        }
        ++rows;
      }
      int64_t nw = 0, nv = 0;
      for (int r = p; r < p + rows; ++r) {
        nw = std::max<int64_t>(nw, g.row[r].nw);
        nv = std::max<int64_t>(nv, g.row[r].nv);
      }
      nw = (nw + (4 << lt) - 1) / (4 << lt);
      nv = (nv + (4 << lt) - 1) / (4 << lt);
      if (nw > 0x7fff || nv > 0x7fff || at + (nw + nv) * R >= INT32_MAX) return false;
      out.desc.push_back(make_int4((int)at, (int)(nw | nv << 16), p, rows << 8 | lt));
      at += (nw + nv) * R;
      p += rows;
    }
  out.idx.reset(new int4[(size_t)std::max<int64_t>(at, 1)]);
  out.val.reset(new T[(size_t)std::max<int64_t>(4 * at, 1)]);
#pragma omp parallel for schedule(static, 64)
  for (int64_t k = 0; k < (int64_t)out.desc.size(); ++k) {
    const int4 d = out.desc[k];
    const int lt = d.w & 255, rows = d.w >> 8, tpr = 1 << lt;
    const int64_t end = d.x + (int64_t)((d.y & 0xffff) + (d.y >> 16)) * R;
    std::fill(out.idx.get() + d.x, out.idx.get() + end, make_int4(-1, -1, -1, -1));
    std::fill(out.val.get() + 4 * (int64_t)d.x, out.val.get() + 4 * end, T(0));
    for (int r = 0; r < rows; ++r) {
      // entry e of the row: slot e / tpr of lane e % tpr
      auto put = [&](int64_t base, int64_t e, int c, double v) {
        const int64_t slot = e >> lt, q = base + (slot >> 2) * R + r * tpr + (e & (tpr - 1));
        (&out.idx[(size_t)q].x)[slot & 3] = c;
        out.val[(size_t)(4 * q + (slot & 3))] = (T)v;
      };
      const GroupRow &gr = g.row[d.z + r];
      for (int e = 0; e < gr.nw; ++e) put(d.x, e, wcol(gr.w[e].col), gr.w[e].val * wscale(gr.w[e].col));
      for (int e = 0; e < gr.nv; ++e) put(d.x + (int64_t)(d.y & 0xffff) * R, e, gr.v[e].col, gr.v[e].val);
    }
  }
  out.slots = 4 * at;
  return true;
}

// Replays a grouped plan's tasks in ticket order: every position written
// once, every index in range, every dependency written by an earlier group.
// Returns the number of violations; x solves the factor for rhs.
template <typename T>
static int64_t grp_emulate(const TriGroups &g, const GrpTasks<T> &m, int KC, const std::vector<double> &rhs,
                           std::vector<double> &x) {
  const int n = g.gptr.back(), R = 32 / KC;
  int64_t bad = 0;
  x.assign((size_t)n, 0.0);
  std::vector<char> done((size_t)n, 0);
  size_t grp = 0;
  for (const int4 &d : m.desc) {
    const int lt = d.w & 255, rows = d.w >> 8, tpr = 1 << lt, nw = d.y & 0xffff, nv = d.y >> 16;
    while (grp + 1 < g.gptr.size() && d.z >= g.gptr[grp + 1]) ++grp;
    if (rows < 1 || rows * tpr > R || d.z < 0 || d.z + rows > g.gptr[grp + 1] || d.x < 0 || nv < 0 ||
        4 * (d.x + (int64_t)(nw + nv) * R) > m.slots) {
      ++bad;
      continue;
    }
    for (int r = 0; r < rows; ++r) {
      T acc = T(0);
      for (int sub = 0; sub < tpr; ++sub)
        for (int s = 0; s < nw + nv; ++s) {
          const size_t q = (size_t)d.x + (size_t)s * R + r * tpr + sub;
          for (int e = 0; e < 4; ++e) {
            const int j = (&m.idx[q].x)[e];
            if (j < 0) continue;
            if (j >= n || (s >= nw && (j >= g.gptr[grp] || !done[j]))) {
              ++bad;
              continue;
            }
            if (s < nw)
              acc += m.val[4 * q + e] * (T)rhs[j];
            else
              acc -= m.val[4 * q + e] * (T)x[j];
          }
        }
      const int p = d.z + r;
      bad += done[p];
      done[p] = 1;
      x[p] = (double)acc;
    }
  }
  for (int p = 0; p < n; ++p) bad += !done[p];
  return bad;
}

// Plan of the grouped solve (k_trsv_grp) for one triangular factor and one
// column width.
template <typename T>
struct DGrp {
  int n = 0, grid = 0, room = 0;  // blocks of a solve, and those that the device has room for
  GrpMat<T> m{};
  int64_t slots = 0;  // stored entries, padding included
  int *orig = nullptr;
};

static int pick_tpr(int64_t nnz, int nr) {
  const double avg = nr > 0 ? (double)nnz / nr : 0.0;
  if (avg <= 8) return 1;
  if (avg <= 16) return 2;
  if (avg <= 32) return 4;
  if (avg <= 64) return 8;
  if (avg <= 128) return 16;
  return 32;
}

// The SELL-32 copy of a CSR matrix (k_spmv_sell): skipped when padding would
// add more than a quarter of the entries, or with MLDG_NO_SELL.  Padding
// slots hold a zero value on an in-range column (the row itself, or the last
// row for the rows past the end of the last slice).
template <typename T>
static void build_sell(Arena &ar, const HostCSR &h, DCSR<T> &d) {
  if (std::getenv("MLDG_NO_SELL") || h.nr == 0 || h.nnz() == 0) return;
  const int ns = (h.nr + 31) / 32;
  std::vector<int> soff((size_t)ns + 1, 0);
  for (int s = 0; s < ns; ++s) {
    int w = 0;
    for (int i = s * 32; i < std::min(h.nr, s * 32 + 32); ++i) w = std::max(w, h.irp[i + 1] - h.irp[i]);
    const int64_t next = (int64_t)soff[s] + 32 * (int64_t)w;
    if (next > INT32_MAX) return;
    soff[s + 1] = (int)next;
  }
  const int64_t slots = soff[ns];
  if (slots * 4 > h.nnz() * 5) return;
  std::vector<T> sv((size_t)slots, T(0));
  const bool rel = d.jd != nullptr;
  std::vector<short> sjd(rel ? (size_t)slots : 0);
  std::vector<int> sja(rel ? 0 : (size_t)slots);
#pragma omp parallel for schedule(static, 256)
  for (int s = 0; s < ns; ++s) {
    const int w = (soff[s + 1] - soff[s]) / 32;
    for (int lane = 0; lane < 32; ++lane) {
      const int i = s * 32 + lane;
      const int len = i < h.nr ? h.irp[i + 1] - h.irp[i] : 0;
      const int pad_col = i < h.nr ? (h.nr == h.nc ? i : 0) : (h.nr == h.nc ? h.nr - 1 : 0);
      for (int k = 0; k < w; ++k) {
        const size_t e = (size_t)soff[s] + 32 * (size_t)k + lane;
        const int col = k < len ? h.ja[h.irp[i] + k] : pad_col;
        if (k < len) sv[e] = (T)h.val[h.irp[i] + k];
        if (rel)
          sjd[e] = (short)(col - i);
        else
          sja[e] = col;
      }
    }
  }
  d.soff = ar.upload(soff);
  d.sval = ar.upload(sv);
  if (rel)
    d.sjd = ar.upload(sjd);
  else
    d.sja = ar.upload(sja);
  d.slots = slots;
}

// FP16 row-scaled copies of a level operator's values (CSR and, when built,
// SELL order): rs_i = max_j |a_ij| rounded to FP32, h_ij = a_ij / rs_i
// rounded to FP32 and then to FP16 (round to nearest even), so |h_ij| <= 1.
static void h16_values(const HostCSR &h, std::vector<float> &sc, std::vector<__half> &hv) {
  sc.assign((size_t)h.nr, 1.f);
  hv.resize(h.val.size());
#pragma omp parallel for schedule(static, 4096)
  for (int i = 0; i < h.nr; ++i) {
    double mx = 0;
    for (int k = h.irp[i]; k < h.irp[i + 1]; ++k) mx = std::max(mx, std::fabs(h.val[k]));
    const float s = mx > 0 ? (float)mx : 1.f;
    sc[i] = s;
    for (int k = h.irp[i]; k < h.irp[i + 1]; ++k) hv[k] = __float2half_rn((float)(h.val[k] / (double)s));
  }
}
template <typename T>
static void make_h16(Arena &ar, const HostCSR &h, DCSR<T> &d) {
  std::vector<float> sc;
  std::vector<__half> hv;
  h16_values(h, sc, hv);
  d.rs = ar.upload(sc);
  d.hval = ar.upload(hv);
  if (d.soff) {
    // the SELL slots in the order build_sell wrote them (padding: zero)
    const int ns = d.nslice();
    std::vector<int> soff((size_t)ns + 1);
    MLDG_CUDA(cudaMemcpy(soff.data(), d.soff, sizeof(int) * soff.size(), cudaMemcpyDeviceToHost));
    std::vector<__half> sh((size_t)d.slots, __float2half_rn(0.f));
#pragma omp parallel for schedule(static, 256)
    for (int s = 0; s < ns; ++s)
      for (int lane = 0; lane < 32; ++lane) {
        const int i = s * 32 + lane;
        if (i >= h.nr) continue;
        for (int k = 0; k < h.irp[i + 1] - h.irp[i]; ++k) sh[(size_t)soff[s] + 32 * (size_t)k + lane] = hv[h.irp[i] + k];
      }
    d.shval = ar.upload(sh);
  }
}

// The HDIA-32 copy of a square CSR matrix (k_spmv_hdia): rows in slices of
// 32, per slice the ascending distinct column offsets j - i of its entries,
// and one value per (offset, row), zero where the row has no entry on that
// offset.  Built only when
// every row is sorted by column (the kernels then sum a row in its stored
// order), no slice has more than kHdiaMaxDiag offsets, and the slices store
// at most an eighth more values than the matrix has entries; MLDG_NO_HDIA
// skips it.  In the FP16 operator form the values are the FP16 row-scaled
// ones of make_h16 (its row scales rs are shared).
constexpr int kHdiaMaxDiag = 512;
template <typename T>
static void build_hdia(Arena &ar, const HostCSR &h, DCSR<T> &d, bool h16) {
  if (std::getenv("MLDG_NO_HDIA") || h.nr == 0 || h.nr != h.nc || h.nnz() == 0) return;
  constexpr int H = 32;
  const int ns = (h.nr + H - 1) / H;
  // the sorted distinct offsets of slice s, in o (cleared first)
  auto slice_offsets = [&](int s, std::vector<int> &o) {
    o.clear();
    for (int i = s * H; i < std::min(h.nr, s * H + H); ++i)
      for (int k = h.irp[i]; k < h.irp[i + 1]; ++k) o.push_back(h.ja[k] - i);
    std::sort(o.begin(), o.end());
    o.erase(std::unique(o.begin(), o.end()), o.end());
  };
  std::vector<int> cnt((size_t)ns, 0);
  int bad = 0;
  // pass 1: offsets per slice (counted), sortedness
#pragma omp parallel reduction(| : bad)
  {
    std::vector<int> o;
#pragma omp for schedule(static, 64)
    for (int s = 0; s < ns; ++s) {
      for (int i = s * H; i < std::min(h.nr, s * H + H); ++i)
        for (int k = h.irp[i] + 1; k < h.irp[i + 1]; ++k) bad |= h.ja[k] <= h.ja[k - 1];
      slice_offsets(s, o);
      cnt[s] = (int)o.size();
      bad |= cnt[s] > kHdiaMaxDiag;
    }
  }
  if (bad) return;
  std::vector<int> dptr((size_t)ns + 1, 0);
  for (int s = 0; s < ns; ++s) dptr[s + 1] = dptr[s] + cnt[s];
  const int64_t slots = (int64_t)H * dptr[ns];
  if (slots * 8 > h.nnz() * 9 || slots > INT32_MAX) return;
  std::vector<int> doff((size_t)dptr[ns]);
  std::vector<float> sc;
  std::vector<__half> hv;
  if (h16) h16_values(h, sc, hv);
  std::vector<T> tv(h16 ? 0 : (size_t)slots, T(0));
  std::vector<__half> th(h16 ? (size_t)slots : 0, __float2half_rn(0.f));
#pragma omp parallel
  {
    std::vector<int> o;
#pragma omp for schedule(static, 64)
    for (int s = 0; s < ns; ++s) {
      slice_offsets(s, o);
      std::copy(o.begin(), o.end(), doff.begin() + dptr[s]);
      for (int i = s * H; i < std::min(h.nr, s * H + H); ++i) {
        size_t q = 0;
        for (int k = h.irp[i]; k < h.irp[i + 1]; ++k) {
          const int off = h.ja[k] - i;
          while (o[q] != off) ++q;  // the row's offsets ascend, like the slice's
          const size_t e = (size_t)H * ((size_t)dptr[s] + q) + (size_t)(i - s * H);
          if (h16)
            th[e] = hv[k];
          else
            tv[e] = (T)h.val[k];
        }
      }
    }
  }
  d.hdptr = ar.upload(dptr);
  d.hdoff = ar.upload(doff);
  if (h16)
    d.hdhval = ar.upload(th);
  else
    d.hdval = ar.upload(tv);
  d.hdslots = slots;
}

// Staged SELL tiles (mldg_spmv_stg.cuh): the SELL-32 slots of the operator,
// in the order build_sell stores them (same widths, same padding columns,
// zero padding values), cut into tiles of consecutive slices whose packed
// block fits kStgBlockMax bytes, and packed: header {slices, slots, col
// offset, val offset}, the slices' slot offsets from the tile's first slot,
// the column offsets (int16 from the row, or int32), the values (T, or the
// FP16 row-scaled values in the FP16 form), each part 16-byte aligned.
// Built only on request (MLDG_STG: offered to the autotuner; MLDG_STG_FORCE:
// used), and not without a SELL copy or when one slice alone exceeds the
// budget.
template <typename T>
static void build_stg_pack(Arena &ar, const HostCSR &h, DCSR<T> &d, bool h16) {
  if (!(std::getenv("MLDG_STG") || std::getenv("MLDG_STG_FORCE")) || !d.soff || h.nr == 0) return;
  const int ns = d.nslice();
  std::vector<int> soff((size_t)ns + 1, 0);
  for (int sl = 0; sl < ns; ++sl) {
    int w = 0;
    for (int i = sl * 32; i < std::min(h.nr, sl * 32 + 32); ++i) w = std::max(w, h.irp[i + 1] - h.irp[i]);
    soff[sl + 1] = soff[sl] + 32 * w;
  }
  if ((int64_t)soff[ns] != d.slots) return;  // not the SELL copy's layout: no tiles
  const bool rel = d.jd != nullptr;
  const int ci = rel ? 2 : 4, vb = h16 ? 2 : (int)sizeof(T);
  auto block_bytes = [&](int s0, int s1) {
    const int slots = soff[s1] - soff[s0];
    return 16 + stg_al16(4 * (s1 - s0 + 1)) + stg_al16(ci * slots) + stg_al16(vb * slots);
  };
  std::vector<int4> tiles;
  int64_t total = 0;
  int tmax = 0;
  for (int s0 = 0; s0 < ns;) {
    if (block_bytes(s0, s0 + 1) > kStgBlockMax) return;
    int s1 = s0 + 1;
    while (s1 < ns && block_bytes(s0, s1 + 1) <= kStgBlockMax) ++s1;
    const int bb = block_bytes(s0, s1);
    if ((total + bb) / 16 > INT32_MAX) return;
    tiles.push_back(make_int4(s0, s1, (int)(total / 16), bb / 16));
    total += bb;
    tmax = std::max(tmax, bb);
    s0 = s1;
  }
  std::vector<float> sc;
  std::vector<__half> hv;
  if (h16) h16_values(h, sc, hv);
  std::vector<uint4> pk((size_t)(total / 16), make_uint4(0, 0, 0, 0));
  unsigned char *base = reinterpret_cast<unsigned char *>(pk.data());
#pragma omp parallel for schedule(dynamic, 64)
  for (int t = 0; t < (int)tiles.size(); ++t) {
    const int4 td = tiles[t];
    unsigned char *blk = base + (size_t)td.z * 16;
    const int nsl = td.y - td.x, slots = soff[td.y] - soff[td.x];
    const int off_col = 16 + stg_al16(4 * (nsl + 1)), off_val = off_col + stg_al16(ci * slots);
    int *hdr = reinterpret_cast<int *>(blk);
    hdr[0] = nsl;
    hdr[1] = slots;
    hdr[2] = off_col;
    hdr[3] = off_val;
    for (int q = 0; q <= nsl; ++q) hdr[4 + q] = soff[td.x + q] - soff[td.x];
    for (int sl = td.x; sl < td.y; ++sl) {
      const int w = (soff[sl + 1] - soff[sl]) / 32;
      for (int lane = 0; lane < 32; ++lane) {
        const int i = sl * 32 + lane;
        const int len = i < h.nr ? h.irp[i + 1] - h.irp[i] : 0;
        const int pad_col = i < h.nr ? (h.nr == h.nc ? i : 0) : (h.nr == h.nc ? h.nr - 1 : 0);
        for (int k = 0; k < w; ++k) {
          const size_t e = (size_t)(soff[sl] - soff[td.x]) + 32 * (size_t)k + lane;
          const int col = k < len ? h.ja[h.irp[i] + k] : pad_col;
          if (rel)
            reinterpret_cast<short *>(blk + off_col)[e] = (short)(col - i);
          else
            reinterpret_cast<int *>(blk + off_col)[e] = col;
          if (k < len) {
            if (h16)
              reinterpret_cast<__half *>(blk + off_val)[e] = hv[h.irp[i] + k];
            else
              reinterpret_cast<T *>(blk + off_val)[e] = (T)h.val[h.irp[i] + k];
          }
        }
      }
    }
  }
  d.tiles = ar.upload(tiles);
  d.pk = ar.upload(pk);
  d.ntiles = (int)tiles.size();
  d.tblock = tmax;
}

template <typename T>
static DCSR<T> to_dev(Arena &ar, const HostCSR &h, bool h16 = false) {
  DCSR<T> d;
  if (!h.present()) return d;
  d.nr = h.nr;
  d.nc = h.nc;
  d.nnz = h.nnz();
  d.irp = ar.upload(h.irp);
  d.ja = ar.upload(h.ja);
  if (h.nr == h.nc && !std::getenv("MLDG_NO_IDX16")) {
    int bad = 0;
#pragma omp parallel for reduction(| : bad) schedule(static, 4096)
    for (int i = 0; i < h.nr; ++i)
      for (int k = h.irp[i]; k < h.irp[i + 1]; ++k) bad |= std::abs(h.ja[k] - i) > 32767;
    if (!bad) {
      std::vector<short> jd(h.ja.size());
#pragma omp parallel for schedule(static, 4096)
      for (int i = 0; i < h.nr; ++i)
        for (int k = h.irp[i]; k < h.irp[i + 1]; ++k) jd[k] = (short)(h.ja[k] - i);
      d.jd = ar.upload(jd);
    }
  }
  std::vector<T> v(h.val.begin(), h.val.end());
  d.val = ar.upload(v);
  d.tpr = pick_tpr(d.nnz, d.nr);
  build_sell(ar, h, d);
  if (h16) make_h16(ar, h, d);
  build_hdia(ar, h, d, h16);
  build_stg_pack(ar, h, d, h16);
  return d;
}

// multi-RHS kernels are compiled for K = 2, 4, 8, 16, 32 columns
template <typename F>
static void kdispatch(int K, F &&f) {
  switch (K) {
    case 2: f(std::integral_constant<int, 2>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    case 32: f(std::integral_constant<int, 32>()); break;
    default: fail(MLDG_ERR_INTERNAL, "bad multi-vector width %d", K);
  }
}
// the ELL triangular solve also serves the single-vector V-cycle (K = 1)
template <typename F>
static void kdispatch_ell(int K, F &&f) {
  if (K == 1)
    f(std::integral_constant<int, 1>());
  else
    kdispatch(K, f);
}
// (K, E, PF) instances of k_trsv_ell: E in {4, 8, 16}, the next task's
// metadata prefetched for E <= 8
template <int V>
using IC = std::integral_constant<int, V>;
template <int KK, typename F>
static void ell_dispatch_k(int E, bool pf, F &f) {
  if constexpr (KK == 1) {
    switch (E) {
      case 4: f(IC<KK>(), IC<4>(), std::true_type()); break;
      case 8: f(IC<KK>(), IC<8>(), std::true_type()); break;
      default: f(IC<KK>(), IC<16>(), std::false_type()); break;
    }
  } else {
    switch (E) {
      case 4: f(IC<KK>(), IC<4>(), std::true_type()); break;
      case 8: f(IC<KK>(), IC<8>(), std::true_type()); break;
      default: f(IC<KK>(), IC<16>(), std::false_type()); break;
    }
  }
}
template <typename F>
static void ell_dispatch(int K, int E, bool pf, F &&f) {
  kdispatch_ell(K, [&](auto kc) { ell_dispatch_k<decltype(kc)::value>(E, pf, f); });
}

static int ilog2(int K) {
  int r = 0;
  while ((1 << r) < K) ++r;
  return r;
}

// ---------------------------------------------------------------------------
// Engine: one precision form of the V-cycle.
struct Engine {
  virtual ~Engine() {}
  virtual void record(char trans) = 0;  // issue one V-cycle: xin (FP64) -> yout (FP64)
  // With kry_io set (inside a CG/FCG solve of an FP32 V-cycle) record()
  // leaves out its two precision casts: the V-cycle starts from the FP32 copy
  // of r that the Krylov kernels write to kry_x32() and ends in kry_y32(),
  // which they read as z.  Both are null for an FP64 V-cycle.
  bool kry_io = false;
  virtual float *kry_x32() { return nullptr; }
  virtual float *kry_y32() { return nullptr; }
  // Multi-RHS V-cycle on K row-interleaved columns: xin_m -> yout_m (FP64,
  // n0 x K interleaved).  ensure_multi allocates the K-wide buffers (true when
  // they were reallocated, which invalidates captured multi graphs).
  virtual bool ensure_multi(int K, char trans) = 0;
  // gives back all that ensure_multi made: the state before its first call
  virtual void release_multi() = 0;
  virtual void record_multi(char trans, int K) = 0;
  double *xin_m = nullptr, *yout_m = nullptr, *col_m = nullptr;
  int mcap = 0;
  virtual void dump_trace() {}
  // After a solve gave up on a dependency wait: put every exchange buffer
  // back to the sentinel and every ticket counter back to zero, as finalize
  // left them, so that the next apply on the handle starts clean.
  virtual void reset_solve_state() = 0;
  int64_t launches = 0;
  // bytes: algorithmic bytes of the recorded launches (each sparse operand of
  // the reference's operation once, each dense vector operand once);
  // impl_bytes: what the chosen implementation reads and writes, which
  // differs where a level's ILU(0) or GS solves run as products with an
  // explicit dense inverse
  int64_t bytes = 0, impl_bytes = 0;
  cudaStream_t st = nullptr;
  int cycle = MLDG_CYCLE_V;  // MLDG_CYCLE_V / _W / _K / _KSYM
  // ---- launch accounting, probe and profile hooks ----
  int cur_lev = 0;
  int probe_kind = 0, probe_lev = 0, probe_idx = 0;
  bool probe_armed = false, pmatch = false;
  int64_t probe_bytes = 0;
  cudaEvent_t pev0 = nullptr, pev1 = nullptr;
  int seen[8][64];
  struct Prof {
    int kind, lev;
    int64_t bytes;
    cudaEvent_t e0, e1;
  };
  std::vector<Prof> *prof = nullptr;
  bool capturing = false;  // inside stream capture: probe events become graph nodes
  // programmatic dependent launch of the streaming kernels (launch_k); off
  // while probe or profile events are recorded between kernels, and with
  // MLDG_NO_PDL
  bool pdl = std::getenv("MLDG_NO_PDL") == nullptr;
  // most blocks of a grouped solve, 0 for no bound: while a batch of systems is
  // captured, whose solves share the SMs
  int grp_blocks = 0;
  int grp_room = 0;  // blocks of a batch's one-column grouped solve that the device has room for
  bool pdl_on() const { return pdl && probe_kind == 0 && !prof; }
  template <typename... KArgs, typename... Args>
  void kl(void (*kern)(KArgs...), int grid, int block, Args... args) {
    launch_k(pdl_on(), kern, grid, block, st, args...);
  }
  void rec(cudaEvent_t e) {
    if (capturing)
      MLDG_CUDA(cudaEventRecordWithFlags(e, st, cudaEventRecordExternal));
    else
      MLDG_CUDA(cudaEventRecord(e, st));
  }
  void begin(int kind) {
    pmatch = false;
    const int lv_ = std::min(cur_lev, 63);
    int &c = seen[kind][lv_];
    if (probe_kind == kind && probe_lev == cur_lev && c == probe_idx) {
      pmatch = true;
      rec(pev0);
    }
    ++c;
    if (prof) {
      Prof e{kind, cur_lev, 0, nullptr, nullptr};
      MLDG_CUDA(cudaEventCreate(&e.e0));
      MLDG_CUDA(cudaEventCreate(&e.e1));
      MLDG_CUDA(cudaEventRecord(e.e0, st));
      prof->push_back(e);
    }
  }
  // b: bytes the launch moves; alg: its algorithmic bytes when they differ
  void end(int64_t b, int64_t alg = -1) {
    if (alg < 0) alg = b;
    launches++;
    bytes += alg;
    impl_bytes += b;
    if (pmatch) {
      rec(pev1);
      probe_bytes = alg;
      probe_armed = true;
      pmatch = false;
    }
    if (prof) {
      prof->back().bytes = alg;
      MLDG_CUDA(cudaEventRecord(prof->back().e1, st));
    }
  }
};

// K identity columns c0 .. c0+K-1 (row-interleaved); rows past n stay zero
template <typename T>
__global__ void k_ident_block(int n, int c0, int K, T *x) {
  const long long tot = (long long)n * K;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / K), c = (int)(t % K);
    x[t] = (i == c0 + c) ? T(1) : T(0);
  }
}
// M[i*n + c0 + c] = y[i*K + c] for the columns that exist
template <typename T>
__global__ void k_scatter_cols(int n, int c0, int K, const T *__restrict__ y, T *__restrict__ M) {
  const long long tot = (long long)n * K;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / K), c = (int)(t % K);
    if (c0 + c < n) M[(size_t)i * n + c0 + c] = y[t];
  }
}
// MT = M^T (n x n), 32 x 32 tiles through shared memory
template <typename T>
__global__ void k_transpose_sq(int n, const T *__restrict__ M, T *__restrict__ MT) {
  __shared__ T tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = by + r, j = bx + threadIdx.x;
    if (i < n && j < n) tile[r][threadIdx.x] = M[(size_t)i * n + j];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = bx + r, j = by + threadIdx.x;
    if (i < n && j < n) MT[(size_t)i * n + j] = tile[threadIdx.x][r];
  }
}

// y = a*x + b*y (b = 1: an axpy as psb_geaxpby(a, x, 1, y))
template <typename T>
__global__ void k_axpby2(int n, T a, const T *__restrict__ x, T b, T *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}
// up to three dot products of T vectors accumulated in FP64, per-block
// partials in the layout of k_dots (summed by k_dots_final)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_dotsT(int n, int np, const T *__restrict__ x0,
                                                      const T *__restrict__ y0, const T *__restrict__ x1,
                                                      const T *__restrict__ y1, const T *__restrict__ x2,
                                                      const T *__restrict__ y2, double *partial) {
  __shared__ double sh[32];
  double s0 = 0, s1 = 0, s2 = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    s0 = fma((double)x0[i], (double)y0[i], s0);
    if (np > 1) s1 = fma((double)x1[i], (double)y1[i], s1);
    if (np > 2) s2 = fma((double)x2[i], (double)y2[i], s2);
  }
  s0 = block_sum(s0, sh);
  s1 = block_sum(s1, sh);
  s2 = block_sum(s2, sh);
  if (threadIdx.x == 0) {
    partial[blockIdx.x * 3 + 0] = s0;
    partial[blockIdx.x * 3 + 1] = s1;
    partial[blockIdx.x * 3 + 2] = s2;
  }
}

template <typename T>
__global__ void k_axpby1(int n, const T *__restrict__ x, T beta, T *y) {
  pdl_enter();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = (beta == T(0)) ? x[i] : fma(beta, y[i], x[i]);
}

struct Handle;

template <typename T>
struct EngineT : Engine {
  struct Lev {
    int n = 0, kind = 0, spre = 1, spost = 1;
    double damp = 1.0;
    int64_t nnz_nd = 0;
    // stored entries of the two triangular factors (ILU(0) L, U or the GS
    // strict triangles): the algorithmic bytes of a level whose solves run
    // as dense products
    int64_t nnz_l = 0, nnz_u = 0;
    DCSR<T> A, AT, P, R, ND, NDT;
    DTri<T> L, U, Lt, Ut;
    T *d = nullptr;
    // ty: residual of the cycle; tz, tw: smoother iterates (never aliasing
    // the smoother's input, which may be ty)
    T *x = nullptr, *y = nullptr, *ty = nullptr, *tw = nullptr, *tz = nullptr, *bufA = nullptr, *bufB = nullptr;
    // K-wide (row-interleaved) counterparts for the multi-RHS V-cycle
    T *xm = nullptr, *ym = nullptr, *tym = nullptr, *twm = nullptr, *tzm = nullptr, *bufAm = nullptr,
      *bufBm = nullptr;
    // windowed cluster solves (k_trsv_win) for both factors of each pair
    bool win = false;
    // single-vector solves through the ELL kernel (k_trsv_ell, K = 1) instead
    bool ell1 = false;
    // FBGS: unscaled strict triangles for sweeps > 1, and which exchange
    // buffer the next single solve writes (one-column and K-column forms)
    DCSR<T> GL, GU;
    int gflip = 0, gflip_m = 0;
    // FBGS: explicit (D+L)^{-1} and (D+U)^{-1} of a small level, when faster
    T *gsF = nullptr, *gsB = nullptr;
    DWin<T> wL, wU, wUt, wLt;
    // replicated-window cluster solves (k_trsv_rep): built (rep_ok) on large
    // ILU(0) levels, used (rep) when the autotuner finds them fastest
    bool rep = false, rep_ok = false;
    DRep<T> rL, rU, rUt, rLt;
    // partitioned solves (k_trsv_blk): built (blk_ok) on ILU(0) levels, used
    // (blk) when the autotuner finds them fastest
    bool blk = false, blk_ok = false;
    DBlk<T> kL, kU, kUt, kLt;
    // grouped solves (k_trsv_grp) of every factor, per log2 of the column
    // width.  A recorded cycle's s-th solve on the level writes x[s % ring] and
    // resets x[(s + ring / 2) % ring]: by then the solve that read it is over
    // (ring 4 for ILU(0) pairs, whose second solve reads the first's; 2 for the
    // single Gauss-Seidel solves).  seq counts the cycle's solves.
    bool grp = false;
    std::vector<double> h_d;  // d on the host: folded into W of the scaled solves
    struct Grp {
      DGrp<T> L, U, Ut, Lt;
      T *x[4] = {};
      int *ctr = nullptr;  // one ticket counter per buffer
      int ring = 4, seq = 0;
      bool refused = false;  // no plan for this width: the level's other solve
      bool built(char trans) const { return (trans == 'N' ? L : Ut).n > 0; }
    } g[6];
    // coarsest level: explicit inverse of its ILU(0) factorisation (and its transpose)
    T *minv = nullptr, *minvT = nullptr;
    T *rp0 = nullptr, *rp1 = nullptr;  // right-hand sides in position order
    // point-Jacobi levels with at most two sweeps (every sweep a first one):
    // ND and ND^T stored with their columns scaled by d (k_jacobi first == 2)
    bool nd_scaled = false;
    // FP16 prolongator values + FP32 row scale (MLDG_PREC_FP32_P16)
    __half *Ph = nullptr;
    float *Pscale = nullptr;
  };
  std::vector<Lev> lv;
  Handle *h = nullptr;
  int *err = nullptr;
  double *xin = nullptr, *yout = nullptr;  // FP64 boundary vectors of level 0
  int nsm = 148;

  // ---- launch helpers ----
  int blocks_for(int64_t threads) const {
    int64_t b = (threads + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)nsm * 16));
  }
  void spmv(const DCSR<T> &A, const T *v, T a1, const T *b, T a0, T *out, T a2) {
    if constexpr (std::is_same<T, float>::value) {
      if (A.h16()) {
        spmv_v<__half>(A, A.hval, A.shval, A.rs, v, a1, b, a0, out, a2, A.hdhval);
        return;
      }
    }
    spmv_v<T>(A, A.val, A.sval, nullptr, v, a1, b, a0, out, a2, A.hdval);
  }
  // values of type V (T, or FP16 with the row scales rs)
  int stg_stages = kStgStages;
  // ring depth of a staged launch: the configured stages, fewer if they would not fit
  int stg_fit(const DCSR<T> &A) const {
    int sgs = stg_stages;
    while (sgs > kStgStages && stg_smem(sgs, A.tblock) > kStgSmemMax) --sgs;
    return sgs;
  }
  StgArgs stg_args(const DCSR<T> &A, const float *rs) {
    StgArgs a{};
    a.ntiles = A.ntiles;
    a.nr = A.nr;
    a.stages = stg_fit(A);
    a.block_bytes = A.tblock;
    a.tiles = A.tiles;
    a.pk = A.pk;
    a.rs = rs;
    a.err = err;
    return a;
  }
  // fill the staged kernels' launch cache for every (kernel, shared memory)
  // pair the operators can launch, before any stream capture
  void stg_prepare() {
    for (auto &L : lv)
      for (DCSR<T> *op : {&L.A, &L.AT, &L.P, &L.R, &L.ND, &L.NDT}) {
        if (!op->tiles) continue;
        const size_t sm = stg_smem(stg_fit(*op), op->tblock);
        auto go = [&](auto vtag) {
          using V = typename decltype(vtag)::type;
          if (op->jd) {
            stg_occ(k_spmv_stg<T, V, short>, sm);
            stg_occ(k_jacobi_stg<T, V, short>, sm);
          } else {
            stg_occ(k_spmv_stg<T, V, int>, sm);
            stg_occ(k_jacobi_stg<T, V, int>, sm);
          }
        };
        if constexpr (std::is_same<T, float>::value) {
          if (op->h16()) {
            go(std::common_type<__half>());
            continue;
          }
        }
        go(std::common_type<T>());
      }
  }
  template <typename V>
  void spmv_stg(const DCSR<T> &A, const float *rs, const T *v, T a1, const T *b, T a0, T *out, T a2) {
    const StgArgs a = stg_args(A, rs);
    const size_t sm = stg_smem(a.stages, a.block_bytes);
    if (A.jd)
      stg_launch(k_spmv_stg<T, V, short>, sm, A.ntiles, nsm, st, a, v, a1, b, a0, out, a2);
    else
      stg_launch(k_spmv_stg<T, V, int>, sm, A.ntiles, nsm, st, a, v, a1, b, a0, out, a2);
  }
  template <typename V>
  void jacobi_stg(const DCSR<T> &ND, const float *rs, const T *d, const T *x, const T *ty, int first, T omega,
                  T alpha, T beta, T *out) {
    const StgArgs a = stg_args(ND, rs);
    const size_t sm = stg_smem(a.stages, a.block_bytes);
    if (ND.jd)
      stg_launch(k_jacobi_stg<T, V, short>, sm, ND.ntiles, nsm, st, a, d, x, ty, first, omega, alpha, beta, out);
    else
      stg_launch(k_jacobi_stg<T, V, int>, sm, ND.ntiles, nsm, st, a, d, x, ty, first, omega, alpha, beta, out);
  }
  template <typename V>
  void spmv_v(const DCSR<T> &A, const V *val, const V *sval, const float *rs, const T *v, T a1, const T *b,
              T a0, T *out, T a2, const V *hdv) {
    const int64_t vec = (int64_t)A.nc * sizeof(T) + (int64_t)A.nr * sizeof(T) * (1 + (b ? 1 : 0) + (a2 != T(0) ? 1 : 0));
    if (A.hdia() && hdv) {
      begin(MLDG_KERNEL_SPMV);
      if (A.hd16)
        kl(k_spmv_hdia<T, V, 16>, blocks_for((int64_t)A.hd_nslice() * 32), 256, A.nr, A.hdptr, A.hdoff, hdv, v, a1,
           b, a0, out, a2, rs);
      else
      kl(k_spmv_hdia<T, V, 4>, blocks_for((int64_t)A.hd_nslice() * 32), 256, A.nr, A.hdptr, A.hdoff, hdv, v, a1,
                                                                                 b, a0, out, a2, rs);
      end(A.mat_bytes() + vec, A.alg_bytes() + vec);
      return;
    }
    if (A.sell == 4 && A.tiles) {
      begin(MLDG_KERNEL_SPMV);
      spmv_stg<V>(A, rs, v, a1, b, a0, out, a2);
      end(A.csr_bytes() + vec, A.alg_bytes() + vec);
      return;
    }
    if (A.sell >= 1 && A.sell <= 3 && A.soff) {
      begin(MLDG_KERNEL_SPMV);
      const int g = blocks_for((int64_t)A.nslice() * 32 / (A.sell == 2 ? 2 : 1));
      if (A.sell == 3) {
        if (A.sjd)
          kl(k_spmv_sellp<T, short, V>, g, 256, A.nr, A.soff, A.sjd, sval, v, a1, b, a0, out, a2, rs);
        else
          kl(k_spmv_sellp<T, int, V>, g, 256, A.nr, A.soff, A.sja, sval, v, a1, b, a0, out, a2, rs);
      } else if (A.sell == 2) {
        if (A.sjd)
          kl(k_spmv_sell<T, short, 2, V>, g, 256, A.nr, A.soff, A.sjd, sval, v, a1, b, a0, out, a2, rs);
        else
          kl(k_spmv_sell<T, int, 2, V>, g, 256, A.nr, A.soff, A.sja, sval, v, a1, b, a0, out, a2, rs);
      } else {
        if (A.sjd)
          kl(k_spmv_sell<T, short, 1, V>, g, 256, A.nr, A.soff, A.sjd, sval, v, a1, b, a0, out, a2, rs);
        else
          kl(k_spmv_sell<T, int, 1, V>, g, 256, A.nr, A.soff, A.sja, sval, v, a1, b, a0, out, a2, rs);
      }
      end(A.mat_bytes() + vec, A.alg_bytes() + vec);
      return;
    }
    const int g = blocks_for((int64_t)A.nr * A.tpr);
    begin(MLDG_KERNEL_SPMV);
    switch (A.tpr) {
#define CASE(K)                                                                                         \
  case K:                                                                                               \
    if (A.jd)                                                                                           \
      kl(k_spmv<T, K, short, V>, g, 256, A.nr, A.irp, A.jd, val, v, a1, b, a0, out, a2, rs);    \
    else                                                                                                \
      kl(k_spmv<T, K, int, V>, g, 256, A.nr, A.irp, A.ja, val, v, a1, b, a0, out, a2, rs);      \
    break;
      CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32)
#undef CASE
      default: fail(MLDG_ERR_INTERNAL, "bad tpr %d", A.tpr);
    }
    end(A.csr_bytes() + vec, A.alg_bytes() + vec);
  }
  void jacobi(const DCSR<T> &ND, const T *d, const T *x, const T *ty, int first, T omega,
              T alpha, T beta, T *out) {
    if constexpr (std::is_same<T, float>::value) {
      if (ND.h16()) {
        jacobi_v<__half>(ND, ND.hval, ND.shval, ND.rs, d, x, ty, first, omega, alpha, beta, out, ND.hdhval);
        return;
      }
    }
    jacobi_v<T>(ND, ND.val, ND.sval, nullptr, d, x, ty, first, omega, alpha, beta, out, ND.hdval);
  }
  template <typename V>
  void jacobi_v(const DCSR<T> &ND, const V *val, const V *sval, const float *rs, const T *d, const T *x,
                const T *ty, int first, T omega, T alpha, T beta, T *out, const V *hdv) {
    const int64_t vec = (int64_t)ND.nr * sizeof(T) * (3 + (first ? 0 : 1) + (beta != T(0) ? 1 : 0));
    if (ND.hdia() && hdv) {
      begin(MLDG_KERNEL_JACOBI);
      if (ND.hd16)
        kl(k_jacobi_hdia<T, V, 16>, blocks_for((int64_t)ND.hd_nslice() * 32), 256, ND.nr, ND.hdptr, ND.hdoff, hdv, d,
           x, ty, first, omega, alpha, beta, out, rs);
      else
      kl(k_jacobi_hdia<T, V, 4>, blocks_for((int64_t)ND.hd_nslice() * 32), 256, 
          ND.nr, ND.hdptr, ND.hdoff, hdv, d, x, ty, first, omega, alpha, beta, out, rs);
      end(ND.mat_bytes() + vec, ND.alg_bytes() + vec);
      return;
    }
    if (ND.sell == 4 && ND.tiles) {
      begin(MLDG_KERNEL_JACOBI);
      jacobi_stg<V>(ND, rs, d, x, ty, first, omega, alpha, beta, out);
      end(ND.csr_bytes() + vec, ND.alg_bytes() + vec);
      return;
    }
    if (ND.sell >= 1 && ND.sell <= 3 && ND.soff) {
      begin(MLDG_KERNEL_JACOBI);
      const int g = blocks_for((int64_t)ND.nslice() * 32 / (ND.sell == 2 ? 2 : 1));
      if (ND.sell == 3) {
        if (ND.sjd)
          kl(k_jacobi_sellp<T, short, V>, g, 256, ND.nr, ND.soff, ND.sjd, sval, d, x, ty, first, omega,
                                                         alpha, beta, out, rs);
        else
          kl(k_jacobi_sellp<T, int, V>, g, 256, ND.nr, ND.soff, ND.sja, sval, d, x, ty, first, omega,
                                                       alpha, beta, out, rs);
      } else if (ND.sell == 2) {
        if (ND.sjd)
          kl(k_jacobi_sell<T, short, 2, V>, g, 256, ND.nr, ND.soff, ND.sjd, sval, d, x, ty, first, omega,
                                                           alpha, beta, out, rs);
        else
          kl(k_jacobi_sell<T, int, 2, V>, g, 256, ND.nr, ND.soff, ND.sja, sval, d, x, ty, first, omega,
                                                         alpha, beta, out, rs);
      } else {
        if (ND.sjd)
          kl(k_jacobi_sell<T, short, 1, V>, g, 256, ND.nr, ND.soff, ND.sjd, sval, d, x, ty, first, omega,
                                                           alpha, beta, out, rs);
        else
          kl(k_jacobi_sell<T, int, 1, V>, g, 256, ND.nr, ND.soff, ND.sja, sval, d, x, ty, first, omega,
                                                         alpha, beta, out, rs);
      }
      end(ND.mat_bytes() + vec, ND.alg_bytes() + vec);
      return;
    }
    const int g = blocks_for((int64_t)ND.nr * ND.tpr);
    begin(MLDG_KERNEL_JACOBI);
    switch (ND.tpr) {
#define CASE(K)                                                                                          \
  case K:                                                                                                \
    if (ND.jd)                                                                                           \
      kl(k_jacobi<T, K, short, V>, g, 256, ND.nr, ND.irp, ND.jd, val, d, x, ty, first, omega,    \
                                                  alpha, beta, out, rs);                                 \
    else                                                                                                 \
      kl(k_jacobi<T, K, int, V>, g, 256, ND.nr, ND.irp, ND.ja, val, d, x, ty, first, omega,      \
                                                alpha, beta, out, rs);                                   \
    break;
      CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32)
#undef CASE
      default: fail(MLDG_ERR_INTERNAL, "bad tpr %d", ND.tpr);
    }
    end(ND.csr_bytes() + vec, ND.alg_bytes() + vec);
  }
  void diag(int n, const T *d, const T *x, T alpha, T beta, T *out) {
    begin(MLDG_KERNEL_VEC);
    kl(k_diag<T>, blocks_for(n), 256, n, d, x, alpha, beta, out);
    end((int64_t)n * sizeof(T) * (3 + (beta != T(0) ? 1 : 0)));
  }
  // precision cast of a boundary vector (k_cast4 when both are 16-byte aligned)
  template <typename A, typename B>
  void cast(int n, const A *x, B *y) {
    if ((((uintptr_t)x | (uintptr_t)y) & 15u) == 0)
      kl(k_cast4<A, B>, blocks_for(((int64_t)n + 3) / 4), 256, n, x, y);
    else
      kl(k_cast<A, B>, blocks_for(n), 256, n, x, y);
  }
  void fill(int n, T v, T *y) {
    begin(MLDG_KERNEL_VEC);
    kl(k_fill<T>, blocks_for(n), 256, n, v, y);
    end((int64_t)n * sizeof(T));
  }
  void trsv(const DTri<T> &t, const T *rhs, const T *scale, T *cur, T *other, T *out, T alpha,
            T beta) {
    TriArgs<T> a;
    a.n = t.n;
    a.rev = t.rev;
    a.nlevels = t.nlevels;
    a.lvl_ptr = t.lvl_ptr;
    a.prow = t.prow;
    a.pirp = t.pirp;
    a.pja = t.pja;
    a.pval = t.pval;
    a.rhs_src = rhs;
    a.rhs_scale = scale;
    a.cur = cur;
    a.other = other;
    a.out = out;
    a.alpha = alpha;
    a.beta = beta;
    a.counters = t.counters;
    a.err = err;
    a.nblk = t.nblk;
    a.blk = t.blk;
    begin(MLDG_KERNEL_TRSV);
    launch_trsv(t, a, st);
    end(t.nnz * (int64_t)(sizeof(T) + 4) + 4 * (2 * (int64_t)t.n + 1) +
        (int64_t)t.n * sizeof(T) *
            (1 + (scale ? 1 : 0) + 1 + (other ? 1 : 0) + (out ? 1 + (beta != T(0)) : 0)));
  }

  void trsv_ell1(const DTri<T> &t, const T *rhs, const T *scale, T *cur, T *other, T *out, T alpha, T beta) {
    begin(MLDG_KERNEL_TRSV);
    launch_ell(t.ell[0], 1, rhs, scale, cur, other, out, alpha, beta);
    end(t.nnz * (int64_t)(sizeof(T) + 4) + 4 * (2 * (int64_t)t.n + 1) +
        (int64_t)t.n * sizeof(T) *
            (1 + (scale ? 1 : 0) + 1 + (other ? 1 : 0) + (out ? 1 + (beta != T(0)) : 0)));
  }
  // Per level: time the ILU pair on the single-vector ELL solve against the
  // level's other solve (sync-free blocks or windowed) and keep the faster.
  void autotune_ilu(int reps) {
    cudaEvent_t e0, e1;
    MLDG_CUDA(cudaEventCreate(&e0));
    MLDG_CUDA(cudaEventCreate(&e1));
    for (auto &L : lv) {
      const bool gs = L.kind == MLDG_SMOOTHER_FBGS;
      if ((L.kind != MLDG_SMOOTHER_BJAC && !gs) || L.minv || L.grp || !L.L.ell[0].ok || !L.U.ell[0].ok ||
          (!gs && (!L.Ut.ell[0].ok || !L.Lt.ell[0].ok)))
        continue;
      // the timed operation: the ILU solve pair, or a forward + backward GS solve
      auto op = [&]() {
        if (gs) {
          fbgs_solve(L, false, L.x, L.ty, T(0));
          fbgs_solve(L, true, L.x, L.ty, T(0));
        } else {
          ilu_apply(L, 'N', L.x, T(0), L.ty);
        }
      };
      // variants: 0 the level's other solve, 1 ELL, 2 replicated-window cluster
      // solve, 3 partitioned solve
      float best[4] = {1e30f, 1e30f, 1e30f, 1e30f};
      for (int v = 0; v < 4; ++v) {
        if (v == 2 && (gs || !L.rep_ok)) continue;
        if (v == 3 && (gs || !L.blk_ok)) continue;
        L.ell1 = v == 1;
        L.rep = v == 2;
        L.blk = v == 3;
        op();  // warm
        MLDG_CUDA(cudaEventRecord(e0, st));
        for (int r = 0; r < reps; ++r) op();
        MLDG_CUDA(cudaEventRecord(e1, st));
        MLDG_CUDA(cudaEventSynchronize(e1));
        MLDG_CUDA(cudaEventElapsedTime(&best[v], e0, e1));
      }
      int pick = 0;
      for (int v = 1; v < 4; ++v)
        if (best[v] < best[pick]) pick = v;
      L.ell1 = pick == 1;
      L.rep = pick == 2;
      L.blk = pick == 3;
      if (std::getenv("MLDG_VERBOSE"))
        std::fprintf(stderr, "mldg: ilu autotune n=%d other %.3f ms ell %.3f ms rep %.3f ms blk %.3f ms -> %s\n",
                     L.n, best[0] / reps, best[1] / reps, best[2] / reps, best[3] / reps,
                     L.blk ? "blk" : (L.rep ? "rep" : (L.ell1 ? "ell" : "other")));
    }
    launches = 0;
    bytes = 0;
    impl_bytes = 0;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }

  void gather(const DWin<T> &w, const T *src, T *dst) { gather(w.n, w.orig, src, dst); }
  void gather(int n, const int *orig, const T *src, T *dst) {
    begin(MLDG_KERNEL_VEC);
    k_gather<T><<<blocks_for(n), 256, 0, st>>>(n, orig, src, (const T *)nullptr, dst);
    end((int64_t)n * (4 + 2 * sizeof(T)));
  }
  // one replicated-window solve; rhs in the plan's position order
  void rsolve(const DRep<T> &w, const T *rhs, T *next, T *out, T beta, T *tpos = nullptr) {
    RepArgs<T> a;
    a.nsteps = w.nsteps;
    a.rmask = w.R - 1;
    a.capB = w.capB;
    a.stage_bytes = w.stage_bytes;
    a.ring_bytes = w.ring_bytes;
    a.linked = w.linked ? 1 : 0;
    a.desc = w.desc;
    a.blocks = w.blocks;
    a.rhs = rhs;
    a.next = w.linked ? next : nullptr;
    a.out = (beta == T(0)) ? out : nullptr;
    a.tpos = (out && beta != T(0)) ? tpos : nullptr;
    a.xp = w.xp;
    a.tail_ptr = w.tail_ptr;
    a.tail = w.tail;
    a.alpha = T(1);
    a.off_bar = w.ring_bytes + kRepD * w.stage_bytes;
    a.vbytes = w.vbytes;
    a.err = err;
    a.trace = w.trace;
    begin(MLDG_KERNEL_TRSV);
    launch_rep(w, a, st);
    end(w.nnz * (int64_t)(sizeof(T) + 4) + 4 * (2 * (int64_t)w.n + 1) +
        (int64_t)w.n * sizeof(T) * (1 + (next ? 2 : 0) + (out ? 1 : 0)) + (next ? 4 * (int64_t)w.n : 0));
    if (out && beta != T(0)) {
      begin(MLDG_KERNEL_VEC);
      k_combine<T><<<blocks_for(w.n), 256, 0, st>>>(w.n, w.orig, tpos, T(1), beta, out);
      end((int64_t)w.n * (4 + 3 * sizeof(T)));
    }
  }
  void wsolve(const DWin<T> &w, const T *rhs, T *next, T *out, T beta, T *tpos = nullptr) {
    WinArgs<T> a;
    a.n = w.n;
    a.nsteps = w.nsteps;
    a.W = w.W;
    a.wshift = w.wshift;
    a.capR = w.capR;
    a.capE = w.capE;
    a.D = w.D;
    a.stage_bytes = w.stage_bytes;
    a.off_win = w.off_win;
    a.off_desc = w.off_desc;
    a.off_bar = w.off_bar;
    a.off_ring = w.off_ring;
    a.desc = w.desc;
    a.orig = w.orig;
    a.pirp = w.pirp;
    a.pja = w.pja;
    a.pval = w.pval;
    a.rhs = rhs;
    a.nextpos = w.nextpos;
    a.nextscale = w.nextscale;
    a.next = next;
    a.out = (beta == T(0)) ? out : nullptr;
    a.tpos = (out && beta != T(0)) ? tpos : nullptr;
    a.alpha = T(1);
    a.beta = T(0);
    a.err = err;
    a.trace = w.trace;
    begin(MLDG_KERNEL_TRSV);
    launch_win(w, a, st);
    end(w.nnz * (int64_t)(sizeof(T) + 4) + 4 * (2 * (int64_t)w.n + 1) +
        (int64_t)w.n * sizeof(T) * (1 + (next ? 2 : 0) + (out ? 1 : 0)) + (next ? 4 * (int64_t)w.n : 0));
    if (out && beta != T(0)) {
      begin(MLDG_KERNEL_VEC);
      k_combine<T><<<blocks_for(w.n), 256, 0, st>>>(w.n, w.orig, tpos, T(1), beta, out);
      end((int64_t)w.n * (4 + 3 * sizeof(T)));
    }
  }

  // one partitioned solve: cur = T^{-1}(scale o rhs); other reset; out = alpha*t + beta*out
  void bsolve(const DBlk<T> &w, const T *rhs, const T *scale, T *cur, T *other, T *out, T alpha, T beta) {
    BlkArgs<T> a;
    a.nblocks = w.nblocks;
    a.wmask = w.W - 1;
    a.stage_bytes = w.stage_bytes;
    a.aux_cap = w.aux_cap;
    a.bstep = w.bstep;
    a.sdesc = w.sdesc;
    a.plan = w.plan;
    a.src = rhs;
    a.scale = scale;
    a.cur = cur;
    a.other = other;
    a.out = out;
    a.alpha = alpha;
    a.beta = beta;
    a.ticket = w.ticket;
    a.err = err;
    begin(MLDG_KERNEL_TRSV);
    launch_blk(w, a, st);
    const int64_t vec = (int64_t)w.n * sizeof(T) *
                        (1 + (scale ? 1 : 0) + 1 + (other ? 1 : 0) + (out ? 1 + (beta != T(0)) : 0));
    end(w.plan_bytes + 4 * ((int64_t)w.nsteps + 1) + vec,
        w.nnz * (int64_t)(sizeof(T) + 4) + 4 * ((int64_t)w.n + 1) + vec);
  }

  // One grouped solve x = (factor)^{-1} (scale o rhs) in position order, the
  // scaling and rhs's order folded into W's columns; out (original order)
  // = x + beta*out when given.  Returns x.
  const T *gsolve(typename Lev::Grp &G, const DGrp<T> &g, int Kw, int64_t nnz, const T *rhs, T *out, T beta) {
    const int s = G.seq % G.ring, r = (G.seq + G.ring / 2) % G.ring;
    ++G.seq;
    GrpArgs<T> a;
    a.m = g.m;
    a.K = Kw;
    a.ncb = Kw / grp_cols<T>(Kw);
    a.rhs = rhs;
    a.x = G.x[s];
    a.reset = G.x[r];
    a.orig = g.orig;
    a.out = out;
    a.alpha = T(1);
    a.beta = beta;
    a.ctr = G.ctr + 32 * s;
    a.ctr_reset = G.ctr + 32 * r;
    a.err = err;
    a.share = grp_blocks > 0 ? 0 : (int)(kGrpShare * g.room);
    a.least = kGrpShareLeast;
    begin(MLDG_KERNEL_TRSV);
    grp_dispatch(Kw, [&](auto kc) {
      if (grp_blocks > 0)
        kl(k_trsv_grp<T, decltype(kc)::value>, std::min(g.grid * (256 / kGrpBatchThreads), grp_blocks),
           kGrpBatchThreads, a);
      else
        kl(k_trsv_grp<T, decltype(kc)::value>, g.grid, 256, a);
    });
    const int64_t vec = (int64_t)g.n * Kw * (int64_t)sizeof(T) * (3 + (out ? 1 + (beta != T(0)) : 0));
    end(g.slots * (int64_t)(sizeof(T) + 4) + 16 * (int64_t)g.m.ntask + vec,
        nnz * (int64_t)(sizeof(T) + 4) + 4 * (2 * (int64_t)g.n + 1) + vec);
    return G.x[s];
  }
  // K dispatched by the columns of a task
  template <typename F>
  static void grp_dispatch(int Kw, F &&f) {
    switch (grp_cols<T>(Kw)) {
      case 1: f(std::integral_constant<int, 1>()); break;
      case 2: f(std::integral_constant<int, 2>()); break;
      case 4: f(std::integral_constant<int, 4>()); break;
      default: f(std::integral_constant<int, (int)(32 / sizeof(T))>());
    }
  }
  // whether a block of Kw columns takes the grouped solve on a level
  static bool grp_for(const Lev &L, int Kw) {
    return L.grp && !L.g[Kw == 1 ? 0 : ilog2(Kw)].refused && (Kw <= kGrpCols || L.nnz_l + L.nnz_u > 2 * kGrpWide * (int64_t)L.n);
  }
  void gpair(Lev &L, int Kw, char trans, const T *x, T beta, T *y) {
    auto &G = L.g[Kw == 1 ? 0 : ilog2(Kw)];
    if (trans == 'N') {
      const T *z = gsolve(G, G.L, Kw, L.nnz_l, x, nullptr, T(0));
      gsolve(G, G.U, Kw, L.nnz_u, z, y, beta);
    } else {
      const T *z = gsolve(G, G.Ut, Kw, L.nnz_u, x, nullptr, T(0));
      gsolve(G, G.Lt, Kw, L.nnz_l, z, y, beta);
    }
  }
  // End of a recorded cycle: the next one starts with x[0] (and x[1] for
  // pairs) at the sentinel and the counters at zero; put back those that the
  // last solves left used (none when a level makes a multiple of ring solves).
  void end_grp(int Kw) {
    const int ki = Kw == 1 ? 0 : ilog2(Kw);
    for (auto &L : lv) {
      auto &G = L.g[ki];
      if (!L.grp || !G.seq) continue;
      for (int b = 0; b < G.ring / 2; ++b)
        for (int s = std::max(0, G.seq - G.ring / 2); s < G.seq; ++s)
          if (s % G.ring == b) {
            begin(MLDG_KERNEL_VEC);
            const int64_t nn = (int64_t)L.n * Kw;
            kl(k_fill<T>, blocks_for(nn), 256, (int)nn, Sentinel<T>::value(), G.x[b]);
            end(nn * (int64_t)sizeof(T));
            kl(k_fill<int>, 1, 32, 1, 0, G.ctr + 32 * b);
          }
      G.seq = 0;
    }
  }

  // ILU solver apply: y = alpha*U^{-1}(d o L^{-1} x) + beta*y, or the 'T' form
  void ilu_apply(Lev &L, char trans, const T *x, T beta, T *y) {
    if (L.minv) {
      const T *M = (trans == 'N') ? L.minv : L.minvT;
      begin(MLDG_KERNEL_VEC);
      kl(k_gemv<T>, blocks_for((int64_t)L.n * 32), 256, L.n, M, x, T(1), beta, y);
      // algorithmic: the two sparse solves and the pivot scaling it replaces
      end((int64_t)L.n * L.n * sizeof(T) + (int64_t)L.n * sizeof(T) * (2 + (beta != T(0))),
          (L.nnz_l + L.nnz_u) * (int64_t)(sizeof(T) + 4) + 8 * ((int64_t)L.n + 1) +
              (int64_t)L.n * sizeof(T) * (3 + (beta != T(0))));
      return;
    }
    if (L.grp) {
      gpair(L, 1, trans, x, beta, y);
      return;
    }
    if (L.blk) {
      if (trans == 'N') {
        bsolve(L.kL, x, nullptr, L.bufA, L.bufB, nullptr, T(1), T(0));
        bsolve(L.kU, L.bufA, L.d, L.bufB, L.bufA, y, T(1), beta);
      } else {
        bsolve(L.kUt, x, nullptr, L.bufA, L.bufB, nullptr, T(1), T(0));
        bsolve(L.kLt, L.bufA, L.d, L.bufB, L.bufA, y, T(1), beta);
      }
      return;
    }
    if (L.ell1) {
      if (trans == 'N') {
        trsv_ell1(L.L, x, nullptr, L.bufA, L.bufB, nullptr, T(1), T(0));
        trsv_ell1(L.U, L.bufA, L.d, L.bufB, L.bufA, y, T(1), beta);
      } else {
        trsv_ell1(L.Ut, x, nullptr, L.bufA, L.bufB, nullptr, T(1), T(0));
        trsv_ell1(L.Lt, L.bufA, L.d, L.bufB, L.bufA, y, T(1), beta);
      }
      return;
    }
    if (L.rep) {
      const DRep<T> &f = (trans == 'N') ? L.rL : L.rUt;
      const DRep<T> &g = (trans == 'N') ? L.rU : L.rLt;
      gather(f.n, f.orig, x, L.rp0);
      rsolve(f, L.rp0, L.rp1, nullptr, T(0));
      rsolve(g, L.rp1, nullptr, y, beta, L.rp0);  // rp0 is free again: results in position order
      return;
    }
    if (L.win) {
      const DWin<T> &f = (trans == 'N') ? L.wL : L.wUt;
      const DWin<T> &g = (trans == 'N') ? L.wU : L.wLt;
      gather(f, x, L.rp0);
      wsolve(f, L.rp0, L.rp1, nullptr, T(0));
      wsolve(g, L.rp1, nullptr, y, beta, L.rp0);  // rp0 is free again: results in position order
      return;
    }
    if (trans == 'N') {
      trsv(L.L, x, nullptr, L.bufA, L.bufB, nullptr, T(1), T(0));
      trsv(L.U, L.bufA, L.d, L.bufB, L.bufA, y, T(1), beta);
    } else {
      trsv(L.Ut, x, nullptr, L.bufA, L.bufB, nullptr, T(1), T(0));
      trsv(L.Lt, L.bufA, L.d, L.bufB, L.bufA, y, T(1), beta);
    }
  }

  // One GS solve out = (D+L)^{-1} rhs (forward) or (D+U)^{-1} rhs (backward)
  // [+ beta*out] on the scaled unit-triangular factors.  Single solves
  // alternate the two exchange buffers (the solve leaves its own buffer
  // holding values and the other one reset); end_fbgs() restores the start
  // state at the end of a recorded cycle.
  void fbgs_solve(Lev &L, bool backward, const T *rhs, T *out, T beta) {
    if (L.gsF) {
      const T *M = backward ? L.gsB : L.gsF;
      begin(MLDG_KERNEL_VEC);
      kl(k_gemv<T>, blocks_for((int64_t)L.n * 32), 256, L.n, M, rhs, T(1), beta, out);
      // algorithmic: the sparse triangular solve (with its diagonal) it replaces
      end((int64_t)L.n * L.n * sizeof(T) + (int64_t)L.n * sizeof(T) * (2 + (beta != T(0))),
          (backward ? L.nnz_u : L.nnz_l) * (int64_t)(sizeof(T) + 4) + 4 * ((int64_t)L.n + 1) +
              (int64_t)L.n * sizeof(T) * (3 + (beta != T(0))));
      return;
    }
    if (L.grp) {
      auto &G = L.g[0];
      gsolve(G, backward ? G.U : G.L, 1, backward ? L.nnz_u : L.nnz_l, rhs, out, beta);
      return;
    }
    const DTri<T> &t = backward ? L.U : L.L;
    T *cur = L.gflip ? L.bufB : L.bufA, *other = L.gflip ? L.bufA : L.bufB;
    L.gflip ^= 1;
    if (L.ell1)
      trsv_ell1(t, rhs, L.d, cur, other, out, T(1), beta);
    else
      trsv(t, rhs, L.d, cur, other, out, T(1), beta);
  }
  void reset_solve_state() override {
    const T sent = Sentinel<T>::value();
    auto refill = [&](T *b, int64_t cnt) {
      if (b && cnt > 0) k_fill<T><<<blocks_for(cnt), 256, 0, st>>>((int)cnt, sent, b);
    };
    for (auto &L : lv) {
      const int n = std::max(L.n, 1);
      refill(L.bufA, n);
      refill(L.bufB, n);
      refill(L.bufAm, (int64_t)n * mcap);
      refill(L.bufBm, (int64_t)n * mcap);
      for (DTri<T> *f : {&L.L, &L.U, &L.Ut, &L.Lt}) {
        if (f->counters) MLDG_CUDA(cudaMemsetAsync(f->counters, 0, 2 * sizeof(int), st));
        for (auto &el : f->ell)
          if (el.ok && el.ctr) MLDG_CUDA(cudaMemsetAsync(el.ctr, 0, sizeof(int) * 32 * (el.S + 1), st));
      }
      for (DRep<T> *r : {&L.rL, &L.rU, &L.rUt, &L.rLt}) refill(r->xp, (int64_t)r->n + 8);
      for (DBlk<T> *k : {&L.kL, &L.kU, &L.kUt, &L.kLt})
        if (k->ticket) MLDG_CUDA(cudaMemsetAsync(k->ticket, 0, 2 * sizeof(int), st));
      for (int Kw = 1; Kw <= 32; Kw *= 2) reset_grp(L, Kw);
      L.gflip = 0;
      L.gflip_m = 0;
    }
    MLDG_CUDA(cudaStreamSynchronize(st));
  }

  void end_fbgs() {
    for (auto &L : lv)
      if (L.kind == MLDG_SMOOTHER_FBGS && L.gflip) {
        fill(L.n, Sentinel<T>::value(), L.bufA);
        L.gflip = 0;
      }
  }
  // jac smoother + GS solver: sweeps forward (pre, sm) or backward (post,
  // sm2) Gauss-Seidel sweeps from a zero start; y = S(x) + beta*y
  void fbgs_smoother(Lev &L, bool post, const T *x, T beta, T *y, int sweeps) {
    if (sweeps == 1) {
      fbgs_solve(L, post, x, y, beta);
      return;
    }
    fbgs_solve(L, post, x, L.tz, T(0));
    for (int s = 1; s < sweeps; ++s) {
      spmv(post ? L.GL : L.GU, L.tz, T(-1), x, T(1), L.tw, T(0));  // wv = x - (U|L) xit
      fbgs_solve(L, post, L.tw, L.tz, T(0));
    }
    k_axpby_impl(L.n, L.tz, beta, y);
  }

  // jac smoother apply with init 'Z': y = alpha*S^sweeps(x) + beta*y, alpha = 1
  void smoother(Lev &L, char trans, const T *x, T beta, T *y, int sweeps, bool post = false) {
    if (L.kind == MLDG_SMOOTHER_FBGS) {
      fbgs_smoother(L, post, x, beta, y, sweeps);
      return;
    }
    const DCSR<T> &ND = (trans == 'N') ? L.ND : L.NDT;
    if (L.kind == MLDG_SMOOTHER_BJAC) {
      if (sweeps == 1 || L.nnz_nd == 0) {
        ilu_apply(L, trans, x, beta, y);
        return;
      }
      // block-Jacobi sweeps with a non-empty off-block part (several ranks'
      // worth of blocks): ty = S(x); ty = S(x - ND ty) ...; y = ty + beta*y
      ilu_apply(L, trans, x, T(0), L.tz);
      for (int s = 1; s < sweeps; ++s) {
        spmv(ND, L.tz, T(-1), x, T(1), L.tw, T(0));
        ilu_apply(L, trans, L.tw, T(0), L.tz);
      }
      k_axpby_impl(L.n, L.tz, beta, y);
      return;
    }
    // point Jacobi (diag solver)
    const T w = (T)L.damp;
    if (sweeps == 1 || L.nnz_nd == 0) {
      diag(L.n, L.d, x, w, beta, y);
      return;
    }
    // sweeps >= 2: first sweep folded into the second (ty = w*d o x on the fly)
    T *src = nullptr;
    T *bufs[2] = {L.tz, L.tw};
    for (int s = 1; s < sweeps; ++s) {
      const bool last = (s == sweeps - 1);
      T *dst = last ? y : bufs[s & 1];
      jacobi(ND, L.d, x, src, s == 1 ? (L.nd_scaled ? 2 : 1) : 0, w, T(1), last ? beta : T(0), dst);
      src = dst;
    }
  }
  void k_axpby_impl(int n, const T *x, T beta, T *y);
  float *kry_x32() override {
    if constexpr (std::is_same<T, float>::value) return lv.empty() ? nullptr : lv[0].x;
    return nullptr;
  }
  float *kry_y32() override {
    if constexpr (std::is_same<T, float>::value) return lv.empty() ? nullptr : lv[0].y;
    return nullptr;
  }

  // V-cycle body (mld_d_inner_mult)
  void vcycle(int l, char trans) {
    cur_lev = l;
    Lev &L = lv[l];
    const int nlev = (int)lv.size();
    const bool pre = (L.spre > 0 && trans == 'N') || (L.spost > 0 && trans != 'N');
    const bool post = (L.spost > 0 && trans == 'N') || (L.spre > 0 && trans != 'N');
    if (l < nlev - 1) {
      Lev &C = lv[l + 1];
      const DCSR<T> &A = (trans == 'N') ? L.A : L.AT;
      if (pre) {
        smoother(L, trans, L.x, T(0), L.y, trans == 'N' ? L.spre : L.spost, trans != 'N');
        spmv(A, L.y, T(-1), L.x, T(1), L.ty, T(0));    // ty = x - op(A) y
        spmv(C.R, L.ty, T(1), nullptr, T(0), C.x, T(0));  // x_{l+1} = R ty
      } else {
        fill(L.n, T(0), L.y);
        spmv(C.R, L.x, T(1), nullptr, T(0), C.x, T(0));
      }
      vcycle(l + 1, trans);
      cur_lev = l;
      prolong(C, L.y);                                   // y += P y_{l+1}
      if (cycle == MLDG_CYCLE_W) {
        // W-cycle: second coarse correction from the new residual (mld_dmlprec_aply.f90:716-745)
        spmv(A, L.y, T(-1), L.x, T(1), L.ty, T(0));
        spmv(C.R, L.ty, T(1), nullptr, T(0), C.x, T(0));
        vcycle(l + 1, trans);
        cur_lev = l;
        prolong(C, L.y);
      }
      if (post) {
        spmv(A, L.y, T(-1), L.x, T(1), L.ty, T(0));
        smoother(L, trans, L.ty, T(1), L.y, trans == 'N' ? L.spost : L.spre, trans == 'N');
      }
    } else {
      smoother(L, trans, L.x, T(0), L.y, L.spre);
    }
  }
  void prolong(Lev &C, T *y);

  // ---- K-cycle (ML_CYCLE = KCYCLE / KCYCLESYM) ----
  // mld_d_inner_k_cycle / mld_dinneritkcycle (mld_dmlprec_aply.f90:811-1184):
  // the inner Krylov step on a level needs its inner products on the host
  // (the second step is taken only if the first left ||w|| > 0.25 ||rhs||),
  // so a K-cycle is issued with host synchronisations and is not captured.
  struct KVec {
    T *w = nullptr, *v = nullptr, *v1 = nullptr, *xk = nullptr, *d0 = nullptr, *d1 = nullptr;
  };
  std::vector<KVec> kvec;
  Arena karena;
  double *kpart = nullptr, *kres = nullptr, *khost = nullptr;
  bool kcycle_mode() const { return cycle == MLDG_CYCLE_K || cycle == MLDG_CYCLE_KSYM; }
  void ensure_k() {
    if (!kvec.empty()) return;
    karena.release();  // of a call whose allocations failed
    std::vector<KVec> made(lv.size());
    for (size_t l = 0; l < lv.size(); ++l) {
      const size_t n = (size_t)std::max(lv[l].n, 1);
      KVec &k = made[l];
      k.w = karena.alloc<T>(n);
      k.v = karena.alloc<T>(n);
      k.v1 = karena.alloc<T>(n);
      k.xk = karena.alloc<T>(n);
      k.d0 = karena.alloc<T>(n);
      k.d1 = karena.alloc<T>(n);
    }
    kpart = karena.alloc<double>(3 * kRedBlocks);
    kres = karena.alloc<double>(4);
    if (!khost) MLDG_CUDA(cudaMallocHost(&khost, 4 * sizeof(double)));
    kvec = std::move(made);
  }
  void copy(int n, const T *x, T *y) { k_axpby_impl(n, x, T(0), y); }
  void axpby2(int n, T a, const T *x, T b, T *y) {
    begin(MLDG_KERNEL_VEC);
    k_axpby2<T><<<blocks_for(n), 256, 0, st>>>(n, a, x, b, y);
    end((int64_t)n * sizeof(T) * 3);
  }
  // up to three inner products, returned on the host (FP64 accumulation)
  void hdots(int n, int np, const T *x0, const T *y0, const T *x1, const T *y1, const T *x2, const T *y2,
             double *r) {
    begin(MLDG_KERNEL_VEC);
    k_dotsT<T><<<kRedBlocks, kRedThreads, 0, st>>>(n, np, x0, y0, x1, y1, x2, y2, kpart);
    end((int64_t)n * sizeof(T) * 2 * np);
    begin(MLDG_KERNEL_VEC);
    k_dots_final<<<1, kRedThreads, 0, st>>>(kRedBlocks, kpart, kres);
    end(3 * kRedBlocks * 8);
    MLDG_CUDA(cudaMemcpyAsync(khost, kres, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    MLDG_CUDA(cudaStreamSynchronize(st));
    for (int q = 0; q < np; ++q) r[q] = khost[q];
  }
  void cycle_at(int l, char trans) {
    if (kcycle_mode())
      kcycle(l, trans);
    else if (cycle == MLDG_CYCLE_ADD)
      addcycle(l, trans);
    else
      vcycle(l, trans);
  }
  // additive cycle (mld_d_inner_add, mld_dmlprec_aply.f90:464-588): smooth x,
  // restrict x itself, recurse, add the prolongated correction.  FBGS levels
  // apply forward then backward GS max(sweeps) times from the previous result.
  void addcycle(int l, char trans) {
    cur_lev = l;
    Lev &L = lv[l];
    if (L.kind == MLDG_SMOOTHER_FBGS) {
      copy(L.n, L.x, L.y);
      for (int k = 0; k < std::max(L.spre, L.spost); ++k) {
        fbgs_solve(L, false, L.y, L.tw, T(0));
        fbgs_solve(L, true, L.tw, L.y, T(0));
      }
    } else {
      smoother(L, trans, L.x, T(0), L.y, L.spre);
    }
    if (l < (int)lv.size() - 1) {
      Lev &C = lv[l + 1];
      spmv(C.R, L.x, T(1), nullptr, T(0), C.x, T(0));
      cycle_at(l + 1, trans);
      cur_lev = l;
      prolong(C, L.y);
    }
  }
  void kcycle(int l, char trans) {
    cur_lev = l;
    Lev &L = lv[l];
    const int nlev = (int)lv.size();
    if (l == nlev - 1) {
      smoother(L, trans, L.x, T(0), L.y, L.spre);
      return;
    }
    Lev &C = lv[l + 1];
    const DCSR<T> &A = (trans == 'N') ? L.A : L.AT;
    smoother(L, trans, L.x, T(0), L.y, trans == 'N' ? L.spre : L.spost, trans != 'N');
    spmv(A, L.y, T(-1), L.x, T(1), L.ty, T(0));
    spmv(C.R, L.ty, T(1), nullptr, T(0), C.x, T(0));
    if (l + 1 <= nlev - 2)
      inneritk(l + 1, trans, cycle == MLDG_CYCLE_K);
    else
      cycle_at(l + 1, trans);
    cur_lev = l;
    prolong(C, L.y);
    spmv(A, L.y, T(-1), L.x, T(1), L.ty, T(0));
    smoother(L, trans, L.ty, T(1), L.y, trans == 'N' ? L.spost : L.spre, trans == 'N');
  }
  void inneritk(int l, char trans, bool gcr) {
    cur_lev = l;
    Lev &L = lv[l];
    KVec &k = kvec[l];
    const int n = L.n;
    double r[3];
    fill(n, T(0), k.xk);
    copy(n, L.x, k.w);
    fill(n, T(0), L.y);
    cycle_at(l, trans);
    cur_lev = l;
    copy(n, L.y, k.d0);
    spmv(L.A, k.d0, T(1), nullptr, T(0), k.v, T(0));  // A, untransposed, as in the reference
    if (gcr)
      hdots(n, 3, k.v, k.w, k.v, k.v, k.w, k.w, r);
    else
      hdots(n, 3, k.d0, k.w, k.d0, k.v, k.w, k.w, r);
    const double delta0 = std::sqrt(r[2]), tau = r[1];
    double alpha = r[0] / tau;
    axpby2(n, (T)(-alpha), k.v, T(1), k.w);
    hdots(n, 1, k.w, k.w, nullptr, nullptr, nullptr, nullptr, r);
    if (std::sqrt(r[0]) <= 0.25 * delta0) {
      axpby2(n, (T)alpha, k.d0, T(1), k.xk);
    } else {
      copy(n, k.w, L.x);
      cycle_at(l, trans);
      cur_lev = l;
      copy(n, L.y, k.d1);
      spmv(L.A, k.d1, T(1), nullptr, T(0), k.v1, T(0));
      if (gcr)
        hdots(n, 3, k.v1, k.v, k.v1, k.v1, k.v1, k.w, r);
      else
        hdots(n, 3, k.d1, k.v, k.d1, k.v1, k.d1, k.w, r);
      const double tau1 = r[0], tau2 = r[1], tau3 = r[2];
      const double tau4 = tau2 - (tau1 * tau1) / tau;
      alpha = alpha - (tau1 * tau3) / (tau * tau4);
      axpby2(n, (T)alpha, k.d0, T(1), k.xk);
      axpby2(n, (T)(tau3 / tau4), k.d1, T(1), k.xk);
    }
    copy(n, k.xk, L.y);
  }
  // Lanes-per-row autotuner: times k_spmv with every TPR on each level's
  // operators (A, A^T, P, R, ND, ND^T) and keeps the fastest.  The
  // off-diagonal parts of point-Jacobi levels are timed in the sweep that
  // reads them (k_jacobi, first sweep: two vector gathers per entry).
  void autotune_spmv(int reps) {
    cudaEvent_t e0, e1;
    MLDG_CUDA(cudaEventCreate(&e0));
    MLDG_CUDA(cudaEventCreate(&e1));
    const auto kept = tune_file_read();
    for (size_t l = 0; l < lv.size(); ++l) {
      Lev &L = lv[l];
      DCSR<T> *ops[6] = {&L.A, &L.AT, &L.P, &L.R, &L.ND, &L.NDT};
      const char *names[6] = {"A", "A^T", "P", "R", "ND", "ND^T"};
      for (int oi = 0; oi < 6; ++oi) {
        DCSR<T> *op = ops[oi];
        if (!op->present() || op->nr == 0) continue;
        char key[128];
        std::snprintf(key, sizeof key, "spmv %d %d %d %d %d %lld", (int)sizeof(T), op->h16() ? 1 : 0, (int)l, oi,
                      op->nr, (long long)op->nnz);
        const auto kc = kept.find(key);
        if (kc != kept.end()) {
          op->tpr = kc->second[0];
          op->sell = kc->second[1];
          op->hd16 = kc->second[2] != 0;
          continue;
        }
        // scratch vectors of this level/its neighbour large enough for nc / nr
        const int nmax = std::max(op->nr, op->nc);
        T *v = scratch_for(nmax, 0), *o = scratch_for(nmax, 1);
        float best = 1e30f;
        int best_t = op->tpr;
        int best_sell = 0;
        // candidates: CSR with 1..32 lanes per row, then the SELL copy with 1
        // and 2 slices per warp iteration (t = -1, -2)
        const bool sweep = oi >= 4 && L.kind == MLDG_SMOOTHER_JACOBI && L.d && op->nr == op->nc;
        auto run = [&]() {
          if (sweep)
            jacobi(*op, L.d, v, nullptr, L.nd_scaled ? 2 : 1, (T)L.damp, T(1), T(0), o);
          else
            spmv(*op, v, T(1), nullptr, T(0), o, T(0));
        };
        // t = -4: the staged SELL kernels; t = -5: the HDIA copy
        const bool has_hd = op->hdptr && (op->h16() ? op->hdhval != nullptr : op->hdval != nullptr);
        bool best_hd16 = false;
        for (int t : {1, 2, 4, 8, 16, 32, -1, -2, -3, -4, -5, -6}) {
          if (t < 0 && t >= -3 && !op->soff) continue;
          if (t == -4 && !op->tiles) continue;
          if (t <= -5 && !has_hd) continue;
          op->sell = t < 0 ? std::min(-t, 5) : 0;
          op->hd16 = t == -6;
          if (t > 0) op->tpr = t;
          run();  // warm
          MLDG_CUDA(cudaEventRecord(e0, st));
          for (int r = 0; r < reps; ++r) run();
          MLDG_CUDA(cudaEventRecord(e1, st));
          MLDG_CUDA(cudaEventSynchronize(e1));
          float ms = 0;
          MLDG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
          if (ms < best) {
            best = ms;
            best_t = t > 0 ? t : best_t;
            best_sell = t < 0 ? std::min(-t, 5) : 0;
            best_hd16 = t == -6;
          }
        }
        op->tpr = best_t;
        op->sell = best_sell;
        op->hd16 = best_hd16;
        tune_file_append(std::string(key) + " " + std::to_string(best_t) + " " + std::to_string(best_sell) + " " +
                         std::to_string(best_hd16 ? 1 : 0));
        if (std::getenv("MLDG_VERBOSE"))
          std::fprintf(stderr, "mldg: spmv autotune level %zu %-4s n=%d nnz=%lld -> %s%d %.4f ms\n", l,
                       names[oi], op->nr, (long long)op->nnz,
                       best_sell >= 5 ? "hdia u" : (best_sell == 4 ? "staged sell" : (best_sell ? "sell" : "csr tpr ")),
                       best_sell >= 5 ? (best_hd16 ? 16 : 4) : (best_sell == 4 ? 1 : (best_sell ? best_sell : best_t)),
                       best / reps);
      }
    }
    launches = 0;
    bytes = 0;
    impl_bytes = 0;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  T *tune_buf[2] = {nullptr, nullptr};
  int tune_n = 0;
  T *scratch_for(int n, int which) {
    if (n > tune_n) fail(MLDG_ERR_INTERNAL, "autotune scratch too small");
    return tune_buf[which];
  }

  // ---- multi-RHS V-cycle: K columns row-interleaved, v[i*K + c] ----
  int K = 2;
  Arena marena;  // K-wide buffers and block tables (grown on demand)
  ~EngineT() override {
    marena.release();
    karena.release();
    if (khost) cudaFreeHost(khost);
  }
  int64_t nk(int n) const { return (int64_t)n * K; }

  // The host side of a factor's grouped plan for Kw columns; W reads the
  // solution of `src` (null: a vector in original order) scaled by `scale` (by
  // original row, or null).
  struct GrpHost {
    const DTri<T> *t = nullptr, *src = nullptr;
    const std::vector<double> *scale = nullptr;
    DGrp<T> *dst = nullptr;
    bool ok = false;
    std::vector<int> orig;
    TriGroups pl;
    GrpTasks<T> tk;
    void build(int Kw) {
      const int n = t->n;
      std::vector<int> dep, at;
      grp_positions(n, t->rev != 0, t->h_prow, t->h_pja, orig, dep);
      if (src) {
        at.resize((size_t)n);
        for (int p = 0; p < n; ++p) at[src->rev ? n - 1 - src->h_prow[p] : src->h_prow[p]] = p;
      }
      int64_t budget = grp_budget(n, Kw);
      if (const char *e = std::getenv("MLDG_GRP_B")) budget = std::max(1, std::atoi(e));
      build_tri_groups(t->h_lvl, t->h_pirp, dep, t->h_pval, budget, kGrpRow, kGrpGrowth, &pl);
      ok = grp_tasks<T>(
          pl, grp_cols<T>(Kw), [&](int c) { return src ? at[orig[c]] : orig[c]; },
          [&](int c) { return scale ? (*scale)[orig[c]] : 1.0; }, tk);
    }
    size_t bytes() const { return (size_t)tk.slots * (sizeof(T) + 4) + 16 * tk.desc.size() + 4 * orig.size(); }
  };
  // its device side
  DGrp<T> upload_grp(Arena &ar, const GrpHost &hp, int Kw) {
    const DTri<T> &t = *hp.t;
    DGrp<T> g;
    const GrpTasks<T> &tk = hp.tk;
    const int n = t.n, KC = grp_cols<T>(Kw);
    g.n = n;
    g.slots = tk.slots;
    g.m.ntask = (int)tk.desc.size();
    g.m.desc = ar.upload(tk.desc);
    g.m.idx = ar.upload(tk.idx.get(), (size_t)tk.slots / 4);
    g.m.val = ar.upload(tk.val.get(), (size_t)tk.slots);
    g.orig = ar.upload(hp.orig);
    // warps in flight: eight groups' tasks, so that a group's tasks have their
    // entries and older values loaded when the group before it is finished
    // (idim=101 level 0: 822 us for four solves with four groups, 680 with eight)
    int nb = 0, nbatch = 0;
    grp_dispatch(Kw, [&](auto kc) {
      MLDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trsv_grp<T, decltype(kc)::value>, 256, 0));
    });
    const int ng = (int)hp.pl.gptr.size() - 1;
    const int64_t ntask = (int64_t)g.m.ntask * (Kw / KC), per = (ntask + ng - 1) / ng;
    const int64_t warps = std::max<int64_t>(32, std::min<int64_t>((Kw > kGrpCols ? 4 : 8) * per, ntask));
    g.room = std::max(nb, 1) * nsm;
    if (Kw == 1) {
      MLDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nbatch, k_trsv_grp<T, 1>, kGrpBatchThreads, 0));
      grp_room = std::max(nbatch, 1) * nsm;
    }
    g.grid = (int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, g.room));
    if (std::getenv("MLDG_VERBOSE"))
      std::fprintf(stderr, "mldg: grp K=%d n=%d levels=%d groups=%d entries %lld slots %lld tasks %d grid %d occ %d\n", Kw, n,
                   t.nlevels, ng, (long long)hp.pl.entries, (long long)g.slots, g.m.ntask, g.grid, nb);
    return g;
  }
  // The grouped plans (of trans 'N' or 'T', or of both: 0) and work vectors of a
  // level for Kw columns; false where they are refused.  All or nothing: what
  // a refusal or a failed allocation leaves behind is given back, and the level
  // sees the plans only when all are there.
  bool build_grp(Lev &L, int Kw, char trans, Arena &ar) {
    auto &G = L.g[Kw == 1 ? 0 : ilog2(Kw)];
    const typename Lev::Grp before = G;
    const Arena::Mark mark = ar.mark();
    auto undo = [&]() {
      ar.release_to(mark);
      G = before;
    };
    try {
      if (try_grp(L, G, Kw, trans, ar)) return true;
    } catch (...) {
      undo();
      throw;
    }
    undo();
    return false;
  }
  bool try_grp(Lev &L, typename Lev::Grp &G, int Kw, char trans, Arena &ar) {
    std::vector<GrpHost> hp;
    auto add = [&](const DTri<T> &t, const DTri<T> *src, const std::vector<double> *scale, DGrp<T> &dst) {
      hp.emplace_back();
      hp.back().t = &t;
      hp.back().src = src;
      hp.back().scale = scale;
      hp.back().dst = &dst;
    };
    const bool gs = L.kind == MLDG_SMOOTHER_FBGS;
    const int ring = gs ? 2 : 4;
    if (gs) {
      add(L.L, nullptr, &L.h_d, G.L);
      add(L.U, nullptr, &L.h_d, G.U);
    } else {
      if (trans != 'T') {
        add(L.L, nullptr, nullptr, G.L);
        add(L.U, &L.L, &L.h_d, G.U);
      }
      if (trans != 'N') {
        add(L.Ut, nullptr, nullptr, G.Ut);
        add(L.Lt, &L.Ut, &L.h_d, G.Lt);
      }
    }
    // a plan that would take most of the memory left is not made: the level
    // keeps its other solve, as where the indices do not reach.  One factor after
    // the other, each on the host only until it is uploaded.
    size_t need = (size_t)ring * L.n * Kw * sizeof(T), avail = 0, total = 0;
    MLDG_CUDA(cudaMemGetInfo(&avail, &total));
    size_t most = avail / 2;
    if (const char *e = std::getenv("MLDG_GRP_MB")) most = std::min(most, (size_t)std::max(0, std::atoi(e)) << 20);
    for (auto &p : hp) {
      p.build(Kw);
      need += p.bytes();
      if (!p.ok || need > most) return false;
      *p.dst = upload_grp(ar, p, Kw);
      p.pl = TriGroups();
      p.tk = GrpTasks<T>();
    }
    if (!G.ctr) {
      G.ring = ring;
      for (int b = 0; b < ring; ++b) G.x[b] = ar.alloc<T>((size_t)L.n * Kw);
      G.ctr = ar.alloc<int>(32 * 4);
      reset_grp(L, Kw);
    }
    return true;
  }
  void reset_grp(Lev &L, int Kw) {
    auto &G = L.g[Kw == 1 ? 0 : ilog2(Kw)];
    if (!G.ctr) return;
    const int64_t nn = (int64_t)L.n * Kw;
    for (int b = 0; b < G.ring; ++b)
      k_fill<T><<<blocks_for(nn), 256, 0, st>>>((int)nn, Sentinel<T>::value(), G.x[b]);
    MLDG_CUDA(cudaMemsetAsync(G.ctr, 0, sizeof(int) * 32 * 4, st));
    G.seq = 0;
  }

  void build_blk_m(DTri<T> &t, int Kw) {
    const int ki = ilog2(Kw), rpw = 32 / Kw;
    const int nl = (int)t.h_lvl.size() - 1;
    std::vector<int2> blk;
    blk.reserve((size_t)t.n / rpw + (size_t)std::max(nl, 0) + 1);
    for (int L = 0; L < nl; ++L)
      for (int p = t.h_lvl[L]; p < t.h_lvl[L + 1]; p += rpw)
        blk.push_back(make_int2(p, std::min(p + rpw, t.h_lvl[L + 1])));
    t.nblkm[ki] = (int)blk.size();
    t.blkm[ki] = marena.upload(blk);
    // as for the single-vector solve: a few dependency levels of blocks in flight
    const int per_level = (t.nblkm[ki] + nl - 1) / std::max(nl, 1);
    const int warps = std::max(32, std::min(4 * per_level, nsm * 32));
    t.gridm[ki] = (warps + 7) / 8;
  }
  template <int KK, int EE, bool PF>
  static int ell_occupancy() {
    int nb = 0;
    MLDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trsv_ell<T, KK, EE, PF>, 256, 0));
    return nb;
  }
  void build_ell(DTri<T> &t, int Kw, Arena &ar) {
    const int ki = ilog2(Kw), rpw = 32 / Kw;
    auto &el = t.ell[ki];
    el = typename DTri<T>::Ell();
    if (std::getenv("MLDG_NO_ELL")) return;
    const int nl = (int)t.h_lvl.size() - 1;
    int64_t npad = 0;
    for (int L = 0; L < nl; ++L) {
      const int cnt = t.h_lvl[L + 1] - t.h_lvl[L];
      npad += (cnt + rpw - 1) / rpw * rpw;
    }
    if (npad * 16 >= (int64_t)INT32_MAX) return;
    // level of every row (transformed index space) to order entries by dependency level
    std::vector<int> lev_of((size_t)t.n, 0);
    int emax = 0;
    for (int L = 0; L < nl; ++L)
      for (int p = t.h_lvl[L]; p < t.h_lvl[L + 1]; ++p) lev_of[t.h_prow[p]] = L;
    for (int p = 0; p < t.n; ++p) emax = std::max(emax, t.h_pirp[p + 1] - t.h_pirp[p]);
    // slots per row: the longest row rounded up to a power of two, at most 16
    // (measured best: wider slot sets cost registers and gained nothing);
    // longer rows spill their oldest dependencies to the overflow
    int ecap = 16;
    if (const char *e = std::getenv("MLDG_ELL_ECAP")) ecap = std::max(4, std::min(ecap, std::atoi(e)));
    int E = 4;
    while (E < emax && E < ecap) E *= 2;
    // padded positions: position -> schedule index (-1 = padding)
    std::vector<int> pos((size_t)npad, -1);
    {
      int64_t pp = 0;
      for (int L = 0; L < nl; ++L) {
        for (int p = t.h_lvl[L]; p < t.h_lvl[L + 1]; ++p) pos[pp++] = p;
        while (pp % rpw) ++pp;
      }
    }
    const int ntask = (int)(npad / rpw);
    std::vector<int2> toff((size_t)ntask);
    int64_t slots = 0;
    // one or two rows per task (K >= 16): uniform E slots, no per-task lookup
    const bool uniform = rpw <= 2;
    for (int tk = 0; tk < ntask; ++tk) {
      int et = 0;
      for (int g = 0; g < rpw; ++g) {
        const int p = pos[(size_t)tk * rpw + g];
        if (p >= 0) et = std::max(et, t.h_pirp[p + 1] - t.h_pirp[p]);
      }
      et = uniform ? E : std::min(et, E);
      toff[tk] = make_int2((int)slots, et);
      slots += (int64_t)et * rpw;
    }
    if (slots >= (int64_t)INT32_MAX) return;
    std::vector<int> prow((size_t)npad, -1), ej((size_t)std::max<int64_t>(slots, 1), -1),
        ovp((size_t)npad + 1, 0);
    std::vector<T> ev((size_t)std::max<int64_t>(slots, 1), T(0));
    // overflow offsets first (a prefix over the positions), then every
    // position fills its slots and overflow range independently
    for (int64_t pp = 0; pp < npad; ++pp) {
      const int p = pos[pp];
      int nov = 0;
      if (p >= 0) nov = std::max(0, t.h_pirp[p + 1] - t.h_pirp[p] - toff[(size_t)(pp / rpw)].y);
      ovp[pp + 1] = ovp[pp] + nov;
    }
    std::vector<int> ovj((size_t)ovp[npad]);
    std::vector<T> ovv((size_t)ovp[npad]);
#pragma omp parallel
    {
      std::vector<int> ord;
#pragma omp for schedule(static, 1024)
      for (int64_t pp = 0; pp < npad; ++pp) {
        const int p = pos[pp];
        if (p < 0) continue;
        const int tk = (int)(pp / rpw), g = (int)(pp % rpw), et = toff[tk].y;
        const int i = t.h_prow[p];
        prow[pp] = t.rev ? t.n - 1 - i : i;
        const int k0 = t.h_pirp[p], len = t.h_pirp[p + 1] - k0;
        ord.resize(len);
        for (int e = 0; e < len; ++e) ord[e] = k0 + e;
        std::stable_sort(ord.begin(), ord.end(),
                         [&](int x, int y) { return lev_of[t.h_pja[x]] < lev_of[t.h_pja[y]]; });
        const int nov = std::max(0, len - et);
        for (int e = 0; e < len; ++e) {
          const int k = ord[e], jj = t.h_pja[k];
          const int oj = t.rev ? t.n - 1 - jj : jj;
          if (e < nov) {
            ovj[(size_t)ovp[pp] + e] = oj;
            ovv[(size_t)ovp[pp] + e] = (T)t.h_pval[k];
          } else {
            const size_t q = (size_t)toff[tk].x + (size_t)(e - nov) * rpw + g;
            ej[q] = oj;
            ev[q] = (T)t.h_pval[k];
          }
        }
      }
    }
    el.npad = (int)npad;
    el.ntask = ntask;
    el.slots = slots;
    el.E = E;
    el.pf = E <= 8;
    if (const char *e = std::getenv("MLDG_ELL_PF")) el.pf = el.pf && e[0] != '0';
    el.S = Kw >= 16 ? 16 : 1;
    if (const char *e = std::getenv("MLDG_ELL_BACKOFF")) el.backoff = std::max(0, std::atoi(e));
    if (const char *e = std::getenv("MLDG_ELL_S")) el.S = std::max(1, std::min(64, std::atoi(e)));
    int nb = 0;
    ell_dispatch(Kw, E, el.pf, [&](auto kc, auto ec, auto pc) {
      nb = ell_occupancy<decltype(kc)::value, decltype(ec)::value, decltype(pc)::value>();
    });
    if (std::getenv("MLDG_VERBOSE"))
      std::fprintf(stderr,
                   "mldg: ell K=%d n=%d rev=%d levels=%d npad=%lld max row entries %d E=%d pf=%d slots %lld "
                   "(entries %lld) overflow %zu S=%d occ %d\n",
                   Kw, t.n, t.rev, nl, (long long)npad, emax, E, (int)el.pf, (long long)slots, (long long)t.nnz,
                   ovj.size(), el.S, nb);
    if (nb < 1) return;
    // every ticket stream needs running warps: grid <= co-resident capacity
    const int per_level = (el.ntask + nl - 1) / std::max(nl, 1);
    int mult = 4;
    if (const char *e = std::getenv("MLDG_ELL_MULT")) mult = std::max(1, std::atoi(e));
    const int64_t warps = std::max<int64_t>(32, std::min<int64_t>((int64_t)mult * per_level, el.ntask));
    el.grid = (int)std::min<int64_t>((warps + 7) / 8, (int64_t)nb * nsm);
    el.grid = std::max(el.grid, (el.S + 7) / 8);
    el.prow = ar.upload(prow);
    if (!uniform) el.toff = ar.upload(toff);
    el.ej = ar.upload(ej);
    el.ev = ar.upload(ev);
    if (!ovj.empty()) {
      el.ovp = ar.upload(ovp);
      el.ovj = ar.upload(ovj);
      el.ovv = ar.upload(ovv);
    }
    if (std::getenv("MLDG_ELL_TRACE")) {
      el.trace = ar.alloc<unsigned long long>((size_t)2 * el.ntask);
      MLDG_CUDA(cudaMemsetAsync(el.trace, 0, sizeof(unsigned long long) * 2 * el.ntask, st));
      el.h_task_level.resize(el.ntask);
      int64_t q = 0;
      for (int L = 0; L < nl; ++L) {
        const int cnt = t.h_lvl[L + 1] - t.h_lvl[L];
        for (int k = 0; k < (cnt + rpw - 1) / rpw; ++k) el.h_task_level[q++] = L;
      }
    }
    el.ctr = ar.alloc<int>((size_t)32 * (el.S + 1));
    MLDG_CUDA(cudaMemsetAsync(el.ctr, 0, sizeof(int) * 32 * (el.S + 1), st));
    el.ok = true;
  }
  // Explicit inverse M^{-1} = U^{-1} diag(d) L^{-1} of a small level's ILU(0)
  // (the operator of its solve pair), computed on the GPU 32 identity columns
  // at a time with the multi-column solves, and its transpose.  Kept when one
  // dense matrix-vector product beats the two dependency-bound solves.
  bool dense_inverse(Lev &L, Arena &ar) {
    const int n = L.n, Kw = 32, ki = 5;
    const bool gs = L.kind == MLDG_SMOOTHER_FBGS;
    if (n < 1 || L.minv || L.gsF || (L.kind != MLDG_SMOOTHER_BJAC && !gs)) return false;
    Arena tmp;
    bool ok = true;
    for (DTri<T> *f : {&L.L, &L.U}) {
      build_ell(*f, Kw, tmp);
      ok = ok && f->ell[ki].ok;
    }
    T *M = nullptr, *MT = nullptr;
    if (ok) {
      const size_t nk = (size_t)n * Kw;
      T *xm = tmp.alloc<T>(nk), *ym = tmp.alloc<T>(nk), *ba = tmp.alloc<T>(nk), *bb = tmp.alloc<T>(nk);
      k_fill<T><<<blocks_for((int64_t)nk), 256, 0, st>>>((int)nk, Sentinel<T>::value(), ba);
      k_fill<T><<<blocks_for((int64_t)nk), 256, 0, st>>>((int)nk, Sentinel<T>::value(), bb);
      M = ar.alloc<T>((size_t)n * n);
      MT = ar.alloc<T>((size_t)n * n);
      const int sK = K;
      K = Kw;
      for (int c0 = 0; c0 < n; c0 += Kw) {
        k_ident_block<T><<<blocks_for((int64_t)nk), 256, 0, st>>>(n, c0, Kw, xm);
        if (gs) {
          // columns of (D+L)^{-1} into M and of (D+U)^{-1} into MT (each exchange pair returns
          // to its start state: the second solve resets the first one's buffer)
          trsv_m(L.L, xm, L.d, ba, bb, ym, T(1), T(0));
          k_scatter_cols<T><<<blocks_for((int64_t)nk), 256, 0, st>>>(n, c0, Kw, ym, M);
          trsv_m(L.U, xm, L.d, bb, ba, ym, T(1), T(0));
          k_scatter_cols<T><<<blocks_for((int64_t)nk), 256, 0, st>>>(n, c0, Kw, ym, MT);
        } else {
          trsv_m(L.L, xm, nullptr, ba, bb, nullptr, T(1), T(0));
          trsv_m(L.U, ba, L.d, bb, ba, ym, T(1), T(0));
          k_scatter_cols<T><<<blocks_for((int64_t)nk), 256, 0, st>>>(n, c0, Kw, ym, M);
        }
      }
      K = sK;
      if (!gs) {
        dim3 tg((n + 31) / 32, (n + 31) / 32), tb(32, 8);
        k_transpose_sq<T><<<tg, tb, 0, st>>>(n, M, MT);
      }
      MLDG_CUDA(cudaStreamSynchronize(st));
    }
    for (DTri<T> *f : {&L.L, &L.U}) f->ell[ki] = typename DTri<T>::Ell();
    tmp.release();
    if (!ok) return false;  // no ELL plans to form the inverse with
    // keep the dense form only if it is faster
    auto op = [&]() {
      if (gs) {
        fbgs_solve(L, false, L.x, L.ty, T(0));
        fbgs_solve(L, true, L.x, L.ty, T(0));
      } else {
        ilu_apply(L, 'N', L.x, T(0), L.ty);
      }
    };
    auto set = [&](bool on) {
      if (gs) {
        L.gsF = on ? M : nullptr;
        L.gsB = on ? MT : nullptr;
      } else {
        L.minv = on ? M : nullptr;
        L.minvT = on ? MT : nullptr;
      }
    };
    cudaEvent_t e0, e1;
    MLDG_CUDA(cudaEventCreate(&e0));
    MLDG_CUDA(cudaEventCreate(&e1));
    float t[2] = {0, 0};
    for (int v = 0; v < 2; ++v) {
      set(v == 1);
      op();
      MLDG_CUDA(cudaEventRecord(e0, st));
      for (int r = 0; r < 3; ++r) op();
      MLDG_CUDA(cudaEventRecord(e1, st));
      MLDG_CUDA(cudaEventSynchronize(e1));
      MLDG_CUDA(cudaEventElapsedTime(&t[v], e0, e1));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (L.grp) reset_grp(L, 1);
    const bool keep = t[1] < t[0] || std::getenv("MLDG_DENSE_INV");
    set(keep);  // (rejected matrices stay in the arena until the handle is freed)
    if (std::getenv("MLDG_VERBOSE"))
      std::fprintf(stderr, "mldg: dense %s inverse n=%d: solves %.3f ms dense %.3f ms -> %s\n", gs ? "GS" : "ILU", n,
                   t[0] / 3, t[1] / 3, keep ? "dense" : "solves");
    launches = 0;
    bytes = 0;
    impl_bytes = 0;
    return keep;
  }
  // K-wide exchange buffers, all-sentinel (bufAm stays so after every solve pair)
  void exchange_m(Lev &L) {
    const size_t n = (size_t)std::max(L.n, 1) * mcap;
    L.bufAm = marena.alloc<T>(n);
    L.bufBm = marena.alloc<T>(n);
    k_fill<T><<<blocks_for((int64_t)n), 256, 0, st>>>((int)n, Sentinel<T>::value(), L.bufAm);
    k_fill<T><<<blocks_for((int64_t)n), 256, 0, st>>>((int)n, Sentinel<T>::value(), L.bufBm);
  }
  void release_multi() override {
    marena.release();
    mcap = 0;
    xin_m = yout_m = col_m = nullptr;
    for (auto &L : lv) {
      L.xm = L.ym = L.tym = L.twm = L.tzm = L.bufAm = L.bufBm = nullptr;
      L.gflip_m = 0;
      for (int q = 1; q < 6; ++q) L.g[q] = typename Lev::Grp();
      for (DTri<T> *t : {&L.L, &L.U, &L.Ut, &L.Lt})
        for (int q = 1; q < 6; ++q) {  // [0] (one column) lives in the main arena
          t->blkm[q] = nullptr;
          t->nblkm[q] = t->gridm[q] = 0;
          t->ell[q] = typename DTri<T>::Ell();
        }
    }
  }
  bool ensure_multi(int Kw, char trans) override {
    bool grown = false;
    if (Kw > mcap) {
      release_multi();
      mcap = Kw;
      const size_t n0 = (size_t)std::max(lv[0].n, 1);
      if ((int64_t)n0 * mcap >= (int64_t)INT32_MAX) fail(MLDG_ERR_SIZE, "n * nrhs too large");
      xin_m = marena.alloc<double>(n0 * mcap);
      yout_m = marena.alloc<double>(n0 * mcap);
      col_m = marena.alloc<double>(n0 * mcap);
      for (size_t l = 0; l < lv.size(); ++l) {
        Lev &L = lv[l];
        const size_t n = (size_t)std::max(L.n, 1) * mcap;
        if (l == 0 && std::is_same<T, double>::value) {
          L.xm = (T *)xin_m;
          L.ym = (T *)yout_m;
        } else {
          L.xm = marena.alloc<T>(n);
          L.ym = marena.alloc<T>(n);
        }
        L.tym = marena.alloc<T>(n);
        L.tzm = marena.alloc<T>(n);
        MLDG_CUDA(cudaMemsetAsync(L.tzm, 0, sizeof(T) * n, st));
        L.twm = marena.alloc<T>(n);
        MLDG_CUDA(cudaMemsetAsync(L.ym, 0, sizeof(T) * n, st));
        MLDG_CUDA(cudaMemsetAsync(L.tym, 0, sizeof(T) * n, st));
        MLDG_CUDA(cudaMemsetAsync(L.twm, 0, sizeof(T) * n, st));
        if ((L.kind == MLDG_SMOOTHER_BJAC || L.kind == MLDG_SMOOTHER_FBGS) && !L.minv &&
            !grp_for(L, mcap)) {
          exchange_m(L);
        }
      }
      grown = true;
    }
    const int ki = ilog2(Kw);
    for (auto &L : lv) {
      if ((L.kind != MLDG_SMOOTHER_BJAC && L.kind != MLDG_SMOOTHER_FBGS) || L.minv) continue;
      if (grp_for(L, Kw)) {
        if (L.g[ki].built(trans) || build_grp(L, Kw, trans, marena)) continue;
        L.g[ki].refused = true;
        grown = true;  // graphs that a width captured with the grouped solve are dropped
        if (!L.bufAm) exchange_m(L);
      }
      for (DTri<T> *t : {&L.L, &L.U, &L.Ut, &L.Lt}) {
        if (!t->present() && L.kind == MLDG_SMOOTHER_FBGS) continue;
        if (!t->present()) fail(MLDG_ERR_INTERNAL, "multi-RHS solve without a level schedule");
        if (!t->blkm[ki]) {
          build_blk_m(*t, Kw);
          build_ell(*t, Kw, marena);
        }
      }
    }
    MLDG_CUDA(cudaStreamSynchronize(st));
    return grown;
  }

  // K columns, and whether the lanes a row leaves share its entries: from 16
  // entries a row (restriction to 910 rows of 187 entries, 32 columns: 62 us
  // unsplit)
  template <typename F>
  static void spmm_dispatch(int K, int64_t nnz, int nr, F &&f) {
    kdispatch(K, [&](auto kc) {
      constexpr int SP = kSpmmSplit<T, decltype(kc)::value>;
      if (SP > 1 && nnz >= 16 * (int64_t)nr)
        f(kc, std::integral_constant<int, SP>());
      else
        f(kc, std::integral_constant<int, 1>());
    });
  }
  void spmm(const DCSR<T> &A, const T *v, T a1, const T *b, T a0, T *out, T a2) {
    begin(MLDG_KERNEL_SPMV);
    spmm_dispatch(K, A.nnz, A.nr, [&](auto kc, auto sp) {
      constexpr int KK = decltype(kc)::value, SP = decltype(sp)::value;
      k_spmm<T, KK, SP><<<blocks_for((int64_t)A.nr * (KK / kVecCols<T, KK>) * SP), 256, 0, st>>>(
          A.nr, A.irp, A.ja, A.val, v, a1, b, a0, out, a2);
    });
    end(A.nnz * (int64_t)(sizeof(T) + 4) + 4 * ((int64_t)A.nr + 1) + nk(A.nc) * (int64_t)sizeof(T) +
        nk(A.nr) * (int64_t)sizeof(T) * (1 + (b ? 1 : 0) + (a2 != T(0) ? 1 : 0)));
  }
  void jacobi_m(const DCSR<T> &ND, const T *d, const T *x, const T *ty, int first, T omega, T alpha, T beta,
                T *out) {
    begin(MLDG_KERNEL_JACOBI);
    spmm_dispatch(K, ND.nnz, ND.nr, [&](auto kc, auto sp) {
      constexpr int KK = decltype(kc)::value, SP = decltype(sp)::value;
      k_jacobi_m<T, KK, SP><<<blocks_for((int64_t)ND.nr * (KK / kVecCols<T, KK>) * SP), 256, 0, st>>>(
          ND.nr, ND.irp, ND.ja, ND.val, d, x, ty, first, omega, alpha, beta, out);
    });
    end(ND.nnz * (int64_t)(sizeof(T) + 4) + 4 * ((int64_t)ND.nr + 1) + (int64_t)ND.nr * sizeof(T) +
        nk(ND.nr) * (int64_t)sizeof(T) * (2 + (first ? 0 : 1) + (beta != T(0) ? 1 : 0)));
  }
  void diag_m(int n, const T *d, const T *x, T alpha, T beta, T *out) {
    begin(MLDG_KERNEL_VEC);
    kdispatch(K, [&](auto kc) {
      constexpr int KK = decltype(kc)::value;
      k_diag_m<T, KK><<<blocks_for(nk(n)), 256, 0, st>>>(n, d, x, alpha, beta, out);
    });
    end((int64_t)n * sizeof(T) + nk(n) * (int64_t)sizeof(T) * (2 + (beta != T(0) ? 1 : 0)));
  }
  void fill_m(int n, T v, T *y) {
    begin(MLDG_KERNEL_VEC);
    k_fill<T><<<blocks_for(nk(n)), 256, 0, st>>>((int)nk(n), v, y);
    end(nk(n) * (int64_t)sizeof(T));
  }
  void axpby_m(int n, const T *x, T beta, T *y) {
    begin(MLDG_KERNEL_VEC);
    k_axpby1<T><<<blocks_for(nk(n)), 256, 0, st>>>((int)nk(n), x, beta, y);
    end(nk(n) * (int64_t)sizeof(T) * (2 + (beta != T(0))));
  }
  void trsv_m(DTri<T> &t, const T *rhs, const T *scale, T *cur, T *other, T *out, T alpha, T beta) {
    TriArgs<T> a;
    a.n = t.n;
    a.rev = t.rev;
    a.nlevels = t.nlevels;
    a.lvl_ptr = t.lvl_ptr;
    a.prow = t.prow;
    a.pirp = t.pirp;
    a.pja = t.pja;
    a.pval = t.pval;
    a.rhs_src = rhs;
    a.rhs_scale = scale;
    a.cur = cur;
    a.other = other;
    a.out = out;
    a.alpha = alpha;
    a.beta = beta;
    a.counters = t.counters;
    a.err = err;
    a.nblk = 0;
    a.blk = nullptr;
    const int ki = ilog2(K);
    begin(MLDG_KERNEL_TRSV);
    const auto &el = t.ell[ki];
    if (el.ok) {
      launch_ell(el, K, rhs, scale, cur, other, out, alpha, beta);
    } else {
      kdispatch(K, [&](auto kc) {
        constexpr int KK = decltype(kc)::value;
        k_trsv_sf_m<T, KK><<<t.gridm[ki], 256, 0, st>>>(a, t.nblkm[ki], t.blkm[ki]);
      });
    }
    end(t.nnz * (int64_t)(sizeof(T) + 4) + 4 * (2 * (int64_t)t.n + 1) + (scale ? (int64_t)t.n * sizeof(T) : 0) +
        nk(t.n) * (int64_t)sizeof(T) * (1 + 1 + (other ? 1 : 0) + (out ? 1 + (beta != T(0)) : 0)));
  }
  void launch_ell(const typename DTri<T>::Ell &el, int Kw, const T *rhs, const T *scale, T *cur, T *other, T *out,
                  T alpha, T beta) {
    {
      EllArgs<T> e;
      e.ntask = el.ntask;
      e.npad = el.npad;
      e.toff = el.toff;
      e.S = el.S;
      e.backoff = el.backoff;
      e.prow = el.prow;
      e.ej = el.ej;
      e.ev = el.ev;
      e.ovp = el.ovp;
      e.ovj = el.ovj;
      e.ovv = el.ovv;
      e.ctr = el.ctr;
      e.trace = el.trace;
      e.rhs_src = rhs;
      e.rhs_scale = scale;
      e.cur = cur;
      e.other = other;
      e.out = out;
      e.alpha = alpha;
      e.beta = beta;
      e.err = err;
      ell_dispatch(Kw, el.E, el.pf, [&](auto kc, auto ec, auto pc) {
        k_trsv_ell<T, decltype(kc)::value, decltype(ec)::value, decltype(pc)::value><<<el.grid, 256, 0, st>>>(e);
      });
    }
  }
  // out = M x + beta*out, M dense n x n (a level's explicit inverse)
  void gemm_m(int n, const T *M, const T *x, T beta, T *out) {
    kdispatch(K, [&](auto kc) {
      constexpr int KK = decltype(kc)::value;
      if constexpr (KK <= 8)
        k_gemm_m_rows<T, KK><<<std::max(1, std::min((n * KK + 127) / 128, nsm * 16)), 128, 0, st>>>(n, M, x, T(1), beta,
                                                                                                 out);
      else
        k_gemm_m_cols<T, KK><<<std::max(1, std::min((n * KK + 127) / 128, nsm * 8)), 256, 0, st>>>(n, M, x, T(1), beta,
                                                                                                out);
    });
  }
  void ilu_apply_m(Lev &L, char trans, const T *x, T beta, T *y) {
    if (L.minv) {
      const T *M = (trans == 'N') ? L.minv : L.minvT;
      begin(MLDG_KERNEL_VEC);
      gemm_m(L.n, M, x, beta, y);
      end((int64_t)L.n * L.n * sizeof(T) + nk(L.n) * (int64_t)sizeof(T) * (2 + (beta != T(0))),
          (L.nnz_l + L.nnz_u) * (int64_t)(sizeof(T) + 4) + 8 * ((int64_t)L.n + 1) +
              (int64_t)L.n * sizeof(T) + nk(L.n) * (int64_t)sizeof(T) * (2 + (beta != T(0))));
      return;
    }
    if (grp_for(L, K)) {
      gpair(L, K, trans, x, beta, y);
      return;
    }
    if (trans == 'N') {
      trsv_m(L.L, x, nullptr, L.bufAm, L.bufBm, nullptr, T(1), T(0));
      trsv_m(L.U, L.bufAm, L.d, L.bufBm, L.bufAm, y, T(1), beta);
    } else {
      trsv_m(L.Ut, x, nullptr, L.bufAm, L.bufBm, nullptr, T(1), T(0));
      trsv_m(L.Lt, L.bufAm, L.d, L.bufBm, L.bufAm, y, T(1), beta);
    }
  }
  // K-wide fbgs_solve / end_fbgs / fbgs_smoother
  void fbgs_solve_m(Lev &L, bool backward, const T *rhs, T *out, T beta) {
    if (L.gsF) {
      const T *M = backward ? L.gsB : L.gsF;
      begin(MLDG_KERNEL_VEC);
      gemm_m(L.n, M, rhs, beta, out);
      end((int64_t)L.n * L.n * sizeof(T) + nk(L.n) * (int64_t)sizeof(T) * (2 + (beta != T(0))),
          (backward ? L.nnz_u : L.nnz_l) * (int64_t)(sizeof(T) + 4) + 4 * ((int64_t)L.n + 1) +
              (int64_t)L.n * sizeof(T) + nk(L.n) * (int64_t)sizeof(T) * (2 + (beta != T(0))));
      return;
    }
    if (grp_for(L, K)) {
      auto &G = L.g[ilog2(K)];
      gsolve(G, backward ? G.U : G.L, K, backward ? L.nnz_u : L.nnz_l, rhs, out, beta);
      return;
    }
    DTri<T> &t = backward ? L.U : L.L;
    T *cur = L.gflip_m ? L.bufBm : L.bufAm, *other = L.gflip_m ? L.bufAm : L.bufBm;
    L.gflip_m ^= 1;
    trsv_m(t, rhs, L.d, cur, other, out, T(1), beta);
  }
  void end_fbgs_m() {
    for (auto &L : lv)
      if (L.kind == MLDG_SMOOTHER_FBGS && L.gflip_m) {
        // the whole allocated width: every K keeps bufAm all-sentinel
        begin(MLDG_KERNEL_VEC);
        const int64_t nn = (int64_t)std::max(L.n, 1) * mcap;
        k_fill<T><<<blocks_for(nn), 256, 0, st>>>((int)nn, Sentinel<T>::value(), L.bufAm);
        end(nn * (int64_t)sizeof(T));
        L.gflip_m = 0;
      }
  }
  void fbgs_smoother_m(Lev &L, bool post, const T *x, T beta, T *y, int sweeps) {
    if (sweeps == 1) {
      fbgs_solve_m(L, post, x, y, beta);
      return;
    }
    fbgs_solve_m(L, post, x, L.tzm, T(0));
    for (int s = 1; s < sweeps; ++s) {
      spmm(post ? L.GL : L.GU, L.tzm, T(-1), x, T(1), L.twm, T(0));
      fbgs_solve_m(L, post, L.twm, L.tzm, T(0));
    }
    axpby_m(L.n, L.tzm, beta, y);
  }
  // the single-vector smoother() with K-wide kernels
  void smoother_m(Lev &L, char trans, const T *x, T beta, T *y, int sweeps, bool post = false) {
    if (L.kind == MLDG_SMOOTHER_FBGS) {
      fbgs_smoother_m(L, post, x, beta, y, sweeps);
      return;
    }
    const DCSR<T> &ND = (trans == 'N') ? L.ND : L.NDT;
    if (L.kind == MLDG_SMOOTHER_BJAC) {
      if (sweeps == 1 || L.nnz_nd == 0) {
        ilu_apply_m(L, trans, x, beta, y);
        return;
      }
      ilu_apply_m(L, trans, x, T(0), L.tzm);
      for (int s = 1; s < sweeps; ++s) {
        spmm(ND, L.tzm, T(-1), x, T(1), L.twm, T(0));
        ilu_apply_m(L, trans, L.twm, T(0), L.tzm);
      }
      axpby_m(L.n, L.tzm, beta, y);
      return;
    }
    const T w = (T)L.damp;
    if (sweeps == 1 || L.nnz_nd == 0) {
      diag_m(L.n, L.d, x, w, beta, y);
      return;
    }
    T *src = nullptr;
    T *bufs[2] = {L.tzm, L.twm};
    for (int s = 1; s < sweeps; ++s) {
      const bool last = (s == sweeps - 1);
      T *dst = last ? y : bufs[s & 1];
      jacobi_m(ND, L.d, x, src, s == 1 ? (L.nd_scaled ? 2 : 1) : 0, w, T(1), last ? beta : T(0), dst);
      src = dst;
    }
  }
  void prolong_m(Lev &C, T *y) {
    if constexpr (std::is_same<T, float>::value) {
      if (C.Ph) {
        begin(MLDG_KERNEL_SPMV);
        kdispatch(K, [&](auto kc) {
          constexpr int KK = decltype(kc)::value;
          k_spmm_h<KK><<<blocks_for(nk(C.P.nr)), 256, 0, st>>>(C.P.nr, C.P.irp, C.P.ja, C.Ph, C.Pscale, C.ym, y);
        });
        end(C.P.nnz * 6 + 4 * ((int64_t)C.P.nr + 1) + (int64_t)C.P.nr * 4 + nk(C.P.nc) * 4 + nk(C.P.nr) * 4 * 2);
        return;
      }
    }
    spmm(C.P, C.ym, T(1), nullptr, T(0), y, T(1));
  }
  // the single-vector vcycle() with K-wide kernels
  void vcycle_m(int l, char trans) {
    cur_lev = l;
    Lev &L = lv[l];
    const int nlev = (int)lv.size();
    const bool pre = (L.spre > 0 && trans == 'N') || (L.spost > 0 && trans != 'N');
    const bool post = (L.spost > 0 && trans == 'N') || (L.spre > 0 && trans != 'N');
    if (l < nlev - 1) {
      Lev &C = lv[l + 1];
      const DCSR<T> &A = (trans == 'N') ? L.A : L.AT;
      if (pre) {
        smoother_m(L, trans, L.xm, T(0), L.ym, trans == 'N' ? L.spre : L.spost, trans != 'N');
        spmm(A, L.ym, T(-1), L.xm, T(1), L.tym, T(0));
        spmm(C.R, L.tym, T(1), nullptr, T(0), C.xm, T(0));
      } else {
        fill_m(L.n, T(0), L.ym);
        spmm(C.R, L.xm, T(1), nullptr, T(0), C.xm, T(0));
      }
      vcycle_m(l + 1, trans);
      cur_lev = l;
      prolong_m(C, L.ym);
      if (cycle == MLDG_CYCLE_W) {
        spmm(A, L.ym, T(-1), L.xm, T(1), L.tym, T(0));
        spmm(C.R, L.tym, T(1), nullptr, T(0), C.xm, T(0));
        vcycle_m(l + 1, trans);
        cur_lev = l;
        prolong_m(C, L.ym);
      }
      if (post) {
        spmm(A, L.ym, T(-1), L.xm, T(1), L.tym, T(0));
        smoother_m(L, trans, L.tym, T(1), L.ym, trans == 'N' ? L.spost : L.spre, trans == 'N');
      }
    } else {
      smoother_m(L, trans, L.xm, T(0), L.ym, L.spre);
    }
  }
  void addcycle_m(int l, char trans) {
    cur_lev = l;
    Lev &L = lv[l];
    if (L.kind == MLDG_SMOOTHER_FBGS) {
      axpby_m(L.n, L.xm, T(0), L.ym);
      for (int k = 0; k < std::max(L.spre, L.spost); ++k) {
        fbgs_solve_m(L, false, L.ym, L.twm, T(0));
        fbgs_solve_m(L, true, L.twm, L.ym, T(0));
      }
    } else {
      smoother_m(L, trans, L.xm, T(0), L.ym, L.spre);
    }
    if (l < (int)lv.size() - 1) {
      Lev &C = lv[l + 1];
      spmm(C.R, L.xm, T(1), nullptr, T(0), C.xm, T(0));
      addcycle_m(l + 1, trans);
      cur_lev = l;
      prolong_m(C, L.ym);
    }
  }
  void record_multi(char trans, int Kw) override {
    if (Kw > mcap) fail(MLDG_ERR_INTERNAL, "multi buffers not allocated for %d columns", Kw);
    if (kcycle_mode()) fail(MLDG_ERR_ARG, "the K-cycle has no multi-column form");
    launches = 0;
    bytes = 0;
    impl_bytes = 0;
    cur_lev = 0;
    probe_armed = false;
    std::memset(seen, 0, sizeof seen);
    K = Kw;
    for (auto &L : lv) L.g[ilog2(Kw)].seq = 0;
    Lev &F = lv[0];
    const int64_t n = nk(F.n);
    if (!std::is_same<T, double>::value) {
      begin(MLDG_KERNEL_VEC);
      k_cast<double, T><<<blocks_for(n), 256, 0, st>>>((int)n, xin_m, F.xm);
      end(n * (8 + (int64_t)sizeof(T)));
    }
    if (lv.size() == 1 && F.kind == MLDG_SMOOTHER_FBGS) {
      const int nsw = std::max(F.spre, F.spost);
      const T *src = F.xm;
      for (int k = 0; k < nsw; ++k) {
        fbgs_solve_m(F, false, src, F.tym, T(0));
        fbgs_solve_m(F, true, F.tym, k == nsw - 1 ? F.ym : F.twm, T(0));
        src = F.twm;
      }
      if (nsw == 0) axpby_m(F.n, F.xm, T(0), F.ym);
    } else if (lv.size() == 1) {
      smoother_m(F, trans, F.xm, T(0), F.ym, F.spre);
    } else if (cycle == MLDG_CYCLE_ADD) {
      addcycle_m(0, trans);
    } else {
      vcycle_m(0, trans);
    }
    end_fbgs_m();
    end_grp(Kw);
    if (!std::is_same<T, double>::value) {
      cur_lev = 0;
      begin(MLDG_KERNEL_VEC);
      k_cast<T, double><<<blocks_for(n), 256, 0, st>>>((int)n, F.ym, yout_m);
      end(n * (8 + (int64_t)sizeof(T)));
    }
  }

  // per-level timing of the last ELL solve of each factor (MLDG_ELL_TRACE)
  void dump_ell_trace() {
    for (size_t l = 0; l < lv.size(); ++l) {
      const DTri<T> *fs[4] = {&lv[l].L, &lv[l].U, &lv[l].Ut, &lv[l].Lt};
      const char *nm[4] = {"L", "U", "Ut", "Lt"};
      for (int q = 0; q < 4; ++q)
        for (int ki = 0; ki < 6; ++ki) {
          const auto &el = fs[q]->ell[ki];
          if (!el.ok || !el.trace) continue;
          std::vector<unsigned long long> tr((size_t)2 * el.ntask);
          cudaMemcpy(tr.data(), el.trace, tr.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
          const int nl = el.h_task_level.empty() ? 0 : el.h_task_level.back() + 1;
          std::vector<unsigned long long> lend(nl, 0), lbeg_min(nl, ~0ull), lbeg_max(nl, 0);
          double dur = 0;
          unsigned long long t_first = ~0ull;
          for (int t = 0; t < el.ntask; ++t) {
            const int L = el.h_task_level[t];
            lend[L] = std::max(lend[L], tr[2 * t + 1]);
            lbeg_min[L] = std::min(lbeg_min[L], tr[2 * t]);
            lbeg_max[L] = std::max(lbeg_max[L], tr[2 * t]);
            dur += (double)(tr[2 * t + 1] - tr[2 * t]);
            t_first = std::min(t_first, tr[2 * t]);
          }
          double step = 0, lag_last = 0, spread = 0;
          for (int L = 1; L < nl; ++L) {
            step += (double)(lend[L] - lend[L - 1]);
            // how long after level L-1 completed did level L's last task start
            lag_last += (double)lbeg_max[L] - (double)lend[L - 1];
            spread += (double)(lend[L] - lbeg_max[L]);
          }
          std::fprintf(stderr,
                       "mldg ell trace: level %zu %s K=%d tasks %d levels %d total %.1f us: per level %.0f ns "
                       "(last task start - prev level end %.0f ns, last start -> level end %.0f ns), "
                       "task duration avg %.0f ns\n",
                       l, nm[q], 1 << ki, el.ntask, nl, (lend[nl - 1] - t_first) * 1e-3,
                       nl > 1 ? step / (nl - 1) : 0.0, nl > 1 ? lag_last / (nl - 1) : 0.0,
                       nl > 1 ? spread / (nl - 1) : 0.0, dur / el.ntask);
        }
    }
  }
  void dump_trace() override {
    dump_ell_trace();
    for (size_t l = 0; l < lv.size(); ++l) {
      const DRep<T> *rs[4] = {&lv[l].rL, &lv[l].rU, &lv[l].rUt, &lv[l].rLt};
      for (int q = 0; q < 4; ++q) {
        if (!rs[q]->trace) continue;
        unsigned long long t[20] = {0};
        cudaMemcpy(t, rs[q]->trace, 20 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
        for (int th = 0; th < 2; ++th) {
          const unsigned long long *u = t + 10 * th;
          if (!u[7]) continue;
          const double k = (double)u[7];
          std::fprintf(stderr,
                       "mldg trace: level %zu rep%d C=%d group %d steps %llu: cycles/step wait(s-2) %.0f mid %.0f "
                       "wait(s-1) %.0f critical %.0f outputs %.0f sync %.0f prepare %.0f | kernel cycles/step %.0f "
                       "ns/step %.0f\n",
                       l, q, rs[q]->C, th, u[7], u[0] / k, u[1] / k, u[2] / k, u[3] / k, u[4] / k, u[5] / k,
                       u[6] / k, u[8] / k, u[9] / k);
        }
      }
    }
    for (size_t l = 0; l < lv.size(); ++l) {
      if (!lv[l].win) continue;
      const DWin<T> *ws[4] = {&lv[l].wL, &lv[l].wU, &lv[l].wUt, &lv[l].wLt};
      for (int q = 0; q < 4; ++q) {
        if (!ws[q]->trace) continue;
        unsigned long long t[16] = {0};
        cudaMemcpy(t, ws[q]->trace, 16 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
        if (!t[4]) continue;
        std::fprintf(stderr,
                     "mldg trace: level %zu win%d C=%d steps %llu: cycles/step wait %.0f compute %.0f barrier %.0f | "
                     "kernel cycles/step %.0f ns/step %.0f (clock %.0f MHz) loop cycles/step %.0f prologue cycles/step %.0f\n",
                     l, q, ws[q]->C, t[4], (double)t[0] / t[4], (double)t[1] / t[4], (double)t[2] / t[4],
                     (double)t[5] / t[4], (double)t[6] / t[4], t[6] ? 1e3 * (double)t[5] / (double)t[6] : 0.0,
                     (double)t[7] / t[4], (double)t[8] / t[4]);
      }
    }
  }

  void record(char trans) override {
    launches = 0;
    bytes = 0;
    impl_bytes = 0;
    cur_lev = 0;
    probe_armed = false;
    std::memset(seen, 0, sizeof seen);
    for (auto &L : lv) L.g[0].seq = 0;
    Lev &F = lv[0];
    if (!std::is_same<T, double>::value && !kry_io) {
      begin(MLDG_KERNEL_VEC);
      cast(F.n, xin, F.x);
      end((int64_t)F.n * (8 + sizeof(T)));
    }
    if (lv.size() == 1 && F.kind == MLDG_SMOOTHER_FBGS) {
      // one level: nswps times forward then backward GS, one sweep each
      const int nsw = std::max(F.spre, F.spost);
      const T *src = F.x;
      for (int k = 0; k < nsw; ++k) {
        fbgs_solve(F, false, src, F.ty, T(0));
        fbgs_solve(F, true, F.ty, k == nsw - 1 ? F.y : F.tw, T(0));
        src = F.tw;
      }
      if (nsw == 0) k_axpby_impl(F.n, F.x, T(0), F.y);
    } else if (lv.size() == 1) {
      smoother(F, trans, F.x, T(0), F.y, F.spre);
    } else if (kcycle_mode()) {
      ensure_k();
      kcycle(0, trans);
    } else if (cycle == MLDG_CYCLE_ADD) {
      addcycle(0, trans);
    } else {
      vcycle(0, trans);
    }
    end_fbgs();
    end_grp(1);
    if (!std::is_same<T, double>::value && !kry_io) {
      cur_lev = 0;
      begin(MLDG_KERNEL_VEC);
      cast(F.n, F.y, yout);
      end((int64_t)F.n * (8 + sizeof(T)));
    }
  }
};

template <typename T>
void EngineT<T>::k_axpby_impl(int n, const T *x, T beta, T *y) {
  begin(MLDG_KERNEL_VEC);
  kl(k_axpby1<T>, blocks_for(n), 256, n, x, beta, y);
  end((int64_t)n * sizeof(T) * (2 + (beta != T(0))));
}

template <typename T>
void EngineT<T>::prolong(Lev &C, T *y) {
  spmv(C.P, C.y, T(1), nullptr, T(0), y, T(1));
}

template <>
void EngineT<float>::prolong(Lev &C, float *y) {
  if (!C.Ph) {
    spmv(C.P, C.y, 1.f, nullptr, 0.f, y, 1.f);
    return;
  }
  const int g = blocks_for((int64_t)C.P.nr * C.P.tpr);
  begin(MLDG_KERNEL_SPMV);
  switch (C.P.tpr) {
#define CASE(K) \
  case K: kl(k_spmv_h<K>, g, 256, C.P.nr, C.P.irp, C.P.ja, C.Ph, C.Pscale, C.y, y); break;
    CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32)
#undef CASE
    default: fail(MLDG_ERR_INTERNAL, "bad tpr");
  }
  end(C.P.nnz * 6 + 4 * ((int64_t)C.P.nr + 1) + (int64_t)C.P.nc * 4 + (int64_t)C.P.nr * 4 * 3);
}

// ---------------------------------------------------------------------------
struct Handle {
  mldg_opts opts{};
  // the CG/FCG kernels being recorded read z in FP32 and write the FP32 copy
  // of r (Engine::kry_io); set while a whole solve or a batch is captured
  bool kio = false;
  // changes at every finalize and destroy: identifies the finalized state
  // that a cached batch graph was captured from
  uint64_t serial = 0;
  int cycle = MLDG_CYCLE_V;
  bool has_fbgs = false;  // a Gauss-Seidel level: trans 'T' is rejected
  std::string last_error;
  std::vector<HostLevel> host;
  int nlev = 0;
  int precision = MLDG_PREC_FP64;
  bool finalized = false;
  Arena arena;
  cudaStream_t st = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::unique_ptr<Engine> eng;
  int *err = nullptr;
  double *xin = nullptr, *yout = nullptr;
  int n0 = 0;
  // graphs per trans
  cudaGraphExec_t gexec[2] = {nullptr, nullptr};
  int64_t glaunch[2] = {0, 0}, gbytes[2] = {0, 0}, gimpl[2] = {0, 0};
  // Krylov state (FP64)
  DCSR<double> A0, A0T;
  // FP64 Krylov state: b, x, the two alternating direction buffers, q = A d,
  // per-block partial sums, the device scalars (KState) and the parameters
  // of the current solve, with pinned host mirrors of both
  double *kb = nullptr, *kx = nullptr, *kd = nullptr, *kd1 = nullptr, *kq = nullptr, *kpart = nullptr;
  KState *kst = nullptr, *hkst = nullptr;
  KParams *kpar = nullptr, *hkpar = nullptr;
  double *hpin = nullptr;  // pinned host scalar mirror
  double last_ms = 0;
  int64_t last_launches = 0;
  int nsm = 148;
  // probe (see mldg_probe_set)
  int probe_kind = 0, probe_lev = 0, probe_idx = 0;
  cudaEvent_t pev0 = nullptr, pev1 = nullptr;
  bool gprobe[2] = {false, false};
  bool pending = false;  // a probed launch was issued and not yet read
  double probe_ms = 0;
  int64_t probe_count = 0, probe_bytes = 0;
  // multi-RHS V-cycle graphs per (trans, log2 K) and the K-wide FP64 Krylov state
  cudaGraphExec_t gexec_m[2][6] = {};
  int64_t glaunch_m[2][6] = {};
  bool gprobe_m[2][6] = {};
  Arena karena;
  int kcap = 0;
  double *kb_m = nullptr, *kx_m = nullptr, *kd_m = nullptr, *kq_m = nullptr, *kpart_m = nullptr;
  KrylovM *ksc_m = nullptr, *hksc_m = nullptr;  // device state, pinned host mirror
  // one whole CG/FCG solve per [method][trans] as a CUDA graph: the initial
  // residual, then a conditional WHILE node repeating V-cycle + iteration
  // until the device-side stopping test clears it; launches of the prefix and
  // of one loop body
  cudaGraphExec_t sgraph[2][2] = {};
  int64_t sglaunch_pre[2][2] = {}, sglaunch_body[2][2] = {};
};

// the GS solvers accept trans = 'N' only (mld_d_gs_solver_apply_vect.f90:68-75)
static void check_trans(const Handle *h, char trans) {
  if (trans != 'N' && h->has_fbgs)
    fail(MLDG_ERR_TRANS, "trans '%c': the Gauss-Seidel smoother (FBGS) applies with trans 'N' only", trans);
}

static void drop_krylov_graphs(Handle *h) {
  for (int m = 0; m < 2; ++m)
    for (int t = 0; t < 2; ++t)
      if (h->sgraph[m][t]) {
        cudaGraphExecDestroy(h->sgraph[m][t]);
        h->sgraph[m][t] = nullptr;
      }
}

static void drop_multi_graphs(Handle *h) {
  for (int t = 0; t < 2; ++t)
    for (int q = 0; q < 6; ++q)
      if (h->gexec_m[t][q]) {
        cudaGraphExecDestroy(h->gexec_m[t][q]);
        h->gexec_m[t][q] = nullptr;
      }
}

// dispatch over (kernel, lanes per row, prefetched entries per lane)
template <typename T, int TPR, int E>
static void launch_trsv_te(const DTri<T> &t, const TriArgs<T> &a, cudaStream_t st) {
  if (t.cta)
    k_trsv_cta<T, TPR, E><<<1, t.threads, t.smem, st>>>(a);
  else
    k_trsv_sf<T, TPR, E><<<t.grid, t.threads, 0, st>>>(a);
}
template <typename T, int TPR>
static void launch_trsv_t(const DTri<T> &t, const TriArgs<T> &a, cudaStream_t st) {
  if (t.mode == 0) {
    if (t.stg.D == 3)
      k_trsv_stg<T, TPR, 3><<<1, t.threads, t.smem, st>>>(a, t.stg, t.desc);
    else if (t.stg.D == 4)
      k_trsv_stg<T, TPR, 4><<<1, t.threads, t.smem, st>>>(a, t.stg, t.desc);
    else
      k_trsv_stg<T, TPR, 6><<<1, t.threads, t.smem, st>>>(a, t.stg, t.desc);
    return;
  }
  if (t.e <= 4)
    launch_trsv_te<T, TPR, 4>(t, a, st);
  else
    launch_trsv_te<T, TPR, 8>(t, a, st);
}
template <typename T>
static void launch_trsv(const DTri<T> &t, const TriArgs<T> &a, cudaStream_t st) {
  switch (t.tpr) {
    case 1: launch_trsv_t<T, 1>(t, a, st); break;
    case 2: launch_trsv_t<T, 2>(t, a, st); break;
    case 4: launch_trsv_t<T, 4>(t, a, st); break;
    case 8: launch_trsv_t<T, 8>(t, a, st); break;
    case 16: launch_trsv_t<T, 16>(t, a, st); break;
    default: launch_trsv_t<T, 32>(t, a, st); break;
  }
}

// Levels with at most this many rows use the single-CTA kernel (the whole
// solution vector in shared memory: 128 KB).
template <typename T>
constexpr int tri_cta_rows() {
  return (int)(128 * 1024 / sizeof(T));
}

// dynamic shared memory of k_trsv_win: 227 KB per block minus its static part
constexpr int kWinSmemMax = 227 * 1024 - 1024;

// Builds the step plan of k_trsv_win for a cluster of C CTAs; returns a plan
// with ok == false when the window cannot hold every dependency or the shared
// memory budget cannot fit the stages.
template <typename T>
static DWin<T> build_win_plan(const HostCSR &m, bool upper, int C) {
  DWin<T> w;
  const int n = m.nr;
  if (n <= 0) return w;
  TriSchedule s;
  build_tri_schedule(n, m.irp.data(), m.ja.data(), m.val.data(), upper, n, &s);
  const int nlev = (int)s.lvl_ptr.size() - 1;
  std::vector<int> posof((size_t)n);
  for (int p = 0; p < n; ++p) posof[s.prow[p]] = p;
  w.n = n;
  w.C = C;
  w.nnz = m.nnz();
  w.h_orig.resize((size_t)n);
  w.h_pos.resize((size_t)n);
  for (int p = 0; p < n; ++p) {
    w.h_orig[p] = upper ? n - 1 - s.prow[p] : s.prow[p];
    w.h_pos[w.h_orig[p]] = p;
  }
  // window: every dependency q of a row in step [sp0, sp1) needs q >= sp1 - W;
  // steps end no later than their level, so the level end bounds the span
  int span = 1;
  for (int L = 0; L < nlev; ++L) {
    const int p1 = s.lvl_ptr[L + 1];
    for (int p = s.lvl_ptr[L]; p < p1; ++p)
      for (int k = s.pirp[p]; k < s.pirp[p + 1]; ++k) span = std::max(span, p1 - posof[s.pja[k]]);
  }
  int W = 32 * C;
  while (W < span + 1) W <<= 1;
  const size_t budget = kWinSmemMax;
  const size_t win_bytes = (size_t)(W / C) * sizeof(T);
  if (win_bytes + 32 * 1024 > budget) return w;
  // capacities: the largest CTA slice of any level with one part per level
  int maxr = 0, maxe = 0;
  for (int L = 0; L < nlev; ++L) {
    const int p0 = s.lvl_ptr[L], p1 = s.lvl_ptr[L + 1], nr = p1 - p0;
    for (int cc = 0; cc < C; ++cc) {
      const int a = p0 + (int)((int64_t)nr * cc / C), b = p0 + (int)((int64_t)nr * (cc + 1) / C);
      maxr = std::max(maxr, b - a);
      maxe = std::max(maxe, s.pirp[b] - s.pirp[a]);
    }
  }
  int capR = std::max(maxr, 1), capE = std::max(maxe, 1);
  int D = 0;
  std::vector<WinDesc> desc;
  std::vector<int> stepends;
  for (int attempt = 0; attempt < 12; ++attempt) {
    // steps: split each level into parts whose CTA slices fit (capR, capE)
    desc.clear();
    stepends.clear();
    bool fits = true;
    for (int L = 0; L < nlev && fits; ++L) {
      const int p0 = s.lvl_ptr[L], p1 = s.lvl_ptr[L + 1], nr = p1 - p0;
      const int ne = s.pirp[p1] - s.pirp[p0];
      int k = std::max(1, std::max((nr + C * capR - 1) / (C * capR), (ne + C * capE - 1) / (C * capE)));
      for (;; ++k) {
        bool good = true;
        for (int j = 0; j < k && good; ++j) {
          const int a0 = p0 + (int)((int64_t)nr * j / k), b0 = p0 + (int)((int64_t)nr * (j + 1) / k);
          for (int cc = 0; cc < C && good; ++cc) {
            const int a = a0 + (int)((int64_t)(b0 - a0) * cc / C), b = a0 + (int)((int64_t)(b0 - a0) * (cc + 1) / C);
            good = (b - a) <= capR && (s.pirp[b] - s.pirp[a]) <= capE;
          }
        }
        if (good) break;
        if (k > nr) {
          fits = false;
          break;
        }
      }
      if (!fits) break;
      for (int j = 0; j < k; ++j) {
        const int a0 = p0 + (int)((int64_t)nr * j / k), b0 = p0 + (int)((int64_t)nr * (j + 1) / k);
        for (int cc = 0; cc < C; ++cc) {
          const int a = a0 + (int)((int64_t)(b0 - a0) * cc / C), b = a0 + (int)((int64_t)(b0 - a0) * (cc + 1) / C);
          desc.push_back(WinDesc{a, b, s.pirp[a], s.pirp[b]});
        }
        stepends.push_back(b0);
      }
    }
    const int nsteps = (int)stepends.size();
    const StageLayout lay = stage_layout<T>(capR, capE);
    const size_t fixed = (size_t)al16((int)win_bytes) + (size_t)al16(nsteps * 16) + 64;
    D = 0;
    if (fits)
      for (int d : {4, 3})
        if (fixed + (size_t)d * lay.bytes <= budget) {
          D = d;
          break;
        }
    if (D) break;
    capR = std::max(1, capR / 2);
    capE = std::max(1, capE / 2);
  }
  if (!D) return w;
  // window check
  {
    int st = 0;
    for (int p = 0; p < n; ++p) {
      while (stepends[st] <= p) ++st;
      const int lim = stepends[st] - W;
      for (int k = s.pirp[p]; k < s.pirp[p + 1]; ++k)
        if (posof[s.pja[k]] < lim) return w;
    }
  }
  w.nsteps = (int)stepends.size();
  w.W = W;
  int ws = 0;
  while ((1 << ws) < W / C) ++ws;
  w.wshift = ws;
  w.D = D;
  w.capR = capR;
  w.capE = capE;
  const StageLayout lay = stage_layout<T>(capR, capE);
  w.stage_bytes = lay.bytes;
  w.off_win = 0;
  w.off_desc = al16((int)win_bytes);
  w.off_bar = w.off_desc + al16(w.nsteps * 16);
  w.off_ring = w.off_bar + 64;
  w.smem = (size_t)w.off_ring + (size_t)D * lay.bytes;
  // lanes per row: few entries per lane (latency), but enough rows per pass
  const double avg = (double)w.nnz / n;
  const double rows_per_slice = (double)n / std::max(1, w.nsteps * C);
  w.tpr = 1;
  while (w.tpr < 32 && avg / w.tpr > 3.0) w.tpr *= 2;
  while (w.tpr > 1 && rows_per_slice * w.tpr > 960) w.tpr /= 2;
  w.h_desc = std::move(desc);
  w.ok = true;
  return w;
}

template <typename T>
static void upload_win(Arena &ar, DWin<T> &w, const HostCSR &m, bool upper) {
  // rebuild the schedule arrays (cheap) and upload with tail padding
  TriSchedule s;
  build_tri_schedule(w.n, m.irp.data(), m.ja.data(), m.val.data(), upper, w.n, &s);
  std::vector<int> posof((size_t)w.n);
  for (int p = 0; p < w.n; ++p) posof[s.prow[p]] = p;
  std::vector<int> orig(w.h_orig);
  orig.resize((size_t)w.n + 4, 0);
  std::vector<int> pirp(s.pirp);
  pirp.resize((size_t)w.n + 1 + 4, (int)w.nnz);
  std::vector<int> pja((size_t)w.nnz + 4, 0);
  for (int64_t k = 0; k < w.nnz; ++k) pja[k] = posof[s.pja[k]];
  std::vector<T> pval((size_t)w.nnz + 4, T(0));
  for (int64_t k = 0; k < w.nnz; ++k) pval[k] = (T)s.pval[k];
  w.orig = ar.upload(orig);
  w.pirp = ar.upload(pirp);
  w.pja = ar.upload(pja);
  w.pval = ar.upload(pval);
  w.desc = ar.upload(w.h_desc);
  if (std::getenv("MLDG_WIN_TRACE")) {
    w.trace = ar.alloc<unsigned long long>(16);
    MLDG_CUDA(cudaMemset(w.trace, 0, 16 * sizeof(unsigned long long)));
  }
}

// the first solve of a pair writes the second one's right-hand side:
// next[pos2(orig)] = d[orig] * t
template <typename T>
static void link_pair(Arena &ar, DWin<T> &first, const DWin<T> &second, const std::vector<double> &d) {
  std::vector<int> np((size_t)first.n + 4, 0);
  std::vector<T> ns((size_t)first.n + 4, T(0));
  for (int p = 0; p < first.n; ++p) {
    const int o = first.h_orig[p];
    np[p] = second.h_pos[o];
    ns[p] = (T)d[o];
  }
  first.nextpos = ar.upload(np);
  first.nextscale = ar.upload(ns);
}

template <typename T, int TPR, int C, int D>
static void launch_win_3(const DWin<T> &w, const WinArgs<T> &a, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    MLDG_CUDA(cudaFuncSetAttribute(k_trsv_win<T, TPR, C, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kWinSmemMax));
    if (C > 8)
      MLDG_CUDA(cudaFuncSetAttribute(k_trsv_win<T, TPR, C, D>,
                                     cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    attr = true;
  }
  if (C == 1) {
    k_trsv_win<T, TPR, C, D><<<1, 512, w.smem, st>>>(a);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(512);
  cfg.dynamicSmemBytes = w.smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  MLDG_CUDA(cudaLaunchKernelEx(&cfg, k_trsv_win<T, TPR, C, D>, a));
}
template <typename T, int TPR, int C>
static void launch_win_2(const DWin<T> &w, const WinArgs<T> &a, cudaStream_t st) {
  if (w.D == 3)
    launch_win_3<T, TPR, C, 3>(w, a, st);
  else
    launch_win_3<T, TPR, C, 4>(w, a, st);
}
template <typename T, int TPR>
static void launch_win_1(const DWin<T> &w, const WinArgs<T> &a, cudaStream_t st) {
  if (w.C == 1)
    launch_win_2<T, TPR, 1>(w, a, st);
  else if (w.C == 4)
    launch_win_2<T, TPR, 4>(w, a, st);
  else
    launch_win_2<T, TPR, 16>(w, a, st);
}
template <typename T>
static void launch_win(const DWin<T> &w, const WinArgs<T> &a, cudaStream_t st) {
  switch (w.tpr) {
    case 1: launch_win_1<T, 1>(w, a, st); break;
    case 2: launch_win_1<T, 2>(w, a, st); break;
    case 4: launch_win_1<T, 4>(w, a, st); break;
    case 8: launch_win_1<T, 8>(w, a, st); break;
    case 16: launch_win_1<T, 16>(w, a, st); break;
    default: launch_win_1<T, 32>(w, a, st); break;
  }
}

// ---- replicated-window cluster solve (k_trsv_rep): plans and launch ----

// Step schedule and entry classes of one factor for a cluster of C CTAs;
// ok == false when a row exceeds the per-lane register capacities or a
// dependency beyond the ring is fewer than kRepFarMin steps back.
template <typename T>
static DRep<T> build_rep_sched(const HostCSR &m, bool upper, int C) {
  DRep<T> w;
  const int n = m.nr;
  if (n <= 0) return w;
  TriSchedule s;
  build_tri_schedule(n, m.irp.data(), m.ja.data(), m.val.data(), upper, n, &s);
  const int nlev = (int)s.lvl_ptr.size() - 1;
  std::vector<int> posof((size_t)n);
  for (int p = 0; p < n; ++p) posof[s.prow[p]] = p;
  w.n = n;
  w.C = C;
  w.nnz = m.nnz();
  w.R = (int)(128 * 1024 / sizeof(T));
  // MLDG_REP_R: a smaller ring (power of two), so that small tests reach the far path
  if (const char *ev = std::getenv("MLDG_REP_R")) {
    const int r = std::atoi(ev);
    if (r >= 1024 && r <= w.R && (r & (r - 1)) == 0) w.R = r;
  }
  w.h_orig.resize((size_t)n);
  w.h_pos.resize((size_t)n);
  for (int p = 0; p < n; ++p) {
    w.h_orig[p] = upper ? n - 1 - s.prow[p] : s.prow[p];
    w.h_pos[w.h_orig[p]] = p;
  }
  // steps: levels, split where wider than the cluster's row slots
  const int maxstep = C * rep_rows<kRepTPR>();
  if (w.R < 2 * maxstep) return w;
  w.step_ptr.push_back(0);
  for (int L = 0; L < nlev; ++L) {
    const int p0 = s.lvl_ptr[L], p1 = s.lvl_ptr[L + 1], nr = p1 - p0;
    const int k = (nr + maxstep - 1) / maxstep;
    for (int j = 1; j <= k; ++j) w.step_ptr.push_back(p0 + (int)((int64_t)nr * j / k));
  }
  w.nsteps = (int)w.step_ptr.size() - 1;
  std::vector<int> step_of((size_t)n);
  for (int st = 0; st < w.nsteps; ++st)
    for (int p = w.step_ptr[st]; p < w.step_ptr[st + 1]; ++p) step_of[p] = st;
  w.pirp = std::move(s.pirp);
  w.val = std::move(s.pval);
  w.dep.resize(s.pja.size());
  w.cls.resize(s.pja.size());
  w.feeds.assign((size_t)n, 0);
  bool ok = true;
#pragma omp parallel for schedule(static) reduction(&& : ok)
  for (int p = 0; p < n; ++p) {
    const int sp = step_of[p], end = w.step_ptr[sp + 1];
    int n1 = 0, nm = 0, no = 0, nf = 0;
    for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k) {
      const int q = posof[s.pja[k]], sq = step_of[q], dist = sp - sq;
      w.dep[k] = q;
      if (dist < 1) ok = false;
      if (end - q <= w.R) {
        w.cls[k] = dist == 1 ? 0 : (dist <= kRepG ? 3 : 1);
        (dist == 1 ? n1 : (dist <= kRepG ? nm : no))++;
      } else {
        w.cls[k] = 2;
        ++nf;
        if (dist < kRepFarMin) ok = false;
      }
    }
    if (n1 > kRepN1 * kRepTPR || nf > kRepNF * kRepTPR || nm > 255 || no > 255) ok = false;
  }
  if (!ok) return w;
  int64_t nfar = 0;
  // a far copy is reset one step after its last reader's step
  w.rst_step.assign((size_t)n, -1);
  for (int p = 0; p < n; ++p)
    for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k)
      if (w.cls[k] == 2) {
        w.feeds[w.dep[k]] = 1;
        w.rst_step[w.dep[k]] = std::max(w.rst_step[w.dep[k]], step_of[p] + 1);
        ++nfar;
      }
  w.nfar = nfar;
  w.ok = true;
  return w;
}

// Per-CTA blocks of a scheduled factor (host memory); with `next`, each row
// also writes the following solve's right-hand side: next[pos'(orig)] = d[orig] * t.
// Sets w.ok = false when the stages and the ring do not fit in shared memory.
template <typename T>
static void build_rep_blocks_host(DRep<T> &w, const DRep<T> *next, const std::vector<double> *d,
                                  std::vector<uint4> &blocks, std::vector<int4> &desc) {
  const int C = w.C, ns = w.nsteps;
  w.linked = next != nullptr;
  desc.assign((size_t)C * ns, make_int4(0, 0, 0, 0));
  auto slice = [&](int c, int st, int &a, int &b) {
    const int P0 = w.step_ptr[st], P1 = w.step_ptr[st + 1];
    a = P0 + (int)((int64_t)(P1 - P0) * c / C);
    b = P0 + (int)((int64_t)(P1 - P0) * (c + 1) / C);
  };
  // far-copy resets of each (CTA, step): position q goes to CTA q % C at its reset step
  std::vector<std::vector<int>> rst((size_t)C * ns);
  std::vector<std::vector<int>> tailv((size_t)C);
  for (int q = 0; q < w.n; ++q)
    if (w.feeds[q]) {
      const int r = w.rst_step[q];
      if (r < ns)
        rst[(size_t)(q % C) * ns + r].push_back(q);
      else
        tailv[(size_t)(q % C)].push_back(q);
    }
  w.h_tail_ptr.assign((size_t)C + 1, 0);
  w.h_tail.clear();
  for (int c = 0; c < C; ++c) {
    w.h_tail.insert(w.h_tail.end(), tailv[c].begin(), tailv[c].end());
    w.h_tail_ptr[c + 1] = (int)w.h_tail.size();
  }
  // ring and far entries of each (CTA, step) slice
  std::vector<int> ne_of((size_t)C * ns), nf_of((size_t)C * ns);
  for (int c = 0; c < C; ++c)
    for (int st = 0; st < ns; ++st) {
      int a, b, ne = 0, nf = 0;
      slice(c, st, a, b);
      for (int p = a; p < b; ++p)
        for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k) (w.cls[k] == 2 ? nf : ne)++;
      ne_of[(size_t)c * ns + st] = ne;
      nf_of[(size_t)c * ns + st] = nf;
    }
  // block sizes (the block of step t lists the far entries of step t + 2), offsets per CTA in step order
  std::vector<int64_t> boff((size_t)C * ns + 1, 0);
  int capB = 16, maxnr = 0;
  for (int c = 0; c < C; ++c)
    for (int st = 0; st < ns; ++st) {
      const size_t i = (size_t)c * ns + st;
      int a, b, a2 = 0, b2 = 0;
      slice(c, st, a, b);
      if (st + kRepG < ns) slice(c, st + kRepG, a2, b2);
      const int nf2 = st + kRepG < ns ? nf_of[i + kRepG] : 0;
      const RepLayout L = rep_layout<T>(b - a, ne_of[i], b2 - a2, nf2, (int)rst[i].size(), w.linked);
      desc[i] = make_int4((int)(boff[i] / 16), L.bytes / 16, a, b - a);
      boff[i + 1] = boff[i] + L.bytes;
      capB = std::max(capB, L.bytes);
      maxnr = std::max(maxnr, b - a);
    }
  w.block_bytes = boff[(size_t)C * ns];
  blocks.assign((size_t)(w.block_bytes / 16), make_uint4(0, 0, 0, 0));
  unsigned char *base = reinterpret_cast<unsigned char *>(blocks.data());
#pragma omp parallel for schedule(dynamic, 16)
  for (int64_t i = 0; i < (int64_t)C * ns; ++i) {
    const int st = (int)(i % ns), c = (int)(i / ns);
    const int4 dd = desc[(size_t)i];
    const int a = dd.z, nr = dd.w;
    int a2 = 0, b2 = 0;
    if (st + kRepG < ns) slice(c, st + kRepG, a2, b2);
    const int nr2 = b2 - a2, nf2 = st + kRepG < ns ? nf_of[(size_t)i + kRepG] : 0;
    unsigned char *blk = base + boff[(size_t)i];
    const int nrst = (int)rst[(size_t)i].size();
    const RepLayout L = rep_layout<T>(nr, ne_of[(size_t)i], nr2, nf2, nrst, w.linked);
    int4 *hdr = reinterpret_cast<int4 *>(blk);
    hdr[0] = make_int4(nr, ne_of[(size_t)i], nf2, a);
    // copies of the descriptors of the blocks copied and prefetched while this one is staged
    hdr[1] = st + kRepD - 1 < ns ? desc[(size_t)i + kRepD - 1] : make_int4(0, 0, 0, 0);
    hdr[2] = st + kRepPF < ns ? desc[(size_t)i + kRepPF] : make_int4(0, 0, 0, 0);
    hdr[3] = make_int4(nr2, nrst, 0, 0);
    std::copy(rst[(size_t)i].begin(), rst[(size_t)i].end(), reinterpret_cast<int *>(blk + L.o_rst));
    int4 *row = reinterpret_cast<int4 *>(blk + L.o_row);
    int *npos = reinterpret_cast<int *>(blk + L.o_npos);
    T *nsc = reinterpret_cast<T *>(blk + L.o_nsc);
    unsigned short *slot = reinterpret_cast<unsigned short *>(blk + L.o_slot);
    T *val = reinterpret_cast<T *>(blk + L.o_val);
    int2 *fr = reinterpret_cast<int2 *>(blk + L.o_fr);
    int *fq = reinterpret_cast<int *>(blk + L.o_fq);
    T *fv = reinterpret_cast<T *>(blk + L.o_fv);
    int e = 0;
    for (int r = 0; r < nr; ++r) {
      const int p = a + r, o = w.h_orig[p];
      const int e0 = e;
      int cnt[4] = {0, 0, 0, 0};
      for (int pass : {0, 3, 1})  // previous step, two to kRepG steps back, older
        for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k)
          if (w.cls[k] == pass) {
            slot[e] = (unsigned short)(w.dep[k] & (w.R - 1));
            val[e] = (T)w.val[k];
            ++e;
            ++cnt[pass];
          }
      row[r] = make_int4(e0, cnt[0] | (cnt[3] << 8) | (cnt[1] << 16) | ((int)w.feeds[p] << 24), 0, o);
      if (w.linked) {
        npos[r] = next->h_pos[o];
        nsc[r] = (T)(*d)[o];
      }
    }
    int f = 0;
    for (int r = 0; r < nr2; ++r) {
      const int p = a2 + r, f0 = f;
      for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k)
        if (w.cls[k] == 2) {
          fq[f] = w.dep[k];
          fv[f] = (T)w.val[k];
          ++f;
        }
      fr[r] = make_int2(f0, f - f0);
    }
  }
  constexpr int PER = 16 / (int)sizeof(T);
  w.capB = capB;
  w.stage_bytes = capB + rep_al16((maxnr + 2 * PER) * (int)sizeof(T));
  w.ring_bytes = w.R * (int)sizeof(T);
  w.smem = (size_t)w.ring_bytes + (size_t)kRepD * w.stage_bytes + 256;  // + the mbarriers
  if (w.smem > (size_t)kWinSmemMax) w.ok = false;
}

template <typename T>
static void build_rep_blocks(Arena &ar, DRep<T> &w, const DRep<T> *next, const std::vector<double> *d) {
  std::vector<uint4> blocks;
  std::vector<int4> desc;
  build_rep_blocks_host(w, next, d, blocks, desc);
  if (!w.ok) return;
  w.desc = ar.upload(desc);
  w.blocks = ar.upload(blocks);
  std::vector<int> vb((size_t)w.nsteps);
  for (int st = 0; st < w.nsteps; ++st) vb[st] = (int)sizeof(T) * (w.step_ptr[st + 1] - w.step_ptr[st]);
  w.vbytes = ar.upload(vb);
  std::vector<int> orig(w.h_orig);
  orig.resize((size_t)w.n + 4, 0);
  w.orig = ar.upload(orig);
  if (w.nfar) {
    // the far copy holds the sentinel until a value is written
    std::vector<T> xs((size_t)w.n + 8, Sentinel<T>::value());
    w.xp = ar.upload(xs);
    w.tail_ptr = ar.upload(w.h_tail_ptr);
    std::vector<int> tl(w.h_tail);
    tl.push_back(0);
    w.tail = ar.upload(tl);
  }
  if (std::getenv("MLDG_REP_TRACE")) {
    w.trace = ar.alloc<unsigned long long>(20);
    MLDG_CUDA(cudaMemset(w.trace, 0, 20 * sizeof(unsigned long long)));
  }
}

// drops the host schedule of a plan (after its blocks and those of the plan
// linked to it are built)
template <typename T>
static void rep_release_sched(DRep<T> &w) {
  std::vector<int>().swap(w.step_ptr);
  std::vector<int>().swap(w.pirp);
  std::vector<int>().swap(w.dep);
  std::vector<double>().swap(w.val);
  std::vector<unsigned char>().swap(w.cls);
  std::vector<unsigned char>().swap(w.feeds);
  std::vector<int>().swap(w.rst_step);
}

template <typename T, int C>
static cudaLaunchConfig_t rep_config(const DRep<T> &w, cudaStream_t st, cudaLaunchAttribute *at) {
  static bool attr = false;
  if (!attr) {
    MLDG_CUDA(cudaFuncSetAttribute(k_trsv_rep<T, kRepTPR, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kWinSmemMax));
    if (C > 8)
      MLDG_CUDA(cudaFuncSetAttribute(k_trsv_rep<T, kRepTPR, C>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kRepThreads);
  cfg.dynamicSmemBytes = w.smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// can a cluster of this plan's shape be resident at all
template <typename T>
static bool rep_fits(const DRep<T> &w) {
  cudaLaunchAttribute at[1];
  int ncl = 0;
  cudaError_t e;
  if (w.C == 8) {
    cudaLaunchConfig_t cfg = rep_config<T, 8>(w, 0, at);
    e = cudaOccupancyMaxActiveClusters(&ncl, k_trsv_rep<T, kRepTPR, 8>, &cfg);
  } else {
    cudaLaunchConfig_t cfg = rep_config<T, 16>(w, 0, at);
    e = cudaOccupancyMaxActiveClusters(&ncl, k_trsv_rep<T, kRepTPR, 16>, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return ncl > 0;
}

template <typename T>
static void launch_rep(const DRep<T> &w, const RepArgs<T> &a, cudaStream_t st) {
  cudaLaunchAttribute at[1];
  if (w.C == 8) {
    cudaLaunchConfig_t cfg = rep_config<T, 8>(w, st, at);
    MLDG_CUDA(cudaLaunchKernelEx(&cfg, k_trsv_rep<T, kRepTPR, 8>, a));
  } else {
    cudaLaunchConfig_t cfg = rep_config<T, 16>(w, st, at);
    MLDG_CUDA(cudaLaunchKernelEx(&cfg, k_trsv_rep<T, kRepTPR, 16>, a));
  }
}

// Host emulation of k_trsv_rep over a plan, in the kernel's order (the rows
// of a step from the ring state after the previous step, values published at
// the end of the step).  Every ring read is checked against the position the
// schedule says it holds, every ring read against the window bound of its
// step, every far read against its kRepFarMin-step distance, and every block
// against its descriptor and the stage capacity; returns the violations.
// rhs_pos: right-hand side in the plan's position order; out[orig] = t;
// next_pos[npos] = nsc * t for a linked plan.
template <typename T>
static int64_t rep_emulate(const DRep<T> &w, const std::vector<uint4> &blocks, const std::vector<int4> &desc,
                           const std::vector<T> &rhs_pos, std::vector<T> &out, std::vector<T> *next_pos) {
  const int R = w.R, C = w.C, ns = w.nsteps, n = w.n;
  constexpr int PER = 16 / (int)sizeof(T);
  std::vector<T> ring((size_t)R, T(0)), xp((size_t)n, T(0));
  std::vector<int> tag((size_t)R, -1), tstep((size_t)R, -1), xstep((size_t)n, 1 << 30);
  std::vector<unsigned char> xvalid((size_t)n, 0);  // far copy written and not yet reset
  std::vector<std::pair<int, T>> pub;
  const unsigned char *base = reinterpret_cast<const unsigned char *>(blocks.data());
  int64_t bad = 0;
  for (int s = 0; s < ns; ++s) {
    pub.clear();
    const int end = w.step_ptr[s + 1];
    for (int c = 0; c < C; ++c) {
      const int4 dd = desc[(size_t)c * ns + s];
      const unsigned char *blk = base + (size_t)dd.x * 16;
      const int4 hdr = *reinterpret_cast<const int4 *>(blk);
      const int4 h3 = reinterpret_cast<const int4 *>(blk)[3];
      const RepLayout L = rep_layout<T>(hdr.x, hdr.y, h3.x, hdr.z, h3.y, w.linked);
      if (hdr.x != dd.w || hdr.w != dd.z || L.bytes != dd.y * 16 || L.bytes > w.capB) ++bad;
      if (s + kRepG < ns && h3.x != desc[(size_t)c * ns + s + kRepG].w) ++bad;
      for (int h = 1; h <= 2; ++h) {
        const int ahead = h == 1 ? kRepD - 1 : kRepPF;
        const int4 want = s + ahead < ns ? desc[(size_t)c * ns + s + ahead] : make_int4(0, 0, 0, 0);
        const int4 got = reinterpret_cast<const int4 *>(blk)[h];
        if (got.x != want.x || got.y != want.y || got.z != want.z || got.w != want.w) ++bad;
      }
      if (hdr.x > rep_rows<kRepTPR>()) ++bad;
      const int r0a = dd.z & ~(PER - 1);
      const int nrc = dd.w > 0 ? (dd.z + dd.w - r0a + PER - 1) / PER : 0;
      if (16 * nrc > w.stage_bytes - w.capB) ++bad;
      const int4 *row = reinterpret_cast<const int4 *>(blk + L.o_row);
      const int *npos = reinterpret_cast<const int *>(blk + L.o_npos);
      const T *nsc = reinterpret_cast<const T *>(blk + L.o_nsc);
      const unsigned short *slot = reinterpret_cast<const unsigned short *>(blk + L.o_slot);
      const T *val = reinterpret_cast<const T *>(blk + L.o_val);
      // far entries of this step's rows: listed in the block of step s - kRepG
      const int2 *fr = nullptr;
      const int *fq = nullptr;
      const T *fv = nullptr;
      if (s >= kRepG) {
        const unsigned char *b2 = base + (size_t)desc[(size_t)c * ns + s - kRepG].x * 16;
        const int4 g0 = *reinterpret_cast<const int4 *>(b2);
        const int4 g3 = reinterpret_cast<const int4 *>(b2)[3];
        if (g3.x != hdr.x) ++bad;
        const RepLayout L2 = rep_layout<T>(g0.x, g0.y, g3.x, g0.z, g3.y, w.linked);
        fr = reinterpret_cast<const int2 *>(b2 + L2.o_fr);
        fq = reinterpret_cast<const int *>(b2 + L2.o_fq);
        fv = reinterpret_cast<const T *>(b2 + L2.o_fv);
      }
      for (int r = 0; r < hdr.x; ++r) {
        const int p = hdr.w + r;
        const int4 ri = row[r];
        const int n1 = ri.y & 0xff, nm = (ri.y >> 8) & 0xff, no = (ri.y >> 16) & 0xff;
        const int nf = fr ? fr[r].y : 0, f0 = fr ? fr[r].x : 0;
        int nfs = 0;
        for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k) nfs += w.cls[k] == 2;
        if (n1 > kRepN1 * kRepTPR || nf > kRepNF * kRepTPR || nf != nfs) ++bad;
        if (ri.w != w.h_orig[p] || ((ri.y >> 24) & 1) != (int)w.feeds[p]) ++bad;
        // the schedule's ring dependencies of p, in block order, and the step
        // distance each class allows: previous step, 2..kRepG back, older
        std::vector<int> qs;
        std::vector<int> lo, hi;
        for (int pass : {0, 3, 1})
          for (int k = w.pirp[p]; k < w.pirp[p + 1]; ++k)
            if (w.cls[k] == pass) {
              qs.push_back(w.dep[k]);
              lo.push_back(pass == 0 ? 1 : (pass == 3 ? 2 : kRepG + 1));
              hi.push_back(pass == 0 ? 1 : (pass == 3 ? kRepG : 1 << 30));
            }
        if ((int)qs.size() != n1 + nm + no) ++bad;
        T acc = T(0);
        for (int e = 0; e < n1 + nm + no; ++e) {
          const int k = ri.x + e, sl = slot[k];
          const int q = e < (int)qs.size() ? qs[e] : -1;
          if (q < 0 || tag[sl] != q || q < end - R) {
            ++bad;
          } else {
            const int dist = s - tstep[sl];
            if (dist < lo[e] || dist > hi[e]) ++bad;
          }
          acc = acc + val[k] * ring[sl];
        }
        for (int f = 0; f < nf; ++f) {
          const int q = fq[f0 + f];
          // written in this solve, not yet reset, far enough back
          if (q < 0 || q >= n || !xvalid[q] || xstep[q] > s - kRepFarMin) ++bad;
          acc = acc + fv[f0 + f] * xp[q];
        }
        const T t = rhs_pos[p] - acc;
        pub.emplace_back(p, t);
        out[ri.w] = t;
        if (w.linked) (*next_pos)[npos[r]] = nsc[r] * t;
        if ((ri.y >> 24) & 1) {
          xp[p] = t;
          xstep[p] = s;
          xvalid[p] = 1;
        }
      }
    }
    for (auto &pv : pub) {
      ring[pv.first & (R - 1)] = pv.second;
      tag[pv.first & (R - 1)] = pv.first;
      tstep[pv.first & (R - 1)] = s;
    }
    // far-copy resets of this step (every reader of them is in an earlier step)
    for (int c = 0; c < C; ++c) {
      const unsigned char *blk = base + (size_t)desc[(size_t)c * ns + s].x * 16;
      const int4 hdr = *reinterpret_cast<const int4 *>(blk);
      const int4 h3 = reinterpret_cast<const int4 *>(blk)[3];
      const RepLayout L = rep_layout<T>(hdr.x, hdr.y, h3.x, hdr.z, h3.y, w.linked);
      const int *rs = reinterpret_cast<const int *>(blk + L.o_rst);
      for (int i = 0; i < h3.y; ++i) {
        const int q = rs[i];
        if (q < 0 || q >= n || !xvalid[q] || q % C != c) ++bad;
        else xvalid[q] = 0;
      }
    }
  }
  // the tail resets leave the far copy clean for the next solve
  for (int c = 0; c < C; ++c)
    for (int i = w.h_tail_ptr[c]; i < w.h_tail_ptr[c + 1]; ++i) {
      const int q = w.h_tail[i];
      if (q < 0 || q >= n || !xvalid[q] || q % C != c) ++bad;
      else xvalid[q] = 0;
    }
  for (int q = 0; q < n; ++q) bad += xvalid[q];
  return bad;
}

// y = U^{-1} diag(d) L^{-1} x through the emulated pair of plans; stats: violations,
// steps of the first plan, far entries of both, plans usable (1/0).
template <typename T>
static void rep_check_pair(const HostCSR &Lf, bool lupper, const HostCSR &Uf, bool uupper,
                           const std::vector<double> &d, int C, const double *x, double *y, long long *stats) {
  DRep<T> f = build_rep_sched<T>(Lf, lupper, C);
  DRep<T> g = build_rep_sched<T>(Uf, uupper, C);
  stats[0] = 0;
  stats[1] = f.nsteps;
  stats[2] = f.nfar + g.nfar;
  stats[3] = 0;
  if (!f.ok || !g.ok) return;
  std::vector<uint4> bf, bg;
  std::vector<int4> df, dg;
  build_rep_blocks_host(f, &g, &d, bf, df);
  build_rep_blocks_host(g, (const DRep<T> *)nullptr, (const std::vector<double> *)nullptr, bg, dg);
  if (!f.ok || !g.ok) return;
  const int n = f.n;
  std::vector<T> rp((size_t)n), nx((size_t)n, T(0)), o1((size_t)n), o2((size_t)n);
  for (int p = 0; p < n; ++p) rp[p] = (T)x[f.h_orig[p]];
  int64_t bad = rep_emulate(f, bf, df, rp, o1, &nx);
  bad += rep_emulate(g, bg, dg, nx, o2, (std::vector<T> *)nullptr);
  for (int i = 0; i < n; ++i) y[i] = (double)o2[i];
  stats[0] = bad;
  stats[3] = 1;
}

// ---- partitioned solve (k_trsv_blk): plan and launch ----
// The factor in lower form (an upper factor with rows and columns reversed)
// is cut into P contiguous blocks of about equal rows + entries.  A block's
// rows are ordered by (global dependency level, row) and grouped into steps
// of one level each, split where a step's plan would exceed kBlkStageCap
// bytes (the pieces of one level are marked, the kernel takes no barrier
// between them).  A dependency on a row of the same block whose ring slot is
// still intact at the end of the reading step's level (rows of one level
// are solved without a barrier between its steps) reads the ring, every
// other one the exchange vector.  The ring holds W values: the smallest
// power of two that covers every local dependency's reach, at most kBlkWMax.
constexpr int kBlkStageCap = 8 * 1024;
constexpr int kBlkWMax = 8192;

template <typename T>
struct HostBlk {
  bool ok = false;
  int n = 0, nblocks = 0, nsteps = 0, W = 0, stage_bytes = 0, aux_cap = 0;
  size_t smem = 0;
  int64_t nnz = 0, plan_bytes = 0;
  std::vector<int> bstep;
  std::vector<int2> sdesc;
  std::vector<uint4> plan;
};

template <typename T>
static HostBlk<T> build_blk_host(const HostCSR &m, bool upper, int P) {
  HostBlk<T> w;
  const int n = m.nr;
  if (n == 0 || P < 1) return w;
  P = std::min(P, n);
  auto orig = [&](int ip) { return upper ? n - 1 - ip : ip; };
  auto lowcol = [&](int j) { return upper ? n - 1 - j : j; };
  std::vector<int> lev((size_t)n, 0);
  for (int ip = 0; ip < n; ++ip) {
    const int o = orig(ip);
    int l = 0;
    for (int k = m.irp[o]; k < m.irp[o + 1]; ++k) {
      const int jp = lowcol(m.ja[k]);
      if (jp >= ip) return w;  // not triangular in this direction
      l = std::max(l, lev[jp] + 1);
    }
    lev[ip] = l;
  }
  // blocks of about equal rows + entries
  const int64_t total = (int64_t)n + m.nnz();
  std::vector<int> bnd((size_t)P + 1, n);
  bnd[0] = 0;
  {
    int64_t acc = 0;
    int b = 1;
    for (int ip = 0; ip < n && b < P; ++ip) {
      const int o = orig(ip);
      acc += 1 + (m.irp[o + 1] - m.irp[o]);
      if (acc * P >= total * b) bnd[b++] = ip + 1;
    }
    for (; b < P; ++b) bnd[b] = n;
  }
  std::vector<int> blk((size_t)n), lpos((size_t)n);
  // per block: positions in (level, row) order
  std::vector<std::vector<int>> order((size_t)P);
#pragma omp parallel for schedule(dynamic, 1)
  for (int b = 0; b < P; ++b) {
    auto &ord = order[b];
    ord.resize((size_t)(bnd[b + 1] - bnd[b]));
    for (int ip = bnd[b]; ip < bnd[b + 1]; ++ip) ord[ip - bnd[b]] = ip;
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return lev[x] < lev[y]; });
    for (size_t q = 0; q < ord.size(); ++q) {
      blk[ord[q]] = b;
      lpos[ord[q]] = (int)q;
    }
  }
  // steps: (block, first local position) ; split on level change or capacity
  struct Step {
    int b, p0, p1, nent;
  };
  std::vector<Step> steps;
  std::vector<int> bstep((size_t)P + 1, 0);
  for (int b = 0; b < P; ++b) {
    bstep[b] = (int)steps.size();
    const auto &ord = order[b];
    int p = 0;
    while (p < (int)ord.size()) {
      Step st{b, p, p, 0};
      const int l = lev[ord[p]];
      while (st.p1 < (int)ord.size() && lev[ord[st.p1]] == l) {
        const int o = orig(ord[st.p1]);
        const int len = m.irp[o + 1] - m.irp[o];
        if (st.p1 > st.p0 && blk_bytes<T>(st.p1 - st.p0 + 1, st.nent + len) > kBlkStageCap) break;
        st.nent += len;
        ++st.p1;
      }
      steps.push_back(st);
      p = st.p1;
    }
  }
  bstep[P] = (int)steps.size();
  const int ns = (int)steps.size();
  // a step continues the level of the block's previous step; the end of each
  // step's level (the rows of a level are solved without a barrier)
  std::vector<int> same((size_t)ns, 0), lvl_end((size_t)ns, 0);
  for (int b = 0; b < P; ++b) {
    for (int s = bstep[b] + 1; s < bstep[b + 1]; ++s)
      same[s] = lev[order[b][steps[s].p0]] == lev[order[b][steps[s - 1].p0]];
    for (int s = bstep[b + 1] - 1; s >= bstep[b]; --s)
      lvl_end[s] = (s + 1 < bstep[b + 1] && same[s + 1]) ? lvl_end[s + 1] : steps[s].p1;
  }
  // ring size: the reach of the local dependencies (capped)
  std::vector<int> step_end((size_t)n);
  for (int s = 0; s < ns; ++s)
    for (int q = steps[s].p0; q < steps[s].p1; ++q) step_end[order[steps[s].b][q]] = lvl_end[s];
  int reach = 1;
  for (int ip = 0; ip < n; ++ip) {
    const int o = orig(ip);
    for (int k = m.irp[o]; k < m.irp[o + 1]; ++k) {
      const int jp = lowcol(m.ja[k]);
      if (blk[jp] == blk[ip]) reach = std::max(reach, step_end[ip] - lpos[jp]);
    }
  }
  int W = 16;
  while (W < reach && W < kBlkWMax) W *= 2;
  // plan blocks
  std::vector<int64_t> boff((size_t)ns + 1, 0);
  int capB = 16, capA = 1;
  for (int s = 0; s < ns; ++s) {
    const int bytes = blk_bytes<T>(steps[s].p1 - steps[s].p0, steps[s].nent);
    boff[s + 1] = boff[s] + bytes;
    capB = std::max(capB, bytes);
    capA = std::max(capA, 2 * (steps[s].p1 - steps[s].p0) + steps[s].nent);
  }
  capA = (capA + 1) & ~1;  // keeps the mbarriers after the aux buffers 8-byte aligned
  if (boff[ns] / 16 > INT32_MAX) return w;
  std::vector<uint4> plan((size_t)(boff[ns] / 16), make_uint4(0, 0, 0, 0));
  std::vector<int2> sdesc((size_t)ns);
#pragma omp parallel for schedule(dynamic, 64)
  for (int s = 0; s < ns; ++s) {
    const Step &st = steps[s];
    const int nr = st.p1 - st.p0;
    unsigned char *base = reinterpret_cast<unsigned char *>(plan.data()) + boff[s];
    int4 *hdr = reinterpret_cast<int4 *>(base);
    *hdr = make_int4(nr, st.nent, same[s], 0);
    int4 *rows = reinterpret_cast<int4 *>(base + 16);
    int *code = reinterpret_cast<int *>(base + 16 + 16 * nr);
    T *val = reinterpret_cast<T *>(base + blk_off_val<T>(nr, st.nent));
    int e = 0;
    for (int q = st.p0; q < st.p1; ++q) {
      const int ip = order[st.b][q];
      const int o = orig(ip);
      rows[q - st.p0] = make_int4(o, e, m.irp[o + 1] - m.irp[o], q);
      for (int k = m.irp[o]; k < m.irp[o + 1]; ++k, ++e) {
        const int jp = lowcol(m.ja[k]);
        const bool ring = blk[jp] == st.b && lpos[jp] >= lvl_end[s] - W;
        code[e] = ring ? (lpos[jp] & (W - 1)) : -(orig(jp) + 1);
        val[e] = (T)m.val[k];
      }
    }
    sdesc[s] = make_int2((int)(boff[s] / 16), (int)((boff[s + 1] - boff[s]) / 16));
  }
  w.n = n;
  w.nblocks = P;
  w.nsteps = ns;
  w.W = W;
  w.stage_bytes = capB;
  w.aux_cap = capA;
  w.nnz = m.nnz();
  w.plan_bytes = boff[ns];
  w.smem = blk_smem<T>(W, capB, capA);
  if (w.smem > 220 * 1024) return w;
  w.bstep = std::move(bstep);
  w.sdesc = std::move(sdesc);
  w.plan = std::move(plan);
  w.ok = true;
  return w;
}

template <typename T>
static DBlk<T> build_blk_plan(Arena &ar, const HostCSR &m, bool upper, int P) {
  DBlk<T> w;
  HostBlk<T> hb = build_blk_host<T>(m, upper, P);
  if (!hb.ok) return w;
  w.n = hb.n;
  w.nblocks = hb.nblocks;
  w.nsteps = hb.nsteps;
  w.W = hb.W;
  w.stage_bytes = hb.stage_bytes;
  w.aux_cap = hb.aux_cap;
  w.nnz = hb.nnz;
  w.plan_bytes = hb.plan_bytes;
  w.smem = hb.smem;
  w.bstep = ar.upload(hb.bstep);
  w.sdesc = ar.upload(hb.sdesc);
  w.plan = ar.upload(hb.plan);
  w.ticket = ar.alloc<int>(2);
  MLDG_CUDA(cudaMemset(w.ticket, 0, 2 * sizeof(int)));
  w.ok = true;
  return w;
}

// Host emulation of k_trsv_blk on a plan: blocks in ticket order, steps in
// order, rows of a step in the kernel's thread order, with every access the
// kernel makes checked against its buffer (plan block inside the plan and
// within the stage, row and entry ranges, ring slots, exchange indices), every
// ring read against the position that slot holds, and every remote read
// against a written value.  Returns the number of violations; t receives the
// solution (original numbering) of t = scale o rhs - T_strict t.
template <typename T>
static int64_t blk_emulate(const HostBlk<T> &w, const HostCSR &m, const std::vector<double> &rhs,
                           const double *scale, std::vector<double> &t) {
  int64_t bad = 0;
  const int n = w.n, W = w.W;
  if (W < 1 || (W & (W - 1)) || (int)w.bstep.size() != w.nblocks + 1 || w.bstep[0] != 0 ||
      w.bstep[w.nblocks] != w.nsteps || w.stage_bytes % 16 || w.smem > 220 * 1024)
    return 1;
  std::vector<double> cur((size_t)n, std::nan(""));
  std::vector<char> written((size_t)n, 0);
  std::vector<double> ring((size_t)W, 0.0);
  t.assign((size_t)n, 0.0);
  const unsigned char *planb = reinterpret_cast<const unsigned char *>(w.plan.data());
  const int64_t plan_size = (int64_t)w.plan.size() * 16;
  for (int b = 0; b < w.nblocks; ++b) {
    std::vector<int> ring_row((size_t)W, -1);  // original row whose value a slot holds
    if (w.bstep[b + 1] < w.bstep[b]) return bad + 1;
    // the steps of one level are solved without a barrier between them: their
    // values become visible at the next level's barrier, and no slot the level
    // reads may be written by it
    std::vector<std::pair<int, double>> pend;  // original row, value
    std::vector<int> pend_slot;
    std::vector<char> read_slot((size_t)W, 0);
    auto flush = [&]() {
      for (size_t q = 0; q < pend.size(); ++q) {
        const int slot = pend_slot[q], row = pend[q].first;
        if (read_slot[slot]) ++bad;  // a slot written while the level still reads it
        ring[slot] = pend[q].second;
        ring_row[slot] = row;
        if (written[row]) ++bad;
        cur[row] = pend[q].second;
        written[row] = 1;
        t[row] = pend[q].second;
      }
      pend.clear();
      pend_slot.clear();
      std::fill(read_slot.begin(), read_slot.end(), 0);
    };
    for (int s = w.bstep[b]; s < w.bstep[b + 1]; ++s) {
      const int2 dsc = w.sdesc[s];
      const int64_t off = (int64_t)dsc.x * 16, bytes = (int64_t)dsc.y * 16;
      if (off < 0 || bytes < 16 || off + bytes > plan_size || bytes > w.stage_bytes) {
        ++bad;
        continue;
      }
      const unsigned char *st = planb + off;
      const int4 hdr = *reinterpret_cast<const int4 *>(st);
      if (hdr.x < 0 || hdr.y < 0 || blk_bytes<T>(hdr.x, hdr.y) > bytes || 2 * hdr.x + hdr.y > w.aux_cap ||
          (hdr.z != 0 && hdr.z != 1) || (hdr.z && s == w.bstep[b])) {
        ++bad;
        continue;
      }
      if (!hdr.z) flush();  // a new level
      const int4 *rows = reinterpret_cast<const int4 *>(st + 16);
      const int *code = reinterpret_cast<const int *>(st + 16 + 16 * hdr.x);
      const T *val = reinterpret_cast<const T *>(st + blk_off_val<T>(hdr.x, hdr.y));
      for (int r = 0; r < hdr.x; ++r) {
        const int4 rw = rows[r];
        if (rw.x < 0 || rw.x >= n || rw.y < 0 || rw.z < 0 || rw.y + rw.z > hdr.y ||
            rw.z != m.irp[rw.x + 1] - m.irp[rw.x]) {
          ++bad;
          continue;
        }
        double acc = 0.0;
        for (int e = rw.y; e < rw.y + rw.z; ++e) {
          const int c = code[e];
          const int k = m.irp[rw.x] + (e - rw.y);  // the CSR entry this slot stands for
          const int dep = m.ja[k];
          if ((double)val[e] != (double)(T)m.val[k]) ++bad;
          double dv = 0.0;
          if (c >= 0) {
            if (c >= W || ring_row[c] != dep) {
              ++bad;
            } else {
              dv = ring[c];
              read_slot[c] = 1;
            }
          } else {
            const int64_t j = -(int64_t)c - 1;
            if (j != dep || !written[j])
              ++bad;
            else
              dv = cur[j];
          }
          acc += (double)val[e] * dv;
        }
        const double sc = scale ? scale[rw.x] : 1.0;
        pend.emplace_back(rw.x, sc * rhs[rw.x] - acc);
        pend_slot.push_back(rw.w & (W - 1));
      }
    }
    flush();
  }
  for (int i = 0; i < n; ++i) bad += !written[i];
  return bad;
}

template <typename T>
static void launch_blk(const DBlk<T> &w, const BlkArgs<T> &a, cudaStream_t st) {
  k_trsv_blk<T><<<w.nblocks, kBlkThreads, w.smem, st>>>(a);
}

template <typename T>
static DTri<T> build_tri_dev(Arena &ar, const HostCSR &m, bool upper, int nsm) {
  DTri<T> t;
  if (!m.present()) return t;
  TriSchedule s;
  const int n = m.nr;
  build_tri_schedule(n, m.irp.data(), m.ja.data(), m.val.data(), upper, std::max(n, 1), &s);
  t.n = n;
  t.rev = upper ? 1 : 0;
  t.nlevels = (int)s.lvl_ptr.size() - 1;
  t.nnz = m.nnz();
  t.lvl_ptr = ar.upload(s.lvl_ptr);
  t.prow = ar.upload(s.prow);
  t.pirp = ar.upload(s.pirp);
  t.pja = ar.upload(s.pja);
  std::vector<T> v(s.pval.begin(), s.pval.end());
  t.pval = ar.upload(v);
  // host copies of the schedule for the ELL and multi-column plans (moved
  // after the uploads; the staged-plan code below only reads lvl_ptr/pirp)
  t.h_lvl = s.lvl_ptr;
  t.h_prow = s.prow;
  t.h_pirp = s.pirp;
  t.h_pja = std::move(s.pja);
  t.h_pval = std::move(s.pval);
  t.counters = ar.alloc<int>(2);
  MLDG_CUDA(cudaMemset(t.counters, 0, 2 * sizeof(int)));
  // lanes per row: smallest power of two with <= 8 entries per lane
  const double avg = n > 0 ? (double)t.nnz / n : 0.0;
  t.tpr = 1;
  while (t.tpr < 32 && avg / t.tpr > 8.0) t.tpr *= 2;
  t.e = (avg / t.tpr <= 4.0) ? 4 : 8;
  t.cta = n <= tri_cta_rows<T>();
  // staged single-CTA plan: solution + level descriptors + D ring stages.
  // Stages are sized for the 95th-percentile level; larger levels are read
  // straight from global memory.  Latency-bound, so few entries per lane.
  if (n <= tri_cta_rows<T>()) {
    std::vector<int4> desc((size_t)t.nlevels);
    std::vector<int> rs, es;
    for (int L = 0; L < t.nlevels; ++L) {
      const int p0 = s.lvl_ptr[L], p1 = s.lvl_ptr[L + 1];
      desc[L] = make_int4(p0, p1, s.pirp[p0], s.pirp[p1]);
      rs.push_back(p1 - p0);
      es.push_back(s.pirp[p1] - s.pirp[p0]);
    }
    auto pct = [](std::vector<int> v, double q) {
      std::sort(v.begin(), v.end());
      return v.empty() ? 1 : std::max(1, v[(size_t)(q * (v.size() - 1))]);
    };
    StageCfg c{};
    c.capR = pct(rs, 0.95);
    c.capE = pct(es, 0.95);
    c.off_y = 0;
    c.off_desc = (int)(((size_t)std::max(n, 1) * sizeof(T) + 15) & ~(size_t)15);
    c.off_ring = c.off_desc + (int)(((size_t)t.nlevels * 16 + 15) & ~(size_t)15);
    const size_t budget = 220 * 1024;
    c.D = 0;
    for (int shrink = 0; shrink < 6 && c.D == 0; ++shrink) {
      c.bytes = (int)(((((size_t)(2 * c.capR + 1 + c.capE) * 4 + 15) & ~(size_t)15) +
                       (size_t)c.capE * sizeof(T) + 15) & ~(size_t)15);
      for (int D : {6, 4, 3})  // ring depths compiled into k_trsv_stg
        if ((size_t)c.off_ring + (size_t)D * c.bytes <= budget) {
          c.D = D;
          break;
        }
      if (c.D == 0) {
        c.capE = std::max(1, c.capE / 2);
        c.capR = std::max(1, c.capR / 2);
      }
    }
    if (c.D >= 3) {
      t.mode = 0;
      t.stg = c;
      t.desc = ar.upload(desc);
      t.threads = 512;
      t.grid = 1;
      t.smem = (size_t)c.off_ring + (size_t)c.D * c.bytes;
      t.tpr = 1;
      while (t.tpr < 32 && avg / t.tpr > 2.0) t.tpr *= 2;
      return t;
    }
  }
  if (t.cta) {
    t.mode = 1;
    t.threads = 512;
    t.grid = 1;
    t.smem = (size_t)std::max(n, 1) * sizeof(T);
  } else {
    t.mode = 2;
    const int rpw = 32 / t.tpr;
    std::vector<int2> blk;
    blk.reserve((size_t)n / rpw + (size_t)t.nlevels + 1);
    for (int L = 0; L < t.nlevels; ++L)
      for (int p = s.lvl_ptr[L]; p < s.lvl_ptr[L + 1]; p += rpw)
        blk.push_back(make_int2(p, std::min(p + rpw, s.lvl_ptr[L + 1])));
    t.nblk = (int)blk.size();
    t.blk = ar.upload(blk);
    // Warps in flight: a few dependency levels' worth of blocks.  More only
    // adds spinning lanes whose polls compete with real traffic in L2.
    const int per_level = (t.nblk + t.nlevels - 1) / std::max(t.nlevels, 1);
    int mult = 4;
    if (const char *e = std::getenv("MLDG_SF_MULT")) mult = std::max(1, std::atoi(e));
    const int warps = std::max(32, std::min(mult * per_level, nsm * 32));
    t.threads = 256;
    t.grid = (warps + 7) / 8;
  }
  return t;
}

template <typename T, int TPR>
static void set_attr_t() {
  const int mx = 224 * 1024;
  MLDG_CUDA(cudaFuncSetAttribute(k_trsv_stg<T, TPR, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
  MLDG_CUDA(cudaFuncSetAttribute(k_trsv_stg<T, TPR, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
  MLDG_CUDA(cudaFuncSetAttribute(k_trsv_stg<T, TPR, 6>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
  MLDG_CUDA(cudaFuncSetAttribute(k_trsv_cta<T, TPR, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
  MLDG_CUDA(cudaFuncSetAttribute(k_trsv_cta<T, TPR, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
}
template <typename T>
static void set_trsv_smem_attr() {
  static bool done = false;
  if (done) return;
  set_attr_t<T, 1>();
  set_attr_t<T, 2>();
  set_attr_t<T, 4>();
  set_attr_t<T, 8>();
  set_attr_t<T, 16>();
  set_attr_t<T, 32>();
  MLDG_CUDA(cudaFuncSetAttribute(k_trsv_blk<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
  done = true;
}

// Coarsest levels up to this size are solved with the explicit inverse of
// their ILU(0) factorisation: the same operator as the two triangular solves
// (U^{-1} diag(d) L^{-1}), applied as one bandwidth-bound matrix-vector
// product instead of a chain of dependency levels.
constexpr int kDenseCoarseRows = 2048;
// intermediate levels up to this size get a GPU-computed explicit inverse
// (n^2 values, 2.1 GB at FP64 for the largest) when it applies faster
constexpr int kDenseInvRows = 16384;

// M = U^{-1} diag(d) L^{-1} (row-major) and its transpose, column by column
static void dense_ilu_inverse(const HostCSR &Lf, const HostCSR &Uf, const std::vector<double> &d,
                              std::vector<double> &M, std::vector<double> &MT) {
  const int n = Lf.nr;
  M.assign((size_t)n * n, 0.0);
  MT.assign((size_t)n * n, 0.0);
#pragma omp parallel
  {
    std::vector<double> t((size_t)n), z((size_t)n);
#pragma omp for schedule(dynamic, 8)
    for (int j = 0; j < n; ++j) {
      for (int i = 0; i < n; ++i) {  // t = L^{-1} e_j
        double s = 0.0;
        for (int k = Lf.irp[i]; k < Lf.irp[i + 1]; ++k) s += Lf.val[k] * t[Lf.ja[k]];
        t[i] = (i == j ? 1.0 : 0.0) - s;
      }
      for (int i = 0; i < n; ++i) t[i] *= d[i];
      for (int i = n - 1; i >= 0; --i) {  // z = U^{-1} t
        double s = 0.0;
        for (int k = Uf.irp[i]; k < Uf.irp[i + 1]; ++k) s += Uf.val[k] * z[Uf.ja[k]];
        z[i] = t[i] - s;
      }
      for (int i = 0; i < n; ++i) {
        M[(size_t)i * n + j] = z[i];
        MT[(size_t)j * n + i] = z[i];
      }
    }
  }
}

template <typename T>
static Engine *make_engine(Handle *h) {
  // MLDG_TIMING: host time of each finalize phase
  std::map<std::string, double> tm;
  auto clk = std::chrono::steady_clock::now();
  auto tick = [&](const char *what) {
    const auto now = std::chrono::steady_clock::now();
    tm[what] += std::chrono::duration<double>(now - clk).count();
    clk = now;
  };
  set_trsv_smem_attr<T>();
  auto owner = std::make_unique<EngineT<T>>();
  EngineT<T> *e = owner.get();
  e->h = h;
  e->st = h->st;
  e->pev0 = h->pev0;
  e->pev1 = h->pev1;
  e->probe_kind = h->probe_kind;
  e->probe_lev = h->probe_lev;
  e->probe_idx = h->probe_idx;
  e->err = h->err;
  e->cycle = h->cycle;
  e->xin = h->xin;
  e->yout = h->yout;
  e->nsm = h->nsm;
  if (const char *ev = std::getenv("MLDG_STG_S")) e->stg_stages = std::max(2, std::min(kStgMaxStages, std::atoi(ev)));
  Arena &ar = h->arena;
  e->lv.resize(h->nlev);
  // triangular solves: the grouped solve, unless the environment asks for one
  // of the others
  bool want_grp = std::getenv("MLDG_NO_GRP") == nullptr;
  for (const char *v : {"MLDG_ELL1", "MLDG_WIN_ALL", "MLDG_REP_FORCE", "MLDG_REP_MIN", "MLDG_BLK", "MLDG_BLK_FORCE"})
    want_grp = want_grp && !std::getenv(v);
  for (int l = 0; l < h->nlev; ++l) {
    HostLevel &H = h->host[l];
    auto &L = e->lv[l];
    L.n = H.A.nr;
    L.kind = H.kind;
    L.spre = H.sweeps_pre;
    L.spost = H.sweeps_post;
    L.damp = H.damp;
    const bool h16 = std::is_same<T, float>::value && h->precision == MLDG_PREC_FP32_H16;
    L.A = to_dev<T>(ar, H.A, h16);
    tick("A upload");
    L.AT = to_dev<T>(ar, transpose(H.A), h16);
    tick("A^T transpose + upload");
    if (l > 0) {
      L.P = to_dev<T>(ar, H.P, h16);
      L.R = to_dev<T>(ar, H.R, h16);
      if (std::is_same<T, float>::value && h->precision == MLDG_PREC_FP32_P16) {
        // FP16 values with an FP32 per-row scale = max |p_ij| of the row
        std::vector<__half> hv(H.P.val.size());
        std::vector<float> sc((size_t)H.P.nr, 1.f);
        for (int i = 0; i < H.P.nr; ++i) {
          double mx = 0;
          for (int k = H.P.irp[i]; k < H.P.irp[i + 1]; ++k) mx = std::max(mx, std::fabs(H.P.val[k]));
          sc[i] = mx > 0 ? (float)mx : 1.f;
          for (int k = H.P.irp[i]; k < H.P.irp[i + 1]; ++k)
            hv[k] = __float2half_rn((float)(H.P.val[k] / sc[i]));
        }
        L.Ph = ar.upload(hv);
        L.Pscale = ar.upload(sc);
      }
    }
    L.nnz_nd = H.ND.nnz();
    if (H.kind == MLDG_SMOOTHER_BJAC || H.kind == MLDG_SMOOTHER_FBGS) {
      L.nnz_l = H.L.nnz();
      L.nnz_u = H.U.nnz();
    }
    tick("matrices (A, A^T, P, R upload)");
    const bool dense_coarse = H.kind == MLDG_SMOOTHER_BJAC && l == h->nlev - 1 && h->nlev > 1 &&
                              L.n <= kDenseCoarseRows && !std::getenv("MLDG_NO_DENSE_COARSE");
    // The grouped solve for every other ILU(0) and GS level, except the large
    // ILU(0) levels with wide rows (a coarse level's, above eight entries a
    // row), which the cluster solve runs faster: the fill of a wide row grows
    // with its square (idim=101 level 1, 129,684 rows of 14 entries: 256 us a
    // cluster solve, 290 us a grouped one; level 0, 3 entries: 356 -> 155 us).
    L.grp = want_grp && L.n > 0 && !dense_coarse &&
            (H.kind == MLDG_SMOOTHER_FBGS ||
             (H.kind == MLDG_SMOOTHER_BJAC &&
              (L.n <= 65536 || H.L.nnz() <= 8 * (int64_t)L.n || std::getenv("MLDG_NO_REP"))));
    // level schedules of the four factors: what the other plans are made from,
    // and the solves that need none (k_trsv_sf, k_trsv_sf_m)
    if (H.kind == MLDG_SMOOTHER_BJAC) {
      L.L = build_tri_dev<T>(ar, H.L, false, h->nsm);
      L.U = build_tri_dev<T>(ar, H.U, true, h->nsm);
      tick("L, U schedules");
      HostCSR Lt = transpose(H.L), Ut = transpose(H.U);
      tick("L^T, U^T transposes");
      L.Ut = build_tri_dev<T>(ar, Ut, false, h->nsm);  // U^T is lower
      L.Lt = build_tri_dev<T>(ar, Lt, true, h->nsm);   // L^T is upper
      if (std::getenv("MLDG_VERBOSE")) {
        const DTri<T> *ts[4] = {&L.L, &L.U, &L.Ut, &L.Lt};
        const char *nm[4] = {"L", "U", "Ut", "Lt"};
        for (int q = 0; q < 4; ++q)
          std::fprintf(stderr,
                       "mldg: level %d %-2s n=%d nnz=%lld levels=%d mode=%d tpr=%d e=%d D=%d "
                       "capR=%d capE=%d smem=%zu grid=%d\n",
                       l, nm[q], ts[q]->n, (long long)ts[q]->nnz, ts[q]->nlevels, ts[q]->mode,
                       ts[q]->tpr, ts[q]->e, ts[q]->stg.D, ts[q]->stg.capR, ts[q]->stg.capE,
                       ts[q]->smem, ts[q]->grid);
      }
    }
    tick("level schedules");
    std::vector<double> dh = H.d;
    if (H.kind == MLDG_SMOOTHER_FBGS) {
      // (D+L)^{-1} and (D+U)^{-1} as unit-triangular solves of the rows
      // scaled by 1/a_ii, the right-hand side scaled by 1/a_ii
      for (double &v : dh) v = 1.0 / v;
      HostCSR Ls = H.L, Us = H.U;
      for (int i = 0; i < Ls.nr; ++i) {
        for (int k = Ls.irp[i]; k < Ls.irp[i + 1]; ++k) Ls.val[k] *= dh[i];
        for (int k = Us.irp[i]; k < Us.irp[i + 1]; ++k) Us.val[k] *= dh[i];
      }
      L.L = build_tri_dev<T>(ar, Ls, false, h->nsm);
      L.U = build_tri_dev<T>(ar, Us, true, h->nsm);
      if (std::max(H.sweeps_pre, H.sweeps_post) > 1) {
        // later sweeps: wv = x - U xit (forward) / x - L xit (backward)
        L.GU = to_dev<T>(ar, H.U);
        L.GL = to_dev<T>(ar, H.L);
      }
    }
    tick("FBGS factors");
    // a refused grouped plan leaves the level to its other solves, planned below
    if (L.grp) {
      L.h_d = dh;
      L.grp = e->build_grp(L, 1, 0, ar);
      tick("grouped plans");
    }
    if (H.kind == MLDG_SMOOTHER_BJAC && !L.grp && !std::getenv("MLDG_NO_WIN")) {
      const int n = H.A.nr;
      // Single-CTA windows win on small levels; large levels stay on the
      // sync-free solve unless MLDG_WIN_ALL asks for clusters everywhere.
      const int C = n > 1000000 ? 16 : (n > 65536 ? 4 : 1);
      const bool try_win = C == 1 || std::getenv("MLDG_WIN_ALL");
      HostCSR Lt = transpose(H.L), Ut = transpose(H.U);
      if (try_win) {
        L.wL = build_win_plan<T>(H.L, false, C);
        L.wU = build_win_plan<T>(H.U, true, C);
        L.wUt = build_win_plan<T>(Ut, false, C);
        L.wLt = build_win_plan<T>(Lt, true, C);
      }
      if (try_win && L.wL.ok && L.wU.ok && L.wUt.ok && L.wLt.ok) {
        L.win = true;
        upload_win(ar, L.wL, H.L, false);
        upload_win(ar, L.wU, H.U, true);
        upload_win(ar, L.wUt, Ut, false);
        upload_win(ar, L.wLt, Lt, true);
        link_pair(ar, L.wL, L.wU, H.d);
        link_pair(ar, L.wUt, L.wLt, H.d);
        L.rp0 = ar.alloc<T>((size_t)n + 8);
        L.rp1 = ar.alloc<T>((size_t)n + 8);
        MLDG_CUDA(cudaMemset(L.rp0, 0, sizeof(T) * ((size_t)n + 8)));
        MLDG_CUDA(cudaMemset(L.rp1, 0, sizeof(T) * ((size_t)n + 8)));
        if (std::getenv("MLDG_VERBOSE")) {
          const DWin<T> *ws[4] = {&L.wL, &L.wU, &L.wUt, &L.wLt};
          for (int q = 0; q < 4; ++q)
            std::fprintf(stderr, "mldg: level %d win%d n=%d C=%d W=%d steps=%d D=%d capR=%d capE=%d tpr=%d smem=%zu\n",
                         l, q, ws[q]->n, ws[q]->C, ws[q]->W, ws[q]->nsteps, ws[q]->D, ws[q]->capR,
                         ws[q]->capE, ws[q]->tpr, ws[q]->smem);
        }
      }
    }
    tick("window plans");
    if (H.ND.present() && L.nnz_nd > 0) {
      if (H.kind == MLDG_SMOOTHER_JACOBI && std::max(H.sweeps_pre, H.sweeps_post) <= 2 &&
          !std::getenv("MLDG_NO_ND_SCALE")) {
        // only first sweeps: ND D and ND^T D (columns scaled by d = 1/a_jj)
        auto colscale = [&](HostCSR m) {
          for (size_t k = 0; k < m.ja.size(); ++k) m.val[k] *= dh[m.ja[k]];
          return m;
        };
        L.ND = to_dev<T>(ar, colscale(H.ND), h16);
        L.NDT = to_dev<T>(ar, colscale(transpose(H.ND)), h16);
        L.nd_scaled = true;
      } else {
        L.ND = to_dev<T>(ar, H.ND, h16);
        L.NDT = to_dev<T>(ar, transpose(H.ND), h16);
      }
    }
    tick("ND");
    if (dense_coarse) {
      std::vector<double> M, MT;
      dense_ilu_inverse(H.L, H.U, H.d, M, MT);
      std::vector<T> m(M.begin(), M.end()), mt(MT.begin(), MT.end());
      L.minv = ar.upload(m);
      L.minvT = ar.upload(mt);
    }
    tick("dense coarsest inverse");
    // replicated-window cluster solves (k_trsv_rep) for the large ILU(0) levels
    {
      int rep_min = 65536;
      if (const char *ev = std::getenv("MLDG_REP_MIN")) rep_min = std::atoi(ev);
      if (H.kind == MLDG_SMOOTHER_BJAC && !L.minv && !L.win && !L.grp && L.n > rep_min && !std::getenv("MLDG_NO_REP")) {
        int C = 16;
        if (const char *ev = std::getenv("MLDG_REP_C")) C = std::atoi(ev) == 8 ? 8 : 16;
        HostCSR Lt = transpose(H.L), Ut = transpose(H.U);
        L.rL = build_rep_sched<T>(H.L, false, C);
        L.rU = build_rep_sched<T>(H.U, true, C);
        L.rUt = build_rep_sched<T>(Ut, false, C);
        L.rLt = build_rep_sched<T>(Lt, true, C);
        DRep<T> *rs[4] = {&L.rL, &L.rU, &L.rUt, &L.rLt};
        bool ok = L.rL.ok && L.rU.ok && L.rUt.ok && L.rLt.ok;
        if (ok) {
          build_rep_blocks(ar, L.rL, &L.rU, &H.d);
          build_rep_blocks(ar, L.rU, (const DRep<T> *)nullptr, (const std::vector<double> *)nullptr);
          build_rep_blocks(ar, L.rUt, &L.rLt, &H.d);
          build_rep_blocks(ar, L.rLt, (const DRep<T> *)nullptr, (const std::vector<double> *)nullptr);
          for (DRep<T> *r : rs) ok = ok && r->ok && rep_fits(*r);
        }
        for (DRep<T> *r : rs) rep_release_sched(*r);
        L.rep_ok = ok;
        if (ok && !L.rp0) {
          L.rp0 = ar.alloc<T>((size_t)L.n + 8);
          L.rp1 = ar.alloc<T>((size_t)L.n + 8);
          MLDG_CUDA(cudaMemset(L.rp0, 0, sizeof(T) * ((size_t)L.n + 8)));
          MLDG_CUDA(cudaMemset(L.rp1, 0, sizeof(T) * ((size_t)L.n + 8)));
        }
        if (std::getenv("MLDG_VERBOSE")) {
          const char *nm[4] = {"L", "U", "Ut", "Lt"};
          for (int q = 0; q < 4; ++q)
            std::fprintf(stderr,
                         "mldg: level %d rep %-2s n=%d C=%d steps=%d R=%d far=%lld capB=%d stage=%d smem=%zu "
                         "blocks=%.1f MB ok=%d\n",
                         l, nm[q], rs[q]->n, rs[q]->C, rs[q]->nsteps, rs[q]->R, (long long)rs[q]->nfar,
                         rs[q]->capB, rs[q]->stage_bytes, rs[q]->smem, rs[q]->block_bytes / 1e6, (int)rs[q]->ok);
        }
      }
    }
    tick("replicated-window plans");
    // partitioned solves (k_trsv_blk) for the ILU(0) levels that keep their
    // solves: built only on request (MLDG_BLK=1, or MLDG_BLK_FORCE), since on
    // the pdegen hierarchies measured so far the other solves are faster
    // (level 0 at idim=160: 2.2 ms per pair vs 1.3 ms; coarse levels far slower)
    {
      int blk_min = 4096;
      if (const char *ev = std::getenv("MLDG_BLK_MIN")) blk_min = std::atoi(ev);
      const bool want = std::getenv("MLDG_BLK") || std::getenv("MLDG_BLK_FORCE");
      if (want && H.kind == MLDG_SMOOTHER_BJAC && !L.minv && L.n >= blk_min && !std::getenv("MLDG_NO_BLK")) {
        int P = std::min(h->nsm, std::max(1, L.n / 1024));
        if (const char *ev = std::getenv("MLDG_BLK_P")) P = std::max(1, std::atoi(ev));
        HostCSR Lt = transpose(H.L), Ut = transpose(H.U);
        L.kL = build_blk_plan<T>(ar, H.L, false, P);
        L.kU = build_blk_plan<T>(ar, H.U, true, P);
        L.kUt = build_blk_plan<T>(ar, Ut, false, P);
        L.kLt = build_blk_plan<T>(ar, Lt, true, P);
        L.blk_ok = L.kL.ok && L.kU.ok && L.kUt.ok && L.kLt.ok;
        if (std::getenv("MLDG_VERBOSE")) {
          const DBlk<T> *ks[4] = {&L.kL, &L.kU, &L.kUt, &L.kLt};
          const char *nm[4] = {"L", "U", "Ut", "Lt"};
          for (int q = 0; q < 4; ++q)
            std::fprintf(stderr, "mldg: level %d blk %-2s n=%d P=%d steps=%d W=%d stage=%d smem=%zu plan=%.1f MB ok=%d\n",
                         l, nm[q], ks[q]->n, ks[q]->nblocks, ks[q]->nsteps, ks[q]->W, ks[q]->stage_bytes,
                         ks[q]->smem, ks[q]->plan_bytes / 1e6, (int)ks[q]->ok);
        }
      }
    }
    tick("partitioned-solve plans");
    std::vector<T> dv(dh.begin(), dh.end());
    L.d = ar.upload(dv);
    const int n = std::max(L.n, 1);
    if (l == 0 && std::is_same<T, double>::value) {
      L.x = (T *)h->xin;
      L.y = (T *)h->yout;
    } else {
      L.x = ar.alloc<T>(n);
      L.y = ar.alloc<T>(n);
    }
    L.ty = ar.alloc<T>(n);
    L.tz = ar.alloc<T>(n);
    MLDG_CUDA(cudaMemset(L.tz, 0, sizeof(T) * n));
    L.tw = ar.alloc<T>(n);
    MLDG_CUDA(cudaMemset(L.y, 0, sizeof(T) * n));
    MLDG_CUDA(cudaMemset(L.ty, 0, sizeof(T) * n));
    MLDG_CUDA(cudaMemset(L.tw, 0, sizeof(T) * n));
    if ((H.kind == MLDG_SMOOTHER_BJAC || H.kind == MLDG_SMOOTHER_FBGS) && !L.grp) {
      L.bufA = ar.alloc<T>(n);
      L.bufB = ar.alloc<T>(n);
      k_fill<T><<<64, 256, 0, h->st>>>(n, Sentinel<T>::value(), L.bufA);
      k_fill<T><<<64, 256, 0, h->st>>>(n, Sentinel<T>::value(), L.bufB);
      tick("vectors, exchange buffers");
      if (!L.minv) {
        bool ok = true;
        for (DTri<T> *f : {&L.L, &L.U, &L.Ut, &L.Lt}) {
          if (!f->present()) continue;  // FBGS: forward and backward factors only
          e->build_ell(*f, 1, ar);
          ok = ok && f->ell[0].ok;
        }
        tick("ELL plans (one column)");
        const char *ev = std::getenv("MLDG_ELL1");
        L.ell1 = ok && !(ev && ev[0] == '0');
      }
    }
  }
  MLDG_CUDA(cudaStreamSynchronize(h->st));
  e->stg_prepare();
  if (h->opts.autotune && !std::getenv("MLDG_NO_AUTOTUNE")) {
    int nmax = 1;
    for (auto &L : e->lv) nmax = std::max(nmax, L.n);
    e->tune_n = nmax;
    e->tune_buf[0] = ar.alloc<T>(nmax);
    e->tune_buf[1] = ar.alloc<T>(nmax);
    k_fill<T><<<64, 256, 0, h->st>>>(nmax, T(1), e->tune_buf[0]);
    tick("ELL plans");
    e->autotune_spmv(5);
    tick("autotune SpMV");
    if (!std::getenv("MLDG_ELL1")) e->autotune_ilu(3);
    MLDG_CUDA(cudaStreamSynchronize(h->st));
  }
  // small intermediate levels: the explicit inverse of their ILU(0) when faster
  // MLDG_REP_FORCE: every level with replicated-window plans uses them (a
  // value above 1: only the levels of at most that many rows)
  if (const char *ev = std::getenv("MLDG_REP_FORCE"))
    for (auto &L : e->lv)
      if (L.rep_ok && (std::atol(ev) <= 1 || L.n <= std::atol(ev))) {
        L.rep = true;
        L.ell1 = false;
        L.blk = false;
        if (std::getenv("MLDG_VERBOSE")) std::fprintf(stderr, "mldg: level n=%d uses rep (forced)\n", L.n);
      }
  // MLDG_BLK_FORCE: every level with partitioned-solve plans uses them
  if (std::getenv("MLDG_BLK_FORCE"))
    for (auto &L : e->lv)
      if (L.blk_ok) {
        L.blk = true;
        L.rep = false;
        L.ell1 = false;
      }
  // MLDG_SELL_FORCE: every operator with a SELL copy uses it (measurement aid)
  if (std::getenv("MLDG_SELL_FORCE"))
    for (auto &L : e->lv)
      for (DCSR<T> *op : {&L.A, &L.AT, &L.P, &L.R, &L.ND, &L.NDT})
        if (op->soff) {
          const int f = std::atoi(std::getenv("MLDG_SELL_FORCE"));
          op->sell = (f >= 1 && f <= 3) ? f : 1;
        }
  // MLDG_HDIA_FORCE: every operator with an HDIA copy uses it (measurement
  // aid and test hook; the value 16 picks the 16-diagonal passes)
  if (std::getenv("MLDG_HDIA_FORCE"))
    for (auto &L : e->lv)
      for (DCSR<T> *op : {&L.A, &L.AT, &L.P, &L.R, &L.ND, &L.NDT})
        if (op->hdptr && (op->h16() ? op->hdhval != nullptr : op->hdval != nullptr))
        {
          op->sell = 5;
          op->hd16 = std::atoi(std::getenv("MLDG_HDIA_FORCE")) == 16;
        }
  // MLDG_STG_FORCE: every operator with staged tiles uses them
  if (std::getenv("MLDG_STG_FORCE"))
    for (auto &L : e->lv)
      for (DCSR<T> *op : {&L.A, &L.AT, &L.P, &L.R, &L.ND, &L.NDT})
        if (op->tiles) op->sell = 4;
  tick("autotune solves");
  if (!std::getenv("MLDG_NO_DENSE_INV"))
    for (int l = 1; l < h->nlev; ++l) {
      auto &L = e->lv[l];
      if ((L.kind == MLDG_SMOOTHER_BJAC || L.kind == MLDG_SMOOTHER_FBGS) && !L.minv && L.n <= kDenseInvRows)
        e->dense_inverse(L, ar);
    }
  tick("dense level inverses");
  if (std::getenv("MLDG_TIMING"))
    for (auto &kv : tm) std::fprintf(stderr, "mldg timing: finalize %-32s %.3f s\n", kv.first.c_str(), kv.second);
  return owner.release();
}

static void check_level(const HostLevel &H, int l, const HostLevel *prev) {
  const int n = H.A.nr;
  if (!H.A.present()) fail(MLDG_ERR_ARG, "level %d: missing A", l);
  if (H.A.nc != n) fail(MLDG_ERR_ARG, "level %d: A must be square", l);
  if (prev) {
    const int nf = prev->A.nr;
    if (!H.P.present() || !H.R.present()) fail(MLDG_ERR_ARG, "level %d: missing P/R", l);
    if (H.P.nr != nf || H.P.nc != n) fail(MLDG_ERR_ARG, "level %d: P must be %d x %d", l, nf, n);
    if (H.R.nr != n || H.R.nc != nf) fail(MLDG_ERR_ARG, "level %d: R must be %d x %d", l, n, nf);
  }
  if ((int)H.d.size() != n) fail(MLDG_ERR_NO_DIAG, "level %d: missing d (length %d)", l, n);
  if (H.kind == MLDG_SMOOTHER_BJAC || H.kind == MLDG_SMOOTHER_FBGS) {
    if (!H.L.present() || !H.U.present()) fail(MLDG_ERR_NO_SOLVER, "level %d: missing L/U", l);
    if (H.L.nr != n || H.U.nr != n) fail(MLDG_ERR_ARG, "level %d: L/U size", l);
    for (int i = 0; i < n; ++i) {
      for (int k = H.L.irp[i]; k < H.L.irp[i + 1]; ++k)
        if (H.L.ja[k] >= i) fail(MLDG_ERR_ARG, "level %d: L not strictly lower at row %d", l, i);
      for (int k = H.U.irp[i]; k < H.U.irp[i + 1]; ++k)
        if (H.U.ja[k] <= i) fail(MLDG_ERR_ARG, "level %d: U not strictly upper at row %d", l, i);
    }
    if (H.kind == MLDG_SMOOTHER_FBGS)
      for (int i = 0; i < n; ++i)
        if (H.d[i] == 0.0) fail(MLDG_ERR_NO_DIAG, "level %d: zero diagonal at row %d (Gauss-Seidel)", l, i);
  } else if (H.kind != MLDG_SMOOTHER_JACOBI) {
    fail(MLDG_ERR_ARG, "level %d: unknown smoother kind %d", l, H.kind);
  }
  if (H.ND.present() && (H.ND.nr != n || H.ND.nc != n)) fail(MLDG_ERR_ARG, "level %d: ND size", l);
  if (H.sweeps_pre < 0 || H.sweeps_post < 0) fail(MLDG_ERR_ARG, "level %d: negative sweeps", l);
}

static void tune_krylov_spmv(Handle *h);

static void batch_evict(uint64_t serial);

static uint64_t next_serial() {
  static std::atomic<uint64_t> ctr{1};
  return ctr.fetch_add(1);
}

static void finalize(Handle *h, int nlev, int precision) {
  if (nlev < 1 || nlev > (int)h->host.size()) fail(MLDG_ERR_ARG, "nlev %d: %zu levels uploaded", nlev, h->host.size());
  for (int l = 0; l < nlev; ++l)
    if (!h->host[l].uploaded) fail(MLDG_ERR_ARG, "level %d not uploaded", l);
  for (int l = 0; l < nlev; ++l) check_level(h->host[l], l, l ? &h->host[l - 1] : nullptr);
  if (precision != MLDG_PREC_FP64 && precision != MLDG_PREC_FP32 && precision != MLDG_PREC_FP32_P16 &&
      precision != MLDG_PREC_FP32_H16)
    fail(MLDG_ERR_ARG, "unknown precision %d", precision);
  // drop any previous device state
  h->finalized = false;
  for (int t = 0; t < 2; ++t)
    if (h->gexec[t]) {
      cudaGraphExecDestroy(h->gexec[t]);
      h->gexec[t] = nullptr;
    }
  drop_multi_graphs(h);
  drop_krylov_graphs(h);
  batch_evict(h->serial);
  h->serial = 0;
  h->eng.reset();
  h->arena.release();
  h->karena.release();
  h->kcap = 0;
  h->nlev = nlev;
  h->has_fbgs = false;
  for (int l = 0; l < nlev; ++l) h->has_fbgs = h->has_fbgs || h->host[l].kind == MLDG_SMOOTHER_FBGS;
  h->precision = precision;
  h->n0 = h->host[0].A.nr;
  const int n0 = std::max(h->n0, 1);
  h->err = h->arena.alloc<int>(1);
  MLDG_CUDA(cudaMemset(h->err, 0, sizeof(int)));
  h->xin = h->arena.alloc<double>(n0);
  h->yout = h->arena.alloc<double>(n0);
  MLDG_CUDA(cudaMemset(h->xin, 0, sizeof(double) * n0));
  MLDG_CUDA(cudaMemset(h->yout, 0, sizeof(double) * n0));
  h->A0 = to_dev<double>(h->arena, h->host[0].A);
  h->A0T = DCSR<double>();
  h->kb = h->arena.alloc<double>(n0);
  h->kx = h->arena.alloc<double>(n0);
  h->kd = h->arena.alloc<double>(n0);
  h->kd1 = h->arena.alloc<double>(n0);
  h->kq = h->arena.alloc<double>(n0);
  // partials: 3 per reduction block, or 2 per block of the fused SpMV
  h->kpart = h->arena.alloc<double>(std::max(3 * kRedBlocks, 2 * 16 * h->nsm));
  h->kst = h->arena.alloc<KState>(1);
  h->kpar = h->arena.alloc<KParams>(1);
  if (!h->hkst) MLDG_CUDA(cudaMallocHost(&h->hkst, sizeof(KState)));
  if (!h->hkpar) MLDG_CUDA(cudaMallocHost(&h->hkpar, sizeof(KParams)));
  if (precision == MLDG_PREC_FP64)
    h->eng.reset(make_engine<double>(h));
  else
    h->eng.reset(make_engine<float>(h));
  h->finalized = true;
  h->serial = next_serial();
  if (h->opts.autotune && !std::getenv("MLDG_NO_AUTOTUNE")) tune_krylov_spmv(h);
  if (std::getenv("MLDG_SELL_FORCE")) h->A0.sell = h->A0.soff != nullptr ? 1 : 0;
  if (std::getenv("MLDG_HDIA_FORCE") && h->A0.hdptr && h->A0.hdval) h->A0.sell = 5;
}

static bool kcycle_handle(const Handle *h) { return h->cycle == MLDG_CYCLE_K || h->cycle == MLDG_CYCLE_KSYM; }

static void run_vcycle(Handle *h, char trans) {
  const int t = (trans == 'N') ? 0 : 1;
  if (h->opts.use_graphs && !kcycle_handle(h)) {
    if (!h->gexec[t]) {
      cudaGraph_t g;
      MLDG_CUDA(cudaStreamBeginCapture(h->st, cudaStreamCaptureModeThreadLocal));
      h->eng->capturing = true;
      try {
        h->eng->record(trans);
      } catch (...) {
        h->eng->capturing = false;
        cudaStreamEndCapture(h->st, &g);
        throw;
      }
      h->eng->capturing = false;
      MLDG_CUDA(cudaStreamEndCapture(h->st, &g));
      MLDG_CUDA(cudaGraphInstantiate(&h->gexec[t], g, 0));
      cudaGraphDestroy(g);
      h->glaunch[t] = h->eng->launches;
      h->gbytes[t] = h->eng->bytes;
      h->gimpl[t] = h->eng->impl_bytes;
      h->gprobe[t] = h->eng->probe_armed;
      if (h->eng->probe_armed) h->probe_bytes = h->eng->probe_bytes;
    }
    MLDG_CUDA(cudaGraphLaunch(h->gexec[t], h->st));
    h->last_launches += h->glaunch[t];
    h->pending = h->gprobe[t];
  } else {
    h->eng->record(trans);
    h->glaunch[t] = h->eng->launches;
    h->gbytes[t] = h->eng->bytes;
    h->gimpl[t] = h->eng->impl_bytes;
    h->last_launches += h->eng->launches;
    h->pending = h->eng->probe_armed;
    if (h->eng->probe_armed) h->probe_bytes = h->eng->probe_bytes;
  }
}

// after a stream synchronisation: account the probed launch, if any
static void probe_collect(Handle *h) {
  if (!h->pending) return;
  float ms = 0;
  MLDG_CUDA(cudaEventElapsedTime(&ms, h->pev0, h->pev1));
  h->probe_ms += ms;
  h->probe_count += 1;
  h->pending = false;
}

static int check_device_error(Handle *h) {
  int e = 0;
  MLDG_CUDA(cudaMemcpy(&e, h->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    // the solve that gave up may have left exchange buffers written and
    // counters advanced: restore them before the handle is used again
    if (h->eng) h->eng->reset_solve_state();
    MLDG_CUDA(cudaMemset(h->err, 0, sizeof(int)));
    fail(MLDG_ERR_TIMEOUT, "a triangular-solve dependency wait exceeded its limit (code %d)", e);
  }
  return 0;
}

static void run_vcycle_multi(Handle *h, char trans, int K) {
  const int t = (trans == 'N') ? 0 : 1, q = ilog2(K);
  if (h->opts.use_graphs) {
    if (!h->gexec_m[t][q]) {
      cudaGraph_t g;
      MLDG_CUDA(cudaStreamBeginCapture(h->st, cudaStreamCaptureModeThreadLocal));
      h->eng->capturing = true;
      try {
        h->eng->record_multi(trans, K);
      } catch (...) {
        h->eng->capturing = false;
        cudaStreamEndCapture(h->st, &g);
        throw;
      }
      h->eng->capturing = false;
      MLDG_CUDA(cudaStreamEndCapture(h->st, &g));
      MLDG_CUDA(cudaGraphInstantiate(&h->gexec_m[t][q], g, 0));
      cudaGraphDestroy(g);
      h->glaunch_m[t][q] = h->eng->launches;
      h->gprobe_m[t][q] = h->eng->probe_armed;
      if (h->eng->probe_armed) h->probe_bytes = h->eng->probe_bytes;
    }
    MLDG_CUDA(cudaGraphLaunch(h->gexec_m[t][q], h->st));
    h->last_launches += h->glaunch_m[t][q];
    h->pending = h->gprobe_m[t][q];
  } else {
    h->eng->record_multi(trans, K);
    h->glaunch_m[t][q] = h->eng->launches;
    h->last_launches += h->eng->launches;
    h->pending = h->eng->probe_armed;
    if (h->eng->probe_armed) h->probe_bytes = h->eng->probe_bytes;
  }
}

// columns [c0, c0+k) of a column-major (ld) FP64 block, host or device, into
// the K-wide interleaved device buffer dst (columns >= k zero)
static void load_block(Handle *h, const double *src, int ld, int k, int K, int mem, double *dst) {
  const int n = h->n0;
  int sld = ld;
  if (mem == MLDG_MEM_HOST) {
    MLDG_CUDA(cudaMemcpy2DAsync(h->eng->col_m, sizeof(double) * n, src, sizeof(double) * ld, sizeof(double) * n, k,
                                cudaMemcpyHostToDevice, h->st));
    src = h->eng->col_m;
    sld = n;
  }
  const int64_t tot = (int64_t)n * K;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, (int64_t)h->nsm * 16));
  k_to_interleaved<double><<<g, 256, 0, h->st>>>(n, k, K, sld, src, dst);
  h->last_launches++;
}
static void store_block(Handle *h, const double *src, int k, int K, int mem, double *dst, int ld) {
  const int n = h->n0;
  const int64_t tot = (int64_t)n * k;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, (int64_t)h->nsm * 16));
  if (mem == MLDG_MEM_HOST) {
    k_from_interleaved<double><<<g, 256, 0, h->st>>>(n, k, K, n, src, h->eng->col_m);
    MLDG_CUDA(cudaMemcpy2DAsync(dst, sizeof(double) * ld, h->eng->col_m, sizeof(double) * n, sizeof(double) * n, k,
                                cudaMemcpyDeviceToHost, h->st));
  } else {
    k_from_interleaved<double><<<g, 256, 0, h->st>>>(n, k, K, ld, src, dst);
  }
  h->last_launches++;
}
static int width_for(int k) {
  int K = 2;
  while (K < k) K *= 2;
  return K;
}
// Buffers and plans for K columns.  Where an allocation fails, the graphs that
// hold the old ones and whatever was half made go, so that the next call
// starts over.
static void prepare_multi(Handle *h, int K, char trans) {
  try {
    if (h->eng->ensure_multi(K, trans)) drop_multi_graphs(h);
  } catch (...) {
    drop_multi_graphs(h);
    h->eng->release_multi();
    throw;
  }
}

// nrhs > 1: blocks of up to 32 columns through the K-wide V-cycle
static void apply_multi(Handle *h, const double *x, double *y, char trans, int nrhs, int ld, int mem) {
  for (int c0 = 0; c0 < nrhs; c0 += 32) {
    const int k = std::min(32, nrhs - c0), K = width_for(k);
    prepare_multi(h, K, trans);
    load_block(h, x + (size_t)c0 * ld, ld, k, K, mem, h->eng->xin_m);
    run_vcycle_multi(h, trans, K);
    store_block(h, h->eng->yout_m, k, K, mem, y + (size_t)c0 * ld, ld);
    if (h->pending) {
      MLDG_CUDA(cudaStreamSynchronize(h->st));
      probe_collect(h);
    }
  }
}

static void apply(Handle *h, const double *x, double *y, char trans, int nrhs, int ld, int mem) {
  if (!h->finalized) fail(MLDG_ERR_NOT_BUILT, "apply before build (mldg_finalize not called)");
  if (trans == 'C') trans = 'T';
  if (trans != 'N' && trans != 'T') fail(MLDG_ERR_TRANS, "invalid trans '%c'", trans);
  check_trans(h, trans);
  if (nrhs < 0) fail(MLDG_ERR_ARG, "nrhs < 0");
  const int n = h->n0;
  if (nrhs > 1 && ld < n) fail(MLDG_ERR_SIZE, "ld %d < n %d", ld, n);
  if (nrhs > 0 && (!x || !y)) fail(MLDG_ERR_ARG, "null vector");
  if (mem != MLDG_MEM_HOST && mem != MLDG_MEM_DEVICE) fail(MLDG_ERR_ARG, "bad mem_kind");
  const cudaMemcpyKind h2d = mem == MLDG_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind d2h = mem == MLDG_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  h->last_launches = 0;
  MLDG_CUDA(cudaEventRecord(h->ev0, h->st));
  const char *em = std::getenv("MLDG_MULTI");
  const bool multi = nrhs > 1 && !(em && em[0] == '0') && !kcycle_handle(h);
  if (multi) apply_multi(h, x, y, trans, nrhs, ld, mem);
  for (int c = 0; c < (multi ? 0 : nrhs); ++c) {
    const size_t off = (size_t)c * (size_t)(nrhs > 1 ? ld : n);
    MLDG_CUDA(cudaMemcpyAsync(h->xin, x + off, sizeof(double) * n, h2d, h->st));
    run_vcycle(h, trans);
    MLDG_CUDA(cudaMemcpyAsync(y + off, h->yout, sizeof(double) * n, d2h, h->st));
    if (h->pending) {
      MLDG_CUDA(cudaStreamSynchronize(h->st));
      probe_collect(h);
    }
  }
  MLDG_CUDA(cudaEventRecord(h->ev1, h->st));
  MLDG_CUDA(cudaStreamSynchronize(h->st));
  float ms = 0;
  MLDG_CUDA(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
  h->last_ms = ms;
  check_device_error(h);
}

// ---------------------------------------------------------------------------
static void spmv64(Handle *h, const DCSR<double> &A, const double *v, double a1, const double *b,
                   double a0, double *out) {
  const int64_t thr = (int64_t)A.nr * A.tpr;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((thr + 255) / 256, (int64_t)h->nsm * 16));
  switch (A.tpr) {
#define CASE(K)                                                                                         \
  case K:                                                                                               \
    if (A.jd)                                                                                           \
      k_spmv<double, K, short><<<g, 256, 0, h->st>>>(A.nr, A.irp, A.jd, A.val, v, a1, b, a0, out, 0.0); \
    else                                                                                                \
      k_spmv<double, K, int><<<g, 256, 0, h->st>>>(A.nr, A.irp, A.ja, A.val, v, a1, b, a0, out, 0.0);   \
    break;
    CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32)
#undef CASE
    default: fail(MLDG_ERR_INTERNAL, "bad tpr");
  }
  h->last_launches++;
}

// The initial residual r = b - A x and the Krylov state (k_kry_init) from
// the parameters in h->kpar; hc != 0 also sets the graph conditional.
static void krylov_prefix(Handle *h, const DCSR<double> &A, cudaGraphConditionalHandle hc) {
  const int n = h->n0;
  spmv64(h, A, h->kx, -1.0, h->kb, 1.0, h->xin);  // r = b - A x
  if (h->kio) {  // the first V-cycle's FP32 input
    k_cast<double, float><<<(int)std::min<int64_t>(((int64_t)n + 255) / 256, (int64_t)h->nsm * 8), 256, 0, h->st>>>(
        n, h->xin, h->eng->kry_x32());
    h->last_launches++;
  }
  k_dots<<<kRedBlocks, kRedThreads, 0, h->st>>>(n, 2, h->kb, h->kb, h->xin, h->xin, nullptr, nullptr,
                                                h->kpart);
  k_kry_init<<<1, kRedThreads, 0, h->st>>>(kRedBlocks, h->kpart, h->kpar, h->kst, hc);
  h->last_launches += 2;
}

// One CG/FCG iteration after the preconditioner apply z = M^{-1} r (in yout):
// three fused kernels (mldg_kernels.cuh, k_kry_*); every kernel returns at
// once when the device state says the solve is done.
template <typename ZT>
static void kry_spmv_z(Handle *h, const DCSR<double> &A, const ZT *z) {
  const bool pdl = h->eng->pdl_on();
  double *r = h->xin;
  if (A.hdia() && A.hdval) {
    const int64_t thr = (int64_t)A.hd_nslice() * 32;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((thr + 255) / 256, (int64_t)h->nsm * 16));
    launch_k(pdl, k_kry_spmv_hdia<ZT>, g, 256, h->st, A.nr, A.hdptr, A.hdoff, A.hdval, z, h->kd, h->kd1, h->kq, r, h->kst,
                                          h->kpart);
    return;
  }
  if (A.sell) {
    // grid: at most 16 blocks per SM (the partials hold 2 per block)
    const int64_t thr = (int64_t)A.nslice() * 32;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((thr + 255) / 256, (int64_t)h->nsm * 16));
    if (A.sjd)
      launch_k(pdl, k_kry_spmv_sell<short, ZT>, g, 256, h->st, A.nr, A.soff, A.sjd, A.sval, z, h->kd, h->kd1, h->kq, r,
                                                   h->kst, h->kpart);
    else
      launch_k(pdl, k_kry_spmv_sell<int, ZT>, g, 256, h->st, A.nr, A.soff, A.sja, A.sval, z, h->kd, h->kd1, h->kq, r,
                                                 h->kst, h->kpart);
    return;
  }
  const int64_t thr = (int64_t)A.nr * A.tpr;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((thr + 255) / 256, (int64_t)h->nsm * 16));
  switch (A.tpr) {
#define CASE(K)                                                                                  \
  case K:                                                                                        \
    if (A.jd)                                                                                    \
      launch_k(pdl, k_kry_spmv<K, short, ZT>, g, 256, h->st, A.nr, A.irp, A.jd, A.val, z, h->kd, h->kd1, h->kq, r, \
                                                 h->kst, h->kpart);                              \
    else                                                                                         \
      launch_k(pdl, k_kry_spmv<K, int, ZT>, g, 256, h->st, A.nr, A.irp, A.ja, A.val, z, h->kd, h->kd1, h->kq, r,   \
                                               h->kst, h->kpart);                                \
    break;
    CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32)
#undef CASE
    default: fail(MLDG_ERR_INTERNAL, "bad tpr");
  }
}

// z: the V-cycle's FP64 output, or its FP32 output when h->kio is set
static void kry_spmv(Handle *h, const DCSR<double> &A) {
  if (h->kio)
    kry_spmv_z<float>(h, A, h->eng->kry_y32());
  else
    kry_spmv_z<double>(h, A, h->yout);
}

static void krylov_iteration(Handle *h, const DCSR<double> &A, cudaGraphConditionalHandle hc) {
  const bool pdl = h->eng->pdl_on();
  const int n = h->n0;
  double *r = h->xin;
  // vector kernels: 8 blocks of 256 threads per SM (64 warps), so that enough
  // loads are in flight to stream the vectors at HBM bandwidth
  const int gv = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n + 255) / 256, (int64_t)h->nsm * 8));
  if (h->kio)
    launch_k(pdl, k_kry_beta<float>, gv, kRedThreads, h->st, n, (const float *)h->eng->kry_y32(), h->kq, r, h->kst,
             h->kpart);
  else
    launch_k(pdl, k_kry_beta<double>, gv, kRedThreads, h->st, n, (const double *)h->yout, h->kq, r, h->kst,
             h->kpart);
  kry_spmv(h, A);
  launch_k(pdl, k_kry_update, gv, kRedThreads, h->st, n, (const double *)h->kd, (const double *)h->kd1,
           (const double *)h->kq, h->kx, r, h->kst, h->kpart, hc, h->kio ? h->eng->kry_x32() : (float *)nullptr);
  h->last_launches += 3;
}

// Lanes per row of the finest matrix in the fused Krylov SpMV, picked by
// timing (finalize): the state is set to a mid-solve iteration on zero
// vectors, and the kernel is timed for each width.
static void tune_krylov_spmv(Handle *h) {
  DCSR<double> &A = h->A0;
  if (!A.present() || A.nr == 0) return;
  char key[128];
  std::snprintf(key, sizeof key, "kry %d %lld", A.nr, (long long)A.nnz);
  {
    const auto kept = tune_file_read();
    const auto kc = kept.find(key);
    if (kc != kept.end()) {
      A.tpr = kc->second[0];
      A.sell = kc->second[1];
      return;
    }
  }
  KState s0 = {};
  s0.bn2 = 1.0;
  s0.it = 1;
  s0.itmax = 1 << 30;
  s0.method = 1;
  s0.beta = 0.5;
  cudaEvent_t e0, e1;
  MLDG_CUDA(cudaEventCreate(&e0));
  MLDG_CUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  int best_t = A.tpr;
  int best_sell = 0;
  for (double *v : {h->kd, h->kd1, h->kq}) MLDG_CUDA(cudaMemsetAsync(v, 0, sizeof(double) * (size_t)h->n0, h->st));
  // t = 0: the SELL copy; t = -1: the HDIA copy
  for (int t : {1, 2, 4, 8, 16, 32, 0, -1}) {
    if (t == 0 && !A.soff) continue;
    if (t == -1 && !(A.hdptr && A.hdval)) continue;
    A.sell = t == 0 ? 1 : (t == -1 ? 5 : 0);
    if (t > 0) A.tpr = t;
    *h->hkst = s0;
    MLDG_CUDA(cudaMemcpyAsync(h->kst, h->hkst, sizeof(KState), cudaMemcpyHostToDevice, h->st));
    kry_spmv(h, A);  // warm
    MLDG_CUDA(cudaEventRecord(e0, h->st));
    for (int r = 0; r < 5; ++r) kry_spmv(h, A);
    MLDG_CUDA(cudaEventRecord(e1, h->st));
    MLDG_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    MLDG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < best) {
      best = ms;
      best_t = t > 0 ? t : best_t;
      best_sell = t == 0 ? 1 : (t == -1 ? 5 : 0);
    }
  }
  A.tpr = best_t;
  A.sell = best_sell;
  tune_file_append(std::string(key) + " " + std::to_string(best_t) + " " + std::to_string(best_sell));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // leave clean vectors behind
  MLDG_CUDA(cudaMemsetAsync(h->kd, 0, sizeof(double) * (size_t)h->n0, h->st));
  MLDG_CUDA(cudaMemsetAsync(h->kd1, 0, sizeof(double) * (size_t)h->n0, h->st));
  MLDG_CUDA(cudaMemsetAsync(h->kq, 0, sizeof(double) * (size_t)h->n0, h->st));
  MLDG_CUDA(cudaStreamSynchronize(h->st));
}

// Captures a whole solve (method, trans) on the handle's own matrix A as one
// graph: prefix, then a WHILE node whose body is the V-cycle and one
// iteration.  The stopping test runs on the device, so the solve makes no
// host round trip; the iteration count is read back afterwards.
// FP32 V-cycle inside a captured CG/FCG solve: no precision casts at its
// ends (Engine::kry_io); MLDG_NO_KRY_IO keeps them
static bool kry_io_ok(Handle *h) { return h->eng->kry_y32() != nullptr && !std::getenv("MLDG_NO_KRY_IO"); }
struct KioScope {  // sets h->kio and the engine's kry_io for one capture
  Handle *h;
  KioScope(Handle *hh, bool on) : h(hh) {
    h->kio = on;
    h->eng->kry_io = on;
  }
  ~KioScope() {
    h->kio = false;
    h->eng->kry_io = false;
  }
};

static void capture_solve(Handle *h, int method, char trans, const DCSR<double> &A) {
  const int t = trans == 'N' ? 0 : 1;
  if (h->sgraph[method][t]) return;
  cudaGraph_t g = nullptr;
  MLDG_CUDA(cudaGraphCreate(&g, 0));
  const int64_t l0 = h->last_launches;
  KioScope kio(h, kry_io_ok(h));
  try {
    cudaGraphConditionalHandle hc;
    MLDG_CUDA(cudaGraphConditionalHandleCreate(&hc, g, 0, cudaGraphCondAssignDefault));
    // prefix, captured into g (a linear chain)
    MLDG_CUDA(cudaStreamBeginCaptureToGraph(h->st, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    try {
      krylov_prefix(h, A, hc);
    } catch (...) {
      cudaGraph_t tmp;
      cudaStreamEndCapture(h->st, &tmp);
      throw;
    }
    cudaGraph_t gout = nullptr;
    MLDG_CUDA(cudaStreamEndCapture(h->st, &gout));
    const int64_t lpre = h->last_launches - l0;
    // the sink of the prefix chain
    size_t nn = 0;
    MLDG_CUDA(cudaGraphGetNodes(g, nullptr, &nn));
    std::vector<cudaGraphNode_t> nodes(nn);
    MLDG_CUDA(cudaGraphGetNodes(g, nodes.data(), &nn));
    cudaGraphNode_t sink = nullptr;
    for (cudaGraphNode_t nd : nodes) {
      size_t nd_out = 0;
      MLDG_CUDA(cudaGraphNodeGetDependentNodes(nd, nullptr, &nd_out));
      if (nd_out == 0) {
        if (sink) fail(MLDG_ERR_INTERNAL, "solve graph: prefix is not a chain");
        sink = nd;
      }
    }
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = hc;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t cn;
    MLDG_CUDA(cudaGraphAddNode(&cn, g, sink ? &sink : nullptr, sink ? 1 : 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const int64_t l1 = h->last_launches;
    MLDG_CUDA(cudaStreamBeginCaptureToGraph(h->st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    h->eng->capturing = true;
    try {
      h->eng->record(trans);
      krylov_iteration(h, A, hc);
    } catch (...) {
      h->eng->capturing = false;
      cudaGraph_t tmp;
      cudaStreamEndCapture(h->st, &tmp);
      throw;
    }
    h->eng->capturing = false;
    MLDG_CUDA(cudaStreamEndCapture(h->st, &gout));
    const int64_t lbody = h->eng->launches + (h->last_launches - l1);
    MLDG_CUDA(cudaGraphInstantiate(&h->sgraph[method][t], g, 0));
    h->sglaunch_pre[method][t] = lpre;
    h->sglaunch_body[method][t] = lbody;
  } catch (...) {
    h->last_launches = l0;
    cudaGraphDestroy(g);
    throw;
  }
  cudaGraphDestroy(g);
  h->last_launches = l0;
}

// Whole solves run as one captured graph unless the handle's V-cycle is not
// graph-captured (K-cycle, use_graphs = 0), a probe brackets a V-cycle launch
// (event nodes cannot sit in a conditional body), or the caller passed its
// own matrix; those run the same kernels with one host check per iteration.
static bool solve_graphable(const Handle *h, bool own_matrix) {
  // MLDG_NO_SOLVE_GRAPH: host-stepped solves (a profiler cannot see the
  // kernels of a graph with conditional nodes; the V-cycle graph stays)
  return own_matrix && h->opts.use_graphs && !kcycle_handle(h) && h->probe_kind == 0 &&
         !std::getenv("MLDG_NO_SOLVE_GRAPH");
}

static void krylov(Handle *h, int method, const mldg_csr *Acsr, const double *b, double *x,
                   double tol, int itmax, int *iters, double *relres, int mem, char trans = 'N') {
  if (!h->finalized) fail(MLDG_ERR_NOT_BUILT, "krylov before build");
  if (method != 0 && method != 1) fail(MLDG_ERR_ARG, "method must be 0 (CG) or 1 (FCG)");
  if (!b || !x) fail(MLDG_ERR_ARG, "null vector");
  check_trans(h, trans);
  if (itmax < 0) fail(MLDG_ERR_ARG, "itmax < 0");
  const int n = h->n0;
  DCSR<double> A = h->A0;
  Arena tmp;
  if (trans != 'N') {
    // A^T of the finest level, built on first use
    if (!h->A0T.present()) h->A0T = to_dev<double>(h->arena, transpose(h->host[0].A));
    A = h->A0T;
  }
  if (Acsr) {
    HostCSR ha = copy_csr(*Acsr, h->opts.index_base, "krylov A", 0);
    if (ha.nr != n || ha.nc != n) fail(MLDG_ERR_SIZE, "krylov A must be %d x %d", n, n);
    A = to_dev<double>(tmp, ha);
  }
  const cudaMemcpyKind h2d = mem == MLDG_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind d2h = mem == MLDG_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  const bool graphed = solve_graphable(h, Acsr == nullptr);
  const int t = trans == 'N' ? 0 : 1;
  if (graphed) capture_solve(h, method, trans, A);  // first use: capture (not timed)
  h->last_launches = 0;
  h->hkpar->tol = tol;
  h->hkpar->itmax = itmax;
  h->hkpar->method = method;
  MLDG_CUDA(cudaEventRecord(h->ev0, h->st));
  MLDG_CUDA(cudaMemcpyAsync(h->kb, b, sizeof(double) * n, h2d, h->st));
  MLDG_CUDA(cudaMemcpyAsync(h->kx, x, sizeof(double) * n, h2d, h->st));
  MLDG_CUDA(cudaMemcpyAsync(h->kpar, h->hkpar, sizeof(KParams), cudaMemcpyHostToDevice, h->st));
  KState *hs = h->hkst;
  if (graphed) {
    MLDG_CUDA(cudaGraphLaunch(h->sgraph[method][t], h->st));
    MLDG_CUDA(cudaMemcpyAsync(hs, h->kst, sizeof(KState), cudaMemcpyDeviceToHost, h->st));
  } else {
    krylov_prefix(h, A, 0);
    MLDG_CUDA(cudaMemcpyAsync(hs, h->kst, sizeof(KState), cudaMemcpyDeviceToHost, h->st));
    MLDG_CUDA(cudaStreamSynchronize(h->st));
    while (!hs->done) {
      run_vcycle(h, trans);  // z = M^{-1} r (or M^{-T} r)
      krylov_iteration(h, A, 0);
      MLDG_CUDA(cudaMemcpyAsync(hs, h->kst, sizeof(KState), cudaMemcpyDeviceToHost, h->st));
      MLDG_CUDA(cudaStreamSynchronize(h->st));
      probe_collect(h);
    }
  }
  MLDG_CUDA(cudaMemcpyAsync(x, h->kx, sizeof(double) * n, d2h, h->st));
  MLDG_CUDA(cudaEventRecord(h->ev1, h->st));
  MLDG_CUDA(cudaStreamSynchronize(h->st));
  if (graphed)
    h->last_launches = h->sglaunch_pre[method][t] + (int64_t)hs->it * h->sglaunch_body[method][t];
  float ms = 0;
  MLDG_CUDA(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
  h->last_ms = ms;
  tmp.release();
  if (iters) *iters = hs->it;
  if (relres) *relres = hs->err;
  check_device_error(h);
}


// ---------------------------------------------------------------------------
// nrhs independent CG/FCG solves sharing the preconditioner, advanced
// together: one K-wide V-cycle, one SpMM and per-column scalars per
// iteration.  A converged column is frozen (its x and r stop changing), so
// each column follows the single-vector krylov() iteration for its own system.
template <int KK>
static void dots_m_t(Handle *h, int nq, const double *x0, const double *y0, const double *x1, const double *y1) {
  k_dots_m<KK><<<kRedBlocksM, 256, 0, h->st>>>(h->n0, nq, x0, y0, x1, y1, h->kpart_m);
  k_dots_m_final<KK><<<1, 2 * KK, 0, h->st>>>(kRedBlocksM, h->kpart_m, h->ksc_m->dots);
  h->last_launches += 2;
}
static void dots_m(Handle *h, int K, int nq, const double *x0, const double *y0, const double *x1,
                   const double *y1) {
  kdispatch(K, [&](auto kc) { dots_m_t<decltype(kc)::value>(h, nq, x0, y0, x1, y1); });
}
static void scal_m(Handle *h, int K, int what) {
  kdispatch(K, [&](auto kc) { k_scal_store_m<decltype(kc)::value><<<1, 32, 0, h->st>>>(h->ksc_m, what); });
  h->last_launches++;
}
static void spmm64(Handle *h, int K, const DCSR<double> &A, const double *v, double a1, const double *b, double a0,
                   double *out) {
  const int64_t thr = (int64_t)A.nr * K / 2;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((thr + 255) / 256, (int64_t)h->nsm * 16));
  kdispatch(K, [&](auto kc) {
    k_spmm<double, decltype(kc)::value, 1><<<g, 256, 0, h->st>>>(A.nr, A.irp, A.ja, A.val, v, a1, b, a0, out, 0.0);
  });
  h->last_launches++;
}
static void ensure_krylov_m(Handle *h, int K) {
  if (!h->hksc_m) MLDG_CUDA(cudaMallocHost(&h->hksc_m, sizeof(KrylovM)));
  if (K <= h->kcap) return;
  h->karena.release();
  h->kcap = 0;  // until every vector is there
  const size_t nk = (size_t)std::max(h->n0, 1) * K;
  h->kb_m = h->karena.alloc<double>(nk);
  h->kx_m = h->karena.alloc<double>(nk);
  h->kd_m = h->karena.alloc<double>(nk);
  h->kq_m = h->karena.alloc<double>(nk);
  h->kpart_m = h->karena.alloc<double>((size_t)2 * 32 * kRedBlocksM);
  h->ksc_m = h->karena.alloc<KrylovM>(1);
  h->kcap = K;
}

static void krylov_multi(Handle *h, int method, const mldg_csr *Acsr, int nrhs, const double *b, int ldb,
                         double *x, int ldx, double tol, int itmax, int *iters, double *relres, int mem) {
  if (!h->finalized) fail(MLDG_ERR_NOT_BUILT, "krylov before build");
  if (method != 0 && method != 1) fail(MLDG_ERR_ARG, "method must be 0 (CG) or 1 (FCG)");
  if (nrhs < 0) fail(MLDG_ERR_ARG, "nrhs < 0");
  if (nrhs > 0 && (!b || !x || !iters || !relres)) fail(MLDG_ERR_ARG, "null argument");
  if (itmax < 0) fail(MLDG_ERR_ARG, "itmax < 0");
  if (mem != MLDG_MEM_HOST && mem != MLDG_MEM_DEVICE) fail(MLDG_ERR_ARG, "bad mem_kind");
  const int n = h->n0;
  if (ldb < n || ldx < n) fail(MLDG_ERR_SIZE, "ldb %d / ldx %d < n %d", ldb, ldx, n);
  if (kcycle_handle(h)) fail(MLDG_ERR_ARG, "the K-cycle is applied column by column: use mldg_krylov per column");
  DCSR<double> A = h->A0;
  Arena tmp;
  if (Acsr) {
    HostCSR ha = copy_csr(*Acsr, h->opts.index_base, "krylov A", 0);
    if (ha.nr != n || ha.nc != n) fail(MLDG_ERR_SIZE, "krylov A must be %d x %d", n, n);
    A = to_dev<double>(tmp, ha);
  }
  h->last_launches = 0;
  MLDG_CUDA(cudaEventRecord(h->ev0, h->st));
  for (int c0 = 0; c0 < nrhs; c0 += 32) {
    const int k = std::min(32, nrhs - c0), K = width_for(k);
    prepare_multi(h, K, 'N');
    ensure_krylov_m(h, K);
    Engine &e = *h->eng;
    double *r = e.xin_m, *z = e.yout_m, *d = h->kd_m, *q = h->kq_m, *xx = h->kx_m, *bb = h->kb_m;
    KrylovM *hs = h->hksc_m;
    load_block(h, b + (size_t)c0 * ldb, ldb, k, K, mem, bb);
    load_block(h, x + (size_t)c0 * ldx, ldx, k, K, mem, xx);
    spmm64(h, K, A, xx, -1.0, bb, 1.0, r);  // r = b - A x
    std::memset(hs, 0, sizeof(KrylovM));
    hs->tol = tol;
    hs->ncols = k;
    MLDG_CUDA(cudaMemcpyAsync(h->ksc_m, hs, sizeof(KrylovM), cudaMemcpyHostToDevice, h->st));
    dots_m(h, K, 2, bb, bb, r, r);
    scal_m(h, K, 3);
    MLDG_CUDA(cudaMemcpyAsync(hs, h->ksc_m, sizeof(KrylovM), cudaMemcpyDeviceToHost, h->st));
    MLDG_CUDA(cudaStreamSynchronize(h->st));
    int it = 0;
    std::vector<int> done(k, 0);
    for (int c = 0; c < k; ++c)
      if (!hs->active[c]) {
        done[c] = 1;
        iters[c0 + c] = 0;
      }
    auto any_active = [&]() {
      for (int c = 0; c < k; ++c)
        if (hs->active[c]) return true;
      return false;
    };
    while (any_active() && it < itmax) {
      ++it;
      run_vcycle_multi(h, 'N', K);  // z = M^{-1} r, all columns
      if (method == 1) {
        if (it > 1) {
          dots_m(h, K, 1, z, q, nullptr, nullptr);
          scal_m(h, K, 0);
        }
      } else {
        dots_m(h, K, 1, r, z, nullptr, nullptr);
        scal_m(h, K, 0);
      }
      const int64_t tot = (int64_t)n * K;
      const int g = (int)std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, (int64_t)h->nsm * 16));
      kdispatch(K, [&](auto kc) {
        constexpr int KK = decltype(kc)::value;
        k_dir_update_m<KK><<<g, 256, 0, h->st>>>(n, method, it == 1 ? 1 : 0, z, d, h->ksc_m);
      });
      spmm64(h, K, A, d, 1.0, nullptr, 0.0, q);  // q = A d
      dots_m(h, K, 2, d, q, d, r);
      scal_m(h, K, 1);
      kdispatch(K, [&](auto kc) {
        constexpr int KK = decltype(kc)::value;
        k_xr_update_m<KK><<<g, 256, 0, h->st>>>(n, method, d, q, xx, r, h->ksc_m);
      });
      dots_m(h, K, 1, r, r, nullptr, nullptr);
      scal_m(h, K, 2);
      h->last_launches += 2;
      MLDG_CUDA(cudaMemcpyAsync(hs, h->ksc_m, sizeof(KrylovM), cudaMemcpyDeviceToHost, h->st));
      MLDG_CUDA(cudaStreamSynchronize(h->st));
      probe_collect(h);
      for (int c = 0; c < k; ++c)
        if (!done[c] && !hs->active[c]) {
          done[c] = 1;
          iters[c0 + c] = it;
        }
    }
    for (int c = 0; c < k; ++c) {
      if (!done[c]) iters[c0 + c] = it;
      relres[c0 + c] = std::sqrt(std::max(hs->rr[c], 0.0)) / hs->bn[c];
      if (std::isnan(hs->rr[c])) relres[c0 + c] = hs->rr[c];
    }
    store_block(h, xx, k, K, mem, x + (size_t)c0 * ldx, ldx);
  }
  MLDG_CUDA(cudaEventRecord(h->ev1, h->st));
  MLDG_CUDA(cudaStreamSynchronize(h->st));
  float ms = 0;
  MLDG_CUDA(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
  h->last_ms = ms;
  tmp.release();
  check_device_error(h);
}

// ---------------------------------------------------------------------------
// Independent systems solved together in ONE graph launch: the prefixes of
// all systems (initial residual and state) as parallel branches, then a
// WHILE node whose body opens, per iteration, an IF branch for every
// unfinished system -- its V-cycle and its CG/FCG iteration
// (krylov_iteration) -- and closes with k_kry_any, which keeps the loop
// going while any system is unfinished.  The branches of one iteration run
// concurrently; nothing returns to the host until every system has
// finished.  Each system runs exactly the kernels mldg_krylov runs for it,
// so the results are the same bits.
struct BatchGraph {
  std::vector<uint64_t> key;  // method, then the handles' serials
  cudaGraphExec_t exec = nullptr;
  KState **dstates = nullptr;  // device array of the systems' states
  cudaGraphConditionalHandle *dhc = nullptr;
  int64_t launches_pre = 0, launches_loop = 0;  // per launch of the prefix / per loop iteration
  std::vector<int64_t> launches_branch;         // per system, one branch
  void release() {
    if (exec) cudaGraphExecDestroy(exec);
    if (dstates) cudaFree(dstates);
    if (dhc) cudaFree(dhc);
    exec = nullptr;
    dstates = nullptr;
    dhc = nullptr;
  }
};
static std::mutex g_batch_mu;
static std::vector<std::unique_ptr<BatchGraph>> g_batch_cache;  // most recent last, at most 4

// drops the cached batch graphs that include a handle (at its finalize or destroy)
static void batch_evict(uint64_t serial) {
  if (serial == 0) return;
  std::lock_guard<std::mutex> lk(g_batch_mu);
  for (size_t k = 0; k < g_batch_cache.size();) {
    const auto &key = g_batch_cache[k]->key;
    if (std::find(key.begin() + 1, key.end(), serial) != key.end()) {
      g_batch_cache[k]->release();
      g_batch_cache.erase(g_batch_cache.begin() + k);
    } else {
      ++k;
    }
  }
}

static cudaGraphNode_t only_sink(cudaGraph_t g) {
  size_t nn = 0;
  MLDG_CUDA(cudaGraphGetNodes(g, nullptr, &nn));
  std::vector<cudaGraphNode_t> nodes(nn);
  MLDG_CUDA(cudaGraphGetNodes(g, nodes.data(), &nn));
  cudaGraphNode_t sink = nullptr;
  for (cudaGraphNode_t nd : nodes) {
    size_t no = 0;
    MLDG_CUDA(cudaGraphNodeGetDependentNodes(nd, nullptr, &no));
    if (no == 0) {
      if (sink) fail(MLDG_ERR_INTERNAL, "batch graph: more than one sink");
      sink = nd;
    }
  }
  if (!sink) fail(MLDG_ERR_INTERNAL, "batch graph: no sink");
  return sink;
}

static void end_capture_quietly(cudaStream_t st) {
  cudaGraph_t tmp = nullptr;
  cudaStreamEndCapture(st, &tmp);
  if (tmp) cudaGraphDestroy(tmp);
}

// Programmatic dependent launch off for the captures of a batch: the early
// scheduled blocks of one system's next kernel would sit on SMs, waiting,
// that the concurrent branches of the other systems need (64 systems at idim
// 24..96: 185 ms with it, against 155 ms without).
// The systems' grouped solves share the SMs by their rows: a solve alone keeps
// two or three blocks an SM waiting, which 64 systems have no room for.
struct NoPdlScope {
  std::vector<std::pair<Engine *, bool>> saved;
  NoPdlScope(int nsys, Handle **hs) {
    double rows = 0;
    for (int i = 0; i < nsys; ++i) rows += hs[i]->n0;
    for (int i = 0; i < nsys; ++i) {
      saved.emplace_back(hs[i]->eng.get(), hs[i]->eng->pdl);
      hs[i]->eng->pdl = false;
      hs[i]->eng->grp_blocks = std::max(kGrpBatchLeast, (int)(hs[i]->eng->grp_room * (hs[i]->n0 / std::max(rows, 1.0))));
    }
  }
  ~NoPdlScope() {
    for (auto &e : saved) {
      e.first->pdl = e.second;
      e.first->grp_blocks = 0;
    }
  }
};

static std::unique_ptr<BatchGraph> capture_batch(int nsys, Handle **hs, int method, cudaStream_t ms) {
  NoPdlScope nopdl(nsys, hs);
  auto bg = std::make_unique<BatchGraph>();
  bg->key.push_back((uint64_t)method);
  for (int i = 0; i < nsys; ++i) bg->key.push_back(hs[i]->serial);
  cudaGraph_t top = nullptr;
  std::vector<cudaEvent_t> evs;
  MLDG_CUDA(cudaGraphCreate(&top, 0));
  try {
    std::vector<KState *> states(nsys);
    for (int i = 0; i < nsys; ++i) states[i] = hs[i]->kst;
    MLDG_CUDA(cudaMalloc(&bg->dstates, sizeof(KState *) * nsys));
    MLDG_CUDA(cudaMemcpy(bg->dstates, states.data(), sizeof(KState *) * nsys, cudaMemcpyHostToDevice));
    cudaGraphConditionalHandle hw;
    MLDG_CUDA(cudaGraphConditionalHandleCreate(&hw, top, 0, cudaGraphCondAssignDefault));
    for (int i = 0; i <= nsys; ++i) {
      cudaEvent_t e;
      MLDG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      evs.push_back(e);
    }
    // prefixes: forked from the master stream, joined before k_kry_any
    MLDG_CUDA(cudaStreamBeginCaptureToGraph(ms, top, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    try {
      MLDG_CUDA(cudaEventRecord(evs[nsys], ms));
      for (int i = 0; i < nsys; ++i) {
        Handle *h = hs[i];
        MLDG_CUDA(cudaStreamWaitEvent(h->st, evs[nsys], 0));
        const int64_t l0 = h->last_launches;
        {
          KioScope kio(h, kry_io_ok(h));
          krylov_prefix(h, h->A0, 0);
        }
        bg->launches_pre += h->last_launches - l0;
        h->last_launches = l0;
        MLDG_CUDA(cudaEventRecord(evs[i], h->st));
        MLDG_CUDA(cudaStreamWaitEvent(ms, evs[i], 0));
      }
      k_kry_any<<<1, 256, 0, ms>>>(bg->dstates, nsys, hw);
    } catch (...) {
      end_capture_quietly(ms);
      throw;
    }
    cudaGraph_t gout = nullptr;
    MLDG_CUDA(cudaStreamEndCapture(ms, &gout));
    bg->launches_pre += 1;
    cudaGraphNode_t sink = only_sink(top);
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = hw;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t wn;
    MLDG_CUDA(cudaGraphAddNode(&wn, top, &sink, 1, &wp));
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    // the IF handles of the branches live in the loop body
    std::vector<cudaGraphConditionalHandle> hc(nsys);
    for (int i = 0; i < nsys; ++i) MLDG_CUDA(cudaGraphConditionalHandleCreate(&hc[i], body, 0, 0));
    MLDG_CUDA(cudaMalloc(&bg->dhc, sizeof(cudaGraphConditionalHandle) * nsys));
    MLDG_CUDA(cudaMemcpy(bg->dhc, hc.data(), sizeof(cudaGraphConditionalHandle) * nsys, cudaMemcpyHostToDevice));
    MLDG_CUDA(cudaStreamBeginCaptureToGraph(ms, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    k_kry_gate<<<1, 256, 0, ms>>>(bg->dstates, bg->dhc, nsys);
    MLDG_CUDA(cudaStreamEndCapture(ms, &gout));
    cudaGraphNode_t gate = only_sink(body);
    std::vector<cudaGraphNode_t> ifs(nsys);
    bg->launches_branch.assign(nsys, 0);
    for (int i = 0; i < nsys; ++i) {
      Handle *h = hs[i];
      cudaGraphNodeParams ip = {};
      ip.type = cudaGraphNodeTypeConditional;
      ip.conditional.handle = hc[i];
      ip.conditional.type = cudaGraphCondTypeIf;
      ip.conditional.size = 1;
      MLDG_CUDA(cudaGraphAddNode(&ifs[i], body, &gate, 1, &ip));
      cudaGraph_t br = ip.conditional.phGraph_out[0];
      const int64_t l0 = h->last_launches;
      MLDG_CUDA(cudaStreamBeginCaptureToGraph(h->st, br, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
      KioScope kio(h, kry_io_ok(h));
      h->eng->capturing = true;
      try {
        h->eng->record('N');
        krylov_iteration(h, h->A0, 0);
      } catch (...) {
        h->eng->capturing = false;
        end_capture_quietly(h->st);
        throw;
      }
      h->eng->capturing = false;
      MLDG_CUDA(cudaStreamEndCapture(h->st, &gout));
      bg->launches_branch[i] = h->eng->launches + (h->last_launches - l0);
      h->last_launches = l0;
    }
    MLDG_CUDA(cudaStreamBeginCaptureToGraph(ms, body, ifs.data(), nullptr, nsys, cudaStreamCaptureModeThreadLocal));
    k_kry_any<<<1, 256, 0, ms>>>(bg->dstates, nsys, hw);
    MLDG_CUDA(cudaStreamEndCapture(ms, &gout));
    bg->launches_loop = 2;  // gate and any
    MLDG_CUDA(cudaGraphInstantiate(&bg->exec, top, 0));
  } catch (...) {
    for (cudaEvent_t e : evs) cudaEventDestroy(e);
    cudaGraphDestroy(top);
    bg->release();
    throw;
  }
  for (cudaEvent_t e : evs) cudaEventDestroy(e);
  cudaGraphDestroy(top);
  return bg;
}

static void krylov_batch(int nsys, Handle **hs, int method, const double *const *b, double *const *x, double tol,
                         int itmax, int *iters, double *relres, int mem, double *ms_out) {
  if (nsys < 0) fail(MLDG_ERR_ARG, "nsys < 0");
  if (nsys == 0) return;
  if (!hs || !b || !x || !iters || !relres) fail(MLDG_ERR_ARG, "null argument");
  if (method != 0 && method != 1) fail(MLDG_ERR_ARG, "method must be 0 (CG) or 1 (FCG)");
  if (itmax < 0) fail(MLDG_ERR_ARG, "itmax < 0");
  if (mem != MLDG_MEM_HOST && mem != MLDG_MEM_DEVICE) fail(MLDG_ERR_ARG, "bad mem_kind");
  const int dev = hs[0]->opts.device;
  for (int i = 0; i < nsys; ++i) {
    if (!hs[i]) fail(MLDG_ERR_ARG, "system %d: null handle", i);
    if (!hs[i]->finalized) fail(MLDG_ERR_NOT_BUILT, "system %d: krylov before build", i);
    if (hs[i]->opts.device != dev) fail(MLDG_ERR_ARG, "system %d: handles on different devices", i);
    if (!solve_graphable(hs[i], true))
      fail(MLDG_ERR_ARG, "system %d: its solve cannot be one graph (K-cycle, use_graphs = 0 or a probe set); "
                         "use mldg_krylov", i);
    if (!b[i] || !x[i]) fail(MLDG_ERR_ARG, "system %d: null vector", i);
    for (int k = 0; k < i; ++k)
      if (hs[k] == hs[i]) fail(MLDG_ERR_ARG, "system %d: handle repeated", i);
  }
  MLDG_CUDA(cudaSetDevice(dev));
  const cudaMemcpyKind h2d = mem == MLDG_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind d2h = mem == MLDG_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  std::lock_guard<std::mutex> lk(g_batch_mu);
  cudaStream_t ms = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  MLDG_CUDA(cudaStreamCreateWithFlags(&ms, cudaStreamNonBlocking));
  MLDG_CUDA(cudaEventCreate(&e0));
  MLDG_CUDA(cudaEventCreate(&e1));
  try {
    // the batch graph of exactly these finalized handles (captured on first use, not timed)
    std::vector<uint64_t> key{(uint64_t)method};
    for (int i = 0; i < nsys; ++i) key.push_back(hs[i]->serial);
    BatchGraph *bg = nullptr;
    for (auto &c : g_batch_cache)
      if (c->key == key) bg = c.get();
    if (!bg) {
      for (int i = 0; i < nsys; ++i) MLDG_CUDA(cudaStreamSynchronize(hs[i]->st));
      g_batch_cache.push_back(capture_batch(nsys, hs, method, ms));
      bg = g_batch_cache.back().get();
      if (g_batch_cache.size() > 4) {
        g_batch_cache.front()->release();
        g_batch_cache.erase(g_batch_cache.begin());
      }
    }
    MLDG_CUDA(cudaEventRecord(e0, ms));
    for (int i = 0; i < nsys; ++i) {
      Handle *h = hs[i];
      const int n = h->n0;
      h->hkpar->tol = tol;
      h->hkpar->itmax = itmax;
      h->hkpar->method = method;
      MLDG_CUDA(cudaMemcpyAsync(h->kb, b[i], sizeof(double) * n, h2d, ms));
      MLDG_CUDA(cudaMemcpyAsync(h->kx, x[i], sizeof(double) * n, h2d, ms));
      MLDG_CUDA(cudaMemcpyAsync(h->kpar, h->hkpar, sizeof(KParams), cudaMemcpyHostToDevice, ms));
    }
    MLDG_CUDA(cudaGraphLaunch(bg->exec, ms));
    for (int i = 0; i < nsys; ++i) {
      Handle *h = hs[i];
      MLDG_CUDA(cudaMemcpyAsync(h->hkst, h->kst, sizeof(KState), cudaMemcpyDeviceToHost, ms));
      MLDG_CUDA(cudaMemcpyAsync(x[i], h->kx, sizeof(double) * h->n0, d2h, ms));
    }
    MLDG_CUDA(cudaEventRecord(e1, ms));
    MLDG_CUDA(cudaStreamSynchronize(ms));
    float t = 0;
    MLDG_CUDA(cudaEventElapsedTime(&t, e0, e1));
    if (ms_out) *ms_out = t;
    int itmax_seen = 0;
    for (int i = 0; i < nsys; ++i) itmax_seen = std::max(itmax_seen, hs[i]->hkst->it);
    for (int i = 0; i < nsys; ++i) {
      Handle *h = hs[i];
      iters[i] = h->hkst->it;
      relres[i] = h->hkst->err;
      h->last_ms = t;
      // this system's own kernels; the batch's gate/any kernels are counted on the first system
      h->last_launches = (int64_t)h->hkst->it * bg->launches_branch[i] +
                         (i == 0 ? bg->launches_pre + (int64_t)itmax_seen * bg->launches_loop : 3);
      check_device_error(h);
    }
  } catch (...) {
    cudaStreamSynchronize(ms);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamDestroy(ms);
    throw;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(ms);
}
}  // namespace mldg

// ===========================================================================
// C ABI
using mldg::Error;
using mldg::Handle;

struct mldg_handle {
  Handle h;
};

#define MLDG_GUARD(hp, body)                                     \
  do {                                                           \
    try {                                                        \
      body;                                                      \
      return MLDG_SUCCESS;                                       \
    } catch (const Error &e_) {                                  \
      if (hp) (hp)->h.last_error = e_.msg;                       \
      return e_.code;                                            \
    } catch (const std::exception &e_) {                         \
      if (hp) (hp)->h.last_error = e_.what();                    \
      return MLDG_ERR_INTERNAL;                                  \
    }                                                            \
  } while (0)

extern "C" int mldg_create(mldg_handle **out, const mldg_opts *opts) {
  if (!out) return MLDG_ERR_ARG;
  *out = nullptr;
  mldg_handle *hp = new mldg_handle();
  Handle &h = hp->h;
  h.opts.device = 0;
  h.opts.index_base = 0;
  h.opts.use_graphs = 1;
  h.opts.autotune = 1;
  if (opts) h.opts = *opts;
  if (h.opts.index_base != 0 && h.opts.index_base != 1) {
    delete hp;
    return MLDG_ERR_ARG;
  }
  try {
    MLDG_CUDA(cudaSetDevice(h.opts.device));
    MLDG_CUDA(cudaStreamCreateWithFlags(&h.st, cudaStreamNonBlocking));
    MLDG_CUDA(cudaEventCreate(&h.ev0));
    MLDG_CUDA(cudaEventCreate(&h.ev1));
    MLDG_CUDA(cudaEventCreate(&h.pev0));
    MLDG_CUDA(cudaEventCreate(&h.pev1));
    MLDG_CUDA(cudaMallocHost(&h.hpin, 4 * sizeof(double)));
    MLDG_CUDA(cudaDeviceGetAttribute(&h.nsm, cudaDevAttrMultiProcessorCount, h.opts.device));
  } catch (const Error &e) {
    delete hp;
    return e.code;
  }
  *out = hp;
  return MLDG_SUCCESS;
}

extern "C" int mldg_upload_level(mldg_handle *hp, int lev, const mldg_level_desc *d) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, {
    Handle &h = hp->h;
    if (!d) mldg::fail(MLDG_ERR_ARG, "null level descriptor");
    if (lev < 0 || lev > 64) mldg::fail(MLDG_ERR_ARG, "level %d out of range", lev);
    if ((int)h.host.size() <= lev) h.host.resize(lev + 1);
    mldg::HostLevel H;
    const int b = h.opts.index_base;
    H.A = mldg::copy_csr(d->A, b, "A", lev);
    H.P = mldg::copy_csr(d->P, b, "P", lev);
    H.R = mldg::copy_csr(d->R, b, "R", lev);
    H.ND = mldg::copy_csr(d->ND, b, "ND", lev);
    H.L = mldg::copy_csr(d->L, b, "L", lev);
    H.U = mldg::copy_csr(d->U, b, "U", lev);
    if (d->d && H.A.present()) H.d.assign(d->d, d->d + H.A.nr);
    H.kind = d->smoother_kind;
    H.sweeps_pre = d->sweeps_pre;
    H.sweeps_post = d->sweeps_post;
    H.damp = d->damping == 0.0 ? 1.0 : d->damping;
    H.uploaded = true;
    h.host[lev] = std::move(H);
    h.finalized = false;
  });
}

extern "C" int mldg_finalize(mldg_handle *hp, int nlev, int precision) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, {
    MLDG_CUDA(cudaSetDevice(hp->h.opts.device));
    mldg::finalize(&hp->h, nlev, precision);
  });
}

extern "C" int mldg_set_cycle(mldg_handle *hp, int cycle) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, {
    Handle &h = hp->h;
    if (cycle < MLDG_CYCLE_V || cycle > MLDG_CYCLE_ADD) mldg::fail(MLDG_ERR_ARG, "unknown cycle %d", cycle);
    if (h.cycle != cycle) {
      h.cycle = cycle;
      for (int t = 0; t < 2; ++t)
        if (h.gexec[t]) {
          cudaGraphExecDestroy(h.gexec[t]);
          h.gexec[t] = nullptr;
        }
      mldg::drop_multi_graphs(&h);
      mldg::drop_krylov_graphs(&h);
      if (h.eng) h.eng->cycle = cycle;
    }
  });
}

extern "C" int mldg_apply(mldg_handle *hp, const double *x, double *y, char trans, int nrhs,
                          int ld, int mem_kind) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, { mldg::apply(&hp->h, x, y, trans, nrhs, ld, mem_kind); });
}

extern "C" int mldg_krylov(mldg_handle *hp, int method, const mldg_csr *A, const double *b,
                           double *x, double tol, int itmax, int *iters, double *relres,
                           int mem_kind) {
  if (!hp) return MLDG_ERR_ARG;
  int it = 0;
  MLDG_GUARD(hp, {
    mldg::krylov(&hp->h, method, A, b, x, tol, itmax, &it, relres, mem_kind);
    if (iters) *iters = it;
    if (it >= itmax && relres && *relres > tol)
      mldg::fail(MLDG_ERR_NOT_CONVERGED, "not converged in %d iterations (relres %.3e)", it, *relres);
  });
}

extern "C" int mldg_krylov_multi(mldg_handle *hp, int method, const mldg_csr *A, int nrhs, const double *b,
                                 int ldb, double *x, int ldx, double tol, int itmax, int *iters, double *relres,
                                 int mem_kind) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, {
    mldg::krylov_multi(&hp->h, method, A, nrhs, b, ldb, x, ldx, tol, itmax, iters, relres, mem_kind);
    for (int c = 0; c < nrhs; ++c)
      if (iters[c] >= itmax && !(relres[c] <= tol))
        mldg::fail(MLDG_ERR_NOT_CONVERGED, "column %d not converged in %d iterations (relres %.3e)", c, iters[c],
                   relres[c]);
  });
}

extern "C" int mldg_krylov_batch(int nsys, mldg_handle *const *hps, int method, const double *const *b,
                                 double *const *x, double tol, int itmax, int *iters, double *relres, int mem_kind,
                                 double *ms) {
  if (nsys > 0 && !hps) return MLDG_ERR_ARG;
  for (int i = 0; i < nsys; ++i)
    if (!hps[i]) return MLDG_ERR_ARG;
  mldg_handle *hp = nsys > 0 ? hps[0] : nullptr;
  std::vector<Handle *> hs((size_t)std::max(nsys, 0));
  for (int i = 0; i < nsys; ++i) hs[i] = &hps[i]->h;
  MLDG_GUARD(hp, {
    try {
      mldg::krylov_batch(nsys, hs.data(), method, b, x, tol, itmax, iters, relres, mem_kind, ms);
    } catch (const Error &e) {
      for (int i = 1; i < nsys; ++i) hps[i]->h.last_error = e.msg;
      throw;
    }
    for (int i = 0; i < nsys; ++i)
      if (iters[i] >= itmax && !(relres[i] <= tol))
        mldg::fail(MLDG_ERR_NOT_CONVERGED, "system %d not converged in %d iterations (relres %.3e)", i, iters[i],
                   relres[i]);
  });
}

extern "C" int mldg_adjoint(mldg_handle *hp, const double *g, double *lambda, double tol, int itmax,
                            int *iters, double *relres, int mem_kind) {
  if (!hp) return MLDG_ERR_ARG;
  int it = 0;
  MLDG_GUARD(hp, {
    mldg::krylov(&hp->h, 1, nullptr, g, lambda, tol, itmax, &it, relres, mem_kind, 'T');
    if (iters) *iters = it;
    if (it >= itmax && relres && *relres > tol)
      mldg::fail(MLDG_ERR_NOT_CONVERGED, "adjoint not converged in %d iterations (relres %.3e)", it, *relres);
  });
}

static void kappa_grad(Handle &h, int idim, const double *kappa, const double *x, const double *lam,
                       double *grad, int mem) {
  if (idim <= 0 || !kappa || !x || !lam || !grad) mldg::fail(MLDG_ERR_ARG, "bad kappa_grad arguments");
  MLDG_CUDA(cudaSetDevice(h.opts.device));
  const long long n = (long long)idim * idim * idim;
  const double hh = 1.0 / (double)(idim + 1);
  const int blocks = (int)std::min<long long>((n + 255) / 256, (long long)h.nsm * 16);
  if (mem == MLDG_MEM_DEVICE) {
    mldg::k_kappa_grad<<<blocks, 256, 0, h.st>>>(idim, 1.0 / (hh * hh), kappa, x, lam, grad);
    MLDG_CUDA(cudaStreamSynchronize(h.st));
    MLDG_CUDA(cudaGetLastError());
    return;
  }
  if (mem != MLDG_MEM_HOST) mldg::fail(MLDG_ERR_ARG, "bad mem_kind");
  mldg::Arena tmp;  // host buffers: staged through device copies
  double *dk = tmp.alloc<double>((size_t)n), *dx = tmp.alloc<double>((size_t)n);
  double *dl = tmp.alloc<double>((size_t)n), *dg = tmp.alloc<double>((size_t)n);
  MLDG_CUDA(cudaMemcpyAsync(dk, kappa, sizeof(double) * n, cudaMemcpyHostToDevice, h.st));
  MLDG_CUDA(cudaMemcpyAsync(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice, h.st));
  MLDG_CUDA(cudaMemcpyAsync(dl, lam, sizeof(double) * n, cudaMemcpyHostToDevice, h.st));
  mldg::k_kappa_grad<<<blocks, 256, 0, h.st>>>(idim, 1.0 / (hh * hh), dk, dx, dl, dg);
  MLDG_CUDA(cudaMemcpyAsync(grad, dg, sizeof(double) * n, cudaMemcpyDeviceToHost, h.st));
  MLDG_CUDA(cudaStreamSynchronize(h.st));
  tmp.release();
}

extern "C" int mldg_kappa_grad(mldg_handle *hp, int idim, const double *kappa, const double *x,
                               const double *lambda, double *grad, int mem_kind) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, { kappa_grad(hp->h, idim, kappa, x, lambda, grad, mem_kind); });
}

extern "C" int mldg_level_info(const mldg_handle *hp, int lev, int64_t *info) {
  if (!hp || !info) return MLDG_ERR_ARG;
  const Handle &h = hp->h;
  if (!h.finalized) return MLDG_ERR_NOT_BUILT;
  if (lev < 0 || lev >= h.nlev) return MLDG_ERR_ARG;
  const mldg::HostLevel &H = h.host[lev];
  info[0] = H.A.nr;
  info[1] = H.A.nnz();
  info[2] = H.P.nnz();
  info[3] = H.L.nnz() + H.U.nnz() + H.ND.nnz();
  info[4] = h.nlev;
  return MLDG_SUCCESS;
}

extern "C" int mldg_last_timing(const mldg_handle *hp, double *ms, int64_t *launches) {
  if (!hp) return MLDG_ERR_ARG;
  if (ms) *ms = hp->h.last_ms;
  if (launches) *launches = hp->h.last_launches;
  return MLDG_SUCCESS;
}

extern "C" int mldg_apply_bytes(const mldg_handle *hp, int64_t *bytes) {
  if (!hp || !bytes) return MLDG_ERR_ARG;
  if (!hp->h.finalized) return MLDG_ERR_NOT_BUILT;
  *bytes = hp->h.gbytes[0];
  return MLDG_SUCCESS;
}

extern "C" int mldg_apply_impl_bytes(const mldg_handle *hp, int64_t *bytes) {
  if (!hp || !bytes) return MLDG_ERR_ARG;
  if (!hp->h.finalized) return MLDG_ERR_NOT_BUILT;
  *bytes = hp->h.gimpl[0];
  return MLDG_SUCCESS;
}

extern "C" int mldg_probe_set(mldg_handle *hp, int kind, int lev, int index) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, {
    Handle &h = hp->h;
    if (kind < 0 || kind > MLDG_KERNEL_VEC || lev < 0 || index < 0)
      mldg::fail(MLDG_ERR_ARG, "bad probe (%d, %d, %d)", kind, lev, index);
    h.probe_kind = kind;
    h.probe_lev = lev;
    h.probe_idx = index;
    for (int t = 0; t < 2; ++t)
      if (h.gexec[t]) {
        cudaGraphExecDestroy(h.gexec[t]);
        h.gexec[t] = nullptr;
      }
    mldg::drop_multi_graphs(&h);
    mldg::drop_krylov_graphs(&h);
    if (h.eng) {
      h.eng->probe_kind = kind;
      h.eng->probe_lev = lev;
      h.eng->probe_idx = index;
    }
    h.probe_ms = 0;
    h.probe_count = 0;
    h.pending = false;
  });
}

extern "C" int mldg_probe_read(mldg_handle *hp, double *total_ms, int64_t *count, int64_t *bytes) {
  if (!hp) return MLDG_ERR_ARG;
  Handle &h = hp->h;
  if (total_ms) *total_ms = h.probe_ms;
  if (count) *count = h.probe_count;
  if (bytes) *bytes = h.probe_bytes;
  h.probe_ms = 0;
  h.probe_count = 0;
  return MLDG_SUCCESS;
}

static void profile_run(Handle &h, char trans, int nrhs, int max, mldg_kernel_stat *stats, int *n) {
  if (!h.finalized) mldg::fail(MLDG_ERR_NOT_BUILT, "profile before build");
  if (trans == 'C') trans = 'T';
  if (trans != 'N' && trans != 'T') mldg::fail(MLDG_ERR_TRANS, "invalid trans");
  mldg::check_trans(&h, trans);
  if (nrhs < 1 || nrhs > 32) mldg::fail(MLDG_ERR_ARG, "profile width must be 1..32");
  const int K = nrhs > 1 ? mldg::width_for(nrhs) : 1;
  if (K > 1) mldg::prepare_multi(&h, K, trans);
  std::vector<mldg::Engine::Prof> prof;
  h.eng->prof = &prof;
  const int pk = h.eng->probe_kind;
  h.eng->probe_kind = 0;
  try {
    if (K > 1)
      h.eng->record_multi(trans, K);
    else
      h.eng->record(trans);
  } catch (...) {
    h.eng->prof = nullptr;
    h.eng->probe_kind = pk;
    throw;
  }
  h.eng->prof = nullptr;
  h.eng->probe_kind = pk;
  MLDG_CUDA(cudaStreamSynchronize(h.st));
  int k = 0;
  for (auto &e : prof) {
    float ms = 0;
    cudaEventElapsedTime(&ms, e.e0, e.e1);
    if (k < max && stats) {
      stats[k].kind = e.kind;
      stats[k].level = e.lev;
      stats[k].bytes = e.bytes;
      stats[k].ms = ms;
    }
    ++k;
    cudaEventDestroy(e.e0);
    cudaEventDestroy(e.e1);
  }
  if (n) *n = k;
  mldg::check_device_error(&h);
}

extern "C" int mldg_profile_multi(mldg_handle *hp, char trans, int nrhs, int max, mldg_kernel_stat *stats,
                                  int *n) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, { profile_run(hp->h, trans, nrhs, max, stats, n); });
}

extern "C" int mldg_profile(mldg_handle *hp, char trans, int max, mldg_kernel_stat *stats, int *n) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, { profile_run(hp->h, trans, 1, max, stats, n); });
}

// ---------------------------------------------------------------------------
// Allocation-free relative residual (see mldg.h).  The scratch of this entry
// point is a file-scope device array: [0, MAX_N) holds the residual r,
// [MAX_N, MAX_N + 3*kRedBlocks) the per-block partials of the two-pass
// reduction, the next 3 doubles its result.  Nothing there needs to start at
// zero: every call overwrites r, every partial and the result before reading
// them.
static __device__ __align__(256) double g_noalloc_scratch[MLDG_NOALLOC_MAX_N + 1024];
static_assert(3 * mldg::kRedBlocks + 3 <= 1024, "scratch tail too small for the partials");

namespace {
std::mutex g_noalloc_mu;
double *g_noalloc_ptr[128] = {nullptr};  // device address of the array, per device

// once per device, with that device current
double *noalloc_scratch(int device) {
  if (device < 0 || device >= 128) mldg::fail(MLDG_ERR_ARG, "device %d out of range", device);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
      mldg::fail(MLDG_ERR_CUDA, "cudaGetSymbolAddress(scratch): %s", cudaGetErrorString(e));
    g_noalloc_ptr[device] = (double *)p;
  }
  return g_noalloc_ptr[device];
}
}  // namespace

static void relres_noalloc(Handle &h, const mldg_csr *A, const double *x, const double *b,
                           double *relres) {
  {
    if (!A || !x || !b || !relres) mldg::fail(MLDG_ERR_ARG, "null argument");
    const int n = A->nrows;
    if (n < 0 || A->ncols != n) mldg::fail(MLDG_ERR_ARG, "A must be square (%d x %d)", n, A->ncols);
    if (n > MLDG_NOALLOC_MAX_N)
      mldg::fail(MLDG_ERR_SIZE, "n = %d exceeds the allocation-free limit MLDG_NOALLOC_MAX_N = %d", n,
                 MLDG_NOALLOC_MAX_N);
    if (n > 0 && (!A->irp || !A->ja || !A->val)) mldg::fail(MLDG_ERR_ARG, "null CSR array");
    MLDG_CUDA(cudaSetDevice(h.opts.device));
    double *scratch = noalloc_scratch(h.opts.device);
    double *r = scratch;
    double *partial = scratch + MLDG_NOALLOC_MAX_N;
    double *res = partial + 3 * mldg::kRedBlocks;
    if (n == 0) {
      *relres = 1.0;
      return;
    }
    // r = b - A x with the row length of A choosing the lanes per row
    int64_t nnz = 0;
    MLDG_CUDA(cudaMemcpyAsync(&nnz, A->irp + n, sizeof(int32_t), cudaMemcpyDeviceToHost, h.st));
    MLDG_CUDA(cudaStreamSynchronize(h.st));
    nnz = (int64_t)(int32_t)nnz;
    const int tpr = mldg::pick_tpr(nnz, n);
    const int64_t thr = (int64_t)n * tpr;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((thr + 255) / 256, (int64_t)h.nsm * 16));
    switch (tpr) {
#define CASE(K)                                                                                 \
  case K:                                                                                       \
    mldg::k_spmv<double, K><<<g, 256, 0, h.st>>>(n, A->irp, A->ja, A->val, x, -1.0, b, 1.0, r, 0.0); \
    break;
      CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32)
#undef CASE
      default: mldg::fail(MLDG_ERR_INTERNAL, "bad tpr");
    }
    // ||b||^2, ||r||^2: per-block partials, then one block in a fixed order
    mldg::k_dots<<<mldg::kRedBlocks, mldg::kRedThreads, 0, h.st>>>(n, 2, b, b, r, r, nullptr, nullptr,
                                                                     partial);
    mldg::k_dots_final<<<1, mldg::kRedThreads, 0, h.st>>>(mldg::kRedBlocks, partial, res);
    double out[3] = {0, 0, 0};
    MLDG_CUDA(cudaMemcpyAsync(out, res, 3 * sizeof(double), cudaMemcpyDeviceToHost, h.st));
    MLDG_CUDA(cudaStreamSynchronize(h.st));
    MLDG_CUDA(cudaGetLastError());
    const double bn = std::sqrt(out[0]);
    *relres = bn == 0.0 ? 1.0 : std::sqrt(out[1]) / bn;
  }
}

extern "C" int mldg_relres_noalloc(mldg_handle *hp, const mldg_csr *A, const double *x,
                                   const double *b, double *relres) {
  if (!hp) return MLDG_ERR_ARG;
  MLDG_GUARD(hp, { relres_noalloc(hp->h, A, x, b, relres); });
}

extern "C" const char *mldg_last_error(const mldg_handle *hp) {
  if (!hp) return "null handle";
  return hp->h.last_error.c_str();
}

extern "C" void mldg_destroy(mldg_handle *hp) {
  if (!hp) return;
  Handle &h = hp->h;
  cudaSetDevice(h.opts.device);
  if (h.st) cudaStreamSynchronize(h.st);
  if (h.eng && (std::getenv("MLDG_WIN_TRACE") || std::getenv("MLDG_ELL_TRACE") || std::getenv("MLDG_REP_TRACE")))
    h.eng->dump_trace();
  for (int t = 0; t < 2; ++t)
    if (h.gexec[t]) cudaGraphExecDestroy(h.gexec[t]);
  mldg::drop_multi_graphs(&h);
  mldg::drop_krylov_graphs(&h);
  mldg::batch_evict(h.serial);
  h.eng.reset();
  h.arena.release();
  h.karena.release();
  if (h.hpin) cudaFreeHost(h.hpin);
  if (h.hkst) cudaFreeHost(h.hkst);
  if (h.hkpar) cudaFreeHost(h.hkpar);
  if (h.hksc_m) cudaFreeHost(h.hksc_m);
  if (h.ev0) cudaEventDestroy(h.ev0);
  if (h.ev1) cudaEventDestroy(h.ev1);
  if (h.pev0) cudaEventDestroy(h.pev0);
  if (h.pev1) cudaEventDestroy(h.pev1);
  if (h.st) cudaStreamDestroy(h.st);
  delete hp;
}

// Test hook (host only, no GPU): builds the replicated-window plans of an
// ILU(0) pair for a cluster of `cluster` CTAs and runs the pair through the
// host emulation of k_trsv_rep.  trans 'N': y = U^{-1} diag(d) L^{-1} x;
// 'T': y = L^{-T} diag(d) U^{-T} x.  stats[4]: plan violations, steps of the
// first solve, far entries, plans usable.
// ---------------------------------------------------------------------------
// ILU(0) factorisation on the GPU (mldg_ilu0.cuh): rows grouped by the
// dependency level of L's pattern (computed on the host, one pass), one
// kernel per level.
namespace mldg {
static const double kIluEpsTol = 1.1102230246251565e-16;  // PSBLAS 3.5 d_epstol

static void ilu0_factor_gpu(int device, const mldg_csr *Ac, int32_t *Lirp, int32_t *Lja, double *Lval,
                            int32_t *Uirp, int32_t *Uja, double *Uval, double *d, int *bad_row, double *ms) {
  if (!Ac || !Lirp || !Lja || !Lval || !Uirp || !Uja || !Uval || !d || !bad_row)
    fail(MLDG_ERR_ARG, "null argument");
  HostCSR a = copy_csr(*Ac, 0, "A", 0);
  const int n = a.nr;
  if (a.nc != n) fail(MLDG_ERR_ARG, "A must be square");
  *bad_row = -1;
  if (n == 0) {
    Lirp[0] = Uirp[0] = 0;
    return;
  }
  // dependency levels of L's pattern, rows in level order
  std::vector<int> lev((size_t)n, 0);
  int nl = 0;
  for (int i = 0; i < n; ++i) {
    int l = 0;
    for (int k = a.irp[i]; k < a.irp[i + 1]; ++k)
      if (a.ja[k] < i) l = std::max(l, lev[a.ja[k]] + 1);
    lev[i] = l;
    nl = std::max(nl, l + 1);
  }
  std::vector<int> lptr((size_t)nl + 1, 0), rows((size_t)n);
  for (int i = 0; i < n; ++i) lptr[lev[i] + 1]++;
  for (int l = 0; l < nl; ++l) lptr[l + 1] += lptr[l];
  {
    std::vector<int> fillp(lptr.begin(), lptr.end() - 1);
    for (int i = 0; i < n; ++i) rows[fillp[lev[i]]++] = i;
  }
  MLDG_CUDA(cudaSetDevice(device));
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  MLDG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  Arena ar;
  try {
    MLDG_CUDA(cudaEventCreate(&e0));
    MLDG_CUDA(cudaEventCreate(&e1));
    MLDG_CUDA(cudaEventRecord(e0, st));
    int *dirp = ar.upload(a.irp), *dja = ar.upload(a.ja), *drows = ar.upload(rows);
    double *dval = ar.upload(a.val);
    int *cl = ar.alloc<int>(n), *cu = ar.alloc<int>(n);
    const int g = (int)std::min<int64_t>(((int64_t)n + 255) / 256, (int64_t)nsm * 16);
    k_ilu0_count<<<g, 256, 0, st>>>(n, dirp, dja, cl, cu);
    std::vector<int> hl((size_t)n), hu((size_t)n);
    MLDG_CUDA(cudaMemcpyAsync(hl.data(), cl, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    MLDG_CUDA(cudaMemcpyAsync(hu.data(), cu, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    MLDG_CUDA(cudaStreamSynchronize(st));
    Lirp[0] = Uirp[0] = 0;
    for (int i = 0; i < n; ++i) {
      Lirp[i + 1] = Lirp[i] + hl[i];
      Uirp[i + 1] = Uirp[i] + hu[i];
    }
    std::vector<int> vl(Lirp, Lirp + n + 1), vu(Uirp, Uirp + n + 1);
    int *dlirp = ar.upload(vl), *duirp = ar.upload(vu);
    const size_t nzl = std::max(1, Lirp[n]), nzu = std::max(1, Uirp[n]);
    int *dlja = ar.alloc<int>(nzl), *duja = ar.alloc<int>(nzu), *dbad = ar.alloc<int>(1);
    double *dlval = ar.alloc<double>(nzl), *duval = ar.alloc<double>(nzu), *dd = ar.alloc<double>(n);
    const int big = INT32_MAX;
    MLDG_CUDA(cudaMemcpyAsync(dbad, &big, sizeof(int), cudaMemcpyHostToDevice, st));
    k_ilu0_split<<<g, 256, 0, st>>>(n, dirp, dja, dval, dlirp, dlja, dlval, duirp, duja, duval, dd);
    for (int l = 0; l < nl; ++l) {
      const int cnt = lptr[l + 1] - lptr[l];
      const int gl = (int)std::min<int64_t>(((int64_t)cnt + 127) / 128, (int64_t)nsm * 8);
      k_ilu0_level<<<gl, 128, 0, st>>>(drows, lptr[l], lptr[l + 1], dlirp, dlja, dlval, duirp, duja, duval, dd,
                                       kIluEpsTol, dbad);
    }
    int bad = big;
    MLDG_CUDA(cudaMemcpyAsync(&bad, dbad, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (Lirp[n] > 0) {
      MLDG_CUDA(cudaMemcpyAsync(Lja, dlja, sizeof(int) * Lirp[n], cudaMemcpyDeviceToHost, st));
      MLDG_CUDA(cudaMemcpyAsync(Lval, dlval, sizeof(double) * Lirp[n], cudaMemcpyDeviceToHost, st));
    }
    if (Uirp[n] > 0) {
      MLDG_CUDA(cudaMemcpyAsync(Uja, duja, sizeof(int) * Uirp[n], cudaMemcpyDeviceToHost, st));
      MLDG_CUDA(cudaMemcpyAsync(Uval, duval, sizeof(double) * Uirp[n], cudaMemcpyDeviceToHost, st));
    }
    MLDG_CUDA(cudaMemcpyAsync(d, dd, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
    MLDG_CUDA(cudaEventRecord(e1, st));
    MLDG_CUDA(cudaStreamSynchronize(st));
    float t = 0;
    MLDG_CUDA(cudaEventElapsedTime(&t, e0, e1));
    if (ms) *ms = t;
    *bad_row = bad == big ? -1 : bad;
  } catch (...) {
    cudaStreamSynchronize(st);
    ar.release();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaStreamDestroy(st);
    throw;
  }
  ar.release();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
}
}  // namespace mldg

// ---------------------------------------------------------------------------
// C = A B on the GPU (mldg_spgemm.cuh), bit for bit the host's Gustavson
// product; rows with more distinct columns than a warp's table takes are
// formed on the host with the same operation order.
namespace mldg {
static void spgemm_host_row(const HostCSR &a, const HostCSR &b, int i, std::vector<int> &cols,
                            std::vector<double> &vals) {
  std::map<int, double> acc;  // column -> value, first contribution assigned
  for (int ka = a.irp[i]; ka < a.irp[i + 1]; ++ka) {
    const int k = a.ja[ka];
    const double av = a.val[ka];
    for (int kb = b.irp[k]; kb < b.irp[k + 1]; ++kb) {
      volatile double p = av * b.val[kb];  // one rounding, as the host build (no contraction)
      auto it = acc.find(b.ja[kb]);
      if (it == acc.end())
        acc.emplace(b.ja[kb], (double)p);
      else
        it->second = it->second + (double)p;
    }
  }
  cols.clear();
  vals.clear();
  for (auto &kv : acc) {
    cols.push_back(kv.first);
    vals.push_back(kv.second);
  }
}

static void spgemm_gpu(int device, const mldg_csr *Ac, const mldg_csr *Bc, int32_t **cirp, int32_t **cja,
                       double **cval, int *cnr, int *cnc, double *ms) {
  HostCSR a = copy_csr(*Ac, 0, "A", 0), b = copy_csr(*Bc, 0, "B", 0);
  if (a.nc != b.nr) fail(MLDG_ERR_SIZE, "spgemm: A is %d x %d, B is %d x %d", a.nr, a.nc, b.nr, b.nc);
  const int m = a.nr;
  MLDG_CUDA(cudaSetDevice(device));
  static bool attr = false;
  if (!attr) {
    MLDG_CUDA(cudaFuncSetAttribute(k_spgemm_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpgSmem));
    MLDG_CUDA(cudaFuncSetAttribute(k_spgemm_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpgSmem));
    attr = true;
  }
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  MLDG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  Arena ar;
  std::vector<int> irp((size_t)m + 1, 0);
  std::vector<int> ja;
  std::vector<double> val;
  try {
    MLDG_CUDA(cudaEventCreate(&e0));
    MLDG_CUDA(cudaEventCreate(&e1));
    MLDG_CUDA(cudaEventRecord(e0, st));
    int *dairp = ar.upload(a.irp), *daja = ar.upload(a.ja), *dbirp = ar.upload(b.irp), *dbja = ar.upload(b.ja);
    double *daval = ar.upload(a.val), *dbval = ar.upload(b.val);
    int *dcnt = ar.alloc<int>((size_t)std::max(m, 1));
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)m + kSpgWarps - 1) / kSpgWarps, (int64_t)nsm * 8));
    if (m > 0) k_spgemm_count<<<g, 32 * kSpgWarps, kSpgSmem, st>>>(m, dairp, daja, dbirp, dbja, dcnt);
    std::vector<int> cnt((size_t)m);
    if (m > 0) MLDG_CUDA(cudaMemcpyAsync(cnt.data(), dcnt, sizeof(int) * m, cudaMemcpyDeviceToHost, st));
    MLDG_CUDA(cudaStreamSynchronize(st));
    // rows left to the host
    std::vector<int> big;
    std::vector<std::vector<int>> bcols;
    std::vector<std::vector<double>> bvals;
    for (int i = 0; i < m; ++i)
      if (cnt[i] < 0) big.push_back(i);
    bcols.resize(big.size());
    bvals.resize(big.size());
#pragma omp parallel for schedule(dynamic, 16)
    for (size_t q = 0; q < big.size(); ++q) spgemm_host_row(a, b, big[q], bcols[q], bvals[q]);
    for (size_t q = 0; q < big.size(); ++q) cnt[big[q]] = (int)bcols[q].size();
    for (int i = 0; i < m; ++i) irp[i + 1] = irp[i] + cnt[i];
    const size_t nnz = (size_t)irp[m];
    int *dcirp = ar.upload(irp);
    int *dcja = ar.alloc<int>(std::max<size_t>(nnz, 1));
    double *dcval = ar.alloc<double>(std::max<size_t>(nnz, 1));
    // the host rows' counts go back as -1 so the fill pass skips them
    for (int i : big) cnt[i] = -1;
    std::vector<int> cflag(cnt);
    int *dflag = ar.upload(cflag);
    if (m > 0)
      k_spgemm_fill<<<g, 32 * kSpgWarps, kSpgSmem, st>>>(m, dairp, daja, daval, dbirp, dbja, dbval, dflag, dcirp,
                                                         dcja, dcval);
    ja.resize(nnz);
    val.resize(nnz);
    if (nnz) {
      MLDG_CUDA(cudaMemcpyAsync(ja.data(), dcja, sizeof(int) * nnz, cudaMemcpyDeviceToHost, st));
      MLDG_CUDA(cudaMemcpyAsync(val.data(), dcval, sizeof(double) * nnz, cudaMemcpyDeviceToHost, st));
    }
    MLDG_CUDA(cudaEventRecord(e1, st));
    MLDG_CUDA(cudaStreamSynchronize(st));
    float t = 0;
    MLDG_CUDA(cudaEventElapsedTime(&t, e0, e1));
    if (ms) *ms = t;
    for (size_t q = 0; q < big.size(); ++q) {
      std::copy(bcols[q].begin(), bcols[q].end(), ja.begin() + irp[big[q]]);
      std::copy(bvals[q].begin(), bvals[q].end(), val.begin() + irp[big[q]]);
    }
  } catch (...) {
    cudaStreamSynchronize(st);
    ar.release();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaStreamDestroy(st);
    throw;
  }
  ar.release();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
  // results in malloc'd arrays owned by the caller (mldg_free)
  *cnr = m;
  *cnc = b.nc;
  *cirp = (int32_t *)std::malloc(sizeof(int32_t) * ((size_t)m + 1));
  *cja = (int32_t *)std::malloc(sizeof(int32_t) * std::max<size_t>(ja.size(), 1));
  *cval = (double *)std::malloc(sizeof(double) * std::max<size_t>(val.size(), 1));
  if (!*cirp || !*cja || !*cval) fail(MLDG_ERR_ALLOC, "spgemm: host allocation failed");
  std::copy(irp.begin(), irp.end(), *cirp);
  std::copy(ja.begin(), ja.end(), *cja);
  std::copy(val.begin(), val.end(), *cval);
}
}  // namespace mldg

extern "C" int mldg_spgemm(int device, const mldg_csr *A, const mldg_csr *B, int32_t **Cirp, int32_t **Cja,
                           double **Cval, int *Cnrows, int *Cncols, double *ms) {
  if (!A || !B || !Cirp || !Cja || !Cval || !Cnrows || !Cncols) return MLDG_ERR_ARG;
  *Cirp = *Cja = nullptr;
  *Cval = nullptr;
  try {
    mldg::spgemm_gpu(device, A, B, Cirp, Cja, Cval, Cnrows, Cncols, ms);
  } catch (const mldg::Error &e) {
    std::free(*Cirp);
    std::free(*Cja);
    std::free(*Cval);
    *Cirp = *Cja = nullptr;
    *Cval = nullptr;
    return e.code;
  }
  return MLDG_SUCCESS;
}

extern "C" void mldg_free(void *p) { std::free(p); }

extern "C" int mldg_ilu0_factor(int device, const mldg_csr *A, int32_t *Lirp, int32_t *Lja, double *Lval,
                                int32_t *Uirp, int32_t *Uja, double *Uval, double *d, int *bad_row, double *ms) {
  try {
    mldg::ilu0_factor_gpu(device, A, Lirp, Lja, Lval, Uirp, Uja, Uval, d, bad_row, ms);
  } catch (const mldg::Error &e) {
    return e.code;
  }
  return (bad_row && *bad_row >= 0) ? 2 : MLDG_SUCCESS;
}

extern "C" int mldg_test_set_spin_limit(int device, int polls) {
  const int v = polls < 0 ? mldg::kSpinLimit : polls;
  if (cudaSetDevice(device) != cudaSuccess) return MLDG_ERR_CUDA;
  if (cudaMemcpyToSymbol(mldg::g_spin_limit, &v, sizeof(int)) != cudaSuccess) return MLDG_ERR_CUDA;
  return cudaDeviceSynchronize() == cudaSuccess ? MLDG_SUCCESS : MLDG_ERR_CUDA;
}

extern "C" int mldg_test_set_alloc_failure(int after) {
  mldg::g_alloc_failure = after;
  return MLDG_SUCCESS;
}

extern "C" int mldg_blk_plan_check(const mldg_csr *Tc, int upper, const double *scale, const double *rhs,
                                   double *t, int nblocks, int fp32, long long *stats) {
  if (!Tc || !rhs || !t || !stats || nblocks < 1) return MLDG_ERR_ARG;
  try {
    mldg::HostCSR m = mldg::copy_csr(*Tc, 0, "T", 0);
    if (m.nr != m.nc) return MLDG_ERR_ARG;
    std::vector<double> r(rhs, rhs + m.nr), out;
    auto run = [&](auto tag) {
      typedef decltype(tag) TT;
      mldg::HostBlk<TT> hb = mldg::build_blk_host<TT>(m, upper != 0, nblocks);
      stats[0] = hb.ok ? mldg::blk_emulate<TT>(hb, m, r, scale, out) : 0;
      stats[1] = hb.nsteps;
      stats[2] = hb.W;
      stats[3] = hb.ok ? 1 : 0;
      stats[4] = hb.nblocks;
      stats[5] = (long long)hb.smem;
    };
    if (fp32)
      run(float());
    else
      run(double());
    if (stats[3]) std::copy(out.begin(), out.end(), t);
  } catch (const mldg::Error &e) {
    return e.code;
  }
  return MLDG_SUCCESS;
}

extern "C" int mldg_grp_plan_check(const mldg_csr *Tc, int upper, const double *scale, const double *rhs, double *t,
                                   int ncols, long long budget, int row, double growth, int fp32, long long *stats) {
  if (!Tc || !rhs || !t || !stats || ncols < 1 || ncols > 32 || (ncols & (ncols - 1))) return MLDG_ERR_ARG;
  try {
    mldg::HostCSR m = mldg::copy_csr(*Tc, 0, "T", 0);
    if (m.nr != m.nc || m.nr < 1) return MLDG_ERR_ARG;
    mldg::TriSchedule s;
    mldg::build_tri_schedule(m.nr, m.irp.data(), m.ja.data(), m.val.data(), upper != 0, m.nr, &s);
    std::vector<int> orig, dep;
    mldg::grp_positions(m.nr, upper != 0, s.prow, s.pja, orig, dep);
    mldg::TriGroups g;
    mldg::build_tri_groups(s.lvl_ptr, s.pirp, dep, s.pval, budget > 0 ? budget : mldg::grp_budget(m.nr, ncols),
                           row > 0 ? row : mldg::kGrpRow, growth > 0 ? growth : mldg::kGrpGrowth, &g);
    const std::vector<double> r(rhs, rhs + m.nr);
    std::vector<double> x;
    auto run = [&](auto tag) {
      typedef decltype(tag) TT;
      const int KC = mldg::grp_cols<TT>(ncols);
      mldg::GrpTasks<TT> tk;
      const bool ok = mldg::grp_tasks<TT>(
          g, KC, [&](int c) { return orig[c]; }, [&](int c) { return scale ? scale[orig[c]] : 1.0; }, tk);
      stats[0] = ok ? mldg::grp_emulate<TT>(g, tk, KC, r, x) : -1;
      stats[1] = (long long)s.lvl_ptr.size() - 1;
      stats[2] = (long long)g.gptr.size() - 1;
      stats[3] = (long long)g.entries;
    };
    if (fp32)
      run(float());
    else
      run(double());
    if (stats[0] < 0) return MLDG_ERR_SIZE;
    for (int p = 0; p < m.nr; ++p) t[orig[p]] = x[p];
  } catch (const mldg::Error &e) {
    return e.code;
  } catch (const std::exception &) {
    return MLDG_ERR_ALLOC;
  }
  return MLDG_SUCCESS;
}

extern "C" int mldg_rep_plan_check(const mldg_csr *Lc, const mldg_csr *Uc, const double *d, const double *x,
                                   double *y, int cluster, int fp32, char trans, long long *stats) {
  if (!Lc || !Uc || !d || !x || !y || !stats || (cluster != 8 && cluster != 16)) return MLDG_ERR_ARG;
  try {
    mldg::HostCSR L = mldg::copy_csr(*Lc, 0, "L", 0), U = mldg::copy_csr(*Uc, 0, "U", 0);
    std::vector<double> dv(d, d + L.nr);
    if (trans == 'N') {
      if (fp32)
        mldg::rep_check_pair<float>(L, false, U, true, dv, cluster, x, y, stats);
      else
        mldg::rep_check_pair<double>(L, false, U, true, dv, cluster, x, y, stats);
    } else {
      mldg::HostCSR Ut = mldg::transpose(U), Lt = mldg::transpose(L);
      if (fp32)
        mldg::rep_check_pair<float>(Ut, false, Lt, true, dv, cluster, x, y, stats);
      else
        mldg::rep_check_pair<double>(Ut, false, Lt, true, dv, cluster, x, y, stats);
    }
  } catch (const mldg::Error &e) {
    return e.code;
  }
  return MLDG_SUCCESS;
}
