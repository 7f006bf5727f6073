// state.cuh -- host-side state of libfemh shared by its translation units: the
// cell hierarchy (levels, work unit lists), the handle, launch bookkeeping, and
// the declaration of the stencil launcher (defined in stencil_launch.cuh,
// instantiated in stencil_*.cu so that its kernels compile in parallel).
#pragma once
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/femh.h"
#include "smem_limits.hpp"
#include "stencil.cuh"

using namespace femh;

namespace femh {
struct BlockCG;   // kernels.cuh
}

namespace femh_engine {

struct FemhError {
  int code;
  std::string msg;
};

#define CK(x)                                                                              \
  do {                                                                                     \
    cudaError_t e_ = (x);                                                                  \
    if (e_ != cudaSuccess) {                                                               \
      char b_[512];                                                                        \
      snprintf(b_, sizeof b_, "%s failed: %s (%s:%d)", #x, cudaGetErrorString(e_), __FILE__, \
               __LINE__);                                                                  \
      throw FemhError{e_ == cudaErrorMemoryAllocation ? FEMH_E_OOM : FEMH_E_CUDA, b_};      \
    }                                                                                      \
  } while (0)

// ------------------------------------------------------------- device mem ---
struct Arena {
  std::vector<void*> ptrs;
  size_t held = 0;            // bytes allocated
  size_t limit = SIZE_MAX;    // FEMH_ARENA_LIMIT_BYTES (tests only): fail like a full device beyond it
  void* get(size_t bytes) {
    if (bytes == 0) bytes = 16;
    if (bytes > limit - held) throw FemhError{FEMH_E_OOM, "device memory limit of this handle reached"};
    void* p = nullptr;
    CK(cudaMalloc(&p, bytes));
    ptrs.push_back(p);
    held += bytes;
    return p;
  }
  template <typename T> T* arr(size_t n) { return static_cast<T*>(get(n * sizeof(T))); }
  void release() {
    for (void* p : ptrs) cudaFree(p);
    ptrs.clear();
    held = 0;
  }
  ~Arena() { release(); }
};

template <typename T>
T* upload(Arena& ar, const std::vector<T>& v, cudaStream_t s) {
  T* d = ar.arr<T>(std::max<size_t>(v.size(), 1));
  if (!v.empty()) CK(cudaMemcpyAsync(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
  return d;
}

struct UnitList {
  std::vector<StencilUnit> su;
  StencilUnit* d_su = nullptr;
  std::vector<NodeUnit> nu;
  NodeUnit* d_nu = nullptr;
  // persistent staged kernel (variant 7): CTA b runs units [cta[b], cta[b+1])
  std::vector<int> cta;
  int* d_cta = nullptr;
  int cta_cap = 0;   // entries allocated at d_cta
};

// Stencil units of one z extent: entries [b, e) of a unit list sorted by z extent.
struct UnitGroups {
  std::vector<int> nz, b, e;
};

struct Level {
  std::vector<CellDesc> cells;
  CellDesc* d_cells = nullptr;
  long long ntot = 0, nodes_smooth = 0;
  int level = 0;
  int NT = 256, maxnz = 1;
  int nz_spec = 0;   // > 0: every cell of the level has this z extent (specialised kernel)
  int chunk = 0;     // x-chunk length of the stencil units (0 = heuristic), set by the autotuner
  int variant = 2;   // stencil kernel (femh_config::stencil_variant numbering)
  bool bulk_ok = false;     // the bulk-copy staged FP32 kernel (variants 5, 7) can run on this level
  bool bulk_ok64 = false;   // the bulk-copy staged FP64 kernel (variant 6) can run on this level
  // cells of several z extents, each one with a compile-time kernel (a batch
  // of uneven cells): the unit lists are sorted by z extent and each extent
  // launches its own specialised kernel
  bool grouped = false;
  UnitGroups gall, gsmooth, g64;
  // level 0 of the mixed modes also runs FP64 operator applies (CG / true
  // residual): they get their own tuned layout (FP64 kernels spill in the
  // layout that suits FP32)
  bool use64 = false;
  int variant64 = 1, chunk64 = 0;
  std::vector<StencilUnit> su64;
  StencilUnit* d_su64 = nullptr;
  std::vector<int> su64_sb, su64_se;
  int *d_su64_sb = nullptr, *d_su64_se = nullptr;
  UnitList all, smooth;      // all cells / cells that continue to a coarser level
  std::vector<int> su_sb, su_se, nu_sb, nu_se;   // slot ranges per cell (all lists)
  int *d_su_sb = nullptr, *d_su_se = nullptr, *d_nu_sb = nullptr, *d_nu_se = nullptr;
  std::vector<int> coarse_list;                  // cells whose coarsest level this is
  int* d_coarse_list = nullptr;
  long long* d_aoff = nullptr;
  long long* d_cell_aoff = nullptr;              // the same by cell (coarsest cells of this level)
  double* d_A = nullptr;
  double* d_Awork = nullptr;
  double* d_Adiag = nullptr;                     // diagonal of the coarse matrices, by node of the level
  int coarse_maxm = 0;
  void* kc = nullptr;     // TC
  float* invd = nullptr;
  float* binv = nullptr;  // node-block Jacobi: [node][6] symmetric 3x3 inverses (block_jacobi)
  void* xa = nullptr;     // level vectors (TV)
  void* xb = nullptr;
  void* bv = nullptr;
};

}  // namespace femh_engine
using namespace femh_engine;

// ============================================================== handle ===
struct femh_handle {
  femh_config cfg{};
  int device = 0;
  cudaStream_t own_stream = nullptr, stream = nullptr;
  std::string err;
  long long launches = 0;
  double K0[576];
  HadK hk{};
  HadK hk_force{};   // Hadamard factors of host_k0_force (femh_force_tensors)
  ElemConst ec{};
  ElemConst* d_ec = nullptr;
  double* d_K0 = nullptr;
  std::vector<double> w_pre, w_post;   // damping weight of each smoothing sweep
  Arena perm;   // lives as long as the handle

  // setup cache
  std::vector<int> shape_key;
  std::vector<double> h_key;
  int prec_key = -1, solver_key = -1, bf16_key = -1;
  Arena setup;
  std::vector<Level> levels;
  int tail = 0;                 // first level of the fused coarse end of the V-cycle (levels.size(): none)
  std::map<std::string, int> tune_cache;   // autotuned x-chunk per level signature
  int ncells = 0;
  std::vector<long long> cell_vox;   // voxels per cell
  std::vector<long long> cell_off;   // fine offsets
  long long nvox = 0;
  // fine-level FP64 arrays
  double* rho_in = nullptr;     // packed input rho
  double* rho_used = nullptr;
  double* kc64 = nullptr;
  double* b64 = nullptr;        // [6][3][nvox]
  double* x64 = nullptr;        // solution chi
  double* r64 = nullptr;
  void* cg_x = nullptr;         // inner CG vectors (TV / TP)
  void* cg_r = nullptr;
  void* cg_p = nullptr;
  void* cg_q = nullptr;
  void* cg_rm = nullptr;        // FP32 copy of the FP64 residual (level-0 rhs of an FP32 V-cycle)
  CGState* d_state = nullptr;
  BlockCG* d_bcg = nullptr;     // block PCG step matrices per cell
  double* d_part_g = nullptr;   // block PCG 6x6 partials [2][sub-slots][36]
  double* d_part_b = nullptr;   // block PCG ||r||^2 partials [sub-slots][6]
  size_t part_g_slots = 0;      // slots of level 0 before any compaction (units keep their slot)
  int bt = 256;                 // block PCG update / direction: threads per CTA
  int bsub = 1;                 // block PCG update / direction: CTAs per level-0 node unit
  int bsub_g = 1;               // block PCG Gram kernels: CTAs per level-0 node unit
  int bsub_e = 1;               // energy kernels: CTAs per level-0 node unit
  std::vector<CGState> state;
  double* d_part_s = nullptr;   // stencil partials [slots][6]
  double* d_part_n = nullptr;   // node partials [slots][6][2]
  double* d_part_z = nullptr;   // node partials [slots][6]
  double* d_part_e = nullptr;   // energy partials [sub-slots][22]; load sums [slots][6][3] before the solve
  double* d_C = nullptr;        // [ncells][36]
  double* d_W = nullptr;        // [ncells][21]
  double* d_stage = nullptr;    // output staging (dCdrho, fields, apply), allocated on first use
  size_t stage_n = 0;           // doubles in d_stage
  // field chain rule: voxels of each field parameter (CSR), cached by the map's hash
  int* d_fmap = nullptr;        // [nparam + 1] offsets, then [nmapped] voxel indices
  size_t fmap_n = 0;            // ints allocated
  unsigned long long fmap_key = 0;
  int fmap_nparam = -1;
  double* d_nrm = nullptr;      // [ncells][6]
  double* d_mean = nullptr;     // [ncells][6][3] net force of the load over its weights (k_rhs)
  bool solved = false;
  bool have_x = false;   // x64 holds the last solution of these cells (warm starts)
  std::vector<double> C_last;

  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  SmemLimits smem_limits;        // kernels whose shared memory limit this handle has raised
  int wait_limit = kWaitLimit;   // try_wait rounds of the staged kernels' stage waits
  int nsm = 1;                   // multiprocessors of the device (persistent stencil CTAs)
  // persistent stencil CTAs are split evenly over the six load cases; the inner
  // solves of defect correction finish their load cases at different times
  // (the CTAs of a finished one would idle), so they run one CTA per unit
  bool persist_ok = true;
  // captured CG loops (pcg), kept until the set-up they run on goes: a capture
  // and its instantiation cost the host milliseconds, as much as a small solve.
  // At most one entry per loop a configuration uses (block, one case at a time).
  struct LoopGraph {
    const void* prec;   // precision tag of pcg<PR>
    const void* kcg;
    int limit, chunk;
    bool block, persist;
    cudaGraphExec_t exec;
    long long kernels;  // kernels of one pass of the loop body
  };
  std::vector<LoopGraph> loops;
  int* d_loop = nullptr;         // CG iterations run on the device in the current solve (WHILE-node count)
  int* d_err = nullptr;   // [0] set by a stencil kernel whose bounded wait ran out,
                          // [1] by k_coef on a NaN, infinite or negative density

  // measurement: per-kernel-class CUDA-event timing (femh_profile), and the
  // count of kernel executions including CUDA-graph replays
  bool prof = false;
  bool capturing = false;
  long long cap_count = 0;
  struct KStat {
    long long launches = 0;
    double ms = 0, bytes = 0;
  };
  std::map<std::string, KStat> kstats;
  struct Pend {
    std::string name;
    cudaEvent_t a, b;
    double bytes;
  };
  std::vector<Pend> pend;
  std::vector<cudaEvent_t> evpool;
};

namespace femh_engine {


#define LAUNCH_CHECK(H)                          \
  do {                                           \
    CK(cudaGetLastError());                      \
    if ((H)->capturing) (H)->cap_count++;        \
    else (H)->launches++;                        \
  } while (0)

// Raises a kernel's dynamic shared memory limit to `bytes`, the most that any
// of its launches takes (the same in every call, see smem_limits.hpp).
template <typename... P>
void allow_smem(femh_handle* H, void (*fn)(P...), int bytes) {
  H->smem_limits.raise((const void*)fn,
                       [&] { CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)); });
}

// Launch of a kernel of the CG loop, as a programmatic dependent of the kernel
// before it (griddep_sync()) while launches are a part of the time.  With more
// voxels the early CTAs only take slots from kernels of several waves, so larger
// sets launch plainly; griddep_sync() then returns at once.  Whole solves, plain
// -> early: Jacobi-PCG FP64 33x45x37 21.6 -> 20.6 ms, 64^3 71.0 -> 69.4, 96^3 312
// -> 309, 112^3 even; multigrid in FP32 48^3 6.23 -> 6.02, 64^3 8.69 -> 8.40, 96^3
// 22.0 -> 21.7, 112^3 even; multigrid in FP64, whose stencils are twice the waves,
// 32^3 3.43 -> 3.34, 56^3 13.3 -> 13.1, 64^3 12.0 -> 12.1, 80^3 24.4 -> 25.0, 96^3
// 29.4 -> 30.7, 128^3 72.1 -> 73.6.
constexpr long long kEarlyLaunchVoxels = 1 << 20, kEarlyLaunchVoxelsF64 = 200000;
inline bool early_launch(const femh_config& c, long long nvox) {
  const bool mg64 = c.solver == FEMH_GMG_PCG && c.precision == FEMH_FP64;
  return nvox <= (mg64 ? kEarlyLaunchVoxelsF64 : kEarlyLaunchVoxels);
}
template <typename... P, typename... A>
void launch(femh_handle* H, void (*fn)(P...), dim3 grid, unsigned block, size_t smem, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = H->stream;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = early_launch(H->cfg, H->nvox) ? 1 : 0;
  CK(cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...));
  LAUNCH_CHECK(H);
}

inline cudaEvent_t pool_event(femh_handle* H) {
  if (!H->evpool.empty()) {
    cudaEvent_t e = H->evpool.back();
    H->evpool.pop_back();
    return e;
  }
  cudaEvent_t e;
  CK(cudaEventCreate(&e));
  return e;
}

// Times the launches issued in its scope when profiling is on (graphs are
// not captured then, so every launch is timed on the handle's stream).
struct Prof {
  femh_handle* H;
  const char* name;
  double bytes;
  cudaEvent_t a = nullptr;
  Prof(femh_handle* h, const char* n, double b) : H(h), name(n), bytes(b) {
    if (H->prof && !H->capturing) {
      a = pool_event(H);
      CK(cudaEventRecord(a, H->stream));
    }
  }
  ~Prof() {
    if (a) {
      cudaEvent_t b = pool_event(H);
      if (cudaEventRecord(b, H->stream) == cudaSuccess) H->pend.push_back({name, a, b, bytes});
    }
  }
};

inline void release_loops(femh_handle* H) {
  for (auto& g : H->loops) cudaGraphExecDestroy(g.exec);
  H->loops.clear();
}

inline void prof_resolve(femh_handle* H) {
  if (H->pend.empty()) return;
  CK(cudaStreamSynchronize(H->stream));
  for (auto& p : H->pend) {
    float ms = 0;
    CK(cudaEventElapsedTime(&ms, p.a, p.b));
    auto& k = H->kstats[p.name];
    k.launches++;
    k.ms += ms;
    k.bytes += p.bytes;
    H->evpool.push_back(p.a);
    H->evpool.push_back(p.b);
  }
  H->pend.clear();
}

// Threads per CTA of a stencil variant on a level: the packed two-row kernel
// needs up to ~160 registers a thread, so it runs 384-thread CTAs where its
// tiles still hold at least two thread rows.
inline int variant_nt(int level_nt, int maxnz, int variant) {
  if ((variant == 4 || variant == 5 || variant == 7) && level_nt > 384 && 384 >= 2 * maxnz) return 384;
  return level_nt;
}

// z extents with compile-time kernels, and their threads per CTA.
inline bool spec_nz(int nz) { return nz == 16 || nz == 24 || nz == 32 || nz == 48 || nz == 64 || nz == 128 || nz == 256; }
inline int spec_nt(int nz) { return (nz == 24 || nz == 48) ? 480 : 512; }

// Row pitch of the staged kernels (variants 5 to 7) for a z extent: the
// smallest class that holds it, 0 if there is none.  Rows are copied in bulk,
// so extents are multiples of 4 (16 bytes); between the classes a CTA's lanes
// beyond nz idle (at most 31% of them from 36 on).  FP32 sweep, ms, best
// unstaged -> staged: 192^3 1.27 -> 0.65, 160^3 0.61 -> 0.49, 112^3 0.236 ->
// 0.163, 96^3 0.139 -> 0.085, 80^3 0.077 -> 0.065; FP64 apply 192^3 2.66 ->
// 1.33, 96^3 0.205 -> 0.125.  At 56 and 40 the two are even, and the autotuner
// times both wherever the staged kernels are eligible.  Below 36 only the
// classes themselves: the row copies would shrink to 48-112 bytes, over a
// hundred a step, on levels that the other kernels finish in microseconds.
inline int stage_class(int nz) {
  if (nz % 4 != 0) return 0;
  for (int c : {16, 24, 32, 48, 64, 96, 128, 192, 256})
    if (nz <= c) return nz == c || nz >= 36 ? c : 0;
  return 0;
}
constexpr int kStageNT32 = 384;   // variants 5, 7: 24 to 2 thread rows
// variant 6: threads a multiple of the pitch; at 192 two thread rows of which
// one is the halo (384 threads: 192^3 apply 1.33 ms; three rows of 576 threads
// hold only 96 registers each and spill: 1.70 ms; unstaged 2.66 ms)
constexpr int stage_nt64(int c) { return c == 192 ? 384 : (c == 24 || c == 48 || c == 96) ? 480 : 512; }

// One stencil launch set over a level (all cells, or those that are smoothed
// there).  T = arithmetic type; in/out/b storage types as given.
template <typename T, int OUT, typename TIn, typename TOut, typename TB, typename TC>
void stencil(femh_handle* H, Level& L, bool smooth_only, const TIn* in, TOut* out, const TB* b, const TC* kc,
             double* part, const CGState* stt, double omega);

}  // namespace femh_engine
