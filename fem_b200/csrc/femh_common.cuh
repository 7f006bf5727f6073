// femh_common.cuh -- shared device-side types of the femh homogenization engine.
//
// Grid conventions (same as the reference, desaic/fem):
//   voxel / node index (i*ny + j)*nz + k, x slowest, z fastest
//   (fast_fem/ArrayUtil.cpp gridToLinearIdx); voxel (i,j,k) has lower corner
//   node (i,j,k); local node a = 4*ax + 2*ay + az (the `oneV` order of
//   fast_fem/FEM3DFun.cpp:58-60); DOF 3*a + c.
// Device vector layout (engine-internal): [rhs][comp][node], the node range of
// every cell of a level packed one after another ("plane stride" = nodes of
// the level over all cells).
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace femh {

constexpr int kNumRhs = 6;

// One periodic cell at one multigrid level.
struct CellDesc {
  int nx, ny, nz;
  int id;            // cell index in the batch (indexes per-cell state)
  int parent;        // index of this cell in the next finer level's table (-1 at the finest)
  int child;         // index in the next coarser level's table (-1 at the cell's coarsest level)
  long long off;     // first node (= first voxel) of this cell in the level arrays
  double h;          // voxel edge at this level
};

// One CTA of the stencil kernel: rows [j0, j0+rows) x planes [i0, i0+len) of a cell.
struct StencilUnit {
  int cell;   // index into the level's CellDesc table
  int j0, rows;
  int i0, len;
  int slot;   // partial-sum slot of this unit inside its cell
};

// Node-parallel work of vector kernels: a contiguous node range of one cell.
struct NodeUnit {
  int cell;
  int slot;
  long long begin, end;   // node range relative to the cell
};

// The element stiffness of a unit cube (E = 1, h = 1) in the Hadamard basis of
// the 2x2x2 node cube.  u_hat_c(k) = sum_a chi_k(a) u_{a,c}, chi_k(a) =
// prod_s (2*bit_s(a)-1)^bit_s(k).  K0 = T^T Kh T with T = H8 (x) I3 and Kh
// block-sparse with 45 nonzeros; these eight numbers are its distinct values
// (derived on the host from the Gauss-integrated K0 and checked there).
struct HadK {
  double A;    // shear pairs  (k=1,c=x)-(k=4,c=z), (1,y)-(2,z), (2,x)-(4,y)
  double Bd;   // normal triple diagonal (4,x),(2,y),(1,z)
  double Bo;   // normal triple off-diagonal
  double D1;   // mixed triple diagonal (3,x),(5,y),(6,z)
  double O1;   // mixed triple off-diagonal
  double D2;   // mixed pairs diagonal (3,y)-(5,x), (3,z)-(6,x), (5,z)-(6,y)
  double O2;   // mixed pairs off-diagonal
  double G;    // k=7 (xyz mixed) diagonal
  double diag; // K0 diagonal entry (all 24 equal for the cube)
};

// Constants of the load and energy kernels, for h = 1 (scaled by h inside).
struct ElemConst {
  double g1[kNumRhs][24];      // K0(E=1,h=1) ue0^I(h=1), DOF 3a+c
  double uhat0[kNumRhs][3][8]; // Hadamard transform of ue0^I(h=1)
};

// Per (cell, load case) CG state, kept on the device so that iterations can be
// captured in a CUDA graph without host round trips.
struct CGState {
  double rz, pq, alpha, beta, rr, bnorm2, rel, scale;
  int iters, active, status, max_iter;
  double tol;
  int outer;        // defect correction: this (cell, rhs) takes part in the current outer step
  int fallback;     // 1: the multigrid preconditioner turned indefinite; Jacobi from then on
  double best;      // smallest relative residual so far (inner solves of defect correction)
  int since;        // iterations since it last halved
};
// An inner (FP32) solve of defect correction stops when its residual has not
// halved for this many iterations: it has reached what its arithmetic resolves,
// and the next outer step (FP64 residual) continues from there.
constexpr int kInnerStallWindow = 200;
// CG_BLOCK_FAIL: a block PCG step matrix turned indefinite; the cell's load
// cases are solved again one at a time.
enum CGStatus : int { CG_RUNNING = 0, CG_CONVERGED = 1, CG_MAXITER = 2, CG_BREAKDOWN = 3, CG_BLOCK_FAIL = 4 };

template <typename T> struct VT { using type = T; };

// Loads of vectors that the loop's kernels write: coherent loads after
// griddep_sync().  A kernel of the loop is resident while the kernel before it
// still writes, so the read-only path (__ldg, ld.global.nc), whose data must
// not change while the kernel runs, is not open to them; nor may they be plain
// reads of `const T* __restrict__` parameters, which the compiler turns into
// that path.  `volatile` keeps them after the wait; they carry no "memory"
// clobber, so other work moves around them (no kernel reads back what it wrote).
__device__ __forceinline__ double ld_val(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ float ld_val(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ float ld_val(const __nv_bfloat16* p) {
  unsigned short v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(__cvta_generic_to_global(p)));
  return __bfloat162float(__ushort_as_bfloat16(v));
}
template <typename T> using LdT = decltype(ld_val((const T*)nullptr));   // what ld_val returns for a T
// Two values from a pair-aligned address.
__device__ __forceinline__ double2 ld_val2(const double* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ float2 ld_val2(const float* p) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ void st_val(double* p, double v) { *p = v; }
__device__ __forceinline__ void st_val(float* p, float v) { *p = v; }
__device__ __forceinline__ void st_val(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// Damped-Jacobi direction at one node: d <- D^-1 d, D the point diagonal
// (inverse id, the same for the 3 components) or, with binv != nullptr, the
// node's 3x3 diagonal block of K (node-block Jacobi; the symmetric inverse
// [xx, yy, zz, xy, xz, yz] stored at binv + 6 g, 8-byte aligned).
template <typename T>
__device__ __forceinline__ void jacobi_dir(const float* __restrict__ binv, long long g, T id, T (&d)[3]) {
  if (binv) {
    const float2 b01 = *reinterpret_cast<const float2*>(binv + 6 * g);
    const float2 b23 = *reinterpret_cast<const float2*>(binv + 6 * g + 2);
    const float2 b45 = *reinterpret_cast<const float2*>(binv + 6 * g + 4);
    const T xx = (T)b01.x, yy = (T)b01.y, zz = (T)b23.x, xy = (T)b23.y, xz = (T)b45.x, yz = (T)b45.y;
    const T d0 = d[0], d1 = d[1], d2 = d[2];
    d[0] = xx * d0 + xy * d1 + xz * d2;
    d[1] = xy * d0 + yy * d1 + yz * d2;
    d[2] = xz * d0 + yz * d1 + zz * d2;
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) d[c] *= id;
  }
}

// First statement of every kernel of the CG loop: waits until the kernel before
// it in the stream is complete and its writes are visible, then lets the next
// one's CTAs be set up.  The loop's kernels are launched as programmatic
// dependents (launch() in state.cuh), so a launch overlaps its predecessor's
// run instead of following its end.  No kernel of the loop may return or touch
// memory before this call: completion of one must imply completion of all
// before it.  After it, what the loop writes is read with coherent loads
// (ld_val, or plain reads through pointers that are not __restrict__).
__device__ __forceinline__ void griddep_sync() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Warp + block reduction of nv doubles; result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_reduce(double (&v)[NV], double* smem /* >= 32*NV */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) smem[warp * NV + q] = v[q];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = (lane < nwarps) ? smem[lane * NV + q] : 0.0;
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
  }
}

}  // namespace femh
