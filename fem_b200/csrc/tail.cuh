// tail.cuh -- the coarse end of the V-cycle in one kernel: one CTA per (cell,
// load case) smooths, restricts, solves and prolongs on every level whose
// vectors fit in its shared memory, down to the dense coarse solve and back.
//
// Why: on these levels (8^3 to 12^3 nodes and below) a launch per sweep is
// latency from end to end -- 17 launches of 4 to 9 us for two smoothed levels
// and the solve, whatever the arithmetic in them.  Measured figures stand at
// the rule that picks the first tail level (tail_level in engine.cu).
#pragma once
#include "kernels.cuh"

namespace femh {

constexpr int kTailLevels = 6;
constexpr int kTailThreads = 512;   // up to 128 registers: the 24 values of a voxel stay in them

struct TailLevel {
  const CellDesc* cells;
  const void* kc;          // TC
  const float* invd;
  const float* binv;       // node-block inverses, or nullptr (point Jacobi with invd)
  const double* A;         // inverses of the coarse matrices of this level's coarsest cells
  const long long* aoff;   // offset of each cell's inverse in A (cells with child < 0)
};
struct TailArgs {
  TailLevel lev[kTailLevels];   // lev[0]: first tail level
  const void* b;                // right-hand side on lev[0], [rhs][comp][node] (T)
  void* x;                      // solution on lev[0] (T)
  long long ntot;               // nodes of lev[0] over all cells
  const CGState* stt;
  HadK k;
  int pre, post;
  double w_pre[8], w_post[8];
};

// Shared memory of a cell of n[0..nl) nodes per level, in values of T: the
// iterate of lev[0], iterate and right-hand side of the deeper levels, and the
// corner contributions [24][n0] of the operator.
__host__ __device__ inline long long tail_values(const int* n, int nl) {
  long long v = 27LL * n[0];
  for (int l = 1; l < nl; ++l) v += 6LL * n[l];
  return v;
}

// Corner contributions of K x of every voxel of one level: F[(3 a + c) n + node].
// Corner a of the voxels is a permutation of the nodes, so every entry is
// written once and a node finds its 8 contributions at its own index.
template <typename T, typename TC>
__device__ __forceinline__ void tail_apply(const T* __restrict__ x, T* __restrict__ F, const CellDesc& cd,
                                           const TC* __restrict__ kc, const HadK& K) {
  const int n = cd.nx * cd.ny * cd.nz;
  for (int e = threadIdx.x; e < n; e += kTailThreads) {
    int i, j, k;
    node_ijk(e, cd.ny, cd.nz, i, j, k);
    const int k1 = k + 1 == cd.nz ? 0 : k + 1;
    const int r00 = e - k, r01 = j + 1 == cd.ny ? r00 - j * cd.nz : r00 + cd.nz;
    const int up = i + 1 == cd.nx ? -i * cd.ny * cd.nz : cd.ny * cd.nz;
    int nd[8] = {r00 + k, r00 + k1, r01 + k, r01 + k1, 0, 0, 0, 0};
#pragma unroll
    for (int a = 0; a < 4; ++a) nd[4 + a] = nd[a] + up;
    T w[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int a = 0; a < 8; ++a) w[c][a] = x[c * n + nd[a]];
      fwht8_fwd(w[c]);
    }
    had_block(w, K, (T)kc[e]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      fwht8_inv(w[c]);
#pragma unroll
      for (int a = 0; a < 8; ++a) F[(3 * a + c) * n + nd[a]] = w[c][a];
    }
  }
}

// b - K x at one node from the corner contributions (b: shared memory or the
// loop's global vector, so not __restrict__).
template <typename T>
__device__ __forceinline__ void tail_residual(const T* __restrict__ F, const T* b, long long bs, int n, int q,
                                              T (&d)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] = b[c * bs + q];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    T y = (T)0;
#pragma unroll
    for (int a = 0; a < 8; ++a) y += F[(3 * a + c) * n + q];
    d[c] -= y;
  }
}

// d <- w D^-1 d at one node of a level.
template <typename T>
__device__ __forceinline__ void tail_jacobi(const TailLevel& L, long long off, int q, T w, T (&d)[3]) {
  jacobi_dir<T>(L.binv, off + q, L.binv ? (T)0 : (T)L.invd[off + q], d);
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] *= w;
}

template <typename T, typename TC>
__global__ void __launch_bounds__(kTailThreads, 1) k_tail(const __grid_constant__ TailArgs a) {
  griddep_sync();
  extern __shared__ __align__(16) unsigned char tail_smem[];
  const int rhs = blockIdx.y, tid = threadIdx.x;
  CellDesc cd[kTailLevels];
  cd[0] = a.lev[0].cells[blockIdx.x];
  if (a.stt && !a.stt[cd[0].id * kNumRhs + rhs].active) return;
  int nl = 1;
  while (nl < kTailLevels && cd[nl - 1].child >= 0) {
    cd[nl] = a.lev[nl].cells[cd[nl - 1].child];
    ++nl;
  }
  const int n0 = cd[0].nx * cd[0].ny * cd[0].nz;
  T* F = reinterpret_cast<T*>(tail_smem);   // [24][n0]
  T* x0 = F + 24 * n0;                      // [3][n0], then [3][n] iterate and [3][n] rhs per deeper level
  const T* b0 = reinterpret_cast<const T*>(a.b) + (long long)rhs * 3 * a.ntot + cd[0].off;

  // ---- down: pre-smooth, residual, restriction
  T* x = x0;
  const T* b = b0;
  long long bs = a.ntot;   // component stride of b
  for (int l = 0; l + 1 < nl; ++l) {
    const CellDesc& c = cd[l];
    const TailLevel& L = a.lev[l];
    const TC* kc = reinterpret_cast<const TC*>(L.kc) + c.off;
    const int n = c.nx * c.ny * c.nz;
    for (int q = tid; q < n; q += kTailThreads) {   // first sweep from a zero guess
      double d[3] = {(double)b[q], (double)b[bs + q], (double)b[2 * bs + q]};
      tail_jacobi<double>(L, c.off, q, a.w_pre[0], d);
#pragma unroll
      for (int s = 0; s < 3; ++s) x[s * n + q] = (T)d[s];
    }
    __syncthreads();
    for (int sw = 1; sw <= a.pre; ++sw) {   // the last pass leaves the residual in F[0..3n)
      tail_apply<T, TC>(x, F, c, kc, a.k);
      __syncthreads();
      if (sw < a.pre) {
        for (int q = tid; q < n; q += kTailThreads) {
          T d[3];
          tail_residual<T>(F, b, bs, n, q, d);
          tail_jacobi<T>(L, c.off, q, (T)a.w_pre[sw], d);
#pragma unroll
          for (int s = 0; s < 3; ++s) x[s * n + q] += d[s];
        }
      } else {
        // in place: entry (0, s, q) of F is read by node q alone before it is written
        for (int q = tid; q < n; q += kTailThreads) {
          T d[3];
          tail_residual<T>(F, b, bs, n, q, d);
#pragma unroll
          for (int s = 0; s < 3; ++s) F[s * n + q] = d[s];
        }
      }
      __syncthreads();
    }
    // full weighting to the next level's right-hand side
    const CellDesc& cc = cd[l + 1];
    const int nc = cc.nx * cc.ny * cc.nz;
    T* xc = x + 3 * n + (l > 0 ? 3 * n : 0);   // past this level's iterate (and rhs)
    T* bc = xc + 3 * nc;
    for (int t = tid; t < 3 * nc; t += kTailThreads) {
      const int s = t / nc, q = t - s * nc;
      int i, j, k;
      node_ijk(q, cc.ny, cc.nz, i, j, k);
      double acc = 0.0;
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        const int ri = wrap(2 * i + dx, c.nx) * c.ny;
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
          const T* row = F + s * n + (ri + wrap(2 * j + dy, c.ny)) * c.nz;
          const double wxy = (dx ? 0.5 : 1.0) * (dy ? 0.5 : 1.0);
          acc += wxy * ((double)row[2 * k] +
                        0.5 * ((double)row[wrap(2 * k - 1, c.nz)] + (double)row[wrap(2 * k + 1, c.nz)]));
        }
      }
      bc[s * nc + q] = (T)acc;
    }
    __syncthreads();
    x = xc;
    b = bc;
    bs = nc;
  }

  // ---- dense solve on the coarsest level: x = A^-1 b, FP64, columns of the
  // symmetric inverse read along rows (coalesced) by groups of threads
  {
    const CellDesc& c = cd[nl - 1];
    const int n = c.nx * c.ny * c.nz, m = 3 * n;
    const double* M = a.lev[nl - 1].A + a.lev[nl - 1].aoff[nl > 1 ? cd[nl - 2].child : (int)blockIdx.x];
    double* sb = reinterpret_cast<double*>(F);             // [m] right-hand side, then [groups][m] partial sums
    // F holds 24 n0 values of T, at least 4 m doubles (m <= 3 n0): room for
    // the right-hand side and `groups` >= 1 sets of partial sums
    const int room = (int)(24LL * n0 * (int)sizeof(T) / 8 / m) - 1;
    const int groups = max(1, min(min(kTailThreads / m, 8), room));
    for (int t = tid; t < m; t += kTailThreads) sb[t] = (double)b[(t % 3) * bs + t / 3];
    __syncthreads();
    double* part = sb + m;
    const int g = tid / m;
    if (groups == 1) {
      for (int t = tid; t < m; t += kTailThreads) {
        double v = 0.0;
#pragma unroll 8
        for (int j = 0; j < m; ++j) v += M[(long long)j * m + t] * sb[j];
        part[t] = v;
      }
    } else if (g < groups) {
      const int t = tid - g * m, j0 = m * g / groups, j1 = m * (g + 1) / groups;
      double v = 0.0;
#pragma unroll 16
      for (int j = j0; j < j1; ++j) v += M[(long long)j * m + t] * sb[j];
      part[g * m + t] = v;
    }
    __syncthreads();
    for (int t = tid; t < m; t += kTailThreads) {
      double v = part[t];
      for (int q = 1; q < groups; ++q) v += part[q * m + t];
      x[(t % 3) * n + t / 3] = (T)v;
    }
    __syncthreads();
  }

  // ---- up: correction and post-smoothing
  for (int l = nl - 2; l >= 0; --l) {
    const CellDesc &c = cd[l], &cc = cd[l + 1];
    const TailLevel& L = a.lev[l];
    const TC* kc = reinterpret_cast<const TC*>(L.kc) + c.off;
    const int n = c.nx * c.ny * c.nz, nc = cc.nx * cc.ny * cc.nz;
    const T* ec = x;
    x = const_cast<T*>(ec) - 3 * n - (l > 0 ? 3 * n : 0);
    if (l == 0) {
      b = b0;
      bs = a.ntot;
    } else {
      b = x + 3 * n;
      bs = n;
    }
    for (int q = tid; q < n; q += kTailThreads) {   // trilinear
      int i, j, k;
      node_ijk(q, c.ny, c.nz, i, j, k);
      const int i0 = (i >> 1) * cc.ny, i1 = wrap((i >> 1) + (i & 1), cc.nx) * cc.ny;
      const int j0 = j >> 1, j1 = wrap(j0 + (j & 1), cc.ny), k0 = k >> 1, k1 = wrap(k0 + (k & 1), cc.nz);
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const T* e = ec + s * nc;
        auto at = [&](int r, int kk) { return (double)e[r * cc.nz + kk]; };
        const double v = ((at(i0 + j0, k0) + at(i0 + j0, k1)) + (at(i0 + j1, k0) + at(i0 + j1, k1))) +
                         ((at(i1 + j0, k0) + at(i1 + j0, k1)) + (at(i1 + j1, k0) + at(i1 + j1, k1)));
        x[s * n + q] = (T)((double)x[s * n + q] + 0.125 * v);
      }
    }
    __syncthreads();
    for (int sw = 0; sw < a.post; ++sw) {
      tail_apply<T, TC>(x, F, c, kc, a.k);
      __syncthreads();
      for (int q = tid; q < n; q += kTailThreads) {
        T d[3];
        tail_residual<T>(F, b, bs, n, q, d);
        tail_jacobi<T>(L, c.off, q, (T)a.w_post[sw], d);
#pragma unroll
        for (int s = 0; s < 3; ++s) x[s * n + q] += d[s];
      }
      __syncthreads();
    }
  }
  T* out = reinterpret_cast<T*>(a.x) + (long long)rhs * 3 * a.ntot + cd[0].off;
  for (int t = tid; t < 3 * n0; t += kTailThreads) {
    const int s = t / n0;
    out[s * a.ntot + (t - s * n0)] = x0[t];
  }
}

}  // namespace femh
