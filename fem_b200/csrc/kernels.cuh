// kernels.cuh -- node-parallel kernels of the femh engine: coefficients, the
// strain-driven right-hand sides, fused CG vector updates with FP64 partial
// sums, per-(cell, load case) scalar finalisation, multigrid transfers, the
// dense FP64 coarse solve, and the FP64 energy reductions (C^H, dC^H/drho,
// dL/drho).
//
// All node-parallel kernels take a NodeUnit table: one CTA per (unit, load
// case), a unit being a contiguous node range of one cell, so that thousands
// of cells of different sizes run in the same launch.
#pragma once
#include <type_traits>

#include "femh_common.cuh"
#include "stencil.cuh"

namespace femh {

// Material law of the per-voxel modulus E(rho) (K0 is built for E = 1).
enum Interp : int { INTERP_SIMP = 0, INTERP_RAMP3 = 1, INTERP_BINARY = 2 };
struct MatLaw {
  int interp;
  int rho_bf16;   // round rho to bf16 before the law (mixed-precision option)
  double E_s, E_min, penal, bin_hi, bin_lo, rho_min, rho_max;
};

// SIMP's usual exponent 3 needs no pow (whose ~100 instructions are half of what
// the density gradient does per voxel besides the field sums).
__host__ __device__ inline double law_coef(const MatLaw& m, double rho) {
  if (m.interp == INTERP_SIMP)
    return m.E_min + (m.penal == 3.0 ? rho * rho * rho : pow(rho, m.penal)) * (m.E_s - m.E_min);
  if (m.interp == INTERP_RAMP3) return m.E_s * rho / (3.0 - 2.0 * rho);
  return rho >= 0.5 ? m.bin_hi : m.bin_lo;
}
__host__ __device__ inline double law_dcoef(const MatLaw& m, double rho) {
  if (m.interp == INTERP_SIMP)
    return m.penal * (m.penal == 3.0 ? rho * rho : pow(rho, m.penal - 1.0)) * (m.E_s - m.E_min);
  if (m.interp == INTERP_RAMP3) {
    const double d = 3.0 - 2.0 * rho;
    return m.E_s * 3.0 / (d * d);
  }
  return 0.0;
}

// (i, j, k) of node n of a cell; n < nx*ny*nz < 2^32, so 32-bit unsigned
// division (far cheaper than 64-bit) is exact.
__device__ __forceinline__ void node_ijk(long long n, int ny, int nz, int& i, int& j, int& k) {
  const unsigned nn = (unsigned)n, p = (unsigned)ny * (unsigned)nz;
  const unsigned ii = nn / p, rem = nn - ii * p, jj = rem / (unsigned)nz;
  i = (int)ii;
  j = (int)jj;
  k = (int)(rem - jj * (unsigned)nz);
}
__device__ __forceinline__ long long lin(int i, int j, int k, int ny, int nz) {
  return ((long long)i * ny + j) * nz + k;
}
__device__ __forceinline__ int wrap(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// ---------------------------------------------------------------- setup ---
// Fine-level stiffness scale kc[e] = E(clamp(rho_e)) * h and the rho actually used.
// A density that is NaN, infinite or negative is not clamped into range but
// reported: *bad = 1 (the host turns it into FEMH_E_ARG before solving).
template <typename TC2>
__global__ void k_coef(const CellDesc* cells, const NodeUnit* units, const double* rho, MatLaw law,
                       double* kc64, TC2* kc2, double* rho_used, int* bad) {
  const NodeUnit u = units[blockIdx.x];
  const CellDesc cd = cells[u.cell];
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    double r = rho[cd.off + n];
    if (!(r >= 0.0) || isinf(r)) {
      *bad = 1;
      r = 0.0;
    }
    r = fmin(fmax(r, law.rho_min), law.rho_max);
    const double kc = law_coef(law, r) * cd.h;
    if (rho_used) rho_used[cd.off + n] = r;
    if (kc64) kc64[cd.off + n] = kc;
    if (kc2) {
      // the inner (FP32) operator may see rho rounded to bf16; the FP64
      // operator that defines the solution always uses rho as given
      const double rb = law.rho_bf16 ? (double)__bfloat162float(__float2bfloat16_rn((float)r)) : r;
      kc2[cd.off + n] = (TC2)(law.rho_bf16 ? law_coef(law, rb) * cd.h : kc);
    }
  }
}

// Rediscretised coarse scale: the coarse voxel's modulus is the mean of its 8
// children's moduli and its edge is 2h, so kc_c = mean(kc_f / h) * 2h =
// 2 mean(kc_f).  avg: 0 arithmetic mean, 1 geometric, 2 harmonic.
template <typename TF, typename TCo>
__global__ void k_coarsen_coef(const CellDesc* fine, const CellDesc* coarse, const NodeUnit* units,
                               const TF* kcf, TCo* kcc, int avg) {
  const NodeUnit u = units[blockIdx.x];
  const CellDesc cc = coarse[u.cell], cf = fine[cc.parent];
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    int i, j, k;
    node_ijk(n, cc.ny, cc.nz, i, j, k);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const double v = (double)kcf[cf.off + lin(2 * i + ((a >> 2) & 1), 2 * j + ((a >> 1) & 1), 2 * k + (a & 1),
                                                cf.ny, cf.nz)];
      s += (avg == 0) ? v : (avg == 1 ? log(v) : 1.0 / v);
    }
    const double m = (avg == 0) ? s / 8.0 : (avg == 1 ? exp(s / 8.0) : 8.0 / s);
    kcc[cc.off + n] = (TCo)(2.0 * m);
  }
}

// Point-Jacobi inverse diagonal: all 24 diagonal entries of the cube's K0 are
// equal, so diag(K)_n = K0diag * sum_{8 voxels at n} kc_e for all 3 components.
template <typename TC>
__global__ void k_invdiag(const CellDesc* cells, const NodeUnit* units, const TC* kc, double diag,
                          float* invd) {
  const NodeUnit u = units[blockIdx.x];
  const CellDesc cd = cells[u.cell];
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    int i, j, k;
    node_ijk(n, cd.ny, cd.nz, i, j, k);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 8; ++a)
      s += (double)kc[cd.off + lin(wrap(i - ((a >> 2) & 1), cd.nx), wrap(j - ((a >> 1) & 1), cd.ny),
                                   wrap(k - (a & 1), cd.nz), cd.ny, cd.nz)];
    invd[cd.off + n] = (float)(1.0 / (diag * s));
  }
}

// Node-block Jacobi: D_n = the 3x3 diagonal block of K at node n = sum over
// the 8 voxels at n of kc_e K0(1)_aa, a = the node's corner in voxel e.  The
// cube's corner blocks are d I + o S_a, S_a(c1, c2) = sigma_c1 sigma_c2 off the
// diagonal, sigma_c = 1 - 2 bit_c(a) (d = K0 diagonal, o = K0[0][1]), so
// D_n = d (sum kc) I + o T_n with T_n(c1, c2) = sum_e kc_e sigma_c1 sigma_c2.
// binv[6 (cd.off + n) + k] = the symmetric inverse, k = xx, yy, zz, xy, xz, yz
// (FP32).
template <typename TC>
__global__ void k_invblock(const CellDesc* cells, const NodeUnit* units, const TC* kc, double d, double o,
                           float* binv) {
  const NodeUnit u = units[blockIdx.x];
  const CellDesc cd = cells[u.cell];
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    int i, j, k;
    node_ijk(n, cd.ny, cd.nz, i, j, k);
    double sum = 0.0, txy = 0.0, txz = 0.0, tyz = 0.0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int ax = (a >> 2) & 1, ay = (a >> 1) & 1, az = a & 1;
      const double ke = (double)kc[cd.off + lin(wrap(i - ax, cd.nx), wrap(j - ay, cd.ny), wrap(k - az, cd.nz), cd.ny,
                                                cd.nz)];
      const double sx = 1.0 - 2.0 * ax, sy = 1.0 - 2.0 * ay, sz = 1.0 - 2.0 * az;
      sum += ke;
      txy += ke * sx * sy;
      txz += ke * sx * sz;
      tyz += ke * sy * sz;
    }
    const double A = d * sum, X = o * txy, Y = o * txz, Z = o * tyz;   // [[A X Y] [X A Z] [Y Z A]]
    const double c00 = A * A - Z * Z, c11 = A * A - Y * Y, c22 = A * A - X * X;
    const double c01 = Y * Z - X * A, c02 = X * Z - Y * A, c12 = X * Y - A * Z;
    const double det = A * c00 + X * c01 + Y * c02;
    const double r = 1.0 / det;
    float* out = binv + 6 * (cd.off + n);
    out[0] = (float)(c00 * r);
    out[1] = (float)(c11 * r);
    out[2] = (float)(c22 * r);
    out[3] = (float)(c01 * r);
    out[4] = (float)(c02 * r);
    out[5] = (float)(c12 * r);
  }
}

// Strain-driven load b^I_n = -sum_{e at n} c_e (K0(h) ue0^I(h))[a_n(e)]
//   = -h * sum_e kc_e g1^I[a_n(e)]  (K0(h) = h K0(1), ue0(h) = h ue0(1), kc = c h),
// without its net force.  The exact load has none, and the solver leaves the
// three translations free, so it needs a load without one; and where the exact
// load is zero (a uniform neighbourhood), rounding must not make one up: a
// node's sum below its rounding bound, 8 u sum |kc_e g1|, is 0.  The net force
// that rounding leaves is taken from the nodes in proportion to the stiffness
// of their voxels, sum kc_e: in equal parts it would load soft voxels out of all
// proportion to theirs (layers of 1 and 1e-12: C_11 off by 2e-9 of itself, now
// below 1e-12) and voxels that have none.
// Two passes over the densities (8 B per node each, against 144 B of load): SUM
// adds the load up, [slot][6][3] partials, and the weights, [slot][6][2] (first
// entry of load case 0); the other writes it less `mean`, its net force over
// the sum of the weights per (cell, load case, component), times the weight.
// One CTA per (unit, load case).
template <bool SUM>
__global__ void k_rhs(const CellDesc* cells, const NodeUnit* units, const double* kc64, const ElemConst* ec,
                      double* __restrict__ b, long long ntot, double* __restrict__ part,
                      double* __restrict__ wpart, const double* __restrict__ mean) {
  const NodeUnit u = units[blockIdx.x];
  const int I = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  double v[4] = {0.0, 0.0, 0.0, 0.0};   // net force, sum of the weights
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    int i, j, k;
    node_ijk(n, cd.ny, cd.nz, i, j, k);
    double acc[3] = {0, 0, 0}, size[3] = {0, 0, 0}, w = 0.0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const double ke = kc64[cd.off + lin(wrap(i - ((a >> 2) & 1), cd.nx), wrap(j - ((a >> 1) & 1), cd.ny),
                                          wrap(k - (a & 1), cd.nz), cd.ny, cd.nz)];
      w += ke;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        acc[c] += ke * ec->g1[I][3 * a + c];
        size[c] += ke * fabs(ec->g1[I][3 * a + c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double f = fabs(acc[c]) <= 8.0 * 1.1102230246251565e-16 * size[c] ? 0.0 : -cd.h * acc[c];
      if (SUM) v[c] += f;
      else b[((long long)I * 3 + c) * ntot + cd.off + n] = f - mean[(cd.id * kNumRhs + I) * 3 + c] * w;
    }
    if (SUM) v[3] += w;
  }
  if (SUM) {
    __shared__ double red[32 * 4];
    block_reduce<4>(v, red);
    if (threadIdx.x == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) part[((long long)u.slot * kNumRhs + I) * 3 + c] = v[c];
      if (I == 0) wpart[(long long)u.slot * kNumRhs * 2] = v[3];
    }
  }
}

// ------------------------------------------------------------- CG pieces ---
// Start of PCG: x = 0 (kept as it is when keep_x: a warm start, with b the
// residual of that x), r = s*b (s = per (cell,rhs) scale), partial ||r||^2.
// With jacobi != 0 also partial r.(invd r) for the Jacobi-preconditioned rz and
// p = invd r.  Partials: [slot][6][2].
template <typename TB, typename TV, typename TP>
__global__ void k_cg_init(const CellDesc* cells, const NodeUnit* units, const TB* __restrict__ b, TV* __restrict__ x, TV* __restrict__ r,
                          TP* __restrict__ p, const float* __restrict__ invd, const CGState* stt, double* __restrict__ part, long long ntot,
                          int jacobi, int keep_x) {
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  const CGState S = stt[cd.id * kNumRhs + rhs];
  double v[2] = {0.0, 0.0};
  if (S.active) {
    #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
      const long long g = cd.off + n;
      const float id = invd[g];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const long long o = ((long long)rhs * 3 + c) * ntot + g;
        const double rv = S.scale * (double)ld_val(b + o);
        if (!keep_x) st_val(x + o, 0.0);
        st_val(r + o, rv);
        v[0] += rv * rv;
        const double z = (double)id * rv;
        v[1] += rv * z;
        if (jacobi) st_val(p + o, z);
      }
    }
  }
  __shared__ double red[64];
  block_reduce<2>(v, red);
  if (threadIdx.x == 0) {
    part[((long long)u.slot * kNumRhs + rhs) * 2 + 0] = v[0];
    part[((long long)u.slot * kNumRhs + rhs) * 2 + 1] = v[1];
  }
}

// x += alpha p ; r -= alpha q ; partial ||r||^2 and, for
// Jacobi, r.(invd r).  For the multigrid preconditioner (z0 != nullptr) it
// also writes the first damped-Jacobi sweep from zero: z0 = omega invd r, and,
// when rm != nullptr, r in the V-cycle's storage type (the level-0 right-hand
// side its sweeps read).
template <typename TV, typename TP, typename TQ, typename TZ>
__global__ void __launch_bounds__(256, 2)
k_cg_update(const CellDesc* cells, const NodeUnit* units, TV* __restrict__ x, TV* __restrict__ r,
            const TP* __restrict__ p, const TQ* __restrict__ q, const float* __restrict__ invd, TZ* __restrict__ z0,
            TZ* __restrict__ rm, double omega, const CGState* stt, double* __restrict__ part, long long ntot,
            const float* __restrict__ binv) {
  griddep_sync();
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  const CGState S = stt[cd.id * kNumRhs + rhs];
  double v[2] = {0.0, 0.0};
  if (S.active) {
    const double al = S.alpha;
    // A thread issues the loads of U nodes before its first store, which later
    // loads cannot pass.  The stores' addresses are formed anew: kept from the
    // loads they would take as many registers as the values.  FP64 with U = 4
    // spills at the 128 registers that two CTAs leave (Jacobi solves, U = 1, 2, 4:
    // 32^3 7.74, 7.53, 7.90 ms; 33x45x37 18.97, 18.97, 20.03).
    constexpr int U = sizeof(TV) == 8 ? 2 : 4;
    const long long base = (long long)rhs * 3 * ntot + cd.off;
    const unsigned end = (unsigned)u.end, bd = blockDim.x;
#pragma unroll 1
    for (unsigned n0 = (unsigned)u.begin + threadIdx.x; n0 < end; n0 += U * bd) {
      LdT<TV> xs[U][3], rs[U][3];
      LdT<TP> ps[U][3];
      LdT<TQ> qs[U][3];
      float ids[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const unsigned n = n0 + k * bd;
        if (n >= end) break;
        ids[k] = invd[cd.off + n];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const long long o = base + c * ntot;
          ps[k][c] = ld_val(p + o + n);
          xs[k][c] = ld_val(x + o + n);
          rs[k][c] = ld_val(r + o + n);
          qs[k][c] = ld_val(q + o + n);
        }
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        unsigned n = n0 + k * bd;
        if (n >= end) break;
        asm volatile("" : "+r"(n));
        const double id = (double)ids[k];
        double rvs[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const long long o = base + c * ntot;
          const double xv = (double)xs[k][c] + al * (double)ps[k][c];
          const double rv = (double)rs[k][c] - al * (double)qs[k][c];
          st_val(x + o + n, xv);
          st_val(r + o + n, rv);
          v[0] += rv * rv;
          v[1] += rv * id * rv;
          if (z0 && !binv) st_val(z0 + o + n, omega * id * rv);
          if (rm) st_val(rm + o + n, rv);
          rvs[c] = rv;
        }
        if (z0 && binv) {   // node-block Jacobi: z0 = omega B r
          jacobi_dir<double>(binv, cd.off + n, 0.0, rvs);
#pragma unroll
          for (int c = 0; c < 3; ++c) st_val(z0 + base + c * ntot + n, omega * rvs[c]);
        }
      }
    }
  }
  __shared__ double red[64];
  block_reduce<2>(v, red);
  if (threadIdx.x == 0) {
    part[((long long)u.slot * kNumRhs + rhs) * 2 + 0] = v[0];
    part[((long long)u.slot * kNumRhs + rhs) * 2 + 1] = v[1];
  }
}

// p = z + beta p, with z = invd r (Jacobi) or z read from zvec (multigrid).
template <typename TP, typename TZ, typename TR>
__global__ void k_cg_dir(const CellDesc* cells, const NodeUnit* units, TP* __restrict__ p, const TZ* __restrict__ zvec,
                         const TR* __restrict__ r, const float* __restrict__ invd, const CGState* stt, long long ntot) {
  griddep_sync();
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  const CGState S = stt[cd.id * kNumRhs + rhs];
  if (!S.active) return;
  const double be = S.beta;
  constexpr int U = 4;   // as in k_cg_update
  const long long base = (long long)rhs * 3 * ntot + cd.off;
  const unsigned end = (unsigned)u.end, bd = blockDim.x;
  // one loop per source of z: a choice at each load would part the loads
  auto pass = [&](auto from_z) {
    constexpr bool MG = decltype(from_z)::value;
#pragma unroll 1
    for (unsigned n0 = (unsigned)u.begin + threadIdx.x; n0 < end; n0 += U * bd) {
      LdT<typename std::conditional<MG, TZ, TR>::type> zs[U][3];
      LdT<TP> ps[U][3];
      float ids[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const unsigned n = n0 + k * bd;
        if (n >= end) break;
        if (!MG) ids[k] = invd[cd.off + n];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const long long o = base + c * ntot;
          if constexpr (MG) zs[k][c] = ld_val(zvec + o + n);
          else zs[k][c] = ld_val(r + o + n);
          ps[k][c] = ld_val(p + o + n);
        }
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        unsigned n = n0 + k * bd;
        if (n >= end) break;
        asm volatile("" : "+r"(n));
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double z = MG ? (double)zs[k][c] : (double)ids[k] * (double)zs[k][c];
          st_val(p + base + c * ntot + n, be == 0.0 ? z : z + be * (double)ps[k][c]);
        }
      }
    }
  };
  if (zvec && !S.fallback) pass(std::true_type{});
  else pass(std::false_type{});
}

// Sum of the partials of one (cell, rhs) over the cell's slot range: one warp,
// lane-strided then a shuffle tree (fixed order: deterministic).  Valid in all lanes.
__device__ __forceinline__ double sum_slots(const double* part, int b, int e, int rhs, int stride,
                                            int comp) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int t = b + lane; t < e; t += 32) s += part[((long long)t * kNumRhs + rhs) * stride + comp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// ------------------------------------------------------ block PCG ---
// Block conjugate gradients over the six load cases of a cell (O'Leary,
// Linear Algebra Appl. 29, 1980): they share the operator and the
// preconditioner, so one Krylov space serves all six and the scalar steps
// become 6x6 matrices.  Each new search block is made K-conjugate to the
// previous one explicitly (the flexible form, as in Notay's flexible CG,
// SIAM J. Sci. Comput. 22, 2000), so an FP32 V-cycle that is symmetric only to
// its rounding keeps the directions conjugate:
//   G = P^T K P,  alpha = G^+ (Z^T R),  X += P alpha,  R -= (K P) alpha,
//   Z = M R,      beta = -G^+ ((K P)^T Z),  P = Z + P beta.
// G^+ solves by Cholesky and drops a direction whose pivot falls below `drop`
// of its diagonal (dependent on the earlier ones to the accuracy of the
// preconditioned block: 1e-12 with an FP64 V-cycle, 1e-8 with an FP32 one).
// Load cases that are not live at the start (a zero right-hand side) stay out
// of every product.
struct BlockCG {
  double g[36];       // P^T K P of the current search block, symmetric, row-major
  double zr[36];      // zr[k * 6 + j] = z_k . r_j
  double alpha[36];   // alpha[i * 6 + j]: weight of direction i in load case j
  double beta[36];    // beta[i * 6 + j]: weight of old direction i in new direction j
  double best;        // smallest worst-case relative residual of the block so far
  int since;          // iterations since that last halved
  int mask;           // load cases in the block (bit j)
  int live;           // 1 while the block iterates
};
// A block whose worst relative residual has not halved for this many
// iterations has stalled: its cell is solved again one load case at a time.
constexpr int kBlockStallWindow = 200;

// G X = s B (6x6, row-major, shared memory) by Cholesky on the columns in mask,
// a column with a pivot below drop times its diagonal dropped (its row of X is
// 0).  Returns false if a pivot is below -1e-8 times its diagonal (G indefinite
// beyond rounding), not finite, or no column is kept.  One warp: lane r holds
// row r of L (r < 6), then lane c solves column c; one thread alone took 10 us
// of divisions in a row, the warp takes ~1.
__device__ __forceinline__ bool chol_solve6(const double* G, const double* B, double sgn, double* X, int mask,
                                            double drop) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, r = min(lane, 5);
  double l[6], inv[6];
  bool ok = true, any = false;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = G[r * 6 + k];
#pragma unroll
    for (int j = 0; j < k; ++j) v -= l[j] * __shfl_sync(full, l[j], k);
    const double d = __shfl_sync(full, v, k), gkk = G[k * 6 + k];
    const bool in = mask >> k & 1;
    if (in && (!isfinite(d) || d < -1e-8 * fabs(gkk))) ok = false;
    const bool use = in && gkk > 0.0 && d > drop * gkk;
    const double lkk = use ? sqrt(d) : 1.0;
    inv[k] = use ? 1.0 / lkk : 0.0;
    l[k] = r == k ? lkk : (r > k ? v * inv[k] : 0.0);
    any = any || use;
  }
  double y[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = sgn * B[k * 6 + r];
#pragma unroll
    for (int j = 0; j < k; ++j) v -= __shfl_sync(full, l[j], k) * y[j];
    y[k] = v * inv[k];
  }
#pragma unroll
  for (int k = 5; k >= 0; --k) {
    double v = y[k];
#pragma unroll
    for (int j = k + 1; j < 6; ++j) v -= __shfl_sync(full, l[k], j) * y[j];
    y[k] = v * inv[k];
  }
  if (lane < 6)
#pragma unroll
    for (int k = 0; k < 6; ++k) X[k * 6 + lane] = y[k];
  __syncwarp();
  return ok && any;
}

// The block kernels split each node unit into S sub-ranges, one CTA each (S
// > 1 gives small cells enough CTAs); partial sums go to sub-slot slot*S + s.
struct SubUnit {
  NodeUnit u;
  long long begin, end;
  long long sub;   // partial-sum index
};
__device__ __forceinline__ SubUnit sub_unit(const NodeUnit* units, int S) {
  const int s = (int)(blockIdx.x % (unsigned)S);
  SubUnit r;
  r.u = units[blockIdx.x / (unsigned)S];
  const long long len = r.u.end - r.u.begin;
  r.begin = r.u.begin + len * s / S;
  r.end = r.u.begin + len * (s + 1) / S;
  r.sub = (long long)r.u.slot * S + s;
  return r;
}

// D += A B on the FP64 tensor cores: A 16 x 8 (lane l holds rows l / 4 and + 8
// of columns l % 4 and + 4), B 8 x 8 (rows l % 4 and + 4, column l / 4), D 16 x 8
// (rows l / 4 and + 8, columns 2 (l % 4) and the next).  Lane l's values of load
// case l / 4 at two nodes serve as rows of A or as columns of B.
__device__ __forceinline__ void dmma1688(double (&d)[4], double lo0, double hi0, double lo1, double hi1, double b0,
                                         double b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(lo0), "d"(hi0), "d"(lo1), "d"(hi1), "d"(b0), "d"(b1));
}
template <typename T>
__device__ __forceinline__ void ld_pair(const T* p, bool vec, bool in0, bool in1, double (&v)[2]) {
  if (vec && in0 && in1) {
    const auto t = ld_val2(p);
    v[0] = (double)t.x;
    v[1] = (double)t.y;
  } else {
    v[0] = in0 ? (double)ld_val(p) : 0.0;
    v[1] = in1 ? (double)ld_val(p + 1) : 0.0;
  }
}

// Partials of the 6x6 matrix A^T B (entry i * 6 + j = a_i . b_j) of one cell's
// block per sub-slot, and with TWO of C^T A as well, A read once; columns
// outside the block's mask read as 0.  A warp takes eight nodes at a time, lane
// l the nodes 2 (l % 4) and the next of load case l / 4, and sums the products
// on the FP64 tensor cores: four registers for both matrices, where a thread
// per node needed 36 accumulators each (72 spilled) and their reduction over
// the CTA.  Z^T R and (K P)^T Z: 128^3 two passes of 125 + 121 us -> one of 215
// (0.52 of measured HBM), 64^3 31 + 29 -> 36; P^T K P 119 -> 113 and 21 -> 17
// (0.82).  Four nodes a lane, four times fewer or more CTAs and 8 x 8 x 4
// products all measured the same within 5%.
template <bool TWO, typename TA, typename TB, typename TC>
__global__ void __launch_bounds__(256)
k_bgram(const CellDesc* cells, const NodeUnit* units, const TA* __restrict__ a, const TB* __restrict__ b,
        const TC* __restrict__ c, const BlockCG* bst, double* __restrict__ part_ab, double* __restrict__ part_ca,
        long long ntot, int nsub) {
  griddep_sync();
  const SubUnit su = sub_unit(units, nsub);
  const CellDesc cd = cells[su.u.cell];
  const int mask = bst[cd.id].live ? bst[cd.id].mask : 0;
  if (!mask) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int i = lane >> 2, q = lane & 3;
  const bool on = i < kNumRhs && (mask >> i & 1);
  // pairs start at even level nodes; with an odd plane stride pairs are loaded one by one
  const bool vec = (ntot & 1) == 0;
  const long long begin = cd.off + su.begin, end = cd.off + su.end;
  double d[4] = {0.0, 0.0, 0.0, 0.0};   // rows 0-7: b_i . a_j, rows 8-15: c_i . a_j
  for (long long g0 = (begin & ~1LL) + 8 * warp; g0 < end; g0 += 8 * nw) {
    const long long g = g0 + 2 * q;
    const bool in0 = on && g >= begin && g < end, in1 = on && g + 1 >= begin && g + 1 < end;
    double av[3][2], bv[3][2], cv[3][2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long long o = ((long long)i * 3 + k) * ntot + g;
      ld_pair(a + o, vec, in0, in1, av[k]);
      ld_pair(b + o, vec, in0, in1, bv[k]);
      if (TWO) ld_pair(c + o, vec, in0, in1, cv[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      dmma1688(d, bv[k][0], TWO ? cv[k][0] : 0.0, bv[k][1], TWO ? cv[k][1] : 0.0, av[k][0], av[k][1]);
  }
  __shared__ double red[TWO ? 2 : 1][8][36];   // per warp
  if (i < kNumRhs && q < 3) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      red[0][warp][(2 * q + h) * 6 + i] = d[h];
      if (TWO) red[TWO ? 1 : 0][warp][i * 6 + 2 * q + h] = d[2 + h];
    }
  }
  __syncthreads();
  if (threadIdx.x < (TWO ? 72 : 36)) {
    const int m = threadIdx.x / 36, k = threadIdx.x % 36;
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += red[m][w][k];
    (m ? part_ca : part_ab)[su.sub * 36 + k] = v;
  }
}

// Sums of a cell's per-slot partials by a 1024-thread CTA in a fixed order
// (deterministic): value v of set q (NQ sets of n[q] values, slots [b[q], e[q])
// of part[q]) is added up by G[q] threads, thread g over the slots b + g,
// b + g + G, ... (coalesced rows, eight loads in flight per thread), then the G
// sums by one thread.  sum n[q] G[q] <= 1024.  out (shared memory, the sets one
// after another) is valid after the call in every thread.  256 threads without
// the unrolling took 24 us of a 128^3 iteration for the three sums of the beta
// step; with the same G for its sets the 4096 slots of ||r||^2 took 25.
template <int NQ>
__device__ __forceinline__ void cta_sums(const double* const (&part)[NQ], const int (&n)[NQ], const int (&G)[NQ],
                                         const int (&b)[NQ], const int (&e)[NQ], double* red, double* out) {
  const int t = threadIdx.x;
  int first = 0, val = 0;   // threads and values of the sets before
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int nq = n[q], Gq = G[q], u = t - first;
    if (u >= 0 && u < nq * Gq) {
      const double* p = part[q] + u % nq;
      const int end = e[q];
      double acc = 0.0;
#pragma unroll 8
      for (int sl = b[q] + u / nq; sl < end; sl += Gq) acc += p[(long long)sl * nq];
      red[t] = acc;
    }
    first += nq * Gq;
  }
  __syncthreads();
  first = 0;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int nq = n[q], Gq = G[q], v = t - val;
    if (v >= 0 && v < nq) {
      double acc = 0.0;
#pragma unroll 8
      for (int g = 0; g < Gq; ++g) acc += red[first + g * nq + v];
      out[t] = acc;
    }
    first += nq * Gq;
    val += nq;
  }
  __syncthreads();
}

// The block stops: its load cases leave the loop with `status`.  One warp.
__device__ __forceinline__ void block_stop(BlockCG& B, CGState* stt, int cell, int mask, int status) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) B.live = 0;
  if (lane < kNumRhs && (mask >> lane & 1)) {
    CGState& S = stt[cell * kNumRhs + lane];
    S.active = 0;
    S.status = status == CG_MAXITER && S.rel < S.tol ? CG_CONVERGED : status;
  }
}

// z_j . r_j of every load case of the block positive: the preconditioner is
// positive on the current residuals.  One warp.
__device__ __forceinline__ bool zr_positive(const double* Z, int mask) {
  const int lane = threadIdx.x & 31;
  const bool mine = lane < kNumRhs && (mask >> lane & 1);
  const double z = mine ? Z[lane * 7] : 1.0;
  return __all_sync(0xffffffffu, z > 0.0 && isfinite(z));
}

// After k_fin_init: the block of each cell is its live load cases.
__global__ void k_binit(BlockCG* bst, const CGState* stt, int ncells) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= ncells) return;
  int mask = 0;
  for (int j = 0; j < kNumRhs; ++j)
    if (stt[cell * kNumRhs + j].active) mask |= 1 << j;
  BlockCG& B = bst[cell];
  B.mask = mask;
  B.live = mask != 0;
  B.best = INFINITY;
  B.since = 0;
  for (int k = 0; k < 36; ++k) B.alpha[k] = B.beta[k] = 0.0;
}

// After the first preconditioner application: Z^T R of the start (beta = 0).
// One 1024-thread CTA per cell.
__global__ void __launch_bounds__(1024) k_bfin_rz(BlockCG* bst, CGState* stt, const int* sb, const int* se,
                                                  const double* part_zr, int ncells, int nsub) {
  const int cell = blockIdx.x, lane = threadIdx.x;
  BlockCG& B = bst[cell];
  if (!B.live) return;
  __shared__ double red[1024], Z[36];
  cta_sums<1>({part_zr}, {36}, {28}, {sb[cell] * nsub}, {se[cell] * nsub}, red, Z);
  if (lane >= 32) return;
  if (!zr_positive(Z, B.mask)) return block_stop(B, stt, cell, B.mask, CG_BLOCK_FAIL);
  for (int k = lane; k < 36; k += 32) B.zr[k] = Z[k];
}

// G = P^T K P, alpha = G^+ Z^T R.  One 1024-thread CTA per cell.
__global__ void __launch_bounds__(1024) k_bfin_alpha(BlockCG* bst, CGState* stt, const int* sb, const int* se,
                                                     const double* part_g, int ncells, double drop, int nsub) {
  griddep_sync();
  const int cell = blockIdx.x, lane = threadIdx.x;
  BlockCG& B = bst[cell];
  if (!B.live) return;
  __shared__ double red[1024], g[36], G[36], A[36], ZR[36];
  cta_sums<1>({part_g}, {36}, {28}, {sb[cell] * nsub}, {se[cell] * nsub}, red, g);
  if (lane >= 32) return;
  for (int k = lane; k < 36; k += 32) {
    const int i = k / 6, j = k % 6;
    G[k] = i <= j ? g[k] : g[j * 6 + i];   // symmetric to the last bit
    ZR[k] = B.zr[k];
  }
  __syncwarp();
  if (!chol_solve6(G, ZR, 1.0, A, B.mask, drop)) return block_stop(B, stt, cell, B.mask, CG_BLOCK_FAIL);
  for (int k = lane; k < 36; k += 32) {
    B.alpha[k] = A[k];
    B.g[k] = G[k];
  }
}

// After the update and the preconditioner: convergence of every load case of
// the block, then beta = -G^+ (K P)^T Z.  One 1024-thread CTA per cell; the
// Gram partials come in nsub_g sub-slots per slot, the ||r||^2 ones in nsub.
__global__ void __launch_bounds__(1024) k_bfin_beta(BlockCG* bst, CGState* stt, const int* sb, const int* se,
                                                    const double* part_upd, const double* part_zr,
                                                    const double* part_qz, int ncells, double drop, int nsub_g,
                                                    int nsub) {
  griddep_sync();
  const int cell = blockIdx.x, lane = threadIdx.x;
  BlockCG& B = bst[cell];
  if (!B.live) return;
  const int b = sb[cell], e = se[cell];
  __shared__ double red[1024], sums[78], T[36], G[36];
  cta_sums<3>({part_zr, part_qz, part_upd}, {36, 36, kNumRhs}, {10, 10, 50}, {b * nsub_g, b * nsub_g, b * nsub},
              {e * nsub_g, e * nsub_g, e * nsub}, red, sums);
  if (lane >= 32) return;
  const double *Z = sums, *Q = sums + 36, *rr = sums + 72;
  const unsigned full = 0xffffffffu;
  const int mask = B.mask;
  const bool mine = lane < kNumRhs && (mask >> lane & 1);
  double rel = 0.0;
  bool conv = true, spent = false, bad = false;
  if (mine) {
    CGState& S = stt[cell * kNumRhs + lane];
    rel = sqrt(rr[lane] / S.bnorm2);
    S.rr = rr[lane];
    S.iters += 1;
    S.rel = rel;
    conv = rel < S.tol;
    spent = S.iters >= S.max_iter;
    bad = !isfinite(rel);
  }
  if (__all_sync(full, conv)) return block_stop(B, stt, cell, mask, CG_CONVERGED);
  if (__any_sync(full, bad)) return block_stop(B, stt, cell, mask, CG_BREAKDOWN);
  if (__any_sync(full, spent)) return block_stop(B, stt, cell, mask, CG_MAXITER);
  double worst = rel;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(full, worst, o));
  worst = __shfl_sync(full, worst, 0);
  const double best = B.best;
  const int since = B.since + 1;
  __syncwarp();
  if (worst < 0.5 * best) {
    if (lane == 0) {
      B.best = worst;
      B.since = 0;
    }
  } else {
    if (lane == 0) B.since = since;
    if (since >= kBlockStallWindow) return block_stop(B, stt, cell, mask, CG_BLOCK_FAIL);
  }
  for (int k = lane; k < 36; k += 32) G[k] = B.g[k];
  __syncwarp();
  if (!zr_positive(Z, mask) || !chol_solve6(G, Q, -1.0, T, mask, drop))
    return block_stop(B, stt, cell, mask, CG_BLOCK_FAIL);
  for (int k = lane; k < 36; k += 32) {
    B.beta[k] = T[k];
    B.zr[k] = Z[k];
  }
}

// X += P alpha, R -= Q alpha (Q = K P) for the load cases of each live block,
// with ||r||^2 partials per load case ([sub-slot][6]) and, for the multigrid, the first
// smoothing sweep z0 = omega D^-1 r and the residual copy rm of the V-cycle.
// BT threads (256, or 64 where the cells are small: see bsub); a node's new
// residuals wait in shared memory for the 3x3 node-block sweep (registers kept
// for 768 threads per SM: 1024 measured slower).
template <int BT, typename TV, typename TP, typename TQ, typename TZ>
__global__ void __launch_bounds__(BT, 768 / BT)
k_bupdate(const CellDesc* cells, const NodeUnit* units, TV* __restrict__ x, TV* __restrict__ r,
          const TP* __restrict__ p, const TQ* __restrict__ q, const float* __restrict__ invd, TZ* __restrict__ z0,
          TZ* __restrict__ rm, double omega, const BlockCG* bst, double* __restrict__ part, long long ntot,
          const float* __restrict__ binv, int nsub) {
  griddep_sync();
  const SubUnit su = sub_unit(units, nsub);
  const CellDesc cd = cells[su.u.cell];
  const int mask = bst[cd.id].live ? bst[cd.id].mask : 0;
  __shared__ double al[36];
  __shared__ double rs[kNumRhs * 3][BT];
  if (threadIdx.x < 36) al[threadIdx.x] = bst[cd.id].alpha[threadIdx.x];
  __syncthreads();
  double v[kNumRhs];
#pragma unroll
  for (int j = 0; j < kNumRhs; ++j) v[j] = 0.0;
  if (mask) {
    for (long long n = su.begin + threadIdx.x; n < su.end; n += blockDim.x) {
      const long long g = cd.off + n;
#pragma unroll 1
      for (int c = 0; c < 3; ++c) {
        double pv[kNumRhs], qv[kNumRhs];
#pragma unroll
        for (int i = 0; i < kNumRhs; ++i) {
          const long long o = ((long long)i * 3 + c) * ntot + g;
          const bool in = mask >> i & 1;
          pv[i] = in ? (double)ld_val(p + o) : 0.0;
          qv[i] = in ? (double)ld_val(q + o) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kNumRhs; ++j) {
          if (!(mask >> j & 1)) continue;
          double dx = 0.0, dr = 0.0;
#pragma unroll
          for (int i = 0; i < kNumRhs; ++i) {
            dx += al[i * 6 + j] * pv[i];
            dr += al[i * 6 + j] * qv[i];
          }
          const long long o = ((long long)j * 3 + c) * ntot + g;
          const double rj = (double)ld_val(r + o) - dr;
          st_val(x + o, (double)ld_val(x + o) + dx);
          st_val(r + o, rj);
          if (rm) st_val(rm + o, rj);
          v[j] += rj * rj;
          rs[j * 3 + c][threadIdx.x] = rj;
        }
      }
      if (z0) {
        const double id = binv ? 0.0 : (double)invd[g];
#pragma unroll 1
        for (int j = 0; j < kNumRhs; ++j) {
          if (!(mask >> j & 1)) continue;
          double d[3] = {rs[j * 3][threadIdx.x], rs[j * 3 + 1][threadIdx.x], rs[j * 3 + 2][threadIdx.x]};
          jacobi_dir<double>(binv, g, id, d);
#pragma unroll
          for (int c = 0; c < 3; ++c) st_val(z0 + ((long long)j * 3 + c) * ntot + g, omega * d[c]);
        }
      }
    }
  }
  __shared__ double red[32 * kNumRhs];
  block_reduce<kNumRhs>(v, red);
  if (threadIdx.x == 0)
#pragma unroll
    for (int j = 0; j < kNumRhs; ++j) part[su.sub * kNumRhs + j] = v[j];
}

// P = Z + P beta for the load cases of each live block (first: P = Z).
template <int BT, typename TP, typename TZ>
__global__ void __launch_bounds__(BT, 1024 / BT)
k_bdir(const CellDesc* cells, const NodeUnit* units, TP* __restrict__ p, const TZ* __restrict__ z,
       const BlockCG* bst, long long ntot, int first, int nsub) {
  griddep_sync();
  const SubUnit su = sub_unit(units, nsub);
  const CellDesc cd = cells[su.u.cell];
  const int mask = bst[cd.id].live ? bst[cd.id].mask : 0;
  __shared__ double be[36];
  if (threadIdx.x < 36) be[threadIdx.x] = first ? 0.0 : bst[cd.id].beta[threadIdx.x];
  __syncthreads();
  if (!mask) return;
  const bool rd = !first;
  for (long long n = su.begin + threadIdx.x; n < su.end; n += blockDim.x) {
    const long long g = cd.off + n;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double pv[kNumRhs], zv[kNumRhs];
#pragma unroll
      for (int i = 0; i < kNumRhs; ++i) {
        const long long o = ((long long)i * 3 + c) * ntot + g;
        const bool in = mask >> i & 1;
        pv[i] = (rd && in) ? (double)ld_val(p + o) : 0.0;
        zv[i] = in ? (double)ld_val(z + o) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < kNumRhs; ++j) {
        if (!(mask >> j & 1)) continue;
        double pj = zv[j];
#pragma unroll
        for (int i = 0; i < kNumRhs; ++i) pj += be[i * 6 + j] * pv[i];
        st_val(p + ((long long)j * 3 + c) * ntot + g, pj);
      }
    }
  }
}

// One warp per (cell, rhs) in the finalisation kernels.
#define FIN_PROLOGUE                                                         \
  const int t = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5); \
  const bool lead = (threadIdx.x & 31) == 0;                                 \
  if (t >= ncells * kNumRhs) return;                                         \
  const int cell = t / kNumRhs, rhs = t % kNumRhs;                           \
  (void)cell;                                                                \
  (void)rhs;

// After k_cg_init: bnorm2, rz (Jacobi) / rr; decide which (cell, rhs) run.
// One thread per (cell, rhs).
// bn2 != nullptr (warm start): ||b||^2 per (cell, rhs), against which the
// residual of the starting x is measured; else the start is x = 0 and r = b.
__global__ void k_fin_init(CGState* stt, const int* slot_begin, const int* slot_end,
                           const double* part, int ncells, int jacobi, const double* bn2) {
  FIN_PROLOGUE
  CGState S = stt[t];
  if (!S.active) return;
  const double rr = sum_slots(part, slot_begin[cell], slot_end[cell], rhs, 2, 0);
  S.bnorm2 = bn2 ? bn2[t] : rr;
  S.rr = rr;
  S.rz = jacobi ? sum_slots(part, slot_begin[cell], slot_end[cell], rhs, 2, 1) : 0.0;
  S.iters = 0;
  S.rel = (S.bnorm2 > 0.0) ? sqrt(rr / S.bnorm2) : 0.0;
  S.best = S.rel;
  S.since = 0;
  if (!(S.bnorm2 > 0.0) || !(rr > 0.0) || S.rel < S.tol) { S.active = 0; S.status = CG_CONVERGED; }
  if (lead) stt[t] = S;
}

// rz for the multigrid preconditioner at start (z . r of the first V-cycle);
// if that is not positive, the pair starts with the Jacobi preconditioner.
// beta = 0 so that the following direction kernel sets p = z.
// part: z.r partials over slot range [zb, ze) of each cell (node units, or the
// stencil units of the sweep that computed them); part_init: the start
// partials over [slot_begin, slot_end).
__global__ void k_fin_rz(CGState* stt, const int* slot_begin, const int* slot_end,
                         const int* zb, const int* ze, const double* part, const double* part_init, int ncells) {
  FIN_PROLOGUE
  CGState S = stt[t];
  if (!S.active) return;
  const double rz_mg = sum_slots(part, zb[cell], ze[cell], rhs, 1, 0);
  const double rz_jac = sum_slots(part_init, slot_begin[cell], slot_end[cell], rhs, 2, 1);
  S.beta = 0.0;
  if (isfinite(rz_mg) && rz_mg > 0.0) {
    S.rz = rz_mg;
  } else {
    S.fallback = 1;
    S.rz = rz_jac;
  }
  if (lead) stt[t] = S;
}

// alpha = rz / (p . K p); breakdown if p.Kp <= 0 or not finite.
__global__ void k_fin_alpha(CGState* stt, const int* slot_begin, const int* slot_end,
                            const double* part, int ncells) {
  griddep_sync();
  FIN_PROLOGUE
  CGState S = stt[t];
  if (!S.active) return;
  const double pq = sum_slots(part, slot_begin[cell], slot_end[cell], rhs, 1, 0);
  S.pq = pq;
  if (!(pq > 0.0) || !isfinite(pq) || !isfinite(S.rz)) {
    S.alpha = 0.0;
    S.active = 0;
    S.status = CG_BREAKDOWN;
  } else {
    S.alpha = S.rz / pq;
  }
  if (lead) stt[t] = S;
}

// After the update (+ preconditioner): convergence test and beta.
// jacobi: rz_new from the update partials; else from the V-cycle partials.
// part_rz: z.r partials over slot range [zb, ze) of each cell.
__global__ void k_fin_beta(CGState* stt, const int* slot_begin, const int* slot_end,
                           const int* zb, const int* ze, const double* part_upd, const double* part_rz,
                           int ncells, int jacobi) {
  griddep_sync();
  FIN_PROLOGUE
  CGState S = stt[t];
  if (!S.active) return;
  const int b = slot_begin[cell], e = slot_end[cell];
  const double rr = sum_slots(part_upd, b, e, rhs, 2, 0);
  const double rz_jac = sum_slots(part_upd, b, e, rhs, 2, 1);
  const double rz_mg = jacobi ? rz_jac : sum_slots(part_rz, zb[cell], ze[cell], rhs, 1, 0);
  const double rzn = (jacobi || S.fallback) ? rz_jac : rz_mg;
  S.rr = rr;
  S.iters += 1;
  S.rel = sqrt(rr / S.bnorm2);
  if (S.rel < S.tol) {
    S.active = 0;
    S.status = CG_CONVERGED;
  } else if (S.iters >= S.max_iter) {
    S.active = 0;
    S.status = CG_MAXITER;
  } else if (S.outer && (S.rel < 0.5 * S.best ? (S.best = S.rel, S.since = 0, false)
                                               : ++S.since >= kInnerStallWindow)) {
    S.active = 0;   // inner solve at its arithmetic's floor: hand back to the outer step
    S.status = CG_MAXITER;
  } else if (!isfinite(rzn) || !(rzn > 0.0)) {
    if (!jacobi && !S.fallback && isfinite(rz_jac) && rz_jac > 0.0) {
      // the V-cycle is not positive definite for this field: restart the
      // search direction with the (always SPD) Jacobi preconditioner
      S.fallback = 1;
      S.beta = 0.0;
      S.rz = rz_jac;
    } else {
      S.active = 0;
      S.status = CG_BREAKDOWN;
    }
  } else {
    S.beta = rzn / S.rz;
    S.rz = rzn;
  }
  if (lead) stt[t] = S;
}

// ---------------------------------------------------------- multigrid ---
// Full-weighting restriction (transpose of trilinear prolongation):
// bc(I) = sum_{d in {-1,0,1}^3} prod_s (1 - |d_s|/2) rf(2I + d).  The weights of a
// fine node add up to 1, so a residual without net force stays one.
// xc != nullptr: also the coarse level's first damped-Jacobi sweep from a zero
// guess, xc = omega * invdc * bc (as stored), on the coarse cells that are
// smoothed there (child >= 0; the others are solved directly).
template <typename TF, typename TCo>
__global__ void k_restrict(const CellDesc* fine, const CellDesc* coarse, const NodeUnit* units,
                           const TF* __restrict__ rf, TCo* __restrict__ bc, TCo* __restrict__ xc,
                           const float* __restrict__ invdc, double omega, const CGState* stt, long long ntf,
                           long long ntc, const float* __restrict__ binvc) {
  griddep_sync();
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cc = coarse[u.cell], cf = fine[cc.parent];
  if (stt && !stt[cc.id * kNumRhs + rhs].active) return;
  const bool smooth = xc != nullptr && cc.child >= 0;
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    int i, j, k;
    node_ijk(n, cc.ny, cc.nz, i, j, k);
    double acc[3] = {0, 0, 0};
    for (int dx = -1; dx <= 1; ++dx) {
      const int fi = wrap(2 * i + dx, cf.nx);
      const double wx = dx ? 0.5 : 1.0;
      for (int dy = -1; dy <= 1; ++dy) {
        const int fj = wrap(2 * j + dy, cf.ny);
        const double wy = wx * (dy ? 0.5 : 1.0);
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz) {
          const int fk = wrap(2 * k + dz, cf.nz);
          const double w = wy * (dz ? 0.5 : 1.0);
          const long long g = cf.off + lin(fi, fj, fk, cf.ny, cf.nz);
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[c] += w * (double)ld_val(rf + ((long long)rhs * 3 + c) * ntf + g);
        }
      }
    }
    const long long g = cc.off + n;
#pragma unroll
    for (int c = 0; c < 3; ++c) st_val(bc + ((long long)rhs * 3 + c) * ntc + g, acc[c]);
    if (smooth) {
      double bs[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) bs[c] = (double)static_cast<TCo>(acc[c]);   // b as stored
      if (binvc) {
        jacobi_dir<double>(binvc, g, 0.0, bs);
      } else {
        const double id = (double)invdc[g];
#pragma unroll
        for (int c = 0; c < 3; ++c) bs[c] *= id;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) st_val(xc + ((long long)rhs * 3 + c) * ntc + g, omega * bs[c]);
    }
  }
}

// Trilinear prolongation and correction: xf(n) += sum_I w(n,I) ec(I).
// Each thread corrects the two fine nodes 2m and 2m+1 of a z row, which share
// the coarse z nodes m and m+1 (fine 2m = coarse m; fine 2m+1 = mean of m, m+1);
// x and y weights are uniform along the row.
// (All multigrid levels have even fine extents, so pairs never straddle rows.)
template <typename TF, typename TCo>
__global__ void k_prolong_add(const CellDesc* __restrict__ fine, const CellDesc* __restrict__ coarse,
                              const NodeUnit* __restrict__ units, TF* __restrict__ xf,
                              const TCo* __restrict__ ec, const CGState* stt, long long ntf, long long ntc) {
  griddep_sync();
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cf = fine[u.cell], cc = coarse[fine[u.cell].child];
  if (stt && !stt[cf.id * kNumRhs + rhs].active) return;
  const long long pb = (u.begin + 1) >> 1, pe = (u.end + 1) >> 1;   // node pairs of the unit
  for (long long pr = pb + threadIdx.x; pr < pe; pr += blockDim.x) {
    const long long n = 2 * pr;
    int i, j, k;
    node_ijk(n, cf.ny, cf.nz, i, j, k);   // k even
    const int ci0 = i >> 1, cj0 = j >> 1, m = k >> 1;
    const int ci1 = wrap(ci0 + (i & 1), cc.nx), cj1 = wrap(cj0 + (j & 1), cc.ny);
    const int m1 = wrap(m + 1, cc.nz);
    const double wx = (i & 1) ? 0.5 : 1.0, wy = (j & 1) ? 0.5 : 1.0;
    double a0[3] = {0, 0, 0}, a1[3] = {0, 0, 0};   // at fine k = 2m and 2m+1
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
      if (ax == 1 && !(i & 1)) break;
      const int ci = ax ? ci1 : ci0;
#pragma unroll
      for (int ay = 0; ay < 2; ++ay) {
        if (ay == 1 && !(j & 1)) break;
        const int cj = ay ? cj1 : cj0;
        const double w = wx * wy;
        const long long g0 = cc.off + lin(ci, cj, m, cc.ny, cc.nz);
        const long long g1 = cc.off + lin(ci, cj, m1, cc.ny, cc.nz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double e0 = (double)ld_val(ec + ((long long)rhs * 3 + c) * ntc + g0);
          const double e1 = (double)ld_val(ec + ((long long)rhs * 3 + c) * ntc + g1);
          a0[c] += w * e0;
          a1[c] += w * 0.5 * (e0 + e1);
        }
      }
    }
    const bool two = n + 1 < u.end;
    TF* px = xf + (long long)rhs * 3 * ntf + cf.off + n;
    LdT<TF> x0[3], x1[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {   // all before the first store
      x0[c] = ld_val(px + c * ntf);
      x1[c] = two ? ld_val(px + c * ntf + 1) : (LdT<TF>)0;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      st_val(px + c * ntf, (double)x0[c] + a0[c]);
      if (two) st_val(px + c * ntf + 1, (double)x1[c] + a1[c]);
    }
  }
}

// z = omega * invd * b  (first damped-Jacobi sweep from a zero start); with
// bcopy != nullptr also b converted to TX.
template <typename TB, typename TX>
__global__ void k_jacobi0(const CellDesc* cells, const NodeUnit* units, const TB* __restrict__ b, TX* __restrict__ x,
                          TX* __restrict__ bcopy, const float* __restrict__ invd, double omega, const CGState* stt,
                          long long ntot, const float* __restrict__ binv) {
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  if (stt && !stt[cd.id * kNumRhs + rhs].active) return;
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x) {
    const long long g = cd.off + n;
    double bv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long o = ((long long)rhs * 3 + c) * ntot + g;
      bv[c] = (double)ld_val(b + o);
      if (bcopy) st_val(bcopy + o, bv[c]);
    }
    if (binv) {
      jacobi_dir<double>(binv, g, 0.0, bv);
    } else {
      const double id = (double)invd[g];
#pragma unroll
      for (int c = 0; c < 3; ++c) bv[c] *= id;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) st_val(x + ((long long)rhs * 3 + c) * ntot + g, omega * bv[c]);
  }
}

// Dense coarse operator, FP64: A = sum_e kc_e K0(1) scattered to the periodic
// DOFs, with the rows and columns of one node zero: the inversion leaves the
// unknowns of zero pivots out, so that node stays put and the solution of a
// right-hand side without net force is A's up to a translation, which no residual
// sees.  It is the node with the largest diagonal (the first of them): it takes
// up the net force that rounding leaves, and a node among soft voxels would yield
// to it (40 iterations instead of 2 on a frame of 1 in 1e-9).  (The mean
// diagonal times the projector on the translations, added to A instead, couples
// every pair of nodes at the stiff voxels' scale: soft voxels lose their digits --
// contrasts of 1e12 made the preconditioner indefinite -- and the unknowns of
// voxels without stiffness no longer drop out.)  diag[node] is A's diagonal, the
// same for the three components.  A is m x m, m = 3 * nodes.  One 96-thread CTA
// per (node, cell) owns the node's three rows, gathers its 8 voxels (one after
// another: a corner pair of two voxels may meet in the same entry) in shared
// memory and writes the rows once.  A CTA per cell that scattered voxel after
// voxel took 66 us at 64 nodes and 162 us at 105; a row owner needs 8 steps
// whatever the size (~4 us).
// Cells whose sweep takes an odd number of block steps start in `work`, so
// that the last step of every cell writes A (k_coarse_sweep).
constexpr int kSweep = 32;   // block size of the coarse inversion
template <typename TC>
__global__ void __launch_bounds__(96) k_coarse_assemble(const CellDesc* cells, const int* list, const TC* kc,
                                                        const double* K0, double* A, double* work,
                                                        const long long* aoff, double* diag) {
  extern __shared__ double rows[];   // [3][m]
  const CellDesc cd = cells[list[blockIdx.x]];
  const int nn = cd.nx * cd.ny * cd.nz, m = 3 * nn, n = blockIdx.y;
  if (n >= nn) return;
  double* M = ((m + kSweep - 1) / kSweep % 2 ? work : A) + aoff[blockIdx.x];
  // the fixed node (every CTA of the cell finds the same one)
  double mx = -1.0;
  int pin = 0;
  for (int q = threadIdx.x; q < nn; q += blockDim.x) {
    int i, j, k;
    node_ijk(q, cd.ny, cd.nz, i, j, k);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 8; ++a)
      s += (double)kc[cd.off + lin(wrap(i - (a >> 2 & 1), cd.nx), wrap(j - (a >> 1 & 1), cd.ny),
                                   wrap(k - (a & 1), cd.nz), cd.ny, cd.nz)];
    if (s > mx) {
      mx = s;
      pin = q;
    }
  }
  auto take = [&](double v, int q) {   // the larger one, the first of equals
    if (v > mx || (v == mx && q < pin)) {
      mx = v;
      pin = q;
    }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    take(__shfl_xor_sync(0xffffffffu, mx, o), __shfl_xor_sync(0xffffffffu, pin, o));
  __shared__ double best[3];
  __shared__ int node[3];
  if (threadIdx.x % 32 == 0) {
    best[threadIdx.x / 32] = mx;
    node[threadIdx.x / 32] = pin;
  }
  for (int t = threadIdx.x; t < 3 * m; t += blockDim.x) rows[t] = 0.0;
  __syncthreads();
  for (int w = 0; w < 3; ++w) take(best[w], node[w]);
  int i, j, k;
  node_ijk(n, cd.ny, cd.nz, i, j, k);
  const int t = threadIdx.x, aq = t / 9, cp = t / 3 % 3, cq = t % 3;   // 72 of the threads: corner, row, column
  for (int ap = 0; ap < 8; ++ap) {
    if (t < 72) {
      const int ei = wrap(i - (ap >> 2 & 1), cd.nx), ej = wrap(j - (ap >> 1 & 1), cd.ny),
                ek = wrap(k - (ap & 1), cd.nz);
      const int nq = (int)lin(wrap(ei + (aq >> 2 & 1), cd.nx), wrap(ej + (aq >> 1 & 1), cd.ny),
                              wrap(ek + (aq & 1), cd.nz), cd.ny, cd.nz);
      rows[cp * m + 3 * nq + cq] +=
          (double)kc[cd.off + lin(ei, ej, ek, cd.ny, cd.nz)] * K0[(3 * ap + cp) * 24 + 3 * aq + cq];
    }
    __syncthreads();
  }
  if (t == 0) diag[cd.off + n] = n == pin ? 0.0 : rows[3 * n];
  for (int q = t; q < 3 * m; q += blockDim.x)
    M[(long long)3 * n * m + q] = n == pin || q % m / 3 == pin ? 0.0 : rows[q];
}

// Explicit inverse of every cell's SPD coarse matrix by symmetric block sweeps
// (the sweep operator of regression, Goodnight, Am. Stat. 33, 1979, with 32 x
// 32 blocks): step k replaces, with D = A_kk^-1,
//   A_kk <- -D,   A_ik <- A_ik D,   A_ij <- A_ij - A_ik D A_kj,
// and after all block steps the matrix is -A^-1 (the last step stores the
// negative).  The Cholesky factorisation and column solves that this replaces
// ran on one CTA per cell, a chain of m pivots each with a pass over the
// trailing matrix: 1.60 ms at m = 192, 26.3 ms at 315, 150 ms at 600.  Here a
// step is one launch whose CTAs (one per lower-triangle tile and cell) each
// invert the 32 x 32 pivot block themselves (32 short pivots in registers,
// the same pivots as Cholesky's) and do the rank-32 update of their tile, so
// the chain is ceil(m / 32) launches of ~16 us.  Steps go from one buffer to the other:
// tiles read the pivot row and column of the previous step while the same
// launch rewrites them.  Tiles i > j are stored twice, so the inverse is
// symmetric to the last bit, which the V-cycle needs to be a symmetric
// preconditioner.  A pivot that is zero up to rounding -- not above kPivotFloor
// times A's diagonal there: the fixed node, voxels without stiffness, parts held by
// nothing else -- leaves its unknown out: its row and column of the inverse are
// zero.
constexpr double kPivotFloor = 32 * 1.1102230246251565e-16;
__global__ void __launch_bounds__(256) k_coarse_sweep(const CellDesc* cells, const int* list, double* A, double* work,
                                                      const long long* aoff, const double* diag, int step) {
  const CellDesc cd = cells[list[blockIdx.x]];
  const int m = 3 * cd.nx * cd.ny * cd.nz, T = (m + kSweep - 1) / kSweep;
  if (step >= T) return;
  // lower-triangle tile (ti, tj) of this CTA
  int ti = (int)((sqrtf(8.f * blockIdx.y + 1.f) - 1.f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.y) ++ti;
  while (ti * (ti + 1) / 2 > (int)blockIdx.y) --ti;
  const int tj = (int)blockIdx.y - ti * (ti + 1) / 2;
  if (ti >= T) return;
  const bool in_work = (T - step) % 2 != 0;
  const double* src = (in_work ? work : A) + aoff[blockIdx.x];
  double* dst = (in_work ? A : work) + aoff[blockIdx.x];
  __shared__ double D[kSweep][kSweep + 1], P[kSweep][kSweep + 1], Q[kSweep][kSweep + 1], U[kSweep][kSweep + 1];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;   // tile column, first of 4 rows (stride 8)
  auto at = [&](int bi, int bj, int r) -> double {   // entry (r, x) of tile (bi, bj), the identity outside
    const int gi = bi * kSweep + r, gj = bj * kSweep + x;
    return gi < m && gj < m ? src[(long long)gi * m + gj] : (bi == bj && r == x ? 1.0 : 0.0);
  };
  double a[4], v[4];
  __shared__ double prow[2][kSweep], pcol[2][kSweep];   // pivot row and column, of this pivot and the next
  __shared__ double least[kSweep];   // pivots up to here are zero
  const int gp = step * kSweep + x;
  const double dg = y == 0 && gp < m ? diag[cd.off + gp / 3] : 0.0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = y + 8 * q;
    v[q] = at(step, step, r);
    P[r][x] = at(ti, step, r);      // A_ik
    Q[r][x] = at(tj, step, r);      // A_jk = A_kj^T
    a[q] = at(ti, tj, r);
    if (r == 0) prow[0][x] = v[q];
    if (x == 0) pcol[0][r] = v[q];
  }
  if (y == 0) least[x] = kPivotFloor * dg;
  // v <- -A_kk^-1: scalar sweeps, one pivot at a time, in registers; a barrier
  // per pivot passes the next pivot's row and column on
  for (int p = 0; p < kSweep; ++p) {
    __syncthreads();
    const double* row = prow[p & 1];
    const double* col = pcol[p & 1];
    const double piv = row[p], cx = row[x];
    const double d = piv > least[p] ? 1.0 / piv : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = y + 8 * q;
      const double cr = col[r];
      v[q] = r == p ? (x == p ? -d : cx * d) : (x == p ? cr * d : v[q] - cr * d * cx);
      if (r == p + 1) prow[(p + 1) & 1][x] = v[q];
      if (x == p + 1) pcol[(p + 1) & 1][r] = v[q];
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) D[y + 8 * q][x] = v[q];
  __syncthreads();
  // U = A_ik D (D holds -A_kk^-1)
  double u[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int p = 0; p < kSweep; ++p) {
    const double dx = D[p][x];
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] -= P[y + 8 * q][p] * dx;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) U[y + 8 * q][x] = u[q];
  __syncthreads();
  const bool krow = ti == step && tj != step;   // tile of the pivot row: (A_jk D)^T
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = krow ? 0.0 : a[q];
#pragma unroll 8
  for (int p = 0; p < kSweep; ++p) {
    const double qx = Q[x][p];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] -= (krow ? D[p][y + 8 * q] : U[y + 8 * q][p]) * qx;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = y + 8 * q;
    if (ti == step && tj == step) v[q] = r >= x ? D[r][x] : D[x][r];   // -D
    else if (tj == step) v[q] = u[q];                                  // A_ik D
    else v[q] = a[q];
    if (step == T - 1) v[q] = -v[q];
  }
  __syncthreads();   // P is free: the tile on its way to the mirrored store
#pragma unroll
  for (int q = 0; q < 4; ++q) P[y + 8 * q][x] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = y + 8 * q;
    const int gi = ti * kSweep + r, gj = tj * kSweep + x;
    if (gi < m && gj < m && gi >= gj) dst[(long long)gi * m + gj] = P[r][x];
    const int hi = tj * kSweep + r, hj = ti * kSweep + x;   // mirrored entry
    if (hi < m && hj < m && hj > hi) dst[(long long)hi * m + hj] = P[x][r];
  }
}

// Coarse solve e = A^{-1} b for one (cell, rhs) per CTA (A^{-1} symmetric).
template <typename TB, typename TX>
__global__ void k_coarse_solve(const CellDesc* cells, const int* list, const double* Ainv,
                               const long long* aoff, const TB* b, TX* x, const CGState* stt,
                               long long ntot) {
  griddep_sync();
  const int cell = list[blockIdx.x], rhs = blockIdx.y;
  const CellDesc cd = cells[cell];
  if (stt && !stt[cd.id * kNumRhs + rhs].active) return;
  const int nn = cd.nx * cd.ny * cd.nz, m = 3 * nn;
  extern __shared__ double sb[];
  for (int t = threadIdx.x; t < m; t += blockDim.x) {
    const int n = t / 3, c = t % 3;
    sb[t] = (double)ld_val(b + ((long long)rhs * 3 + c) * ntot + cd.off + n);
  }
  __syncthreads();
  const double* M = Ainv + aoff[blockIdx.x];
  // one warp per row t (A^{-1} is symmetric: row t is read contiguously), the
  // row's dot product split over the lanes and summed by shuffles
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int t = warp; t < m; t += nw) {
    const double* Mr = M + (long long)t * m;
    double s = 0.0;
    for (int j = lane; j < m; j += 32) s += Mr[j] * sb[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const int n = t / 3, c = t % 3;
      st_val(x + ((long long)rhs * 3 + c) * ntot + cd.off + n, s);
    }
  }
}

// ------------------------------------------------------- energy kernels ---
// Per voxel: u^I = ue0^I(h) + chi^I (6 load cases) and the 21 pairs
// s_IJ = u^I . K0(1) u^J.  Modes:
//   C partials:   sum_e kc_e s_IJ       (-> C^H = sum / (|Y|))     [sub-slot][22]
//   dC/drho:      out[t][e] = c'(rho_e) h s_t / |Y|
//   dL/drho:      out[e] = c'(rho_e) h sum_t W_t s_t / |Y|
enum EnergyMode : int { EN_C = 0, EN_DCDRHO = 1, EN_GRAD = 2 };

// K0 in the 18 strain modes of the voxel, in which it is diagonal:
// s_IJ = sum_k w_k phi_k^I phi_k^J.  The modes are the Hadamard coefficients
// that carry energy, combined to the eigenvectors of Kh's 3x3 and 2x2 blocks
// (a block d I + o J has the sum with weight (d + 2 o) / 3 and two differences
// with (d - o) / 2 and (d - o) / 6, or (d +- o) / 2 for a pair; the shear pairs
// have the sum only).  The macro strains reach the first six modes.
struct EnergyModes {
  double nsum, nd1, nd2, shear, msum, md1, md2, psum, pdif, cube;   // weights
  double m0[kNumRhs][6];   // unit macro strains (h = 1): normal sum, differences 1 and 2, shear xz, yz, xy
};
inline EnergyModes energy_modes(const HadK& k, const ElemConst& ec) {
  EnergyModes m{};
  m.nsum = (k.Bd + 2 * k.Bo) / 3;
  m.nd1 = (k.Bd - k.Bo) / 2;
  m.nd2 = (k.Bd - k.Bo) / 6;
  m.shear = k.A;
  m.msum = (k.D1 + 2 * k.O1) / 3;
  m.md1 = (k.D1 - k.O1) / 2;
  m.md2 = (k.D1 - k.O1) / 6;
  m.psum = (k.D2 + k.O2) / 2;
  m.pdif = (k.D2 - k.O2) / 2;
  m.cube = k.G;
  for (int I = 0; I < kNumRhs; ++I) {
    const auto& u = ec.uhat0[I];
    const double n0 = u[0][4], n1 = u[1][2], n2 = u[2][1];
    m.m0[I][0] = n0 + n1 + n2;
    m.m0[I][1] = n0 - n1;
    m.m0[I][2] = n0 + n1 - 2 * n2;
    m.m0[I][3] = u[0][1] + u[2][4];
    m.m0[I][4] = u[1][1] + u[2][2];
    m.m0[I][5] = u[0][2] + u[1][4];
  }
  return m;
}

struct EnergyArgs {
  const CellDesc* cells;
  const NodeUnit* units;
  const double* chi;      // [6][3][ntot] FP64
  const double* kc64;     // c_e * h
  const double* rho;      // rho actually used (clamped)
  const double* W;        // [cell][21] symmetric weights for EN_GRAD
  double* part;           // EN_C: [sub-slot][22]
  double* out;            // EN_DCDRHO: [21][ntot]; EN_GRAD: [ntot]
  long long ntot;
  int nsub;               // CTAs per node unit
  EnergyModes m;
  MatLaw law;
};

// 18 modes of one load case of a voxel: chi = its x component (components ntot
// apart), nd = the 8 corner nodes, m0 = the macro strain's modes.
__device__ __forceinline__ void energy_phi(const double* __restrict__ chi, long long ntot, const unsigned (&nd)[8],
                                           double h, const double (&m0)[6], double (&f)[18]) {
  double w[3][8];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int a8 = 0; a8 < 8; ++a8) w[c][a8] = chi[c * ntot + nd[a8]];
    fwht8_fwd(w[c]);
  }
  f[0] = w[0][4] + w[1][2] + w[2][1] + h * m0[0];
  f[1] = w[0][4] - w[1][2] + h * m0[1];
  f[2] = w[0][4] + w[1][2] - 2.0 * w[2][1] + h * m0[2];
  f[3] = w[0][1] + w[2][4] + h * m0[3];
  f[4] = w[1][1] + w[2][2] + h * m0[4];
  f[5] = w[0][2] + w[1][4] + h * m0[5];
  f[6] = w[0][3] + w[1][5] + w[2][6];
  f[7] = w[0][3] - w[1][5];
  f[8] = w[0][3] + w[1][5] - 2.0 * w[2][6];
  f[9] = w[1][3] + w[0][5];
  f[10] = w[1][3] - w[0][5];
  f[11] = w[2][3] + w[0][6];
  f[12] = w[2][3] - w[0][6];
  f[13] = w[2][5] + w[1][6];
  f[14] = w[2][5] - w[1][6];
  f[15] = w[0][7];
  f[16] = w[1][7];
  f[17] = w[2][7];
}

// Two threads per voxel: a warp's lower half holds the modes of load cases 0-2
// of 16 voxels, its upper half those of cases 3-5 of the same voxels; mode by
// mode they exchange their three values and each adds up 12 of the pairs
// (its own 6; three across; the three pairs (i, i + 3) in both halves).
// One thread per voxel needed the 144 coefficients of all cases at once and
// spilled; this takes 108 registers of modes and one pass over the fields.
// Bound by its instruction mix at 12 warps per SM: per 16 voxels ~525 FP64
// operations, 72 loads and 108 shuffles a lane, and prefetching the next
// fields changes nothing.  96^3: 206 -> 137 us (table) and 140 (gradient),
// 0.35 of measured HBM for the table; 24^3 both 46 -> 14 us (more CTAs).
// Pair p of half h is entry kEnergyPair[h][p] of the lower triangle.
__device__ constexpr signed char kEnergyPair[2][12] = {
    {0, 1, 3, 2, 4, 5, /* (0,4) (0,5) (1,5) */ 10, 15, 16, /* (0,3) (1,4) (2,5) */ 6, 11, 17},
    {9, 13, 18, 14, 19, 20, /* (3,1) (3,2) (4,2) */ 7, 8, 12, /* as in half 0 */ 6, 11, 17}};

template <int MODE>
__global__ void __launch_bounds__(128, 3) k_energy(EnergyArgs a) {
  const SubUnit su = sub_unit(a.units, a.nsub);
  const CellDesc cd = a.cells[su.u.cell];
  const double vol = (double)cd.nx * cd.ny * cd.nz * cd.h * cd.h * cd.h;
  const int half = (threadIdx.x >> 4) & 1;
  const int lane16 = threadIdx.x & 15, warp = threadIdx.x >> 5;
  const double* chi = a.chi + (long long)half * 9 * a.ntot + cd.off;
  double acc[12], rsum = 0.0;
#pragma unroll
  for (int p = 0; p < 12; ++p) acc[p] = 0.0;
  for (long long e0 = su.begin + warp * 16; e0 < su.end; e0 += 64) {
    const bool in = e0 + lane16 < su.end;
    const long long e = in ? e0 + lane16 : su.end - 1;   // idle lanes repeat the last voxel, unweighted
    int i, j, k;
    node_ijk(e, cd.ny, cd.nz, i, j, k);
    unsigned nd[8];
#pragma unroll
    for (int a8 = 0; a8 < 8; ++a8)
      nd[a8] = (unsigned)lin(wrap(i + ((a8 >> 2) & 1), cd.nx), wrap(j + ((a8 >> 1) & 1), cd.ny),
                             wrap(k + (a8 & 1), cd.nz), cd.ny, cd.nz);
    double f[3][18];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double m0[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) m0[t] = half ? a.m.m0[q + 3][t] : a.m.m0[q][t];
      energy_phi(chi + (long long)q * 3 * a.ntot, a.ntot, nd, cd.h, m0, f[q]);
    }
    double s[12];
#pragma unroll
    for (int p = 0; p < 12; ++p) s[p] = 0.0;
#pragma unroll
    for (int t = 0; t < 18; ++t) {
      const double w = t == 0 ? a.m.nsum : t == 1 ? a.m.nd1 : t == 2 ? a.m.nd2 : t < 6 ? a.m.shear : t == 6 ? a.m.msum
                       : t == 7 ? a.m.md1 : t == 8 ? a.m.md2 : t < 15 ? (t % 2 ? a.m.psum : a.m.pdif) : a.m.cube;
      const double x0 = f[0][t], x1 = f[1][t], x2 = f[2][t];
      const double y0 = __shfl_xor_sync(0xffffffffu, x0, 16), y1 = __shfl_xor_sync(0xffffffffu, x1, 16),
                   y2 = __shfl_xor_sync(0xffffffffu, x2, 16);
      const double w0 = w * x0, w1 = w * x1, w2 = w * x2;
      s[0] += w0 * x0;
      s[1] += w0 * x1;
      s[2] += w0 * x2;
      s[3] += w1 * x1;
      s[4] += w1 * x2;
      s[5] += w2 * x2;
      s[6] += w0 * y1;
      s[7] += w0 * y2;
      s[8] += w1 * y2;
      s[9] += w0 * y0;
      s[10] += w1 * y1;
      s[11] += w2 * y2;
    }
    if (MODE == EN_C) {
      const double ke = in ? a.kc64[cd.off + e] : 0.0;
#pragma unroll
      for (int p = 0; p < 12; ++p) acc[p] += ke * s[p];
      if (in) rsum += a.rho[cd.off + e];
    } else {
      const double dc = law_dcoef(a.law, a.rho[cd.off + e]) * cd.h / vol;
      if (MODE == EN_DCDRHO) {
        if (in) {
#pragma unroll
          for (int p = 0; p < 12; ++p)
            if (p < 9 || half == 0) a.out[(long long)kEnergyPair[half][p] * a.ntot + cd.off + e] = dc * s[p];
        }
      } else {
        double g = 0.0;
#pragma unroll
        for (int p = 0; p < 12; ++p)
          if (p < 9 || half == 0) g += a.W[cd.id * 21 + kEnergyPair[half][p]] * s[p];
        g += __shfl_xor_sync(0xffffffffu, g, 16);
        if (in && half == 0) a.out[cd.off + e] = dc * g;
      }
    }
  }
  if (MODE == EN_C) {   // over each half warp, then over the warps, in a fixed order
    __shared__ double red[4][2][13];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
#pragma unroll
      for (int p = 0; p < 12; ++p) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], o);
      rsum += __shfl_xor_sync(0xffffffffu, rsum, o);
    }
    if (lane16 == 0) {
#pragma unroll
      for (int p = 0; p < 12; ++p) red[warp][half][p] = acc[p];
      red[warp][half][12] = rsum;
    }
    __syncthreads();
    if (threadIdx.x < 25) {   // 0-11: half 0's pairs and the density; 12-20: half 1's
      const int t = threadIdx.x, hf = t >= 13, p = t < 13 ? t : t - 13;
      if (!hf || p < 9) {
        double v = 0.0;
        for (int w = 0; w < 4; ++w) v += red[w][hf][p];
        a.part[su.sub * 22 + (p == 12 ? 21 : kEnergyPair[hf][p])] = v;
      }
    }
  }
}

// C^H of each cell from its energy partials, one warp per (cell, pair), lanes
// over the sub-slots and a shuffle tree (fixed order).  One thread per pair
// chased the slots one load after another: 564 us at 192^3.
__global__ void k_energy_fin(const CellDesc* cells, const int* slot_begin, const int* slot_end,
                             const double* part, double* C, double* dens, int ncells, int nsub) {
  const int t = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (t >= ncells * 22) return;
  const int cell = t / 22, q = t % 22;
  const CellDesc cd = cells[cell];
  const double nvx = (double)cd.nx * cd.ny * cd.nz;
  const double vol = nvx * cd.h * cd.h * cd.h;
  double s = 0.0;
  const long long end = (long long)slot_end[cell] * nsub;
#pragma unroll 4
  for (long long sl = (long long)slot_begin[cell] * nsub + lane; sl < end; sl += 32) s += part[sl * 22 + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane != 0) return;
  if (q == 21) {
    dens[cell] = s / nvx;
    return;
  }
  int I = 0;
  while ((I + 1) * (I + 2) / 2 <= q) ++I;
  const int J = q - I * (I + 1) / 2;
  C[cell * 36 + I * 6 + J] = s / vol;
  C[cell * 36 + J * 6 + I] = s / vol;
}

// ------------------------------------------------------- misc vector ops ---
// dst = src (cast), per load case, over all nodes of the units.
template <typename TD, typename TS>
__global__ void k_copy(const CellDesc* cells, const NodeUnit* units, TD* __restrict__ dst, const TS* __restrict__ src,
                       const CGState* stt, long long ntot) {
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  if (stt && !stt[cd.id * kNumRhs + rhs].active) return;
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long o = ((long long)rhs * 3 + c) * ntot + cd.off + n;
      st_val(dst + o, (double)ld_val(src + o));
    }
}

// Defect correction: x64 += d / scale (d from the inner solve).
template <typename TD>
__global__ void k_dc_accum(const CellDesc* cells, const NodeUnit* units, double* __restrict__ x64, const TD* __restrict__ d,
                           const CGState* stt, long long ntot) {
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  const CGState S = stt[cd.id * kNumRhs + rhs];
  if (!S.outer) return;
  const double inv = 1.0 / S.scale;
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long o = ((long long)rhs * 3 + c) * ntot + cd.off + n;
      x64[o] += inv * (double)ld_val(d + o);
    }
}


// Partial a.b per (unit, rhs) into part[slot][6] (stride 1).
template <typename TA, typename TB2>
__global__ void k_dot(const CellDesc* cells, const NodeUnit* units, const TA* __restrict__ a, const TB2* __restrict__ b,
                      const CGState* stt, double* __restrict__ part, long long ntot) {
  griddep_sync();
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  double acc[1] = {0.0};
  if (!stt || stt[cd.id * kNumRhs + rhs].active) {
    #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const long long o = ((long long)rhs * 3 + c) * ntot + cd.off + n;
        acc[0] += (double)ld_val(a + o) * (double)ld_val(b + o);
      }
  }
  __shared__ double red[32];
  block_reduce<1>(acc, red);
  if (threadIdx.x == 0) part[(long long)u.slot * kNumRhs + rhs] = acc[0];
}

// Partial ||v||^2 per (unit, rhs) into part[slot][6] (stride 1).
template <typename TV>
__global__ void k_norm2(const CellDesc* cells, const NodeUnit* units, const TV* __restrict__ v, double* __restrict__ part,
                        long long ntot) {
  const NodeUnit u = units[blockIdx.x];
  const int rhs = blockIdx.y;
  const CellDesc cd = cells[u.cell];
  double acc[1] = {0.0};
  #pragma unroll 4
  for (long long n = u.begin + threadIdx.x; n < u.end; n += blockDim.x)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double x = (double)ld_val(v + ((long long)rhs * 3 + c) * ntot + cd.off + n);
      acc[0] += x * x;
    }
  __shared__ double red[32];
  block_reduce<1>(acc, red);
  if (threadIdx.x == 0) part[(long long)u.slot * kNumRhs + rhs] = acc[0];
}

// Condition of the CUDA-graph WHILE node around the captured CG iterations
// (one CTA): another pass of `chunk` iterations while some listed cell still
// iterates, the iteration budget `limit` is not spent, and -- for a batch --
// more than half of the `listed` cells still iterate (otherwise the host
// compacts the unit lists to the live cells and relaunches).  loop[0] counts
// the iterations run in this solve, so the loop always ends.
__global__ void k_while_cond(cudaGraphConditionalHandle h, const CGState* stt, int ncells,
                             int listed, int* loop, int chunk, int limit) {
  griddep_sync();
  __shared__ int alive;
  if (threadIdx.x == 0) alive = 0;
  __syncthreads();
  int mine = 0;
  for (int c = threadIdx.x; c < ncells; c += blockDim.x) {
    bool a = false;
#pragma unroll
    for (int r = 0; r < kNumRhs; ++r) a = a || stt[c * kNumRhs + r].active != 0;
    mine += a ? 1 : 0;
  }
  if (mine) atomicAdd(&alive, mine);   // integer count: exact in any order
  __syncthreads();
  if (threadIdx.x == 0) {
    const int done = loop[0] + chunk;
    loop[0] = done;
    const bool more = alive > 0 && done <= limit && !(ncells > 1 && 2 * alive <= listed);
    cudaGraphSetConditional(h, more ? 1u : 0u);
  }
}

// Field chain rule of fast_fem FEM3DFun::df (fast_fem/FEM3DFun.cpp:252-266)
// for piecewise-constant fields: every voxel belongs to one field parameter
// with weight 1, so grad[p] = sum over the voxels of p of (dL/drho_e + c).
// One warp per parameter, its voxels in a fixed order (CSR built on the host):
// deterministic, no atomics.
__global__ void k_param_sum(const int* __restrict__ ptr, const int* __restrict__ vox,
                            const double* __restrict__ dLdrho, double c, double* __restrict__ out, int nparam) {
  const int p = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= nparam) return;
  double s = 0.0;
  for (int q = ptr[p] + lane; q < ptr[p + 1]; q += 32) s += dLdrho[vox[q]] + c;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[p] = s;
}


// Net force over the sum of the weights per (cell, load case, component), from
// k_rhs's sums.
__global__ void k_rhs_mean(const int* slot_begin, const int* slot_end, const double* part, const double* wpart,
                           double* mean, int ncells) {
  FIN_PROLOGUE
  const double w = sum_slots(wpart, slot_begin[cell], slot_end[cell], 0, 2, 0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double v = sum_slots(part, slot_begin[cell], slot_end[cell], rhs, 3, c);
    if (lead) mean[t * 3 + c] = w > 0.0 ? v / w : 0.0;
  }
}

__global__ void k_sum_slots(const int* slot_begin, const int* slot_end, const double* part, double* out,
                            int ncells) {
  FIN_PROLOGUE
  const double v = sum_slots(part, slot_begin[cell], slot_end[cell], rhs, 1, 0);
  if (lead) out[t] = v;
}

// Full-cell displacement on (nx+1)(ny+1)(nz+1) nodes for load case I: periodic
// chi (with node 0 at zero) plus the macro-strain affine field, the jump
// eps (X - X0) on the + faces included (fast_fem/FEM3DFun.cpp:31-56
// copyPeriodicU).  Layout [node][3].
__global__ void k_full_field(const CellDesc* cells, int cell, const double* chi, int I, double* out,
                             long long ntot) {
  const CellDesc cd = cells[cell];
  const int Nx = cd.nx + 1, Ny = cd.ny + 1, Nz = cd.nz + 1;
  const long long total = (long long)Nx * Ny * Nz;
  double eps[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  if (I < 3) eps[I][I] = 1.0;
  if (I == 3) eps[1][2] = eps[2][1] = 0.5;
  if (I == 4) eps[0][2] = eps[2][0] = 0.5;
  if (I == 5) eps[0][1] = eps[1][0] = 0.5;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    node_ijk(t, Ny, Nz, i, j, k);
    const long long n0 = cd.off + lin(i % cd.nx, j % cd.ny, k % cd.nz, cd.ny, cd.nz);
    const double X[3] = {i * cd.h, j * cd.h, k * cd.h};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double aff = eps[c][0] * X[0] + eps[c][1] * X[1] + eps[c][2] * X[2];
      const double* x = chi + ((long long)I * 3 + c) * ntot;
      out[3 * t + c] = x[n0] - x[cd.off] + aff;
    }
  }
}

}  // namespace femh

namespace femh {
// [6][3][node] (engine) <-> [6][node][3] (reference layout) for one cell;
// pin (to the reference layout only): every field relative to its node 0.
template <bool TO_AOS>
__global__ void k_layout(const double* src, double* dst, long long off, long long nn, long long ntot, int pin) {
  const long long total = nn * 18;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int I = (int)(t / (3 * nn));
    const long long rem = t - (long long)I * 3 * nn;
    const long long n = rem / 3;
    const int c = (int)(rem - n * 3);
    const long long eng = ((long long)I * 3 + c) * ntot + off + n;   // engine index
    const long long ref = t;                                          // [I][n][c] of this cell
    if (TO_AOS) dst[ref] = pin ? src[eng] - src[eng - n] : src[eng];
    else dst[eng] = src[ref];
  }
}
}  // namespace femh
