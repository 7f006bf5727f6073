// stencil_launch.cuh -- launches of the stencil kernels of stencil.cuh on a
// level's unit lists: variant and storage rules, compile-time z extents.
// Included by the stencil_*.cu files, which instantiate stencil() explicitly.
#pragma once
#include "state.cuh"

// ======================================================== kernel launch ===
namespace femh_engine {

template <typename T, int NT, int OUT, int NZ, typename TIn, typename TOut, typename TB, typename TC>
void stencil_go(femh_handle* H, dim3 grid, size_t smem, const StencilArgs<TIn, TOut, TB, TC>& a, int variant) {
  if constexpr (std::is_same<T, float>::value) {
    if (variant == 3) {   // two load cases per CTA in packed FP32x2 lanes
      auto fn3 = stencilp_kernel<NT, OUT, NZ, TIn, TOut, TB, TC>;
      allow_smem(H, fn3, 227 * 1024);
      launch(H, fn3, dim3(grid.x, kNumRhs / 2), NT, smem, a);
      return;
    }
  }
  if (variant == 2) {
    auto fn2 = stencil2_kernel<T, NT, OUT, NZ, TIn, TOut, TB, TC>;
    allow_smem(H, fn2, 200 * 1024);
    launch(H, fn2, grid, NT, smem, a);
    return;
  }
  auto fn = stencil_kernel<T, NT, OUT, NZ, TIn, TOut, TB, TC>;
  allow_smem(H, fn, 200 * 1024);
  launch(H, fn, grid, NT, smem, a);
}

// Two voxel rows per thread in packed FP32x2 lanes (variant 4).
template <int NT, int OUT, int NZ, typename TIn, typename TOut, typename TB, typename TC>
void stencil_go4(femh_handle* H, dim3 grid, size_t smem, const StencilArgs<TIn, TOut, TB, TC>& a) {
  auto fn = stencil2p_kernel<NT, OUT, NZ, TIn, TOut, TB, TC>;
  allow_smem(H, fn, 200 * 1024);
  launch(H, fn, grid, NT, smem, a);
}

// Two voxel rows per thread in packed FP32x2 lanes, inputs staged by bulk copies (variant 5).
template <int NT, int OUT, int NZ>
void stencil_go5(femh_handle* H, dim3 grid, size_t smem, const StencilArgs<float, float, float, float>& a) {
  auto fn = stencil2b_kernel<NT, OUT, NZ>;
  allow_smem(H, fn, 200 * 1024);   // (a few bytes of static shared memory come on top)
  launch(H, fn, grid, NT, smem, a);
}

// FP64 operator, one voxel row per thread, inputs staged by bulk copies (variant 6).
template <int NT, int OUT, int NZ, typename TIn>
void stencil_go6(femh_handle* H, dim3 grid, const StencilArgs<TIn, double, double, double>& a) {
  constexpr int smem = stage1b_cta_bytes(NT, NZ, (int)sizeof(TIn), stage1b_blocks(NT, NZ, (int)sizeof(TIn), OUT));
  auto fn = stencil1b_kernel<NT, OUT, NZ, TIn>;
  allow_smem(H, fn, smem);
  launch(H, fn, grid, NT, smem, a);
}

// T = arithmetic type; in/out/b storage types as given.
template <typename T, int OUT, typename TIn, typename TOut, typename TB, typename TC>
void stencil(femh_handle* H, Level& L, bool smooth_only, const TIn* in, TOut* out, const TB* b,
             const TC* kc, double* part, const CGState* stt, double omega) {
  const bool use64 = sizeof(T) == 8 && L.use64 && !smooth_only;
  UnitList& ul = smooth_only ? L.smooth : L.all;
  const std::vector<StencilUnit>& units = use64 ? L.su64 : ul.su;
  if (units.empty()) return;
  int variant = use64 ? L.variant64 : L.variant;
  if (!std::is_same<T, float>::value) {   // packed-FP32 kernels: FP64 twin with the same units
    if (variant == 3) variant = 1;
    if (variant == 4 || variant == 5 || variant == 7) variant = 2;
  } else if (variant == 6) {   // the staged FP64 kernel's FP32 twin takes the same units
    variant = 2;
  }
  if (variant == 6) {   // bulk-copy staging: FP64 output / rhs / coefficients, aligned rows
    const bool ok = std::is_same<TOut, double>::value && std::is_same<TB, double>::value &&
                    std::is_same<TC, double>::value &&
                    (std::is_same<TIn, double>::value || std::is_same<TIn, float>::value);
    auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    if (!(ok && L.bulk_ok64 && al(in) && al(out) && al(kc) && al(L.invd) && (!b || al(b)) && L.ntot % 4 == 0))
      variant = 2;
  }
  bool persistent = false;
  if (variant == 7) {   // the staged kernel as persistent CTAs over the list's CTA table
    persistent = !use64 && !L.grouped && ul.cta.size() >= 2 && H->persist_ok;
    variant = 5;
  }
  if (variant == 5) {   // bulk-copy staging: FP32 storage, 16-byte aligned rows, eligible level
    const bool f32 = std::is_same<TIn, float>::value && std::is_same<TOut, float>::value &&
                     std::is_same<TB, float>::value && std::is_same<TC, float>::value;
    auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    if (!(f32 && L.bulk_ok && al(in) && al(out) && al(kc) && al(L.invd) && (!b || al(b)) && L.ntot % 4 == 0)) {
      variant = 4;
      persistent = false;
    }
  }
  StencilArgs<TIn, TOut, TB, TC> a;
  a.cells = L.d_cells;
  a.units = use64 ? L.d_su64 : ul.d_su;
  a.u = in;
  a.out = out;
  a.b = b;
  a.kc = kc;
  a.invd = L.invd;
  a.partials = part;
  a.stt = stt;
  a.ntot = L.ntot;
  a.k = H->hk;
  a.omega = omega;
  a.err = H->d_err;
  a.wait_limit = H->wait_limit;
  a.cta_units = persistent ? ul.d_cta : nullptr;
  a.binv = (OUT == OUT_JACOBI || OUT == OUT_JACOBI_DOT) ? L.binv : nullptr;
  {
    const HadK& k = H->hk;
    const double kv[8] = {k.A, k.Bd - k.Bo, k.Bo, k.D1 - k.O1, k.O1, k.D2 - k.O2, k.O2, k.G};
    for (int i = 0; i < 8; ++i) a.kp[i] = make_float2((float)kv[i], (float)kv[i]);
  }
  dim3 grid((unsigned)(persistent ? ul.cta.size() - 1 : units.size()), kNumRhs);
  static const char* mode_names[] = {"apply", "apply_dot", "jacobi", "jacobi_dot", "resid"};
  char nm[64];
  snprintf(nm, sizeof nm, "stencil_%s_%s_L%d", sizeof(T) == 8 ? "f64" : "f32", mode_names[OUT], L.level);
  // algorithmic bytes: only (cell, load case) pairs still iterating move data
  double nodes = 0.0;
  if (H->prof) {
    for (const auto& cd : L.cells) {
      if (smooth_only && cd.child < 0) continue;
      int act = kNumRhs;
      if (stt) {
        act = 0;
        for (int q = 0; q < kNumRhs; ++q) act += H->state[cd.id * kNumRhs + q].active ? 1 : 0;
      }
      nodes += (double)cd.nx * cd.ny * cd.nz * act / kNumRhs;
    }
  }
  double per = 18.0 * (sizeof(TIn) + sizeof(TOut)) + sizeof(TC);
  if (OUT >= OUT_JACOBI) per += 18.0 * sizeof(TB) + (OUT == OUT_RESID ? 0.0 : (L.binv ? 24.0 : 4.0));
  std::string key(nm);
  Prof prof_(H, H->prof ? H->kstats.emplace(key, femh_handle::KStat{}).first->first.c_str() : nm, nodes * per);
  // launch on units of one z extent (nz_spec > 0: compile-time kernels) or on
  // the level's runtime-z kernels (nz_spec = 0), lnt threads per CTA
  auto launch = [&](int nz_spec, int lnt, int maxnz, dim3 grid, const StencilArgs<TIn, TOut, TB, TC>& a) {
    const size_t smem =
        variant == 3 ? sizeof(float4) * 12 * (size_t)lnt + 2 * sizeof(float2) * (size_t)(12 * lnt + 3 * maxnz) +
                             64 * sizeof(double)
        : variant == 2 ? sizeof(T) * (size_t)(2 * (6 * lnt + 3 * maxnz) + 24 * lnt) + 16 + 64 * sizeof(double)
                       : 2 * sizeof(T) * (size_t)(15 * lnt + 3 * maxnz) + 16 + 64 * sizeof(double);
    if constexpr (std::is_same<T, double>::value && std::is_same<TOut, double>::value &&
                  std::is_same<TB, double>::value && std::is_same<TC, double>::value &&
                  (std::is_same<TIn, double>::value || std::is_same<TIn, float>::value)) {
      if (variant == 6) {
        const int c = stage_class(nz_spec > 0 ? nz_spec : maxnz);
        switch (c) {
          case 16: stencil_go6<stage_nt64(16), OUT, 16>(H, grid, a); return;
          case 24: stencil_go6<stage_nt64(24), OUT, 24>(H, grid, a); return;
          case 32: stencil_go6<stage_nt64(32), OUT, 32>(H, grid, a); return;
          case 48: stencil_go6<stage_nt64(48), OUT, 48>(H, grid, a); return;
          case 64: stencil_go6<stage_nt64(64), OUT, 64>(H, grid, a); return;
          case 96: stencil_go6<stage_nt64(96), OUT, 96>(H, grid, a); return;
          case 128: stencil_go6<stage_nt64(128), OUT, 128>(H, grid, a); return;
          case 192: stencil_go6<stage_nt64(192), OUT, 192>(H, grid, a); return;
          case 256: stencil_go6<stage_nt64(256), OUT, 256>(H, grid, a); return;
          default: throw FemhError{FEMH_E_ARG, "staged FP64 stencil on an ineligible level"};
        }
      }
    }
    if constexpr (std::is_same<TIn, float>::value && std::is_same<TOut, float>::value &&
                  std::is_same<TB, float>::value && std::is_same<TC, float>::value) {
      if (variant == 5) {
        const int c = stage_class(nz_spec > 0 ? nz_spec : maxnz);
        const size_t sm5 = stencil2b_smem_bytes(kStageNT32, c);
        switch (c) {
          case 16: stencil_go5<kStageNT32, OUT, 16>(H, grid, sm5, a); return;
          case 24: stencil_go5<kStageNT32, OUT, 24>(H, grid, sm5, a); return;
          case 32: stencil_go5<kStageNT32, OUT, 32>(H, grid, sm5, a); return;
          case 48: stencil_go5<kStageNT32, OUT, 48>(H, grid, sm5, a); return;
          case 64: stencil_go5<kStageNT32, OUT, 64>(H, grid, sm5, a); return;
          case 96: stencil_go5<kStageNT32, OUT, 96>(H, grid, sm5, a); return;
          case 128: stencil_go5<kStageNT32, OUT, 128>(H, grid, sm5, a); return;
          case 192: stencil_go5<kStageNT32, OUT, 192>(H, grid, sm5, a); return;
          default: throw FemhError{FEMH_E_ARG, "bulk-copy stencil on an ineligible level"};
        }
      }
    }
    if constexpr (std::is_same<T, float>::value) {
      if (variant == 4) {
        const int nt = variant_nt(lnt, maxnz, 4);
        const size_t sm4 =
            sizeof(float2) * 18 * (size_t)nt + sizeof(float) * (6 * (size_t)maxnz + 2) + 64 * sizeof(double);
        if (nt == 384) {
          switch (nz_spec) {
            case 16: stencil_go4<384, OUT, 16>(H, grid, sm4, a); return;
            case 24: stencil_go4<384, OUT, 24>(H, grid, sm4, a); return;
            case 32: stencil_go4<384, OUT, 32>(H, grid, sm4, a); return;
            case 48: stencil_go4<384, OUT, 48>(H, grid, sm4, a); return;
            case 64: stencil_go4<384, OUT, 64>(H, grid, sm4, a); return;
            case 128: stencil_go4<384, OUT, 128>(H, grid, sm4, a); return;
            default: stencil_go4<384, OUT, 0>(H, grid, sm4, a); return;
          }
        }
        if (nz_spec == 256) {
          stencil_go4<512, OUT, 256>(H, grid, sm4, a);
          return;
        }
        switch (nt) {
          case 128: stencil_go4<128, OUT, 0>(H, grid, sm4, a); return;
          case 256: stencil_go4<256, OUT, 0>(H, grid, sm4, a); return;
          case 512: stencil_go4<512, OUT, 0>(H, grid, sm4, a); return;
          default: throw FemhError{FEMH_E_ARG, "unsupported stencil block size"};
        }
      }
    }
    switch (nz_spec) {   // compile-time z extent (threads fixed per extent)
      case 16: stencil_go<T, 512, OUT, 16>(H, grid, smem, a, variant); return;
      case 24: stencil_go<T, 480, OUT, 24>(H, grid, smem, a, variant); return;
      case 32: stencil_go<T, 512, OUT, 32>(H, grid, smem, a, variant); return;
      case 48: stencil_go<T, 480, OUT, 48>(H, grid, smem, a, variant); return;
      case 64: stencil_go<T, 512, OUT, 64>(H, grid, smem, a, variant); return;
      case 128: stencil_go<T, 512, OUT, 128>(H, grid, smem, a, variant); return;
      case 256: stencil_go<T, 512, OUT, 256>(H, grid, smem, a, variant); return;
      default: break;
    }
    switch (lnt) {
      case 128: stencil_go<T, 128, OUT, 0>(H, grid, smem, a, variant); break;
      case 256: stencil_go<T, 256, OUT, 0>(H, grid, smem, a, variant); break;
      case 512: stencil_go<T, 512, OUT, 0>(H, grid, smem, a, variant); break;
      default: throw FemhError{FEMH_E_ARG, "unsupported stencil block size"};
    }
  };
  if (!L.grouped) {
    launch(L.nz_spec, L.NT, L.maxnz, grid, a);
    return;
  }
  // cells of several compile-time z extents: one launch per extent
  const UnitGroups& gr = use64 ? L.g64 : (smooth_only ? L.gsmooth : L.gall);
  for (size_t gi = 0; gi < gr.nz.size(); ++gi) {
    StencilArgs<TIn, TOut, TB, TC> ag = a;
    ag.units = a.units + gr.b[gi];
    launch(gr.nz[gi], spec_nt(gr.nz[gi]), gr.nz[gi], dim3((unsigned)(gr.e[gi] - gr.b[gi]), kNumRhs), ag);
  }
}

}  // namespace femh_engine
