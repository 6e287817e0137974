// efe_launch.cuh -- tile sizing and launch of the kernels of one element shape.
#pragma once
#include <algorithm>

#include "efe_kernels.cuh"

namespace efe {

// Tile shapes of the element pass.  Variant 0: about 128 material points per CTA (one per
// thread in phase A), 128 threads, at most 72 KB of shared memory so that three CTAs share an SM.
// Variant 1: about 256 points and 256 threads per CTA, up to 110 KB (one or two CTAs per SM).
// The autotuner (edelweissfe_gb300/autotune.py) picks one per group by timing both.
constexpr int SMALL_TILE = 4;
template <int SHAPE, int RULE, int FORM, typename KT, int VARIANT>
struct TileOf {
  // variant 0: 128 threads, ~128 points, 3 CTAs/SM where they fit; 1: 256 threads, ~256 points;
  // 2: variant 0's tile with 4 CTAs/SM where shared memory allows (the compiler then holds the
  // kernel to 128 registers per thread); SMALL_TILE: about 16 points, for groups that fill few SMs
  static constexpr int NQ = RuleInfo<RULE>::NQ;
  static constexpr size_t per_element = LayoutOf<SHAPE, RULE, FORM, KT, 1>::bytes;
  static constexpr size_t budget = VARIANT == 1 ? 110 * 1024 : 72 * 1024;
  static constexpr int points = VARIANT == 1 ? 256 : VARIANT == SMALL_TILE ? 16 : 128;
  static constexpr int fit = (int)(budget / per_element);
  static constexpr int want = (points + NQ - 1) / NQ;
  static constexpr int e0 = fit < want ? fit : want;
  static constexpr int EPB = e0 < 1 ? 1 : (e0 > 32 ? 32 : e0);
  static constexpr int NT = VARIANT == 1 ? 256 : VARIANT == SMALL_TILE && ShapeInfo<SHAPE>::NN <= 8 ? 64 : 128;
  static constexpr size_t bytes = LayoutOf<SHAPE, RULE, FORM, KT, EPB>::bytes;
  static constexpr int MINB = VARIANT == 1 ? 1
                              : (VARIANT == 2 && bytes <= 56 * 1024) ? 4
                              : (bytes <= 72 * 1024 ? 3 : 1);
};
// The warp tile of small-strain Hexa8 with an FP32 tangent (efe_ss3.cuh), one shape for all variants: six CTAs of
// four warps per SM hold the kernel to 80 registers (48 B of spills); five CTAs (96 registers) or four (128) run in 1.00
// and 1.04 times its time on 262144 elements, 1.02 and 1.05 times on 65231.
template <int VARIANT>
struct WarpTile {
  static constexpr int NT = VARIANT == SMALL_TILE ? 32 : 128, EPB = SS3Hexa8Layout<NT>::EPB, MINB = VARIANT == SMALL_TILE ? 1 : 6;
  static constexpr size_t bytes = SS3Hexa8Layout<NT>::bytes;
};
// The two-element tile of Hexa20 3x3x3 with an FP32 tangent (efe_ss3.cuh), one shape for all variants, the number 3 of the
// former tensor-core tile among them: five CTAs per SM (96 registers).  Small strain, 13824 elements: four (128 registers)
// or six (80) run in 1.03 and 1.17 times its time; total Lagrangian, 2730 elements: four in 1.16, six in 1.03.
template <bool TL>
struct Hexa20Tile {
  static constexpr int NT = Hexa20Layout<TL>::NT, EPB = Hexa20Layout<TL>::EPB, MINB = 5;
  static constexpr size_t bytes = Hexa20Layout<TL>::bytes;
};
template <int SHAPE, int RULE, int FORM, typename KT, int VARIANT = 0>
struct Tile
    : std::conditional<FORM == SS3 && ss3_warp_tile<SHAPE, RULE, KT>(), WarpTile<VARIANT>,
                       typename std::conditional<(FORM == SS3 || FORM == TLH) && ss3_hexa20_tile<SHAPE, RULE, KT>(),
                                                 Hexa20Tile<FORM == TLH>,
                                                 TileOf<SHAPE, RULE, FORM, KT, VARIANT>>::type>::type {};

template <int SHAPE, int RULE, int FORM, typename KT, bool FF, int VARIANT>
cudaError_t launch_assemble_variant(const GroupArgs& g, cudaStream_t st) {
  using T = Tile<SHAPE, RULE, FORM, KT, VARIANT>;
  static_assert(T::bytes <= 200 * 1024, "tile does not fit in shared memory");
  auto kern = assemble_kernel<SHAPE, RULE, FORM, KT, T::EPB, T::NT, T::MINB, FF>;
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::bytes);
  if (err != cudaSuccess) return err;
  const int64_t grid = (g.nElements + T::EPB - 1) / T::EPB;
  if (grid == 0) return cudaSuccess;
  kern<<<(unsigned)grid, T::NT, T::bytes, st>>>(g);
  return cudaGetLastError();
}

template <int SHAPE, int RULE, int FORM, typename KT, bool FF = false>
cudaError_t launch_assemble(const GroupArgs& g, cudaStream_t st) {
  // the small-strain solids and the Hexa20 tile form their B-products in integers in either mode
  constexpr bool ffTile = FF && FORM != SS3 && !(FORM == TLH && ss3_hexa20_tile<SHAPE, RULE, KT>());
  // A small group's ordinary tiles leave most SMs without one, and a tile's phases one after the other are then the
  // whole time: small tiles up to two per SM.  320 CPE4 elements (fp64) 11 us against 19, 1200 CPE8R 20 against 45, 512
  // C3D8TL (mixed) 15 against 19, 1000 C3D8 (mixed) 18.4 against 19.5; beyond, 1000 C3D8 (fp64) 32 against 28 and 4000 CPE4
  // 35 against 22.
  using Small = Tile<SHAPE, RULE, FORM, KT, SMALL_TILE>;
  if constexpr (Small::EPB < Tile<SHAPE, RULE, FORM, KT, 0>::EPB) {
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return err;
    if (g.nElements <= (int64_t)2 * sms * Small::EPB)
      return launch_assemble_variant<SHAPE, RULE, FORM, KT, ffTile, SMALL_TILE>(g, st);
  }
  if (g.tileVariant == 1) return launch_assemble_variant<SHAPE, RULE, FORM, KT, ffTile, 1>(g, st);
  if constexpr (Tile<SHAPE, RULE, FORM, KT, 2>::MINB != Tile<SHAPE, RULE, FORM, KT, 0>::MINB) {
    if (g.tileVariant == 2) return launch_assemble_variant<SHAPE, RULE, FORM, KT, ffTile, 2>(g, st);
  }
  return launch_assemble_variant<SHAPE, RULE, FORM, KT, ffTile, 0>(g, st);
}

template <int SHAPE, int RULE>
cudaError_t launch_geometry(int64_t nEl, int64_t elOffset, const int32_t* conn, const double* coords,
                            const double* thickness, double* G, float* G32, float* Glo, double* S,
                            int32_t* status, const Hexa20Fix& fix, cudaStream_t st) {
  const int64_t n = nEl * RuleInfo<RULE>::NQ;
  if (n == 0) return cudaSuccess;
  const int nt = 128;
  geometry_kernel<SHAPE, RULE><<<(unsigned)((n + nt - 1) / nt), nt, 0, st>>>(nEl, elOffset, conn, coords, thickness,
                                                                             G, G32, Glo, S, status, fix);
  return cudaGetLastError();
}

template <int SHAPE, int RULE>
cudaError_t launch_body_force(int64_t nSel, const int32_t* elems, const int32_t* conn, const int32_t* nodeDof,
                              const double* S, const double* f, double* P, cudaStream_t st) {
  const int64_t n = nSel * ShapeInfo<SHAPE>::NN;
  if (n == 0) return cudaSuccess;
  const int nt = 128;
  body_force_kernel<SHAPE, RULE><<<(unsigned)((n + nt - 1) / nt), nt, 0, st>>>(nSel, elems, conn, nodeDof, S, f[0], f[1],
                                                                               ShapeInfo<SHAPE>::DIM == 3 ? f[2] : 0.0, P);
  return cudaGetLastError();
}

struct AdjointArgs {
  int64_t nEl;
  const int32_t* conn;
  const int32_t* nodeDof;
  const double* coords;
  const double* U;
  const double* lam;
  const double* props;
  int nProps, material;
  const double* thickness;
  Hexa20Fix fix;
  double* gX;
  double* gP;
};

template <int SHAPE, int RULE>
cudaError_t launch_adjoint_tl(const AdjointArgs& a, cudaStream_t st);

// reverse mode of one small-strain element pass (efe_adjoint_ss.cuh)
struct SSAdjointArgs {
  int64_t nEl;
  int32_t nProps, material;
  int32_t planeStress;  // 2D groups: 1 for plane stress (local Newton on eps33), 0 for plane strain
  const int32_t* conn;
  const int32_t* nodeDof;
  const double* props;
  const double* geomG;
  const double* geomS;
  const double* stateBefore;  // [S][nPts]
  const double* dU;           // [nDof]
  const double* Pbar;         // [nDof] or null
  const double* barIn;        // [S][nPts] or null
  double* barOut;             // [S][nPts] or null (accumulated)
  double* dUbar;              // [nDof] (accumulated)
  double* gProps;             // [nEl][nProps] or null (accumulated)
  // nodal coordinate adjoints [nNodes][dim] (accumulated) or null; coords and the Hexa20 table for
  // the Jacobian of the Hexa20 quirk
  double* gX;
  const double* coords;
  Hexa20Fix fix;
};

template <int SHAPE, int RULE>
cudaError_t launch_adjoint_ss(const SSAdjointArgs& a, cudaStream_t st);

// form selector: small strain 3D/2D, total Lagrangian hyperelastic, total Lagrangian hypoelastic 3D/2D
template <int SHAPE, int RULE, typename KT, bool FF = false>
cudaError_t launch_form(int form, const GroupArgs& g, cudaStream_t st) {
  constexpr int DIM = ShapeInfo<SHAPE>::DIM;
  if constexpr (DIM == 3) {
    switch (form) {
      case SS3: return launch_assemble<SHAPE, RULE, SS3, KT, FF>(g, st);
      case TLH: return launch_assemble<SHAPE, RULE, TLH, KT, FF>(g, st);
      case TLV3: return launch_assemble<SHAPE, RULE, TLV3, KT>(g, st);
    }
  } else {
    switch (form) {
      case SS2: return launch_assemble<SHAPE, RULE, SS2, KT>(g, st);
      case TLH: return launch_assemble<SHAPE, RULE, TLH, KT, FF>(g, st);
      case TLV2: return launch_assemble<SHAPE, RULE, TLV2, KT>(g, st);
    }
  }
  return cudaErrorInvalidValue;
}

template <int SHAPE, int RULE>
cudaError_t launch_rule(int form, int kprec, const GroupArgs& g, cudaStream_t st) {
  if (kprec == EFE_K_FP32_FF) return launch_form<SHAPE, RULE, float, true>(form, g, st);
  return kprec == EFE_K_FP32 ? launch_form<SHAPE, RULE, float>(form, g, st)
                             : launch_form<SHAPE, RULE, double>(form, g, st);
}

// per-shape entry points (one translation unit each, compiled in parallel)
cudaError_t assemble_quad4(int rule, int form, int kprec, const GroupArgs& g, cudaStream_t st);
cudaError_t assemble_quad8(int rule, int form, int kprec, const GroupArgs& g, cudaStream_t st);
cudaError_t assemble_hexa8(int rule, int form, int kprec, const GroupArgs& g, cudaStream_t st);
cudaError_t assemble_hexa20(int rule, int form, int kprec, const GroupArgs& g, cudaStream_t st);
#define EFE_BODY_DECL(name)                                                                                \
  cudaError_t body_force_##name(int rule, int64_t nSel, const int32_t* elems, const int32_t* conn,            \
                                const int32_t* nodeDof, const double* S, const double* f, double* P, cudaStream_t st);
EFE_BODY_DECL(quad4)
EFE_BODY_DECL(quad8)
EFE_BODY_DECL(hexa8)
EFE_BODY_DECL(hexa20)
#undef EFE_BODY_DECL
// the persistent pass over up to MAX_PERSISTENT_GROUPS groups of each of its element types
// (groups[k][0 .. nGroups[k]) for type k of persistent_type_index)
cudaError_t persistent_groups(int kprec, const GroupArgs (*groups)[MAX_PERSISTENT_GROUPS], const int* nGroups,
                              unsigned long long* counter, cudaStream_t st);
// same pass with the work counter in the library's static scratch array; *needed = tile indices
// the counter runs through (written before the range check)
cudaError_t persistent_groups_noalloc(int kprec, const GroupArgs (*groups)[MAX_PERSISTENT_GROUPS], const int* nGroups,
                                      int64_t* needed, cudaStream_t st);
// FMA-chain probe of the FP64 / FP32 pipe (efe_probe.cu)
cudaError_t fma_probe(int fp64, int blocks, int64_t iterations, void* sink, cudaStream_t st);
int64_t fma_probe_flops(int blocks, int64_t iterations);
// device linear solve (efe_solve.cu)
cudaError_t csr_spmv(const EfePcg& s, const double* x, double* y, cudaStream_t st);
cudaError_t csr_gemv(const EfeCsr& a, const double* x, double alpha, double beta, double* y, cudaStream_t st);
cudaError_t csr_gemv_pairs(const EfeCsr& a, const float2* xf, double alpha, double beta, double* y,
                           cudaStream_t st);
cudaError_t chebyshev_step(int64_t n, const double* dinv, const double* r, double c1, double c2, int accumulate,
                           double* d, double* z, float2* dff, cudaStream_t st);
cudaError_t split_pairs(int64_t n, const double* x, float2* xf, cudaStream_t st);
cudaError_t pcg_start(const EfePcg& s, const double* b, cudaStream_t st);
// CG iterations (efe_pcg.cu); blockCols: first column of every node block or null; every > 0: test
// r.r <= tol2 each `every` iterations and stop one such batch later
cudaError_t pcg_run(const EfePcg& s, const int32_t* blockCols, int64_t nnz, int64_t k0, int nIter, int every, double tol2,
                    cudaStream_t st);
cudaError_t adjoint_ss_quad4(int rule, const SSAdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_ss_quad8(int rule, const SSAdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_ss_hexa8(int rule, const SSAdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_ss_hexa20(int rule, const SSAdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_tl_quad4(int rule, const AdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_tl_quad8(int rule, const AdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_tl_hexa8(int rule, const AdjointArgs& a, cudaStream_t st);
cudaError_t adjoint_tl_hexa20(int rule, const AdjointArgs& a, cudaStream_t st);
#define EFE_GEOMETRY_DECL(name)                                                                          \
  cudaError_t geometry_##name(int rule, int64_t nEl, int64_t off, const int32_t* conn, const double* coords, \
                              const double* th, double* G, float* G32, float* Glo, double* S,                 \
                              int32_t* status, const Hexa20Fix& fix, cudaStream_t st);
EFE_GEOMETRY_DECL(quad4)
EFE_GEOMETRY_DECL(quad8)
EFE_GEOMETRY_DECL(hexa8)
EFE_GEOMETRY_DECL(hexa20)
#undef EFE_GEOMETRY_DECL

}  // namespace efe
