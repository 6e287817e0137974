// efe_ss3.cuh -- the small-strain solid element pass (von Mises, linear elastic; Hexa8, Hexa20), and the total-Lagrangian
// Neo-Hooke one of Hexa20 3x3x3 with an FP32 tangent, with their B-products in fixed-point integers (efe_fixed.cuh);
// included by efe_kernels.cuh.
//
// What is left to the FP64 pipe, which bound this pass in every mode, is the material update (92 instructions per point,
// 53 with an FP32 tangent).  The strain increment de = B dU (9 products per node and point), the residual
// s B^T sigma (9 again) and, with an FP64 tangent, the element stiffness (27 per node pair and point) are sums
// over few terms of one scale per element, so they run as integer multiply-adds and are exact apart from the
// rounding of the operands.
//
// Scales (biased exponents), one per component, as the components of dN/dX (thin elements) and of the increment
// (plates, rotations) differ in size by their nature: component d of the element's dN/dX has D_d, a point the same shift
// t <= 0 of all three (its dN/dX is smaller), so that D_d + t holds it; component c of dU has U_c.  A normal strain is one
// sum, a shear two, of the scales D_j + U_i and D_i + U_j.  A row c of the residual has E_c, the largest s sigma_cd times
// dN/dX_d of the element: the point's factors are rounded relative to E_c - D_d - t, nine instead of six.  The FP64 tangent's
// coefficients (c12 s and c44 s; a s) have em_c and em_a over the points' c 2^2t; its sums (j, k) then em_c + D_j + D_k, the
// flow direction's em_a + Z_j + Z_k with Z_j the largest n_jd dN/dX_d.
//
// Measured, von Mises plastic increment, kernel time before (FP64 sums) and with integers: C3D8, FP64 tangent, 29667
// elements 1027 -> 346 us; FP32 tangent, 262144 elements 1322 -> 992 us; C3D20, FP64 tangent, 2448 elements 1640 -> 321
// us; FP32 tangent, 13824 elements 675 -> 383 us (with one scale for all components 363, 985, 326 and 381).  Norm of the
// error against 113-bit arithmetic, before and now: C3D8, 12 x 11 x 10, P 1.11e-15 -> 1.01e-15, K 4.66e-16 -> 4.62e-16,
// stress 7.4e-16 -> 5.0e-16; C3D20, 9 x 8 x 5, P 3.10e-15 -> 2.97e-15, K 1.31e-15 -> 1.29e-15; FP32 K of C3D8 6.35e-8 ->
// 6.23e-8.  In plates of 1 : 10^5 every strain is within the rounding of its own FP64 sum.
//
// FP64 tangent: K_ab = sum_q  c12 s G_a (x) G_b + c44 s (G_b (x) G_a + G_a . G_b I) - a s nG_a (x) nG_b.  The
// operands c12 s G, c44 s G, -a s nG and nG of every point and node are formed once (integer products of the
// digits); a node pair then takes 27 products per point.
#pragma once

namespace efe {

template <int SHAPE, int RULE, typename KT, int EPB>
struct SS3Layout {
  static constexpr int DIM = 3, NN = ShapeInfo<SHAPE>::NN, NQ = RuleInfo<RULE>::NQ, NDOF = 3 * NN, NP = EPB * NQ;
  static constexpr bool F64 = std::is_same<KT, double>::value;
  // odd strides per point: consecutive points fall on different banks
  static constexpr int GS = NDOF | 1, SV = (2 * NDOF) | 1, DS = 9;
  static constexpr size_t u_off = 0;                                         // double, then fx [EPB][NDOF]
  static constexpr size_t g_off = u_off + 8 * EPB * NDOF;                    // fx [NP][GS]: dN/dX
  static constexpr size_t d_off = g_off + 8 * NP * GS;                       // [NP][DS]: strain, then s sigma (double, fx)
  static constexpr size_t k_off = d_off + 8 * NP * DS;                       // F64: fx [4][NP][GS], else KT [NP][SV]
  // flow direction n: double, then fx (F64), or float where the tangent's vectors are formed per point and node
  static constexpr size_t n_off = (k_off + (F64 ? (size_t)32 * NP * GS : (size_t)4 * NP * SV) + 7) / 8 * 8;  // [NP][DS]
  static constexpr size_t c_off = (n_off + (F64 || NN > 8 || NQ > 8 ? sizeof(KT) * NP * DS : 0) + 7) / 8 * 8;  // KT [NP][3]: coefficients
  static constexpr size_t mc_off = (c_off + sizeof(KT) * NP * 3 + 15) / 16 * 16;  // VMConst [EPB]
  static constexpr size_t rl_off = mc_off + sizeof(VMConst) * EPB;                // int [EPB][NN]
  static constexpr int ES = 14;                                                   // scales of an element: U, D, E, Z, em_c, em_a
  static constexpr size_t e_off = rl_off + sizeof(int) * EPB * NN;                // int [EPB][ES]; [NP][3]: a point's maxima; [NP]: t
  static constexpr size_t bytes = e_off + sizeof(int) * (ES * EPB + 4 * NP);
};

__device__ __forceinline__ int fx_max_exponent(int em, double x) { return max(em, fx_exponent(x)); }

// Where the factors of a point's rows lie: digit of (row c, direction d), from the Voigt value of the same place; a shear
// value has one for each of its rows.
__device__ __forceinline__ constexpr int row_slot(int c, int d) {
  return c == 0 ? (d == 0 ? 0 : 2 + d) : c == 1 ? (d == 0 ? 6 : d == 1 ? 1 : 5) : (d == 2 ? 2 : 7 + d);
}
// The digits of Voigt value f of a point in its row's scale: E[c] - D[d] - t, with E and D the element's.
__device__ __forceinline__ void row_digits(fx* out, double x, int f, const int* E, const int* D, int t) {
  const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
  if (f >= 3) out[f + 3] = fx_make(x, E[j] - D[i] - t);
  out[f] = fx_make(x, E[i] - D[j] - t);
}

template <int SHAPE, int RULE, typename KT, int EPB, int NT>
__device__ __forceinline__ void assemble_tile_ss3(const GroupArgs& g, const int64_t e0, unsigned char* smem) {
  using L = SS3Layout<SHAPE, RULE, KT, EPB>;
  constexpr int NN = L::NN, NQ = L::NQ, NDOF = L::NDOF, NP = L::NP, GS = L::GS, SV = L::SV, DS = L::DS, ES = L::ES;
  constexpr bool F64 = L::F64;
  // one thread forms a point's digits and strain where a point has few nodes (the tile has a thread per point)
  constexpr bool PERPOINT = NN == 8 && NP <= NT;
  double* su = reinterpret_cast<double*>(smem + L::u_off);
  fx* suf = reinterpret_cast<fx*>(smem + L::u_off);
  fx* sg = reinterpret_cast<fx*>(smem + L::g_off);
  double* sd = reinterpret_cast<double*>(smem + L::d_off);
  fx* sdf = reinterpret_cast<fx*>(smem + L::d_off);
  KT* sv = reinterpret_cast<KT*>(smem + L::k_off);
  fx* sset = reinterpret_cast<fx*>(smem + L::k_off);
  KT* sn = reinterpret_cast<KT*>(smem + L::n_off);
  fx* snf = reinterpret_cast<fx*>(smem + L::n_off);
  KT* sc = reinterpret_cast<KT*>(smem + L::c_off);
  fx* scf = reinterpret_cast<fx*>(smem + L::c_off);
  VMConst* smc = reinterpret_cast<VMConst*>(smem + L::mc_off);
  int* srl = reinterpret_cast<int*>(smem + L::rl_off);
  int* sem = reinterpret_cast<int*>(smem + L::e_off);
  constexpr int eU = 0, eD = 3, eE = 6, eZ = 9, eC = 12, eA = 13;  // of an element's ES
  int *semp = sem + ES * EPB, *semt = semp + 3 * NP;
  const int tid = threadIdx.x;
  const int64_t nEl = g.nElements, stride = nEl * NQ;
  const int nLoc = nEl - e0 < EPB ? (int)(nEl - e0) : EPB, np = nLoc * NQ;
  // the shift of a point whose components have the exponents e
  auto shift = [&](const int* e, const int* el) { return max(max(e[0] - el[eD], e[1] - el[eD + 1]), e[2] - el[eD + 2]); };

  // ---- dU relative to the element's first node (sum_a dN_a/dX = 0), row lengths, material constants, dN/dX
  for (int t = tid; t < ES * EPB + 3 * NP; t += NT) sem[t] = 0;
  if (!PERPOINT) __syncthreads();
  double G[PERPOINT ? 3 : 1][PERPOINT ? NN : 1];
  int eg[3] = {0, 0, 0};
  if constexpr (PERPOINT) {
    if (tid < np) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < NN; ++a) G[c][a] = g.geomG[(int64_t)(c * NN + a) * stride + e0 * NQ + tid];
    }
  } else {
    for (int t = tid; t < np * NN; t += NT) {
      const int a = t / np, r = t - a * np;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        atomicMax(semp + r * 3 + c, fx_exponent(g.geomG[(int64_t)(c * NN + a) * stride + e0 * NQ + r]));
    }
  }
  for (int t = tid; t < nLoc * NN; t += NT) {
    const int le = t / NN, a = t - le * NN;
    const int64_t e = e0 + le;
    double* u = su + le * NDOF + a * 3;
    u[0] = u[1] = u[2] = 0.0;
    const int32_t node = g.conn[e * NN + a], node0 = g.conn[e * NN];
    if (!in_bounds(g, node, g.nNodes, e) || !in_bounds(g, node0, g.nNodes, e)) continue;
    srl[le * NN + a] = g.nodeRowLen[node];
    const int32_t dof = g.nodeDof[node], dof0 = g.nodeDof[node0];
    if (!in_bounds(g, dof, g.nDof - 2, e) || !in_bounds(g, dof0, g.nDof - 2, e)) continue;
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = g.dU[dof + c] - g.dU[dof0 + c];
  }
  // the last warp, which has the least of the gather
  for (int le = NT - 1 - tid; le < nLoc; le += NT)
    smc[le] = vm_const<!F64>(g.props + (e0 + le) * g.nProps, g.material == EFE_MAT_VON_MISES);
  __syncthreads();
  for (int t = tid; t < nLoc * NDOF; t += NT) atomicMax(sem + t / NDOF * ES + eU + t % 3, fx_exponent(su[t]));
  if constexpr (PERPOINT) {
    if (tid < np) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int a = 0; a < NN; ++a) eg[c] = fx_max_exponent(eg[c], G[c][a]);
        atomicMax(sem + tid / NQ * ES + eD + c, eg[c]);
      }
    }
  } else {
    for (int t = tid; t < np * 3; t += NT) atomicMax(sem + t / (3 * NQ) * ES + eD + t % 3, semp[t]);
  }
  __syncthreads();

  // ---- digits of dU and dN/dX; the FP32 tangent's dN/dX
  for (int t = tid; t < nLoc * NDOF; t += NT) suf[t] = fx_make(su[t], sem[t / NDOF * ES + eU + t % 3]);
  if constexpr (PERPOINT) {
    if (tid < np) {
      const int* el = sem + tid / NQ * ES;
      const int t = shift(eg, el);
      semt[tid] = t;
#pragma unroll
      for (int c = 0; c < 3; ++c) eg[c] = el[eD + c] + t;
#pragma unroll
      for (int a = 0; a < NN; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          sg[tid * GS + a * 3 + c] = fx_make(G[c][a], eg[c]);
          if constexpr (!F64) sv[tid * SV + a * 6 + c] = ff_split_rn_bits(G[c][a]).h;
        }
    }
  } else {
    for (int k = tid; k < np * NN; k += NT) {
      const int a = k / np, r = k - a * np;
      const int* el = sem + r / NQ * ES;
      const int t = shift(semp + r * 3, el);
      if (a == 0) semt[r] = t;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double x = g.geomG[(int64_t)(c * NN + a) * stride + e0 * NQ + r];
        sg[r * GS + a * 3 + c] = fx_make(x, el[eD + c] + t);
        if constexpr (!F64) sv[r * SV + a * 6 + c] = ff_split_rn_bits(x).h;
      }
    }
  }
  __syncthreads();

  // ---- strain increment (element.py:322), Voigt 11, 22, 33, 12, 13, 23 with engineering shears
  double de[6] = {0, 0, 0, 0, 0, 0};
  if constexpr (PERPOINT) {
    if (tid < np) {
      const fx* gp = sg + tid * GS;
      const fx* up = suf + tid / NQ * NDOF;
      const int* eu = sem + tid / NQ * ES + eU;
      FxSum s[9] = {};
#pragma unroll
      for (int a = 0; a < NN; ++a) {
        const fx gx = gp[a * 3], gy = gp[a * 3 + 1], gz = gp[a * 3 + 2];
        const fx ux = up[a * 3], uy = up[a * 3 + 1], uz = up[a * 3 + 2];
        fx_fma(s[0], gx, ux);
        fx_fma(s[1], gy, uy);
        fx_fma(s[2], gz, uz);
        fx_fma(s[3], gy, ux);
        fx_fma(s[4], gz, ux);
        fx_fma(s[5], gz, uy);
        fx_fma(s[6], gx, uy);
        fx_fma(s[7], gx, uz);
        fx_fma(s[8], gy, uz);
      }
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
        int em = eg[j] + eu[i];
        int64_t v = fx_int(s[f], -1);
        if (f >= 3) v = fx_add(v, em, fx_int(s[f + 3], -1), eg[i] + eu[j]);
        de[f] = fx_value(v, em + 1);
      }
    }
  } else {
    for (int t = tid; t < np * 6; t += NT) {
      const int f = t / np, r = t - f * np;
      const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
      const fx* gp = sg + r * GS;
      const fx* up = suf + r / NQ * NDOF;
      FxSum s{0, 0}, s2{0, 0};
      for (int a = 0; a < NN; ++a) {
        fx_fma(s, gp[a * 3 + j], up[a * 3 + i]);
        if (f >= 3) fx_fma(s2, gp[a * 3 + i], up[a * 3 + j]);
      }
      const int *el = sem + r / NQ * ES, t0 = semt[r];
      int em = el[eD + j] + el[eU + i] + t0;
      const int64_t v = fx_add(fx_int(s, -1), em, fx_int(s2, -1), f >= 3 ? el[eD + i] + el[eU + j] + t0 : em);
      sd[r * DS + f] = fx_value(v, em + 1);
    }
    __syncthreads();
  }

  // ---- material points (a thread per point): state, s sigma, the tangent's coefficients and flow direction
  for (int t = tid; t < np; t += NT) {
    const int le = t / NQ;
    const int64_t e = e0 + le, pt = e0 * NQ + t;
    const double s = g.geomS[pt];
    double sig[6], eps[6], kappa = 0.0;
    for (int f = 0; f < 6; ++f) {
      sig[f] = g.stateRef[(int64_t)f * stride + pt];
      eps[f] = g.stateRef[(int64_t)(6 + f) * stride + pt];
    }
    const bool hasM = g.material != EFE_MAT_LINEAR_ELASTIC;
    if (hasM) kappa = g.stateRef[(int64_t)12 * stride + pt];
    if constexpr (!PERPOINT)
      for (int f = 0; f < 6; ++f) de[f] = sd[t * DS + f];
    bool ok = true;
    typename std::conditional<F64, Tangent3, TangentF32>::type T;
    if (g.material == EFE_MAT_LINEAR_ELASTIC)
      linear_elastic_3d(smc[le], sig, de, T);
    else if constexpr (F64)
      ok = von_mises_3d<false>(smc[le], sig, de, kappa, T);
    else
      ok = von_mises_3d_f32(smc[le], sig, de, kappa, T);
    bool finite = true;
    int* el = sem + le * ES;
    const int t0 = semt[t];
    int es[3] = {0, 0, 0};
    for (int f = 0; f < 6; ++f) {
      g.stateTemp[(int64_t)f * stride + pt] = sig[f];
      g.stateTemp[(int64_t)(6 + f) * stride + pt] = eps[f] + de[f];
      finite = finite && finite_bits(sig[f]);
      const double ss = sig[f] * s;
      sd[t * DS + f] = ss;
      const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2), ef = fx_exponent(ss);
      es[i] = max(es[i], ef + el[eD + j]);
      es[j] = max(es[j], ef + el[eD + i]);
    }
    if (hasM) g.stateTemp[(int64_t)12 * stride + pt] = kappa;
    if (!ok) report(g.status, EFE_STATUS_CUTBACK, g.elementOffset + e, 1);
    if (!finite) atomicOr(g.status, EFE_STATUS_NONFINITE);
    for (int c = 0; c < 3; ++c) atomicMax(el + eE + c, es[c] + t0);
    const double c[3] = {T.c12 * s, T.c44 * s, T.a * s};
    if constexpr (F64) {
      int ez[3] = {0, 0, 0};
      for (int f = 0; f < 6; ++f) {
        sn[t * DS + f] = T.n[f];
        const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2), ef = fx_exponent(T.n[f]);
        ez[i] = max(ez[i], ef + el[eD + j]);
        ez[j] = max(ez[j], ef + el[eD + i]);
      }
      for (int k = 0; k < 3; ++k) {
        sc[t * 3 + k] = c[k];
        atomicMax(el + eZ + k, ez[k]);
      }
      atomicMax(el + eC, max(fx_exponent(c[0]), fx_exponent(c[1])) + 2 * t0);
      atomicMax(el + eA, fx_exponent(c[2]) + 2 * t0);
    } else {
      for (int k = 0; k < 3; ++k) sc[t * 3 + k] = ff_split_rn_bits(c[k]).h;
      const float* n = T.n;
      if constexpr (PERPOINT) {
        for (int a = 0; a < NN; ++a) {
          KT* v = sv + t * SV + a * 6;
          const KT gx = v[0], gy = v[1], gz = v[2];
          v[3] = n[0] * gx + n[3] * gy + n[4] * gz;
          v[4] = n[3] * gx + n[1] * gy + n[5] * gz;
          v[5] = n[4] * gx + n[5] * gy + n[2] * gz;
        }
      } else {
        for (int f = 0; f < 6; ++f) sn[t * DS + f] = n[f];
      }
    }
  }
  __syncthreads();

  // ---- digits of the per-point factors
  for (int t = tid; t < np * 6; t += NT) {
    const int r = t / 6, f = t - r * 6;
    const int* el = sem + r / NQ * ES;
    row_digits(sdf + r * DS, sd[r * DS + f], f, el + eE, el + eD, semt[r]);
    if constexpr (F64) row_digits(snf + r * DS, sn[r * DS + f], f, el + eZ, el + eD, 0);
  }
  if constexpr (F64) {
    for (int t = tid; t < np * 3; t += NT) {
      const int r = t / 3;
      scf[t] = fx_make(sc[t], sem[r / NQ * ES + (t - r * 3 == 2 ? eA : eC)] - 2 * semt[r]);
    }
  }
  if constexpr (F64 || !PERPOINT) {
    if constexpr (F64) __syncthreads();
    // the tangent's operands per point and node
    for (int t = tid; t < np * NN; t += NT) {
      const int a = t / np, r = t - a * np;
      if constexpr (F64) {
        const fx gx = sg[r * GS + a * 3], gy = sg[r * GS + a * 3 + 1], gz = sg[r * GS + a * 3 + 2];
        const fx* n = snf + r * DS;
        FxSum z[3] = {};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          fx_fma(z[c], n[row_slot(c, 0)], gx);
          fx_fma(z[c], n[row_slot(c, 1)], gy);
          fx_fma(z[c], n[row_slot(c, 2)], gz);
        }
        const fx c0 = scf[r * 3], c1 = scf[r * 3 + 1], c2 = scf[r * 3 + 2];
        fx* v = sset + (size_t)r * GS + a * 3;
        const fx gv[3] = {gx, gy, gz};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const fx zc = fx_split(fx_int(z[c], -3));  // three products: scale Z_c + t - 1020
          v[c] = fx_mul(c0, gv[c]);
          v[(size_t)NP * GS + c] = fx_mul(c1, gv[c]);
          v[(size_t)2 * NP * GS + c] = fx_mul(c2, zc);
          v[(size_t)3 * NP * GS + c] = zc;
        }
      } else {
        const KT* n = sn + r * DS;
        KT* v = sv + r * SV + a * 6;
        const KT gx = v[0], gy = v[1], gz = v[2];
        v[3] = n[0] * gx + n[3] * gy + n[4] * gz;
        v[4] = n[3] * gx + n[1] * gy + n[5] * gz;
        v[5] = n[4] * gx + n[5] * gy + n[2] * gz;
      }
    }
  }
  __syncthreads();

  // ---- residual and flux (NIST.computeElements, nonlinearimplicitstatic.py:837-844): P_e[a][c] = -sum_q s sigma[c] . G_a
  for (int t = tid; t < nLoc * NDOF; t += NT) {
    const int le = t / NDOF, k = t - le * NDOF, a = k / 3, c = k - 3 * a;
    const int64_t e = e0 + le;
    const int v0 = row_slot(c, 0), v1 = row_slot(c, 1), v2 = row_slot(c, 2);
    constexpr int R = NQ > 8 ? -2 : 0;
    FxSum s[3] = {};  // one for each direction: 27 products at most
    for (int q = 0; q < NQ; ++q) {
      const fx* gp = sg + (le * NQ + q) * GS + a * 3;
      const fx* dp = sdf + (le * NQ + q) * DS;
      fx_fma(s[0], dp[v0], gp[0]);
      fx_fma(s[1], dp[v1], gp[1]);
      fx_fma(s[2], dp[v2], gp[2]);
    }
    const double pe = -fx_value(fx_int(s[0], R) + fx_int(s[1], R) + fx_int(s[2], R), sem[le * ES + eE + c] - R);
    const int32_t node = g.conn[e * NN + a];
    if (!in_bounds(g, node, g.nNodes, e)) continue;
    const int32_t dof = g.nodeDof[node] + c;
    if (!in_bounds(g, dof, g.nDof, e)) continue;
    atomicAdd(g.P + dof, pe);
    atomicAdd(g.F + dof, fabs(pe));
  }

  // ---- tangent blocks of the node pairs a <= b (the element tangents are symmetric), each scattered twice
  KT* K = reinterpret_cast<KT*>(g.Kdata);
  constexpr int NPAIR = NN * (NN + 1) / 2;
  for (int t = tid; t < nLoc * NPAIR; t += NT) {
    const int le = t / NPAIR;
    int r = t - le * NPAIR, a = 0;
    while (r >= NN - a) {
      r -= NN - a;
      ++a;
    }
    const int b = a + r;
    const int64_t e = e0 + le;
    KT acc[3][3];
    if constexpr (F64) {
      FxSum s1[3][3] = {}, s2[3][3] = {}, s3[3][3] = {};
#pragma unroll 1
      for (int q = 0; q < NQ; ++q) {
        const fx* va = sset + (size_t)(le * NQ + q) * GS + a * 3;
        const fx* zb = sset + (size_t)(3 * NP + le * NQ + q) * GS + b * 3;
        const fx* gb = sg + (le * NQ + q) * GS + b * 3;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const fx la = va[j], ma = va[(size_t)NP * GS + j], ta = va[(size_t)2 * NP * GS + j];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            fx_fma(s1[j][k], la, gb[k]);
            fx_fma(s2[j][k], ma, gb[k]);
            fx_fma(s3[j][k], ta, zb[k]);
          }
        }
      }
      // The first two sums in units of em_c - 1022 + D_j + D_k, the third of em_a - 3062 + Z_j + Z_k, added at the coarser
      // of them with B guard bits: as many as the largest of the 27 sums leaves (six of them add up)
      int top = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) top |= fx_bits(s1[j][k]) | fx_bits(s2[j][k]) | fx_bits(s3[j][k]);
      const int B = min(__clz(top) - 5, 26);
      const int* el = sem + le * ES;
      const int ec = el[eC] - 1022, ea = el[eA] - 3062, D[3] = {el[eD], el[eD + 1], el[eD + 2]}, Z[3] = {el[eZ], el[eZ + 1], el[eZ + 2]};
      const int Dm = max(D[0], max(D[1], D[2]));
      int64_t dot = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j) dot += fx_down(fx_int(s2[j][j], B), 2 * (Dm - D[j]));
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int cjk = ec + D[j] + D[k], ajk = ea + Z[j] + Z[k], em = max(j == k ? ec + 2 * Dm : cjk, ajk);
          int64_t v = fx_down(fx_int(s1[j][k], B) + fx_int(s2[k][j], B), em - cjk) - fx_down(fx_int(s3[j][k], B), em - ajk);
          if (j == k) v += fx_down(dot, em - ec - 2 * Dm);
          acc[j][k] = fx_value(v, em - B);
        }
    } else {
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[j][k] = KT(0);
      for (int q = 0; q < NQ; ++q) {
        const KT* cq = sc + (le * NQ + q) * 3;
        const KT* va = sv + (le * NQ + q) * SV + a * 6;
        const KT* vb = sv + (le * NQ + q) * SV + b * 6;
        const KT Lq = cq[0], Mq = cq[1], Aq = cq[2];
        const KT dot = va[0] * vb[0] + va[1] * vb[1] + va[2] * vb[2];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int k = 0; k < 3; ++k)
            acc[j][k] += Lq * va[j] * vb[k] + Mq * ((j == k ? dot : KT(0)) + va[k] * vb[j]) - Aq * va[3 + j] * vb[3 + k];
      }
    }
    // Ke[(a,j),(b,k)] -> CSR (row = dof(b,k), col = dof(a,j)) = slot(a,b) + k*rowLen(b) + j
    const int32_t slot = g.pairSlot[(e * NN + a) * NN + b];
    const int rl = srl[le * NN + b];
    if (!in_bounds(g, slot, g.nnz, e) || !in_bounds(g, slot + (int64_t)2 * (rl + 1), g.nnz, e)) continue;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k) kadd(K + slot + (int64_t)k * rl + j, acc[j][k]);
    if (a != b) {  // Ke[(b,k),(a,j)] = Ke[(a,j),(b,k)] -> (row = dof(a,j), col = dof(b,k))
      const int32_t slot2 = g.pairSlot[(e * NN + b) * NN + a];
      const int rl2 = srl[le * NN + a];
      if (!in_bounds(g, slot2, g.nnz, e) || !in_bounds(g, slot2 + (int64_t)2 * (rl2 + 1), g.nnz, e)) continue;
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) kadd(K + slot2 + (int64_t)j * rl2 + k, acc[j][k]);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Hexa8 with 2x2x2 points and an FP32 tangent: a warp works on four elements, a lane per point, the eight lanes of an
// element also holding its eight nodes.  The scales are maxima and the residual a transposing sum over eight lanes;
// the point's row of shared memory holds the digits of dN/dX and then, in their place, the tangent's vectors.  The only
// wait for other warps is for the elements' material constants (FP64 divisions, formed by one warp for all).  262144
// elements: 992 us; latency of the chain through a warp's phases binds it (the FP64
// pipe is about half busy), hence few registers and 24 warps per SM.
template <int NT>
struct SS3Hexa8Layout {
  static constexpr int NW = NT / 32, EPB = 4 * NW;
  // a point's row in doublewords: 24 digits of dN/dX, then the floats (dN/dX, n dN/dX) of 8 nodes; 3 coefficients; 27,
  // odd, so that consecutive points fall on different banks
  static constexpr int SV = 27;
  static constexpr size_t v_off = 0;                                            // fx [NW][32][SV]
  static constexpr size_t u_off = v_off + sizeof(fx) * NW * 32 * SV;            // fx [NW][4][24]
  static constexpr size_t mc_off = (u_off + sizeof(fx) * NW * 96 + 15) / 16 * 16;  // VMConst [EPB]
  static constexpr size_t rl_off = mc_off + sizeof(VMConst) * EPB;              // int [NW][32]
  static constexpr size_t bytes = rl_off + sizeof(int) * NW * 32;
};

template <int NT>
__device__ __forceinline__ void assemble_tile_ss3_hexa8(const GroupArgs& g, const int64_t e0, unsigned char* smem) {
  using L = SS3Hexa8Layout<NT>;
  constexpr int NN = 8, NQ = 8, SV = L::SV;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, le = lane >> 3, q = lane & 7;
  fx* sv = reinterpret_cast<fx*>(smem + L::v_off) + wid * 32 * SV;
  fx* su = reinterpret_cast<fx*>(smem + L::u_off) + wid * 96;
  VMConst* smc = reinterpret_cast<VMConst*>(smem + L::mc_off);
  int* srl = reinterpret_cast<int*>(smem + L::rl_off) + wid * 32;
  float* K = reinterpret_cast<float*>(g.Kdata);
  const int64_t nEl = g.nElements, stride = nEl * NQ, eS = e0 + wid * 4, e = eS + le, pt = eS * NQ + lane;
  const bool vm = g.material == EFE_MAT_VON_MISES, live = e < nEl;
  fx* row = sv + lane * SV;
  if (wid == L::NW - 1 && lane < L::EPB && e0 + lane < nEl) smc[lane] = vm_const<true>(g.props + (e0 + lane) * g.nProps, vm);

  // ---- the node's dU relative to the element's first node, digits of it and of the point's dN/dX
  int32_t dof = -1;
  int eg[3] = {0, 0, 0}, eu[3] = {0, 0, 0};  // scales of the point's dN/dX and of dU
  {
    double u[3] = {0.0, 0.0, 0.0};
    double G[3][NN];
    int rl = 0;
    if (live) {
      const int32_t node = g.conn[e * NN + q];
      if (in_bounds(g, node, g.nNodes, e)) {
        rl = g.nodeRowLen[node];
        const int32_t d = g.nodeDof[node];
        if (in_bounds(g, d, g.nDof - 2, e)) {
          dof = d;
#pragma unroll
          for (int c = 0; c < 3; ++c) u[c] = g.dU[d + c];
        }
      }
      const double* gp = g.geomG + pt;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < NN; ++a) G[c][a] = gp[(int64_t)(c * NN + a) * stride];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < NN; ++a) eg[c] = fx_max_exponent(eg[c], G[c][a]);
    }
    srl[lane] = rl;
    int D[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      u[c] -= __shfl_sync(0xffffffffu, u[c], lane & 24);
      eu[c] = fx_exponent(u[c]);
      D[c] = eg[c];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        eu[c] = max(eu[c], __shfl_xor_sync(0xffffffffu, eu[c], o));
        D[c] = max(D[c], __shfl_xor_sync(0xffffffffu, D[c], o));
      }
      su[lane * 3 + c] = fx_make(u[c], eu[c]);
    }
    if (live) {
      const int t = max(max(eg[0] - D[0], eg[1] - D[1]), eg[2] - D[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) eg[c] = D[c] + t;
#pragma unroll
      for (int a = 0; a < NN; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) row[a * 3 + c] = fx_make(G[c][a], eg[c]);
    }
  }
  __syncthreads();

  // ---- strain increment (element.py:322), material update, state
  int es[3] = {0, 0, 0};  // scales of the residual's rows
  double sig[6] = {0, 0, 0, 0, 0, 0}, s = 0.0;
  float n[6], cf[3];
  if (live) {
    s = g.geomS[pt];
    double de[6], kappa = 0.0;
#pragma unroll
    for (int f = 0; f < 6; ++f) sig[f] = g.stateRef[(int64_t)f * stride + pt];
    const bool hasM = g.material != EFE_MAT_LINEAR_ELASTIC;
    if (hasM) kappa = g.stateRef[(int64_t)12 * stride + pt];
    {
      FxSum acc[9] = {};
      const fx* up = su + le * 24;
#pragma unroll
      for (int a = 0; a < NN; ++a) {
        const fx ux = up[a * 3], uy = up[a * 3 + 1], uz = up[a * 3 + 2];
        const fx gx = row[a * 3], gy = row[a * 3 + 1], gz = row[a * 3 + 2];
        fx_fma(acc[0], gx, ux);
        fx_fma(acc[1], gy, uy);
        fx_fma(acc[2], gz, uz);
        fx_fma(acc[3], gy, ux);
        fx_fma(acc[4], gz, ux);
        fx_fma(acc[5], gz, uy);
        fx_fma(acc[6], gx, uy);
        fx_fma(acc[7], gx, uz);
        fx_fma(acc[8], gy, uz);
      }
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
        int em = eg[j] + eu[i];
        int64_t v = fx_int(acc[f], -1);
        if (f >= 3) v = fx_add(v, em, fx_int(acc[f + 3], -1), eg[i] + eu[j]);
        de[f] = fx_value(v, em + 1);
      }
    }
    bool ok = true;
    TangentF32 T;
    const VMConst& mc = smc[wid * 4 + le];
    if (vm)
      ok = von_mises_3d_f32(mc, sig, de, kappa, T);
    else
      linear_elastic_3d(mc, sig, de, T);
    bool finite = true;
    // all loads before the first store, which they could not pass
#pragma unroll
    for (int f = 0; f < 6; ++f) de[f] += g.stateRef[(int64_t)(6 + f) * stride + pt];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      g.stateTemp[(int64_t)f * stride + pt] = sig[f];
      g.stateTemp[(int64_t)(6 + f) * stride + pt] = de[f];
      finite = finite && finite_bits(sig[f]);
      n[f] = T.n[f];
    }
    if (hasM) g.stateTemp[(int64_t)12 * stride + pt] = kappa;
    if (!ok) report(g.status, EFE_STATUS_CUTBACK, g.elementOffset + e, 1);
    if (!finite) atomicOr(g.status, EFE_STATUS_NONFINITE);
    cf[0] = ff_split_rn_bits(T.c12 * s).h;
    cf[1] = ff_split_rn_bits(T.c44 * s).h;
    cf[2] = ff_split_rn_bits(T.a * s).h;
  }
  // ---- residual: s sigma . G_a of the point for every node, summed over the element's points by exchanges that leave
  // node q's three sums in lane q
  {
    // s sigma exactly as integers, then their digits in the rows' scales
    const int e1 = fx_exponent(s) - 1022;  // of s sigma: that of sigma and this
    int ef[6];
    fx d[9];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
      ef[f] = fx_exponent(sig[f]) + e1;
      es[i] = max(es[i], ef[f] + eg[j]);
      es[j] = max(es[j], ef[f] + eg[i]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) es[c] = max(es[c], __shfl_xor_sync(0xffffffffu, es[c], o));
    const fx sd = fx_make(s, e1 + 1022);
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
      FxSum p{0, 0};
      fx_fma(p, fx_make(sig[f], ef[f] - e1), sd);
      const int64_t v = live ? fx_int(p, -1) : 0;
      d[f] = fx_split(fx_shift(v, min(es[i] - eg[j] - ef[f], 62)));  // rounded: an operand
      if (f >= 3) d[f + 3] = fx_split(fx_shift(v, min(es[j] - eg[i] - ef[f], 62)));
    }
    auto force = [&](int a, int c) {
      FxSum r{0, 0};
      fx_fma(r, d[row_slot(c, 0)], row[a * 3]);
      fx_fma(r, d[row_slot(c, 1)], row[a * 3 + 1]);
      fx_fma(r, d[row_slot(c, 2)], row[a * 3 + 2]);
      return (long long)fx_int(r);
    };
    if (!live)
#pragma unroll
      for (int k = 0; k < 24; ++k) row[k] = fx{0, 0};
    const bool b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
    double pe[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      long long t[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const long long lo = force(a, c), hi = force(a + 4, c);
        t[a] = (b2 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b2 ? lo : hi, 4);
      }
      const long long x0 = (b1 ? t[2] : t[0]) + __shfl_xor_sync(0xffffffffu, b1 ? t[0] : t[2], 2);
      const long long x1 = (b1 ? t[3] : t[1]) + __shfl_xor_sync(0xffffffffu, b1 ? t[1] : t[3], 2);
      pe[c] = -fx_value((b0 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, b0 ? x0 : x1, 1), es[c]);
    }
    if (dof >= 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        atomicAdd(g.P + dof + c, pe[c]);
        atomicAdd(g.F + dof + c, fabs(pe[c]));
      }
    }
  }
  // ---- the tangent's vectors in the place of the digits, from the upper ones: 29 bits of the largest of their component.
  // The FP32 sums round at 24 of it: errors of K with all bits, or with dN/dX itself rounded, are the same within 1 %.
  if (live) {
    const float sx = fx_unit(eg[0]), sy = fx_unit(eg[1]), sz = fx_unit(eg[2]);
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      const float gx = fx_float(row[a * 3], sx), gy = fx_float(row[a * 3 + 1], sy), gz = fx_float(row[a * 3 + 2], sz);
      float2* v = reinterpret_cast<float2*>(row + a * 3);
      v[0] = make_float2(gx, gy);
      v[1] = make_float2(gz, n[0] * gx + n[3] * gy + n[4] * gz);
      v[2] = make_float2(n[3] * gx + n[1] * gy + n[5] * gz, n[4] * gx + n[5] * gy + n[2] * gz);
    }
    float2* v = reinterpret_cast<float2*>(row + 24);
    v[0] = make_float2(cf[0], cf[1]);
    v[1] = make_float2(cf[2], 0.0f);
  }
  __syncwarp();

  // ---- tangent: the 36 node pairs as (a, a + d mod 8), d = 0 .. 3 for every a and d = 4 for a < 4
  const int nLoc = nEl - eS < 4 ? (int)(nEl - eS) : 4;
  for (int t = lane; t < nLoc * 36; t += 32) {
    const int el = t / 36, r = t - el * 36, a = r & 7, b = (a + (r >> 3)) & 7;
    const int64_t ee = eS + el;
    const int32_t slot = g.pairSlot[(ee * NN + a) * NN + b], slot2 = g.pairSlot[(ee * NN + b) * NN + a];
    float acc[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, dot = 0.0f;
    const float2* base = reinterpret_cast<const float2*>(sv + el * NQ * SV);
#pragma unroll 2
    for (int p = 0; p < NQ; ++p) {
      const float2 *va = base + p * SV + a * 3, *vb = base + p * SV + b * 3, *cq = base + p * SV + 24;
      const float2 a0 = va[0], a1 = va[1], a2 = va[2], b0 = vb[0], b1 = vb[1], b2 = vb[2], c0 = cq[0], c1 = cq[1];
      const float ga[3] = {a0.x, a0.y, a1.x}, na[3] = {a1.y, a2.x, a2.y};
      const float gb[3] = {b0.x, b0.y, b1.x}, nb[3] = {b1.y, b2.x, b2.y};
      float lg[3], mg[3], tn[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        lg[j] = c0.x * ga[j];
        mg[j] = c0.y * ga[j];
        tn[j] = -c1.x * na[j];
        dot = fmaf(mg[j], gb[j], dot);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[j][k] = fmaf(tn[j], nb[k], fmaf(mg[k], gb[j], fmaf(lg[j], gb[k], acc[j][k])));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) acc[j][j] += dot;
    // Ke[(a,j),(b,k)] -> CSR (row = dof(b,k), col = dof(a,j)) = slot(a,b) + k*rowLen(b) + j, and its transpose
    const int rb = srl[el * NN + b], ra = srl[el * NN + a];
    if (!in_bounds(g, slot, g.nnz, ee) || !in_bounds(g, slot + (int64_t)2 * (rb + 1), g.nnz, ee)) continue;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k) kadd(K + slot + (int64_t)k * rb + j, acc[j][k]);
    if (a == b) continue;
    if (!in_bounds(g, slot2, g.nnz, ee) || !in_bounds(g, slot2 + (int64_t)2 * (ra + 1), g.nnz, ee)) continue;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k) kadd(K + slot2 + (int64_t)j * ra + k, acc[j][k]);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Hexa20 with 3x3x3 points and an FP32 tangent, small strain or (TL) total-Lagrangian Neo-Hooke: two elements on four
// warps.  A point's row of shared memory holds the digits of dN/dX and then, in their place, the tangent's vectors; a
// thread forms the blocks of 2 x 2 nodes (14 loads of shared memory for 174 arithmetic instructions per point), and K_e goes
// to the CSR rows through shared memory, so that the lanes of a warp share the sectors that L2 adds to (the adds alone: 110
// us on 13824 elements, 264 us by node pairs).
//
// The Neo-Hooke tangent (displacementtlelement/element.py:408-412) takes two vectors per node too, h = F^-T dN/dX and
// g = F dN/dX: with c1 = sB and c3 = c4 in every variant, B h = g and dN_a/dX . dN_b/dX = h_a . g_b,
//   K_ab[j][k] = sum_q s (c2 h_a[j] h_b[k] + c3 (g_a[j] h_b[k] + h_a[j] g_b[k]) - sI h_a[k] h_b[j] + c1 delta_jk h_a . g_b).
//
// 13824 elements: small strain (von Mises) 675 -> 383 us, where a tensor-core tile (tcgen05, TF32 hi/lo) ran; TL 704 ->
// 463 us, mixed-ff 606 -> 463 us, against the same.  That tile's serial phases (operand conversion, FP64 update on one
// warp, MMA waits) with twelve warps per SM bound it, not the products; its tangent was 8e-7 off, this one 7e-8.  Here
// the issue slots (63 % used, small strain) and the waits of the phases with a thread per point bind.
template <bool TL>
struct Hexa20Layout {
  static constexpr int EPB = 2, NT = 128, NN = 20, NQ = 27, NDOF = 60, NP = EPB * NQ, NB = 55;  // NB: node blocks A <= B
  // a point's row in doublewords: 60 digits, then the floats (dN/dX, n dN/dX) of 20 nodes; odd
  static constexpr int SV = 61, DS = 9, SN = TL ? 21 : 9, SK = 61;
  static constexpr size_t v_off = 0;                            // fx [NP][SV]
  static constexpr size_t u_off = v_off + 8 * NP * SV;          // fx [EPB][NDOF]
  static constexpr size_t d_off = u_off + 8 * EPB * NDOF;       // int64 [NP][DS]: half of the strain (H); fx: s sigma (s P)
  static constexpr size_t k_bytes = 4 * EPB * NDOF * SK;        // K_e, in their place: float [EPB][NDOF][SK]
  static_assert(k_bytes <= d_off + 8 * NP * DS, "K_e fits the area of the operands");
  static constexpr size_t c_off = (d_off + 8 * NP * DS + 15) / 16 * 16;  // float4 [NP]: coefficients of the tangent
  // float [NP][SN]: flow direction, or F^-1 and F, and the units of dN/dX's digits
  static constexpr size_t n_off = c_off + 16 * NP;
  static constexpr size_t mc_off = (n_off + 4 * NP * SN + 15) / 16 * 16;  // VMConst [EPB]
  static constexpr size_t sl_off = mc_off + sizeof(VMConst) * EPB;        // int [EPB][NN][NN]: pair slots
  static constexpr size_t rl_off = sl_off + 4 * EPB * NN * NN;            // int [EPB][NN]: row lengths
  // int [4 warps][EPB][3]: an element's maxima; [EPB][3]: scales of dU, of the residual's rows
  static constexpr size_t e_off = rl_off + 4 * EPB * NN;
  static constexpr size_t bytes = e_off + 4 * 18 * EPB;
  // before the flow direction, in its place: int [NP][4]: a point's maxima (of 1, two halves of 2, of 3); [NP][3]: scales of
  // its dN/dX
  static_assert(SN >= 7, "scales in the place of the flow direction");
  static_assert(TL || 5 * (bytes + 1024) <= 196 * 1024, "the rest of the SM's 256 KB is L1 in steps: above this 28 KB instead of 60");
};

// Total-Lagrangian Neo-Hooke update of one point from H (displacementtlelement/element.py:386-414): state, strain, s P =
// s tau F^-T = s sB F + s sI F^-T, and for the tangent c = (c2, c3, -sI, c1) s and n = F^-1, F.
__device__ __forceinline__ void hexa20_neo_hooke(const GroupArgs& g, int64_t e, int64_t pt, int64_t stride, double s,
                                                 const double H[9], double sP[9], float4* c, float* n) {
  const double* props = g.props + e * g.nProps;
  double F[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) F[i][j] = (i == j ? 1.0 : 0.0) + H[i * 3 + j];
  // Green-Lagrange E = 1/2 (H + H^T + H^T H) (:386), order 11, 22, 33, 12, 23, 13
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const int i = f < 3 ? f : (f == 4 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
    const double E = 0.5 * ((H[i * 3 + j] + H[j * 3 + i]) + (H[i] * H[j] + H[3 + i] * H[3 + j] + H[6 + i] * H[6 + j]));
    g.auxTemp[(int64_t)f * stride + pt] = E;
    g.stateTemp[(int64_t)(6 + f) * stride + pt] = f < 3 ? E : 2.0 * E;
  }
  double iF[3][3];
  iF[0][0] = F[1][1] * F[2][2] - F[1][2] * F[2][1];
  iF[1][0] = F[1][2] * F[2][0] - F[1][0] * F[2][2];
  iF[2][0] = F[1][0] * F[2][1] - F[1][1] * F[2][0];
  const double J = F[0][0] * iF[0][0] + F[0][1] * iF[1][0] + F[0][2] * iF[2][0];
  iF[0][1] = F[0][2] * F[2][1] - F[0][1] * F[2][2];
  iF[0][2] = F[0][1] * F[1][2] - F[0][2] * F[1][1];
  iF[1][1] = F[0][0] * F[2][2] - F[0][2] * F[2][0];
  iF[1][2] = F[0][2] * F[1][0] - F[0][0] * F[1][2];
  iF[2][1] = F[0][1] * F[2][0] - F[0][0] * F[2][1];
  iF[2][2] = F[0][0] * F[1][1] - F[0][1] * F[1][0];
  const double rJ = 1.0 / J;
  double B[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const int i = f < 3 ? f : (f == 4 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
    B[f] = F[i][0] * F[j][0] + F[i][1] * F[j][1] + F[i][2] * F[j][2];
  }
  const NeoHookeScalars o =
      neo_hooke_scalars(g.material, props[0], props[1], J, B[0] + B[1] + B[2], F[0][0] + F[1][1] + F[2][2]);
  bool finite = true;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const double tau = f < 3 ? o.sB * B[f] + o.sI : o.sB * B[f];
    g.stateTemp[(int64_t)f * stride + pt] = tau;
    finite = finite && finite_bits(tau);
  }
  g.stateTemp[(int64_t)12 * stride + pt] = o.energy;
  if (!finite) atomicOr(g.status, EFE_STATUS_NONFINITE);
  const double aF = s * o.sB, aI = s * o.sI, aIJ = aI * rJ;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      sP[i * 3 + j] = fma(aIJ, iF[j][i], aF * F[i][j]);
      n[j * 3 + i] = ff_split_rn_bits(iF[j][i] * rJ).h;
      n[9 + i * 3 + j] = ff_split_rn_bits(F[i][j]).h;
    }
  *c = make_float4(ff_split_rn_bits(o.c2 * s).h, ff_split_rn_bits(o.c3 * s).h, ff_split_rn_bits(-aI).h,
                   ff_split_rn_bits(o.c1 * s).h);
}

template <bool TL>
__device__ __forceinline__ void assemble_tile_hexa20(const GroupArgs& g, const int64_t e0, unsigned char* smem) {
  using L = Hexa20Layout<TL>;
  constexpr int NN = L::NN, NQ = L::NQ, NDOF = L::NDOF, NP = L::NP, SV = L::SV, DS = L::DS, SN = L::SN, EPB = L::EPB, NT = L::NT;
  const double* Ux = TL ? g.U : g.dU;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  fx* sv = reinterpret_cast<fx*>(smem + L::v_off);
  fx* su = reinterpret_cast<fx*>(smem + L::u_off);
  int64_t* sde = reinterpret_cast<int64_t*>(smem + L::d_off);
  fx* sd = reinterpret_cast<fx*>(smem + L::d_off);
  float4* sc = reinterpret_cast<float4*>(smem + L::c_off);
  float* sn = reinterpret_cast<float*>(smem + L::n_off);
  VMConst* smc = reinterpret_cast<VMConst*>(smem + L::mc_off);
  int* sps = reinterpret_cast<int*>(smem + L::sl_off);
  int* srl = reinterpret_cast<int*>(smem + L::rl_off);
  int *sem = reinterpret_cast<int*>(sn), *semG = sem + 4 * NP;
  int *semD = reinterpret_cast<int*>(smem + L::e_off), *emu = semD + 12 * EPB, *ems = emu + 3 * EPB;
  const int64_t nEl = g.nElements, stride = nEl * NQ;
  const int nLoc = nEl - e0 < EPB ? (int)(nEl - e0) : EPB;
  const bool vm = g.material == EFE_MAT_VON_MISES;

  for (int t = tid; t < nLoc * NN * NN; t += NT) cp_async4(sps + t, g.pairSlot + e0 * NN * NN + t);
  // ---- dN/dX: two threads per point, 30 values each; dU relative to the element's first node: warps 0 and 1; the
  // material constants: two lanes of warp 3 that have no points
  {
    const int part = tid / NP, r = tid - part * NP;
    const bool live = part < 2 && r < nLoc * NQ;
    constexpr int H = NDOF / 2;
    double G[H];
    if (live) {
      const double* gp = g.geomG + (int64_t)(part * H) * stride + e0 * NQ + r;
#pragma unroll
      for (int i = 0; i < H; ++i) G[i] = gp[(int64_t)i * stride];
    }
    const int le = wid;
    if (le < EPB) {
      double u[3] = {0.0, 0.0, 0.0};
      const int64_t e = e0 + le;
      if (lane < NN && le < nLoc) {
        const int32_t node = g.conn[e * NN + lane], node0 = g.conn[e * NN];
        int rl = 0;
        if (in_bounds(g, node, g.nNodes, e) && in_bounds(g, node0, g.nNodes, e)) {
          rl = g.nodeRowLen[node];
          const int32_t dof = g.nodeDof[node], dof0 = g.nodeDof[node0];
          if (in_bounds(g, dof, g.nDof - 2, e) && in_bounds(g, dof0, g.nDof - 2, e)) {
#pragma unroll
            for (int c = 0; c < 3; ++c) u[c] = Ux[dof + c] - Ux[dof0 + c];
          }
        }
        srl[le * NN + lane] = rl;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int eu = __reduce_max_sync(0xffffffffu, fx_exponent(u[c]));
        if (lane < NN) su[le * NDOF + lane * 3 + c] = fx_make(u[c], eu);
        if (lane == 0) emu[le * 3 + c] = eu;
      }
    }
    // the first part's values are component 0 of all nodes and 1 of ten, the second's 1 of the others and 2 of all
    int em0 = 0, em1 = 0;
    if (live) {
      int m[3] = {0, 0, 0};
#pragma unroll
      for (int i = 0; i < H; ++i) m[i / 10] = fx_max_exponent(m[i / 10], G[i]);
      em0 = part ? m[0] : max(m[0], m[1]);
      em1 = part ? max(m[1], m[2]) : m[2];
      sem[r * 4 + part * 2] = em0;
      sem[r * 4 + part * 2 + 1] = em1;
    }
#pragma unroll
    for (int el = 0; el < EPB; ++el)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const bool mine = live && r / NQ == el && (c == 1 || c == 2 * part);
        const int m = __reduce_max_sync(0xffffffffu, mine ? (c == part ? em0 : em1) : 0);
        if (lane == 0) semD[(wid * EPB + el) * 3 + c] = m;
      }
    if (!TL && wid == 3 && lane >= 32 - nLoc) {
      const int k = 31 - lane;
      smc[k] = vm_const<true>(g.props + (e0 + k) * g.nProps, vm);
    }
    __syncthreads();
    if (live) {
      const int *pm = sem + r * 4, *dm = semD + r / NQ * 3;
      int D[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) D[c] = max(max(dm[c], dm[3 * EPB + c]), max(dm[6 * EPB + c], dm[9 * EPB + c]));
      const int t = max(max(pm[0] - D[0], max(pm[1], pm[2]) - D[1]), pm[3] - D[2]);
      if (part == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) semG[r * 3 + c] = D[c] + t;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const int la = part * H + i, c = la / NN, a = la - c * NN;
        sv[r * SV + a * 3 + c] = fx_make(G[i], (i < 10 ? (part ? D[1] : D[0]) : i < 20 ? (part ? D[2] : D[0]) : (part ? D[2] : D[1])) + t);
      }
    }
  }
  __syncthreads();

  // ---- strain increment (element.py:322): two warps per element, a lane per point, ten nodes each
  const int le = wid >> 1, half = wid & 1, pr = le * NQ + lane;
  const bool live = le < nLoc && lane < NQ;
  int eg[3] = {0, 0, 0}, eu[3] = {0, 0, 0};
  if (live)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      eg[c] = semG[pr * 3 + c];
      eu[c] = emu[le * 3 + c];
    }
  const int64_t e = e0 + le, pt = e * NQ + lane;
  const bool hasM = g.material != EFE_MAT_LINEAR_ELASTIC;
  constexpr int NS = TL ? 9 : 6;
  int64_t st[NS];
  double sig[6], kappa = 0.0, s = 0.0;
  if (live && half == 0) {
    if constexpr (!TL) {
#pragma unroll
      for (int f = 0; f < 6; ++f) sig[f] = g.stateRef[(int64_t)f * stride + pt];
      if (hasM) kappa = g.stateRef[(int64_t)12 * stride + pt];
    }
    s = g.geomS[pt];
  }
  if (live) {
    FxSum acc[9] = {};
    const fx *gp = sv + pr * SV + half * 30, *up = su + le * NDOF + half * 30;
#pragma unroll 5
    for (int a = 0; a < NN / 2; ++a) {
      const fx u[3] = {up[a * 3], up[a * 3 + 1], up[a * 3 + 2]}, G[3] = {gp[a * 3], gp[a * 3 + 1], gp[a * 3 + 2]};
      if constexpr (TL) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) fx_fma(acc[i * 3 + j], u[i], G[j]);
      } else {
        fx_fma(acc[0], G[0], u[0]);
        fx_fma(acc[1], G[1], u[1]);
        fx_fma(acc[2], G[2], u[2]);
        fx_fma(acc[3], G[1], u[0]);
        fx_fma(acc[4], G[2], u[0]);
        fx_fma(acc[5], G[2], u[1]);
        fx_fma(acc[6], G[0], u[1]);
        fx_fma(acc[7], G[0], u[2]);
        fx_fma(acc[8], G[1], u[2]);
      }
    }
#pragma unroll
    for (int f = 0; f < NS; ++f) {
      const int i = f < 3 ? f : (f == 5 ? 1 : 0), j = f < 3 ? f : (f == 3 ? 1 : 2);
      st[f] = fx_int(acc[f], -1);
      if (!TL && f >= 3) {
        int em = eg[j] + eu[i];
        st[f] = fx_add(st[f], em, fx_int(acc[f + 3], -1), eg[i] + eu[j]);
      }
      if (half) sde[pr * DS + f] = st[f];
    }
  }
  __syncthreads();

  // ---- material points: one warp of each element
  if (half == 0) {
    int es[3] = {0, 0, 0};
    double ss[NS] = {};  // s sigma, or s P = s tau F^-T
    if (live) {
      double de[NS];  // the strain increment, or H
#pragma unroll
      for (int f = 0; f < NS; ++f) {
        const int i = TL ? f / 3 : f < 3 ? f : (f == 5 ? 1 : 0), j = TL ? f % 3 : f < 3 ? f : (f == 3 ? 1 : 2);
        const int em = TL || f < 3 ? eg[j] + eu[i] : max(eg[j] + eu[i], eg[i] + eu[j]);
        de[f] = fx_value(st[f] + sde[pr * DS + f], em + 1);
      }
      if constexpr (TL) {
        hexa20_neo_hooke(g, e, pt, stride, s, de, ss, sc + pr, sn + pr * SN);
      } else {
        double eps[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) eps[f] = g.stateRef[(int64_t)(6 + f) * stride + pt];
        bool ok = true;
        TangentF32 T;
        if (vm)
          ok = von_mises_3d_f32(smc[le], sig, de, kappa, T);
        else
          linear_elastic_3d(smc[le], sig, de, T);
        bool finite = true;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
          g.stateTemp[(int64_t)f * stride + pt] = sig[f];
          g.stateTemp[(int64_t)(6 + f) * stride + pt] = eps[f] + de[f];
          finite = finite && finite_bits(sig[f]);
          ss[f] = s * sig[f];
          sn[pr * SN + f] = T.n[f];
        }
        if (hasM) g.stateTemp[(int64_t)12 * stride + pt] = kappa;
        if (!ok) report(g.status, EFE_STATUS_CUTBACK, g.elementOffset + e, 1);
        if (!finite) atomicOr(g.status, EFE_STATUS_NONFINITE);
        sc[pr] = make_float4(ff_split_rn_bits(T.c12 * s).h, ff_split_rn_bits(T.c44 * s).h, ff_split_rn_bits(T.a * s).h,
                             0.0f);
      }
#pragma unroll
      for (int f = 0; f < NS; ++f) {
        const int i = TL ? f / 3 : f < 3 ? f : (f == 5 ? 1 : 0), j = TL ? f % 3 : f < 3 ? f : (f == 3 ? 1 : 2);
        const int ef = fx_exponent(ss[f]);
        es[i] = max(es[i], ef + eg[j]);
        if (!TL) es[j] = max(es[j], ef + eg[i]);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      es[c] = __reduce_max_sync(0xffffffffu, es[c]);
      if (lane == 0) ems[le * 3 + c] = es[c];
    }
    if (live)
#pragma unroll
      for (int f = 0; f < NS; ++f) {
        if constexpr (TL)
          sd[pr * DS + f] = fx_make(ss[f], es[f / 3] - eg[f % 3]);
        else
          reinterpret_cast<double*>(sd)[pr * DS + f] = ss[f];
      }
  } else if (live) {
#pragma unroll
    for (int c = 0; c < 3; ++c) sn[pr * SN + SN - 3 + c] = fx_unit(eg[c]);
  }
  __syncthreads();
  // small strain: digits of the nine row factors by both warps (13824 elements: 12 us less than by one)
  if constexpr (!TL) {
    if (live) {
      const int es[3] = {ems[le * 3], ems[le * 3 + 1], ems[le * 3 + 2]};
#pragma unroll
      for (int f = 0; f < NS; ++f)
        if ((f >= 4) == half) row_digits(sd + pr * DS, reinterpret_cast<const double*>(sd)[pr * DS + f], f, es, eg, 0);
    }
    __syncthreads();
  }

  // ---- residual and flux (NIST.computeElements, nonlinearimplicitstatic.py:837-844): 60 threads per element
  {
    const int el = tid >> 6, k = tid & 63;
    if (k < NDOF && el < nLoc) {
      const int a = k / 3, c = k - 3 * a;
      const int64_t e = e0 + el;
      const int v0 = TL ? 3 * c : row_slot(c, 0), v1 = TL ? 3 * c + 1 : row_slot(c, 1), v2 = TL ? 3 * c + 2 : row_slot(c, 2);
      FxSum s[3] = {};  // one for each direction: 27 products
      const fx *gp = sv + el * NQ * SV + a * 3, *dp = sd + el * NQ * DS;
#pragma unroll 3
      for (int q = 0; q < NQ; ++q) {
        fx_fma(s[0], dp[q * DS + v0], gp[q * SV]);
        fx_fma(s[1], dp[q * DS + v1], gp[q * SV + 1]);
        fx_fma(s[2], dp[q * DS + v2], gp[q * SV + 2]);
      }
      const double pe = -fx_value(fx_int(s[0], -2) + fx_int(s[1], -2) + fx_int(s[2], -2), ems[el * 3 + c] + 2);
      const int32_t node = g.conn[e * NN + a];
      if (in_bounds(g, node, g.nNodes, e)) {
        const int32_t dof = g.nodeDof[node] + c;
        if (in_bounds(g, dof, g.nDof, e)) {
          atomicAdd(g.P + dof, pe);
          atomicAdd(g.F + dof, fabs(pe));
        }
      }
    }
  }
  __syncthreads();

  // ---- the tangent's vectors in the place of the digits (as in the Hexa8 tile)
  if (live) {
    const float *unit = sn + pr * SN + SN - 3, ux = unit[0], uy = unit[1], uz = unit[2];
    float n[TL ? 18 : 6];
#pragma unroll
    for (int f = 0; f < (TL ? 18 : 6); ++f) n[f] = sn[pr * SN + f];
    fx* row = sv + pr * SV + half * 30;
#pragma unroll 5
    for (int a = 0; a < NN / 2; ++a) {
      const float gx = fx_float(row[a * 3], ux), gy = fx_float(row[a * 3 + 1], uy), gz = fx_float(row[a * 3 + 2], uz);
      float x[6];
      if constexpr (TL) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          x[i] = n[i] * gx + n[3 + i] * gy + n[6 + i] * gz;                    // h = F^-T dN/dX
          x[3 + i] = n[9 + 3 * i] * gx + n[10 + 3 * i] * gy + n[11 + 3 * i] * gz;  // F dN/dX
        }
      } else {
        x[0] = gx, x[1] = gy, x[2] = gz;
        x[3] = n[0] * gx + n[3] * gy + n[4] * gz;
        x[4] = n[3] * gx + n[1] * gy + n[5] * gz;
        x[5] = n[4] * gx + n[5] * gy + n[2] * gz;
      }
      float2* v = reinterpret_cast<float2*>(row + a * 3);
      v[0] = make_float2(x[0], x[1]);
      v[1] = make_float2(x[2], x[3]);
      v[2] = make_float2(x[4], x[5]);
    }
  }
  __syncthreads();

  // ---- tangent: blocks of the nodes (2A, 2A + 1) x (2B, 2B + 1), A <= B, 64 threads per element
  const int el = tid >> 6;
  int B = tid & 63, A = 0;
  const bool has = B < L::NB && el < nLoc;
  float acc[2][2][3][3] = {};
  if (has) {
    while (B >= NN / 2 - A) {
      B -= NN / 2 - A;
      ++A;
    }
    B += A;
    float dot[2][2] = {};
    const float2* base = reinterpret_cast<const float2*>(sv + el * NQ * SV);
#pragma unroll 1
    for (int q = 0; q < NQ; ++q) {
      float ga[2][3], na[2][3], gb[2][3], nb[2][3];
      const float4 c = sc[el * NQ + q];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 *va = base + q * SV + (2 * A + x) * 3, *vb = base + q * SV + (2 * B + x) * 3;
        const float2 a0 = va[0], a1 = va[1], a2 = va[2], b0 = vb[0], b1 = vb[1], b2 = vb[2];
        ga[x][0] = a0.x, ga[x][1] = a0.y, ga[x][2] = a1.x, na[x][0] = a1.y, na[x][1] = a2.x, na[x][2] = a2.y;
        gb[x][0] = b0.x, gb[x][1] = b0.y, gb[x][2] = b1.x, nb[x][0] = b1.y, nb[x][1] = b2.x, nb[x][2] = b2.y;
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float lg[3], mg[3], tn[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          lg[j] = TL ? fmaf(c.y, na[x][j], c.x * ga[x][j]) : c.x * ga[x][j];
          mg[j] = (TL ? c.z : c.y) * ga[x][j];
          tn[j] = TL ? c.y * ga[x][j] : -c.z * na[x][j];
        }
#pragma unroll
        for (int y = 0; y < 2; ++y) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            dot[x][y] = TL ? fmaf(c.w * ga[x][j], nb[y][j], dot[x][y]) : fmaf(mg[j], gb[y][j], dot[x][y]);
#pragma unroll
            for (int k = 0; k < 3; ++k)
              acc[x][y][j][k] += fmaf(tn[j], nb[y][k], fmaf(mg[k], gb[y][j], lg[j] * gb[y][k]));
          }
        }
      }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int j = 0; j < 3; ++j) acc[x][y][j][j] += dot[x][y];
  }
  cp_async_wait_all();
  __syncthreads();

  // ---- K_e[(b, k)][(a, j)] over the operands (the element tangents are symmetric), then a warp per node b: its three
  // CSR rows, 30 lanes for the columns (a, j) of ten nodes: slot(a, b) + k rowLen(b) + j
  float* sK = reinterpret_cast<float*>(smem) + el * NDOF * L::SK;
  if (has) {
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int ca = (2 * A + x) * 3 + j, cb = (2 * B + y) * 3 + k;
            sK[cb * L::SK + ca] = acc[x][y][j][k];
            if (A != B) sK[ca * L::SK + cb] = acc[x][y][j][k];
          }
  }
  __syncthreads();
  {
    float* K = reinterpret_cast<float*>(g.Kdata);
    const int a0 = lane / 3, j = lane - 3 * a0;
    if (lane < 30) {
      for (int t = wid; t < nLoc * NN; t += NT / 32) {
        const int m = t / NN, b = t - m * NN, rl = srl[m * NN + b];
        const int64_t e = e0 + m;
        const float* row = reinterpret_cast<const float*>(smem) + (m * NDOF + 3 * b) * L::SK;
#pragma unroll
        for (int a = a0; a < NN; a += 10) {
          const int32_t slot = sps[(m * NN + a) * NN + b];
          if (!in_bounds(g, slot, g.nnz, e) || !in_bounds(g, slot + (int64_t)2 * (rl + 1), g.nnz, e)) continue;
#pragma unroll
          for (int k = 0; k < 3; ++k) atomicAdd(K + slot + (int64_t)k * rl + j, row[k * L::SK + 3 * a + j]);
        }
      }
    }
  }
}

}  // namespace efe
