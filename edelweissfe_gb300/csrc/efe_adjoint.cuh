// efe_adjoint.cuh -- adjoint of the total-Lagrangian hyperelastic element residual.
//
// For L = lambda^T P(X, U, mu, K), with P the element residual of DisplacementTLElement with a
// Neo-Hooke material (displacementtlelement/element.py:389-414: P_a -= s tau h_a, s = det J w t,
// h_a = F^-T dN_a/dX, tau the Kirchhoff stress), the kernel returns dL/dX (nodal reference
// coordinates) and dL/dmu, dL/dK per element, by reverse-mode differentiation written out by hand:
//
//   L = -s phi,  phi = P : Lambda,  Lambda = sum_a lambda_a (x) dN_a/dX
//   P = tau F^-T = sB F + sI F^-T = dphi/dLambda,  tau = sB B + sI I  (sB = c1 for every variant)
//   dphi/dF  = c1 Lambda + (c2 F^-T : Lambda + c3 F : Lambda) F^-T + c4 (F^-T : Lambda) F
//              - sI F^-T Lambda^T F^-T
// (the terms c1 M^T F and F^-T Lambda^T sB B F^-T, M = Lambda F^-1, cancel), then through
// F = I + H, H = sum_a U_a (x) G_a, and Lambda to G = J^-1 dN/dxi, and through J = dN/dxi . X (with the
// Hexa20 third-row term of the reference) and s = det J w t to X:
//   dL/dJ = s J^-T (dphi/dF^T H + P^T Lambda - phi I)
// Parameter derivatives use dtau/dmu, dtau/dK of each variant.
//
// The sums over the nodes (J, and H and Lambda before their product with J^-T) and the element's nodal sums of
// dL/dJ dN/dxi run in fixed-point integers (efe_fixed.cuh), H and Lambda also through that product: the FP64 pipe, which
// binds the kernel, is left with about 380 instructions per point.  Each component of the nodal values, of J^-T and of
// dL/dJ has a scale of its own: in thin elements they differ in size.  Nodal values are staged once per element, relative
// to its first node (sum_a dN_a = 0), and dN/dxi once per CTA, whose elements are strided by the grid.  Four CTAs per
// SM (128 registers): 32768 C3D8TL elements in 227 us, about 160 of them the FP64 pipe's, against 486 with float-float
// sums and products by M; 2048 C3D20TL 122 against 282 us; 20000 CPE8RTL 52 against 108 us.
#pragma once
#include "efe_launch.cuh"

namespace efe {

// d tau / d mu = aB B + aI I and d tau / d K = bI I of the three Neo-Hooke variants (of neo_hooke_scalars)
__device__ inline void neo_hooke_param_derivatives(int material, double mu, double K, double J, double I1, double& aB,
                                                   double& aI, double& bI) {
  if (material == EFE_MAT_NEOHOOKE_WA) {
    aB = 1.0;
    aI = -(2.0 / 3.0) * (J * J - J) - 1.0;
    bI = J * J - J;
  } else if (material == EFE_MAT_NEOHOOKE_WB) {
    const double J23 = pow(J, 2.0 / 3.0);
    aB = 1.0 / J23;
    aI = -I1 / (3.0 * J23);
    bI = (J * J - 1.0 / (J * J)) / 4.0;
  } else {
    const double p = pow(J, 2.0 / 3.0 - K / mu);
    const double lnJ = log(J);
    aB = 1.0;
    aI = -p * (1.0 + (K / mu) * lnJ);
    bI = p * lnJ;
  }
}

// Elements and shared memory of a CTA of 128 threads, a thread per point.
template <int SHAPE, int RULE>
struct AdjointTLLayout {
  static constexpr int DIM = ShapeInfo<SHAPE>::DIM, NN = ShapeInfo<SHAPE>::NN, NQ = RuleInfo<RULE>::NQ, NDOF = DIM * NN;
  static constexpr int NT = 128, EPB = NT / NQ < 32 ? NT / NQ : 32, NP = EPB * NQ;
  // the Hexa20 Jacobian's third row differs from dN/dxi's: a row of its own
  static constexpr int ROWS = SHAPE == EFE_HEXA20 ? 4 : DIM, DS = (ROWS * NN) | 1, JS = (DIM * DIM) | 1, XS = (3 * NDOF) | 1;
  static constexpr size_t d_off = 0;                          // fx [NQ][DS]: dN/dxi
  static constexpr size_t x_off = d_off + 8 * NQ * DS;        // double, then fx [EPB][XS: X, U, lambda][NN][DIM]
  static constexpr size_t j_off = x_off + 8 * EPB * XS;       // double, then fx [NP][JS]: dL/dJ
  static constexpr int ES = 4 * DIM;                          // scales of an element: components of X, U, lambda, dL/dJ
  static constexpr size_t e_off = j_off + 8 * NP * JS;        // int [EPB][ES], [1] dN/dxi
  static constexpr size_t bytes = e_off + 4 * (ES * EPB + 1);
  static_assert(NN <= 31 && NQ <= 31, "products of a fixed-point sum");
};

// cofactor matrix of A / det A, transposed: the inverse; 2D blocks carry A[2][2] = 1
template <int DIM>
__device__ __forceinline__ double adjoint_inverse(const double A[3][3], double B[3][3]) {
  if constexpr (DIM == 2) {
    const double d = A[0][0] * A[1][1] - A[0][1] * A[1][0], r = 1.0 / d;
    B[0][0] = A[1][1] * r;
    B[0][1] = -A[0][1] * r;
    B[1][0] = -A[1][0] * r;
    B[1][1] = A[0][0] * r;
    return d;
  } else {
    B[0][0] = A[1][1] * A[2][2] - A[1][2] * A[2][1];
    B[1][0] = A[1][2] * A[2][0] - A[1][0] * A[2][2];
    B[2][0] = A[1][0] * A[2][1] - A[1][1] * A[2][0];
    const double d = A[0][0] * B[0][0] + A[0][1] * B[1][0] + A[0][2] * B[2][0], r = 1.0 / d;
    B[0][0] *= r;
    B[1][0] *= r;
    B[2][0] *= r;
    B[0][1] = (A[0][2] * A[2][1] - A[0][1] * A[2][2]) * r;
    B[0][2] = (A[0][1] * A[1][2] - A[0][2] * A[1][1]) * r;
    B[1][1] = (A[0][0] * A[2][2] - A[0][2] * A[2][0]) * r;
    B[1][2] = (A[0][2] * A[1][0] - A[0][0] * A[1][2]) * r;
    B[2][1] = (A[0][1] * A[2][0] - A[0][0] * A[2][1]) * r;
    B[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * r;
    return d;
  }
}

// gX is [nNodes][dim], gP is [nElements][2] (mu, K); both are accumulated into (the caller zeroes them).
template <int SHAPE, int RULE>
__global__ void __launch_bounds__(128, 4) adjoint_tl_kernel(AdjointArgs ar) {
  using L = AdjointTLLayout<SHAPE, RULE>;
  constexpr int DIM = L::DIM, NN = L::NN, NQ = L::NQ, NDOF = L::NDOF, NT = L::NT, EPB = L::EPB, DS = L::DS, JS = L::JS,
                XS = L::XS, ES = L::ES;
  extern __shared__ __align__(16) unsigned char smem[];
  fx* sD = reinterpret_cast<fx*>(smem + L::d_off);
  double* sXd = reinterpret_cast<double*>(smem + L::x_off);
  fx* sX = reinterpret_cast<fx*>(smem + L::x_off);
  double* sJd = reinterpret_cast<double*>(smem + L::j_off);
  fx* sJ = reinterpret_cast<fx*>(smem + L::j_off);
  int* sem = reinterpret_cast<int*>(smem + L::e_off);
  int* semD = sem + ES * EPB;
  const int tid = threadIdx.x;
  const int le = tid / NQ, q = tid - le * NQ;
  double xi, eta, zeta, w;
  quadrature_point(RULE, q, xi, eta, zeta, w);
  // Jacobian table row 2 of Hexa20 carries (zeta - xi) * inv(A)[5] (the reference's _J3D20); that
  // row does not sum to zero over the nodes, so its sum times X_0 is added back in FP64
  const double quirk = (SHAPE == EFE_HEXA20) ? (zeta - xi) : 0.0;
  double rs = 0.0;
  if constexpr (SHAPE == EFE_HEXA20)
    for (int a = 0; a < NN; ++a) rs += ar.fix.r[a % 20];
  if (tid == 0) *semD = 0;
  __syncthreads();
  {
    const double p[3] = {eta, xi, zeta};
    double D[L::ROWS][NN];
    if (tid < NQ) {
      shape_derivatives<SHAPE>(p, D);
      int em = 0;
      if constexpr (SHAPE == EFE_HEXA20)
        for (int a = 0; a < NN; ++a) D[3][a] = D[2][a] + quirk * ar.fix.r[a % 20];
#pragma unroll
      for (int r = 0; r < L::ROWS; ++r)
#pragma unroll
        for (int a = 0; a < NN; ++a) em = max(em, fx_exponent(D[r][a]));
      atomicMax(semD, em);
    }
    __syncthreads();
    if (tid < NQ) {
#pragma unroll
      for (int r = 0; r < L::ROWS; ++r)
#pragma unroll
        for (int a = 0; a < NN; ++a) sD[q * DS + a * L::ROWS + r] = fx_make(D[r][a], *semD);
    }
  }

  for (int64_t e0 = (int64_t)blockIdx.x * EPB; e0 < ar.nEl; e0 += (int64_t)gridDim.x * EPB) {
    const int nLoc = ar.nEl - e0 < EPB ? (int)(ar.nEl - e0) : EPB;
    for (int t = tid; t < ES * EPB; t += NT) sem[t] = 0;
    __syncthreads();
    // ---- nodal values relative to the element's first node
    for (int t = tid; t < nLoc * NN; t += NT) {
      const int l = t / NN, a = t - l * NN;
      const int32_t* en = ar.conn + (e0 + l) * NN;
      const int64_t n = en[a], n0 = en[0];
      const int64_t dof = ar.nodeDof[n], dof0 = ar.nodeDof[n0];
      double v[3][DIM];
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        v[0][c] = ar.coords[n * DIM + c] - ar.coords[n0 * DIM + c];
        v[1][c] = ar.U[dof + c] - ar.U[dof0 + c];
        v[2][c] = ar.lam[dof + c] - ar.lam[dof0 + c];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          sXd[l * XS + k * NDOF + a * DIM + c] = v[k][c];
          atomicMax(sem + l * ES + k * DIM + c, fx_exponent(v[k][c]));
        }
    }
    __syncthreads();
    for (int t = tid; t < nLoc * 3 * NDOF; t += NT) {
      const int l = t / (3 * NDOF), r = t - l * 3 * NDOF;
      sX[l * XS + r] = fx_make(sXd[l * XS + r], sem[l * ES + r / NDOF * DIM + r % DIM]);
    }
    __syncthreads();

    // ---- a thread per point
    const int64_t e = e0 + le;
    const bool live = le < nLoc;
    if (live) {
      const int emD = *semD;
      int* el = sem + le * ES;
      // sum_a v_a[c] D[r][a] as integers, V[c][r]
      auto nodal = [&](int k, int row2, FxSum V[DIM][DIM]) {
#pragma unroll
        for (int c = 0; c < DIM; ++c)
#pragma unroll
          for (int r = 0; r < DIM; ++r) V[c][r] = FxSum{0, 0};
        const fx *xp = sX + le * XS + k * NDOF, *dp = sD + q * DS;
#pragma unroll 4
        for (int a = 0; a < NN; ++a) {
          fx d[DIM];
#pragma unroll
          for (int r = 0; r < DIM; ++r) d[r] = dp[a * L::ROWS + (r == 2 ? row2 : r)];
#pragma unroll
          for (int c = 0; c < DIM; ++c) {
            const fx x = xp[a * DIM + c];
#pragma unroll
            for (int r = 0; r < DIM; ++r) fx_fma(V[c][r], x, d[r]);
          }
        }
      };
      double J[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 1}}, iJ[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 1}};
      {
        FxSum V[DIM][DIM];
        nodal(0, L::ROWS - 1, V);
#pragma unroll
        for (int c = 0; c < DIM; ++c)
#pragma unroll
          for (int r = 0; r < DIM; ++r) J[r][c] = fx_value(fx_int(V[c][r]), emD + el[c]);
      }
      if constexpr (SHAPE == EFE_HEXA20) {
        const int64_t n0 = ar.conn[e * NN];
#pragma unroll
        for (int c = 0; c < DIM; ++c) J[2][c] += quirk * rs * ar.coords[n0 * DIM + c];
      }
      const double detJ = adjoint_inverse<DIM>(J, iJ);
      // H and Lambda: the nodal sums times J^-T
      double F[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}, H[DIM][DIM], Lam[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
      {
        int ei[DIM];
        fx iJf[DIM][DIM];
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          ei[c] = 0;
#pragma unroll
          for (int r = 0; r < DIM; ++r) ei[c] = max(ei[c], fx_exponent(iJ[c][r]));
#pragma unroll
          for (int r = 0; r < DIM; ++r) iJf[c][r] = fx_make(iJ[c][r], ei[c]);
        }
        constexpr int B = NN > 8 ? 5 : (NN > 4 ? 4 : 3);  // |sum| <= NN 2^58 as an operand of 57 bits
#pragma unroll
        for (int k = 1; k < 3; ++k) {
          FxSum V[DIM][DIM];
          nodal(k, 2, V);
#pragma unroll
          for (int i = 0; i < DIM; ++i) {
            const int em = emD + el[k * DIM + i] - 1023 + B;  // the operand's scale: its value is V 2^(em - 1079)
            fx v[DIM];
#pragma unroll
            for (int r = 0; r < DIM; ++r) v[r] = fx_split(fx_int(V[i][r], -B));
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
              FxSum t{0, 0};
#pragma unroll
              for (int r = 0; r < DIM; ++r) fx_fma(t, v[r], iJf[j][r]);
              const double x = fx_value(fx_int(t), em + ei[j]);
              if (k == 1) {
                H[i][j] = x;
                F[i][j] += x;
              } else {
                Lam[i][j] = x;
              }
            }
          }
        }
      }
      const double th = (DIM == 2 && ar.thickness) ? ar.thickness[e] : 1.0;
      const double s = detJ * w * th;
      double iF[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 1}};
      const double Jf = adjoint_inverse<DIM>(F, iF);
      double I1 = DIM == 2 ? 1.0 : 0.0, trM = 0.0, MB = 0.0;  // F : F, F^-T : Lambda, F : Lambda
#pragma unroll
      for (int i = 0; i < DIM; ++i)
#pragma unroll
        for (int j = 0; j < DIM; ++j) {
          I1 = fma(F[i][j], F[i][j], I1);
          trM = fma(iF[j][i], Lam[i][j], trM);
          MB = fma(F[i][j], Lam[i][j], MB);
        }
      const double mu = ar.props[e * ar.nProps + 0], Kb = ar.props[e * ar.nProps + 1];
      const NeoHookeScalars o = neo_hooke_scalars(ar.material, mu, Kb, Jf, I1, F[0][0] + F[1][1] + F[2][2]);
      const double phi = o.sB * MB + o.sI * trM;
      {
        double aB, aI, bI;
        neo_hooke_param_derivatives(ar.material, mu, Kb, Jf, I1, aB, aI, bI);
        atomicAdd(ar.gP + 2 * e + 0, -s * (aB * MB + aI * trM));
        atomicAdd(ar.gP + 2 * e + 1, -s * (bI * trM));
      }
      // E = s (dphi/dF^T H + P^T Lambda - phi I), a row i of dphi/dF and P at a time
      double E[DIM][DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k)
#pragma unroll
        for (int c = 0; c < DIM; ++c) E[k][c] = k == c ? -phi : 0.0;
      const double cI = o.c2 * trM + o.c3 * MB, cF = o.c4 * trM;
#pragma unroll
      for (int i = 0; i < DIM; ++i) {
        double T[DIM];  // row i of F^-T Lambda^T
#pragma unroll
        for (int l = 0; l < DIM; ++l) {
          T[l] = 0.0;
#pragma unroll
          for (int m = 0; m < DIM; ++m) T[l] = fma(iF[m][i], Lam[l][m], T[l]);
        }
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          double Q = 0.0;
#pragma unroll
          for (int l = 0; l < DIM; ++l) Q = fma(T[l], iF[k][l], Q);
          const double fb = fma(o.c1, Lam[i][k], fma(cI, iF[k][i], fma(cF, F[i][k], -o.sI * Q)));
          const double P = fma(o.sB, F[i][k], o.sI * iF[k][i]);
#pragma unroll
          for (int c = 0; c < DIM; ++c) E[k][c] = fma(fb, H[i][c], fma(P, Lam[i][c], E[k][c]));
        }
      }
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        int ej = 0;
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          double v = 0.0;
#pragma unroll
          for (int k = 0; k < DIM; ++k) v = fma(iJ[k][r], E[k][c], v);
          v *= s;
          sJd[tid * JS + r * DIM + c] = v;
          ej = max(ej, fx_exponent(v));
        }
        atomicMax(el + 3 * DIM + c, ej);
      }
    }
    __syncthreads();
    if (live) {
#pragma unroll
      for (int k = 0; k < DIM * DIM; ++k) sJ[tid * JS + k] = fx_make(sJd[tid * JS + k], sem[le * ES + 3 * DIM + k % DIM]);
    }
    __syncthreads();
    // ---- the element's nodal sums: gX[a][c] += sum_q sum_r dL/dJ[r][c] D[r][a]
    for (int t = tid; t < nLoc * NDOF; t += NT) {
      const int l = t / NDOF, k = t - l * NDOF, a = k / DIM, c = k - a * DIM;
      FxSum acc[DIM] = {};
      for (int p = 0; p < NQ; ++p)
#pragma unroll
        for (int r = 0; r < DIM; ++r)
          fx_fma(acc[r], sJ[(l * NQ + p) * JS + r * DIM + c], sD[p * DS + a * L::ROWS + (r == 2 ? L::ROWS - 1 : r)]);
      int64_t v = 0;
#pragma unroll
      for (int r = 0; r < DIM; ++r) v += fx_int(acc[r], -2);
      atomicAdd(ar.gX + (int64_t)ar.conn[(e0 + l) * NN + a] * DIM + c, fx_value(v, *semD + sem[l * ES + 3 * DIM + c] + 2));
    }
    __syncthreads();
  }
}

template <int SHAPE, int RULE>
cudaError_t launch_adjoint_tl(const AdjointArgs& a, cudaStream_t st) {
  using L = AdjointTLLayout<SHAPE, RULE>;
  if (a.nEl == 0) return cudaSuccess;
  auto kern = adjoint_tl_kernel<SHAPE, RULE>;
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::bytes);
  if (err != cudaSuccess) return err;
  int dev = 0, sms = 0, perSM = 0;
  if ((err = cudaGetDevice(&dev)) != cudaSuccess) return err;
  if ((err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return err;
  if ((err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kern, L::NT, L::bytes)) != cudaSuccess) return err;
  if (perSM < 1) return cudaErrorInvalidConfiguration;
  const int64_t tiles = (a.nEl + L::EPB - 1) / L::EPB;
  kern<<<(unsigned)std::min<int64_t>(tiles, (int64_t)sms * perSM), L::NT, L::bytes, st>>>(a);
  return cudaGetLastError();
}

}  // namespace efe
