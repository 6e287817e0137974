// efe_pcg.cu -- preconditioned conjugate gradients as one persistent kernel (efe_pcg_iterate,
// efe_pcg_solve): the Newton correction (the reference's linearSolve,
// solvers/nonlinearimplicitstatic.py:727-751) and the adjoint systems.
//
// One cooperative launch of one CTA per SM (small systems: one cluster) runs many iterations.  An iteration has
// two phases, with a sum over the grid behind the first and a grid barrier behind the second:
//   A  Ap = A p and the sums p.Ap, Ap.M^-1 Ap
//   B  x += alpha p, r -= alpha Ap, z = M^-1 r, p = z + beta p, and the sum r.z
// alpha = r.z / p.Ap needs the sums of A; so does beta, predicted as beta = alpha (Ap.M^-1 Ap) / p.Ap - 1 (from
// r_new.z_new = alpha^2 Ap.M^-1 Ap - r.z), while the r.z of the next alpha is the sum formed in B (G. Meurant,
// "Multitasking the conjugate gradient method on the CRAY X-MP/48", Parallel Computing 5, 1987; T. Chen and
// E. Carson, "Predict-and-recompute conjugate gradient variants", SIAM J. Sci. Comput. 42, 2020, measure the same
// convergence as the two-sum form).  That takes one of three synchronisations and a pass over p and z out of the
// iteration.  Every CTA sums the partials of all CTAs in the same order, so a solve is bitwise repeatable.
//
// Phase A is bound by the matrix stream and the issue rate (FP32 values) or by the FP64 pipe (FP64 values: this
// part issues FP64 at 1/64 of its FP32 rate, 16 cycles of an SM per warp instruction).  The rows of a chunk of
// consecutive nodes are one contiguous range of the CSR data: a warp fetches its next chunk with bulk copies into
// shared memory while the other warps work on theirs, which keeps the stream going without registers (the first
// chunks of the next product arrive under phase B's barrier: K does not change).  PB > 1: the PB rows of a node
// share one list of node blocks of PB columns (4 / PB^2 bytes of column index per entry instead of 4, one gather of
// PB consecutive values of p per block).  LPG lanes work on one node's rows.
//
// Precision: FP32 tangents multiply in float-float arithmetic against p held as float pairs (~48 bits, ff_madd),
// FP64 tangents in FP64; vectors and scalars are FP64.
//
// Measured (a solve's time by its iterations, set-up included; before: a product, an update and a direction kernel per
// iteration, replayed as a graph): 64^3 Hexa8, FP32 values 208 -> 75 us (phase A 55 us for 288 MB, 5.2 TB/s; the two
// synchronisations 8, B 10), 32^3 Hexa8, FP64 values 56 -> 31 us (phase A 16 us, its FP64 work alone 15); 40 x 8 plate 16.0
// -> 6.0 us; Hexa20, whose corner nodes' chunks are longer than a copy, 24 x 24 x 12, FP32 48 -> 43 us, FP64 76 -> 53.
//
// The grid's scalars lie in slots of their epoch (efe_pcg_slots.cuh).  Every wait is bounded; one that gives up (about two
// seconds) ends the launch with work[5] = -1.
#include "efe_launch.cuh"
#include "efe_pcg_slots.cuh"

#include <type_traits>

namespace efe {

namespace {

// work layout (doubles): [0..1] r.z by iteration parity, [2] r.r, [3] p.Ap, [4] arrival counters,
// [5] 1 when the solve has ended (-1: a wait gave up), [6] iterations run, [7] 1 when the last test asked to
// stop, [8 ..) the slots (efe_pcg_slots.cuh)
constexpr int PART0 = 8, MAX_GRID = 512;
static_assert(PART0 + pcg_slots(MAX_GRID) * PCG_SLOT_DOUBLES <= EFE_PCG_WORK_DOUBLES, "work layout");
static_assert(sizeof(ulonglong2) == PCG_SLOT_DOUBLES * sizeof(double), "a slot");
constexpr int MAX_WARPS = 16;
constexpr int MAX_CLUSTER = 8;
constexpr int BARRIER_LIMIT = 1 << 22;  // polls of another CTA's arrival (about two seconds) before it gives up
constexpr int COPY_LIMIT = 1 << 22;     // polls of a bulk copy's completion

struct CgArgs {
  int64_t n;
  const int32_t* indptr;
  const int32_t* cols;  // column of every entry (PB = 1) or first column of every node block
  const void* K;
  const uint8_t* freeMask;
  const double* dinv;
  double *x, *r, *p, *Ap;
  float2* pf;
  double* work;
  int64_t k0;
  int nIter, every;  // every > 0: test the residual each `every` iterations
  double tol2;
  int capK, capC;  // bytes of a warp's copy (values, columns)
};

// ---------------------------------------------------------------- float-float (as in efe_solve.cu)
__device__ __forceinline__ void ff_acc(float& h, float& l, float a, float b) {
  const float s = __fadd_rn(h, a);
  const float bb = __fsub_rn(s, h);
  const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fsub_rn(a, bb));
  l = __fadd_rn(l, __fadd_rn(err, b));
  h = s;
}
__device__ __forceinline__ void ff_madd(float& h, float& l, float k, float xh, float xl) {
  const float p = __fmul_rn(k, xh);
  float e = __fmaf_rn(k, xh, -p);
  e = __fmaf_rn(k, xl, e);
  ff_acc(h, l, p, e);
}

// ---------------------------------------------------------------- copies
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// global -> shared, both 16-byte aligned, bytes a multiple of 16; policy: the L2 eviction priority
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
      : "memory");
}

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------- scalars across the grid
// Slot of one CTA: the two halves of a double, each with the epoch it belongs to in the same 8-byte word: a
// reader that sees both epochs has the whole value, without fences.
__device__ __forceinline__ void post(ulonglong2* slot, double v, uint32_t epoch) {
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&slot->x), "l"((b << 32) | epoch) : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&slot->y), "l"((b & 0xffffffff00000000ull) | epoch) : "memory");
}
__device__ __forceinline__ void arrive(uint32_t* counter) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
}
// polls the counter until it reaches target; false: gave up
__device__ __forceinline__ bool await(const uint32_t* counter, uint32_t target) {
  uint32_t seen = 0;
  int it = 0;
#pragma unroll 1
  for (; it < BARRIER_LIMIT; ++it) {
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
    if ((int32_t)(seen - target) >= 0) break;
  }
  return it < BARRIER_LIMIT;
}
// CTAs of one cluster: a barrier that also makes their global writes visible to each other, and a store into
// another CTA's copy of a shared variable.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void store_remote(double* p, int cta, double v) {
  uint32_t addr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_addr(p)), "r"(cta));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
// Sum over the slots of all CTAs in slot order by a warp (every lane gets it); false: gave up.  The caller has
// seen every CTA arrive, so the values are there or on their way, and stay until the caller's own next arrival.
__device__ __forceinline__ bool gather_sum(const ulonglong2* slots, int nSlots, uint32_t epoch, int lane, double& sum) {
  double v = 0.0;
  bool ok = true;
#pragma unroll 1
  for (int i0 = lane; i0 < nSlots; i0 += 32 * 5) {
    uint64_t x[5], y[5];
#pragma unroll
    for (int u = 0; u < 5; ++u) {  // up to 160 slots in flight
      const int i = i0 + 32 * u;
      x[u] = y[u] = epoch;
      if (i < nSlots) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x[u]) : "l"(&slots[i].x) : "memory");
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(y[u]) : "l"(&slots[i].y) : "memory");
      }
    }
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int i = i0 + 32 * u;
      int it = 0;
#pragma unroll 1
      for (; ((uint32_t)x[u] != epoch || (uint32_t)y[u] != epoch) && it < BARRIER_LIMIT; ++it) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x[u]) : "l"(&slots[i].x) : "memory");
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(y[u]) : "l"(&slots[i].y) : "memory");
      }
      if (it == BARRIER_LIMIT) ok = false;
      if (i < nSlots) v += __longlong_as_double((long long)((x[u] >> 32) | (y[u] & 0xffffffff00000000ull)));
    }
  }
  sum = warp_sum(v);
  return __all_sync(0xffffffffu, ok);
}

// z = M^-1 r on one block of BS consecutive DOFs (BS = 1: point Jacobi; 2, 3: the inverse of the
// node's diagonal block, [BS][BS] row-major per block)
template <int BS>
__device__ __forceinline__ void precondition(const double* dinv, const double r[BS], double z[BS]) {
#pragma unroll
  for (int i = 0; i < BS; ++i) {
    double v = 0.0;
#pragma unroll
    for (int j = 0; j < BS; ++j) v = fma(dinv[i * BS + j], r[j], v);
    z[i] = v;
  }
}

// The rows a CTA owns in phase B: slabs of R consecutive rows, (k gridDim + blockIdx) R.
struct Slab {
  int n, R;
  __device__ __forceinline__ int row(int i) const {
    const int k = i / R;
    return (k * (int)gridDim.x + (int)blockIdx.x) * R + (i - k * R);
  }
  // one past the last index i of this CTA
  __device__ __forceinline__ int count() const {
    const int per = (int)gridDim.x * R, full = n / per, rest = n - full * per - (int)blockIdx.x * R;
    return full * R + (rest < 0 ? 0 : (rest < R ? rest : R));
  }
};

// Ap . M^-1 Ap over this CTA's rows (BS > 1; with BS = 1 the product's epilogue forms it).
template <int BS>
__device__ __forceinline__ double preconditioned_norm(const CgArgs& a, const Slab& sl) {
  double w = 0.0;
  const int nb = sl.count() / BS;
#pragma unroll 1
  for (int k = threadIdx.x; k < nb; k += blockDim.x) {
    const int row = sl.row(k * BS);
    double q[BS], t[BS], d[BS * BS];
#pragma unroll
    for (int c = 0; c < BS; ++c) q[c] = a.Ap[row + c];
#pragma unroll
    for (int c = 0; c < BS * BS; ++c) d[c] = a.dinv[(int64_t)row * BS + c];
    precondition<BS>(d, q, t);
#pragma unroll
    for (int c = 0; c < BS; ++c) w = fma(q[c], t[c], w);
  }
  return w;
}

template <bool FF>
__device__ __forceinline__ void store_p(const CgArgs& a, int i, double v) {
  a.p[i] = v;
  if constexpr (FF) {
    const ff h = ff_split_rn_bits(v);
    a.pf[i] = make_float2(h.h, h.l);
  }
}

// Phase B over this CTA's rows; with known == false beta is not known yet and p stays.
template <int BS, bool FF>
__device__ __forceinline__ void update_vectors(const CgArgs& a, const Slab& sl, double alpha, double beta, bool known,
                                               bool needRR, double& rz, double& rr) {
  constexpr int U = BS == 1 ? 3 : 1;  // blocks in flight per thread
  const int nb = sl.count() / BS;
#pragma unroll 1
  for (int k0 = threadIdx.x; k0 < nb; k0 += U * blockDim.x) {
    double x[U][BS], r[U][BS], p[U][BS], q[U][BS], d[U][BS * BS];
    int row[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * blockDim.x;
      row[u] = k < nb ? sl.row(k * BS) : -1;
      if (row[u] >= 0) {
#pragma unroll
        for (int c = 0; c < BS; ++c) {
          p[u][c] = a.p[row[u] + c];
          q[u][c] = a.Ap[row[u] + c];
          x[u][c] = a.x[row[u] + c];
          r[u][c] = a.r[row[u] + c];
        }
#pragma unroll
        for (int c = 0; c < BS * BS; ++c) d[u][c] = a.dinv[(int64_t)row[u] * BS + c];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (row[u] >= 0) {
        double z[BS];
#pragma unroll
        for (int c = 0; c < BS; ++c) {
          a.x[row[u] + c] = fma(alpha, p[u][c], x[u][c]);
          r[u][c] = fma(-alpha, q[u][c], r[u][c]);
          a.r[row[u] + c] = r[u][c];
        }
        precondition<BS>(d[u], r[u], z);
#pragma unroll
        for (int c = 0; c < BS; ++c) {
          rz = fma(r[u][c], z[c], rz);
          if (needRR) rr = fma(r[u][c], r[u][c], rr);
          if (known) store_p<FF>(a, row[u] + c, fma(beta, p[u][c], z[c]));
        }
      }
    }
  }
}

// p = M^-1 r + beta p over this CTA's rows, where beta had to wait for the sum.
template <int BS, bool FF>
__device__ __forceinline__ void update_direction(const CgArgs& a, const Slab& sl, double beta) {
  const int nb = sl.count() / BS;
#pragma unroll 1
  for (int k = threadIdx.x; k < nb; k += blockDim.x) {
    const int row = sl.row(k * BS);
    double r[BS], z[BS], d[BS * BS];
#pragma unroll
    for (int c = 0; c < BS; ++c) r[c] = a.r[row + c];
#pragma unroll
    for (int c = 0; c < BS * BS; ++c) d[c] = a.dinv[(int64_t)row * BS + c];
    precondition<BS>(d, r, z);
#pragma unroll
    for (int c = 0; c < BS; ++c) store_p<FF>(a, row + c, fma(beta, a.p[row + c], z[c]));
  }
}

// ---------------------------------------------------------------- the product
// Row sums of one lane over the node blocks of its group.
template <typename KT, bool FF, int PB, int LPG>
struct RowSum {
  float h[FF ? PB : 1], l[FF ? PB : 1];
  double v[FF ? 1 : PB];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int c = 0; c < PB; ++c) {
      if constexpr (FF)
        h[c] = l[c] = 0.f;
      else
        v[c] = 0.0;
    }
  }
  typedef typename std::conditional<FF, float2, double>::type X;
  __device__ __forceinline__ static void gather(const CgArgs& a, int col, X x[PB]) {
#pragma unroll
    for (int j = 0; j < PB; ++j) {
      if constexpr (FF)
        x[j] = a.pf[col + j];
      else
        x[j] = a.p[col + j];
    }
  }
  // block at k: its row c at k + c len
  __device__ __forceinline__ void add(const KT* k, int len, const X x[PB]) {
#pragma unroll
    for (int j = 0; j < PB; ++j)
#pragma unroll
      for (int c = 0; c < PB; ++c) {
        if constexpr (FF)
          ff_madd(h[c], l[c], (float)k[c * len + j], x[j].x, x[j].y);
        else
          v[c] = fma((double)k[c * len + j], x[j], v[c]);
      }
  }
  // the lane's blocks sl, sl + LPG, ... of a group with nb blocks; U gathers in flight
  __device__ __forceinline__ void product(const CgArgs& a, const KT* k, const int32_t* cols, int nb, int sl) {
    constexpr int U = 3;
    const int len = nb * PB;
#pragma unroll 1
    for (int t = sl; t < nb; t += U * LPG) {
      X x[U][PB];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u == 0 || t + u * LPG < nb) gather(a, cols[t + u * LPG], x[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u == 0 || t + u * LPG < nb) add(k + PB * (t + u * LPG), len, x[u]);
    }
  }
  // Sum over the group's lanes: two exchanges leave one row per lane (row sl & 3, or sl & 1), the others
  // sum it over the rest of the group; every lane returns its row's sum.
  __device__ __forceinline__ double reduce(int sl) const {
    const bool odd = sl & 1, hi = sl & 2;
    if constexpr (FF) {
      float H = h[0], L = l[0];
      if constexpr (PB > 1) {
        H = odd ? h[1] : h[0];
        L = odd ? l[1] : l[0];
        ff_acc(H, L, __shfl_xor_sync(0xffffffffu, odd ? h[0] : h[1], 1), __shfl_xor_sync(0xffffffffu, odd ? l[0] : l[1], 1));
      }
      if constexpr (PB > 2) {
        float c = h[2], d = l[2];
        ff_acc(c, d, __shfl_xor_sync(0xffffffffu, h[2], 1), __shfl_xor_sync(0xffffffffu, l[2], 1));
        const float sH = hi ? H : c, sL = hi ? L : d;
        if (hi) H = c, L = d;
        ff_acc(H, L, __shfl_xor_sync(0xffffffffu, sH, 2), __shfl_xor_sync(0xffffffffu, sL, 2));
      }
#pragma unroll
      for (int o = PB == 1 ? 1 : (PB == 2 ? 2 : 4); o < LPG; o <<= 1)
        ff_acc(H, L, __shfl_xor_sync(0xffffffffu, H, o), __shfl_xor_sync(0xffffffffu, L, o));
      return f2d_bits(H) + f2d_bits(L);
    } else {
      double V = v[0];
      if constexpr (PB > 1) V = (odd ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 1);
      if constexpr (PB > 2) {
        const double w = v[2] + __shfl_xor_sync(0xffffffffu, v[2], 1);
        V = (hi ? w : V) + __shfl_xor_sync(0xffffffffu, hi ? V : w, 2);
      }
#pragma unroll
      for (int o = PB == 1 ? 1 : (PB == 2 ? 2 : 4); o < LPG; o <<= 1) V += __shfl_xor_sync(0xffffffffu, V, o);
      return V;
    }
  }
};

template <typename KT, bool FF, int PB, int BS, int LPG, bool CL>
__global__ void __launch_bounds__(MAX_WARPS * 32, 1) pcg_kernel(CgArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bars[MAX_WARPS];
  __shared__ double red[3 * MAX_WARPS * 32];  // block sums: one value per thread each of p.Ap, Ap.M^-1 Ap, r.z
  __shared__ double sums[4], scalar[2], all[2][4 * MAX_CLUSTER];  // CL: block sums of every CTA, written by them
  __shared__ int shDead;
  constexpr int GPW = 32 / LPG, PB2 = PB * PB;
  constexpr int AK = 16 / (int)sizeof(KT), AC = 4;  // entries per 16 bytes
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int sl = lane % LPG, grp = lane / LPG;
  const int n = (int)a.n, nGroups = n / PB, nChunks = (nGroups + GPW - 1) / GPW;  // int32 CSR: n < 2^31
  const int W = gridDim.x * nw, w0 = blockIdx.x * nw + wid;
  if (a.every > 0 && a.work[5] != 0.0) return;  // ended in an earlier launch (the same answer in every CTA)
  const int stageBytes = a.capK + a.capC;
  const int stage0 = wid * stageBytes;
  uint64_t* bar = bars + wid;
  if (lane == 0) mbar_init(bar, 1);
  if (tid == 0) shDead = 0;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();

  const KT* K = static_cast<const KT*>(a.K);
  const int32_t total = a.indptr[n];
  const bool aligned = ((reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(a.cols)) & 15) == 0;
  uint64_t policy;
  if ((int64_t)total * (int64_t)sizeof(KT) > 64ll << 20)  // larger than what L2 keeps beside the vectors
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  else
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));

  // One chunk as a lane sees it: its group's first entry b and blocks nb; the chunk's first entry kb, and
  // whether the chunk is copied to shared memory (the 16-byte aligned range around its entries must fit
  // a stage and stay inside the arrays).
  struct Desc {
    int b, nb, kb;
    bool staged;
  };
  struct Ends {
    int b, e;
  };
  auto ends = [&](int c) {  // first and one past the last entry of this lane's group (equal past the end)
    const int g = c * GPW + grp, r = (c < nChunks && g < nGroups) ? g * PB : n;
    return Ends{a.indptr[r], a.indptr[r < n ? r + PB : n]};
  };
  auto issue = [&](const Ends& q) {  // describes the chunk and starts its copy
    Desc d;
    d.b = q.b;
    d.nb = (q.e - q.b) / PB2;
    d.kb = __shfl_sync(0xffffffffu, q.b, 0);
    const int ke = __shfl_sync(0xffffffffu, q.e, 31);
    const int k0 = d.kb & ~(AK - 1), c0 = (d.kb / PB2) & ~(AC - 1);
    const int64_t k1 = ((int64_t)ke + AK - 1) & ~(int64_t)(AK - 1), c1 = ((int64_t)(ke / PB2) + AC - 1) & ~(int64_t)(AC - 1);
    const int64_t bk = (k1 - k0) * (int)sizeof(KT), bc = (c1 - c0) * 4;
    d.staged = aligned && ke > d.kb && bk <= a.capK && bc <= a.capC && k1 <= total && c1 <= total / PB2;
    if (lane == 0 && d.staged) {
      unsigned char* dst = smem + stage0;
      mbar_expect(bar, (uint32_t)(bk + bc));
      bulk_copy(dst, K + k0, (uint32_t)bk, bar, policy);
      bulk_copy(dst + a.capK, a.cols + c0, (uint32_t)bc, bar, policy);
    }
    return d;
  };

  uint32_t phase = 0;  // parity of the copy's next completion
  bool dead = false;   // a wait gave up: no more waits, the kernel runs out
  uint32_t epoch = 0, arrivals = 0, passes = 0;
  ulonglong2* slots = reinterpret_cast<ulonglong2*>(a.work + PART0);  // pcg_slots(gridDim) of them
  uint32_t* counters = reinterpret_cast<uint32_t*>(a.work + 4);       // arrivals at the sums, at the barrier
  const int ng = gridDim.x;
  double rz = a.work[a.k0 & 1], rr = 0.0, pAp = 0.0;
  bool rzKnown = true, stopNext = a.every > 0 && a.work[7] != 0.0, done = false;

  constexpr bool cross = BS > 1 && BS != PB;  // phase B's rows are not the ones this CTA multiplied
  const Slab slab{n, cross ? (int)blockDim.x * BS : nw * GPW * PB};

  // The sums over the grid of m values per thread (red[k * blockDim + thread]) into sums[0 .. m).  Warp k sums value
  // k: FP64 instructions cost the same for 1 or 32 active lanes, so one warp adding a value per thread takes a
  // fraction of a shuffle tree in every warp.  Sums in a fixed order, the same in every CTA.
  auto grid_sums = [&](int m) {
    ++epoch;
    ++arrivals;
    if (cross && !CL) asm volatile("fence.acq_rel.gpu;" ::: "memory");
    __syncthreads();
    if (wid < m) {
      const double* vals = red + wid * blockDim.x;
      double s = 0.0, s2 = 0.0;
      int i = lane;
#pragma unroll 1
      for (; i + 32 < (int)blockDim.x; i += 64) {
        s += vals[i];
        s2 += vals[i + 32];
      }
      if (i < (int)blockDim.x) s += vals[i];
      s = warp_sum(s + s2);
      if constexpr (CL) {
        if (lane < ng) store_remote(&all[epoch & 1][wid * MAX_CLUSTER + blockIdx.x], lane, s);
      } else {
        ulonglong2* set = slots + pcg_slot(epoch, wid, ng);
        if (lane == 0) {
          post(set + blockIdx.x, s, epoch);
          if (wid == 0) arrive(counters);
          if (!dead && !await(counters, arrivals * ng)) dead = true;
        }
        __syncwarp();
        dead = __shfl_sync(0xffffffffu, (int)dead, 0);
        if (!dead && !gather_sum(set, ng, epoch, lane, s)) dead = true;
        if (cross) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        if (lane == 0) {
          sums[wid] = s;
          if (dead) shDead = 1;
        }
      }
    }
    if constexpr (CL) {
      cluster_sync();
      if (wid == 0) {  // lane (k, CTA): three exchanges sum every value over the CTAs
        double s = lane % MAX_CLUSTER < ng ? all[epoch & 1][lane] : 0.0;
#pragma unroll
        for (int o = 1; o < MAX_CLUSTER; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane % MAX_CLUSTER == 0) sums[lane / MAX_CLUSTER] = s;
      }
    }
    __syncthreads();
  };

  if constexpr (CL) {
    for (int i = tid; i < 2 * 4 * MAX_CLUSTER; i += blockDim.x) (&all[0][0])[i] = 0.0;
    cluster_sync();
  }
  const bool resident = nChunks <= W;  // every warp has one chunk at most: its copy stays
  bool landed = false;
  Desc d = issue(ends(w0));
  double rzPart = 0.0, rrPart = 0.0;
#pragma unroll 1
  for (int it = 0; it < a.nIter; ++it) {
    // ---- A: Ap = A p, p.Ap and (BS = 1) Ap.M^-1 Ap
    double acc = 0.0, w = 0.0;
#pragma unroll 1
    for (int c = w0; c < nChunks; c += W) {
      const Ends nx = ends(resident ? nChunks : c + W);  // the chunk copied next
      // this lane's row of the result
      const int g = c * GPW + grp, row = PB == 1 ? 0 : (sl & 3), rIdx = g * PB + row;
      const bool mine = g < nGroups && (PB == 1 ? sl == 0 : sl < PB);
      double pr = 0.0, dr = 0.0;
      bool isFree = true;
      if (mine) {
        pr = a.p[rIdx];
        if constexpr (BS == 1) dr = a.dinv[rIdx];
        isFree = !a.freeMask || a.freeMask[rIdx];
      }
      RowSum<KT, FF, PB, LPG> sum;
      sum.zero();
      if (d.staged) {
        if (!landed) {
          if (!dead && !mbar_wait(bar, phase, COPY_LIMIT)) dead = true;
          phase ^= 1u;
          landed = resident;
        }
        const unsigned char* src = smem + stage0;
        sum.product(a, reinterpret_cast<const KT*>(src) + (d.b - (d.kb & ~(AK - 1))),
                    reinterpret_cast<const int32_t*>(src + a.capK) + (d.b / PB2 - ((d.kb / PB2) & ~(AC - 1))), d.nb, sl);
      } else {
        sum.product(a, K + d.b, a.cols + d.b / PB2, d.nb, sl);
      }
      __syncwarp();
      if (c + W < nChunks) d = issue(nx);
      const double v = sum.reduce(sl);
      if (mine) {
        const double y = isFree ? v : pr;
        a.Ap[rIdx] = y;
        acc = fma(pr, y, acc);
        if constexpr (BS == 1) w = fma(y * y, dr, w);
      }
    }
    if constexpr (BS > 1) {
      if (cross) {  // other CTAs' Ap: one more round before it can be read
        red[tid] = 0.0;
        grid_sums(1);
      } else {
        __syncthreads();
      }
      w = preconditioned_norm<BS>(a, slab);
    }
    red[tid] = acc;
    red[blockDim.x + tid] = w;
    if (!rzKnown) red[2 * blockDim.x + tid] = rzPart;
    grid_sums(rzKnown ? 2 : 3);
    if (!rzKnown) rz = sums[2];
    if (wid == 0) {
      // alpha = r.z / p.Ap, beta = alpha (Ap.M^-1 Ap / p.Ap) - 1: one division, by two lanes
      const double den = sums[0], q = (lane == 0 ? rz : sums[1]) / (den != 0.0 ? den : 1.0);
      const double t = __shfl_sync(0xffffffffu, q, 1);
      if (lane == 0) {
        const bool move = den != 0.0 && rz != 0.0;
        scalar[0] = move ? q : 0.0;
        scalar[1] = move ? fma(q, t, -1.0) : 0.0;
      }
    }
    pAp = sums[0];
    __syncthreads();
    // ---- B: x, r, p
    const bool lastIt = it + 1 == a.nIter;
    const bool test = a.every > 0 && (a.k0 + it + 1) % a.every == 0;
    rzPart = rrPart = 0.0;
    // A predicted beta carries an error of about 1e-16, and p a part 1e-16 / sqrt(beta) of the old direction: below
    // 1e-3 (a residual that falls by 30 in one iteration) beta is formed from the sum instead.
    const double betaPredicted = scalar[1];
    const bool known = betaPredicted >= 1e-3;
    update_vectors<BS, FF>(a, slab, scalar[0], betaPredicted, known, lastIt || test, rzPart, rrPart);
    rzKnown = false;
    if (lastIt || test || !known) {
      red[tid] = rzPart;
      red[blockDim.x + tid] = rrPart;
      grid_sums(2);
      if (!known) update_direction<BS, FF>(a, slab, rz != 0.0 ? sums[0] / rz : 0.0);
      rz = sums[0];
      if (lastIt || test) rr = sums[1];
      rzKnown = true;
      if (test) {
        if (stopNext) done = true;
        stopNext = !(rr > a.tol2) || pAp == 0.0;  // met, NaN or breakdown
      }
      if (blockIdx.x == 0 && tid == 0 && (lastIt || done)) {
        a.work[(a.k0 + it + 1) & 1] = rz;
        a.work[2] = rr;
        a.work[3] = pAp;
        if (a.every > 0) {
          if (done)  // unless a wait gave up
            atomicCAS(reinterpret_cast<unsigned long long*>(a.work + 5), 0ull, (unsigned long long)__double_as_longlong(1.0));
          a.work[6] = (double)(a.k0 + it + 1);
          a.work[7] = stopNext ? 1.0 : 0.0;
        }
      }
      if (lastIt || done) break;
    }
    // the first copies of the next product run under the barrier; behind it everybody's p is visible
    if (!resident) d = issue(ends(w0));
    if constexpr (CL) {
      cluster_sync();
      continue;
    }
    ++passes;
    __syncthreads();
    if (tid == 0) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      arrive(counters + 1);
      if (!dead && !await(counters + 1, passes * ng)) dead = true;
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      if (dead) shDead = 1;
    }
    __syncthreads();
    if (shDead) {  // gave up: let the copy land before the CTA ends
      if (!resident && w0 < nChunks && d.staged) mbar_wait(bar, phase, COPY_LIMIT);
      break;
    }
  }
  if ((dead || shDead) && lane == 0) atomicMin(reinterpret_cast<long long*>(a.work + 5), __double_as_longlong(-1.0));
}

int pcg_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 1;
  return sms;
}


template <typename KT, bool FF, int PB, int BS, int LPG, bool CL>
cudaError_t launch(CgArgs a, int warps, cudaStream_t st) {
  auto kern = pcg_kernel<KT, FF, PB, BS, LPG, CL>;
  const size_t bytes = (size_t)warps * (a.capK + a.capC);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  const int64_t nChunks = (a.n / PB + 32 / LPG - 1) / (32 / LPG);
  int64_t grid = (nChunks + warps - 1) / warps;
  if (grid > pcg_sms()) grid = pcg_sms();
  if (grid > (CL ? MAX_CLUSTER : MAX_GRID)) grid = CL ? MAX_CLUSTER : MAX_GRID;
  if (grid < 1) grid = 1;
  if constexpr (CL) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)grid;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
  }
  // the counters, and the slots, whose epochs start from 0 in every launch
  if ((e = cudaMemsetAsync(a.work + 4, 0, sizeof(double), st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(a.work + PART0, 0, (size_t)pcg_slots((int)grid) * sizeof(ulonglong2), st)) != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kern), dim3((unsigned)grid), dim3(warps * 32), args, bytes, st);
}

// Which lanes, warps and CTAs.  Four lanes per node group measured fastest where ten or more warps' copies fit
// an SM (64^3 Hexa8, FP32 values: 75 us an iteration, 88 with eight lanes; 32^3, FP64 values: 29 against 33); where they
// do not, eight.  Per-entry columns the same (64^3: 151 against 198 us; the three kernels of before 173), but eight
// as long as every warp has one chunk at most (10 x 10 x 5 Hexa20: 11 us against 12), and for FP64 values whose number is
// not known, as the longer rows of Hexa20 would not fit (16 x 16 x 8: 24 us against 30).  A system that leaves SMs
// without work takes four warps per CTA (12^3 Hexa8: 12 us against 16 with sixteen), and one that fits 64 warps runs as
// one cluster of eight CTAs, whose barriers cost a third of the grid's (40 x 8 plate: 7.0 us an iteration against
// 9.2; at 8^3 Hexa8, 92 warps, the grid is ahead by 15 %).
template <typename KT, bool FF, int PB, int BS>
cudaError_t dispatch(CgArgs a, int64_t nnz, cudaStream_t st) {
  constexpr int budget = 227 * 1024 - 14 * 1024;  // shared memory of a CTA less the static arrays
  // a warp's copy: its chunk's entries, 15 % more than on average (longer chunks are read from global memory),
  // and their column list; all that sixteen warps can have if the number of entries is not known
  const int64_t groups = a.n / PB;
  auto stage = [&](int lpg) {
    int64_t entries = budget / MAX_WARPS * (PB * PB) / ((int)sizeof(KT) * PB * PB + 4) - 16;
    if (nnz > 0)
      entries = std::min<int64_t>((int64_t)(1.15 * ((double)nnz / (double)groups) * (32 / lpg)) + 16, 24 * 1024 / (int)sizeof(KT));
    a.capK = (int)((entries * (int)sizeof(KT) + 31) / 16 * 16);
    a.capC = (int)((entries / (PB * PB) * 4 + 47) / 16 * 16);
    return a.capK + a.capC;
  };
  const bool eight = PB == 1 && ((groups + 3) / 4 <= (int64_t)pcg_sms() * MAX_WARPS || (nnz <= 0 && sizeof(KT) == 8));
  const int lpg = eight || 10 * stage(4) > budget ? 8 : 4;
  const int64_t chunks = (groups + 32 / lpg - 1) / (32 / lpg);
  const int most = std::min(MAX_WARPS, budget / stage(lpg));
  const bool cluster = chunks <= 64 && most >= 8;
  int warps = (int)std::min<int64_t>(most, std::max<int64_t>(4, (chunks + pcg_sms() - 1) / pcg_sms()));
  if (cluster) warps = (int)std::max<int64_t>(1, (chunks + MAX_CLUSTER - 1) / MAX_CLUSTER);
  warps = std::max(warps, 3);  // a warp for each sum
  if (lpg == 4) {
    if constexpr (PB > 1) {  // per-entry columns: not in a system of 64 warps
      if (cluster) return launch<KT, FF, PB, BS, 4, true>(a, warps, st);
    }
    return launch<KT, FF, PB, BS, 4, false>(a, warps, st);
  }
  return cluster ? launch<KT, FF, PB, BS, 8, true>(a, warps, st) : launch<KT, FF, PB, BS, 8, false>(a, warps, st);
}

// PB and BS in step: the instances are BS = 1 and BS = PB, and BS = 2, 3 with per-entry columns
template <typename KT, bool FF>
cudaError_t by_block(const CgArgs& a, int bs, int pb, int64_t nnz, cudaStream_t st) {
  if (pb == 3) return bs == 1 ? dispatch<KT, FF, 3, 1>(a, nnz, st) : dispatch<KT, FF, 3, 3>(a, nnz, st);
  if (pb == 2) return bs == 1 ? dispatch<KT, FF, 2, 1>(a, nnz, st) : dispatch<KT, FF, 2, 2>(a, nnz, st);
  if (bs == 1) return dispatch<KT, FF, 1, 1>(a, nnz, st);
  return bs == 2 ? dispatch<KT, FF, 1, 2>(a, nnz, st) : dispatch<KT, FF, 1, 3>(a, nnz, st);
}

}  // namespace

cudaError_t pcg_run(const EfePcg& s, const int32_t* blockCols, int64_t nnz, int64_t k0, int nIter, int every, double tol2,
                    cudaStream_t st) {
  if (nIter <= 0) return cudaSuccess;
  CgArgs a{};
  a.n = s.n;
  a.indptr = s.indptr;
  a.K = s.Kdata;
  a.freeMask = s.freeMask;
  a.dinv = s.dinv;
  a.x = s.x;
  a.r = s.r;
  a.p = s.p;
  a.Ap = s.Ap;
  a.work = s.work;
  a.k0 = k0;
  a.nIter = nIter;
  a.every = every;
  a.tol2 = tol2;
  int pb = blockCols && s.patternBlock > 1 && s.n % s.patternBlock == 0 ? s.patternBlock : 1;
  if (s.kPrecision != EFE_K_FP64) a.pf = reinterpret_cast<float2*>(s.pFF);
  if ((s.blockSize > 1 && s.blockSize != pb) || (s.kPrecision != EFE_K_FP64 && !a.pf)) pb = 1;
  a.cols = pb > 1 ? blockCols : s.indices;
  if (s.kPrecision == EFE_K_FP64) return by_block<double, false>(a, s.blockSize, pb, nnz, st);
  if (a.pf) return by_block<float, true>(a, s.blockSize, pb, nnz, st);
  if (s.blockSize == 1) return dispatch<float, false, 1, 1>(a, nnz, st);
  return s.blockSize == 2 ? dispatch<float, false, 1, 2>(a, nnz, st) : dispatch<float, false, 1, 3>(a, nnz, st);
}

}  // namespace efe
