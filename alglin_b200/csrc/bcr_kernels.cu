// BorderedCR device kernels, FP64 path (sm_100a).
//
// One cyclic-reduction (CR) level is one launch of k_factor_level: every pair
// (jp = j-k, j) of the level is independent, and one warp eliminates one pair.
// The warp stages the pair's row blocks in shared memory as one
// (2n + nr) x (3n + nx) work matrix
//
//                x_j      x_jp     x_jpp    xb
//   TOP    [  E_jp  |  D_jp  |   0    | B_jp ]   row block jp
//   BOTTOM [  D_j   |   0    |  E_j   | B_j  ]   row block j
//   border [  C_j   |   0    |   0    |  0   ]   nr border rows
//
// and eliminates x_j from it: partial-pivot LU or Householder QR on the 2n x n
// panel (buildT, BABD_BorderedCR.cc:845-898), applied to the trailing columns
// (applyT, cc:917-982) and, through the U rows, to the border rows (the C/F
// Schur updates of factorize_block, cc:1107-1154).  After elimination
//   rows 0..n-1   hold the U-row  [U | D'_j | E'_j | B'_j ]  (back-substitution)
//   rows n..2n-1  hold the reduced row [0 | D'_jp | E'_jp | B'_jp]
//   border rows   hold [C_j U^-1 | dC_jp | dC_jpp | dF]
// dC_jp is added to C_jp by the owning warp (no other pair of the level writes
// C_jp); dC_jpp goes to a per-block scratch slot and is added to C_jpp by
// k_border_fix after the level, because C_jpp is also C_jp of pair j+2k.
// The F updates dF go to a per-block slot and are summed in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "bcr_device.h"

namespace bcr {

static constexpr int WARPS_PANEL = 4;
static constexpr size_t SMEM_MAX = 227 * 1024;
static constexpr int CTA_KERNEL_MIN_N = 24;  // n above this: one CTA per pair
static constexpr long COMPACT_GRID = 148 * 8;  // CTAs of a sweep over a compacted batch map

template <typename T>
struct FactorArgs {
  Dims d;
  const double *D0, *E0, *B0, *C0;  // loaded matrix, read at the first level
  T *D, *E, *B, *C;                  // working blocks
  T* Tm;
  unsigned char* P;
  T* Rbuf;
  double* Fbuf;  // the F Schur updates are accumulated in FP64 in every precision
  const double* F0;  // loaded F (read by the tree schedule's root)
  StatusWords* st;
  int k, first, ldw;
  // right-hand sides eliminated together with the factorization (forward
  // sweep fused into the pair kernel); nrf == 0 when not fused
  double* x;
  int ldx, nrf;
  double* XB;
  // pair range of a single-system launch, [qb, qe) of the level (qe == 0: all)
  long qb, qe;
};

// element of a block: the loaded FP64 matrix at the first level, the working
// copy (type T) afterwards
template <typename T>
__device__ __forceinline__ T ldsrc(bool first, const double* orig, const T* work, size_t i) {
  return first ? T(orig[i]) : work[i];
}

// the same where another CTA of the same launch may have written the element
// (persistent batch launches): served by L2, never by a stale L1 line
template <bool COH, typename T>
__device__ __forceinline__ T ldsrc_c(bool first, const double* orig, const T* work, size_t i) {
  if constexpr (COH) return first ? T(__ldcg(orig + i)) : __ldcg(work + i);
  else return ldsrc(first, orig, work, i);
}

// Element of a batch of loads, 0 where p is false.  volatile keeps the loads of
// an unrolled batch together: scheduled by the compiler, each one waits for the
// use of the one before (the same 262 KB read by one CTA: 80,000 cycles from
// DRAM, against 13,000).
__device__ __forceinline__ double ld_batch(bool p, const double* a) {
  double v;
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f64 %0, 0d0000000000000000; @q ld.global.f64 %0, [%1]; }\n"
               : "=d"(v)
               : "l"(a), "r"((unsigned)p));
  return v;
}
__device__ __forceinline__ float ld_batch(bool p, const float* a) {
  float v;
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f32 %0, 0f00000000; @q ld.global.f32 %0, [%1]; }\n"
               : "=f"(v)
               : "l"(a), "r"((unsigned)p));
  return v;
}

// the same through L2 (elements that another CTA of the launch may have written)
__device__ __forceinline__ double ld_batch_cg(bool p, const double* a) {
  double v;
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f64 %0, 0d0000000000000000; @q ld.global.cg.f64 %0, [%1]; }\n"
               : "=d"(v)
               : "l"(a), "r"((unsigned)p)
               : "memory");
  return v;
}
__device__ __forceinline__ float ld_batch_cg(bool p, const float* a) {
  float v;
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f32 %0, 0f00000000; @q ld.global.cg.f32 %0, [%1]; }\n"
               : "=f"(v)
               : "l"(a), "r"((unsigned)p)
               : "memory");
  return v;
}
template <bool COH, typename T>
__device__ __forceinline__ T ld_batch_c(bool p, const T* a) {
  if constexpr (COH) return ld_batch_cg(p, a);
  else return ld_batch(p, a);
}

// Pair range of one worker (warp or CTA).  Single system: a grid-stride loop
// over the level's pairs.  Batch: map entry e (by default the CTA's index)
// holds pairs [q0, q1) of system cmap[e].sys, whose arguments come from the
// table; the level is the batch's.
__device__ __forceinline__ void take_level(FactorArgs<float>& a, const FactorArgs<float>& a0) { a.k = a0.k; a.first = a0.first; }
__device__ __forceinline__ void take_level(FactorArgs<double>& a, const FactorArgs<double>& a0) { a.k = a0.k; a.first = a0.first; }

// a batch system whose refinement has converged skips the sweeps (the
// SweepArgs overload below; found at instantiation)
template <typename A>
__device__ __forceinline__ bool system_active(const A&) { return true; }

// the pair range a single-system factorization launch is limited to (sweeps: all)
template <typename T>
__device__ __forceinline__ void launch_pair_range(const FactorArgs<T>& a, long& qb, long& qe) { qb = a.qb; qe = a.qe; }
template <typename A>
__device__ __forceinline__ void launch_pair_range(const A&, long&, long&) {}

template <bool BATCH, typename A>
__device__ __forceinline__ void pair_range(const A& a0, const A* tab, const BatchCta* cmap, int workers, int worker,
                                           A& a, long& q0, long& q1, long& qs, long entry = -1) {
  if constexpr (BATCH) {
    const BatchCta c = cmap[entry < 0 ? (long)blockIdx.x : entry];
    a = tab[c.sys];
    take_level(a, a0);
    q0 = c.q0 + worker;
    q1 = system_active(a) ? c.q1 : q0;
    qs = workers;
  } else {
    q0 = (long)blockIdx.x * workers + worker;
    q1 = pairs_at_level(a0.d.nblock, a0.k);
    qs = (long)gridDim.x * workers;
    long qb = 0, qe = 0;
    launch_pair_range(a0, qb, qe);
    if (qe > 0) { q0 += qb; q1 = qe; }
  }
}

// Map entries of one CTA of a batched sweep: entry b alone (one CTA per
// entry), or, when ecnt is given (the compacted maps of the refinement
// passes, whose length the device wrote), entries b, b + grid, ... below
// *ecnt.  Single systems: the body once.
template <bool BATCH, typename F>
__device__ __forceinline__ void for_entries(const long* ecnt, F&& body) {
  if constexpr (BATCH) {
    const long cnt = ecnt ? *ecnt : (long)gridDim.x;
    for (long e = blockIdx.x; e < cnt; e += gridDim.x) body(e);
  } else {
    body(-1L);
  }
}

// the same through the read-only path; every load of a pair kernel's load
// phase is independent of the shared-memory stores that follow it
template <typename T>
__device__ __forceinline__ T ldg_src(bool first, const double* orig, const T* work, size_t i) {
  if constexpr (sizeof(T) == 8)
    return __ldg(first ? orig + i : reinterpret_cast<const double*>(work) + i);
  else
    return first ? T(__ldg(orig + i)) : __ldg(work + i);
}

template <typename T>
__device__ __forceinline__ void load2(const T* p, T& a, T& b) {
  if constexpr (sizeof(T) == 8) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    a = v.x; b = v.y;
  } else {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x; b = v.y;
  }
}

template <typename T>
__device__ __forceinline__ void store2(T* p, T a, T b) {
  if constexpr (sizeof(T) == 8) *reinterpret_cast<double2*>(p) = make_double2(a, b);
  else *reinterpret_cast<float2*>(p) = make_float2(a, b);
}

__host__ __device__ inline int odd_ld(int r) { return r | 1; }

// pairs of large blocks go to one CTA each (work matrix in a global slab)
bool use_cta_kernel(const Dims& d) {
  return d.n > CTA_KERNEL_MIN_N || panel_smem_per_warp(d, 8) > SMEM_MAX;
}

size_t cta_slab_elems(const Dims& d) { return (size_t)(2 * d.n + d.nr) * (3 * d.n + d.nx); }

size_t panel_smem_per_warp(const Dims& d, int elem_bytes) {
  const int R = 2 * d.n + d.nr, NC = 3 * d.n + d.nx;
  size_t b = (size_t)odd_ld(R) * NC * elem_bytes + (size_t)d.n * (elem_bytes + sizeof(int));
  return b;
}

template <typename T> __device__ void block_argmax(T& v, int& idx, T* sv, int* si);
template <typename T> __device__ T block_sum(T v, T* sv);

// ---------------------------------------------------------------------------
// warp-level elimination of x_j from the staged work matrix
// ---------------------------------------------------------------------------
template <typename T>
__device__ int warp_eliminate_lu(T* W, int ldw, int n, int R, int NC, int* ipiv, int lane) {
  const int n2 = 2 * n;
  for (int i = 0; i < n; ++i) {
    T* ci = W + (size_t)i * ldw;
    T best = T(-1);
    int bi = i;  // stays in range even when every candidate is NaN
    for (int r = i + lane; r < n2; r += 32) {
      T v = dev_abs(ci[r]);
      if (v > best) { best = v; bi = r; }
    }
    warp_argmax(best, bi);
    if (lane == 0) ipiv[i] = bi;
    const T pv = ci[bi];
    __syncwarp();  // every lane holds the pivot before column i is swapped
    if (pv == T(0)) return i + 1;  // LAPACK getrf INFO
    if (bi != i)
      for (int c = lane; c < NC; c += 32) {
        T* col = W + (size_t)c * ldw;
        T t = col[i]; col[i] = col[bi]; col[bi] = t;
      }
    __syncwarp();
    const T rinv = T(1) / pv;
    for (int r = i + 1 + lane; r < R; r += 32) ci[r] *= rinv;
    __syncwarp();
    for (int c = i + 1 + lane; c < NC; c += 32) {
      T* col = W + (size_t)c * ldw;
      const T u = col[i];
      if (u != T(0))
        for (int r = i + 1; r < R; ++r) col[r] -= ci[r] * u;
    }
    __syncwarp();
  }
  return 0;
}

// Householder QR (optionally with column pivoting) of the panel; the border
// rows are eliminated with the finished R rows.  Returns i+1 if R(i,i) == 0.
template <typename T, bool PIVOT>
__device__ int warp_eliminate_qr(T* W, int ldw, int n, int R, int NC, int* ipiv, T* tau, int lane) {
  const int n2 = 2 * n;
  for (int i = 0; i < n; ++i) {
    if (PIVOT) {
      // largest remaining column 2-norm over the panel rows i..2n-1
      T best = T(-1);
      int bc = i;
      for (int c = i + lane; c < n; c += 32) {
        const T* col = W + (size_t)c * ldw;
        T s = T(0);
        for (int r = i; r < n2; ++r) s += col[r] * col[r];
        if (s > best) { best = s; bc = c; }
      }
      warp_argmax(best, bc);
      if (lane == 0) ipiv[i] = bc;
      if (bc != i)
        for (int r = lane; r < R; r += 32) {
          T t = W[(size_t)i * ldw + r];
          W[(size_t)i * ldw + r] = W[(size_t)bc * ldw + r];
          W[(size_t)bc * ldw + r] = t;
        }
      __syncwarp();
    } else if (lane == 0) {
      ipiv[i] = i;
    }
    T* v = W + (size_t)i * ldw;
    const T alpha = v[i];
    T s = T(0);
    for (int r = i + 1 + lane; r < n2; r += 32) s += v[r] * v[r];
    s = warp_sum(s);
    T t = T(0), beta = alpha;
    if (s != T(0)) {
      T nrm = sqrt(alpha * alpha + s);
      beta = alpha >= T(0) ? -nrm : nrm;
      t = (beta - alpha) / beta;
      const T sc = T(1) / (alpha - beta);
      for (int r = i + 1 + lane; r < n2; r += 32) v[r] *= sc;
    }
    __syncwarp();
    if (lane == 0) { v[i] = beta; tau[i] = t; }
    __syncwarp();
    if (beta == T(0)) return i + 1;
    if (t != T(0))
      for (int c = i + 1 + lane; c < NC; c += 32) {
        T* col = W + (size_t)c * ldw;
        T w = col[i];
        for (int r = i + 1; r < n2; ++r) w += v[r] * col[r];
        w *= t;
        col[i] -= w;
        for (int r = i + 1; r < n2; ++r) col[r] -= w * v[r];
      }
    __syncwarp();
    if (R > n2) {
      const T rb = T(1) / beta;
      for (int r = n2 + lane; r < R; r += 32) v[r] *= rb;
      __syncwarp();
      for (int c = i + 1 + lane; c < NC; c += 32) {
        T* col = W + (size_t)c * ldw;
        const T u = col[i];
        if (u != T(0))
          for (int r = n2; r < R; ++r) col[r] -= v[r] * u;
      }
      __syncwarp();
    }
  }
  return 0;
}

template <typename T, int SEL, bool BATCH = false>
__global__ void __launch_bounds__(WARPS_PANEL * 32) k_factor_level(FactorArgs<T> a0, const FactorArgs<T>* tab,
                                                               const BatchCta* cmap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  FactorArgs<T> ab;  // this CTA's system (batch only)
  long q0, q1, qs;
  pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs);
  const FactorArgs<T>& a = BATCH ? ab : a0;
  const Dims d = a.d;
  const int n = d.n, nr = d.nr, nx = d.nx, nb = d.nblock;
  const int n2 = 2 * n, R = n2 + nr, NC = 3 * n + nx, ldw = a.ldw;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  const size_t wsz = (size_t)ldw * NC;
  T* W = reinterpret_cast<T*>(smem_raw) + warp * wsz;
  T* tau = reinterpret_cast<T*>(smem_raw) + wpb * wsz + warp * n;
  int* ipiv = reinterpret_cast<int*>(reinterpret_cast<T*>(smem_raw) + wpb * wsz + wpb * n) + warp * n;
  const int k = a.k;
  const bool first = a.first != 0;

  for (long q = q0; q < q1; q += qs) {
    const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
    // ---------------------------------------------------------------- load
    {
      const size_t oj = (size_t)j * nn, ojp = (size_t)jp * nn;
      for (int idx = lane; idx < (int)nn; idx += 32) {
        const int i = idx % n, c = idx / n;
        T ejp, djp, dj, ej;
        if (first) {
          ejp = T(a.E0[ojp + idx]); djp = T(a.D0[ojp + idx]);
          dj = T(a.D0[oj + idx]);   ej = T(a.E0[oj + idx]);
        } else {
          ejp = a.E[ojp + idx]; djp = a.D[ojp + idx];
          dj = a.D[oj + idx];   ej = a.E[oj + idx];
        }
        W[(size_t)c * ldw + i] = ejp;
        W[(size_t)(n + c) * ldw + i] = djp;
        W[(size_t)(n2 + c) * ldw + i] = T(0);
        W[(size_t)c * ldw + n + i] = dj;
        W[(size_t)(n + c) * ldw + n + i] = T(0);
        W[(size_t)(n2 + c) * ldw + n + i] = ej;
      }
      for (int idx = lane; idx < (int)nnx; idx += 32) {
        const int i = idx % n, c = idx / n;
        const size_t o1 = (size_t)jp * nnx + idx, o2 = (size_t)j * nnx + idx;
        W[(size_t)(3 * n + c) * ldw + i] = first ? T(a.B0[o1]) : a.B[o1];
        W[(size_t)(3 * n + c) * ldw + n + i] = first ? T(a.B0[o2]) : a.B[o2];
      }
      for (int idx = lane; idx < (int)nrn; idx += 32) {
        const int r = idx % nr, c = idx / nr;
        const size_t o = (size_t)j * nrn + idx;
        W[(size_t)c * ldw + n2 + r] = first ? T(a.C0[o]) : a.C[o];
        W[(size_t)(n + c) * ldw + n2 + r] = T(0);
        W[(size_t)(n2 + c) * ldw + n2 + r] = T(0);
      }
      for (int idx = lane; idx < (int)nrnx; idx += 32) {
        const int r = idx % nr, c = idx / nr;
        W[(size_t)(3 * n + c) * ldw + n2 + r] = T(0);
      }
    }
    __syncwarp();
    // ----------------------------------------------------------- eliminate
    int info;
    if (SEL == SEL_LU) info = warp_eliminate_lu<T>(W, ldw, n, R, NC, ipiv, lane);
    else if (SEL == SEL_QR) info = warp_eliminate_qr<T, false>(W, ldw, n, R, NC, ipiv, tau, lane);
    else info = warp_eliminate_qr<T, true>(W, ldw, n, R, NC, ipiv, tau, lane);
    __syncwarp();
    if (info != 0) {
      if (lane == 0) report(a.st, DEV_ZERO_PIVOT, j, info, k);
      continue;
    }
    // ---------------------------------------------------------------- store
    {
      T* Tj = a.Tm + (size_t)j * szT(d);
      for (int idx = lane; idx < (int)(2 * nn); idx += 32) {
        const int r = idx % n2, c = idx / n2;
        Tj[idx] = W[(size_t)c * ldw + r];
      }
      if (SEL != SEL_LU)
        for (int i = lane; i < n; i += 32) Tj[2 * nn + i] = tau[i];
      __syncwarp();
      // row map (getrf row order) and column map (QRP) from the swap sequence,
      // built in the tau scratch (already stored)
      unsigned char* Pj = a.P + (size_t)j * szP(d);
      unsigned char* mp = reinterpret_cast<unsigned char*>(tau);
      if (lane == 0) {
        if (SEL == SEL_LU) {
          for (int r = 0; r < n2; ++r) mp[r] = (unsigned char)r;
          for (int i = 0; i < n; ++i) { unsigned char t = mp[i]; mp[i] = mp[ipiv[i]]; mp[ipiv[i]] = t; }
        } else {
          for (int r = 0; r < n2; ++r) mp[r] = (unsigned char)r;
          for (int i = 0; i < n; ++i) mp[n2 + i] = (unsigned char)i;
          if (SEL == SEL_QRP)
            for (int i = 0; i < n; ++i) { unsigned char t = mp[n2 + i]; mp[n2 + i] = mp[n2 + ipiv[i]]; mp[n2 + ipiv[i]] = t; }
        }
      }
      __syncwarp();
      for (int i = lane; i < (SEL == SEL_LU ? n2 : 3 * n); i += 32) Pj[i] = mp[i];
      const size_t oj = (size_t)j * nn, ojp = (size_t)jp * nn;
      for (int idx = lane; idx < (int)nn; idx += 32) {
        const int i = idx % n, c = idx / n;
        a.D[oj + idx] = W[(size_t)(n + c) * ldw + i];
        a.E[oj + idx] = W[(size_t)(n2 + c) * ldw + i];
        a.D[ojp + idx] = W[(size_t)(n + c) * ldw + n + i];
        a.E[ojp + idx] = W[(size_t)(n2 + c) * ldw + n + i];
      }
      for (int idx = lane; idx < (int)nnx; idx += 32) {
        const int i = idx % n, c = idx / n;
        a.B[(size_t)j * nnx + idx] = W[(size_t)(3 * n + c) * ldw + i];
        a.B[(size_t)jp * nnx + idx] = W[(size_t)(3 * n + c) * ldw + n + i];
      }
      for (int idx = lane; idx < (int)nrn; idx += 32) {
        const int r = idx % nr, c = idx / nr;
        const size_t oc = (size_t)jp * nrn + idx;
        a.C[(size_t)j * nrn + idx] = W[(size_t)c * ldw + n2 + r];
        const T cjp = first ? T(a.C0[oc]) : a.C[oc];
        a.C[oc] = cjp + W[(size_t)(n + c) * ldw + n2 + r];
        a.Rbuf[(size_t)j * nrn + idx] = W[(size_t)(n2 + c) * ldw + n2 + r];
      }
      for (int idx = lane; idx < (int)nrnx; idx += 32) {
        const int r = idx % nr, c = idx / nr;
        a.Fbuf[(size_t)j * nrnx + idx] = W[(size_t)(3 * n + c) * ldw + n2 + r];
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// register-resident LU pair elimination for n <= N <= 16 (lane = panel row)
//
// Lane l < 2n holds row l of the work matrix [panel | x_jp | x_jpp | xb] in
// registers.  Row interchanges are not performed physically: every lane keeps
// the LAPACK row position of its row (mypos), and the swap of positions i and
// p at step i (getrf's ipiv) is replayed on those positions, so the final
// positions reproduce the row order of getrf exactly.  The pivot row of each
// step is broadcast through shared memory; the nr border rows are spread over
// the lanes by column (lane c holds column c, and c+32) and are eliminated with
// the same pivot rows, which yields C_j U^-1 and the C/F Schur updates.
// ---------------------------------------------------------------------------
// pairs [q0, q1) step qs of one system and level, one per warp
template <typename T, int N, int NXM, int NRM, bool COH>
__device__ __forceinline__ void rows_body(const FactorArgs<T>& a, long q0, long q1, long qs) {
  constexpr int NC = 3 * N + NXM;
  constexpr int NCP = (NC + 1) & ~1;
  constexpr int SLOTS = (NC + 31) / 32;
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ __align__(16) T ubuf[4][NCP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Dims d = a.d;
  const int n = d.n, nr = d.nr, nx = d.nx, n2 = 2 * n;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  T* ub = ubuf[warp];
  const int k = a.k;
  const bool first = a.first != 0;
  const bool act = lane < n2, top = lane < n;
  const int ri = top ? lane : lane - n;

  for (long q = q0; q < q1; q += qs) {
    const int j = k + (int)(2L * k * q), jp = j - k;
    T row[NC];
    {
      // panel: E_jp (TOP) / D_j (BOTTOM); x_jp column: D_jp / 0; x_jpp: 0 / E_j
      const size_t op = top ? (size_t)jp * nn : (size_t)j * nn;
      const size_t ob = (size_t)(top ? jp : j) * nnx;
#pragma unroll
      for (int c = 0; c < N; ++c) {
        T pv = T(0), xv = T(0);
        if (act && c < n) {
          const size_t o = op + (size_t)c * n + ri;
          pv = top ? ldsrc_c<COH>(first, a.E0, a.E, o) : ldsrc_c<COH>(first, a.D0, a.D, o);
          xv = top ? ldsrc_c<COH>(first, a.D0, a.D, o) : ldsrc_c<COH>(first, a.E0, a.E, o);
        }
        row[c] = pv;
        row[N + c] = top ? xv : T(0);
        row[2 * N + c] = top ? T(0) : xv;
      }
#pragma unroll
      for (int c = 0; c < NXM; ++c)
        row[3 * N + c] = (act && c < nx) ? ldsrc_c<COH>(first, a.B0, a.B, ob + (size_t)c * n + ri) : T(0);
    }
    T cr[NRM][SLOTS];
#pragma unroll
    for (int r = 0; r < NRM; ++r)
#pragma unroll
      for (int sl = 0; sl < SLOTS; ++sl) cr[r][sl] = T(0);
    if (lane < n) {
      const size_t oc = (size_t)j * nrn + (size_t)lane * nr;
#pragma unroll
      for (int r = 0; r < NRM; ++r)
        if (r < nr) cr[r][0] = ldsrc_c<COH>(first, a.C0, a.C, oc + r);
    }

    int mypos = lane, mykey = 0, info = 0;
    bool done = !act;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (i < n) {
        T v = done ? T(-1) : dev_abs(row[i]);
        if (v != v) v = T(-0.5);  // NaN never wins against a number
        int key = done ? 0x7fffffff : mypos;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const T ov = __shfl_xor_sync(FULL, v, o);
          const int ok = __shfl_xor_sync(FULL, key, o);
          if (ov > v || (ov == v && ok < key)) { v = ov; key = ok; }
        }
        const unsigned m = __ballot_sync(FULL, !done && mypos == key);
        const int p = __ffs(m) - 1;
        if (lane == i) mykey = key;
        if (!done && mypos == i && lane != p) mypos = key;
        if (lane == p) {
          mypos = i;
#pragma unroll
          for (int c = (i & ~1); c < NCP; c += 2)
            store2(&ub[c], row[c], c + 1 < NC ? row[c + 1] : T(0));
        }
        __syncwarp();
        const T piv = ub[i];
        if (piv == T(0) && info == 0) info = i + 1;
        const T rinv = piv != T(0) ? T(1) / piv : T(0);
        if (!done && lane != p) {
          const T l = row[i] * rinv;
          row[i] = l;
#pragma unroll
          for (int c = i + 1; c < NC; ++c) row[c] = fma(-l, ub[c], row[c]);
        }
        if (lane == p) done = true;
#pragma unroll
        for (int r = 0; r < NRM; ++r) {
          if (r < nr) {
            const T mr = __shfl_sync(FULL, cr[r][0], i) * rinv;
            if (lane == i) cr[r][0] = mr;
            else if (lane > i && lane < NC) cr[r][0] = fma(-mr, ub[lane], cr[r][0]);
#pragma unroll
            for (int sl = 1; sl < SLOTS; ++sl)
              if (lane + 32 * sl < NC) cr[r][sl] = fma(-mr, ub[lane + 32 * sl], cr[r][sl]);
          }
        }
        __syncwarp();
      }
    }
    if (info != 0) {
      if (lane == 0) report(a.st, DEV_ZERO_PIVOT, j, info, k);
      continue;
    }
    // ---------------------------------------------------------------- store
    if (act) {
      T* Tj = a.Tm + (size_t)j * szT(d);
      const bool urow = mypos < n;
      const int rr = urow ? mypos : mypos - n;
      const size_t blk = urow ? (size_t)j : (size_t)jp;
      T* Dd = a.D + blk * nn + rr;
      T* Ed = a.E + blk * nn + rr;
      T* Bd = a.B + blk * nnx + rr;
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (c < n) {
          Tj[(size_t)mypos + (size_t)c * n2] = row[c];
          Dd[(size_t)c * n] = row[N + c];
          Ed[(size_t)c * n] = row[2 * N + c];
        }
#pragma unroll
      for (int c = 0; c < NXM; ++c)
        if (c < nx) Bd[(size_t)c * n] = row[3 * N + c];
    }
    if (act) a.P[(size_t)j * szP(d) + mypos] = (unsigned char)lane;
#pragma unroll
    for (int sl = 0; sl < SLOTS; ++sl) {
      const int col = lane + 32 * sl;
      if (col >= NC) continue;
#pragma unroll
      for (int r = 0; r < NRM; ++r) {
        if (r >= nr) continue;
        const T v = cr[r][sl];
        if (col < N) {
          if (col < n) a.C[(size_t)j * nrn + (size_t)col * nr + r] = v;
        } else if (col < 2 * N) {
          const int c = col - N;
          if (c < n) {
            const size_t o = (size_t)jp * nrn + (size_t)c * nr + r;
            a.C[o] = ldsrc_c<COH>(first, a.C0, a.C, o) + v;
          }
        } else if (col < 3 * N) {
          const int c = col - 2 * N;
          if (c < n) a.Rbuf[(size_t)j * nrn + (size_t)c * nr + r] = v;
        } else {
          const int c = col - 3 * N;
          if (c < nx) a.Fbuf[(size_t)j * nrnx + (size_t)c * nr + r] = v;
        }
      }
    }
  }
}

template <typename T, int N, int NXM, int NRM, bool BATCH = false>
__global__ void __launch_bounds__(128) k_factor_lu_rows(FactorArgs<T> a0, const FactorArgs<T>* tab,
                                                         const BatchCta* cmap) {
  const int warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  FactorArgs<T> ab;  // this CTA's system (batch only)
  long q0, q1, qs;
  pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs);
  rows_body<T, N, NXM, NRM, false>(BATCH ? ab : a0, q0, q1, qs);
}

template <typename T> __device__ __forceinline__ T rcp_rn(T x);
template <> __device__ __forceinline__ double rcp_rn<double>(double x) { return __drcp_rn(x); }
template <> __device__ __forceinline__ float rcp_rn<float>(float x) { return __frcp_rn(x); }

#include "bcr_qr.cuh"

// ---------------------------------------------------------------------------
// Tensor-core LU pair elimination for n == N (N = 8 or 16), nr <= 8, nx <= 8.
//
//   phase 1 (SIMT, lane = panel row): partial-pivot LU of the 2N x N panel
//     [E_jp; D_j] in registers, with getrf's row order replayed on positions
//     (mypos) and the pivot chosen by exact integer reductions on the bits of
//     |a| (largest |a|, then smallest position: the idamax rule).  The columns
//     already eliminated are reused, Gauss-Jordan style, for the operator that
//     the eliminations apply to the trailing columns,
//       G = [ L^-1 ; -M L^-1 ; -(C_j U^-1) L^-1 ]      ((2N+8) x N),
//     so that no triangular solve follows.  The nr border rows are spread over
//     the warp.
//   phase 2 (FP64 tensor cores, mma.sync m8n8k4): one GEMM
//       [U-row | reduced row | border update] = G (PW)_top + [0; (PW)_bot; 0]
//     over the 2N + nx trailing columns [x_jp | x_jpp | xb].
//
// Bound by the pivot steps' dependency chains (4 warps per scheduler) and the L1
// data pipe (66% busy: 1,333 wavefronts and 3,323 instructions per pair with a
// right-hand side, level 1 of n = 16).  With unrolled steps, keeping the
// operator in the eliminated columns instead of solving X L = [I; -M; -C']
// after the LU took a pair from 3,093 to 2,616 instructions and level 1 of
// 40,000 blocks from 179 to 165 us.
//
// T_j and C_j hold the operator form: T_j = [L^-1 below the diagonal, U on and
// above it; -M L^-1], C_j = -C_j U^-1 L^-1.  The forward sweep applies them as
// one matrix-vector product (SweepArgs::op).
// ---------------------------------------------------------------------------
// Pivot candidate of one lane: |a| as an integer key (upper word + 1, lower
// word; NaN below every number, finished rows below everything) and the
// reciprocal of a by Newton-Raphson steps r <- r + r (1 - a r) from the
// hardware's approximation, which doubles the correct bits each time (FP64:
// about 20, 40, 80; FP32: 23, then rounding): at most one unit in the last
// place off for the magnitudes tc_plain_pivot() accepts (measured: the correctly
// rounded value for every such FP32 number and for 3.8e9 random FP64 numbers), and
// free of the range branches of a correctly rounded reciprocal, which would cut
// the step into pieces the scheduler cannot overlap.
__device__ __forceinline__ void tc_candidate(double v, bool done, unsigned& hi, unsigned& lo, double& rc) {
  const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
  hi = done ? 0u : h > 0x7ff00000u ? 1u : h + 1u;
  lo = (unsigned)__double2loint(v);
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  r = fma(fma(-v, r, 1.0), r, r);
  rc = fma(fma(-v, r, 1.0), r, r);
}
__device__ __forceinline__ void tc_candidate(float v, bool done, unsigned& hi, unsigned& lo, float& rc) {
  const unsigned h = __float_as_uint(v) & 0x7fffffffu;
  hi = done ? 0u : h > 0x7f800000u ? 1u : h + 1u;
  lo = 0u;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  rc = fmaf(fmaf(-v, r, 1.0f), r, r);
}
// the pivot's magnitude (key hi) is a normal number whose reciprocal is one too
template <typename T>
__device__ __forceinline__ bool tc_plain_pivot(unsigned hi) {
  return sizeof(T) == 8 ? hi - 0x00200000u < 0x7fc00000u - 0x00200000u : hi - 0x01000000u < 0x7e000000u - 0x01000000u;
}

__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <int N, typename T = double>
struct TcShape {
  static constexpr int MT = 2 * N + 8;             // GEMM rows: U-row, reduced row, border (padded)
  static constexpr int NTILES = (2 * N + 8 + 7) / 8;  // trailing columns 2N + nx, nx <= 8
  static constexpr int NTP = NTILES * 8;
  // trailing rows, compact: a TOP row keeps [D_jp | B_jp | x_jp], a BOTTOM row
  // [E_j | B_j | x_j]; the structurally zero half of each row is not stored
  static constexpr int LDW = NTP - N + 1;
  static constexpr int PC = (NTILES + 1) / 2;      // column tiles per product pass
  static constexpr int LDG = N + 4;                 // operator rows (16B aligned, conflict-free A loads)
  static constexpr int KSTEPS = N / 4;
  static constexpr int MTILES = MT / 8;
  static constexpr int WS = 2 * N * LDW;            // doubles: the 2N panel rows' trailing part
  static constexpr int GS = MT * LDG;
  static constexpr size_t BYTES = (size_t)(WS + GS) * sizeof(T) + 2 * N * sizeof(int);
};

// element (row, col) of the trailing part from the compact rows
template <int N, typename T>
__device__ __forceinline__ T tc_w(const T* Wt, int row, int col) {
  constexpr int LDW = TcShape<N>::LDW;
  const bool top = row < N;
  if (col < N) return top ? Wt[row * LDW + col] : T(0);
  if (col < 2 * N) return top ? T(0) : Wt[row * LDW + col - N];
  return Wt[row * LDW + col - N];
}

size_t tc_smem_per_warp(int n) {
  return n == 16 ? TcShape<16>::BYTES : n == 8 ? TcShape<8>::BYTES : 0;
}
template <typename T>
static size_t tc_smem_per_warp_t(int n) {
  return n == 16 ? TcShape<16, T>::BYTES : n == 8 ? TcShape<8, T>::BYTES : 0;
}

__host__ __device__ inline int lowbit(int v) { return v & -v; }
__host__ __device__ inline void tree_children(int j, int nb, int& c1, int& c2);

// Per-pair extras of the tree-scheduled factorization (k_factor_tree_tc):
// gather = the C_jpp contributions of earlier levels are added to C_j at load
// (Rbuf[j - K'] for K' = 1, 2, ..., gather; 0 in the level-by-level launches,
// where k_border_fix adds them after each level); c1, c2 = the nodes whose F
// and xb partial sums are added to this pair's own (0: none).
struct TcTree {
  int gather, c1, c2;
};

// Coherent load of an element that another warp of the same launch may have
// written (tree schedule): bypasses L1, served by L2.
__device__ __forceinline__ double ldw(const double* p) { return __ldcg(p); }

// Eliminates x_j from the pair (jp = j - k, j); see the comment above.
// Returns false (after reporting) when the panel has an exactly-zero pivot; the
// outputs of that pair are then not written.
//
// The nr <= NRM border rows are spread over the whole warp: lane = r * LPR +
// cg holds columns cg*CPL .. cg*CPL + CPL - 1 of border row r (LPR = 32 / NRM
// lanes per row), so their eliminations (C_j U^-1, then -C' L^-1) run in the
// same instructions as everyone else instead of on nr lanes alone.
//
// PAD: blocks of order n < N, as the leading part of blocks of order N.  Panel
// lanes are N apart (TOP row r on lane r, BOTTOM row r on lane N + r); the lanes
// and columns beyond n hold zeros or are never stored.  Positions are those of
// the 2n rows; in shared memory the reduced rows start at row N.
template <int N, int NRM, typename T = double, bool PAD = false>
__device__ __forceinline__ bool tc_pair(const FactorArgs<T>& a, int j, int k, bool first, T* Wt, int lane,
                                        const TcTree& tr) {
  using S = TcShape<N, T>;
  constexpr unsigned FULL = 0xffffffffu;
  T* Gs = Wt + S::WS;
  int* rowof = reinterpret_cast<int*>(Gs + S::GS);
  const Dims d = a.d;
  const int nr = d.nr, nx = d.nx;
  const int n = PAD ? d.n : N, n2 = 2 * n;
  const size_t nn = (size_t)n * n;
  const size_t nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  const int nrf = a.nrf;             // fused right-hand sides
  const bool top = lane < N;
  const int ri = lane & (N - 1);
  const bool act = lane < 2 * N && ri < n;
  const int g = lane >> 2, t = lane & 3;
  const int jp = j - k;
  // block elements: the loaded FP64 matrix at the first level, the working
  // copy (type T) after it; always through L2 (see ldw)
  using SrcT = typename std::conditional<sizeof(T) == 8, double, T>::type;
  const SrcT* srcD = first ? (const SrcT*)a.D0 : (const SrcT*)a.D;
  const SrcT* srcE = first ? (const SrcT*)a.E0 : (const SrcT*)a.E;
  const SrcT* srcB = first ? (const SrcT*)a.B0 : (const SrcT*)a.B;
  const SrcT* srcC = first ? (const SrcT*)a.C0 : (const SrcT*)a.C;
  auto lds = [&](const SrcT* base, const double* orig, size_t i) -> T {
    if constexpr (sizeof(T) == 8) return ldw(base + i);
    else return first ? T(ldw(orig + i)) : __ldcg(base + i);
  };
  // ------------------------------------------------------------ load
  constexpr int LPR = 32 / NRM, CPL = N / LPR;   // border layout (see above)
  const int br = lane / LPR, bc0 = (lane % LPR) * CPL;
  const bool blive = br < nr;
  T rowA[N], cb[CPL];
  double cs1[2] = {0.0, 0.0}, cs2[2] = {0.0, 0.0};  // children's F / xb sums (tree)
  auto load_panel = [&]() {
    const size_t po = top ? (size_t)jp * nn : (size_t)j * nn;
    const SrcT* Pm = (top ? srcE : srcD) + po;
    const double* Po = (top ? a.E0 : a.D0) + po;
#pragma unroll
    for (int c = 0; c < N; ++c) rowA[c] = act && (!PAD || c < n) ? lds(Pm, Po, (size_t)c * n + ri) : T(0);
#pragma unroll
    for (int q = 0; q < CPL; ++q)
      cb[q] = blive && (!PAD || bc0 + q < n) ? lds(srcC, a.C0, (size_t)j * nrn + (size_t)(bc0 + q) * nr + br) : T(0);
    // C_jpp contributions of the pairs (j - 2K', j - K') of earlier levels,
    // K' = 1, 2, ..., gather: loaded eight levels at a time so that their
    // latencies overlap, then added in level order
    for (int e0 = 0; e0 < 31 && (1 << e0) <= tr.gather; e0 += 8) {
      T v[8][CPL];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int kk = e0 + e < 31 ? 1 << (e0 + e) : 0;
        const bool on = blive && kk != 0 && kk <= tr.gather;
#pragma unroll
        for (int q = 0; q < CPL; ++q)
          v[e][q] = on ? T(__ldcg(a.Rbuf + (size_t)(j - kk) * nrn + (size_t)(bc0 + q) * nr + br)) : T(0);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int q = 0; q < CPL; ++q) cb[q] += v[e][q];
    }
  };
  load_panel();
  {
    // the children's F / xb partial sums of the two border-tile elements this
    // lane holds in the product (row 2N + g, columns 2N + 2t + {0, 1})
    if ((tr.c1 | tr.c2) && g < nr) {
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int cl = 2 * t + hh;
        const double* base = nullptr;
        size_t stride = 0, e = 0;
        if (cl < nx) { base = a.Fbuf; stride = nrnx; e = (size_t)cl * nr + g; }
        else if (cl < nx + nrf) { base = a.XB; stride = (size_t)nr * nrf; e = (size_t)(cl - nx) * nr + g; }
        if (base) {
          if (tr.c1) cs1[hh] = ldw(base + (size_t)tr.c1 * stride + e);
          if (tr.c2) cs2[hh] = ldw(base + (size_t)tr.c2 * stride + e);
        }
      }
    }
    // trailing columns in the original row order: TOP [D_jp 0 B_jp], BOTTOM [0 E_j
    // B_j] and the fused right-hand sides (TOP x_jp, BOTTOM x_j); columns beyond
    // them are not set (they feed outputs that are not stored).  Compile-time
    // trip counts: every load of the pair is issued before the first one is
    // consumed, so a lone pair pays one memory latency
    const SrcT* Djp = srcD + (size_t)jp * nn;
    const SrcT* Ej = srcE + (size_t)j * nn;
    const double* Djp0 = a.D0 + (size_t)jp * nn;
    const double* Ej0 = a.E0 + (size_t)j * nn;
#pragma unroll
    for (int it = 0; it < N * N / 32; ++it) {
      const int c = it * (32 / N) + lane / N;
      if (!PAD || (ri < n && c < n)) {
        Wt[ri * S::LDW + c] = lds(Djp, Djp0, (size_t)c * n + ri);
        Wt[(N + ri) * S::LDW + c] = lds(Ej, Ej0, (size_t)c * n + ri);
      }
    }
    if (act) {
      T* Wr = Wt + lane * S::LDW + N;
      const size_t bo = (size_t)(top ? jp : j) * nnx + ri;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nx) Wr[c] = lds(srcB + bo, a.B0 + bo, (size_t)c * n);
      const double* xr = a.x + (size_t)(top ? jp : j) * n + ri;
      for (int c = 0; c < nrf; ++c) Wr[nx + c] = T(ldw(xr + (size_t)c * a.ldx));
    }
    if (PAD) {  // rows of the product that no panel row fills
      if (lane < 2 * N) rowof[lane] = 0;
      __syncwarp();
    }
  }
  // ------------------- phase 1: panel LU with the operator rows in place
  // After step i a row not yet a pivot is orig_r + sum_{c <= i} X_r[c] orig(pivot c):
  // eliminating column i frees its register, which takes X_r[i] = -l, and the
  // same multiplier updates the X of the earlier columns with the pivot row's
  // X, so one run of N - 1 fused multiply-adds per step yields U, L^-1 (the
  // pivot rows' X, strictly lower), -M L^-1 and -C' L^-1 (see the comment above).
  // The registers rotate: rowA[0] is column i, a step moves every column one
  // register down and puts X_r[i] at the end, so that the steps are one rolled
  // loop that stays in the instruction cache (column c is at (c - i) mod N).
  // The pivot is found by reductions: the largest |a| (upper, then lower word),
  // then the smallest (position, lane).  Reciprocals of zero, tiny or huge pivots
  // need the correctly rounded routine, whose branch would wait for the search at
  // each step: such a pivot is only noted, and the panel run again with it.
  const int pos0 = act ? (top ? ri : n + ri) : 63;
  int mypos = pos0, info = 0;
  bool done = !act, bad = false;
  for (int attempt = 0;; ++attempt) {
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const T v0 = rowA[0];
      unsigned hi, lo;
      T rc;
      tc_candidate(v0, done, hi, lo, rc);
      const unsigned hmax = __reduce_max_sync(FULL, hi);
      bool in = hi == hmax;
      if constexpr (sizeof(T) == 8) {
        const unsigned lmax = __reduce_max_sync(FULL, in ? lo : 0u);
        in = in && lo == lmax;
      }
      const unsigned best = __reduce_min_sync(FULL, in ? ((unsigned)mypos << 5) | lane : 0xffffffffu);
      const int p = (int)(best & 31u), pmin = (int)(best >> 5);
      bad = bad || !tc_plain_pivot<T>(hmax);
      if (attempt) {
        if (!tc_plain_pivot<T>(hmax)) rc = v0 != T(0) ? rcp_rn(v0) : T(0);
        if (info == 0 && __shfl_sync(FULL, v0, p) == T(0)) info = i + 1;
      }
      const bool isp = lane == p;
      mypos = isp ? i : (mypos == i ? pmin : mypos);
      T* prow = Gs + i * S::LDG;  // the reciprocal, then the pivot row from column i + 1 on
      if (isp) {
        store2(&prow[0], rc, rowA[1]);
#pragma unroll
        for (int c = 2; c < N; c += 2) store2(&prow[c], rowA[c], rowA[c + 1]);
      }
      __syncwarp();
      done = done || isp;
      T u0, u1;
      load2(&prow[0], u0, u1);
      const T rinv = u0;
      const T l = done ? T(0) : v0 * rinv;
      rowA[0] = fma(-l, u1, rowA[1]);
#pragma unroll
      for (int c = 2; c < N; c += 2) {
        load2(&prow[c], u0, u1);
        rowA[c - 1] = fma(-l, u0, rowA[c]);
        rowA[c] = fma(-l, u1, rowA[c + 1]);
      }
      rowA[N - 1] = done ? v0 : -l;
      {  // border rows: multiplier from the lane holding column i of the row
        T ci = cb[0];
#pragma unroll
        for (int q = 1; q < CPL; ++q) ci = (i & (CPL - 1)) == q ? cb[q] : ci;
        const T lb = __shfl_sync(FULL, ci, (lane & ~(LPR - 1)) | (i / CPL)) * rinv;
#pragma unroll
        for (int q = 0; q < CPL; ++q) {
          const int at = (bc0 + q - i) & (N - 1);
          cb[q] = at == 0 ? -lb : fma(-lb, prow[at], cb[q]);
        }
      }
    }
    if (!bad || attempt) break;
    load_panel();
    mypos = pos0;
    done = !act;
  }
  if (info != 0) {
    if (lane == 0) report(a.st, DEV_ZERO_PIVOT, j, info, k);
    __syncwarp();
    return false;
  }
  if (PAD) {  // the rest of the rotation
#pragma unroll 1
    for (int i = n; i < N; ++i) {
      const T v0 = rowA[0];
#pragma unroll
      for (int c = 1; c < N; ++c) rowA[c - 1] = rowA[c];
      rowA[N - 1] = v0;
    }
  }
  // panel factors T_j in getrf row order (operator form: [L^-1 \ U; -M L^-1],
  // the unit diagonal of L^-1 not stored), pivots, the border operator
  // -C_j U^-1 L^-1; operator rows of the reduced and border rows for the product
  {
    T* Tj = a.Tm + (size_t)j * szT(d);
    if (act) {
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (!PAD || c < n) Tj[(size_t)mypos + (size_t)c * n2] = rowA[c];
      const int gr = mypos < n ? mypos : mypos - n + N;  // row of the product
      rowof[gr] = lane;
      a.P[(size_t)j * szP(d) + mypos] = (unsigned char)pos0;
      if (mypos >= n) {
#pragma unroll
        for (int c = 0; c < N; c += 2) store2(&Gs[gr * S::LDG + c], rowA[c], rowA[c + 1]);
      }
    }
#pragma unroll
    for (int q = 0; q < CPL; ++q) {
      if (blive && (!PAD || bc0 + q < n)) a.C[(size_t)j * nrn + (size_t)(bc0 + q) * nr + br] = cb[q];
      // border rows of G (zero for rows >= nr, and rows NRM..7 of the tile)
      Gs[(2 * N + br) * S::LDG + bc0 + q] = blive ? cb[q] : T(0);
      if constexpr (NRM < 8) Gs[(2 * N + NRM + br) * S::LDG + bc0 + q] = T(0);
    }
  }
  __syncwarp();
  // ----------------------------------------- phase 2: the product
  // G = [L^-1; -M L^-1; -C' L^-1] times (PW)_top: rows 0..N-1 of Gs hold L^-1
  // below the diagonal and U from the diagonal on, so those fragments are masked
  // to unit lower triangular (the tiles above the diagonal are skipped).
  // FP64 tensor cores (DMMA 8x8x4) for double, the FP32 pipe for float, with
  // the same accumulator layout; two passes over the column tiles keep the
  // accumulators within budget
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    constexpr int PC = S::PC;
    T acc[S::MTILES][PC][2];
#pragma unroll
    for (int mt = 0; mt < S::MTILES; ++mt)
#pragma unroll
      for (int ni = 0; ni < PC; ++ni) {
        const int nt = pass * PC + ni;
        const int row = mt * 8 + g;
        T c0 = T(0), c1 = T(0);
        if (nt < S::NTILES && row >= N && row < 2 * N) {  // (PW)_bot
          const int orow = rowof[row];
          c0 = tc_w<N>(Wt, orow, nt * 8 + 2 * t);
          c1 = tc_w<N>(Wt, orow, nt * 8 + 2 * t + 1);
        }
        acc[mt][ni][0] = c0;
        acc[mt][ni][1] = c1;
      }
    if constexpr (sizeof(T) == 8) {
#pragma unroll
      for (int ks = 0; ks < S::KSTEPS; ++ks) {
        double bfr[PC];
        const int orow = rowof[ks * 4 + t];
#pragma unroll
        for (int ni = 0; ni < PC; ++ni) {
          const int nt = pass * PC + ni;
          bfr[ni] = nt < S::NTILES ? tc_w<N>(Wt, orow, nt * 8 + g) : 0.0;
        }
#pragma unroll
        for (int mt = 0; mt < S::MTILES; ++mt) {
          if (mt * 8 < N && ks * 4 >= mt * 8 + 8) continue;  // above the diagonal of L^-1
          // (row r of L^-1 is stored from column r on, see phase 1)
          const int dk = ks * 4 + t - (mt * 8 + g);
          double afr = Gs[(mt * 8 + g) * S::LDG + (mt * 8 < N ? dk & (N - 1) : ks * 4 + t)];
          if (mt * 8 < N && ks * 4 + 3 >= mt * 8) afr = dk < 0 ? afr : dk == 0 ? 1.0 : 0.0;
#pragma unroll
          for (int ni = 0; ni < PC; ++ni)
            if (pass * PC + ni < S::NTILES) dmma_8x8x4(acc[mt][ni][0], acc[mt][ni][1], afr, bfr[ni]);
        }
      }
    } else {
      // element (8mt+g, 8nt+2t+h) += sum over kk of G(8mt+g, kk) (PW)_top(kk, 8nt+2t+h)
#pragma unroll 4
      for (int kk = 0; kk < N; ++kk) {
        const int orow = rowof[kk];
        T bv[PC][2];
#pragma unroll
        for (int ni = 0; ni < PC; ++ni) {
          const int nt = pass * PC + ni;
          bv[ni][0] = nt < S::NTILES ? tc_w<N>(Wt, orow, nt * 8 + 2 * t) : T(0);
          bv[ni][1] = nt < S::NTILES ? tc_w<N>(Wt, orow, nt * 8 + 2 * t + 1) : T(0);
        }
#pragma unroll
        for (int mt = 0; mt < S::MTILES; ++mt) {
          const int dk = kk - (mt * 8 + g);
          T av = Gs[(mt * 8 + g) * S::LDG + (mt * 8 < N ? dk & (N - 1) : kk)];
          if (mt * 8 < N) av = dk < 0 ? av : dk == 0 ? T(1) : T(0);
#pragma unroll
          for (int ni = 0; ni < PC; ++ni) {
            acc[mt][ni][0] = fma(av, bv[ni][0], acc[mt][ni][0]);
            acc[mt][ni][1] = fma(av, bv[ni][1], acc[mt][ni][1]);
          }
        }
      }
    }
    // ------------------------------------------------------------ store
    // accumulator element (row 8mt+g, column 8nt+2t+h) straight to its block:
    // rows [0,N) U-row, [N,2N) reduced row, [2N, 2N+nr) border updates;
    // columns [0,N) x_jp, [N,2N) x_jpp, [2N, 2N+nx) xb
    {
#pragma unroll
      for (int mt = 0; mt < S::MTILES; ++mt) {
        const int row = mt * 8 + g;
#pragma unroll
        for (int ni = 0; ni < PC; ++ni)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const int nt = pass * PC + ni;
            if (nt >= S::NTILES) continue;
            const int col = nt * 8 + 2 * t + hh;
            const T v = acc[mt][ni][hh];
            const int cj = col < N ? col : col < 2 * N ? col - N : col - 2 * N;  // column within its block
            if (mt * 8 < 2 * N) {  // panel rows (compile-time per mt)
              const bool ur = mt * 8 < N;
              const int rr = ur ? row : row - N;
              if (PAD && rr >= n) continue;
              const size_t blk = ur ? (size_t)j : (size_t)jp;
              if (nt * 8 < N) {
                if (!PAD || cj < n) a.D[blk * nn + (size_t)cj * n + rr] = v;
              } else if (nt * 8 < 2 * N) {
                if (!PAD || cj < n) a.E[blk * nn + (size_t)cj * n + rr] = v;
              } else if (cj < nx) {
                a.B[blk * nnx + (size_t)cj * n + rr] = v;
              } else if (cj < nx + nrf) {
                a.x[(size_t)(cj - nx) * a.ldx + blk * n + rr] = (double)v;
              }
            } else {
              const int rr = row - 2 * N;
              if (rr < nr) {
                if (nt * 8 < N) {
                  const size_t o = (size_t)jp * nrn + (size_t)cj * nr + rr;
                  if (!PAD || cj < n) a.C[o] = lds(srcC, a.C0, o) + v;
                } else if (nt * 8 < 2 * N) {
                  if (!PAD || cj < n) a.Rbuf[(size_t)j * nrn + (size_t)cj * nr + rr] = v;
                } else if (cj < nx) {
                  // own F update plus the partial sums of the child nodes (tree)
                  const size_t e = (size_t)cj * nr + rr;
                  a.Fbuf[(size_t)j * nrnx + e] = (double)v + cs1[hh] + cs2[hh];
                } else if (cj < nx + nrf) {
                  const size_t e = (size_t)(cj - nx) * nr + rr, nrr = (size_t)nr * nrf;
                  a.XB[(size_t)j * nrr + e] = (double)v + cs1[hh] + cs2[hh];
                }
              }
            }
          }
      }
    }
  }  // pass
  __syncwarp();
  return true;
}

// BOOK: the border bookkeeping of the tree schedule (see k_factor_tree_tc)
// in level-by-level launches: every pair gathers the C_j updates of the lower
// levels and adds its children's F / xb partial sums, so no border fix-up or
// reduction launch is needed between or after the levels (k_tree_root
// finishes C_nblock, F and xb after the last level).
// resident CTAs of 4 warps the register budget is sized for: FP32 pairs take
// half the shared memory and fewer registers, so more of them fit on an SM
template <typename T>
constexpr int tc_min_blocks() { return sizeof(T) == 8 ? 4 : 6; }

template <int N, bool BATCH = false, bool BOOK = false, int NRM = 8, typename T = double, bool PAD = false>
__global__ void __launch_bounds__(128, tc_min_blocks<T>())
    k_factor_lu_tc(FactorArgs<T> a0, const FactorArgs<T>* tab, const BatchCta* cmap) {
  using S = TcShape<N, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  FactorArgs<T> ab;  // this CTA's system (batch only)
  long q0, q1, qs;
  pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs);
  const FactorArgs<T>& a = BATCH ? ab : a0;
  T* Wt = reinterpret_cast<T*>(smem_raw + (size_t)warp * S::BYTES);
  TcTree tr{0, 0, 0};
  for (long q = q0; q < q1; q += qs) {
    const int j = a.k + (int)(2L * a.k * q);
    if constexpr (BOOK) {
      tr.gather = a.k / 2;
      tree_children(j, a.d.nblock, tr.c1, tr.c2);
    }
    tc_pair<N, NRM, T, PAD>(a, j, a.k, a.first != 0, Wt, lane, tr);
  }
}

// ---------------------------------------------------------------------------
// The whole cyclic reduction of one system in one launch (tree schedule).
//
// Node j >= 1 is the pair (j - K, j) of level K = lowbit(j).  Its TOP row
// jp = j - K is final once the pair (jp, jp + K/2) -- node j - K/2 -- is done
// (K >= 2); its BOTTOM row j once the last pair of row j's own chain, node
// j + k'' (k'' the largest power of two below K with j + k'' < nblock), is
// done.  So each node waits for at most two children, and each node has one
// parent: the next pair of row jp's chain (node jp + 2K, when jp is a multiple
// of 4K and jp + 2K < nblock), otherwise the pair that eliminates row jp
// (node jp); node jp = 0 is the root.  Warps take the level-1 nodes (the
// leaves) from a counter; a warp that finishes a node adds one to its
// parent's arrival counter, and the warp that brings the count to the
// parent's number of children carries on with the parent.  No warp ever
// waits for another: the schedule needs no grid barrier and cannot stall.
//
// The border bookkeeping of the level-by-level schedule moves into the tree:
// the C_jpp updates a pair leaves in Rbuf[j] are gathered by the node that
// eliminates that block (or, for C_nblock, by the root), and the F and xb
// updates are summed up the tree (each node adds its children's partial sums
// to its own, in a fixed order), so results are bit-reproducible run to run.
// ---------------------------------------------------------------------------
// parent node of node j, 0 for the root
__host__ __device__ inline int tree_parent(int j, int nb) {
  const int K = lowbit(j), jp = j - K;
  if ((jp & (4 * K - 1)) == 0 && jp + 2 * K < nb) return jp + 2 * K;
  return jp;
}
// children of node j (0: none): the TOP child, then the BOTTOM child
__host__ __device__ inline void tree_children(int j, int nb, int& c1, int& c2) {
  const int K = lowbit(j);
  c1 = K >= 2 ? j - K / 2 : 0;
  c2 = 0;
  if (K >= 2 && j + 1 < nb) {
    int kk = K / 2;
    while (j + kk >= nb) kk >>= 1;
    c2 = j + kk;
  }
}

struct TreeArgs {
  int* cnt;         // [nblock] arrival counters (zero at launch)
  int* leaf;        // next level-1 node to take (zero at launch)
  double* Ffin;     // out: F0 + all F updates (nr x nx, FP64)
  double* xb;       // fused solve: rows of xb in x (+= sum of the xb updates), or null
};

// Work of the root: C_nblock with the C_jpp updates of the pairs whose jpp is
// nblock (one per level at most, in level order), F = F0 + sum of every F
// update, xb += sum of every xb update.
template <int N>
__device__ void tree_root(const FactorArgs<double>& a, const TreeArgs& ta, int root, int lane) {
  const Dims d = a.d;
  const int nb = d.nblock, nr = d.nr, nx = d.nx;
  const size_t nrn = (size_t)nr * N, nrnx = (size_t)nr * nx;
  // the contributing pair of each level (0: none), found before any load so
  // that every load is in flight at once
  int src[31];
#pragma unroll
  for (int lev = 0; lev < 31; ++lev) {
    const int K = 1 << lev;
    const long np = K < nb ? pairs_at_level(nb, K) : 0;
    const int jl = np > 0 ? (int)(K * (2 * np - 1)) : 0;
    src[lev] = (np > 0 && jl + K >= nb) ? jl : 0;
  }
  for (size_t e = lane; e < nrn; e += 32) {
    double v[31];
#pragma unroll
    for (int lev = 0; lev < 31; ++lev) v[lev] = src[lev] ? ldw(a.Rbuf + (size_t)src[lev] * nrn + e) : 0.0;
    double s = ldw(a.C + (size_t)nb * nrn + e);
#pragma unroll
    for (int lev = 0; lev < 31; ++lev) s += v[lev];
    a.C[(size_t)nb * nrn + e] = s;
  }
  for (size_t e = lane; e < nrnx; e += 32) {
    const int r = (int)(e % nr), c = (int)(e / nr);
    ta.Ffin[e] = a.F0[(size_t)c * nr + r] + ldw(a.Fbuf + (size_t)root * nrnx + e);
  }
  if (ta.xb) {
    for (int e = lane; e < nr * a.nrf; e += 32) {
      const int r = e % nr, c = e / nr;
      ta.xb[(size_t)c * a.ldx + r] += ldw(a.XB + (size_t)root * nr * a.nrf + e);
    }
  }
}

// The top levels of the cyclic reduction (at most TOP_WARPS pairs each) in one
// launch of one CTA: each level's pairs go one per warp, then the CTA applies
// the level's C_jpp updates (k_border_fix's work) before the next level; one
// launch replaces two per level, whose fixed cost dominates there.
constexpr int TOP_WARPS = 16;

template <int N, int NRM, bool PAD = false>
__global__ void __launch_bounds__(TOP_WARPS * 32, 1) k_factor_top_tc(FactorArgs<double> a, int k_first) {
  using S = TcShape<N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* Wt = reinterpret_cast<double*>(smem_raw + (size_t)warp * S::BYTES);
  const TcTree none{0, 0, 0};
  const int nb = a.d.nblock;
  const size_t nrn = (size_t)a.d.nr * a.d.n;
  for (int k = k_first; k < nb; k *= 2) {
    const long np = pairs_at_level(nb, k);
    for (long q = warp; q < np; q += TOP_WARPS)
      tc_pair<N, NRM, double, PAD>(a, k + (int)(2L * k * q), k, k == 1, Wt, lane, none);
    __syncthreads();
    for (size_t e = threadIdx.x; e < (size_t)np * nrn; e += blockDim.x) {
      const long q = (long)(e / nrn);
      const size_t idx = e % nrn;
      const int j = k + (int)(2L * k * q), jpp = min(j + k, nb);
      a.C[(size_t)jpp * nrn + idx] += ldw(a.Rbuf + (size_t)j * nrn + idx);
    }
    __syncthreads();
  }
}

// the root work after level-by-level launches with the tree bookkeeping
template <int N>
__global__ void __launch_bounds__(32) k_tree_root(FactorArgs<double> a, TreeArgs ta, int root) {
  tree_root<N>(a, ta, root, threadIdx.x);
}

template <int N, int NRM>
__global__ void __launch_bounds__(128, 4) k_factor_tree_tc(FactorArgs<double> a, TreeArgs ta) {
  using S = TcShape<N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* Wt = reinterpret_cast<double*>(smem_raw + (size_t)warp * S::BYTES);
  const int nb = a.d.nblock;
  const long leaves = pairs_at_level(nb, 1);
  for (;;) {
    int q = 0;
    if (lane == 0) q = atomicAdd(ta.leaf, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= leaves) break;
    int j = 2 * q + 1;
    for (;;) {
      const int K = lowbit(j);
      TcTree tr;
      tr.gather = K / 2;
      tree_children(j, nb, tr.c1, tr.c2);
      tc_pair<N, NRM>(a, j, K, K == 1, Wt, lane, tr);
      const int par = tree_parent(j, nb);
      if (par == 0) {  // the root: every pair is done
        __threadfence();
        tree_root<N>(a, ta, j, lane);
        break;
      }
      // publish this node's results, then count the arrival at the parent
      __threadfence();
      int old = 0;
      if (lane == 0) old = atomicAdd(ta.cnt + par, 1);
      old = __shfl_sync(0xffffffffu, old, 0);
      int c1, c2;
      tree_children(par, nb, c1, c2);
      const int expected = (c1 != 0) + (c2 != 0);
      if (old + 1 < expected) break;  // the other child's warp will carry on
      __threadfence();                // acquire: the children's results are visible
      j = par;
    }
  }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory"); }

// ---------------------------------------------------------------------------
// LU pair kernel for n = 16 and n = 32 in either precision, and for 16 < n < 32
// padded.  One CTA per pair: 2N panel threads (one panel row each, in registers)
// plus one warp whose first nr lanes hold the border rows C_j.  As in the
// warp-per-pair kernel: register panel LU with the getrf pivot rule (the pivot
// search spans the panel warps: each posts its best candidate row and its
// reciprocal, one barrier per column, double-buffered by column parity) that
// keeps the operator G = [L^-1; -M L^-1; -C' L^-1] in the eliminated columns;
// then one product G * (P W)_top, on the
// FP64 tensor cores (DMMA 8x8x4) for double, as a 3xTF32 split on the tensor
// cores for float at n = 32, on the FP32 pipe for float at n = 16.
// ---------------------------------------------------------------------------
template <typename T, int N>
struct GrpShape {
  static constexpr int TPP = 2 * N;        // panel threads, one per panel row
  static constexpr int NTH = TPP + 32;     // + the border warp
  static constexpr int NWP = TPP / 32;     // warps in the pivot search
  static constexpr int NWA = NTH / 32;
  static constexpr int MT = 2 * N + 8;     // product rows: U-row, reduced row, border (nr <= 8)
  static constexpr int NTC = 2 * N + 8;    // trailing columns: x_jp, x_jpp, xb (nx <= 8)
  // trailing rows, compact: a TOP row keeps [D_jp | B_jp], a BOTTOM row
  // [E_j | B_j]; the structurally zero half of each row is not stored
  static constexpr int LDW = N + 8 + 1;
  static constexpr int LDG = N + 4;        // G rows (16-byte aligned rows, conflict-free fragments)
  static constexpr int LDS = N + 2;
  // FP64 product: DMMA tiles, warp w owns row tiles [w*RTW, (w+1)*RTW)
  static constexpr int MTILES = MT / 8, NTILES = NTC / 8;
  static constexpr int RTW = (MTILES + NWA - 1) / NWA;
  static constexpr int PC = NTILES % 3 == 0 ? 3 : NTILES;  // column tiles per pass
  // FP32 product: TR x TC thread grid, RPT x CPT elements per thread
  static constexpr int TR = 8, TC = NTH / TR;
  static constexpr int RPT = MT / TR, CPT = NTC / TC;
  static constexpr size_t BYTES =
      (size_t)(2 * N * LDW + MT * LDG + 2 * NWP * LDS) * sizeof(T) + (size_t)(2 * NWP * 4 + 2 * N) * sizeof(int);
  static_assert(MT % TR == 0 && NTC % TC == 0 && NTILES % PC == 0, "product tiling");
};

// element (row, col) of the trailing part of the work matrix from the compact
// rows: columns [0,N) x_jp (TOP rows only), [N,2N) x_jpp (BOTTOM rows only),
// [2N, 2N+8) xb
template <typename T, int N>
__device__ __forceinline__ T w_at(const T* Wt, int row, int col) {
  constexpr int LDW = GrpShape<T, N>::LDW;
  const bool top = row < N;
  if (col < N) return top ? Wt[row * LDW + col] : T(0);
  if (col < 2 * N) return top ? T(0) : Wt[row * LDW + col - N];
  return Wt[row * LDW + col - N];
}

// G * (P W)_top + [0; (P W)_bot; 0] -> the U-row of block j, the reduced row of
// block jp and the border updates (C_jp, the C_jpp buffer, the F buffer)
template <typename T, int N>
struct GrpProduct;

template <int N>
struct GrpProduct<double, N> {
  using S = GrpShape<double, N>;
  template <typename Out>
  __device__ static void run(const double* Wt, const double* Gs, const int* rowof, int t, Out out) {
    const int w = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    const int mt0 = w * S::RTW;
#pragma unroll
    for (int pass = 0; pass < S::NTILES / S::PC; ++pass) {
      double acc[S::RTW][S::PC][2];
#pragma unroll
      for (int mi = 0; mi < S::RTW; ++mi)
#pragma unroll
        for (int ni = 0; ni < S::PC; ++ni) {
          const int row = (mt0 + mi) * 8 + g, col = (pass * S::PC + ni) * 8 + 2 * q;
          double c0 = 0.0, c1 = 0.0;
          if (mt0 + mi < S::MTILES && row >= N && row < 2 * N) {
            const int orow = rowof[row];
            c0 = w_at<double, N>(Wt, orow, col);
            c1 = w_at<double, N>(Wt, orow, col + 1);
          }
          acc[mi][ni][0] = c0;
          acc[mi][ni][1] = c1;
        }
#pragma unroll
      for (int ks = 0; ks < N / 4; ++ks) {
        double bfr[S::PC];
        const int orow = rowof[ks * 4 + q];
#pragma unroll
        for (int ni = 0; ni < S::PC; ++ni) bfr[ni] = w_at<double, N>(Wt, orow, (pass * S::PC + ni) * 8 + g);
#pragma unroll
        for (int mi = 0; mi < S::RTW; ++mi) {
          if (mt0 + mi < S::MTILES) {
            const double afr = Gs[((mt0 + mi) * 8 + g) * S::LDG + ks * 4 + q];
#pragma unroll
            for (int ni = 0; ni < S::PC; ++ni) dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], afr, bfr[ni]);
          }
        }
      }
#pragma unroll
      for (int mi = 0; mi < S::RTW; ++mi)
        if (mt0 + mi < S::MTILES)
#pragma unroll
          for (int ni = 0; ni < S::PC; ++ni)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
              out((mt0 + mi) * 8 + g, (pass * S::PC + ni) * 8 + 2 * q + hh, acc[mi][ni][hh]);
    }
  }
};

template <int N>
struct GrpProduct<float, N> {
  using S = GrpShape<float, N>;
  template <typename Out>
  __device__ static void run(const float* Wt, const float* Gs, const int* rowof, int t, Out out) {
    const int tr = t % S::TR, tc = t / S::TR;
    float acc[S::RPT][S::CPT];
#pragma unroll
    for (int ii = 0; ii < S::RPT; ++ii) {
      const int row = tr + S::TR * ii;
#pragma unroll
      for (int jj = 0; jj < S::CPT; ++jj)
        acc[ii][jj] = (row >= N && row < 2 * N) ? w_at<float, N>(Wt, rowof[row], tc + S::TC * jj) : 0.0f;
    }
#pragma unroll 4
    for (int kk = 0; kk < N; ++kk) {
      const int orow = rowof[kk];
      float bv[S::CPT], av[S::RPT];
#pragma unroll
      for (int jj = 0; jj < S::CPT; ++jj) bv[jj] = w_at<float, N>(Wt, orow, tc + S::TC * jj);
#pragma unroll
      for (int ii = 0; ii < S::RPT; ++ii) av[ii] = Gs[(tr + S::TR * ii) * S::LDG + kk];
#pragma unroll
      for (int ii = 0; ii < S::RPT; ++ii)
#pragma unroll
        for (int jj = 0; jj < S::CPT; ++jj) acc[ii][jj] = fmaf(av[ii], bv[jj], acc[ii][jj]);
    }
#pragma unroll
    for (int ii = 0; ii < S::RPT; ++ii)
#pragma unroll
      for (int jj = 0; jj < S::CPT; ++jj) out(tr + S::TR * ii, tc + S::TC * jj, acc[ii][jj]);
  }
};

// FP32 n=32: the product on the tensor cores as a 3xTF32 split
// (mma.sync m16n8k8: a*b ~ a_small*b_big + a_big*b_small + a_big*b_big with
// a_big = tf32(a), a_small = tf32(a - a_big), FP32 accumulators), close to
// FP32 accuracy at a tenth of the FMA product's instructions.  Warp w owns
// column tiles [3w, 3w+3) of all five 16-row tiles (rows >= 72 are padding).
__device__ __forceinline__ unsigned to_tf32(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void split_tf32(float x, unsigned& big, unsigned& small) {
  big = to_tf32(x);
  small = to_tf32(x - __uint_as_float(big));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <>
struct GrpProduct<float, 32> {
  static constexpr int N = 32;
  using S = GrpShape<float, N>;
  static constexpr int M16 = (S::MT + 15) / 16, NPW = S::NTILES / S::NWA;
  static_assert(S::NTILES % S::NWA == 0, "column tiles per warp");
  template <typename Out>
  __device__ static void run(const float* Wt, const float* Gs, const int* rowof, int t, Out out) {
    const int w = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    float acc[M16][NPW][4];
    // [0; (P W)_bot; 0]: accumulator element c0..c3 = (row r, col c), (r, c+1),
    // (r+8, c), (r+8, c+1) with r = 16 mi + g, c = 8 nt + 2q
#pragma unroll
    for (int mi = 0; mi < M16; ++mi)
#pragma unroll
      for (int ni = 0; ni < NPW; ++ni) {
        const int col = (w * NPW + ni) * 8 + 2 * q;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = mi * 16 + g + 8 * h;
          const bool bot = row >= N && row < 2 * N;
          const int orow = bot ? rowof[row] : 0;
          acc[mi][ni][2 * h] = bot ? w_at<float, N>(Wt, orow, col) : 0.0f;
          acc[mi][ni][2 * h + 1] = bot ? w_at<float, N>(Wt, orow, col + 1) : 0.0f;
        }
      }
#pragma unroll
    for (int ks = 0; ks < N / 8; ++ks) {
      // B fragment of (P W)_top: (k = 8 ks + q, col = 8 nt + g) and k + 4
      const int o0 = rowof[ks * 8 + q], o1 = rowof[ks * 8 + q + 4];
      unsigned bb[NPW][2], bs[NPW][2];
#pragma unroll
      for (int ni = 0; ni < NPW; ++ni) {
        const int col = (w * NPW + ni) * 8 + g;
        split_tf32(w_at<float, N>(Wt, o0, col), bb[ni][0], bs[ni][0]);
        split_tf32(w_at<float, N>(Wt, o1, col), bb[ni][1], bs[ni][1]);
      }
#pragma unroll
      for (int mi = 0; mi < M16; ++mi) {
        // A fragment of G: (r, k), (r + 8, k), (r, k + 4), (r + 8, k + 4)
        const int r0 = mi * 16 + g, r1 = r0 + 8, kk = ks * 8 + q;
        const float av[4] = {r0 < S::MT ? Gs[r0 * S::LDG + kk] : 0.0f, r1 < S::MT ? Gs[r1 * S::LDG + kk] : 0.0f,
                             r0 < S::MT ? Gs[r0 * S::LDG + kk + 4] : 0.0f,
                             r1 < S::MT ? Gs[r1 * S::LDG + kk + 4] : 0.0f};
        unsigned ab[4], as[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split_tf32(av[e], ab[e], as[e]);
#pragma unroll
        for (int ni = 0; ni < NPW; ++ni) {
          mma_tf32(acc[mi][ni], as, bb[ni][0], bb[ni][1]);
          mma_tf32(acc[mi][ni], ab, bs[ni][0], bs[ni][1]);
          mma_tf32(acc[mi][ni], ab, bb[ni][0], bb[ni][1]);
        }
      }
    }
#pragma unroll
    for (int mi = 0; mi < M16; ++mi)
#pragma unroll
      for (int ni = 0; ni < NPW; ++ni)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = mi * 16 + g + 8 * h, col = (w * NPW + ni) * 8 + 2 * q;
          if (row < S::MT) {
            out(row, col, acc[mi][ni][2 * h]);
            out(row, col + 1, acc[mi][ni][2 * h + 1]);
          }
        }
  }
};

// CTAs per SM the register budget is sized for (FP64 n=32 is shared-memory
// bound at 5, FP32 n=32 register bound at 6)
template <typename T, int N>
constexpr int grp_min_blocks() { return N == 32 ? (sizeof(T) == 8 ? 5 : 6) : 4; }

// 8-byte asynchronous copy to shared memory (completion: cp_async_wait)
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// Pairs [q0, q1) step qs of one system and level, one per CTA.  PAD: blocks of
// order n < N as the leading part of blocks of order N (see tc_pair).
//
// The pivot steps are one rolled loop over rotating registers (a step moves every
// column one register down and puts the operator's new column at the end, as in
// lub_panel), so that its code stays in the instruction cache: unrolled, with the
// triangular solve that the operator then needed, instruction fetch was the
// largest stall (3.3 of 12 cycles per issue, now 0.5).  The trailing columns
// arrive by asynchronous copies while the panel is factored.  n = 32, 8,192
// pairs: FP64 596 -> 509 us, FP32 506 -> 406 us; n = 20 (padded), 10,000 pairs:
// 728 us in the shared-memory kernel, 492 us.  Bound by the step's chain of
// reductions and its barrier.
template <typename T, int N, bool COH, bool PAD = false>
__device__ __forceinline__ void grp_body(const FactorArgs<T>& a, long q0, long q1, long qs) {
  using S = GrpShape<T, N>;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr bool ASYNC = sizeof(T) == 8 && !COH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_info;
  T* Wt = reinterpret_cast<T*>(smem_raw);          // [2N][LDW] trailing columns, original rows
  T* Gs = Wt + 2 * N * S::LDW;                     // [MT][LDG] operator rows
  T* slot = Gs + S::MT * S::LDG;                   // [2][NWP][LDS] candidate: reciprocal, then its row from the next column on
  int* hdr = reinterpret_cast<int*>(slot + 2 * S::NWP * S::LDS);  // [2][NWP][4] |a| (two words), position and thread
  int* rowof = hdr + 2 * S::NWP * 4;               // row of the product -> panel row
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const Dims d = a.d;
  const int nr = d.nr, nx = d.nx;
  const int n = PAD ? d.n : N, n2 = 2 * n;
  const size_t nn = (size_t)n * n;
  const size_t nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  const int k = a.k;
  const bool first = a.first != 0;
  const bool panel = t < 2 * N;                 // panel row t
  const bool top = t < N;
  const int ri = t & (N - 1);
  const bool act = panel && ri < n;
  const bool brow = !panel && t - 2 * N < nr;   // border row t - 2N
  const int pos0 = act ? (top ? ri : n + ri) : 255;

  for (long qq = q0; qq < q1; qq += qs) {
    const int j = k + (int)(2L * k * qq), jp = j - k;
    __syncthreads();  // the previous pair's readers of Wt/Gs are done
    if (t == 0) s_info = 0;
    if (PAD && t < 2 * N) rowof[t] = 0;  // rows of the product that no panel row fills
    // ------------------------------------------------------------ load
    T row[N];
    auto load_rows = [&](const auto* D, const auto* E, const auto* C) {
      const auto* P = panel ? (top ? E + (size_t)jp * nn : D + (size_t)j * nn) + ri
                            : C + (size_t)j * nrn + (t - 2 * N);
      const int st = panel ? n : nr;
#pragma unroll
      for (int c = 0; c < N; ++c) row[c] = T(ld_batch_c<COH>((act || brow) && (!PAD || c < n), P + (size_t)c * st));
    };
    auto load = [&](const auto* D, const auto* E, const auto* Bm, const auto* C) {
      // trailing columns, compact: TOP rows [D_jp B_jp], BOTTOM rows [E_j B_j]; one
      // element of both per thread and round
      constexpr int IT = (N * N + S::NTH - 1) / S::NTH, IB = (8 * N + S::NTH - 1) / S::NTH;
      if constexpr (ASYNC) {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
          const int idx = t + S::NTH * it, r = idx & (N - 1), c = idx / N;
          if (idx < N * N && (!PAD || (r < n && c < n))) {
            cp_async8(Wt + r * S::LDW + c, D + (size_t)jp * nn + (size_t)c * n + r);
            cp_async8(Wt + (N + r) * S::LDW + c, E + (size_t)j * nn + (size_t)c * n + r);
          }
        }
#pragma unroll
        for (int it = 0; it < IB; ++it) {
          const int idx = t + S::NTH * it, r = idx & (N - 1), c = idx / N;
          if (c < nx && (!PAD || r < n)) {
            cp_async8(Wt + r * S::LDW + N + c, Bm + (size_t)jp * nnx + (size_t)c * n + r);
            cp_async8(Wt + (N + r) * S::LDW + N + c, Bm + (size_t)j * nnx + (size_t)c * n + r);
          }
        }
        cp_async_commit();
      }
      load_rows(D, E, C);
      if constexpr (!ASYNC) {
        constexpr int H = 4;  // rounds in flight
        for (int i0 = 0; i0 < IT; i0 += H) {
          T vd[H], ve[H];
#pragma unroll
          for (int u = 0; u < H; ++u) {
            const int idx = t + S::NTH * (i0 + u), r = idx & (N - 1), c = idx / N;
            const bool in = idx < N * N && (!PAD || (r < n && c < n));
            vd[u] = T(ld_batch_c<COH>(in, D + (size_t)jp * nn + (size_t)c * n + r));
            ve[u] = T(ld_batch_c<COH>(in, E + (size_t)j * nn + (size_t)c * n + r));
          }
#pragma unroll
          for (int u = 0; u < H; ++u) {
            const int idx = t + S::NTH * (i0 + u), r = idx & (N - 1), c = idx / N;
            if (idx < N * N) {
              Wt[r * S::LDW + c] = vd[u];
              Wt[(N + r) * S::LDW + c] = ve[u];
            }
          }
        }
        T vt[IB], vb[IB];
#pragma unroll
        for (int it = 0; it < IB; ++it) {
          const int idx = t + S::NTH * it, r = idx & (N - 1), c = idx / N;
          const bool in = c < nx && (!PAD || r < n);
          vt[it] = T(ld_batch_c<COH>(in, Bm + (size_t)jp * nnx + (size_t)c * n + r));
          vb[it] = T(ld_batch_c<COH>(in, Bm + (size_t)j * nnx + (size_t)c * n + r));
        }
#pragma unroll
        for (int it = 0; it < IB; ++it) {
          const int idx = t + S::NTH * it, r = idx & (N - 1), c = idx / N;
          if (c < 8) {
            Wt[r * S::LDW + N + c] = vt[it];
            Wt[(N + r) * S::LDW + N + c] = vb[it];
          }
        }
      }
    };
    if (first) load(a.D0, a.E0, a.B0, a.C0);
    else load(a.D, a.E, a.B, a.C);
    // ------------------- phase 1: panel LU with the operator rows in place
    // (zero, tiny and huge pivots are only noted, and the panel run again with
    // their reciprocals: see tc_pair)
    int mypos = pos0;
    bool done = !act, used = false, bad = false;  // border and idle lanes never pivot
    for (int attempt = 0;; ++attempt) {
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      // row[0] is column i
      const int par = i & 1;
      const T v0 = row[0];
      if (w < S::NWP) {
        unsigned hi, lo;
        T rc;
        tc_candidate(v0, done, hi, lo, rc);
        const unsigned hmax = __reduce_max_sync(FULL, hi);
        unsigned lmax = 0u;
        bool in = hi == hmax && !done;
        if constexpr (sizeof(T) == 8) {
          lmax = __reduce_max_sync(FULL, hi == hmax ? lo : 0u);
          in = in && lo == lmax;
        }
        const unsigned best = __reduce_min_sync(FULL, in ? ((unsigned)mypos << 5) | lane : 0xffffffffu);
        if (attempt && hmax != 0u && !tc_plain_pivot<T>(hmax)) rc = v0 != T(0) ? rcp_rn(v0) : T(0);
        // where no candidate is left (hmax = 0, best all ones) lane 31 posts zeros
        if ((best & 31u) == (unsigned)lane) {
          reinterpret_cast<int4*>(hdr)[par * S::NWP + w] =
              make_int4((int)hmax, (int)lmax, (int)((best >> 5 << 8) | t), 0);
          T* sl = slot + (par * S::NWP + w) * S::LDS;
          store2(sl, rc, row[1]);
#pragma unroll
          for (int c = 2; c < N; c += 2) store2(sl + c, row[c], row[c + 1]);
        }
      }
      __syncthreads();
      int wb = 0;
      int4 hw = reinterpret_cast<const int4*>(hdr)[par * S::NWP];
      if (S::NWP == 2) {
        const int4 h1 = reinterpret_cast<const int4*>(hdr)[par * S::NWP + 1];
        const unsigned hi0 = (unsigned)hw.x, hi1 = (unsigned)h1.x;
        const unsigned lo0 = (unsigned)hw.y, lo1 = (unsigned)h1.y;
        if (hi1 > hi0 || (hi1 == hi0 && (lo1 > lo0 || (lo1 == lo0 && h1.z < hw.z)))) {
          wb = 1;
          hw = h1;
        }
      }
      bad = bad || !tc_plain_pivot<T>((unsigned)hw.x);
      const int p = hw.z & 255, pmin = (hw.z >> 8) & 255;
      const T* u = slot + (par * S::NWP + wb) * S::LDS;
      mypos = mypos == i ? pmin : mypos;
      if (t == p) {
        mypos = i;
        done = used = true;
        if (attempt && v0 == T(0) && s_info == 0) s_info = i + 1;
      }
      T u0, u1;
      load2(u, u0, u1);
      const T l = used ? T(0) : v0 * u0;
      row[0] = fma(-l, u1, row[1]);
#pragma unroll
      for (int c = 2; c < N; c += 2) {
        load2(u + c, u0, u1);
        row[c - 1] = fma(-l, u0, row[c]);
        row[c] = fma(-l, u1, row[c + 1]);
      }
      row[N - 1] = used ? v0 : -l;
    }
      if (!bad || attempt) break;
      if (first) load_rows(a.D0, a.E0, a.C0);
      else load_rows(a.D, a.E, a.C);
      mypos = pos0;
      done = !act;
      used = false;
      __syncthreads();  // the last step's readers of the slots are done
    }
    if (PAD) {  // the rest of the rotation
#pragma unroll 1
      for (int i = n; i < N; ++i) {
        const T v0 = row[0];
#pragma unroll
        for (int c = 1; c < N; ++c) row[c - 1] = row[c];
        row[N - 1] = v0;
      }
    }
    // panel factors T_j in getrf row order (operator form), row map, the border
    // operator; operator rows for the product (pivot rows: unit lower triangle)
    __syncthreads();
    if (s_info != 0) {
      if (t == 0) report(a.st, DEV_ZERO_PIVOT, j, s_info, k);
      if constexpr (ASYNC) cp_async_wait<0>();
      continue;
    }
    if (act) {
      T* Tj = a.Tm + (size_t)j * szT(d);
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (!PAD || c < n) Tj[(size_t)mypos + (size_t)c * n2] = row[c];
      const int gr = mypos < n ? mypos : mypos - n + N;
      rowof[gr] = t;
      a.P[(size_t)j * szP(d) + mypos] = (unsigned char)pos0;
      T* G = Gs + gr * S::LDG;
      const int dg = mypos < n ? mypos : N;  // unit diagonal
#pragma unroll
      for (int c = 0; c < N; c += 2)
        store2(G + c, c < dg ? row[c] : c == dg ? T(1) : T(0), c + 1 < dg ? row[c + 1] : c + 1 == dg ? T(1) : T(0));
    } else if (!panel && t - 2 * N < 8) {
      T* Cj = a.C + (size_t)j * nrn + (t - 2 * N);
      T* G = Gs + t * S::LDG;
#pragma unroll
      for (int c = 0; c < N; ++c) {
        if (brow && (!PAD || c < n)) Cj[(size_t)c * nr] = row[c];
        G[c] = brow ? row[c] : T(0);
      }
    }
    if constexpr (ASYNC) cp_async_wait<0>();
    __syncthreads();
    // ------------------------------------------ phase 2: G * (P W)_top
    GrpProduct<T, N>::run(Wt, Gs, rowof, t, [&](int prow, int col, T v) {
      const int cj = col < N ? col : col < 2 * N ? col - N : col - 2 * N;
      if (prow < 2 * N) {
        const bool ur = prow < N;
        const int rr = ur ? prow : prow - N;
        const size_t blk = ur ? (size_t)j : (size_t)jp;
        if (PAD && rr >= n) return;
        if (col < N) {
          if (!PAD || cj < n) a.D[blk * nn + (size_t)cj * n + rr] = v;
        } else if (col < 2 * N) {
          if (!PAD || cj < n) a.E[blk * nn + (size_t)cj * n + rr] = v;
        } else if (cj < nx) {
          a.B[blk * nnx + (size_t)cj * n + rr] = v;
        }
      } else {
        const int rr = prow - 2 * N;
        if (rr < nr) {
          if (col < N) {
            const size_t o = (size_t)jp * nrn + (size_t)cj * nr + rr;
            if (!PAD || cj < n) a.C[o] = ldsrc_c<COH>(first, a.C0, a.C, o) + v;
          } else if (col < 2 * N) {
            if (!PAD || cj < n) a.Rbuf[(size_t)j * nrn + (size_t)cj * nr + rr] = v;
          } else if (cj < nx) {
            a.Fbuf[(size_t)j * nrnx + (size_t)cj * nr + rr] = (double)v;
          }
        }
      }
    });
  }
}

template <typename T, int N, bool BATCH = false, bool PAD = false>
__global__ void __launch_bounds__(2 * N + 32, grp_min_blocks<T, N>())
    k_factor_lu_grp(FactorArgs<T> a0, const FactorArgs<T>* tab, const BatchCta* cmap) {
  FactorArgs<T> ab;  // this CTA's system (batch only)
  long q0, q1, qs;
  pair_range<BATCH>(a0, tab, cmap, 1, 0, ab, q0, q1, qs);
  grp_body<T, N, false, PAD>(BATCH ? ab : a0, q0, q1, qs);
}

// ---------------------------------------------------------------------------
// Large blocks, FP32 LU where the tensor-core kernel does not apply: blocked
// right-looking elimination of the pair's work matrix (one CTA per pair, the matrix in the CTA's global slab, L2
// resident).  The panel columns go in blocks of BLK_W: a block is factored in
// shared memory with the getrf pivot rule (border rows eliminated, never
// pivots), its row interchanges are applied to every other column, the
// BLK_W rows of the trailing columns are solved with the block's unit lower
// triangle, and the rows below are updated with one product of depth BLK_W
// (FMA tiles).  FP64 blocks go to k_factor_lu_lub.  The result equals the unblocked elimination (getrf on the panel followed by
// the trailing updates) up to rounding order.
// ---------------------------------------------------------------------------
constexpr int BLK_W = 32;
constexpr int BLK_ROWS_MAX = 512;  // 2n + nr of the blocked kernel

// W[c*R + rowp[r]] -= sum_m L[m*LD + r] * W[c*R + rowp[k0 + m]] for positions r in
// [r0, R), c in [c0, NC), m < w; L: the factored block in shared memory (column m,
// position r); rowp: position -> row of W.  4 x 4 outputs per thread.
template <typename T>
__device__ void blk_update(T* W, int R, int NC, const T* Lsm, int LD, int k0, int w, int r0, int c0,
                           const int* rowp) {
  const int tid = threadIdx.x, bs = blockDim.x;
  const int rows = R - r0, cols = NC - c0;
  if (rows <= 0 || cols <= 0) return;
  const int tr = (rows + 3) / 4, tc = (cols + 3) / 4;
  for (int t = tid; t < tr * tc; t += bs) {
    const int rb = r0 + (t % tr) * 4, cb = c0 + (t / tr) * 4;
    T acc[4][4] = {};
#pragma unroll 4
    for (int m = 0; m < w; ++m) {
      T av[4], bv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        av[u] = rb + u < R ? Lsm[(size_t)m * LD + rb + u] : T(0);
        bv[u] = cb + u < NC ? W[(size_t)(cb + u) * R + rowp[k0 + m]] : T(0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fma(av[u], bv[v], acc[u][v]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v)
        if (rb + u < R && cb + v < NC) W[(size_t)(cb + v) * R + rowp[rb + u]] -= acc[u][v];
  }
}

// Blocked right-looking LU of the first npiv columns of the R x NC column-major
// matrix W (ld R) by one CTA: the getrf pivot rule among positions [i, ncand)
// (rows at positions >= ncand are eliminated but never pivots), the
// interchanges kept in the position -> row map s_perm (rows of W never move;
// s_perm holds the identity on entry), each block of BLK_W columns factored in
// shared memory Pb (BLK_W x R), the block's rows of the columns right of it
// solved with its unit lower triangle, the rows below updated with one product
// of depth BLK_W.  Returns the LAPACK info: 0, or the first zero pivot + 1.
template <typename T>
__device__ int blk_eliminate(T* W, int R, int NC, int npiv, int ncand, T* Pb, int* s_perm, T* sv, int* si) {
  const int tid = threadIdx.x, bs = blockDim.x;
  int info = 0;
  for (int kb = 0; kb < npiv && info == 0; kb += BLK_W) {
    const int w = npiv - kb < BLK_W ? npiv - kb : BLK_W;
    // stage the block's columns (all rows) in shared memory
    for (int e = tid; e < w * R; e += bs) {
      const int r = e % R, c = e / R;
      Pb[(size_t)c * R + r] = W[(size_t)(kb + c) * R + s_perm[r]];
    }
    __syncthreads();
    for (int i = 0; i < w; ++i) {
      const int gi = kb + i;
      T* ci = Pb + (size_t)i * R;
      T best = T(-1);
      int bi = gi;  // stays in range even when every candidate is NaN
      for (int r = gi + tid; r < ncand; r += bs) {
        const T v = dev_abs(ci[r]);
        if (v > best) { best = v; bi = r; }
      }
      block_argmax(best, bi, sv, si);
      const T pv = ci[bi];
      __syncthreads();  // every thread holds the pivot before the rows are swapped
      if (pv == T(0)) { info = gi + 1; break; }
      if (bi != gi && tid < w) {
        T* col = Pb + (size_t)tid * R;
        const T t = col[gi]; col[gi] = col[bi]; col[bi] = t;
      }
      if (bi != gi && tid == w) { const int t = s_perm[gi]; s_perm[gi] = s_perm[bi]; s_perm[bi] = t; }
      __syncthreads();
      // one thread per row below the pivot: its multiplier, then its update
      const T rinv = T(1) / pv;
      for (int r = gi + 1 + tid; r < R; r += bs) {
        const T l = ci[r] * rinv;
        ci[r] = l;
        for (int c = i + 1; c < w; ++c) Pb[(size_t)c * R + r] -= l * Pb[(size_t)c * R + gi];
      }
      __syncthreads();
    }
    if (info != 0) break;
    // the factored block back to the slab (by position)
    for (int e = tid; e < w * R; e += bs) {
      const int r = e % R, c = e / R;
      W[(size_t)(kb + c) * R + s_perm[r]] = Pb[(size_t)c * R + r];
    }
    __syncthreads();
    // rows [kb, kb+w) of the columns right of the block: unit lower solve
    for (int c = kb + w + tid; c < NC; c += bs) {
      T* col = W + (size_t)c * R;
      T y[BLK_W];
#pragma unroll
      for (int r = 0; r < BLK_W; ++r) y[r] = r < w ? col[s_perm[kb + r]] : T(0);
#pragma unroll
      for (int m = 0; m < BLK_W; ++m) {
#pragma unroll
        for (int r = m + 1; r < BLK_W; ++r)
          if (r < w) y[r] = fma(-Pb[(size_t)m * R + kb + r], y[m], y[r]);
      }
#pragma unroll
      for (int r = 0; r < BLK_W; ++r)
        if (r < w) col[s_perm[kb + r]] = y[r];
    }
    __syncthreads();
    // rows below the block: one product of depth w
    blk_update<T>(W, R, NC, Pb, R, kb, w, kb + w, kb + w, s_perm);
    __syncthreads();
  }
  return info;
}

template <typename T>
__global__ void __launch_bounds__(256, 2) k_factor_lu_blocked(FactorArgs<T> a, T* slab, size_t slab_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T sv[32];
  __shared__ int si[32];
  __shared__ int s_perm[BLK_ROWS_MAX];  // position -> row of the slab (rows never move)
  const int tid = threadIdx.x, bs = blockDim.x;
  const Dims d = a.d;
  const int n = d.n, nr = d.nr, nx = d.nx, nb = d.nblock;
  const int n2 = 2 * n, R = n2 + nr, NC = 3 * n + nx;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  T* Pb = reinterpret_cast<T*>(smem_raw);  // [BLK_W][R] the current panel block, column-major
  T* W = slab + (size_t)blockIdx.x * slab_elems;
  const int k = a.k;
  const long np = pairs_at_level(nb, k);
  const bool first = a.first != 0;
  for (long q = blockIdx.x; q < np; q += gridDim.x) {
    const int j = k + (int)(2L * k * q), jp = j - k;
    const size_t oj = (size_t)j * nn, ojp = (size_t)jp * nn;
    // ------------------------------------------------------------ load
    // groups of UL elements per thread: the group's loads are issued before its stores
    constexpr int UL = 4;
    for (int base = 0; base < (int)nn; base += bs * UL) {
      T ejp[UL], djp[UL], dj[UL], ej[UL];
#pragma unroll
      for (int u = 0; u < UL; ++u) {
        const int idx = base + tid + u * bs;
        const bool in = idx < (int)nn;
        ejp[u] = in ? ldg_src(first, a.E0, a.E, ojp + idx) : T(0);
        djp[u] = in ? ldg_src(first, a.D0, a.D, ojp + idx) : T(0);
        dj[u] = in ? ldg_src(first, a.D0, a.D, oj + idx) : T(0);
        ej[u] = in ? ldg_src(first, a.E0, a.E, oj + idx) : T(0);
      }
#pragma unroll
      for (int u = 0; u < UL; ++u) {
        const int idx = base + tid + u * bs;
        if (idx < (int)nn) {
          const int i = idx % n, c = idx / n;
          W[(size_t)c * R + i] = ejp[u];
          W[(size_t)(n + c) * R + i] = djp[u];
          W[(size_t)(n2 + c) * R + i] = T(0);
          W[(size_t)c * R + n + i] = dj[u];
          W[(size_t)(n + c) * R + n + i] = T(0);
          W[(size_t)(n2 + c) * R + n + i] = ej[u];
        }
      }
    }
    for (int idx = tid; idx < (int)nnx; idx += bs) {
      const int i = idx % n, c = idx / n;
      W[(size_t)(3 * n + c) * R + i] = ldsrc(first, a.B0, a.B, (size_t)jp * nnx + idx);
      W[(size_t)(3 * n + c) * R + n + i] = ldsrc(first, a.B0, a.B, (size_t)j * nnx + idx);
    }
    for (int idx = tid; idx < (int)nrn; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      W[(size_t)c * R + n2 + r] = ldsrc(first, a.C0, a.C, (size_t)j * nrn + idx);
      W[(size_t)(n + c) * R + n2 + r] = T(0);
      W[(size_t)(n2 + c) * R + n2 + r] = T(0);
    }
    for (int idx = tid; idx < (int)nrnx; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      W[(size_t)(3 * n + c) * R + n2 + r] = T(0);
    }
    for (int r = tid; r < R; r += bs) s_perm[r] = r;
    __syncthreads();
    // ------------------------------------------------- blocked elimination
    const int info = blk_eliminate<T>(W, R, NC, n, n2, Pb, s_perm, sv, si);
    if (info != 0) {
      if (tid == 0) report(a.st, DEV_ZERO_PIVOT, j, info, k);
      __syncthreads();
      continue;
    }
    // ---------------------------------------------------------------- store
    T* Tj = a.Tm + (size_t)j * szT(d);
    for (int base = 0; base < (int)(2 * nn); base += bs * UL) {
      T v[UL];
#pragma unroll
      for (int u = 0; u < UL; ++u) {
        const int idx = base + tid + u * bs;
        v[u] = idx < (int)(2 * nn) ? W[(size_t)(idx / n2) * R + s_perm[idx % n2]] : T(0);
      }
#pragma unroll
      for (int u = 0; u < UL; ++u) {
        const int idx = base + tid + u * bs;
        if (idx < (int)(2 * nn)) Tj[idx] = v[u];
      }
    }
    unsigned char* Pj = a.P + (size_t)j * szP(d);
    // row map (getrf order): the original row at each position
    for (int r = tid; r < n2; r += bs) Pj[r] = (unsigned char)s_perm[r];
    for (int i = tid; i < n; i += bs) Pj[n2 + i] = (unsigned char)i;
    for (int base = 0; base < (int)nn; base += bs * UL) {
      T v0[UL], v1[UL], v2[UL], v3[UL];
#pragma unroll
      for (int u = 0; u < UL; ++u) {
        const int idx = base + tid + u * bs;
        const int i = idx % n, c = idx / n;
        const bool in = idx < (int)nn;
        const int pu = in ? s_perm[i] : 0, pr = in ? s_perm[n + i] : 0;
        v0[u] = in ? W[(size_t)(n + c) * R + pu] : T(0);
        v1[u] = in ? W[(size_t)(n2 + c) * R + pu] : T(0);
        v2[u] = in ? W[(size_t)(n + c) * R + pr] : T(0);
        v3[u] = in ? W[(size_t)(n2 + c) * R + pr] : T(0);
      }
#pragma unroll
      for (int u = 0; u < UL; ++u) {
        const int idx = base + tid + u * bs;
        if (idx < (int)nn) {
          a.D[oj + idx] = v0[u];
          a.E[oj + idx] = v1[u];
          a.D[ojp + idx] = v2[u];
          a.E[ojp + idx] = v3[u];
        }
      }
    }
    for (int idx = tid; idx < (int)nnx; idx += bs) {
      const int i = idx % n, c = idx / n;
      a.B[(size_t)j * nnx + idx] = W[(size_t)(3 * n + c) * R + s_perm[i]];
      a.B[(size_t)jp * nnx + idx] = W[(size_t)(3 * n + c) * R + s_perm[n + i]];
    }
    for (int idx = tid; idx < (int)nrn; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      const size_t oc = (size_t)jp * nrn + idx;
      a.C[(size_t)j * nrn + idx] = W[(size_t)c * R + n2 + r];
      const T cjp = first ? T(a.C0[oc]) : a.C[oc];
      a.C[oc] = cjp + W[(size_t)(n + c) * R + n2 + r];
      a.Rbuf[(size_t)j * nrn + idx] = W[(size_t)(n2 + c) * R + n2 + r];
    }
    for (int idx = tid; idx < (int)nrnx; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      a.Fbuf[(size_t)j * nrnx + idx] = W[(size_t)(3 * n + c) * R + n2 + r];
    }
    __syncthreads();
  }
}

#include "bcr_umma.cuh"

// ---------------------------------------------------------------------------
// Large blocks: one CTA eliminates one pair; the (2n+nr) x (3n+nx) work
// matrix lives in a global scratch slab of the CTA (column-major, ld = R),
// which stays in L2 while the CTA works on it.  Same elimination as the warp
// kernels (getrf pivot rule, dlarfg reflectors, border rows eliminated by the
// U rows), parallelised over the CTA's threads with block barriers.
// ---------------------------------------------------------------------------
template <typename T, int SEL>
__global__ void __launch_bounds__(256) k_factor_cta(FactorArgs<T> a, T* slab, size_t slab_elems) {
  __shared__ T sv[32];
  __shared__ int si[32];
  __shared__ T s_tau[256];
  __shared__ int s_piv[256];
  const int tid = threadIdx.x, bs = blockDim.x;
  const Dims d = a.d;
  const int n = d.n, nr = d.nr, nx = d.nx, nb = d.nblock;
  const int n2 = 2 * n, R = n2 + nr, NC = 3 * n + nx;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  T* W = slab + (size_t)blockIdx.x * slab_elems;
  const int k = a.k;
  const long np = pairs_at_level(nb, k);
  const bool first = a.first != 0;
  for (long q = blockIdx.x; q < np; q += gridDim.x) {
    const int j = k + (int)(2L * k * q), jp = j - k;
    const size_t oj = (size_t)j * nn, ojp = (size_t)jp * nn;
    // ------------------------------------------------------------ load
    for (int idx = tid; idx < (int)nn; idx += bs) {
      const int i = idx % n, c = idx / n;
      T ejp, djp, dj, ej;
      if (first) {
        ejp = T(a.E0[ojp + idx]); djp = T(a.D0[ojp + idx]); dj = T(a.D0[oj + idx]); ej = T(a.E0[oj + idx]);
      } else {
        ejp = a.E[ojp + idx]; djp = a.D[ojp + idx]; dj = a.D[oj + idx]; ej = a.E[oj + idx];
      }
      W[(size_t)c * R + i] = ejp;
      W[(size_t)(n + c) * R + i] = djp;
      W[(size_t)(n2 + c) * R + i] = T(0);
      W[(size_t)c * R + n + i] = dj;
      W[(size_t)(n + c) * R + n + i] = T(0);
      W[(size_t)(n2 + c) * R + n + i] = ej;
    }
    for (int idx = tid; idx < (int)nnx; idx += bs) {
      const int i = idx % n, c = idx / n;
      const size_t o1 = (size_t)jp * nnx + idx, o2 = (size_t)j * nnx + idx;
      W[(size_t)(3 * n + c) * R + i] = first ? T(a.B0[o1]) : a.B[o1];
      W[(size_t)(3 * n + c) * R + n + i] = first ? T(a.B0[o2]) : a.B[o2];
    }
    for (int idx = tid; idx < (int)nrn; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      const size_t o = (size_t)j * nrn + idx;
      W[(size_t)c * R + n2 + r] = first ? T(a.C0[o]) : a.C[o];
      W[(size_t)(n + c) * R + n2 + r] = T(0);
      W[(size_t)(n2 + c) * R + n2 + r] = T(0);
    }
    for (int idx = tid; idx < (int)nrnx; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      W[(size_t)(3 * n + c) * R + n2 + r] = T(0);
    }
    __syncthreads();
    // ----------------------------------------------------------- eliminate
    int info = 0;
    for (int i = 0; i < n && info == 0; ++i) {
      T* ci = W + (size_t)i * R;
      if (SEL == SEL_QRP) {
        // column with the largest remaining 2-norm over the panel rows
        T best = T(-1);
        int bc = i;
        for (int c = i + tid; c < n; c += bs) {
          const T* col = W + (size_t)c * R;
          T s2 = T(0);
          for (int r = i; r < n2; ++r) s2 += col[r] * col[r];
          if (s2 > best) { best = s2; bc = c; }
        }
        block_argmax(best, bc, sv, si);
        if (tid == 0) s_piv[i] = bc;
        if (bc != i)
          for (int r = tid; r < R; r += bs) {
            T t = ci[r]; ci[r] = W[(size_t)bc * R + r]; W[(size_t)bc * R + r] = t;
          }
        __syncthreads();
      }
      if (SEL == SEL_LU) {
        T best = T(-1);
        int bi = i;
        for (int r = i + tid; r < n2; r += bs) {
          T v = dev_abs(ci[r]);
          if (v > best) { best = v; bi = r; }
        }
        block_argmax(best, bi, sv, si);
        if (tid == 0) s_piv[i] = bi;
        const T pv = ci[bi];
        __syncthreads();  // every thread holds the pivot before column i is swapped
        if (pv == T(0)) { info = i + 1; break; }
        if (bi != i)
          for (int c = tid; c < NC; c += bs) {
            T* col = W + (size_t)c * R;
            T t = col[i]; col[i] = col[bi]; col[bi] = t;
          }
        __syncthreads();
        const T rinv = T(1) / pv;
        for (int r = i + 1 + tid; r < R; r += bs) ci[r] *= rinv;
        __syncthreads();
      } else {
        const T alpha = ci[i];
        T s2 = T(0);
        for (int r = i + 1 + tid; r < n2; r += bs) s2 += ci[r] * ci[r];
        s2 = block_sum(s2, sv);
        T tt = T(0), beta = alpha;
        if (s2 != T(0)) {
          const T nrm = sqrt(alpha * alpha + s2);
          beta = alpha >= T(0) ? -nrm : nrm;
          tt = (beta - alpha) / beta;
          const T sc = T(1) / (alpha - beta);
          for (int r = i + 1 + tid; r < n2; r += bs) ci[r] *= sc;
        }
        __syncthreads();
        if (tid == 0) { ci[i] = beta; s_tau[i] = tt; if (SEL == SEL_QR) s_piv[i] = i; }
        __syncthreads();
        if (beta == T(0)) { info = i + 1; break; }
        if (tt != T(0))
          for (int c = i + 1 + tid; c < NC; c += bs) {
            T* col = W + (size_t)c * R;
            T w = col[i];
            for (int r = i + 1; r < n2; ++r) w += ci[r] * col[r];
            w *= tt;
            col[i] -= w;
            for (int r = i + 1; r < n2; ++r) col[r] -= w * ci[r];
          }
        __syncthreads();
        if (R > n2) {
          const T rb = T(1) / beta;
          for (int r = n2 + tid; r < R; r += bs) ci[r] *= rb;
          __syncthreads();
        }
      }
      // rank-1 update of the rows below i (LU) or of the border rows (QR/QRP)
      const int r0 = SEL == SEL_LU ? i + 1 : n2;
      const int rows = R - r0, cols = NC - i - 1;
      if (rows > 0 && cols > 0) {
        const long tot = (long)rows * cols;
        for (long e = tid; e < tot; e += bs) {
          const int r = r0 + (int)(e % rows), c = i + 1 + (int)(e / rows);
          T* col = W + (size_t)c * R;
          col[r] -= ci[r] * col[i];
        }
      }
      __syncthreads();
    }
    if (info != 0) {
      if (tid == 0) report(a.st, DEV_ZERO_PIVOT, j, info, k);
      __syncthreads();
      continue;
    }
    // ---------------------------------------------------------------- store
    T* Tj = a.Tm + (size_t)j * szT(d);
    for (int idx = tid; idx < (int)(2 * nn); idx += bs) {
      const int r = idx % n2, c = idx / n2;
      Tj[idx] = W[(size_t)c * R + r];
    }
    if (SEL != SEL_LU)
      for (int i = tid; i < n; i += bs) Tj[2 * nn + i] = s_tau[i];
    unsigned char* Pj = a.P + (size_t)j * szP(d);
    if (tid == 0) {
      // row map (getrf order) or QRP column map from the swap sequence
      unsigned char mp[768];
      for (int r = 0; r < n2; ++r) mp[r] = (unsigned char)r;
      for (int i = 0; i < n; ++i) mp[n2 + i] = (unsigned char)i;
      if (SEL == SEL_LU)
        for (int i = 0; i < n; ++i) { unsigned char t = mp[i]; mp[i] = mp[s_piv[i]]; mp[s_piv[i]] = t; }
      if (SEL == SEL_QRP)
        for (int i = 0; i < n; ++i) { unsigned char t = mp[n2 + i]; mp[n2 + i] = mp[n2 + s_piv[i]]; mp[n2 + s_piv[i]] = t; }
      for (int r = 0; r < 3 * n; ++r) Pj[r] = mp[r];
    }
    for (int idx = tid; idx < (int)nn; idx += bs) {
      const int i = idx % n, c = idx / n;
      a.D[oj + idx] = W[(size_t)(n + c) * R + i];
      a.E[oj + idx] = W[(size_t)(n2 + c) * R + i];
      a.D[ojp + idx] = W[(size_t)(n + c) * R + n + i];
      a.E[ojp + idx] = W[(size_t)(n2 + c) * R + n + i];
    }
    for (int idx = tid; idx < (int)nnx; idx += bs) {
      const int i = idx % n, c = idx / n;
      a.B[(size_t)j * nnx + idx] = W[(size_t)(3 * n + c) * R + i];
      a.B[(size_t)jp * nnx + idx] = W[(size_t)(3 * n + c) * R + n + i];
    }
    for (int idx = tid; idx < (int)nrn; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      const size_t oc = (size_t)jp * nrn + idx;
      a.C[(size_t)j * nrn + idx] = W[(size_t)c * R + n2 + r];
      const T cjp = first ? T(a.C0[oc]) : a.C[oc];
      a.C[oc] = cjp + W[(size_t)(n + c) * R + n2 + r];
      a.Rbuf[(size_t)j * nrn + idx] = W[(size_t)(n2 + c) * R + n2 + r];
    }
    for (int idx = tid; idx < (int)nrnx; idx += bs) {
      const int r = idx % nr, c = idx / nr;
      a.Fbuf[(size_t)j * nrnx + idx] = W[(size_t)(3 * n + c) * R + n2 + r];
    }
    __syncthreads();
  }
}

// copy of loaded FP64 blocks into the working precision
template <typename T>
__global__ void k_convert_blocks(const double* src, T* dst, size_t count) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x)
    dst[e] = T(src[e]);
}

// C_jpp += dC_jpp for every pair of the level (one writer per target block)
template <typename T>
__global__ void k_border_fix(Dims d, T* C, const T* Rbuf, int k) {
  const long np = pairs_at_level(d.nblock, k);
  const size_t nrn = (size_t)d.nr * d.n;
  const size_t total = (size_t)np * nrn;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const long q = (long)(e / nrn);
    const int idx = (int)(e % nrn);
    const int j = k + (int)(2L * k * q), jpp = min(j + k, d.nblock);
    C[(size_t)jpp * nrn + idx] += Rbuf[(size_t)j * nrn + idx];
  }
}

// ---------------------------------------------------------------------------
// deterministic sums of per-block m-vectors (m <= 256) over blocks
// [first, first+count): CTA g reduces a fixed chunk of blocks with a fixed
// thread-to-block map and a fixed shared-memory tree, so the result does not
// depend on timing.  With out == nullptr the CTA writes its partial to
// part[g]; otherwise (one CTA) it writes out = base + sum (column height h).
// ---------------------------------------------------------------------------
template <typename T>
__device__ void reduce_tree_body(const T* buf, int stride, long first, long count, int m, long chunk,
                                 T* part, const T* base, int h, int ldb, T* out, int ldo, int blk) {
  __shared__ T red[256];
  const int tid = threadIdx.x;
  const int S = 256 / m;  // items reduced in parallel per element
  const int e = tid % m, g = tid / m;
  const long b0 = first + (long)blk * chunk;
  const long b1 = min(first + count, b0 + chunk);
  T a0 = T(0), a1 = T(0);
  if (g < S) {  // eight loads in flight
    const T* p = buf + e;
    for (long b = b0 + g; b < b1; b += 8 * S) {
      T v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = ld_batch(b + u * S < b1, p + (size_t)(b + u * S) * stride);
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        a0 += v[u];
        a1 += v[u + 1];
      }
    }
  }
  red[tid] = a0 + a1;
  __syncthreads();
  for (int w = 1; w < S; w *= 2) {
    if (g < S && g % (2 * w) == 0 && g + w < S) red[tid] += red[tid + w * m];
    __syncthreads();
  }
  if (g == 0) {
    const T s = red[e];
    if (out) {
      const int r = e % h, c = e / h;
      out[(size_t)c * ldo + r] = (base ? base[(size_t)c * ldb + r] : T(0)) + s;
    } else {
      part[(size_t)blk * m + e] = s;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_reduce_tree(const T* buf, int stride, long first, long count,
                                                     int m, long chunk, T* part, const T* base, int h,
                                                     int ldb, T* out, int ldo) {
  reduce_tree_body(buf, stride, first, count, m, chunk, part, base, h, ldb, out, ldo, (int)blockIdx.x);
}

// ---------------------------------------------------------------------------
// solve sweeps (forward, cc:1615-1795; backward, cc:1805-2075)
// ---------------------------------------------------------------------------
// factors of type T (FP64, or FP32 for the mixed path); vectors always FP64
template <typename T>
struct SweepArgs {
  Dims d;
  const T *D, *E, *B, *C, *Tm;
  const unsigned char* P;
  double* x;
  int ldx, nrhs;
  double* XB;
  int k, ldw, sel;
  int op;           // T_j and C_j hold the operator form, by blocks of op columns (launch argument; 0: L and M)
  const int* done;  // batch, mixed path: nonzero once this system's refinement converged
};

template <typename T>
__device__ __forceinline__ bool system_active(const SweepArgs<T>& a) { return !(a.done && *a.done); }

__device__ __forceinline__ void take_level(SweepArgs<float>& a, const SweepArgs<float>& a0) { a.k = a0.k; }
__device__ __forceinline__ void take_level(SweepArgs<double>& a, const SweepArgs<double>& a0) { a.k = a0.k; }

#include "bcr_lub.cuh"

template <typename T, bool BATCH = false>
__global__ void __launch_bounds__(WARPS_PANEL * 32) k_forward_level(SweepArgs<T> a0, const SweepArgs<T>* tab,
                                                                const BatchCta* cmap, const long* ecnt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  for_entries<BATCH>(ecnt, [&](long entry) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    SweepArgs<T> ab;  // this CTA's system (batch only)
    long q0, q1, qs;
    pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs, entry);
    const SweepArgs<T>& a = BATCH ? ab : a0;
    const Dims d = a.d;
    const int n = d.n, nr = d.nr, n2 = 2 * n, nrhs = a.nrhs, ldw = a.ldw, k = a.k;
    double* W = reinterpret_cast<double*>(smem_raw) + (size_t)warp * ldw * nrhs;
    for (long q = q0; q < q1; q += qs) {
      const int j = k + (int)(2L * k * q), jp = j - k;
      const T* Tj = a.Tm + (size_t)j * szT(d);
      const unsigned char* Pj = a.P + (size_t)j * szP(d);
      for (int idx = lane; idx < n2 * nrhs; idx += 32) {
        const int pos = idx % n2, c = idx / n2;
        const int r = a.sel == SEL_LU ? Pj[pos] : pos;  // original row at this position
        const size_t o = (size_t)c * a.ldx + (r < n ? (size_t)jp * n + r : (size_t)j * n + (r - n));
        W[(size_t)c * ldw + pos] = a.x[o];
      }
      __syncwarp();
      if (a.sel == SEL_LU) {
        for (int i = 0; i < n; ++i) {
          for (int r = i + 1 + lane; r < n2; r += 32) {
            const double l = Tj[(size_t)i * n2 + r];
            for (int c = 0; c < nrhs; ++c) W[(size_t)c * ldw + r] -= l * W[(size_t)c * ldw + i];
          }
          __syncwarp();
        }
      } else {
        for (int i = 0; i < n; ++i) {
          const double t = Tj[2 * (size_t)n * n + i];
          const T* v = Tj + (size_t)i * n2;
          for (int c = 0; c < nrhs; ++c) {
            double* w = W + (size_t)c * ldw;
            double s = 0.0;
            for (int r = i + 1 + lane; r < n2; r += 32) s += double(v[r]) * w[r];
            s = warp_sum(s);
            s = (s + w[i]) * t;
            __syncwarp();
            if (lane == 0) w[i] -= s;
            for (int r = i + 1 + lane; r < n2; r += 32) w[r] -= s * double(v[r]);
            __syncwarp();
          }
        }
      }
      __syncwarp();
      for (int idx = lane; idx < n * nrhs; idx += 32) {
        const int i = idx % n, c = idx / n;
        a.x[(size_t)c * a.ldx + (size_t)jp * n + i] = W[(size_t)c * ldw + n + i];
        a.x[(size_t)c * a.ldx + (size_t)j * n + i] = W[(size_t)c * ldw + i];
      }
      if (nr > 0) {
        const T* Cj = a.C + (size_t)j * nr * n;
        for (int idx = lane; idx < nr * nrhs; idx += 32) {
          const int r = idx % nr, c = idx / nr;
          double s = 0.0;
          for (int i = 0; i < n; ++i) s += double(Cj[(size_t)i * nr + r]) * W[(size_t)c * ldw + i];
          a.XB[(size_t)j * nr * nrhs + idx] = -s;
        }
      }
      __syncwarp();
    }
  });
}

template <typename T, bool BATCH = false>
__global__ void __launch_bounds__(WARPS_PANEL * 32) k_backward_level(SweepArgs<T> a0, const SweepArgs<T>* tab,
                                                                 const BatchCta* cmap, const long* ecnt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  for_entries<BATCH>(ecnt, [&](long entry) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    SweepArgs<T> ab;  // this CTA's system (batch only)
    long q0, q1, qs;
    pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs, entry);
    const SweepArgs<T>& a = BATCH ? ab : a0;
    const Dims d = a.d;
    const int n = d.n, nx = d.nx, n2 = 2 * n, nrhs = a.nrhs, k = a.k, nb = d.nblock;
    double* Y = reinterpret_cast<double*>(smem_raw) + (size_t)warp * a.ldw;
    const size_t xb_off = (size_t)(nb + 1) * n + d.qx;
    for (long q = q0; q < q1; q += qs) {
      const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
      const T* Dj = a.D + (size_t)j * n * n;
      const T* Ej = a.E + (size_t)j * n * n;
      const T* Bj = a.B + (size_t)j * n * nx;
      const T* Tj = a.Tm + (size_t)j * szT(d);
      for (int c = 0; c < nrhs; ++c) {
        double* xc = a.x + (size_t)c * a.ldx;
        for (int i = lane; i < n; i += 32) {
          double s = xc[(size_t)j * n + i];
          for (int m = 0; m < n; ++m) s -= Dj[(size_t)m * n + i] * xc[(size_t)jp * n + m];
          for (int m = 0; m < n; ++m) s -= Ej[(size_t)m * n + i] * xc[(size_t)jpp * n + m];
          for (int m = 0; m < nx; ++m) s -= Bj[(size_t)m * n + i] * xc[xb_off + m];
          Y[i] = s;
        }
        __syncwarp();
        for (int i = n - 1; i >= 0; --i) {
          const double xi = Y[i] / double(Tj[(size_t)i * n2 + i]);
          __syncwarp();
          if (lane == 0) Y[i] = xi;
          for (int r = lane; r < i; r += 32) Y[r] -= Tj[(size_t)i * n2 + r] * xi;
          __syncwarp();
        }
        const unsigned char* cmap = a.P + (size_t)j * szP(d) + 2 * n;
        for (int i = lane; i < n; i += 32) xc[(size_t)j * n + (a.sel == SEL_QRP ? cmap[i] : i)] = Y[i];
        __syncwarp();
      }
    }
  });
}

// ---------------------------------------------------------------------------
// register-resident sweeps for n <= N <= 16: one warp per pair.
//
// forward (forward, cc:1615-1719): lane = position r < 2n of the stacked
//   [x_jp; x_j]; the row map gathers the original row with one shuffle, the
//   unit-lower L and M are applied by n broadcast steps (LU) or the n
//   Householder reflectors by warp reductions (QR/QRP); xb partial -C'_j x_j.
// backward (backward, cc:1805-2075): lanes 0..15 form D'_j x_jp, lanes
//   16..31 E'_j x_jpp for row i = lane & 15; the halves are combined, the B'_j
//   xb term added and U solved by n broadcast steps (QRP: column-map scatter).
// All loads of a pair are issued before the first use.
// ---------------------------------------------------------------------------
template <typename TF, int N, int NRM, bool LU, bool BATCH = false>
__global__ void __launch_bounds__(256, 2) k_forward_rows(SweepArgs<TF> a0, const SweepArgs<TF>* tab,
                                                         const BatchCta* cmap, const long* ecnt) {
  for_entries<BATCH>(ecnt, [&](long entry) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    SweepArgs<TF> ab;  // this CTA's system (batch only)
    long q0, q1, qs;
    pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs, entry);
    const SweepArgs<TF>& a = BATCH ? ab : a0;
    const Dims d = a.d;
    const int n = d.n, nr = d.nr, n2 = 2 * n, nrhs = a.nrhs, k = a.k;
    const bool act = lane < n2;
    constexpr bool lu = LU;
    const bool op = a0.op != 0;
    for (long q = q0; q < q1; q += qs) {
      const int j = k + (int)(2L * k * q), jp = j - k;
      const TF* Tj = a.Tm + (size_t)j * szT(d);
      double t[N];
  #pragma unroll
      for (int c = 0; c < N; ++c) t[c] = (act && c < n) ? double(Tj[(size_t)c * n2 + lane]) : 0.0;
      double tau[LU ? 1 : N];
  #pragma unroll
      for (int c = 0; c < (LU ? 1 : N); ++c) tau[c] = (!lu && c < n) ? Tj[2 * (size_t)n * n + c] : 0.0;
      const int src = (act && lu) ? (int)a.P[(size_t)j * szP(d) + lane] : lane;
      double cp[NRM];
      const TF* Cj = a.C + (size_t)j * nr * n;
  #pragma unroll
      for (int r = 0; r < NRM; ++r) cp[r] = (lane < n && r < nr) ? Cj[(size_t)lane * nr + r] : 0.0;
      for (int col = 0; col < nrhs; ++col) {
        double* xc = a.x + (size_t)col * a.ldx;
        const double orig = act ? (lane < n ? xc[(size_t)jp * n + lane] : xc[(size_t)j * n + lane - n]) : 0.0;
        double w = __shfl_sync(FULL, orig, src);
        const double b = w;
        if (lu && op) {  // the operator form: one product (see k_forward_pipe)
          double w2 = 0.0;
  #pragma unroll
          for (int i = 0; i < N; i += 2) {
            const double b0 = __shfl_sync(FULL, b, i), b1 = __shfl_sync(FULL, b, i + 1);
            if (i < n && lane > i) w = fma(t[i], b0, w);
            if (i + 1 < n && lane > i + 1) w2 = fma(t[i + 1], b1, w2);
          }
          w += w2;
        } else if (lu) {
  #pragma unroll
          for (int i = 0; i < N; ++i) {
            if (i < n) {
              const double wi = __shfl_sync(FULL, w, i);
              if (lane > i && act) w = fma(-t[i], wi, w);
            }
          }
        } else {
  #pragma unroll
          for (int i = 0; i < N; ++i) {
            if (i < n) {
              const double v = (lane > i && act) ? t[i] : (lane == i ? 1.0 : 0.0);
              double sdot = warp_sum(v * w);
              w = fma(-tau[LU ? 0 : i] * sdot, v, w);
            }
          }
        }
        if (act) {
          if (lane < n) xc[(size_t)j * n + lane] = w;
          else xc[(size_t)jp * n + lane - n] = w;
        }
        const double wt = lane < n ? (lu && op ? b : -w) : 0.0;
  #pragma unroll
        for (int r = 0; r < NRM; ++r) {
          if (r < nr) {
            const double sr = warp_sum(cp[r] * wt);
            if (lane == 0) a.XB[(size_t)j * nr * nrhs + (size_t)col * nr + r] = sr;
          }
        }
      }
    }
  });
}

template <typename TF, int N, int NXM, bool BATCH = false>
__global__ void __launch_bounds__(256, 2) k_backward_rows(SweepArgs<TF> a0, const SweepArgs<TF>* tab,
                                                          const BatchCta* cmap, const long* ecnt) {
  for_entries<BATCH>(ecnt, [&](long entry) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    SweepArgs<TF> ab;  // this CTA's system (batch only)
    long q0, q1, qs;
    pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs, entry);
    const SweepArgs<TF>& a = BATCH ? ab : a0;
    const Dims d = a.d;
    const int n = d.n, nx = d.nx, nb = d.nblock, n2 = 2 * n, nrhs = a.nrhs, k = a.k;
    const int i = lane & 15;
    const bool hi = lane >= 16, rowok = i < n;
    const bool qrp = a.sel == SEL_QRP;
    const size_t xb_off = (size_t)(nb + 1) * n + d.qx;
    for (long q = q0; q < q1; q += qs) {
      const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
      const TF* Mt = (hi ? a.E : a.D) + (size_t)j * n * n;
      const TF* Tj = a.Tm + (size_t)j * szT(d);
      const TF* Bj = a.B + (size_t)j * n * nx;
      double m[N], u[N], bb[NXM];
  #pragma unroll
      for (int c = 0; c < N; ++c) m[c] = (rowok && c < n) ? Mt[(size_t)c * n + i] : 0.0;
  #pragma unroll
      for (int c = 0; c < N; ++c) u[c] = (!hi && rowok && c < n) ? Tj[(size_t)c * n2 + i] : 0.0;
  #pragma unroll
      for (int c = 0; c < NXM; ++c) bb[c] = (!hi && rowok && c < nx) ? Bj[(size_t)c * n + i] : 0.0;
      // 1 / U(i,i): pick the diagonal element first, then one division per lane
      double ud = 1.0;
  #pragma unroll
      for (int c = 0; c < N; ++c)
        if (c == i) ud = u[c];
      const double rdi = (!hi && rowok) ? 1.0 / ud : 0.0;
      const int dst = (qrp && !hi && rowok) ? (int)a.P[(size_t)j * szP(d) + n2 + i] : i;
      for (int col = 0; col < nrhs; ++col) {
        double* xc = a.x + (size_t)col * a.ldx;
        const double xv = rowok ? (hi ? xc[(size_t)jpp * n + i] : xc[(size_t)jp * n + i]) : 0.0;
        const double xj = (!hi && rowok) ? xc[(size_t)j * n + i] : 0.0;
        double xbv[NXM];
  #pragma unroll
        for (int c = 0; c < NXM; ++c) xbv[c] = c < nx ? xc[xb_off + c] : 0.0;
        double s = 0.0;
  #pragma unroll
        for (int c = 0; c < N; ++c) {
          if (c < n) {
            const double xcv = __shfl_sync(FULL, xv, (lane & 16) | c);
            s = fma(m[c], xcv, s);
          }
        }
        s += __shfl_xor_sync(FULL, s, 16);
  #pragma unroll
        for (int c = 0; c < NXM; ++c) s = fma(bb[c], xbv[c], s);
        double y = xj - s;
  #pragma unroll
        for (int ii = N - 1; ii >= 0; --ii) {
          if (ii < n) {
            const double xi = __shfl_sync(FULL, y * rdi, ii);
            if (i == ii) y = xi;
            else if (i < ii) y = fma(-u[ii], xi, y);
          }
        }
        if (!hi && rowok) xc[(size_t)j * n + dst] = y;
      }
    }
  });
}

// ---------------------------------------------------------------------------
// Backward sweep for n = 8 or 16 (FP64 or FP32 factors; single systems and
// batch classes, see PipeItems): the same pair arithmetic as k_backward_rows (lane i < n: U-row i with D'_j, U and B'_j;
// lane 16 + i: E'_j row i), with the factors of the warp's NEXT pair copied
// into shared memory by cp.async (16-byte chunks, straight from the blocks'
// column-major layout, which is also the conflict-free layout for lane = row)
// while the current pair is computed, so every warp keeps a pair's worth of
// loads in flight.  Two buffers per warp.
// ---------------------------------------------------------------------------
template <int N, int NXM, typename T = double>
struct BwdBuf {
  static constexpr int DE = N * N, BB = N * NXM, U = N * N;
  static constexpr int WORDS = 2 * DE + BB + U;  // D', E', B', U (rows 0..N-1 of T)
  static constexpr size_t BYTES = (size_t)2 * WORDS * sizeof(T);  // two buffers
};

// the factors of pair q (level stride k) into one buffer (every lane issues
// its share), in 16-byte chunks of V elements; for n = 8, 16 every block (D',
// E', B', the U columns of T) starts and ends on a 16-byte boundary in FP64
// and FP32
template <int N, int NXM, typename T>
__device__ __forceinline__ void bwd_stage(const SweepArgs<T>& a, int k, long q, T* buf, int lane) {
  using Bf = BwdBuf<N, NXM, T>;
  constexpr int V = 16 / (int)sizeof(T);
  const Dims d = a.d;
  constexpr int n = N;
  const int nx = d.nx;
  const int j = k + (int)(2L * k * q);
  const T* Dj = a.D + (size_t)j * n * n;
  const T* Ej = a.E + (size_t)j * n * n;
  const T* Bj = a.B + (size_t)j * n * nx;
  const T* Tj = a.Tm + (size_t)j * szT(d);
  // D', E': n*n elements each
  for (int c = lane; c < n * n / V; c += 32) {
    cp_async16(buf + V * c, Dj + V * c);
    cp_async16(buf + Bf::DE + V * c, Ej + V * c);
  }
  for (int c = lane; c < n * nx / V; c += 32) cp_async16(buf + 2 * Bf::DE + V * c, Bj + V * c);
  // U: column col of T holds rows 0..n-1 of U at Tj + col * 2n
  for (int c = lane; c < n * n / V; c += 32) {
    const int col = (V * c) / n, r = (V * c) % n;
    cp_async16(buf + 2 * Bf::DE + Bf::BB + col * n + r, Tj + (size_t)col * 2 * n + r);
  }
}

// Work items of a warp in the pipelined sweeps.  Single system: pair q =
// item, items first, first + step, ... below the level's pair count.  Batch:
// item = entry of the level's sweep map (the full map: nent entries; or the
// compacted map of the systems still refining: *ecnt entries), the warp's
// pair is entry.q0 + warp, and the system's arguments come from the table.
template <bool BATCH, typename T>
struct PipeItems {
  SweepArgs<T> a0;
  const SweepArgs<T>* tab;
  const BatchCta* map;
  long cnt, first, step;
  int warp;
  __device__ PipeItems(const SweepArgs<T>& a, const SweepArgs<T>* t, const BatchCta* m, const long* ecnt,
                       long nent, int wpb, int w)
      : a0(a), tab(t), map(m), warp(w) {
    if constexpr (BATCH) {
      cnt = ecnt ? *ecnt : nent;
      first = blockIdx.x;
      step = gridDim.x;
    } else {
      cnt = pairs_at_level(a.d.nblock, a.k);
      first = (long)blockIdx.x * wpb + w;
      step = (long)gridDim.x * wpb;
    }
  }
  // the warp's pair of item it (false: none for this warp)
  __device__ bool pair(long it, int& sys, long& q) const {
    if constexpr (BATCH) {
      const BatchCta c = map[it];
      sys = c.sys;
      q = c.q0 + warp;
      if (q >= c.q1) return false;
      const int* dn = tab[sys].done;
      return !(dn && *dn);
    } else {
      sys = 0;
      q = it;
      return true;
    }
  }
  __device__ const SweepArgs<T>& args(int sys) const {
    if constexpr (BATCH) return tab[sys];
    else return a0;
  }
};

// Eight right-hand sides of one pair of the backward sweep (FP64): the products
// D' X_jp, E' X_jpp and B' X_b on the tensor cores, then the triangle with four
// columns per half warp.  buf: the pair's staged factors (overwritten).  COH: x
// may have been written earlier in this launch.
//
// One column at a time, 50 shuffles and as many multiply-adds repeat for every
// column, and the triangle's chain of N shuffles is walked once per column: 8
// right-hand sides of 30,000 blocks of order 16 took 128 us at level 1, and take
// 47 us here; the factor's 16.6 MB pass is 3 us of that.  Taken from two
// right-hand sides on, where it already is the faster one (the whole solve of
// that size: 389 to 318 us for 2, 487 to 323 us for 3, 780 to 490 us with the
// factorization for 8); a single one stays with the scalar code, which does an
// eighth of the work.
template <int N, int NXM, bool COH>
__device__ __forceinline__ void bwd_multi(const SweepArgs<double>& a, int j, int jp, int jpp, double* buf, int lane) {
  using Bf = BwdBuf<N, NXM, double>;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int MT = N / 8, KS = N / 4;
  const Dims d = a.d;
  const int nx = d.nx, nrhs = a.nrhs, g = lane >> 2, q = lane & 3, i = lane & 15, hb = lane >> 4;
  const size_t xb_off = (size_t)(d.nblock + 1) * N + d.qx;
  const bool rowok = i < N;
  double u[N];
#pragma unroll
  for (int c = 0; c < N; ++c) u[c] = rowok ? buf[2 * Bf::DE + Bf::BB + c * N + i] : 0.0;
  double ud = 1.0;
#pragma unroll
  for (int c = 0; c < N; ++c)
    if (c == i) ud = u[c];
  const double rdi = rowok ? 1.0 / ud : 0.0;
  const int dst = a.sel == SEL_QRP && rowok ? (int)a.P[(size_t)j * szP(d) + 2 * N + i] : i;
  // -[D' E' B'] as A fragments, kept for all chunks of columns
  double fd[MT][KS], fe[MT][KS], fb[MT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      fd[mt][ks] = -buf[(4 * ks + q) * N + 8 * mt + g];
      fe[mt][ks] = -buf[Bf::DE + (4 * ks + q) * N + 8 * mt + g];
    }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      const int c = 4 * ks + q;
      fb[mt][ks] = c < nx ? -buf[2 * Bf::DE + (c < NXM ? c : 0) * N + 8 * mt + g] : 0.0;
    }
  }
  for (int c0 = 0; c0 < nrhs; c0 += 8) {
    const int nc = min(8, nrhs - c0);
    double* xc = a.x + (size_t)c0 * a.ldx;
    double bd[KS], be[KS], bb[2], acc[MT][2];
    const double* xg = xc + (size_t)min(g, nc - 1) * a.ldx;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      bd[ks] = ld_batch_c<COH>(g < nc, xg + (size_t)jp * N + 4 * ks + q);
      be[ks] = ld_batch_c<COH>(g < nc, xg + (size_t)jpp * N + 4 * ks + q);
    }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) bb[ks] = ld_batch_c<COH>(g < nc && 4 * ks + q < nx, xg + xb_off + 4 * ks + q);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        acc[mt][h] = ld_batch_c<COH>(2 * q + h < nc, xc + (size_t)min(2 * q + h, nc - 1) * a.ldx + (size_t)j * N + 8 * mt + g);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        dmma_8x8x4(acc[mt][0], acc[mt][1], fd[mt][ks], bd[ks]);
        dmma_8x8x4(acc[mt][0], acc[mt][1], fe[mt][ks], be[ks]);
      }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) dmma_8x8x4(acc[mt][0], acc[mt][1], fb[mt][ks], bb[ks]);
    // to lane = row through the buffer's first block
    __syncwarp();
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) buf[(2 * q + h) * N + 8 * mt + g] = acc[mt][h];
    __syncwarp();
    double y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = rowok ? buf[(4 * hb + e) * N + i] : 0.0;
#pragma unroll
    for (int ii = N - 1; ii >= 0; --ii) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double xi = __shfl_sync(FULL, y[e] * rdi, (lane & 16) | ii);
        y[e] = i == ii ? xi : i < ii ? fma(-u[ii], xi, y[e]) : y[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (rowok && 4 * hb + e < nc) xc[(size_t)(4 * hb + e) * a.ldx + (size_t)j * N + dst] = y[e];
  }
}

template <int N, int NXM, typename T = double, bool BATCH = false>
__global__ void __launch_bounds__(256, 2) k_backward_pipe(SweepArgs<T> a0, const SweepArgs<T>* tab,
                                                          const BatchCta* map, const long* ecnt, long nent) {
  using Bf = BwdBuf<N, NXM, T>;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  T* bufs = reinterpret_cast<T*>(smem_raw) + (size_t)warp * 2 * Bf::WORDS;
  const PipeItems<BATCH, T> items(a0, tab, map, ecnt, nent, wpb, warp);
  const int k = a0.k;
  const int i = lane & 15;
  long it = items.first;
  int sys = 0;
  long q = 0;
  bool have = it < items.cnt && items.pair(it, sys, q);
  if (have) bwd_stage<N, NXM, T>(items.args(sys), k, q, bufs, lane);
  cp_async_commit();
  int cur = 0;
  for (; it < items.cnt; it += items.step) {
    int sysn = 0;
    long qn = 0;
    const bool haven = it + items.step < items.cnt && items.pair(it + items.step, sysn, qn);
    if (haven) bwd_stage<N, NXM, T>(items.args(sysn), k, qn, bufs + (cur ^ 1) * Bf::WORDS, lane);
    cp_async_commit();
    if (have) {
      const SweepArgs<T>& a = items.args(sys);
      const Dims d = a.d;
      constexpr int n = N;
      const int nx = d.nx, nb = d.nblock, nrhs = a.nrhs;
      const bool hi = lane >= 16, rowok = i < n;
      const bool qrp = a.sel == SEL_QRP;
      const size_t xb_off = (size_t)(nb + 1) * n + d.qx;
      const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
      // the right-hand side values, loaded while the factors arrive
      double xv0 = 0.0, xj0 = 0.0;
      if (nrhs >= 1) {
        xv0 = rowok ? (hi ? a.x[(size_t)jpp * n + i] : a.x[(size_t)jp * n + i]) : 0.0;
        xj0 = (!hi && rowok) ? a.x[(size_t)j * n + i] : 0.0;
      }
      const int dst = (qrp && !hi && rowok) ? (int)a.P[(size_t)j * szP(d) + 2 * n + i] : i;
      cp_async_wait<1>();  // this pair's factors (the next pair's may still be in flight)
      __syncwarp();
      T* buf = bufs + cur * Bf::WORDS;
      const bool multi = sizeof(T) == 8 && nrhs > 1;
      if constexpr (sizeof(T) == 8) {
        if (multi) bwd_multi<N, NXM, false>(a, j, jp, jpp, buf, lane);
      }
      if (!multi) {
        double m[N], u[N], bb[NXM];
#pragma unroll
        for (int c = 0; c < N; ++c) m[c] = (rowok && c < n) ? buf[(hi ? Bf::DE : 0) + c * n + i] : 0.0;
#pragma unroll
        for (int c = 0; c < N; ++c) u[c] = (!hi && rowok && c < n) ? buf[2 * Bf::DE + Bf::BB + c * n + i] : 0.0;
#pragma unroll
        for (int c = 0; c < NXM; ++c) bb[c] = (!hi && rowok && c < nx) ? buf[2 * Bf::DE + c * n + i] : 0.0;
        double ud = 1.0;
#pragma unroll
        for (int c = 0; c < N; ++c)
          if (c == i) ud = u[c];
        const double rdi = (!hi && rowok) ? 1.0 / ud : 0.0;
        for (int col = 0; col < nrhs; ++col) {
          double* xc = a.x + (size_t)col * a.ldx;
          const double xv = col == 0 ? xv0 : (rowok ? (hi ? xc[(size_t)jpp * n + i] : xc[(size_t)jp * n + i]) : 0.0);
          const double xj = col == 0 ? xj0 : ((!hi && rowok) ? xc[(size_t)j * n + i] : 0.0);
          double xbv[NXM];
#pragma unroll
          for (int c = 0; c < NXM; ++c) xbv[c] = c < nx ? xc[xb_off + c] : 0.0;
          double sacc = 0.0;
#pragma unroll
          for (int c = 0; c < N; ++c) {
            if (c < n) {
              const double xcv = __shfl_sync(FULL, xv, (lane & 16) | c);
              sacc = fma(m[c], xcv, sacc);
            }
          }
          sacc += __shfl_xor_sync(FULL, sacc, 16);
#pragma unroll
          for (int c = 0; c < NXM; ++c) sacc = fma(bb[c], xbv[c], sacc);
          double y = xj - sacc;
#pragma unroll
          for (int ii = N - 1; ii >= 0; --ii) {
            if (ii < n) {
              const double xi = __shfl_sync(FULL, y * rdi, ii);
              if (i == ii) y = xi;
              else if (i < ii) y = fma(-u[ii], xi, y);
            }
          }
          if (!hi && rowok) xc[(size_t)j * n + dst] = y;
        }
      }
    }
    __syncwarp();  // every lane is done with this buffer before it is refilled
    cur ^= 1;
    have = haven;
    sys = sysn;
    q = qn;
  }
  cp_async_wait<0>();
}

// The top levels of the backward sweep (at most 16 pairs each) in one launch
// of one CTA of 16 warps, levels in order with a barrier between them; the
// pair arithmetic is k_backward_rows'.
template <int N, int NXM, typename T = double>
__global__ void __launch_bounds__(512, 1) k_backward_top(SweepArgs<T> a, int k_top, int k_min) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Dims d = a.d;
  const int n = d.n, nx = d.nx, nb = d.nblock, nrhs = a.nrhs;
  const int i = lane & 15;
  const bool hi = lane >= 16, rowok = i < n;
  const bool qrp = a.sel == SEL_QRP;
  const size_t xb_off = (size_t)(nb + 1) * n + d.qx;
  if constexpr (sizeof(T) == 8) {
    if (nrhs > 1) {  // eight right-hand sides at once (the launch brings BwdBuf::WORDS per warp)
      extern __shared__ __align__(16) unsigned char smem_raw[];
      T* buf = reinterpret_cast<T*>(smem_raw) + (size_t)warp * BwdBuf<N, NXM, T>::WORDS;
      for (int k = k_top; k >= k_min && k > 0; k /= 2) {
        const long np = pairs_at_level(nb, k);
        for (long q = warp; q < np; q += 16) {
          const int j = k + (int)(2L * k * q);
          bwd_stage<N, NXM, T>(a, k, q, buf, lane);
          cp_async_commit();
          cp_async_wait<0>();
          __syncwarp();
          bwd_multi<N, NXM, true>(a, j, j - k, min(j + k, nb), buf, lane);
          __syncwarp();
        }
        __syncthreads();
      }
      return;
    }
  }
  for (int k = k_top; k >= k_min && k > 0; k /= 2) {
    const long np = pairs_at_level(nb, k);
    for (long q = warp; q < np; q += 16) {
      const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
      const T* Mt = (hi ? a.E : a.D) + (size_t)j * n * n;
      const T* Tj = a.Tm + (size_t)j * szT(d);
      const T* Bj = a.B + (size_t)j * n * nx;
      double m[N], u[N], bb[NXM];
#pragma unroll
      for (int c = 0; c < N; ++c) m[c] = (rowok && c < n) ? Mt[(size_t)c * n + i] : 0.0;
#pragma unroll
      for (int c = 0; c < N; ++c) u[c] = (!hi && rowok && c < n) ? Tj[(size_t)c * 2 * n + i] : 0.0;
#pragma unroll
      for (int c = 0; c < NXM; ++c) bb[c] = (!hi && rowok && c < nx) ? Bj[(size_t)c * n + i] : 0.0;
      double ud = 1.0;
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (c == i) ud = u[c];
      const double rdi = (!hi && rowok) ? 1.0 / ud : 0.0;
      const int dst = (qrp && !hi && rowok) ? (int)a.P[(size_t)j * szP(d) + 2 * n + i] : i;
      for (int col = 0; col < nrhs; ++col) {
        double* xc = a.x + (size_t)col * a.ldx;
        const double xv = rowok ? (hi ? __ldcg(xc + (size_t)jpp * n + i) : __ldcg(xc + (size_t)jp * n + i)) : 0.0;
        const double xj = (!hi && rowok) ? xc[(size_t)j * n + i] : 0.0;
        double xbv[NXM];
#pragma unroll
        for (int c = 0; c < NXM; ++c) xbv[c] = c < nx ? __ldcg(xc + xb_off + c) : 0.0;
        double sacc = 0.0;
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (c < n) {
            const double xcv = __shfl_sync(FULL, xv, (lane & 16) | c);
            sacc = fma(m[c], xcv, sacc);
          }
        }
        sacc += __shfl_xor_sync(FULL, sacc, 16);
#pragma unroll
        for (int c = 0; c < NXM; ++c) sacc = fma(bb[c], xbv[c], sacc);
        double y = xj - sacc;
#pragma unroll
        for (int ii = N - 1; ii >= 0; --ii) {
          if (ii < n) {
            const double xi = __shfl_sync(FULL, y * rdi, ii);
            if (i == ii) y = xi;
            else if (i < ii) y = fma(-u[ii], xi, y);
          }
        }
        if (!hi && rowok) xc[(size_t)j * n + dst] = y;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Forward sweep for LU factors, n = 8 or 16 (FP64 or FP32; single systems and
// batch classes, see PipeItems): the pair arithmetic of k_forward_rows (lane = position r < 2n of the stacked
// [x_jp; x_j], row map gathered by one shuffle, n broadcast steps of L and M,
// xb partial -C'_j x_j; with the operator form, one matrix-vector product
// whose terms do not depend on each other), with the factors of the warp's NEXT pair (the 2n x n
// L\U and M block of T, and C_j) copied into shared memory by cp.async while
// the current pair is computed, and the next pair's row-map entry read into a
// register one pair ahead.  Two buffers per warp.
// ---------------------------------------------------------------------------
template <int N, int NRM, typename T = double>
struct FwdBuf {
  static constexpr int TT = 2 * N * N, CC = N * NRM;
  static constexpr int WORDS = TT + CC;                        // T_j (2n x n), C_j (n x nr)
  static constexpr size_t BYTES = (size_t)2 * WORDS * sizeof(T);  // two buffers
};

// the factors of pair q (level stride k) into one buffer, in 16-byte chunks
// of V elements (for n = 8, 16 both blocks are multiples of 16 bytes in FP64
// and FP32)
template <int N, int NRM, typename T>
__device__ __forceinline__ void fwd_stage(const SweepArgs<T>& a, int k, long q, T* buf, int lane) {
  using Bf = FwdBuf<N, NRM, T>;
  constexpr int V = 16 / (int)sizeof(T);
  const Dims d = a.d;
  constexpr int n = N;
  const int nr = d.nr;
  const int j = k + (int)(2L * k * q);
  const T* Tj = a.Tm + (size_t)j * szT(d);
  const T* Cj = a.C + (size_t)j * nr * n;
  for (int c = lane; c < 2 * n * n / V; c += 32) cp_async16(buf + V * c, Tj + V * c);
  for (int c = lane; c < n * nr / V; c += 32) cp_async16(buf + Bf::TT + V * c, Cj + V * c);
}

// Eight right-hand sides of one pair of the forward sweep (FP64, operator form):
// one product [L^-1; -M L^-1; -C' L^-1] X on the tensor cores (see bwd_multi).
// src: the original row at position `lane`; buf: the pair's staged T_j and C_j.
template <int N, int NRM>
__device__ __forceinline__ void fwd_multi(const SweepArgs<double>& a, int j, int jp, int src, const double* buf,
                                          int lane) {
  using Bf = FwdBuf<N, NRM, double>;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int MT = 2 * N / 8, KS = N / 4;
  const Dims d = a.d;
  const int nr = d.nr, nrhs = a.nrhs, g = lane >> 2, q = lane & 3;
  double f[MT + 1][KS];
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    const int c = 4 * ks + q;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const double v = buf[c * 2 * N + 8 * mt + g];
      f[mt][ks] = 8 * mt + g > c ? v : 0.0;  // strictly below the diagonal; the rest of row k is U
    }
    f[MT][ks] = g < nr ? buf[Bf::TT + c * nr + (g < nr ? g : 0)] : 0.0;
  }
  // the vector element at this lane's rows
  auto at = [&](int r, int c) { return a.x + (size_t)c * a.ldx + (r < N ? (size_t)jp * N + r : (size_t)j * N + r - N); };
  int rk[KS], rm[MT];
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) rk[ks] = __shfl_sync(FULL, src, 4 * ks + q);
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) rm[mt] = __shfl_sync(FULL, src, 8 * mt + g);
  for (int c0 = 0; c0 < nrhs; c0 += 8) {
    const int nc = min(8, nrhs - c0);
    double b[KS], acc[MT + 1][2];
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) b[ks] = ld_batch(g < nc, at(rk[ks], c0 + min(g, nc - 1)));
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) acc[mt][h] = ld_batch(2 * q + h < nc, at(rm[mt], c0 + min(2 * q + h, nc - 1)));
    acc[MT][0] = acc[MT][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
      for (int mt = 0; mt <= MT; ++mt) dmma_8x8x4(acc[mt][0], acc[mt][1], f[mt][ks], b[ks]);
    __syncwarp();  // every lane's reads are done
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (2 * q + h < nc) {
        const int c = c0 + 2 * q + h;
        double* xc = a.x + (size_t)c * a.ldx;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int r = 8 * mt + g;
          if (8 * mt < N) xc[(size_t)j * N + r] = acc[mt][h];
          else xc[(size_t)jp * N + r - N] = acc[mt][h];
        }
        if (g < nr) a.XB[(size_t)j * nr * nrhs + (size_t)c * nr + g] = acc[MT][h];
      }
  }
}

template <int N, int NRM, typename T = double, bool BATCH = false>
__global__ void __launch_bounds__(256, 2) k_forward_pipe(SweepArgs<T> a0, const SweepArgs<T>* tab,
                                                         const BatchCta* map, const long* ecnt, long nent) {
  using Bf = FwdBuf<N, NRM, T>;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  T* bufs = reinterpret_cast<T*>(smem_raw) + (size_t)warp * 2 * Bf::WORDS;
  const PipeItems<BATCH, T> items(a0, tab, map, ecnt, nent, wpb, warp);
  const int k = a0.k;
  const bool op = a0.op != 0;
  // the row-map entry of a pair (read a pair ahead, into a register)
  auto row_src = [&](const SweepArgs<T>& a, long q) -> int {
    const int j = k + (int)(2L * k * q);
    return lane < 2 * a.d.n ? (int)a.P[(size_t)j * szP(a.d) + lane] : lane;
  };
  long it = items.first;
  int sys = 0, src_next = lane;
  long q = 0;
  bool have = it < items.cnt && items.pair(it, sys, q);
  if (have) {
    fwd_stage<N, NRM, T>(items.args(sys), k, q, bufs, lane);
    src_next = row_src(items.args(sys), q);
  }
  cp_async_commit();
  int cur = 0;
  for (; it < items.cnt; it += items.step) {
    const int src = src_next;
    int sysn = 0;
    long qn = 0;
    const bool haven = it + items.step < items.cnt && items.pair(it + items.step, sysn, qn);
    if (haven) {
      fwd_stage<N, NRM, T>(items.args(sysn), k, qn, bufs + (cur ^ 1) * Bf::WORDS, lane);
      src_next = row_src(items.args(sysn), qn);
    }
    cp_async_commit();
    if (have) {
      const SweepArgs<T>& a = items.args(sys);
      const Dims d = a.d;
      constexpr int n = N, n2 = 2 * N;
      const int nr = d.nr, nrhs = a.nrhs;
      const bool act = lane < n2;
      const int j = k + (int)(2L * k * q), jp = j - k;
      // the first right-hand side's values, loaded while the factors arrive
      const double orig0 = act ? (lane < n ? a.x[(size_t)jp * n + lane] : a.x[(size_t)j * n + lane - n]) : 0.0;
      cp_async_wait<1>();  // this pair's factors (the next pair's may still be in flight)
      __syncwarp();
      const T* buf = bufs + cur * Bf::WORDS;
      const bool multi = sizeof(T) == 8 && op && nrhs > 1;
      if constexpr (sizeof(T) == 8) {
        if (multi) fwd_multi<N, NRM>(a, j, jp, src, buf, lane);
      }
      if (!multi) {
        double t[N], cp[NRM];
#pragma unroll
        for (int c = 0; c < N; ++c) t[c] = (act && (!op || lane > c)) ? double(buf[c * n2 + lane]) : 0.0;
#pragma unroll
        for (int r = 0; r < NRM; ++r) cp[r] = (lane < n && r < nr) ? double(buf[Bf::TT + lane * nr + r]) : 0.0;
        for (int col = 0; col < nrhs; ++col) {
          double* xc = a.x + (size_t)col * a.ldx;
          const double orig =
              col == 0 ? orig0 : (act ? (lane < n ? xc[(size_t)jp * n + lane] : xc[(size_t)j * n + lane - n]) : 0.0);
          const double b = __shfl_sync(FULL, orig, src);
          double w = b, w2 = 0.0;
          if (op) {  // one product with the operator: no serial chain
#pragma unroll
            for (int i = 0; i < N; i += 2) {
              w = fma(t[i], __shfl_sync(FULL, b, i), w);
              w2 = fma(t[i + 1], __shfl_sync(FULL, b, i + 1), w2);
            }
            w += w2;
          } else {
#pragma unroll
            for (int i = 0; i < N; ++i) {
              const double wi = __shfl_sync(FULL, w, i);
              if (lane > i && act) w = fma(-t[i], wi, w);
            }
          }
          if (act) {
            if (lane < n) xc[(size_t)j * n + lane] = w;
            else xc[(size_t)jp * n + lane - n] = w;
          }
          // operator form: -C' L^-1 times the permuted rows; else -C' times y
          const double wt = lane < n ? (op ? b : -w) : 0.0;
#pragma unroll
          for (int r = 0; r < NRM; ++r) {
            if (r < nr) {
              const double sr = warp_sum(cp[r] * wt);
              if (lane == 0) a.XB[(size_t)j * nr * nrhs + (size_t)col * nr + r] = sr;
            }
          }
        }
      }
    }
    __syncwarp();  // every lane is done with this buffer before it is refilled
    cur ^= 1;
    have = haven;
    sys = sysn;
    q = qn;
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// sweeps for n = 32: one warp per pair, lane i holds panel positions i and
// 32 + i (forward) or U-row i (backward); x values are exchanged by shuffles
// and every factor element is read once, coalesced
// ---------------------------------------------------------------------------
// Factors in operator form (k_factor_lu_grp): one product with the permuted rows,
// 16 columns of both rows read in one batch, up to four right-hand sides on each.
template <typename TF, int NRM, bool BATCH = false>
__global__ void __launch_bounds__(256, 2) k_forward_rows32(SweepArgs<TF> a0, const SweepArgs<TF>* tab,
                                                           const BatchCta* cmap, const long* ecnt) {
  for_entries<BATCH>(ecnt, [&](long entry) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int n = 32, n2 = 64, RH = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    SweepArgs<TF> ab;  // this CTA's system (batch only)
    long q0, q1, qs;
    pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs, entry);
    const SweepArgs<TF>& a = BATCH ? ab : a0;
    const Dims d = a.d;
    const int nr = d.nr, nrhs = a.nrhs, k = a.k;
    for (long q = q0; q < q1; q += qs) {
      const int j = k + (int)(2L * k * q), jp = j - k;
      const TF* Tj = a.Tm + (size_t)j * szT(d);
      const unsigned char* Pj = a.P + (size_t)j * szP(d);
      const int s0 = Pj[lane], s1 = Pj[n + lane];  // original rows at positions lane, 32 + lane
      const TF* Cj = a.C + (size_t)j * nr * n;
      for (int col0 = 0; col0 < nrhs; col0 += RH) {
        const int nc = min(RH, nrhs - col0);
        double* xc = a.x + (size_t)col0 * a.ldx;
        double b[RH], w0[RH], w1[RH];
        TF t0[16], t1[16], cp[NRM];
        auto load = [&](int c0) {
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            t0[u] = ld_batch(lane > c0 + u, Tj + (size_t)(c0 + u) * n2 + lane);
            t1[u] = ld_batch(true, Tj + (size_t)(c0 + u) * n2 + n + lane);
          }
        };
        load(0);
#pragma unroll
        for (int r = 0; r < NRM; ++r) cp[r] = ld_batch(r < nr, Cj + (size_t)lane * nr + r);
        double ot[RH], ob[RH];
#pragma unroll
        for (int c = 0; c < RH; ++c) {
          ot[c] = ld_batch(c < nc, xc + (size_t)c * a.ldx + (size_t)jp * n + lane);
          ob[c] = ld_batch(c < nc, xc + (size_t)c * a.ldx + (size_t)j * n + lane);
        }
#pragma unroll
        for (int c = 0; c < RH; ++c)
          if (c < nc) {
            const double a0t = __shfl_sync(FULL, ot[c], s0 & 31), a0b = __shfl_sync(FULL, ob[c], s0 & 31);
            const double a1t = __shfl_sync(FULL, ot[c], s1 & 31), a1b = __shfl_sync(FULL, ob[c], s1 & 31);
            w0[c] = b[c] = s0 < n ? a0t : a0b;
            w1[c] = s1 < n ? a1t : a1b;
          }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int c = 0; c < RH; ++c)
            if (c < nc) {
#pragma unroll
              for (int u = 0; u < 16; ++u) {
                const double bi = __shfl_sync(FULL, b[c], 16 * h + u);
                w0[c] = fma(double(t0[u]), bi, w0[c]);
                w1[c] = fma(double(t1[u]), bi, w1[c]);
              }
            }
          if (h == 0) load(16);
        }
#pragma unroll
        for (int c = 0; c < RH; ++c)
          if (c < nc) {
            xc[(size_t)c * a.ldx + (size_t)j * n + lane] = w0[c];
            xc[(size_t)c * a.ldx + (size_t)jp * n + lane] = w1[c];
#pragma unroll
            for (int r = 0; r < NRM; ++r) {
              if (r < nr) {
                const double sr = warp_sum(double(cp[r]) * b[c]);
                if (lane == 0) a.XB[(size_t)j * nr * nrhs + (size_t)(col0 + c) * nr + r] = sr;
              }
            }
          }
      }
    }
  });
}

template <typename TF, int NXM, bool BATCH = false>
__global__ void __launch_bounds__(256, 2) k_backward_rows32(SweepArgs<TF> a0, const SweepArgs<TF>* tab,
                                                            const BatchCta* cmap, const long* ecnt) {
  for_entries<BATCH>(ecnt, [&](long entry) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int n = 32, n2 = 64, RH = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    SweepArgs<TF> ab;  // this CTA's system (batch only)
    long q0, q1, qs;
    pair_range<BATCH>(a0, tab, cmap, wpb, warp, ab, q0, q1, qs, entry);
    const SweepArgs<TF>& a = BATCH ? ab : a0;
    const Dims d = a.d;
    const int nx = d.nx, nb = d.nblock, nrhs = a.nrhs, k = a.k;
    const bool qrp = a.sel == SEL_QRP;
    const size_t xb_off = (size_t)(nb + 1) * n + d.qx;
    for (long q = q0; q < q1; q += qs) {
      const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
      const TF* Dj = a.D + (size_t)j * n * n;
      const TF* Ej = a.E + (size_t)j * n * n;
      const TF* Bj = a.B + (size_t)j * n * nx;
      const TF* Tj = a.Tm + (size_t)j * szT(d);
      const int dst = qrp ? (int)a.P[(size_t)j * szP(d) + n2 + lane] : lane;
      for (int col0 = 0; col0 < nrhs; col0 += RH) {
        const int nc = min(RH, nrhs - col0);
        double* xc = a.x + (size_t)col0 * a.ldx;
        TF m[32];
        auto load = [&](const TF* M, int ld, int from) {  // columns from `from` on
#pragma unroll
          for (int c = 0; c < 32; ++c) m[c] = ld_batch(c >= from, M + (size_t)c * ld + lane);
        };
        load(Dj, n, 0);
        TF bb[NXM];
#pragma unroll
        for (int c = 0; c < NXM; ++c) bb[c] = ld_batch(c < nx, Bj + (size_t)c * n + lane);
        double xa[RH], xz[RH], y[RH];
#pragma unroll
        for (int c = 0; c < RH; ++c) {
          xa[c] = ld_batch(c < nc, xc + (size_t)c * a.ldx + (size_t)jp * n + lane);
          xz[c] = ld_batch(c < nc, xc + (size_t)c * a.ldx + (size_t)jpp * n + lane);
          y[c] = ld_batch(c < nc, xc + (size_t)c * a.ldx + (size_t)j * n + lane);
        }
        auto subtract = [&](const double (&x)[RH]) {  // y -= M x
#pragma unroll
          for (int c = 0; c < RH; ++c)
            if (c < nc) {
              double s0 = 0.0, s1 = 0.0;
#pragma unroll
              for (int u = 0; u < 32; u += 2) {
                s0 = fma(double(m[u]), __shfl_sync(FULL, x[c], u), s0);
                s1 = fma(double(m[u + 1]), __shfl_sync(FULL, x[c], u + 1), s1);
              }
              y[c] -= s0 + s1;
            }
        };
        subtract(xa);
        load(Ej, n, 0);
#pragma unroll
        for (int c = 0; c < RH; ++c)
          if (c < nc) {
            double s = 0.0;
#pragma unroll
            for (int e = 0; e < NXM; ++e) s = fma(double(bb[e]), e < nx ? xc[(size_t)c * a.ldx + xb_off + e] : 0.0, s);
            y[c] -= s;
          }
        subtract(xz);
        load(Tj, n2, lane);  // U, on and right of the diagonal
        double ud = 1.0;
#pragma unroll
        for (int c = 0; c < 32; ++c)
          if (c == lane) ud = double(m[c]);
        const double rdi = 1.0 / ud;
#pragma unroll
        for (int c = 0; c < RH; ++c)
          if (c < nc) {
            double v = y[c];
#pragma unroll
            for (int u = 31; u >= 0; --u) {
              const double xi = __shfl_sync(FULL, v * rdi, u);
              v = lane == u ? xi : fma(-double(m[u]), lane < u ? xi : 0.0, v);
            }
            xc[(size_t)c * a.ldx + (size_t)j * n + dst] = v;
          }
      }
    }
  });
}

#include "bcr_sweep_big.cuh"

// ---------------------------------------------------------------------------
// last block (load_and_factorize_last, cc:1281-1374; solve_last, cc:1385-1479)
// one CTA; the Nr x Nc matrix lives in global memory (L2 resident)
// ---------------------------------------------------------------------------
template <typename T>
__device__ void last_assemble_range(Dims d, const T* D, const T* E, const T* B, const T* C,
                                    const double* H, const double* Cq, const double* Ffin, double* Hl,
                                    int e0, int es) {
  const int n = d.n, Nr = d.Nr, Nc = d.Nc, qx = d.qx, nr = d.nr, m = n + d.qr;
  const int total = Nr * Nc;
  const T* CN = C + (size_t)d.nblock * nr * n;
  for (int e = e0; e < total; e += es) {
    const int r = e % Nr, c = e / Nr;
    double v = 0.0;
    if (r < n) {
      if (c < n) v = D[(size_t)c * n + r];
      else if (c < 2 * n) v = E[(size_t)(c - n) * n + r];
      else if (c >= 2 * n + qx) v = B[(size_t)(c - 2 * n - qx) * n + r];
    } else if (r < n + m) {
      v = H[(size_t)c * m + (r - n)];
    } else {
      const int rr = r - n - m;
      if (c < n) v = C[(size_t)c * nr + rr];
      else if (c < 2 * n) v = CN[(size_t)(c - n) * nr + rr];
      else if (c < 2 * n + qx) v = Cq[(size_t)(c - 2 * n) * nr + rr];
      else v = Ffin[(size_t)(c - 2 * n - qx) * nr + rr];
    }
    Hl[e] = v;
  }
}

template <typename T>
__global__ void k_last_assemble(Dims d, const T* D, const T* E, const T* B, const T* C,
                                const double* H, const double* Cq, const double* Ffin, double* Hl) {
  last_assemble_range(d, D, E, B, C, H, Cq, Ffin, Hl, blockIdx.x * blockDim.x + threadIdx.x,
                      gridDim.x * blockDim.x);
}

template <typename T>
__device__ void block_argmax(T& v, int& idx, T* sv, int* si) {
  warp_argmax(v, idx);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) { sv[w] = v; si[w] = idx; }
  __syncthreads();
  if (w == 0) {
    v = lane < nw ? sv[lane] : T(-1);
    idx = lane < nw ? si[lane] : 0x7fffffff;
    warp_argmax(v, idx);
    if (lane == 0) { sv[0] = v; si[0] = idx; }
  }
  __syncthreads();
  v = sv[0];
  idx = si[0];
}

template <typename T>
__device__ T block_sum(T v, T* sv) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) sv[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < nw ? sv[lane] : T(0);
    v = warp_sum(v);
    if (lane == 0) sv[0] = v;
  }
  __syncthreads();
  return sv[0];
}

// buffers of the last block (one CTA works on them)
struct LastBufs {
  double* A;    // Nr x Nc (ld Nr): the assembled block, then its factors
  double* A2;   // copy for the fallback solver (null when there is none)
  int* piv;     // row pivots [0, L), column pivots [L, 2L), L = max(Nr, Nc)
  double* tau;  // Householder scalars
  double* U;    // SVD: W = U*S, max(Nr,Nc) x min(Nr,Nc)
  double* V;    // SVD: min x min
  double* S;    // SVD: singular values
};

__device__ inline int last_kind_of(int sel_last, int M, int N) {
  switch (sel_last) {
    case LAST_LU: return FACT_LU;
    case LAST_LUPQ: return FACT_LUPQ;
    case LAST_QR: return FACT_QR;
    case LAST_QRP: return FACT_QRP;
    default: return M >= N ? FACT_SVD : FACT_SVD_T;  // SVD, LSS, LSY, PINV
  }
}

// Minimum-norm least-squares factorization of the SVD family (the solvers
// SVD, LSS, LSY and PINV of the reference's LapackWrapper): one-sided Jacobi
// on W = A (or A^T when Nr < Nc), rotations of a pair of columns p < q by the
// angle that makes them orthogonal, skipped when |g| <= 1e-15 sqrt(a b); the
// pairs of a sweep follow the round-robin (circle) schedule, so the Np/2 pairs
// of a round are independent and run one per warp; at most 80 sweeps, ending
// at the first sweep without a rotation.  On return W = U*S is split into
// unit columns U and S.
__device__ void last_svd(Dims d, const double* A, LastBufs b, StatusWords* st) {
  __shared__ int rotated;
  const int M = d.Nr, N = d.Nc, tid = threadIdx.x, bs = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = bs >> 5;
  const bool tr = M < N;
  const int Mp = tr ? N : M, Np = tr ? M : N;
  double* W = b.U;
  double* V = b.V;
  for (int e = tid; e < Mp * Np; e += bs) {
    const int i = e % Mp, j = e / Mp;
    W[(size_t)j * Mp + i] = tr ? A[(size_t)i * M + j] : A[(size_t)j * M + i];
  }
  for (int e = tid; e < Np * Np; e += bs) V[e] = (e % Np == e / Np) ? 1.0 : 0.0;
  __syncthreads();
  const int P = Np + (Np & 1);
  for (int sweep = 0; sweep < 80; ++sweep) {
    if (tid == 0) rotated = 0;
    __syncthreads();
    for (int r = 0; r < P - 1; ++r) {
      for (int k = warp; k < P / 2; k += nw) {
        int p0, q0;
        if (k == 0) { p0 = P - 1; q0 = r; }
        else { p0 = (r + k) % (P - 1); q0 = (r - k + P - 1) % (P - 1); }
        const int p = min(p0, q0), q = max(p0, q0);
        if (q >= Np) continue;
        double* wp = W + (size_t)p * Mp;
        double* wq = W + (size_t)q * Mp;
        double a = 0.0, bb = 0.0, g = 0.0;
        for (int i = lane; i < Mp; i += 32) {
          const double x = wp[i], y = wq[i];
          a = fma(x, x, a);
          bb = fma(y, y, bb);
          g = fma(x, y, g);
        }
        a = warp_sum(a);
        bb = warp_sum(bb);
        g = warp_sum(g);
        if (fabs(g) <= 1e-15 * sqrt(a * bb) || g == 0.0) continue;
        const double zeta = (bb - a) / (2.0 * g);
        const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
        for (int i = lane; i < Mp; i += 32) {
          const double x = wp[i], y = wq[i];
          wp[i] = c * x - s * y;
          wq[i] = s * x + c * y;
        }
        double* vp = V + (size_t)p * Np;
        double* vq = V + (size_t)q * Np;
        for (int i = lane; i < Np; i += 32) {
          const double x = vp[i], y = vq[i];
          vp[i] = c * x - s * y;
          vq[i] = s * x + c * y;
        }
        if (lane == 0) rotated = 1;
      }
      __syncthreads();
    }
    const int any = rotated;
    __syncthreads();
    if (!any) break;
  }
  for (int j = warp; j < Np; j += nw) {
    double* wj = W + (size_t)j * Mp;
    double s2 = 0.0;
    for (int i = lane; i < Mp; i += 32) s2 = fma(wj[i], wj[i], s2);
    const double sj = sqrt(warp_sum(s2));
    if (lane == 0) b.S[j] = sj;
    if (sj > 0.0)
      for (int i = lane; i < Mp; i += 32) wj[i] /= sj;
  }
  if (tid == 0) st->kind = tr ? FACT_SVD_T : FACT_SVD;
  __syncthreads();
}

// load_and_factorize_last (cc:1281-1374) with the reference's last-block
// solvers: LU (getrf), LUPQ (complete pivoting), QR (geqrf), QRP (geqp3: the
// column of largest remaining 2-norm first), and the SVD family
// Last blocks of order <= LAST_SMALL (configs with n <= 16 and small borders):
// the LU of a batch's systems runs out of shared memory (the general loop below
// works in global memory, a round trip per column; single systems take
// k_last_lu_blocked), and the solves give every right-hand side a warp, its
// values in registers.  Same pivot rule (largest |a|, first row on ties, NaN
// never chosen), same operation order.
constexpr int LAST_SMALL = 64;

template <typename T>
__device__ void last_lu_small(Dims d, LastBufs b, StatusWords* st) {
  __shared__ T As[LAST_SMALL * (LAST_SMALL + 1)];
  __shared__ T s_pv;
  __shared__ int s_p;
  const int N = d.Nc, ld = N + 1, tid = threadIdx.x, bs = blockDim.x;
  T* A = b.A;
  for (int c = tid / 32; c < N; c += bs / 32)  // one column per warp: coalesced, all loads in flight
    for (int r = tid & 31; r < N; r += 32) As[c * ld + r] = A[(size_t)c * N + r];
  __syncthreads();
  for (int i = 0; i < N; ++i) {
    if (tid < 32) {  // pivot of column i: largest |a| over rows >= i, first row on ties, NaN never
      T best = T(-2);
      int bi = 0x7fffffff;
      for (int r = i + tid; r < N; r += 32) {
        T v = dev_abs(As[i * ld + r]);
        if (!(v == v)) v = T(-1);
        if (v > best) { best = v; bi = r; }
      }
      // upper words of |a| first (one reduction); the exact argmax only on a tie
      const unsigned key = best < T(0) ? 0u : (unsigned)((unsigned long long)__double_as_longlong((double)best) >> 32) + 1u;
      const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
      const unsigned m = __ballot_sync(0xffffffffu, key == kmax);
      if (__popc(m) == 1 && kmax > 0) {
        bi = __shfl_sync(0xffffffffu, bi, __ffs(m) - 1);
      } else {
        warp_argmax(best, bi);
      }
      if (tid == 0) { s_p = bi; s_pv = As[i * ld + bi]; }
    }
    __syncthreads();
    const int p = s_p;
    const T pv = s_pv;
    if (pv == T(0)) {
      if (tid == 0) report(st, DEV_LAST_SINGULAR, -1, i + 1, -1);
      return;
    }
    if (tid == 0) b.piv[i] = p;
    if (p != i)
      for (int c = tid; c < N; c += bs) {
        const T t = As[c * ld + i]; As[c * ld + i] = As[c * ld + p]; As[c * ld + p] = t;
      }
    __syncthreads();
    const T rinv = T(1) / pv;
    for (int r = i + 1 + tid; r < N; r += bs) As[i * ld + r] *= rinv;
    __syncthreads();
    {  // trailing update: thread -> row (tid % 64), columns every bs/64
      const int r = i + 1 + (tid & 63), cs = bs >> 6;
      if (r < N) {
        const T m = As[i * ld + r];
        for (int c = i + 1 + (tid >> 6); c < N; c += cs)
          As[c * ld + r] = fma(-m, As[c * ld + i], As[c * ld + r]);
      }
    }
    __syncthreads();
  }
  for (int c = tid / 32; c < N; c += bs / 32)
    for (int r = tid & 31; r < N; r += 32) A[(size_t)c * N + r] = As[c * ld + r];
  if (tid == 0) st->kind = FACT_LU;
}

template <typename T>
__device__ void last_factor_body(Dims d, LastBufs b, int sel_last, StatusWords* st) {
  __shared__ T sv[32];
  __shared__ int si[32];
  const int M = d.Nr, N = d.Nc, tid = threadIdx.x, bs = blockDim.x;
  const int kind = last_kind_of(sel_last, M, N);
  T* A = b.A;
  int* piv = b.piv;
  T* tau = b.tau;
  if (kind == FACT_SVD || kind == FACT_SVD_T) {
    last_svd(d, A, b, st);
    return;
  }
  if (kind == FACT_LU && M == N && N <= LAST_SMALL) {
    last_lu_small<T>(d, b, st);
    return;
  }
  if (kind == FACT_LU) {
    if (M != N) { if (tid == 0) report(st, DEV_BAD_SHAPE, -1, 0, -1); return; }
    for (int i = 0; i < N; ++i) {
      T best = T(-1);
      int bi = i;  // stays in range even when every candidate is NaN
      for (int r = i + tid; r < N; r += bs) {
        T v = dev_abs(A[(size_t)i * N + r]);
        if (v > best) { best = v; bi = r; }
      }
      block_argmax(best, bi, sv, si);
      if (tid == 0) piv[i] = bi;
      const T pv = A[(size_t)i * N + bi];
      __syncthreads();  // every thread holds the pivot before column i is swapped
      if (pv == T(0)) { if (tid == 0) report(st, DEV_LAST_SINGULAR, -1, i + 1, -1); return; }
      if (bi != i)
        for (int c = tid; c < N; c += bs) {
          T t = A[(size_t)c * N + i]; A[(size_t)c * N + i] = A[(size_t)c * N + bi]; A[(size_t)c * N + bi] = t;
        }
      __syncthreads();
      const T rinv = T(1) / pv;
      for (int r = i + 1 + tid; r < N; r += bs) A[(size_t)i * N + r] *= rinv;
      __syncthreads();
      const int L = N - i - 1;
      for (int e = tid; e < L * L; e += bs) {
        const int r = i + 1 + e % L, c = i + 1 + e / L;
        A[(size_t)c * N + r] -= A[(size_t)i * N + r] * A[(size_t)c * N + i];
      }
      __syncthreads();
    }
  } else if (kind == FACT_LUPQ) {
    if (M != N) { if (tid == 0) report(st, DEV_BAD_SHAPE, -1, 0, -1); return; }
    const int L = M > N ? M : N;
    for (int i = 0; i < N; ++i) {
      // largest |a| of the trailing block, first in column-major order on ties
      const int w = N - i;
      T best = T(-1);
      int bidx = i * N + i;
      for (int e = tid; e < w * w; e += bs) {
        const int r = i + e % w, c = i + e / w;
        const T v = dev_abs(A[(size_t)c * N + r]);
        const int idx = c * N + r;
        if (v > best || (v == best && idx < bidx)) { best = v; bidx = idx; }
      }
      block_argmax(best, bidx, sv, si);
      const int pr = bidx % N, pc = bidx / N;
      if (tid == 0) { piv[i] = pr; piv[L + i] = pc; }
      __syncthreads();
      if (best == T(0)) { if (tid == 0) report(st, DEV_LAST_SINGULAR, -1, i + 1, -1); return; }
      if (pr != i)
        for (int c = tid; c < N; c += bs) {
          T t = A[(size_t)c * N + i]; A[(size_t)c * N + i] = A[(size_t)c * N + pr]; A[(size_t)c * N + pr] = t;
        }
      __syncthreads();
      if (pc != i)
        for (int r = tid; r < N; r += bs) {
          T t = A[(size_t)i * N + r]; A[(size_t)i * N + r] = A[(size_t)pc * N + r]; A[(size_t)pc * N + r] = t;
        }
      __syncthreads();
      const T pv = A[(size_t)i * N + i];
      __syncthreads();
      for (int r = i + 1 + tid; r < N; r += bs) A[(size_t)i * N + r] /= pv;
      __syncthreads();
      const int Lr = N - i - 1;
      for (int e = tid; e < Lr * Lr; e += bs) {
        const int r = i + 1 + e % Lr, c = i + 1 + e / Lr;
        A[(size_t)c * N + r] -= A[(size_t)i * N + r] * A[(size_t)c * N + i];
      }
      __syncthreads();
    }
  } else {  // Householder QR (QRP: largest remaining column first), M >= N
    if (M < N) { if (tid == 0) report(st, DEV_BAD_SHAPE, -1, 0, -1); return; }
    const int L = M > N ? M : N;
    if (kind == FACT_QRP)
      for (int c = tid; c < N; c += bs) piv[L + c] = c;
    __syncthreads();
    for (int i = 0; i < N; ++i) {
      if (kind == FACT_QRP) {
        T best = T(-1);
        int bc = i;
        for (int c = i + tid; c < N; c += bs) {
          const T* col = A + (size_t)c * M;
          T s2 = T(0);
          for (int r = i; r < M; ++r) s2 += col[r] * col[r];
          if (s2 > best) { best = s2; bc = c; }
        }
        block_argmax(best, bc, sv, si);
        if (bc != i) {
          for (int r = tid; r < M; r += bs) {
            T t = A[(size_t)i * M + r]; A[(size_t)i * M + r] = A[(size_t)bc * M + r]; A[(size_t)bc * M + r] = t;
          }
          if (tid == 0) { const int t = piv[L + i]; piv[L + i] = piv[L + bc]; piv[L + bc] = t; }
        }
        __syncthreads();
      }
      T* v = A + (size_t)i * M;
      const T alpha = v[i];
      T s = T(0);
      for (int r = i + 1 + tid; r < M; r += bs) s += v[r] * v[r];
      s = block_sum(s, sv);
      T t = T(0), beta = alpha;
      if (s != T(0)) {
        const T nrm = sqrt(alpha * alpha + s);
        beta = alpha >= T(0) ? -nrm : nrm;
        t = (beta - alpha) / beta;
        const T sc = T(1) / (alpha - beta);
        for (int r = i + 1 + tid; r < M; r += bs) v[r] *= sc;
      }
      __syncthreads();
      if (tid == 0) { v[i] = beta; tau[i] = t; }
      __syncthreads();
      if (beta == T(0)) { if (tid == 0) report(st, DEV_LAST_SINGULAR, -1, i + 1, -1); return; }
      if (t != T(0))
        for (int c = i + 1 + tid; c < N; c += bs) {
          T* col = A + (size_t)c * M;
          T w = col[i];
          for (int r = i + 1; r < M; ++r) w += v[r] * col[r];
          w *= t;
          col[i] -= w;
          for (int r = i + 1; r < M; ++r) col[r] -= w * v[r];
        }
      __syncthreads();
    }
  }
  if (tid == 0) st->kind = kind;
}

// the select_last2 fallback (cc:1347-1369): when the chosen solver failed on
// the last block, factor the saved copy with the SVD family instead
__device__ void last_fallback_body(Dims d, LastBufs b, StatusWords* st) {
  const int code = st->code;
  __syncthreads();
  if (code != DEV_LAST_SINGULAR && code != DEV_BAD_SHAPE) return;
  if (threadIdx.x == 0) *st = StatusWords{0, 0, 0, 0, 0};
  __syncthreads();
  last_svd(d, b.A2, b, st);
}

// 1 / d is a normal number, so that x * (1 / d) stands for the quotient x / d; else
// (d below 2^-1024, where 1 / d overflows, or at the upper end of the range, where
// it loses bits) the last block's solves divide, whose longer latency each of the
// N dependent steps pays
__device__ __forceinline__ bool reciprocal_is_normal(double rd) {
  const double a = fabs(rd);
  return a >= 2.2250738585072014e-308 && a <= 1.7976931348623157e308;
}

// b <- (L U)^-1 P b with the factors by original row (FACT_LU_ROWS), N <= 512:
// position r on thread r (the CTA has at least N threads), blocks of 32 columns.
// Each thread reads its row's 32 elements of a block in one batch, a block ahead
// of the one being solved, so that the 2 N / 32 steps do not wait for memory
// (195 us at N = 288 with eight loads at a time, interleaved with their uses).
__device__ void last_solve_rows(const double* A, const int* piv, int N, double* b, double* tmp) {
  const int tid = threadIdx.x, bs = blockDim.x, lane = tid & 31;
  constexpr unsigned FULL = 0xffffffffu;
  const int nblk = (N + 31) / 32;
  for (int r = tid; r < N; r += bs) tmp[r] = b[piv[r]];
  __syncthreads();
  for (int r = tid; r < N; r += bs) b[r] = tmp[r];
  const int pr = tid < N ? piv[tid] : 0;
  double m[32];
  auto load = [&](int kb, bool lower) {
#pragma unroll
    for (int u = 0; u < 32; ++u) {
      const int c = 32 * kb + u;
      m[u] = ld_batch(tid < N && c < N && (lower ? c < tid : c >= tid), A + (size_t)c * N + pr);
    }
  };
  load(0, true);
  __syncthreads();
  for (int kb = 0; kb < nblk; ++kb) {
    if (tid / 32 == kb) {  // the warp with the diagonal block
      const int r = tid;
      double v = r < N ? b[r] : 0.0;
#pragma unroll
      for (int u = 0; u < 31; ++u) {
        const double vc = __shfl_sync(FULL, v, u);
        if (lane > u) v = fma(-m[u], vc, v);
      }
      if (r < N) b[r] = v;
    }
    __syncthreads();
    if (tid >= 32 * (kb + 1) && tid < N) {
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int u = 0; u < 32; u += 2) {
        s0 = fma(m[u], b[min(32 * kb + u, N - 1)], s0);
        s1 = fma(m[u + 1], b[min(32 * kb + u + 1, N - 1)], s1);
      }
      b[tid] -= s0 + s1;
    }
    if (kb + 1 < nblk) load(kb + 1, true);
    else load(nblk - 1, false);
    __syncthreads();
  }
  for (int kb = nblk - 1; kb >= 0; --kb) {
    if (tid / 32 == kb) {
      const int r = tid;
      double ud = 1.0;
#pragma unroll
      for (int u = 0; u < 32; ++u)
        if (u == lane) ud = m[u];
      double v = r < N ? b[r] : 0.0;
      const double rdi = r < N ? 1.0 / ud : 0.0;
      if (__all_sync(FULL, r >= N || reciprocal_is_normal(rdi))) {
#pragma unroll
        for (int u = 31; u >= 0; --u) {
          const double xi = __shfl_sync(FULL, v * rdi, u);
          v = lane == u ? xi : fma(-m[u], lane < u ? xi : 0.0, v);
        }
      } else {
#pragma unroll
        for (int u = 31; u >= 0; --u) {
          const double xi = __shfl_sync(FULL, r < N ? v / ud : 0.0, u);
          v = lane == u ? xi : fma(-m[u], lane < u ? xi : 0.0, v);
        }
      }
      if (r < N) b[r] = v;
    }
    __syncthreads();
    if (tid < 32 * kb) {
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int u = 0; u < 32; u += 2) {
        s0 = fma(m[u], b[min(32 * kb + u, N - 1)], s0);
        s1 = fma(m[u + 1], b[min(32 * kb + u + 1, N - 1)], s1);
      }
      b[tid] -= s0 + s1;
    }
    if (kb > 0) load(kb - 1, false);
    __syncthreads();
  }
}

// shared memory that a launch may ask for without raising the kernel's limit: 48 KB
// less the 34 KB that last_solve_body holds statically
constexpr size_t LAST_SOLVE_UNASKED = 14 * 1024;
template <typename T>
__device__ void last_solve_body(Dims d, LastBufs lb, const StatusWords* st, T* x, int ldx, int nrhs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = d.n, M = d.Nr, N = d.Nc, tid = threadIdx.x, bs = blockDim.x;
  const int L = M > N ? M : N;
  T* b = reinterpret_cast<T*>(smem_raw);
  T* tmp = b + L;
  __shared__ T sv[32];
  // the whole L\U of a small last block (order <= LAST_SMALL, ld order + 1)
  __shared__ T big[LAST_SMALL * (LAST_SMALL + 1)];
  const int kind = st->kind;
  if ((kind == FACT_LU || kind == FACT_LU_ROWS) && M == N && N <= LAST_SMALL) {
    // L\U in position order in shared memory; a warp per right-hand side, its
    // values in registers (lane = rows lane and lane + 32)
    __shared__ int perm[LAST_SMALL];
    const bool rows = kind == FACT_LU_ROWS;
    if (rows) {
      for (int r = tid; r < N; r += bs) perm[r] = lb.piv[r];
    } else if (tid == 0) {  // getrf's interchanges
      for (int r = 0; r < N; ++r) perm[r] = r;
      for (int i = 0; i < N; ++i) {
        const int p = lb.piv[i], t = perm[i];
        perm[i] = perm[p];
        perm[p] = t;
      }
    }
    __syncthreads();
    for (int e = tid; e < N * N; e += bs) {
      const int c = e / N, r = e % N;
      big[c * (N + 1) + r] = lb.A[(size_t)c * N + (rows ? perm[r] : r)];
    }
    __syncthreads();
    const int lane = tid & 31, r0 = lane, r1 = lane + 32, ld = N + 1;
    const size_t off = (size_t)d.nblock * n;
    const T d0 = r0 < N ? big[r0 * ld + r0] : T(1), d1 = r1 < N ? big[r1 * ld + r1] : T(1);
    const T rd0 = T(1) / d0, rd1 = T(1) / d1;
    const bool plain = __all_sync(0xffffffffu, reciprocal_is_normal(rd0) && reciprocal_is_normal(rd1));
    for (int c = tid >> 5; c < nrhs; c += bs >> 5) {
      T* xc = x + (size_t)c * ldx;
      auto at = [&](int r) -> T& { return r < n ? xc[r] : xc[off + (r - n)]; };
      T x0 = r0 < N ? at(perm[r0]) : T(0), x1 = r1 < N ? at(perm[r1]) : T(0);
      __syncwarp();
      for (int i = 0; i < N; ++i) {
        const T bi = __shfl_sync(0xffffffffu, i < 32 ? x0 : x1, i & 31);
        if (r0 > i && r0 < N) x0 = fma(-big[i * ld + r0], bi, x0);
        if (r1 > i && r1 < N) x1 = fma(-big[i * ld + r1], bi, x1);
      }
      for (int i = N - 1; i >= 0; --i) {
        const T y = i < 32 ? x0 : x1;
        const T xi = __shfl_sync(0xffffffffu, plain ? y * (i < 32 ? rd0 : rd1) : y / (i < 32 ? d0 : d1), i & 31);
        x0 = r0 == i ? xi : r0 < i ? fma(-big[i * ld + r0], xi, x0) : x0;
        x1 = r1 == i ? xi : r1 < i ? fma(-big[i * ld + r1], xi, x1) : x1;
      }
      if (r0 < N) at(r0) = x0;
      if (r1 < N) at(r1) = x1;
    }
    return;
  }
  const T* A = lb.A;
  const int* piv = lb.piv;
  const T* tau = lb.tau;
  const size_t off = (size_t)d.nblock * n;
  T tol = T(0);
  if (kind == FACT_SVD || kind == FACT_SVD_T) {
    const int Np = kind == FACT_SVD ? N : M;
    T smax = T(0);
    for (int j = tid; j < Np; j += bs) smax = fmax(smax, lb.S[j]);
    for (int o = 16; o > 0; o >>= 1) smax = fmax(smax, __shfl_xor_sync(0xffffffffu, smax, o));
    if ((tid & 31) == 0) sv[tid >> 5] = smax;
    __syncthreads();
    if (tid == 0) {
      T m = T(0);
      for (int w = 0; w < (bs >> 5); ++w) m = fmax(m, sv[w]);
      sv[0] = m;
    }
    __syncthreads();
    tol = sv[0] * T(1e-12);
    __syncthreads();
  }
  for (int c = 0; c < nrhs; ++c) {
    T* xc = x + (size_t)c * ldx;
    for (int r = tid; r < M; r += bs) b[r] = r < n ? xc[r] : xc[off + (r - n)];
    __syncthreads();
    if (kind == FACT_SVD || kind == FACT_SVD_T) {
      // x = V S^+ U^T b (Nr >= Nc) or x = U S^+ V^T b (Nr < Nc)
      const bool trn = kind == FACT_SVD_T;
      const int Mp = trn ? N : M, Np = trn ? M : N;
      const int lane = tid & 31, warp = tid >> 5, nw = bs >> 5;
      for (int j = warp; j < Np; j += nw) {
        const T sj = lb.S[j];
        T s = T(0);
        if (sj > tol) {
          const T* col = trn ? lb.V + (size_t)j * Np : lb.U + (size_t)j * Mp;
          const int len = trn ? Np : Mp;
          for (int i = lane; i < len; i += 32) s = fma(col[i], b[i], s);
          s = warp_sum(s) / sj;
        }
        if (lane == 0) tmp[j] = s;
      }
      __syncthreads();
      const int nout = trn ? Mp : Np;
      for (int i = tid; i < nout; i += bs) {
        T s = T(0);
        for (int j = 0; j < Np; ++j)
          s = fma(trn ? lb.U[(size_t)j * Mp + i] : lb.V[(size_t)j * Np + i], tmp[j], s);
        b[i] = s;
      }
      __syncthreads();
    } else {
      if (kind == FACT_LU || kind == FACT_LUPQ) {
        if (tid == 0)
          for (int i = 0; i < N; ++i) {
            const int p = piv[i];
            if (p != i) { T t = b[i]; b[i] = b[p]; b[p] = t; }
          }
        __syncthreads();
        for (int i = 0; i < N; ++i) {
          const T bi = b[i];
          for (int r = i + 1 + tid; r < N; r += bs) b[r] -= A[(size_t)i * N + r] * bi;
          __syncthreads();
        }
      } else if (kind == FACT_LU_ROWS) {
        last_solve_rows(A, piv, N, b, tmp);
      } else {
        for (int i = 0; i < N; ++i) {
          const T* v = A + (size_t)i * M;
          T s = T(0);
          for (int r = i + 1 + tid; r < M; r += bs) s += v[r] * b[r];
          s = block_sum(s, sv);
          s = (s + b[i]) * tau[i];
          __syncthreads();
          if (tid == 0) b[i] -= s;
          for (int r = i + 1 + tid; r < M; r += bs) b[r] -= s * v[r];
          __syncthreads();
        }
      }
      const int lda = (kind == FACT_LU || kind == FACT_LUPQ) ? N : M;
      if (kind == FACT_LU_ROWS) {  // done above
      } else {
        for (int i = N - 1; i >= 0; --i) {
          const T xi = b[i] / A[(size_t)i * lda + i];
          __syncthreads();
          if (tid == 0) b[i] = xi;
          for (int r = tid; r < i; r += bs) b[r] -= A[(size_t)i * lda + r] * xi;
          __syncthreads();
        }
      }
      if (kind == FACT_LUPQ) {
        if (tid == 0)
          for (int i = N - 1; i >= 0; --i) {
            const int q = piv[L + i];
            if (q != i) { T t = b[i]; b[i] = b[q]; b[q] = t; }
          }
        __syncthreads();
      } else if (kind == FACT_QRP) {
        for (int i = tid; i < N; i += bs) tmp[piv[L + i]] = b[i];
        __syncthreads();
        for (int i = tid; i < N; i += bs) b[i] = tmp[i];
        __syncthreads();
      }
    }
    for (int r = tid; r < N; r += bs) {
      if (r < n) xc[r] = b[r];
      else xc[off + (r - n)] = b[r];
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void k_last_factor(Dims d, LastBufs b, int sel_last, StatusWords* st) {
  last_factor_body<T>(d, b, sel_last, st);
}

// load_and_factorize_last with LU for larger blocks (cc:1319-1346, getrf): the
// blocked elimination of the pair kernels on the whole block, FP64 tensor-core
// products, rows left in place (kind FACT_LU_ROWS, piv[pos] = row)
__global__ void __launch_bounds__(512, 1) k_last_lu_blocked(Dims d, LastBufs b, StatusWords* st) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LubShared<512> sh;
  const int N = d.Nc, tid = threadIdx.x;
  if (d.Nr != N || N > LUB_ROWS_MAX) {
    if (tid == 0) report(st, DEV_BAD_SHAPE, -1, 0, -1);
    return;
  }
  const int info = lub_square(sh, reinterpret_cast<double*>(smem_raw), b.A, N, b.piv);
  if (info != 0) {
    if (tid == 0) report(st, DEV_LAST_SINGULAR, -1, info, -1);
    return;
  }
  if (tid == 0) st->kind = FACT_LU_ROWS;
}

__global__ void k_last_fallback(Dims d, LastBufs b, StatusWords* st) { last_fallback_body(d, b, st); }

template <typename T>
__global__ void __launch_bounds__(512, 1) k_last_solve(Dims d, LastBufs b, const StatusWords* st, T* x, int ldx, int nrhs) {
  last_solve_body<T>(d, b, st, x, ldx, nrhs);
}

static LastBufs last_bufs(const DevState& s) {
  LastBufs b;
  b.A = s.Hl; b.A2 = s.Al; b.piv = s.piv_l; b.tau = s.tau_l; b.U = s.Ul; b.V = s.Vl; b.S = s.Sl;
  return b;
}

// ---------------------------------------------------------------------------
// Mv with the loaded matrix (add_Mv, cc:2118-2166): res = alpha*A*x + beta*res
// ---------------------------------------------------------------------------
// ABS: |A| * 1 (row sums of absolute values, for ||A||_inf); x is not read.
// Otherwise, with rowsum non-null, the same pass also writes |A| * 1 there.
template <bool ABS>
__global__ void k_mv_rows(Dims d, const double* D, const double* E, const double* B, double alpha,
                          const double* x, double beta, double* res, double* rowsum = nullptr) {
  const int n = d.n, nx = d.nx;
  const size_t rows = (size_t)d.nblock * n;
  const size_t xb_off = (size_t)(d.nblock + 1) * n + d.qx;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < rows;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t k = e / n;
    const int i = (int)(e % n);
    const double* Dk = D + k * n * n;
    const double* Ek = E + k * n * n;
    const double* Bk = B + k * n * nx;
    // column by column, eight loads of the matrix in flight (see ld_batch);
    // x is the same for a block's rows and comes from L1
    double s = 0.0, sa = 0.0;
    auto run = [&](const double* M, int cols, const double* v) {
      for (int c0 = 0; c0 < cols; c0 += 8) {
        double mv[8], xv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) mv[u] = ld_batch(c0 + u < cols, M + (size_t)(c0 + u) * n + i);
#pragma unroll
        for (int u = 0; u < 8; ++u) xv[u] = ABS ? 0.0 : ld_batch(c0 + u < cols, v + c0 + u);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          s = ABS ? s + fabs(mv[u]) : fma(mv[u], xv[u], s);
          sa += fabs(mv[u]);
        }
      }
    };
    run(Dk, n, x + k * n);
    run(Ek, n, x + (k + 1) * n);
    run(Bk, nx, x + xb_off);
    if constexpr (ABS) {
      res[e] = s;
    } else {
      res[e] = (beta == 0.0 ? 0.0 : beta * res[e]) + alpha * s;
      if (rowsum) rowsum[e] = sa;
    }
  }
}

// C_k x_k per block: 64 elements per CTA round, the columns of each over four
// threads (eight loads in flight), added in a fixed order
template <bool ABS>
__global__ void __launch_bounds__(256) k_mv_cpart(Dims d, const double* C, const double* x, double* part) {
  __shared__ double sp[4][64];
  const int n = d.n, nr = d.nr, t = threadIdx.x & 63, h = threadIdx.x >> 6;
  const size_t total = (size_t)(d.nblock + 1) * nr;
  const int c_lo = n * h / 4, c_hi = n * (h + 1) / 4;
  for (size_t e0 = (size_t)blockIdx.x * 64; e0 < total; e0 += (size_t)gridDim.x * 64) {
    const size_t e = e0 + t, k = e / nr;
    const int r = (int)(e % nr);
    const bool live = e < total;
    const double* Ck = C + k * nr * n;
    double s = 0.0;
    for (int c0 = c_lo; c0 < c_hi; c0 += 8) {
      double cv[8], xv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) cv[u] = ld_batch(live && c0 + u < c_hi, Ck + (size_t)(c0 + u) * nr + r);
#pragma unroll
      for (int u = 0; u < 8; ++u) xv[u] = ABS ? 0.0 : ld_batch(live && c0 + u < c_hi, x + k * n + c0 + u);
#pragma unroll
      for (int u = 0; u < 8; ++u) s = ABS ? s + fabs(cv[u]) : fma(cv[u], xv[u], s);
    }
    sp[h][t] = s;
    __syncthreads();
    if (h == 0 && live) part[e] = ((s + sp[1][t]) + sp[2][t]) + sp[3][t];
    __syncthreads();
  }
}

// H rows and the nr border rows (Csum = sum_k C_k x_k precomputed): 32 rows per
// CTA, the columns over its 16 warps, eight loads in flight each, the partial
// sums added in warp order (one thread per row took 130 us at 144 rows)
constexpr int MVT_W = 16;
template <bool ABS>
__global__ void __launch_bounds__(32 * MVT_W) k_mv_tail(Dims d, const double* H, const double* Cq, const double* F,
                          const double* Csum, double alpha, const double* x, double beta,
                          double* res) {
  __shared__ double part[MVT_W][32];
  const int n = d.n, m = n + d.qr, nr = d.nr, qx = d.qx, nx = d.nx, Nc = d.Nc;
  const size_t r0 = (size_t)d.nblock * n;
  const size_t xN = (size_t)d.nblock * n, xq = (size_t)(d.nblock + 1) * n;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = blockIdx.x * 32 + lane;
  double s = 0.0;
  // columns of [H0 HN Hq Hp] or, for a border row, of [Cq F] (qx + nx of them)
  const bool top = r < m, live = r < m + nr;
  const int cols = top ? Nc : qx + nx;
  for (int c0 = w; c0 < Nc; c0 += 8 * MVT_W) {
    double mv[8], xv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int c = c0 + u * MVT_W, rr = r - m;
      const bool in = live && c < cols;
      const double* M = top ? H + (size_t)c * m + r : c < qx ? Cq + (size_t)c * nr + rr : F + (size_t)(c - qx) * nr + rr;
      const size_t xi = !top ? xq + c : c < n ? (size_t)c : c < 2 * n ? xN + (c - n) : xq + (c - 2 * n);
      mv[u] = ld_batch(in, M);
      xv[u] = ABS ? 0.0 : ld_batch(in, x + xi);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) s = ABS ? s + fabs(mv[u]) : fma(mv[u], xv[u], s);
  }
  part[w][lane] = s;
  __syncthreads();
  if (w == 0 && live) {
    s = top ? 0.0 : Csum[r - m];
#pragma unroll
    for (int o = 0; o < MVT_W; ++o) s += part[o][lane];
    const size_t o = r0 + r;
    res[o] = ABS ? s : (beta == 0.0 ? 0.0 : beta * res[o]) + alpha * s;
  }
}

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------
// Raise a kernel's dynamic shared-memory limit once per process and kernel;
// later calls (for instance inside a CUDA graph capture) only launch.
template <typename K>
static void smem_limit_once(K* kernel, size_t bytes, size_t unasked = 32 * 1024) {
  if (bytes <= unasked) return;  // 48 KB less what a kernel may hold statically
  static const void* keys[64];
  static size_t done[64];
  static int used = 0;
  const void* key = reinterpret_cast<const void*>(kernel);
  int slot = 0;
  while (slot < used && keys[slot] != key) ++slot;
  if (slot < used && done[slot] >= bytes) return;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (slot == used && used < 64) { keys[used] = key; ++used; }
  if (slot < 64) done[slot] = bytes;
}

// CTAs of `kernel` resident on one SM (cached per kernel)
template <typename K>
static int resident_ctas(K* kernel, int threads, size_t smem) {
  static const void* keys[64];
  static int value[64];
  static int used = 0;
  const void* key = reinterpret_cast<const void*>(kernel);
  for (int i = 0; i < used; ++i)
    if (keys[i] == key) return value[i];
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem) != cudaSuccess || nb < 1) nb = 1;
  if (used < 64) { keys[used] = key; value[used] = nb; ++used; }
  return nb;
}

static int grid_for(long work_items, int per_cta, int cap) {
  long g = (work_items + per_cta - 1) / per_cta;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

// the first failed launch of this thread since launch_error() was last asked
static thread_local cudaError_t first_launch_error = cudaSuccess;

static void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    fprintf(stderr, "alglin_b200: launch of %s failed: %s\n", what, cudaGetErrorString(e));
    if (first_launch_error == cudaSuccess) first_launch_error = e;
  }
}

cudaError_t launch_error() {
  const cudaError_t e = first_launch_error, last = cudaGetLastError();
  first_launch_error = cudaSuccess;
  return e != cudaSuccess ? e : last;
}

// sums of per-block m-vectors, m = h x cols (column-major, height h), in pieces of
// at most 256 elements, one after the other: groups of whole columns, or for
// h > 256 the rows of one column
static void reduce_blocks(DevState& s, const double* buf, long first, long count, int m, int h,
                          const double* base, int ldb, double* out, int ldo, cudaStream_t st) {
  if (m <= 0 || h <= 0) return;
  const int cols = m / h, cw = h <= 256 ? 256 / h : 1, hw = std::min(h, 256);
  // about 96 parts: enough CTAs to have the sums in flight, few enough for the
  // one CTA that adds the parts (16,383 sums of 64 elements took 46 us in 16
  // parts of 1,024); whole rounds of the CTA's 256 / (column height) groups
  const long unit = 256 / (std::min(cols, cw) * hw) * 8;
  const long chunk = std::max(unit, (count / 96 + unit) / unit * unit);
  const int nparts = count > 0 ? (int)((count + chunk - 1) / chunk) : 0;
  for (int c0 = 0; c0 < cols; c0 += cw)
    for (int r0 = 0; r0 < h; r0 += hw) {
      const int hn = std::min(hw, h - r0), mm = std::min(cw, cols - c0) * hn;
      const double* bb = buf + (size_t)c0 * h + r0;
      const double* ba = base ? base + (size_t)c0 * ldb + r0 : nullptr;
      double* oo = out + (size_t)c0 * ldo + r0;
      if (nparts > 1) {
        k_reduce_tree<double><<<nparts, 256, 0, st>>>(bb, m, first, count, mm, chunk, s.part, nullptr, hn,
                                                      0, nullptr, 0);
        check_launch("k_reduce_tree");
        k_reduce_tree<double><<<1, 256, 0, st>>>(s.part, mm, 0, nparts, mm, nparts, nullptr, ba, hn, ldb,
                                                 oo, ldo);
      } else {
        k_reduce_tree<double><<<1, 256, 0, st>>>(bb, m, first, count, mm, chunk, nullptr, ba, hn, ldb, oo,
                                                 ldo);
      }
      check_launch("k_reduce_tree");
    }
}

// ---------------------------------------------------------------------------
// working arrays of one precision
// ---------------------------------------------------------------------------
template <typename T>
struct WorkSet {
  T *D, *E, *B, *C, *Tm, *Rbuf;
  T* slab;
};

static WorkSet<double> work_set(DevState& s, double*) {
  return {s.D, s.E, s.B, s.C, s.T, s.Rbuf, reinterpret_cast<double*>(s.slab)};
}
static WorkSet<float> work_set(DevState& s, float*) {
  return {s.Df, s.Ef, s.Bf, s.Cf, s.Tf, s.Rbuff, reinterpret_cast<float*>(s.slab)};
}

// ---------------------------------------------------------------------------
// pair-kernel choice for the factorization
// ---------------------------------------------------------------------------
using LubKernel = void (*)(FactorArgs<double>, double*, size_t, int);
static LubKernel lub_kernel(const LubPlan& p) {
  if (p.threads == 256)
    return p.depth == 32 ? k_factor_lu_lub<256, 4> : p.depth == 48 ? k_factor_lu_lub<256, 6> : k_factor_lu_lub<256, 8>;
  return p.depth == 32 ? k_factor_lu_lub<512, 4> : p.depth == 48 ? k_factor_lu_lub<512, 6> : k_factor_lu_lub<512, 8>;
}

// Clusters of 2, 4 and 8 CTAs of k_factor_lu_lub that are resident at once (a
// cluster lies within one of the GPU's processing clusters, so that of 8 CTAs
// fewer than 148 / 8 fit); asked for once per thread and shape.
static void lub_clusters(LubPlan& p) {
  static_assert(LUB_SLICES_MAX == 8, "one entry per cluster size");
  struct Entry {
    LubKernel kernel;
    size_t smem;
    int nc[3];
  };
  thread_local Entry cache[16];
  thread_local int used = 0;
  const LubKernel kernel = lub_kernel(p);
  int slot = 0;
  while (slot < std::min(used, 16) && (cache[slot].kernel != kernel || cache[slot].smem != p.smem)) ++slot;
  if (slot == std::min(used, 16)) {
    slot = used++ % 16;
    if (used == 32) used = 16;
    Entry& en = cache[slot];
    en.kernel = kernel;
    en.smem = p.smem;
    for (int i = 0; i < 3; ++i) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1024);
      cfg.blockDim = dim3((unsigned)p.threads);
      cfg.dynamicSmemBytes = p.smem;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2u << i;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      en.nc[i] = 0;
      if (cudaOccupancyMaxActiveClusters(&en.nc[i], kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        en.nc[i] = 0;
      }
    }
  }
  for (int i = 0; i < 3; ++i) p.clusters[i] = cache[slot].nc[i];
}

template <typename T>
struct FactorPlan {
  void (*cta)(FactorArgs<T>, T*, size_t) = nullptr;  // CTA per pair (large n)
  void (*blk)(FactorArgs<T>, T*, size_t) = nullptr;  // CTA per pair, blocked LU (large n, FP32)
  size_t blk_smem = 0;
  LubPlan lub;                                       // CTA or cluster per pair, blocked LU (large n, FP64)
  void (*umma)(FactorArgs<T>, T*, size_t) = nullptr;  // CTA per pair, tcgen05 products (FP32, large n)
  size_t umma_smem = 0;
  void (*tc)(FactorArgs<T>, const FactorArgs<T>*, const BatchCta*) = nullptr;               // tensor-core LU (FP64, n = 8, 16)
  size_t tc_smem = 0;
  void (*tree)(FactorArgs<double>, TreeArgs) = nullptr;  // tc pairs, whole reduction in one launch
  int tree_ctas = 0;
  // tc pairs level by level with the tree's border bookkeeping (single systems)
  void (*tcb)(FactorArgs<double>, const FactorArgs<double>*, const BatchCta*) = nullptr;
  void (*top)(FactorArgs<double>, int) = nullptr;  // the top levels in one CTA (single systems)
  void (*root)(FactorArgs<double>, TreeArgs, int) = nullptr;
  void (*grp)(FactorArgs<T>, const FactorArgs<T>*, const BatchCta*) = nullptr;              // CTA of 2n threads per pair (n = 16, 32)
  size_t grp_smem = 0;
  int grp_threads = 0, grp_ctas = 0;
  void (*rows)(FactorArgs<T>, const FactorArgs<T>*, const BatchCta*) = nullptr;             // register LU (n <= 16)
  void (*qr)(FactorArgs<T>, const FactorArgs<T>*, const BatchCta*) = nullptr;               // warp QR / QRP (n <= 16)
  void (*smem_k)(FactorArgs<T>, const FactorArgs<T>*, const BatchCta*) = nullptr;           // shared-memory kernel
  size_t smem = 0;
  int wpb = 1;
  int tc_cols = 0;                                   // trailing-column capacity of tc
};

// the warp-per-pair LU kernel eliminates the pairs of this state (its factors
// are in operator form, which the forward sweep has to know).  Orders other than
// 8 and 16 run as their leading parts: at n = 12, 20,011 blocks, level 1 takes
// 82 us against 148 in the register kernel (k_factor_lu_rows), a lone pair 11
// against 16 us; up to n = 4 with borders it takes, that kernel stays.  The tree
// and gather schedules are FP64 only and unpadded.
static bool tc_pair_selected(const DevState& s) {
  const Dims d = s.d;
  if (s.sel != SEL_LU || d.nr > 8 || d.nx > 8 || !s.use_tc) return false;
  if (d.n != 16 && d.n != 8)  // padded to 8 or 16
    return d.n < 16 && (s.pair_kernel == PAIR_AUTO || s.pair_kernel == PAIR_TC) &&
           (d.n > 4 || d.nr > 4 || d.nx > 4);
  return s.pair_kernel == PAIR_AUTO || s.pair_kernel == PAIR_TC ||
         (!s.mixed && (s.pair_kernel == PAIR_TREE || s.pair_kernel == PAIR_TC_GATHER));
}

// The register QR kernel against the shared-memory one on a level of np pairs.  Its
// cost is a whole warp's registers per step, in two passes where the work matrix
// has more than 32 columns; the other's shrinks with the order and with every
// column beyond a multiple of 32 eliminated.  Few pairs (up to two per scheduler):
// the chain of a lone pair decides, 0.80 to 1.02 of the other's time from order 7
// on in one pass, 0.81 to 0.98 at 12 and 13 and 0.79 to 0.90 at 10 and 11 in two
// passes (1.00 to 1.10 there below 36 columns; 1.01 to 1.15 at 7 to 9).  Many
// pairs: the work does, 0.70 to 1.05 from order 12 and 39 columns on, and 1.05 to
// 2.1 below, for which that kernel stays.
static bool qr_warp_faster(const Dims& d, long np) {
  const int cols = 3 * d.n + d.nx;
  if (d.n >= 12 && cols >= 39) return true;
  if (np > 148L * 8) return false;
  return cols <= 32 ? d.n >= 7 : d.n >= 12 || (d.n >= 10 && cols >= 36);
}

template <typename T>
static FactorPlan<T> plan_factor(const DevState& s) {
  const Dims d = s.d;
  const int n = d.n;
  FactorPlan<T> p;
  const size_t per_warp = panel_smem_per_warp(d, (int)sizeof(T));
  p.wpb = (int)(SMEM_MAX / per_warp);
  if (p.wpb > WARPS_PANEL) p.wpb = WARPS_PANEL;
  if (p.wpb < 1) p.wpb = 1;
  p.smem = per_warp * p.wpb;
  p.smem_k = s.sel == SEL_LU ? k_factor_level<T, SEL_LU>
           : s.sel == SEL_QR ? k_factor_level<T, SEL_QR> : k_factor_level<T, SEL_QRP>;
  if (p.smem <= SMEM_MAX) smem_limit_once(p.smem_k, p.smem);
  if constexpr (sizeof(T) == 8) {
    if (tc_pair_selected(s)) {
      const int N = n <= 8 ? 8 : 16;
      p.tc_smem = tc_smem_per_warp(N) * 4;
      // border rows spread over the warp: 8 lanes per row when nr <= 4, else 4
      const bool r4 = d.nr <= 4;
      if (n != N) {
        if (N == 16) p.tc = r4 ? k_factor_lu_tc<16, false, false, 4, T, true> : k_factor_lu_tc<16, false, false, 8, T, true>;
        else p.tc = r4 ? k_factor_lu_tc<8, false, false, 4, T, true> : k_factor_lu_tc<8, false, false, 8, T, true>;
      } else if (n == 16) p.tc = r4 ? k_factor_lu_tc<16, false, false, 4> : k_factor_lu_tc<16, false, false, 8>;
      else p.tc = r4 ? k_factor_lu_tc<8, false, false, 4> : k_factor_lu_tc<8, false, false, 8>;
      smem_limit_once(p.tc, p.tc_smem);
      p.tc_cols = 2 * n + 8;
      if (s.tree_cnt) {  // single systems (batches keep their own level loop)
        if (n != N) {
          if (N == 16) p.top = r4 ? k_factor_top_tc<16, 4, true> : k_factor_top_tc<16, 8, true>;
          else p.top = r4 ? k_factor_top_tc<8, 4, true> : k_factor_top_tc<8, 8, true>;
        } else if (n == 16) p.top = r4 ? k_factor_top_tc<16, 4> : k_factor_top_tc<16, 8>;
        else p.top = r4 ? k_factor_top_tc<8, 4> : k_factor_top_tc<8, 8>;
        smem_limit_once(p.top, tc_smem_per_warp(N) * TOP_WARPS);
      }
      if (s.pair_kernel == PAIR_TC_GATHER && n == N && s.tree_cnt && d.nblock >= 2) {
        if (n == 16) p.tcb = r4 ? k_factor_lu_tc<16, false, true, 4> : k_factor_lu_tc<16, false, true, 8>;
        else p.tcb = r4 ? k_factor_lu_tc<8, false, true, 4> : k_factor_lu_tc<8, false, true, 8>;
        p.root = n == 16 ? k_tree_root<16> : k_tree_root<8>;
        smem_limit_once(p.tcb, p.tc_smem);
      }
      // the tree schedule (single systems with at least one pair), on request:
      // its top levels run one pair per warp along a serial chain, which costs
      // more than the level-by-level launches save at the sizes measured
      if (s.pair_kernel == PAIR_TREE && n == N && s.tree_cnt && d.nblock >= 2) {
        if (n == 16) p.tree = r4 ? k_factor_tree_tc<16, 4> : k_factor_tree_tc<16, 8>;
        else p.tree = r4 ? k_factor_tree_tc<8, 4> : k_factor_tree_tc<8, 8>;
        smem_limit_once(p.tree, p.tc_smem);
        p.tree_ctas = 148 * resident_ctas(p.tree, 128, p.tc_smem);
      }
    }
  } else {
    // FP32 factors (mixed path): the same warp-per-pair kernel with FP32
    // products, level by level, no fused right-hand sides
    if (tc_pair_selected(s)) {
      const int N = n <= 8 ? 8 : 16;
      p.tc_smem = tc_smem_per_warp_t<T>(N) * 4;
      const bool r4 = d.nr <= 4;
      if (n != N) {
        if (N == 16) p.tc = r4 ? k_factor_lu_tc<16, false, false, 4, T, true> : k_factor_lu_tc<16, false, false, 8, T, true>;
        else p.tc = r4 ? k_factor_lu_tc<8, false, false, 4, T, true> : k_factor_lu_tc<8, false, false, 8, T, true>;
      } else if (n == 16) p.tc = r4 ? k_factor_lu_tc<16, false, false, 4, T> : k_factor_lu_tc<16, false, false, 8, T>;
      else p.tc = r4 ? k_factor_lu_tc<8, false, false, 4, T> : k_factor_lu_tc<8, false, false, 8, T>;
      smem_limit_once(p.tc, p.tc_smem);
      p.tc_cols = 2 * n + 8;
    }
  }
  // orders between 16 and 32 run as the leading part of a block of order 32
  const bool grp_ok = s.sel == SEL_LU && d.nr <= 8 && d.nx <= 8 &&
                      ((n > 16 && n <= 32) || (n == 16 && (sizeof(T) == 4 || s.pair_kernel == PAIR_GRP)));
  if (!p.tc && grp_ok && (s.pair_kernel == PAIR_AUTO || s.pair_kernel == PAIR_GRP)) {
    if (n > 16) {
      p.grp = n == 32 ? k_factor_lu_grp<T, 32> : k_factor_lu_grp<T, 32, false, true>;
      p.grp_smem = GrpShape<T, 32>::BYTES;
    } else {
      p.grp = k_factor_lu_grp<T, 16>;
      p.grp_smem = GrpShape<T, 16>::BYTES;
    }
    p.grp_threads = (n > 16 ? 64 : 32) + 32;
    smem_limit_once(p.grp, p.grp_smem);
    p.grp_ctas = 148 * resident_ctas(p.grp, p.grp_threads, p.grp_smem);
  }
  if (!p.tc && !p.grp && s.sel == SEL_LU && d.nr <= 4 && d.nx <= 4 && s.pair_kernel != PAIR_CTA &&
      s.pair_kernel != PAIR_SMEM) {
    if (n <= 4) p.rows = k_factor_lu_rows<T, 4, 4, 4>;
    else if (n <= 8) p.rows = k_factor_lu_rows<T, 8, 4, 4>;
    else if (n <= 16) p.rows = k_factor_lu_rows<T, 16, 4, 4>;
  }
  // QR panels in registers where some level gains (see qr_warp_faster); a forced
  // family keeps the shared-memory kernels
  if (s.sel != SEL_LU && n <= 16 && d.nr <= 8 && n + d.nx <= 32 && s.pair_kernel == PAIR_AUTO && qr_warp_faster(d, 1)) {
    p.qr = s.sel == SEL_QR ? k_factor_qr_warp<T, false> : k_factor_qr_warp<T, true>;
    smem_limit_once(p.qr, QrShape<T>::BYTES * 4);
  }
  const bool smem_fits = per_warp <= SMEM_MAX;
  if (!p.tc && !p.grp && !p.rows && !p.qr &&
      (use_cta_kernel(d) || s.pair_kernel == PAIR_CTA || !smem_fits) &&
      (s.pair_kernel != PAIR_SMEM || !smem_fits)) {
    p.cta = s.sel == SEL_LU ? k_factor_cta<T, SEL_LU>
          : s.sel == SEL_QR ? k_factor_cta<T, SEL_QR> : k_factor_cta<T, SEL_QRP>;
    if constexpr (sizeof(T) == 8) {
      p.lub = s.sel == SEL_LU ? lub_plan(2 * n + d.nr, n) : LubPlan{};
      if (p.lub.threads) {
        smem_limit_once(lub_kernel(p.lub), p.lub.smem);
        lub_clusters(p.lub);
      }
    } else {
      const size_t bsm = (size_t)BLK_W * (2 * n + d.nr) * sizeof(T);
      if (s.sel == SEL_LU && n <= 128 && 2 * n + d.nr <= BLK_ROWS_MAX && bsm <= SMEM_MAX) {
        p.blk = k_factor_lu_blocked<T>;
        p.blk_smem = bsm;
        smem_limit_once(p.blk, bsm);
      }
    }
    if constexpr (sizeof(T) == 4) {
      if (s.sel == SEL_LU && umma_fits(d) && (s.pair_kernel == PAIR_AUTO || s.pair_kernel == PAIR_UMMA)) {
        p.umma = k_factor_lu_umma;
        p.umma_smem = umma_layout(d).bytes;
        smem_limit_once(p.umma, p.umma_smem);
      }
    }
  }
  return p;
}

// number of right-hand sides the factorization can carry (0: none)
template <typename T>
static int fusable_rhs(const DevState& s, const FactorPlan<T>& p, int nrhs) {
  if (!p.tc || nrhs < 1 || nrhs > 16) return 0;
  return 2 * s.d.n + s.d.nx + nrhs <= p.tc_cols ? nrhs : 0;
}

// one level of k_factor_lu_lub (see lub_grid)
static void launch_lub(const FactorArgs<double>& a, double* slab, size_t slab_elems, int slab_ctas, const LubPlan& p,
                       long np, cudaStream_t st) {
  const LubGrid g = lub_grid(p, np, 2 * a.d.n + a.d.nx, slab_ctas);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.ctas);
  cfg.blockDim = dim3((unsigned)p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g.slices;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, lub_kernel(p), a, slab, slab_elems, p.bw);
}

// every CR level: pair eliminations and the C_jpp border fix-up.  Returns true
// when the tree schedule ran, which also leaves F (s.Ffin), C_nblock and, for
// fused right-hand sides, xb complete.
template <typename T>
static bool factor_levels(DevState& s, const FactorPlan<T>& p, const WorkSet<T>& w, double* x, int ldx,
                          int nrf, cudaStream_t st) {
  const Dims d = s.d;
  const int n = d.n, nb = d.nblock;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * d.nx, nrn = (size_t)d.nr * n;
  cudaMemsetAsync(s.st, 0, sizeof(StatusWords), st);
  // blocks not touched by the first level: the unpaired tail and C_nblock
  if (nb % 2 == 1) {
    const size_t t = (size_t)(nb - 1);
    k_convert_blocks<T><<<1, 256, 0, st>>>(s.D0 + t * nn, w.D + t * nn, nn);
    k_convert_blocks<T><<<1, 256, 0, st>>>(s.E0 + t * nn, w.E + t * nn, nn);
    if (nnx) k_convert_blocks<T><<<1, 256, 0, st>>>(s.B0 + t * nnx, w.B + t * nnx, nnx);
    if (nrn) k_convert_blocks<T><<<1, 256, 0, st>>>(s.C0 + t * nrn, w.C + t * nrn, nrn);
  }
  if (nrn) k_convert_blocks<T><<<1, 256, 0, st>>>(s.C0 + (size_t)nb * nrn, w.C + (size_t)nb * nrn, nrn);
  FactorArgs<T> a;
  a.d = d;
  a.D0 = s.D0; a.E0 = s.E0; a.B0 = s.B0; a.C0 = s.C0;
  a.D = w.D; a.E = w.E; a.B = w.B; a.C = w.C;
  a.Tm = w.Tm; a.P = s.P; a.Rbuf = w.Rbuf; a.Fbuf = s.Fbuf; a.st = s.st;
  a.ldw = odd_ld(2 * n + d.nr);
  a.x = x; a.ldx = ldx; a.nrf = nrf; a.XB = s.XB;
  a.qb = a.qe = 0;
  if constexpr (sizeof(T) == 8) {
    if (p.tree || p.tcb) {
      a.F0 = s.F0;
      TreeArgs ta;
      ta.cnt = s.tree_cnt;
      ta.leaf = s.tree_cnt + nb;
      ta.Ffin = s.Ffin;
      ta.xb = (nrf > 0 && d.nr > 0) ? x + (size_t)(nb + 1) * n + d.qr : nullptr;
      if (p.tree) {
        cudaMemsetAsync(s.tree_cnt, 0, (size_t)(nb + 1) * sizeof(int), st);
        const long leaves = pairs_at_level(nb, 1);
        p.tree<<<grid_for(leaves, 4, p.tree_ctas), 128, p.tc_smem, st>>>(a, ta);
        check_launch("k_factor_tree_tc");
        return true;
      }
      int root = 1;
      for (int k = 1; k < nb; k *= 2) {
        a.k = k;
        a.first = (k == 1);
        root = k;  // the pair (0, k) of the top level
        // level 1 has no gathers and no children: the plain instantiation
        (k == 1 ? p.tc : p.tcb)<<<grid_for(pairs_at_level(nb, k), 4, 148 * 16), 128, p.tc_smem, st>>>(
            a, nullptr, nullptr);
        check_launch("k_factor_lu_tc");
      }
      p.root<<<1, 32, 0, st>>>(a, ta, root);
      check_launch("k_tree_root");
      return true;
    }
  }
  for (int k = 1; k < nb; k *= 2) {
    a.k = k;
    a.first = (k == 1);
    const long np = pairs_at_level(nb, k);
    if constexpr (sizeof(T) == 8) {
      if (p.tc && p.top && np <= TOP_WARPS) {  // this level and every one above it
        p.top<<<1, TOP_WARPS * 32, tc_smem_per_warp(n <= 8 ? 8 : 16) * TOP_WARPS, st>>>(a, k);
        check_launch("k_factor_top_tc");
        break;
      }
    }
    if (p.umma) p.umma<<<grid_for(np, 1, 148), UM_NT, p.umma_smem, st>>>(a, w.slab, s.slab_elems);
    else if (p.lub.threads) {
      if constexpr (sizeof(T) == 8) launch_lub(a, w.slab, s.slab_elems, s.slab_ctas, p.lub, np, st);
    } else if (p.blk) p.blk<<<grid_for(np, 1, s.slab_ctas), 256, p.blk_smem, st>>>(a, w.slab, s.slab_elems);
    else if (p.cta) p.cta<<<grid_for(np, 1, s.slab_ctas), 256, 0, st>>>(a, w.slab, s.slab_elems);
    else if (p.grp) p.grp<<<grid_for(np, 1, p.grp_ctas), p.grp_threads, p.grp_smem, st>>>(a, nullptr, nullptr);
    else if (p.tc) p.tc<<<grid_for(np, 4, 148 * 16), 128, p.tc_smem, st>>>(a, nullptr, nullptr);
    else if (p.rows) p.rows<<<grid_for(np, 4, 148 * 16), 128, 0, st>>>(a, nullptr, nullptr);
    else if (p.qr && qr_warp_faster(d, np)) p.qr<<<grid_for(np, 4, 148 * 16), 128, QrShape<T>::BYTES * 4, st>>>(a, nullptr, nullptr);
    else p.smem_k<<<grid_for(np, p.wpb, 148 * 16), p.wpb * 32, p.smem, st>>>(a, nullptr, nullptr);
    check_launch("k_factor_level");
    if (nrn) {
      const long tot = np * (long)nrn;
      k_border_fix<T><<<grid_for(tot, 256, 148 * 8), 256, 0, st>>>(d, w.C, w.Rbuf, k);
      check_launch("k_border_fix");
    }
  }
  return false;
}

// F = F0 + sum of the Schur updates (FP64); assemble and factor the last block (FP64)
template <typename T>
static void factor_last(DevState& s, const WorkSet<T>& w, cudaStream_t st, bool f_done = false) {
  const Dims d = s.d;
  const int nrnx = d.nr * d.nx;
  if (nrnx > 0 && !f_done)
    reduce_blocks(s, s.Fbuf, 1, d.nblock - 1, nrnx, d.nr, s.F0, d.nr, s.Ffin, d.nr, st);
  k_last_assemble<T><<<grid_for((long)d.Nr * d.Nc, 256, 64), 256, 0, st>>>(
      d, w.D, w.E, w.B, w.C, s.H, s.Cq, s.Ffin, s.Hl);
  check_launch("k_last_assemble");
  if (s.sel_last2) {  // a copy of the assembled block for the fallback solver
    cudaMemcpyAsync(s.Al, s.Hl, (size_t)d.Nr * d.Nc * 8, cudaMemcpyDeviceToDevice, st);
  }
  const LastBufs lb = last_bufs(s);
  if (s.sel_last == LAST_LU && d.Nr == d.Nc && d.Nc >= 1 && d.Nc <= LUB_ROWS_MAX) {
    const size_t sm = lub_last_smem(d.Nc);
    smem_limit_once(k_last_lu_blocked, sm);
    k_last_lu_blocked<<<1, 512, sm, st>>>(d, lb, s.st);
    check_launch("k_last_lu_blocked");
  } else {
    k_last_factor<double><<<1, 512, 0, st>>>(d, lb, s.sel_last, s.st);
    check_launch("k_last_factor");
  }
  if (s.sel_last2) {
    k_last_fallback<<<1, 512, 0, st>>>(d, lb, s.st);
    check_launch("k_last_fallback");
  }
}

template <typename T>
static void factorize_t(DevState& s, cudaStream_t st) {
  T* tag = nullptr;
  const WorkSet<T> w = work_set(s, tag);
  const FactorPlan<T> p = plan_factor<T>(s);
  const bool tree = factor_levels(s, p, w, nullptr, 0, 0, st);
  factor_last(s, w, st, tree);
}

void launch_factorize(DevState& s, cudaStream_t st) {
  if (s.mixed) factorize_t<float>(s, st);
  else factorize_t<double>(s, st);
}

// sweep kernels for one chunk of right-hand sides
template <typename T>
struct SweepPlan {
  void (*fwd)(SweepArgs<T>, const SweepArgs<T>*, const BatchCta*, const long*) = nullptr;
  void (*bwd)(SweepArgs<T>, const SweepArgs<T>*, const BatchCta*, const long*) = nullptr;
  // n = 8, 16 single systems: pipelined forward (LU) and backward levels,
  // the backward top in one CTA
  void (*fwd_pipe)(SweepArgs<T>, const SweepArgs<T>*, const BatchCta*, const long*, long) = nullptr;
  size_t fwd_pipe_smem = 0;
  int op = 0;  // the factors are in operator form, by blocks of op columns
  void (*bwd_pipe)(SweepArgs<T>, const SweepArgs<T>*, const BatchCta*, const long*, long) = nullptr;
  size_t bwd_pipe_smem = 0;
  void (*bwd_top)(SweepArgs<T>, int, int) = nullptr;
  size_t bwd_top_smem = 0;  // with several right-hand sides
  // CTA per pair (16 < n, see bcr_sweep_big.cuh): threads, shared memory per right-hand side
  void (*fwd_big)(SweepArgs<T>) = nullptr;
  void (*bwd_big)(SweepArgs<T>) = nullptr;
  int fwd_big_nt = 0, bwd_big_nt = 0;
  size_t fwd_big_smem = 0, bwd_big_smem = 0;
};

template <typename T>
static SweepPlan<T> plan_sweeps(const DevState& s) {
  const Dims d = s.d;
  const int n = d.n;
  SweepPlan<T> p;
  if (d.nr <= 8 && d.nx <= 8 && n <= 16) {
    const bool lu = s.sel == SEL_LU, r4 = d.nr <= 4, x4 = d.nx <= 4;
#define BCR_FWD(NN) (r4 ? (lu ? k_forward_rows<T, NN, 4, true> : k_forward_rows<T, NN, 4, false>) \
                        : (lu ? k_forward_rows<T, NN, 8, true> : k_forward_rows<T, NN, 8, false>))
#define BCR_BWD(NN) (x4 ? k_backward_rows<T, NN, 4> : k_backward_rows<T, NN, 8>)
    if (n <= 4) { p.fwd = BCR_FWD(4); p.bwd = BCR_BWD(4); }
    else if (n <= 8) { p.fwd = BCR_FWD(8); p.bwd = BCR_BWD(8); }
    else { p.fwd = BCR_FWD(16); p.bwd = BCR_BWD(16); }
#undef BCR_FWD
#undef BCR_BWD
  }
  if ((n == 16 || n == 8) && s.sel == SEL_LU && d.nr <= 8) {  // both precisions
    const bool r4 = d.nr <= 4;
    if (n == 16) {
      p.fwd_pipe = r4 ? k_forward_pipe<16, 4, T> : k_forward_pipe<16, 8, T>;
      p.fwd_pipe_smem = 8 * (r4 ? FwdBuf<16, 4, T>::BYTES : FwdBuf<16, 8, T>::BYTES);
    } else {
      p.fwd_pipe = r4 ? k_forward_pipe<8, 4, T> : k_forward_pipe<8, 8, T>;
      p.fwd_pipe_smem = 8 * (r4 ? FwdBuf<8, 4, T>::BYTES : FwdBuf<8, 8, T>::BYTES);
    }
    smem_limit_once(p.fwd_pipe, p.fwd_pipe_smem);
  }
  if ((n == 16 || n == 8) && d.nx <= 8) {  // both precisions
    const bool x4 = d.nx <= 4;
    if (n == 16) {
      p.bwd_pipe = x4 ? k_backward_pipe<16, 4, T> : k_backward_pipe<16, 8, T>;
      p.bwd_pipe_smem = 8 * (x4 ? BwdBuf<16, 4, T>::BYTES : BwdBuf<16, 8, T>::BYTES);
      p.bwd_top = x4 ? k_backward_top<16, 4, T> : k_backward_top<16, 8, T>;
    } else {
      p.bwd_pipe = x4 ? k_backward_pipe<8, 4, T> : k_backward_pipe<8, 8, T>;
      p.bwd_pipe_smem = 8 * (x4 ? BwdBuf<8, 4, T>::BYTES : BwdBuf<8, 8, T>::BYTES);
      p.bwd_top = x4 ? k_backward_top<8, 4, T> : k_backward_top<8, 8, T>;
    }
    smem_limit_once(p.bwd_pipe, p.bwd_pipe_smem);
    if (sizeof(T) == 8) p.bwd_top_smem = p.bwd_pipe_smem;  // one buffer for each of twice the warps
    smem_limit_once(p.bwd_top, p.bwd_top_smem);
  }
  if (n == 32) {
    if (s.sel == SEL_LU && d.nr <= 8) p.fwd = d.nr <= 4 ? k_forward_rows32<T, 4> : k_forward_rows32<T, 8>;
    if (d.nx <= 8) p.bwd = d.nx <= 4 ? k_backward_rows32<T, 4> : k_backward_rows32<T, 8>;
  }
  if (n > 16 && n <= 128) {
    if (s.sel == SEL_LU && !p.fwd) {
      p.fwd_big = n <= 32 ? k_forward_lm<64, T> : n <= 64 ? k_forward_lm<128, T> : k_forward_lm<256, T>;
      const int rw = n <= 32 ? 64 : n <= 64 ? 128 : 256;
      p.fwd_big_nt = rw * (rw / 64);
      p.fwd_big_smem = (size_t)rw * 8;
    }
    if (!p.bwd) {
      const int rb = n <= 32 ? 32 : n <= 64 ? 64 : 128;
      p.bwd_big = n <= 32 ? k_backward_big<32, T> : n <= 64 ? k_backward_big<64, T> : k_backward_big<128, T>;
      p.bwd_big_nt = rb * (rb / 32);
      p.bwd_big_smem = (size_t)(3 * rb + p.bwd_big_nt) * 8;
      smem_limit_once(p.bwd_big, p.bwd_big_smem * SWB_RHS);
    }
  }
  // the form of the factors follows the kernel that made them
  const FactorPlan<T> fp = plan_factor<T>(s);
  if (fp.tc || fp.grp) p.op = n;
  if (n == 32 && s.sel == SEL_LU && !fp.grp) {  // L and M
    p.fwd = nullptr;
    p.fwd_big = k_forward_lm<64, T>;
    p.fwd_big_nt = 64;
    p.fwd_big_smem = 64 * 8;
  }
  if (n > 16 && n < 32 && fp.grp) {
    p.fwd_big = k_forward_op<64, T>;
    p.fwd_big_nt = 128;
    p.fwd_big_smem = (size_t)(3 * 64 + 64) * 8;
  }
  if constexpr (sizeof(T) == 8) {
    if (fp.lub.threads) {
      const int rw = n <= 64 ? 128 : 256;
      p.op = fp.lub.bw;
      p.fwd_big = n <= 64 ? k_forward_op<128, T> : k_forward_op<256, T>;
      p.fwd_big_nt = 2 * rw;
      p.fwd_big_smem = (size_t)(3 * rw + 64) * 8;
      smem_limit_once(p.fwd_big, p.fwd_big_smem * SWB_RHS);
    }
  }
  return p;
}

template <typename T>
static SweepArgs<T> sweep_args(DevState& s, const WorkSet<T>& w, double* x, int ldx, int nrhs) {
  SweepArgs<T> a;
  a.d = s.d;
  a.D = w.D; a.E = w.E; a.B = w.B; a.C = w.C; a.Tm = w.Tm; a.P = s.P;
  a.x = x; a.ldx = ldx; a.nrhs = nrhs; a.XB = s.XB; a.sel = s.sel;
  a.op = 0;
  a.done = nullptr;
  return a;
}

static int top_level(int nb) {
  int K = 1;
  while (K < nb) K *= 2;
  return K;
}

// xb += sum of the per-block -C'_j x_j contributions
static void reduce_xb(DevState& s, double* x, int ldx, int nrhs, cudaStream_t st) {
  const Dims d = s.d;
  if (d.nr > 0) {
    double* xb = x + (size_t)(d.nblock + 1) * d.n + d.qr;
    reduce_blocks(s, s.XB, 1, d.nblock - 1, d.nr * nrhs, d.nr, xb, ldx, xb, ldx, st);
  }
}

template <typename T>
static void forward_levels(DevState& s, const SweepPlan<T>& p, const WorkSet<T>& w, double* x, int ldx,
                           int nrhs, cudaStream_t st) {
  const Dims d = s.d;
  SweepArgs<T> a = sweep_args(s, w, x, ldx, nrhs);
  a.ldw = odd_ld(2 * d.n);
  a.op = p.op;
  const size_t smem_f = (size_t)a.ldw * nrhs * 8 * WARPS_PANEL;
  smem_limit_once(k_forward_level<T>, smem_f);
  for (int K = 1; K < d.nblock; K *= 2) {
    a.k = K;
    const long np = pairs_at_level(d.nblock, K);
    if (p.fwd_big)
      p.fwd_big<<<grid_for(np, 1, 148 * 32), p.fwd_big_nt, p.fwd_big_smem * std::min(nrhs, SWB_RHS), st>>>(a);
    else if (p.fwd_pipe)
      p.fwd_pipe<<<grid_for(np, 8, 148 * 2), 256, p.fwd_pipe_smem, st>>>(a, nullptr, nullptr, nullptr, 0);
    else if (p.fwd) p.fwd<<<grid_for(np, 8, 148 * 32), 256, 0, st>>>(a, nullptr, nullptr, nullptr);
    else k_forward_level<T><<<grid_for(np, WARPS_PANEL, 148 * 16), WARPS_PANEL * 32, smem_f, st>>>(a, nullptr, nullptr, nullptr);
    check_launch("k_forward_level");
  }
  reduce_xb(s, x, ldx, nrhs, st);
}

template <typename T>
static void last_and_backward(DevState& s, const SweepPlan<T>& p, const WorkSet<T>& w, double* x, int ldx,
                              int nrhs, cudaStream_t st) {
  const Dims d = s.d;
  const size_t smem_l = 2 * (size_t)(d.Nr > d.Nc ? d.Nr : d.Nc) * 8;
  smem_limit_once(k_last_solve<double>, smem_l, LAST_SOLVE_UNASKED);
  k_last_solve<double><<<1, 512, smem_l, st>>>(d, last_bufs(s), s.st, x, ldx, nrhs);
  check_launch("k_last_solve");
  SweepArgs<T> a = sweep_args(s, w, x, ldx, nrhs);
  a.ldw = d.n;
  const size_t smem_b = (size_t)d.n * 8 * WARPS_PANEL;
  if (p.bwd_pipe) {
    // the levels with at most 16 pairs (the top) in one CTA, then one
    // pipelined launch per level below.  (With several right-hand sides too: one
    // launch per level at the top made an uncaptured solve of 64 blocks wait for
    // its launches, 46 against 37 us at n = 8 with 2 right-hand sides.)
    int k = top_level(d.nblock) / 2, k_split = 0;
    for (int kk = k; kk > 0 && !k_split; kk /= 2)
      if (pairs_at_level(d.nblock, kk) > 16) k_split = kk;
    if (k > k_split) {
      p.bwd_top<<<1, 512, nrhs > 1 ? p.bwd_top_smem : 0, st>>>(a, k, k_split * 2 > 0 ? k_split * 2 : 1);
      check_launch("k_backward_top");
    }
    for (int kk = k_split; kk > 0; kk /= 2) {
      a.k = kk;
      const long np = pairs_at_level(d.nblock, kk);
      p.bwd_pipe<<<grid_for(np, 8, 148 * 2), 256, p.bwd_pipe_smem, st>>>(a, nullptr, nullptr, nullptr, 0);
      check_launch("k_backward_pipe");
    }
    return;
  }
  for (int k = top_level(d.nblock); (k /= 2) > 0;) {
    a.k = k;
    const long np = pairs_at_level(d.nblock, k);
    if (p.bwd_big)
      p.bwd_big<<<grid_for(np, 1, 148 * 32), p.bwd_big_nt, p.bwd_big_smem * std::min(nrhs, SWB_RHS), st>>>(a);
    else if (p.bwd) p.bwd<<<grid_for(np, 8, 148 * 32), 256, 0, st>>>(a, nullptr, nullptr, nullptr);
    else k_backward_level<T><<<grid_for(np, WARPS_PANEL, 148 * 16), WARPS_PANEL * 32, smem_b, st>>>(a, nullptr, nullptr, nullptr);
    check_launch("k_backward_level");
  }
}

// right-hand sides are independent: sweep them in chunks of at most 16 columns
template <typename T>
static void solve_t(DevState& s, double* x, int ldx, int nrhs, cudaStream_t st) {
  T* tag = nullptr;
  const WorkSet<T> w = work_set(s, tag);
  const SweepPlan<T> p = plan_sweeps<T>(s);
  for (int c0 = 0; c0 < nrhs; c0 += 16) {
    const int nc = nrhs - c0 < 16 ? nrhs - c0 : 16;
    double* xc = x + (size_t)c0 * ldx;
    forward_levels(s, p, w, xc, ldx, nc, st);
    last_and_backward(s, p, w, xc, ldx, nc, st);
  }
}

void launch_solve(DevState& s, double* x, int ldx, int nrhs, cudaStream_t st) {
  if (s.mixed) solve_t<float>(s, x, ldx, nrhs, st);
  else solve_t<double>(s, x, ldx, nrhs, st);
}

// factorize and solve in one pass: when the pair kernel can carry the right-
// hand sides, their forward elimination rides in the factorization's GEMM and
// the separate forward sweep disappears
template <typename T>
static void factorize_solve_t(DevState& s, double* x, int ldx, int nrhs, cudaStream_t st) {
  T* tag = nullptr;
  const WorkSet<T> w = work_set(s, tag);
  const FactorPlan<T> fp = plan_factor<T>(s);
  const int nrf = fusable_rhs(s, fp, nrhs);
  if (nrf == 0) {
    launch_factorize(s, st);
    launch_solve(s, x, ldx, nrhs, st);
    return;
  }
  const bool tree = factor_levels(s, fp, w, x, ldx, nrf, st);
  if (!tree) reduce_xb(s, x, ldx, nrf, st);
  factor_last(s, w, st, tree);
  last_and_backward(s, plan_sweeps<T>(s), w, x, ldx, nrf, st);
}

void launch_factorize_solve(DevState& s, double* x, int ldx, int nrhs, cudaStream_t st) {
  // FP32 factors (mixed path): the right-hand sides are eliminated in FP32,
  // which is the accuracy of the solve with those factors anyway; the caller
  // refines the result
  if (s.mixed) factorize_solve_t<float>(s, x, ldx, nrhs, st);
  else factorize_solve_t<double>(s, x, ldx, nrhs, st);
}

// Factorize + solve with the matrix uploaded from host memory in chunks of
// 2^m consecutive blocks on the copy stream cst, each chunk's own CR levels
// (the pairs lying inside it) launched on st as soon as it has arrived: the
// tc pair kernels with the tree's border bookkeeping write nothing outside a
// chunk but their own Rbuf/Fbuf/XB slots, so chunks need no fix-up and the
// upload overlaps the factorization.  The levels spanning chunks, the root,
// the last block and the backward sweep follow.  Returns false (nothing
// enqueued) when the shape does not take this path.
bool launch_upload_factorize_solve(DevState& s, const HostMatrix& hm, double* x, int ldx, int nrhs,
                                   cudaStream_t st, cudaStream_t cst, cudaEvent_t* ev, int nev) {
  if (s.mixed || !s.tree_cnt) return false;
  const Dims d = s.d;
  const int n = d.n, nb = d.nblock;
  if (nb < 2048 || nev < 2) return false;
  PairKernel saved = (PairKernel)s.pair_kernel;
  if (saved != PAIR_AUTO && saved != PAIR_TC_GATHER) return false;
  s.pair_kernel = PAIR_TC_GATHER;
  const FactorPlan<double> p = plan_factor<double>(s);
  s.pair_kernel = saved;
  if (!p.tc || !p.tcb || !p.root) return false;
  const int nrf = fusable_rhs(s, p, nrhs);
  if (nrf != nrhs) return false;
  // chunks: a power of two of blocks, at most nev of them
  int chunk = 1024;
  while ((long)chunk * nev < nb) chunk *= 2;
  const int nchunks = (nb + chunk - 1) / chunk;
  double* tag = nullptr;
  const WorkSet<double> w = work_set(s, tag);
  const size_t nn = (size_t)n * n, nnx = (size_t)n * d.nx, nrn = (size_t)d.nr * n;
  // the small arrays first, then the chunks
  auto up = [&](double* dst, const double* src, size_t cnt) {
    if (cnt) cudaMemcpyAsync(dst, src, cnt * 8, cudaMemcpyHostToDevice, cst);
  };
  up(s.Cq, hm.Cq, (size_t)d.nr * d.qx);
  up(s.F0, hm.F, (size_t)d.nr * d.nx);
  up(s.H, hm.H, (size_t)(n + d.qr) * d.Nc);
  FactorArgs<double> a;
  a.d = d;
  a.D0 = s.D0; a.E0 = s.E0; a.B0 = s.B0; a.C0 = s.C0;
  a.D = w.D; a.E = w.E; a.B = w.B; a.C = w.C;
  a.Tm = w.Tm; a.P = s.P; a.Rbuf = w.Rbuf; a.Fbuf = s.Fbuf; a.st = s.st;
  a.ldw = odd_ld(2 * n + d.nr);
  a.x = x; a.ldx = ldx; a.nrf = nrf; a.XB = s.XB;
  a.F0 = s.F0;
  cudaMemsetAsync(s.st, 0, sizeof(StatusWords), st);
  for (int c = 0; c < nchunks; ++c) {
    const long b0 = (long)c * chunk, b1 = std::min<long>(b0 + chunk, nb);
    up(s.D0 + b0 * nn, hm.D + b0 * nn, (size_t)(b1 - b0) * nn);
    up(s.E0 + b0 * nn, hm.E + b0 * nn, (size_t)(b1 - b0) * nn);
    up(s.B0 + b0 * nnx, hm.B + b0 * nnx, (size_t)(b1 - b0) * nnx);
    const long c1 = c == nchunks - 1 ? nb + 1 : b1;  // the last chunk also brings C_nblock
    up(s.C0 + b0 * nrn, hm.C + b0 * nrn, (size_t)(c1 - b0) * nrn);
    cudaEventRecord(ev[c % nev], cst);
    cudaStreamWaitEvent(st, ev[c % nev], 0);
    if (c == nchunks - 1) {  // blocks no pair of the first level touches: the odd tail and C_nblock
      if (nb % 2 == 1) {
        const size_t t = (size_t)(nb - 1);
        k_convert_blocks<double><<<1, 256, 0, st>>>(s.D0 + t * nn, w.D + t * nn, nn);
        k_convert_blocks<double><<<1, 256, 0, st>>>(s.E0 + t * nn, w.E + t * nn, nn);
        if (nnx) k_convert_blocks<double><<<1, 256, 0, st>>>(s.B0 + t * nnx, w.B + t * nnx, nnx);
        if (nrn) k_convert_blocks<double><<<1, 256, 0, st>>>(s.C0 + t * nrn, w.C + t * nrn, nrn);
      }
      if (nrn) k_convert_blocks<double><<<1, 256, 0, st>>>(s.C0 + (size_t)nb * nrn, w.C + (size_t)nb * nrn, nrn);
    }
    // the levels whose pairs lie inside [b0, b1): j = k (2q + 1) with b0 < j < b1
    for (int k = 1; k < chunk; k *= 2) {
      const long qb = b0 / (2L * k), np = pairs_at_level(nb, k);
      const long qe = std::min<long>(np, (b1 + k - 1) / (2L * k));  // j < b1
      if (qe <= qb) continue;
      a.k = k;
      a.first = k == 1;
      a.qb = qb;
      a.qe = qe;
      (k == 1 ? p.tc : p.tcb)<<<grid_for(qe - qb, 4, 148 * 16), 128, p.tc_smem, st>>>(a, nullptr, nullptr);
      check_launch("k_factor_lu_tc (chunk)");
    }
  }
  a.qb = a.qe = 0;
  TreeArgs ta;
  ta.cnt = s.tree_cnt;
  ta.leaf = s.tree_cnt + nb;
  ta.Ffin = s.Ffin;
  ta.xb = (nrf > 0 && d.nr > 0) ? x + (size_t)(nb + 1) * n + d.qr : nullptr;
  int root = 1;
  for (int k = 1; k < nb; k *= 2) {
    root = k;
    if (k < chunk) continue;
    a.k = k;
    a.first = 0;
    p.tcb<<<grid_for(pairs_at_level(nb, k), 4, 148 * 16), 128, p.tc_smem, st>>>(a, nullptr, nullptr);
    check_launch("k_factor_lu_tc");
  }
  p.root<<<1, 32, 0, st>>>(a, ta, root);
  check_launch("k_tree_root");
  factor_last(s, w, st, true);
  last_and_backward(s, plan_sweeps<double>(s), w, x, ldx, nrf, st);
  return true;
}

bool factorize_solve_fuses(const DevState& s, int nrhs) {
  if (s.mixed) return false;
  return fusable_rhs(s, plan_factor<double>(s), nrhs) == nrhs;
}

// rowsum (value pass only): the block rows' |A| * 1 from the same reads;
// skip_rows (ABS pass only): the block rows are already done
template <bool ABS>
static void mv_t(DevState& s, double alpha, const double* x, double beta, double* res, cudaStream_t st,
                 double* rowsum = nullptr, bool skip_rows = false) {
  const Dims d = s.d;
  const long rows = (long)d.nblock * d.n;
  if (rows > 0 && !skip_rows) {
    k_mv_rows<ABS><<<grid_for(rows, 256, 148 * 8), 256, 0, st>>>(d, s.D0, s.E0, s.B0, alpha, x, beta, res,
                                                                  rowsum);
    check_launch("k_mv_rows");
  }
  const int nr = d.nr;
  double* Csum = s.Ffin;  // unused when nr == 0
  if (nr > 0) {
    const long tot = (long)(d.nblock + 1) * nr;
    k_mv_cpart<ABS><<<grid_for(tot, 64, 148 * 8), 256, 0, st>>>(d, s.C0, x, s.mv_part);
    check_launch("k_mv_cpart");
    Csum = s.mv_part + (size_t)(d.nblock + 1) * nr;
    reduce_blocks(s, s.mv_part, 0, d.nblock + 1, nr, nr, nullptr, nr, Csum, nr, st);
  }
  k_mv_tail<ABS><<<(d.n + d.qr + nr + 31) / 32, 32 * MVT_W, 0, st>>>(d, s.H, s.Cq, s.F0, Csum, alpha, x, beta, res);
  check_launch("k_mv_tail");
}

void launch_mv(DevState& s, double alpha, const double* x, double beta, double* res, cudaStream_t st) {
  mv_t<false>(s, alpha, x, beta, res, st);
}

// out[slot] = max |v_i| over i < len (exact, order independent)
// inf-norms of up to three vectors, one per blockIdx.y
struct AbsMax {
  const double* v[3];
  long len[3];
};
__global__ void __launch_bounds__(256) k_absmax(AbsMax a, unsigned long long* out) {
  const double* v = a.v[blockIdx.y];
  const long len = a.len[blockIdx.y], step = (long)gridDim.x * blockDim.x;
  double m = 0.0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += 4 * step) {
    double t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = ld_batch(i + u * step < len, v + i + u * step);
#pragma unroll
    for (int u = 0; u < 4; ++u) m = fmax(m, fabs(t[u]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  // one atomic per CTA: a few hundred on one address, not a few thousand
  __shared__ double sm[8];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int o = 1; o < 8; ++o) m = fmax(m, sm[o]);
    atomicMax(out + blockIdx.y, (unsigned long long)__double_as_longlong(m));
  }
}

__global__ void k_axpy(double* y, const double* x, long len) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long)gridDim.x * blockDim.x)
    y[i] += x[i];
}

// r = b - A x and the three inf-norms |r|, |x|, |b| into out[0..2]; with rowsum
// (an nrows-long scratch) non-null, also ||A||_inf into *normA, the block rows'
// |A| sums taken from the residual's own reads of the matrix
void launch_residual(DevState& s, const double* b, const double* x, double* r, unsigned long long* out,
                     cudaStream_t st, double* rowsum, unsigned long long* normA) {
  const Dims d = s.d;
  const long nrows = (long)d.n * (d.nblock + 1) + d.qr + d.nr;
  const long ncols = (long)d.n * (d.nblock + 1) + d.qx + d.nx;
  cudaMemcpyAsync(r, b, (size_t)nrows * 8, cudaMemcpyDeviceToDevice, st);
  mv_t<false>(s, -1.0, x, 1.0, r, st, rowsum);
  if (rowsum) {
    mv_t<true>(s, 1.0, nullptr, 0.0, rowsum, st, nullptr, true);  // border and last rows
    cudaMemsetAsync(normA, 0, sizeof(unsigned long long), st);
    k_absmax<<<grid_for(nrows, 256, 148 * 2), 256, 0, st>>>(AbsMax{{rowsum}, {nrows}}, normA);
  }
  cudaMemsetAsync(out, 0, 3 * sizeof(unsigned long long), st);
  k_absmax<<<dim3(grid_for(nrows, 256, 148 * 2), 3), 256, 0, st>>>(AbsMax{{r, x, b}, {nrows, ncols, nrows}}, out);
  check_launch("k_absmax");
}

void launch_axpy(double* y, const double* x, long len, cudaStream_t st) {
  k_axpy<<<grid_for(len, 256, 148 * 4), 256, 0, st>>>(y, x, len);
  check_launch("k_axpy");
}

// ---------------------------------------------------------------------------
// batches of independent systems (FP64, internal LU)
// ---------------------------------------------------------------------------
struct LastDesc {
  Dims d;
  const double *D0, *E0, *B0, *C0, *H, *Cq, *F0, *Fbuf, *XB;
  void *Dw, *Ew, *Bw, *Cw;  // working blocks: FP64, or FP32 on the mixed path
  double *Ffin, *Hl, *tau, *x;
  int* piv;
  int kind, ldx;
  StatusWords* st;
  LastBufs lb;
  const int* done;  // mixed path: the system's refinement converged (skip its solve)
};

// status reset and the blocks the first level does not touch (odd tail, C_N)
template <typename T>
__global__ void __launch_bounds__(256) kb_begin(const LastDesc* t) {
  const LastDesc& L = t[blockIdx.x];
  const Dims d = L.d;
  const int nb = d.nblock;
  const size_t nn = (size_t)d.n * d.n, nnx = (size_t)d.n * d.nx, nrn = (size_t)d.nr * d.n;
  T* D = static_cast<T*>(L.Dw);
  T* E = static_cast<T*>(L.Ew);
  T* B = static_cast<T*>(L.Bw);
  T* C = static_cast<T*>(L.Cw);
  if (threadIdx.x == 0) *L.st = StatusWords{0, 0, 0, 0, 0};
  if (nb % 2 == 1) {
    const size_t b = (size_t)(nb - 1);
    for (size_t e = threadIdx.x; e < nn; e += blockDim.x) {
      D[b * nn + e] = T(L.D0[b * nn + e]);
      E[b * nn + e] = T(L.E0[b * nn + e]);
    }
    for (size_t e = threadIdx.x; e < nnx; e += blockDim.x) B[b * nnx + e] = T(L.B0[b * nnx + e]);
    for (size_t e = threadIdx.x; e < nrn; e += blockDim.x) C[b * nrn + e] = T(L.C0[b * nrn + e]);
  }
  for (size_t e = threadIdx.x; e < nrn; e += blockDim.x) C[(size_t)nb * nrn + e] = T(L.C0[(size_t)nb * nrn + e]);
}

// C_jpp += dC_jpp for the pairs of each chunk (one writer per target block)
template <typename T>
__global__ void __launch_bounds__(128) kb_border_fix(const FactorArgs<T>* tab, const BatchCta* cmap, int k) {
  const BatchCta c = cmap[blockIdx.x];
  const FactorArgs<T>& a = tab[c.sys];
  const Dims d = a.d;
  const size_t nrn = (size_t)d.nr * d.n;
  for (long q = c.q0; q < c.q1; ++q) {
    const int j = k + (int)(2L * k * q), jpp = min(j + k, d.nblock);
    for (size_t e = threadIdx.x; e < nrn; e += blockDim.x) a.C[(size_t)jpp * nrn + e] += a.Rbuf[(size_t)j * nrn + e];
  }
}

// ---------------------------------------------------------------------------
// Persistent batch factorization: one launch per class works through the
// (system, level, pair range) items of every level, in level order, with a
// per-system level schedule.  A CTA takes the next item from a counter and
// waits (bounded) until that system's previous level is complete; systems
// advance independently, so a deep system does not hold up shallow ones and
// no level ever waits for the whole batch.  The worker that finishes the last
// item of a (system, level) applies that level's C_jpp updates (the work of
// kb_border_fix) and then publishes the level.  Items are taken in level order,
// so every item an item waits for was taken earlier by a running CTA: the
// waits always end.  A wait that exceeds its limit (about a second) reports
// DEV_TIMEOUT for the system and skips the item's pairs.
// ---------------------------------------------------------------------------
struct BatchQueue {
  int* next;         // next item (zero at launch)
  int* done_pairs;   // per system: pairs finished, cumulative over levels
  int* level_done;   // per system: levels published (border fix-up included)
  long items;
};

// pairs of levels 0..L of a system of nb blocks
__device__ __forceinline__ long pairs_through_level(int nb, int L) {
  long s = 0;
  for (int l = 0; l <= L; ++l) s += pairs_at_level(nb, 1 << l);
  return s;
}

// CTA-wide: the next item; false when the queue is empty
template <typename T>
__device__ bool queue_next(const BatchQueue& qu, const BatchCta* items, const FactorArgs<T>* tab,
                           FactorArgs<T>& a, BatchCta& c, bool& ok) {
  __shared__ long s_it;
  __shared__ int s_ok;
  __syncthreads();  // the previous item's readers of s_it / s_ok are done
  if (threadIdx.x == 0) {
    const long it = atomicAdd(qu.next, 1);
    int good = 1;
    if (it < qu.items) {
      const BatchCta ci = items[it];
      if (ci.pad > 0) {
        const volatile int* flag = qu.level_done + ci.sys;
        unsigned spins = 0;
        while (*flag < ci.pad) {
          if (++spins > (1u << 23)) { good = 0; break; }
          __nanosleep(100);
        }
        __threadfence();
      }
    }
    s_it = it;
    s_ok = good;
  }
  __syncthreads();
  const long it = s_it;
  if (it >= qu.items) return false;
  __threadfence();  // acquire: the system's previous level is visible to every thread
  c = items[it];
  ok = s_ok != 0;
  a = tab[c.sys];
  a.k = 1 << c.pad;
  a.first = c.pad == 0;
  if (!ok && threadIdx.x == 0) report(a.st, DEV_TIMEOUT, -1, 0, a.k);
  return true;
}

// The C_jpp updates of every pair of (system, level): C_jpp += Rbuf[j], four
// elements per thread and round with their loads in flight together
template <typename T>
__device__ void level_fixup(const FactorArgs<T>& a, const BatchCta& c, int tid, int nthr) {
  const Dims d = a.d;
  const int k = 1 << c.pad;
  const size_t nrn = (size_t)d.nr * d.n;
  const long np = pairs_at_level(d.nblock, k);
  const size_t tot = (size_t)np * nrn;
  for (size_t e0 = tid; e0 < tot; e0 += 4 * (size_t)nthr) {
    size_t oc[4];
    T cv[4], rv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t e = e0 + u * (size_t)nthr;
      oc[u] = 0;
      cv[u] = rv[u] = T(0);
      if (e < tot) {
        const long q = (long)(e / nrn);
        const size_t idx = e % nrn;
        const int j = k + (int)(2L * k * q), jpp = min(j + k, d.nblock);
        oc[u] = (size_t)jpp * nrn + idx;
        cv[u] = __ldcg(a.C + oc[u]);
        rv[u] = __ldcg(a.Rbuf + (size_t)j * nrn + idx);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (e0 + u * (size_t)nthr < tot) a.C[oc[u]] = cv[u] + rv[u];
  }
}

// CTA-wide: count the item's pairs; the CTA completing the (system, level)
// applies the level's C_jpp updates and publishes the level
template <typename T>
__device__ void queue_done(const BatchQueue& qu, const FactorArgs<T>& a, const BatchCta& c) {
  __shared__ int s_last;
  __threadfence();  // release: this thread's results of the item
  __syncthreads();  // every pair of the item is finished
  if (threadIdx.x == 0) {
    __threadfence();
    const long cnt = c.q1 - c.q0;
    const int old = atomicAdd(qu.done_pairs + c.sys, (int)cnt);
    s_last = (long)old + cnt == pairs_through_level(a.d.nblock, c.pad);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  level_fixup<T>(a, c, threadIdx.x, blockDim.x);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicExch(qu.level_done + c.sys, c.pad + 1);
  }
}

// The same per warp, for the warp-per-pair families: each warp takes, waits
// for and publishes its own items, so no warp ever waits at a CTA barrier for
// another warp's item.
template <typename T>
__device__ bool queue_next_warp(const BatchQueue& qu, const BatchCta* items, const FactorArgs<T>* tab,
                                FactorArgs<T>& a, BatchCta& c, bool& ok) {
  const int lane = threadIdx.x & 31;
  long it = 0;
  int good = 1;
  if (lane == 0) {
    it = atomicAdd(qu.next, 1);
    if (it < qu.items) {
      const BatchCta ci = items[it];
      if (ci.pad > 0) {
        const volatile int* flag = qu.level_done + ci.sys;
        unsigned spins = 0;
        while (*flag < ci.pad) {
          if (++spins > (1u << 23)) { good = 0; break; }
          __nanosleep(100);
        }
        __threadfence();
      }
    }
  }
  it = __shfl_sync(0xffffffffu, it, 0);
  good = __shfl_sync(0xffffffffu, good, 0);
  if (it >= qu.items) return false;
  __threadfence();
  c = items[it];
  ok = good != 0;
  a = tab[c.sys];
  a.k = 1 << c.pad;
  a.first = c.pad == 0;
  if (!ok && lane == 0) report(a.st, DEV_TIMEOUT, -1, 0, a.k);
  return true;
}

template <typename T>
__device__ void queue_done_warp(const BatchQueue& qu, const FactorArgs<T>& a, const BatchCta& c) {
  const int lane = threadIdx.x & 31;
  __threadfence();
  __syncwarp();
  int last = 0;
  if (lane == 0) {
    const long cnt = c.q1 - c.q0;
    const int old = atomicAdd(qu.done_pairs + c.sys, (int)cnt);
    last = (long)old + cnt == pairs_through_level(a.d.nblock, c.pad);
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return;
  __threadfence();
  level_fixup<T>(a, c, lane, 32);
  __threadfence();
  __syncwarp();
  if (lane == 0) atomicExch(qu.level_done + c.sys, c.pad + 1);
}

template <typename T, int N, int NXM, int NRM>
__global__ void __launch_bounds__(128) kp_factor_rows(const FactorArgs<T>* tab, const BatchCta* items, BatchQueue qu) {
  FactorArgs<T> a;
  BatchCta c;
  bool ok;
  while (queue_next_warp(qu, items, tab, a, c, ok)) {
    if (ok) rows_body<T, N, NXM, NRM, true>(a, c.q0, c.q1, 1);
    queue_done_warp(qu, a, c);
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(2 * N + 32, grp_min_blocks<T, N>())
    kp_factor_grp(const FactorArgs<T>* tab, const BatchCta* items, BatchQueue qu) {
  FactorArgs<T> a;
  BatchCta c;
  bool ok;
  while (queue_next(qu, items, tab, a, c, ok)) {
    if (ok) grp_body<T, N, true>(a, c.q0, c.q1, 1);
    queue_done(qu, a, c);
  }
}

template <int N, typename T = double>
__global__ void __launch_bounds__(128, tc_min_blocks<T>())
    kp_factor_tc(const FactorArgs<T>* tab, const BatchCta* items, BatchQueue qu) {
  using S = TcShape<N, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T* Wt = reinterpret_cast<T*>(smem_raw + (size_t)warp * S::BYTES);
  FactorArgs<T> a;
  BatchCta c;
  bool ok;
  while (queue_next_warp(qu, items, tab, a, c, ok)) {
    const TcTree tr{0, 0, 0};
    if (ok)
      for (long q = c.q0; q < c.q1; ++q)
        tc_pair<N, 8, T>(a, a.k + (int)(2L * a.k * q), a.k, a.first != 0, Wt, lane, tr);
    queue_done_warp(qu, a, c);
  }
}

// F = F0 + sum of the Schur updates, one CTA per system (fixed order)
__global__ void __launch_bounds__(256) kb_reduce_F(const LastDesc* t) {
  const LastDesc& L = t[blockIdx.x];
  const Dims d = L.d;
  const int m = d.nr * d.nx;
  if (m == 0) return;
  const long cnt = d.nblock - 1;
  reduce_tree_body(L.Fbuf, m, 1, cnt, m, cnt > 0 ? cnt : 1, (double*)nullptr, L.F0, d.nr, d.nr, L.Ffin, d.nr, 0);
}

template <typename T>
__global__ void __launch_bounds__(256) kb_last_assemble(const LastDesc* t) {
  const LastDesc& L = t[blockIdx.x];
  last_assemble_range(L.d, static_cast<const T*>(L.Dw), static_cast<const T*>(L.Ew), static_cast<const T*>(L.Bw),
                      static_cast<const T*>(L.Cw), L.H, L.Cq, L.Ffin, L.Hl, (int)threadIdx.x, (int)blockDim.x);
}

__global__ void __launch_bounds__(512) kb_last_factor(const LastDesc* t) {
  const LastDesc& L = t[blockIdx.x];
  if (L.st->code != 0) return;  // a pair of this system already failed
  __syncthreads();
  last_factor_body<double>(L.d, L.lb, L.kind, L.st);
}

// xb += sum of the per-block -C'_j x_j contributions, one CTA per system
__global__ void __launch_bounds__(256) kb_reduce_xb(const LastDesc* t, int nrhs) {
  const LastDesc& L = t[blockIdx.x];
  const Dims d = L.d;
  if (d.nr == 0 || (L.done && *L.done)) return;
  const int m = d.nr * nrhs;
  const long cnt = d.nblock - 1;
  double* xb = L.x + (size_t)(d.nblock + 1) * d.n + d.qr;
  reduce_tree_body(L.XB, m, 1, cnt, m, cnt > 0 ? cnt : 1, (double*)nullptr, (const double*)xb, d.nr, L.ldx, xb,
                   L.ldx, 0);
}

__global__ void __launch_bounds__(256) kb_last_solve(const LastDesc* t, int nrhs) {
  const LastDesc& L = t[blockIdx.x];
  if (L.done && *L.done) return;
  last_solve_body<double>(L.d, L.lb, L.st, L.x, L.ldx, nrhs);
}

// ---------------------------------------------------------------------------
// FP64 residual of the mixed batch path, one CTA per system:
// r = b - A xs with the loaded matrix (add_Mv, cc:2118-2166), written into the
// system's right-hand-side slot, and |r|, |xs|, |b| (and |A|_inf when asked)
// into nrm[1..3] (nrm[0]); the worst |r|/(|A||x|+|b|) of the batch goes to
// *worst (bits of a non-negative double, so an integer max orders them)
// ---------------------------------------------------------------------------
struct ResDesc {
  Dims d;
  const double *D0, *E0, *B0, *C0, *Cq, *F0, *H;
  double* xs;          // the refined solution
  const double* b;
  double *r, *nrm;     // nrm: |A|, |r|, |x|, |b|, |r|/(|A||x|+|b|)
  int* done;
};

__device__ double block_max(double v, double* sv) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) sv[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < nw ? sv[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) sv[0] = v;
  }
  __syncthreads();
  return sv[0];
}

// a batch map with its launch shape: one CTA per entry, or a fixed grid over
// a compacted map whose length (ecnt) the device wrote
struct SweepMap {
  const BatchCta* map;
  const long* ecnt;
  unsigned grid;
};

// r = b - (D_k x_k + E_k x_{k+1} + B_k xb) on block rows [k0, k1) of one
// system, written into the rhs slot; the largest |r| and (with_A) the largest
// row sum of |A| over this thread's rows
__device__ __forceinline__ void res_block_rows(const ResDesc& R, long k0, long k1, int with_A, double& mr,
                                               double& ma) {
  const Dims d = R.d;
  const int n = d.n, nx = d.nx;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx;
  const size_t xb = (size_t)(d.nblock + 1) * n + d.qx;
  const double* xs = R.xs;
  for (long e = k0 * n + threadIdx.x; e < k1 * n; e += blockDim.x) {
    const size_t k = (size_t)(e / n);
    const int i = (int)(e % n);
    const double* Dk = R.D0 + k * nn;
    const double* Ek = R.E0 + k * nn;
    const double* Bk = R.B0 + k * nnx;
    double s = 0.0, sa = 0.0;
    for (int c = 0; c < n; ++c) {
      s = fma(Dk[(size_t)c * n + i], xs[k * n + c], s);
      s = fma(Ek[(size_t)c * n + i], xs[(k + 1) * n + c], s);
      if (with_A) sa += fabs(Dk[(size_t)c * n + i]) + fabs(Ek[(size_t)c * n + i]);
    }
    for (int c = 0; c < nx; ++c) {
      s = fma(Bk[(size_t)c * n + i], xs[xb + c], s);
      if (with_A) sa += fabs(Bk[(size_t)c * n + i]);
    }
    const double r = R.b[e] - s;
    R.r[e] = r;
    mr = fmax(mr, fabs(r));
    ma = fmax(ma, sa);
  }
}

// non-negative doubles order like their bit patterns
__device__ __forceinline__ void atomic_max_nonneg(double* p, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)__double_as_longlong(v));
}

// Block rows covered by the level-1 pairs [q0, q1) of each map entry
// (rows 2 q0 .. 2 q1 - 1), spread over many CTAs: the full sweep map on the
// first residual of a solve, the compacted map of the systems just corrected
// afterwards (ecnt: its length).  The largest |r| and |A| row sum of each
// entry go to nrm[5], nrm[6] of its system.
__global__ void __launch_bounds__(128) kb_residual_rows(const ResDesc* t, const BatchCta* map, const long* ecnt,
                                                        int with_A) {
  __shared__ double sv[32];
  const long cnt = ecnt ? *ecnt : (long)gridDim.x;
  for (long e = blockIdx.x; e < cnt; e += gridDim.x) {
    const BatchCta c = map[e];
    const ResDesc& R = t[c.sys];
    if (*R.done) continue;  // uniform over the CTA
    double mr = 0.0, ma = 0.0;
    res_block_rows(R, 2 * c.q0, 2 * c.q1, with_A, mr, ma);
    mr = block_max(mr, sv);
    ma = block_max(ma, sv);
    if (threadIdx.x == 0) {
      atomic_max_nonneg(R.nrm + 5, mr);
      if (with_A) atomic_max_nonneg(R.nrm + 6, ma);
    }
  }
}

// The rest of the residual, one CTA per system still refining: block rows
// from 2 * (level-1 pairs) on (the odd tail; every row when nblock = 1), the
// boundary rows (H), the border rows (a CTA-wide sum over every block
// column), |x| and |b|; then the norms with kb_residual_rows' maxima,
// |r|/(|A||x|+|b|), the converged flag and the batch-worst figure (bits of a
// non-negative double, so an integer max orders them).  Bit for bit the
// residual of add_Mv (cc:2118-2166) on the loaded FP64 matrix.
__global__ void __launch_bounds__(256, 2) kb_residual(const ResDesc* t, int with_A, double tol,
                                                   unsigned long long* worst) {
  __shared__ double sv[32];
  const ResDesc& R = t[blockIdx.x];
  if (*R.done) {  // converged earlier: its last figure still counts for the batch
    if (threadIdx.x == 0) atomicMax(worst, (unsigned long long)__double_as_longlong(R.nrm[4]));
    return;
  }
  const Dims d = R.d;
  const int n = d.n, nb = d.nblock, nr = d.nr, nx = d.nx, qx = d.qx, m = n + d.qr, Nc = d.Nc;
  const int tid = threadIdx.x, bs = blockDim.x;
  const size_t nrn = (size_t)nr * n;
  const size_t xN = (size_t)nb * n, xq = (size_t)(nb + 1) * n, xb = xq + qx;
  const double* xs = R.xs;
  double mr = 0.0, ma = 0.0;
  res_block_rows(R, 2 * pairs_at_level(nb, 1), nb, with_A, mr, ma);
  // boundary rows (H)
  for (int row = tid; row < m; row += bs) {
    double s = 0.0, sa = 0.0;
    for (int c = 0; c < Nc; ++c) {
      const size_t xi = c < n ? (size_t)c : (c < 2 * n ? xN + (c - n) : xq + (c - 2 * n));
      const double h = R.H[(size_t)c * m + row];
      s = fma(h, xs[xi], s);
      sa += fabs(h);
    }
    const size_t o = xN + row;
    const double r = R.b[o] - s;
    R.r[o] = r;
    mr = fmax(mr, fabs(r));
    ma = fmax(ma, with_A ? sa : 0.0);
  }
  // border rows, four at a time: one walk over every block column
  // accumulates four rows, each row's terms in the same order as a walk of
  // its own; then one CTA reduction per row.  A thread's columns e = tid,
  // tid + bs, ... are loaded RES_U at a time before any is added, so a lone
  // long system (the late refinement passes) pays one load latency per RES_U
  // columns; the additions keep the column order.
  constexpr int RES_U = 4;
  const long tot = (long)(nb + 1) * n;
  const long dk = bs / n;
  const int dc = bs % n;
  for (int r0 = 0; r0 < nr; r0 += 4) {
    double s4[4] = {0.0, 0.0, 0.0, 0.0}, a4[4] = {0.0, 0.0, 0.0, 0.0};
    size_t k = (size_t)(tid / n);  // block and column of element e
    int c = tid % n;
    for (long e0 = tid; e0 < tot; e0 += (long)RES_U * bs) {
      double xv[RES_U], cv[RES_U][4];
#pragma unroll
      for (int u = 0; u < RES_U; ++u) {
        const bool on = e0 + (long)u * bs < tot;
        const double* cp = R.C0 + k * nrn + (size_t)c * nr + r0;
        xv[u] = on ? xs[k * n + c] : 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i) cv[u][i] = (on && r0 + i < nr) ? cp[i] : 0.0;
        k += dk;
        c += dc;
        if (c >= n) { c -= n; ++k; }
      }
#pragma unroll
      for (int u = 0; u < RES_U; ++u) {
        if (e0 + (long)u * bs >= tot) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (r0 + i < nr) {
            s4[i] = fma(cv[u][i], xv[u], s4[i]);
            a4[i] += fabs(cv[u][i]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = r0 + i;
      if (rr >= nr) break;
      double s = s4[i], sa = a4[i];
      for (int c = tid; c < qx; c += bs) { s = fma(R.Cq[(size_t)c * nr + rr], xs[xq + c], s); sa += fabs(R.Cq[(size_t)c * nr + rr]); }
      for (int c = tid; c < nx; c += bs) { s = fma(R.F0[(size_t)c * nr + rr], xs[xb + c], s); sa += fabs(R.F0[(size_t)c * nr + rr]); }
      s = block_sum(s, sv);
      sa = block_sum(sa, sv);
      if (tid == 0) {
        const size_t o = xN + m + rr;
        const double r = R.b[o] - s;
        R.r[o] = r;
        mr = fmax(mr, fabs(r));
        ma = fmax(ma, with_A ? sa : 0.0);
      }
    }
  }
  const long nrows = (long)n * (nb + 1) + d.qr + nr;
  const long ncols = (long)n * (nb + 1) + qx + nx;
  // |x| and |b|: maxima are exact in any order, so eight loads per round
  double mx = 0.0, mb = 0.0;
  for (long e0 = tid; e0 < ncols; e0 += 8L * bs) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = e0 + (long)u * bs < ncols ? fabs(xs[e0 + (long)u * bs]) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) mx = fmax(mx, v[u]);
  }
  for (long e0 = tid; e0 < nrows; e0 += 8L * bs) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = e0 + (long)u * bs < nrows ? fabs(R.b[e0 + (long)u * bs]) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) mb = fmax(mb, v[u]);
  }
  mr = block_max(mr, sv);
  mx = block_max(mx, sv);
  mb = block_max(mb, sv);
  if (with_A) ma = block_max(ma, sv);
  if (tid == 0) {
    mr = fmax(mr, R.nrm[5]);  // the block rows of kb_residual_rows
    if (with_A) R.nrm[0] = fmax(ma, R.nrm[6]);
    R.nrm[5] = 0.0;           // ready for the next residual
    R.nrm[6] = 0.0;
    R.nrm[1] = mr;
    R.nrm[2] = mx;
    R.nrm[3] = mb;
    const double den = R.nrm[0] * mx + mb;
    double rel = den > 0.0 ? mr / den : (mr > 0.0 ? INFINITY : 0.0);
    if (rel != rel) rel = INFINITY;
    R.nrm[4] = rel;
    if (rel <= tol) *R.done = 1;
    atomicMax(worst, (unsigned long long)__double_as_longlong(rel));
  }
}

// x_sol += d for the systems still refining (d was solved in place of r):
// the x blocks of each map entry's level-1 pairs (2 q0 .. 2 q1 - 1) ...
__global__ void __launch_bounds__(128) kb_correct_rows(const ResDesc* t, const BatchCta* map, const long* ecnt) {
  const long cnt = ecnt ? *ecnt : (long)gridDim.x;
  for (long e = blockIdx.x; e < cnt; e += gridDim.x) {
    const BatchCta c = map[e];
    const ResDesc& R = t[c.sys];
    if (*R.done) continue;
    const long n = R.d.n;
    for (long i = 2 * c.q0 * n + threadIdx.x; i < 2 * c.q1 * n; i += blockDim.x) R.xs[i] += R.r[i];
  }
}

// ... and the rest of x, one CTA per system
__global__ void __launch_bounds__(256) kb_correct(const ResDesc* t) {
  const ResDesc& R = t[blockIdx.x];
  if (*R.done) return;
  const Dims d = R.d;
  const long ncols = (long)d.n * (d.nblock + 1) + d.qx + d.nx;
  for (long i = 2 * pairs_at_level(d.nblock, 1) * d.n + threadIdx.x; i < ncols; i += blockDim.x)
    R.xs[i] += R.r[i];
}

// the level-1 entries of the sweep map: all of them, or the compacted ones
static SweepMap level1_map(const BatchClass& c, bool compact) {
  if (!compact) return {c.smap, nullptr, (unsigned)c.scnt[0]};
  return {c.cmap, c.ccnt, (unsigned)std::min<long>(c.scnt[0], COMPACT_GRID)};
}

void batch_residual(BatchClass& c, int with_A, double tol, unsigned long long* worst, cudaStream_t st,
                    bool compact) {
  if (c.nsys == 0) return;
  compact = compact && c.cmap != nullptr;
  if (c.levels > 0 && c.scnt[0] > 0) {
    const SweepMap m = level1_map(c, compact);
    kb_residual_rows<<<m.grid, 128, 0, st>>>(static_cast<const ResDesc*>(c.rd), m.map, m.ecnt, with_A);
    check_launch("kb_residual_rows");
  }
  kb_residual<<<c.nsys, 256, 0, st>>>(static_cast<const ResDesc*>(c.rd), with_A, tol, worst);
  check_launch("kb_residual");
}

void batch_correct(BatchClass& c, cudaStream_t st) {
  if (c.nsys == 0) return;
  const bool compact = c.cmap != nullptr;
  if (c.levels > 0 && c.scnt[0] > 0) {
    const SweepMap m = level1_map(c, compact);
    kb_correct_rows<<<m.grid, 128, 0, st>>>(static_cast<const ResDesc*>(c.rd), m.map, m.ecnt);
    check_launch("kb_correct_rows");
  }
  kb_correct<<<c.nsys, 256, 0, st>>>(static_cast<const ResDesc*>(c.rd));
  check_launch("kb_correct");
}

bool batch_family_ok(int fam, const Dims& d, bool mixed) {
  if (d.nr > 8 || d.nx > 8) return false;
  switch (fam) {
    case PAIR_TC: return d.n == 8 || d.n == 16;
    case PAIR_GRP: return d.n == 16 || d.n == 32;
    case PAIR_ROWS: return d.n <= 16 && d.nr <= 4 && d.nx <= 4;
    default: return false;
  }
}

static void build_map(const std::vector<DevState>& sys, int levels, int chunk, std::vector<BatchCta>& map,
                      std::vector<long>& off, std::vector<long>& cnt) {
  off.assign(levels, 0);
  cnt.assign(levels, 0);
  // within a level the deepest systems come first: their chains of levels are
  // the longest, so the persistent launch starts them first
  std::vector<size_t> order(sys.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(),
                   [&](size_t x, size_t y) { return sys[x].d.nblock > sys[y].d.nblock; });
  for (int L = 0; L < levels; ++L) {
    const int k = 1 << L;
    off[L] = (long)map.size();
    for (size_t i : order) {
      const long np = pairs_at_level(sys[i].d.nblock, k);
      for (long q0 = 0; q0 < np; q0 += chunk) {
        BatchCta c;
        c.sys = (int)i;
        c.pad = L;  // the level (the persistent launch reads it)
        c.q0 = q0;
        c.q1 = q0 + chunk < np ? q0 + chunk : np;
        map.push_back(c);
      }
    }
    cnt[L] = (long)map.size() - off[L];
  }
}

template <typename X>
static int upload_table(void*& dst, const std::vector<X>& v) {
  if (cudaMalloc(&dst, std::max<size_t>(v.size(), 1) * sizeof(X)) != cudaSuccess) return 1;
  if (!v.empty() && cudaMemcpy(dst, v.data(), v.size() * sizeof(X), cudaMemcpyHostToDevice) != cudaSuccess) return 1;
  return 0;
}

void batch_free(BatchClass& c) {
  if (c.qbuf) cudaFree(c.qbuf);
  c.qbuf = nullptr;
  for (void** p : {&c.fa, &c.sf, &c.sb, &c.ld, &c.rd})
    if (*p) { cudaFree(*p); *p = nullptr; }
  if (c.fmap) { cudaFree(c.fmap); c.fmap = nullptr; }
  if (c.smap) { cudaFree(c.smap); c.smap = nullptr; }
  if (c.cmap) { cudaFree(c.cmap); c.cmap = nullptr; }
  if (c.ccnt) { cudaFree(c.ccnt); c.ccnt = nullptr; }
  c.foff.clear(); c.fcnt.clear(); c.soff.clear(); c.scnt.clear();
}

template <typename T>
static int batch_build_t(BatchClass& c, const std::vector<DevState>& sys, int nrhs) {
  c.nsys = (int)sys.size();
  c.nrhs = nrhs;
  c.levels = 0;
  c.nrm = c.nxm = 0;
  size_t lmax = 0;
  std::vector<FactorArgs<T>> fa(sys.size());
  std::vector<SweepArgs<T>> sf(sys.size()), sb(sys.size());
  std::vector<LastDesc> ld(sys.size());
  std::vector<ResDesc> rd(sys.size());
  T* tag = nullptr;
  for (size_t i = 0; i < sys.size(); ++i) {
    DevState s = sys[i];
    const Dims d = s.d;
    const WorkSet<T> w = work_set(s, tag);
    c.n = d.n;
    c.nrm = std::max(c.nrm, d.nr);
    c.nxm = std::max(c.nxm, d.nx);
    int K = 1, lev = 0;
    while (K < d.nblock) { K *= 2; ++lev; }
    c.levels = std::max(c.levels, lev);
    lmax = std::max<size_t>(lmax, (size_t)std::max(d.Nr, d.Nc));
    FactorArgs<T> a{};
    a.d = d;
    a.D0 = s.D0; a.E0 = s.E0; a.B0 = s.B0; a.C0 = s.C0;
    a.D = w.D; a.E = w.E; a.B = w.B; a.C = w.C; a.Tm = w.Tm; a.P = s.P;
    a.Rbuf = w.Rbuf; a.Fbuf = s.Fbuf; a.st = s.st;
    a.ldw = odd_ld(2 * d.n + d.nr);
    a.x = nullptr; a.ldx = 0; a.nrf = 0; a.XB = s.XB;
    fa[i] = a;
    SweepArgs<T> sw{};
    sw.d = d;
    sw.D = w.D; sw.E = w.E; sw.B = w.B; sw.C = w.C; sw.Tm = w.Tm; sw.P = s.P;
    sw.x = s.bx; sw.ldx = s.bldx; sw.nrhs = nrhs; sw.XB = s.XB; sw.sel = SEL_LU;
    sw.done = s.bdone;
    sw.ldw = odd_ld(2 * d.n);
    sf[i] = sw;
    sw.ldw = d.n;
    sb[i] = sw;
    LastDesc l{};
    l.d = d;
    l.D0 = s.D0; l.E0 = s.E0; l.B0 = s.B0; l.C0 = s.C0; l.H = s.H; l.Cq = s.Cq; l.F0 = s.F0;
    l.Fbuf = s.Fbuf; l.XB = s.XB;
    l.Dw = w.D; l.Ew = w.E; l.Bw = w.B; l.Cw = w.C;
    l.Ffin = s.Ffin; l.Hl = s.Hl; l.tau = s.tau_l; l.x = s.bx;
    l.piv = s.piv_l; l.kind = s.sel_last; l.ldx = s.bldx; l.st = s.st;
    l.lb = last_bufs(s);
    l.done = s.bdone;
    ld[i] = l;
    ResDesc r{};
    r.d = d;
    r.D0 = s.D0; r.E0 = s.E0; r.B0 = s.B0; r.C0 = s.C0; r.Cq = s.Cq; r.F0 = s.F0; r.H = s.H;
    r.xs = s.bsol; r.b = s.bb; r.r = s.bx; r.nrm = s.bnrm; r.done = s.bdone;
    rd[i] = r;
  }
  c.last_smem = 2 * lmax * 8;
  std::vector<BatchCta> fmap, smap;
  build_map(sys, c.levels, c.chunk, fmap, c.foff, c.fcnt);
  build_map(sys, c.levels, 8, smap, c.soff, c.scnt);
  int bad = upload_table(c.fa, fa) | upload_table(c.sf, sf) | upload_table(c.sb, sb) | upload_table(c.ld, ld) |
            upload_table(c.rd, rd);
  void* m1 = nullptr;
  void* m2 = nullptr;
  bad |= upload_table(m1, fmap) | upload_table(m2, smap);
  c.fmap = static_cast<BatchCta*>(m1);
  c.smap = static_cast<BatchCta*>(m2);
  c.items = (long)fmap.size();
  if (cudaMalloc(&c.qbuf, (1 + 2 * (size_t)c.nsys) * sizeof(int)) != cudaSuccess) bad = 1;
  if (c.mixed && c.levels > 0) {  // compacted maps of the refinement passes
    if (cudaMalloc(&c.cmap, std::max<size_t>(smap.size(), 1) * sizeof(BatchCta)) != cudaSuccess) bad = 1;
    if (cudaMalloc(&c.ccnt, (size_t)c.levels * sizeof(long)) != cudaSuccess) bad = 1;
  }
  return bad;
}

int batch_build(BatchClass& c, const std::vector<DevState>& sys, int nrhs) {
  batch_free(c);
  return c.mixed ? batch_build_t<float>(c, sys, nrhs) : batch_build_t<double>(c, sys, nrhs);
}

// one batched launch of the class's pair kernel at level `L`
template <typename T>
static void batch_pairs(BatchClass& c, int L, cudaStream_t st) {
  const long cnt = c.fcnt[L];
  if (cnt == 0) return;
  FactorArgs<T> a0{};
  a0.k = 1 << L;
  a0.first = L == 0;
  const FactorArgs<T>* tab = static_cast<const FactorArgs<T>*>(c.fa);
  const BatchCta* map = c.fmap + c.foff[L];
  const unsigned g = (unsigned)cnt;
  if (c.fam == PAIR_TC) {
    const size_t sm = tc_smem_per_warp_t<T>(c.n) * 4;
    if (c.n == 16) {
      smem_limit_once(k_factor_lu_tc<16, true, false, 8, T>, sm);
      k_factor_lu_tc<16, true, false, 8, T><<<g, 128, sm, st>>>(a0, tab, map);
    } else {
      smem_limit_once(k_factor_lu_tc<8, true, false, 8, T>, sm);
      k_factor_lu_tc<8, true, false, 8, T><<<g, 128, sm, st>>>(a0, tab, map);
    }
    check_launch("batched pair kernel");
  }
  if (c.fam == PAIR_GRP) {
    if (c.n == 32) {
      smem_limit_once(k_factor_lu_grp<T, 32, true>, GrpShape<T, 32>::BYTES);
      k_factor_lu_grp<T, 32, true><<<g, 96, GrpShape<T, 32>::BYTES, st>>>(a0, tab, map);
    } else {
      smem_limit_once(k_factor_lu_grp<T, 16, true>, GrpShape<T, 16>::BYTES);
      k_factor_lu_grp<T, 16, true><<<g, 64, GrpShape<T, 16>::BYTES, st>>>(a0, tab, map);
    }
  } else if (c.fam == PAIR_ROWS) {
    if (c.n <= 4) k_factor_lu_rows<T, 4, 4, 4, true><<<g, 128, 0, st>>>(a0, tab, map);
    else if (c.n <= 8) k_factor_lu_rows<T, 8, 4, 4, true><<<g, 128, 0, st>>>(a0, tab, map);
    else k_factor_lu_rows<T, 16, 4, 4, true><<<g, 128, 0, st>>>(a0, tab, map);
  }
  check_launch("batched pair kernel");
  if (c.nrm > 0) {
    kb_border_fix<T><<<g, 128, 0, st>>>(tab, map, 1 << L);
    check_launch("kb_border_fix");
  }
}

// every level of every system of the class in one persistent launch
template <typename T>
static void batch_pairs_persistent(BatchClass& c, cudaStream_t st) {
  if (c.items == 0) return;
  cudaMemsetAsync(c.qbuf, 0, (1 + 2 * (size_t)c.nsys) * sizeof(int), st);
  BatchQueue qu{c.qbuf, c.qbuf + 1, c.qbuf + 1 + c.nsys, c.items};
  const FactorArgs<T>* tab = static_cast<const FactorArgs<T>*>(c.fa);
  auto grid = [&](auto* kern, int threads, size_t smem) {
    return grid_for(c.items, 1, 148 * resident_ctas(kern, threads, smem));
  };
  if (c.fam == PAIR_TC) {
    const size_t sm = tc_smem_per_warp_t<T>(c.n) * 4;
    if (c.n == 16) {
      smem_limit_once(kp_factor_tc<16, T>, sm);
      kp_factor_tc<16, T><<<grid(kp_factor_tc<16, T>, 128, sm), 128, sm, st>>>(tab, c.fmap, qu);
    } else {
      smem_limit_once(kp_factor_tc<8, T>, sm);
      kp_factor_tc<8, T><<<grid(kp_factor_tc<8, T>, 128, sm), 128, sm, st>>>(tab, c.fmap, qu);
    }
    check_launch("kp_factor_tc");
    return;
  }
  if (c.fam == PAIR_GRP) {
    if (c.n == 32) {
      auto* kern = kp_factor_grp<T, 32>;
      smem_limit_once(kern, GrpShape<T, 32>::BYTES);
      kern<<<grid(kern, 96, GrpShape<T, 32>::BYTES), 96, GrpShape<T, 32>::BYTES, st>>>(tab, c.fmap, qu);
    } else {
      auto* kern = kp_factor_grp<T, 16>;
      smem_limit_once(kern, GrpShape<T, 16>::BYTES);
      kern<<<grid(kern, 64, GrpShape<T, 16>::BYTES), 64, GrpShape<T, 16>::BYTES, st>>>(tab, c.fmap, qu);
    }
  } else if (c.fam == PAIR_ROWS) {
    auto* kern = c.n <= 4 ? kp_factor_rows<T, 4, 4, 4> : c.n <= 8 ? kp_factor_rows<T, 8, 4, 4>
                                                                   : kp_factor_rows<T, 16, 4, 4>;
    kern<<<grid(kern, 128, 0), 128, 0, st>>>(tab, c.fmap, qu);
  }
  check_launch("persistent batched pair kernel");
}

template <typename T>
static void batch_factorize_t(BatchClass& c, cudaStream_t st) {
  const LastDesc* ld = static_cast<const LastDesc*>(c.ld);
  kb_begin<T><<<c.nsys, 256, 0, st>>>(ld);
  check_launch("kb_begin");
  if (c.persist) {
    batch_pairs_persistent<T>(c, st);
  } else {
    for (int L = 0; L < c.levels; ++L) batch_pairs<T>(c, L, st);
  }
  kb_reduce_F<<<c.nsys, 256, 0, st>>>(ld);
  kb_last_assemble<T><<<c.nsys, 256, 0, st>>>(ld);
  kb_last_factor<<<c.nsys, 512, 0, st>>>(ld);
  check_launch("batched last block");
}

void batch_factorize(BatchClass& c, cudaStream_t st) {
  if (c.nsys == 0) return;
  c.op = c.fam == PAIR_TC || c.fam == PAIR_GRP ? c.n : 0;
  if (c.mixed) batch_factorize_t<float>(c, st);
  else batch_factorize_t<double>(c, st);
}

// the sweep map of level L: the full map (one CTA per entry), or on the
// refinement passes the compacted map of the systems still refining, walked by
// a fixed grid (the launch is captured before the length is known)
static SweepMap sweep_map(const BatchClass& c, int L, bool compact) {
  if (!compact) return {c.smap + c.soff[L], nullptr, (unsigned)c.scnt[L]};
  return {c.cmap + c.soff[L], c.ccnt + L, (unsigned)std::min<long>(c.scnt[L], COMPACT_GRID)};
}

template <typename T, int N>
static void batch_sweeps_rows(BatchClass& c, cudaStream_t st, bool forward, int L, const SweepMap& m) {
  const bool r4 = c.nrm <= 4, x4 = c.nxm <= 4;
  SweepArgs<T> a0{};
  a0.k = 1 << L;
  a0.op = c.op;
  if constexpr (N == 8 || N == 16) {
    if (c.n == N) {  // pipelined: a fixed grid walks the level's map entries
      const long nent = c.scnt[L];
      const unsigned g = (unsigned)std::min<long>(nent, 148 * 2);
      if (forward) {
        const SweepArgs<T>* tab = static_cast<const SweepArgs<T>*>(c.sf);
        auto* kern = r4 ? k_forward_pipe<N, 4, T, true> : k_forward_pipe<N, 8, T, true>;
        const size_t sm = 8 * (r4 ? FwdBuf<N, 4, T>::BYTES : FwdBuf<N, 8, T>::BYTES);
        smem_limit_once(kern, sm);
        kern<<<g, 256, sm, st>>>(a0, tab, m.map, m.ecnt, nent);
      } else {
        const SweepArgs<T>* tab = static_cast<const SweepArgs<T>*>(c.sb);
        auto* kern = x4 ? k_backward_pipe<N, 4, T, true> : k_backward_pipe<N, 8, T, true>;
        const size_t sm = 8 * (x4 ? BwdBuf<N, 4, T>::BYTES : BwdBuf<N, 8, T>::BYTES);
        smem_limit_once(kern, sm);
        kern<<<g, 256, sm, st>>>(a0, tab, m.map, m.ecnt, nent);
      }
      return;
    }
  }
  if (forward) {
    const SweepArgs<T>* tab = static_cast<const SweepArgs<T>*>(c.sf);
    if (r4) k_forward_rows<T, N, 4, true, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
    else k_forward_rows<T, N, 8, true, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
  } else {
    const SweepArgs<T>* tab = static_cast<const SweepArgs<T>*>(c.sb);
    if (x4) k_backward_rows<T, N, 4, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
    else k_backward_rows<T, N, 8, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
  }
}

template <typename T>
static void batch_sweep_level(BatchClass& c, cudaStream_t st, bool forward, int L, bool compact) {
  if (c.scnt[L] == 0) return;
  const SweepMap m = sweep_map(c, L, compact);
  if (c.n <= 4) batch_sweeps_rows<T, 4>(c, st, forward, L, m);
  else if (c.n <= 8) batch_sweeps_rows<T, 8>(c, st, forward, L, m);
  else if (c.n <= 16) batch_sweeps_rows<T, 16>(c, st, forward, L, m);
  else if (c.n == 32) {
    SweepArgs<T> a0{};
    a0.k = 1 << L;
    if (forward) {
      const SweepArgs<T>* tab = static_cast<const SweepArgs<T>*>(c.sf);
      if (c.nrm <= 4) k_forward_rows32<T, 4, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
      else k_forward_rows32<T, 8, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
    } else {
      const SweepArgs<T>* tab = static_cast<const SweepArgs<T>*>(c.sb);
      if (c.nxm <= 4) k_backward_rows32<T, 4, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
      else k_backward_rows32<T, 8, true><<<m.grid, 256, 0, st>>>(a0, tab, m.map, m.ecnt);
    }
  } else {
    SweepArgs<T> a0{};
    a0.k = 1 << L;
    if (forward) {
      const size_t sm = (size_t)odd_ld(2 * c.n) * c.nrhs * 8 * WARPS_PANEL;
      smem_limit_once(k_forward_level<T, true>, sm);
      k_forward_level<T, true><<<m.grid, WARPS_PANEL * 32, sm, st>>>(a0, static_cast<const SweepArgs<T>*>(c.sf),
                                                                     m.map, m.ecnt);
    } else {
      const size_t sm = (size_t)c.n * 8 * WARPS_PANEL;
      k_backward_level<T, true><<<m.grid, WARPS_PANEL * 32, sm, st>>>(a0, static_cast<const SweepArgs<T>*>(c.sb),
                                                                      m.map, m.ecnt);
    }
  }
  check_launch(forward ? "batched forward sweep" : "batched backward sweep");
}

template <typename T>
static void batch_solve_t(BatchClass& c, cudaStream_t st, bool compact) {
  const LastDesc* ld = static_cast<const LastDesc*>(c.ld);
  for (int L = 0; L < c.levels; ++L) batch_sweep_level<T>(c, st, true, L, compact);
  kb_reduce_xb<<<c.nsys, 256, 0, st>>>(ld, c.nrhs);
  smem_limit_once(kb_last_solve, c.last_smem, LAST_SOLVE_UNASKED);
  kb_last_solve<<<c.nsys, 256, c.last_smem, st>>>(ld, c.nrhs);
  for (int L = c.levels - 1; L >= 0; --L) batch_sweep_level<T>(c, st, false, L, compact);
  check_launch("batched solve");
}

void batch_solve(BatchClass& c, cudaStream_t st, bool compact) {
  if (c.nsys == 0) return;
  compact = compact && c.cmap != nullptr;
  if (c.mixed) batch_solve_t<float>(c, st, compact);
  else batch_solve_t<double>(c, st, compact);
}

// Compacted sweep maps of the systems still refining: entry e of the full map
// is kept when its system has not converged, at a free position of its level
// (one atomic per warp and level; the pairs of a level are independent, so
// the order within a level does not change any result)
struct LevelOffsets {
  long off[32];
};

__global__ void __launch_bounds__(256) kb_compact_map(const LastDesc* ld, const BatchCta* smap, long nent,
                                                      LevelOffsets lo, BatchCta* cmap, long* ccnt) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  BatchCta c{};
  bool keep = false;
  if (e < nent) {
    c = smap[e];
    const int* dn = ld[c.sys].done;
    keep = !(dn && *dn);
  }
  const unsigned act = __ballot_sync(0xffffffffu, keep);
  if (!keep) return;
  const int L = c.pad;  // the entry's level
  const unsigned grp = __match_any_sync(act, L);
  const int leader = __ffs(grp) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(reinterpret_cast<unsigned long long*>(ccnt + L), (unsigned long long)__popc(grp));
  base = __shfl_sync(grp, base, leader);
  const long pos = (long)base + __popc(grp & ((1u << lane) - 1u));
  cmap[lo.off[L] + pos] = c;
}

void batch_compact(BatchClass& c, cudaStream_t st) {
  if (c.nsys == 0 || !c.cmap || c.levels == 0) return;
  const long nent = c.soff[c.levels - 1] + c.scnt[c.levels - 1];
  LevelOffsets lo{};
  for (int L = 0; L < c.levels; ++L) lo.off[L] = c.soff[L];
  cudaMemsetAsync(c.ccnt, 0, sizeof(long) * c.levels, st);
  if (nent > 0)
    kb_compact_map<<<(unsigned)((nent + 255) / 256), 256, 0, st>>>(static_cast<const LastDesc*>(c.ld), c.smap, nent,
                                                                    lo, c.cmap, c.ccnt);
  check_launch("kb_compact_map");
}

}  // namespace bcr
