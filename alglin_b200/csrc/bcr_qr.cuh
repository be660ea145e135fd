// QR / QRP pair kernel for n <= 16, nr <= 8, n + nx <= 32: one warp per pair,
// lane = column of the work matrix, its 2n <= 32 rows in registers; included by
// bcr_kernels.cu.
//
// Step i: the lane that holds column i posts the column in shared memory, every
// lane forms its product with it (for the posting lane that is the norm), and the
// Householder scalars (dlarfg's, from the product and the diagonal element) are
// the same arithmetic in every lane, so the reflector is applied without another
// exchange:
//   d = sum_{r>i} x_r a_r,  w = t (a_i + sc d),  a_i -= w,  a_r -= (w sc) x_r.
// The nr border rows of a column are eliminated with the finished row of R.
// The registers rotate by one row per step, so that one rolled loop covers all
// steps (row i of R leaves through shared memory; after n steps the registers
// hold the reduced rows).  Columns beyond the first pass's (the panel and x_jp,
// or all of them when they fit in a warp) replay the reflectors in a second pass.
// Bound by the FP64 pipe and the posting's latency; the shared-memory kernel this
// replaces walked the whole work matrix there, one lane per column with every
// element loaded and stored at each step: a lone pair at n = 16 took 62 us and
// takes 30, level 1 of 20,011 blocks 444 and 229 us (the scales of the columns took
// 2% of that back).  For which orders and levels it is the faster one:
// qr_warp_faster.
#pragma once

template <typename T>
struct QrShape {
  static constexpr int ROWS = 32, NS = 10;  // scalars of a step: t, sc, then the border multipliers
  static constexpr int V = 16 * ROWS, SC = 16 * NS, S = ROWS * 33;
  static constexpr size_t BYTES = (size_t)(V + SC + S) * sizeof(T) + 16;  // + the column map
};

__device__ __forceinline__ double qr_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float qr_sqrt(float x) { return sqrtf(x); }

// Exponents of the columns.  The products x_r a_r are of the elements as they are,
// without the reflector's scale, so a column whose largest element is not within
// 2^+-MOST is divided by a power of two first (exactly; QR commutes with it, and
// the column's results are multiplied again): the products of two columns then
// stay in the range, wherever in it the columns lie.
__device__ __forceinline__ unsigned qr_key(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned qr_key(float v) { return __float_as_uint(v) & 0x7fffffffu; }
template <typename T>
struct QrRange {
  static constexpr bool F64 = sizeof(T) == 8;
  static constexpr int MANT = F64 ? 20 : 23, BIAS = F64 ? 1023 : 127, MOST = F64 ? 250 : 30, CLAMP = F64 ? 1000 : 120;
};
__device__ __forceinline__ void qr_pow2(int e, double& p) { p = __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ void qr_pow2(int e, float& p) { p = __int_as_float((127 + e) << 23); }

template <typename T, bool PIVOT>
__device__ __forceinline__ void qr_pair(const FactorArgs<T>& a, int j, T* Vs, int lane) {
  using Q = QrShape<T>;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int RW = Q::ROWS, NS = Q::NS, NRM = 8;
  T* Sc = Vs + Q::V;
  T* S = Sc + Q::SC;
  unsigned char* cmap = reinterpret_cast<unsigned char*>(S + Q::S);
  const Dims d = a.d;
  const int n = d.n, nr = d.nr, nx = d.nx, n2 = 2 * n, NC = 3 * n + nx, k = a.k, jp = j - k;
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  const size_t oj = (size_t)j * nn, ojp = (size_t)jp * nn;
  const bool first = a.first != 0;
  const int W0 = NC <= 32 ? NC : n2;  // columns of the first pass
  const int hr = lane & 15, hc = lane >> 4;
  const bool rok = hr < n;
  int info = 0, cpos = lane;
  auto src = [&](const double* orig, const T* work, size_t i) -> T { return ldsrc(first, orig, work, i); };
  for (int c0 = 0; c0 < NC; c0 += c0 == 0 ? W0 : 32) {
    const int nc = c0 == 0 ? W0 : NC - c0;  // columns of this pass (n + nx <= 32 in the second)
    __syncwarp();
    // stage the pass's columns (half a warp per column, every load in flight
    // before the first store), then one column per lane
    const int c = c0 + lane;
    const bool live = lane < nc, panel = live && c < n;
    T cb[NRM];
    auto load = [&](const auto* D, const auto* E, const auto* B, const auto* C) {
      T vt[16], vb[16];
#pragma unroll
      for (int it = 0; it < 16; ++it) {
        const int cc = 2 * it + hc, cg = c0 + cc;
        const bool in = rok && cc < nc;
        const size_t o = (size_t)(cg < n ? cg : cg < n2 ? cg - n : cg < 3 * n ? cg - n2 : cg - 3 * n) * n + hr;
        const auto* pt = cg < n ? E + ojp : cg < n2 ? D + ojp : B + (size_t)jp * nnx;
        const auto* pb = cg < n ? D + oj : cg < 3 * n ? E + oj : B + (size_t)j * nnx;
        vt[it] = T(ld_batch(in && (cg < n2 || cg >= 3 * n), pt + o));
        vb[it] = T(ld_batch(in && (cg < n || cg >= n2), pb + o));
      }
#pragma unroll
      for (int r = 0; r < NRM; ++r) cb[r] = T(ld_batch(panel && r < nr, C + (size_t)j * nrn + (size_t)c * nr + r));
#pragma unroll
      for (int it = 0; it < 16; ++it)
        if (rok) {
          S[hr * 33 + 2 * it + hc] = vt[it];
          S[(n + hr) * 33 + 2 * it + hc] = vb[it];
        }
    };
    if (first) load(a.D0, a.E0, a.B0, a.C0);
    else load(a.D, a.E, a.B, a.C);
    __syncwarp();
    T v[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) v[r] = live && r < n2 ? S[r * 33 + lane] : T(0);
    __syncwarp();
    T un = T(1);  // this lane's column was divided by un
    {
      using Rg = QrRange<T>;
      unsigned key = 0u;
#pragma unroll
      for (int r = 0; r < RW; ++r) key = max(key, qr_key(v[r]));
      const int ex = (int)(key >> Rg::MANT) - Rg::BIAS;
      const bool out = key != 0u && ex <= Rg::BIAS && (ex > Rg::MOST || ex < -Rg::MOST);
      if (__any_sync(FULL, out)) {
        const int e = out ? min(max(ex, -Rg::CLAMP), Rg::CLAMP) : 0;
        T sc;
        qr_pow2(e, un);
        qr_pow2(-e, sc);
#pragma unroll
        for (int r = 0; r < RW; ++r) v[r] *= sc;
#pragma unroll
        for (int r = 0; r < NRM; ++r) cb[r] *= sc;
      }
    }
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      T* x = Vs + i * RW;
      T* sc = Sc + i * NS;
      if (c0 == 0) {
        if constexpr (PIVOT) {
          // largest remaining column 2-norm, first position on ties
          T q0 = T(0), q1 = T(0);
#pragma unroll
          for (int r = 0; r < RW; r += 2) {
            q0 = v[r] * v[r] + q0;
            q1 = v[r + 1] * v[r + 1] + q1;
          }
          const bool cand = panel && cpos >= i;
          T best = cand ? (q0 + q1) * un * un : T(-1);
          if (!(best == best)) best = T(-0.5);  // NaN loses against every number
          int at = cand ? cpos : 64;
          warp_argmax(best, at);
          const int prev = cpos;
          if (panel && prev == at) cpos = i;
          else if (panel && prev == i) cpos = at;
        }
        const bool post = PIVOT ? panel && cpos == i : lane == i;
        if (post) {
#pragma unroll
          for (int r = 0; r < RW; r += 2) store2(&x[r], v[r], v[r + 1]);
        }
        __syncwarp();
        const unsigned who = PIVOT ? (unsigned)(__ffs(__ballot_sync(FULL, post)) - 1) : (unsigned)i;
        T d0 = T(0), d1 = T(0);
        T u0, u1;
        load2(&x[0], u0, u1);
        const T alpha = u0;
        d1 = u1 * v[1];
#pragma unroll
        for (int r = 2; r < RW; r += 2) {
          load2(&x[r], u0, u1);
          d0 = fma(u0, v[r], d0);
          d1 = fma(u1, v[r + 1], d1);
        }
        const T dd = d0 + d1;
        const T s = __shfl_sync(FULL, dd, who);
        T beta = alpha, t = T(0), scl = T(0);
        if (s != T(0)) {
          const T nrm = qr_sqrt(alpha * alpha + s);
          beta = alpha >= T(0) ? -nrm : nrm;
          scl = rcp_rn(alpha - beta);
        }
        if (beta == T(0) && info == 0) info = i + 1;
        const T rb = beta != T(0) ? rcp_rn(beta) : T(0);
        if (s != T(0)) t = (beta - alpha) * rb;
        const T w = t * fma(scl, dd, v[0]), ws = w * scl;
        const bool own = (unsigned)lane == who;
        const T r0 = own ? beta : v[0] - w;
        // the border multipliers C_j(r, i) / R(i, i)
        T l[NRM];
#pragma unroll
        for (int r = 0; r < NRM; ++r) {
          l[r] = r < nr ? __shfl_sync(FULL, cb[r], who) * rb : T(0);
          cb[r] = own ? l[r] : PIVOT && panel && cpos < i ? cb[r] : !PIVOT && panel && lane < i ? cb[r] : fma(-l[r], r0, cb[r]);
        }
        if (lane == 0) {
          sc[0] = t;
          sc[1] = scl;
#pragma unroll
          for (int r = 0; r < NRM; ++r) sc[2 + r] = l[r];
        }
        S[i * 33 + lane] = r0 * un;  // row i of R and of the trailing columns
        // apply and move one row up; finished panel columns are not used again
        v[0] = fma(-ws, x[1], v[1]);
#pragma unroll
        for (int r = 2; r < RW; r += 2) {
          load2(&x[r], u0, u1);
          v[r - 1] = fma(-ws, u0, v[r]);
          v[r] = fma(-ws, u1, v[r + 1]);
        }
        v[RW - 1] = T(0);
      } else {
        T d0 = T(0), d1 = T(0), u0, u1;
        load2(&x[0], u0, u1);
        d1 = u1 * v[1];
#pragma unroll
        for (int r = 2; r < RW; r += 2) {
          load2(&x[r], u0, u1);
          d0 = fma(u0, v[r], d0);
          d1 = fma(u1, v[r + 1], d1);
        }
        const T t = sc[0], scl = sc[1];
        const T w = t * fma(scl, d0 + d1, v[0]), ws = w * scl;
        const T r0 = v[0] - w;
#pragma unroll
        for (int r = 0; r < NRM; ++r) cb[r] = fma(-sc[2 + r], r0, cb[r]);
        S[i * 33 + lane] = r0 * un;
        v[0] = fma(-ws, x[1], v[1]);
#pragma unroll
        for (int r = 2; r < RW; r += 2) {
          load2(&x[r], u0, u1);
          v[r - 1] = fma(-ws, u0, v[r]);
          v[r] = fma(-ws, u1, v[r + 1]);
        }
        v[RW - 1] = T(0);
      }
    }
    if (info != 0) {
      if (lane == 0) report(a.st, DEV_ZERO_PIVOT, j, info, k);
      return;
    }
    // the reduced rows below the rows of R
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (r < n) S[(n + r) * 33 + lane] = v[r] * un;
    if (c0 == 0) {
      if (panel) cmap[cpos] = (unsigned char)lane;
    }
    __syncwarp();
    // ------------------------------------------------------------ store
    if (c0 == 0) {
      // T_j: R above the diagonal (by final column position), the scaled
      // reflectors below it, tau; the row map (identity) and the column map
      T* Tj = a.Tm + (size_t)j * szT(d);
      unsigned char* Pj = a.P + (size_t)j * szP(d);
      for (int p = 0; p < n; ++p) {
        const int lc = PIVOT ? cmap[p] : p;
        if (lane < n2) {
          const T tv = lane <= p ? S[lane * 33 + lc] : Vs[p * RW + (lane - p)] * Sc[p * NS + 1];
          Tj[(size_t)p * n2 + lane] = tv;
        }
      }
      if (lane < n) {
        Tj[2 * nn + lane] = Sc[lane * NS];
        Pj[n2 + lane] = PIVOT ? cmap[lane] : (unsigned char)lane;
      }
      if (lane < n2) Pj[lane] = (unsigned char)lane;
      if (panel) {
        const int p = PIVOT ? cpos : lane;
#pragma unroll
        for (int r = 0; r < NRM; ++r)
          if (r < nr) a.C[(size_t)j * nrn + (size_t)p * nr + r] = cb[r];
      }
    }
    for (int cc = hc; cc < nc; cc += 2) {
      const int cg = c0 + cc;
      if (rok && cg >= n) {
        const T u = S[hr * 33 + cc], q = S[(n + hr) * 33 + cc];
        if (cg < n2) {
          a.D[oj + (size_t)(cg - n) * n + hr] = u;
          a.D[ojp + (size_t)(cg - n) * n + hr] = q;
        } else if (cg < 3 * n) {
          a.E[oj + (size_t)(cg - n2) * n + hr] = u;
          a.E[ojp + (size_t)(cg - n2) * n + hr] = q;
        } else {
          a.B[(size_t)j * nnx + (size_t)(cg - 3 * n) * n + hr] = u;
          a.B[(size_t)jp * nnx + (size_t)(cg - 3 * n) * n + hr] = q;
        }
      }
    }
    if (live && c >= n) {
#pragma unroll
      for (int r = 0; r < NRM; ++r)
        if (r < nr) {
          if (c < n2) {
            const size_t o = (size_t)jp * nrn + (size_t)(c - n) * nr + r;
            a.C[o] = src(a.C0, a.C, o) + cb[r] * un;
          } else if (c < 3 * n) {
            a.Rbuf[(size_t)j * nrn + (size_t)(c - n2) * nr + r] = cb[r] * un;
          } else {
            a.Fbuf[(size_t)j * nrnx + (size_t)(c - 3 * n) * nr + r] = (double)(cb[r] * un);
          }
        }
    }
  }
  __syncwarp();
}

template <typename T, bool PIVOT>
__global__ void __launch_bounds__(128, 4) k_factor_qr_warp(FactorArgs<T> a, const FactorArgs<T>*, const BatchCta*) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T* Vs = reinterpret_cast<T*>(smem_raw + (size_t)warp * QrShape<T>::BYTES);
  const long np = pairs_at_level(a.d.nblock, a.k);
  for (long q = (long)blockIdx.x * 4 + warp; q < np; q += (long)gridDim.x * 4)
    qr_pair<T, PIVOT>(a, a.k + (int)(2L * a.k * q), Vs, lane);
}
