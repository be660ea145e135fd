// Sweeps of one pair by one CTA for 16 < n <= 128, single systems, included by
// bcr_kernels.cu.
//
// Each thread owns a row and a run of 32 columns and reads those 32 elements in
// one batch of loads (ld_batch), so that a pair costs two or three memory round
// trips instead of one for every few columns; the serial parts (32 x 32
// triangles) run on the warp that holds the triangle in its registers.  Right-
// hand sides go through in chunks of SWB_RHS.  Bound by memory latency at the
// levels with few pairs: at n = 128 a lone pair took 52 us forward and 62 us
// backward with loads that the compiler interleaved with their uses, and takes
// 8.8 and 14.5 us (FP64); 1,024 blocks, all levels: 585 -> 144 and 660 -> 224 us.
#pragma once

constexpr int SWB_RHS = 8;

// sum of m[u] * x[u], u < 32, in two chains; x 16-byte aligned in shared memory
template <typename T>
__device__ __forceinline__ double dot32(const T (&m)[32], const double* x) {
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int u = 0; u < 32; u += 2) {
    const double2 v = *reinterpret_cast<const double2*>(x + u);
    s0 = fma(double(m[u]), v.x, s0);
    s1 = fma(double(m[u + 1]), v.y, s1);
  }
  return s0 + s1;
}

// x of the pair's rows in getrf order into y[c][RW]
template <int RW, int NT, typename T>
__device__ __forceinline__ void fwd_gather(const SweepArgs<T>& a, int j, int jp, int col0, int nc, double (*y)[RW]) {
  const int n = a.d.n;
  const unsigned char* Pj = a.P + (size_t)j * szP(a.d);
  for (int e = threadIdx.x; e < RW * nc; e += NT) {
    const int p = e % RW, c = e / RW;
    double v = 0.0;
    if (p < 2 * n) {
      const int r = Pj[p];
      const double* xc = a.x + (size_t)(col0 + c) * a.ldx;
      v = r < n ? xc[(size_t)jp * n + r] : xc[(size_t)j * n + (r - n)];
    }
    y[c][p] = v;
  }
}

// results to x_j (positions below n) and x_jp
template <int RW, int NT, typename T>
__device__ __forceinline__ void fwd_scatter(const SweepArgs<T>& a, int j, int jp, int col0, int nc,
                                            const double (*y)[RW]) {
  const int n = a.d.n;
  for (int e = threadIdx.x; e < RW * nc; e += NT) {
    const int p = e % RW, c = e / RW;
    double* xc = a.x + (size_t)(col0 + c) * a.ldx;
    if (p < n) xc[(size_t)j * n + p] = y[c][p];
    else if (p < 2 * n) xc[(size_t)jp * n + p - n] = y[c][p];
  }
}

// XB_j = sgn * C_j v (v[c][RW], first n entries), one border row per warp; four in
// the CTAs of two warps, where one after the other cost a solve of 60 blocks of
// n = 17 with 12 border rows 6 us of 100
template <int RW, int NT, typename T>
__device__ __forceinline__ void fwd_border(const SweepArgs<T>& a, int j, int col0, int nc, const double (*v)[RW],
                                           double sgn) {
  constexpr int U = RW / 64, W = NT / 32, G = W == 2 ? 4 : 1;
  const int n = a.d.n, nr = a.d.nr, lane = threadIdx.x & 31;
  const T* Cj = a.C + (size_t)j * nr * n;
  for (int r0 = threadIdx.x >> 5; r0 < nr; r0 += G * W) {
    T cv[G][U];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = lane + 32 * u, r = r0 + g * W;
        cv[g][u] = ld_batch(i < n && r < nr, Cj + (size_t)i * nr + r);
      }
    for (int c = 0; c < nc; ++c) {
      double s[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        s[g] = 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (lane + 32 * u < n) s[g] = fma(double(cv[g][u]), v[c][lane + 32 * u], s[g]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] += shfl_xor(s[g], o);
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (lane == 0 && r0 + g * W < nr) a.XB[(size_t)j * nr * a.nrhs + (size_t)(col0 + c) * nr + r0 + g * W] = sgn * s[g];
    }
  }
}

// Forward sweep with factors in operator form by blocks of op <= 64 columns
// (k_factor_lu_lub; padded k_factor_lu_grp): two threads per row, each with 32 of the block's columns.
// RW: rows, at least 2n.
template <int RW, typename T>
__global__ void __launch_bounds__(2 * RW, RW == 64 ? 4 : 256 / RW) k_forward_op(SweepArgs<T> a) {
  constexpr int NT = 2 * RW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double(*y)[RW] = reinterpret_cast<double(*)[RW]>(smem_raw);
  double(*raw)[RW] = y + min(a.nrhs, SWB_RHS);    // the blocks' rows before their block
  double(*part)[RW] = raw + min(a.nrhs, SWB_RHS);
  double(*blk)[64] = reinterpret_cast<double(*)[64]>(part + min(a.nrhs, SWB_RHS));
  const int tid = threadIdx.x, h = tid / RW, r = tid % RW;
  const Dims d = a.d;
  const int n = d.n, n2 = 2 * n, k = a.k, bw = a.op;
  const long np = pairs_at_level(d.nblock, k);
  for (long q = blockIdx.x; q < np; q += gridDim.x) {
    const int j = k + (int)(2L * k * q), jp = j - k;
    const T* Tj = a.Tm + (size_t)j * szT(d);
    for (int col0 = 0; col0 < a.nrhs; col0 += SWB_RHS) {
      const int nc = min(SWB_RHS, a.nrhs - col0);
      T m[32];
      auto load = [&](int kb) {  // strictly left of the diagonal
        const int lim = min(min(bw, n - kb), r - kb);
#pragma unroll
        for (int u = 0; u < 32; ++u) {
          const int c = 32 * h + u;
          m[u] = ld_batch(r < n2 && c < lim, Tj + (size_t)(kb + c) * n2 + r);
        }
      };
      load(0);
      fwd_gather<RW, NT>(a, j, jp, col0, nc, y);
      __syncthreads();
      for (int kb = 0; kb < n; kb += bw) {
        const int w = min(bw, n - kb);
        for (int e = tid; e < 64 * nc; e += NT) {
          const int i = e & 63, c = e >> 6;
          const double v = i < w ? y[c][kb + i] : 0.0;
          blk[c][i] = v;
          if (i < w) raw[c][kb + i] = v;
        }
        __syncthreads();
        double s[SWB_RHS];
#pragma unroll
        for (int c = 0; c < SWB_RHS; ++c)
          if (c < nc) s[c] = dot32(m, &blk[c][32 * h]);
        if (kb + bw < n) load(kb + bw);
        if (h) {
#pragma unroll
          for (int c = 0; c < SWB_RHS; ++c)
            if (c < nc) part[c][r] = s[c];
        }
        __syncthreads();
        if (!h && r >= kb) {
#pragma unroll
          for (int c = 0; c < SWB_RHS; ++c)
            if (c < nc) y[c][r] += s[c] + part[c][r];
        }
        __syncthreads();
      }
      fwd_scatter<RW, NT>(a, j, jp, col0, nc, y);
      fwd_border<RW, NT>(a, j, col0, nc, raw, 1.0);
      __syncthreads();
    }
  }
}

// Forward sweep with L and M (FP32 factors of the tensor-core kernel; factors of
// k_factor_level, k_factor_cta and k_factor_lu_blocked in either precision): a
// thread per row and run of 32 columns.  RW: rows, at least 2n; RW / 64 runs.  The
// triangles' elements wait in shared memory as doubles, each for the lane that wrote
// it: 1,024 threads leave 64 registers, and the 31 converted values of the serial
// part were spilled (a lone pair of n = 128: 22 -> 16 us).  The instances of 1,024
// threads still spill about 270 bytes, of the 32 elements that wait for their use.
template <int RW, typename T>
__global__ void __launch_bounds__(RW * (RW / 64), 1) k_forward_lm(SweepArgs<T> a) {
  constexpr int NT = RW * (RW / 64);
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double(*y)[RW] = reinterpret_cast<double(*)[RW]>(smem_raw);
  __shared__ double tri[RW / 64][32][32];  // [triangle][column][row]
  const int tid = threadIdx.x, h = tid / RW, r = tid % RW, lane = tid & 31;
  const Dims d = a.d;
  const int n = d.n, n2 = 2 * n, k = a.k;
  const long np = pairs_at_level(d.nblock, k);
  for (long q = blockIdx.x; q < np; q += gridDim.x) {
    const int j = k + (int)(2L * k * q), jp = j - k;
    const T* Tj = a.Tm + (size_t)j * szT(d);
    T m[32];  // strictly left of the diagonal
#pragma unroll
    for (int u = 0; u < 32; ++u) {
      const int c = 32 * h + u;
      m[u] = ld_batch(r < n2 && c < n && c < r, Tj + (size_t)c * n2 + r);
    }
    if (r / 32 == h) {
#pragma unroll
      for (int u = 0; u < 32; ++u) tri[h][u][lane] = -double(m[u]);
    }
    for (int col0 = 0; col0 < a.nrhs; col0 += SWB_RHS) {
      const int nc = min(SWB_RHS, a.nrhs - col0);
      fwd_gather<RW, NT>(a, j, jp, col0, nc, y);
      __syncthreads();
      for (int b = 0; 32 * b < n; ++b) {
        if (h == b && r / 32 == b) {  // the warp of the diagonal block
          for (int c = 0; c < nc; ++c) {
            double v = y[c][r];
#pragma unroll 8
            for (int u = 0; u < 31; ++u) {
              const double vc = __shfl_sync(FULL, v, u);
              v = fma(tri[b][u][lane], lane > u ? vc : 0.0, v);
            }
            // rows below n of a partial last block are updated here too
            y[c][r] = v;
          }
        }
        __syncthreads();
        if (h == b && r / 32 > b)
          for (int c = 0; c < nc; ++c) y[c][r] -= dot32(m, &y[c][32 * b]);
        __syncthreads();
      }
      fwd_scatter<RW, NT>(a, j, jp, col0, nc, y);
      fwd_border<RW, NT>(a, j, col0, nc, y, -1.0);
      __syncthreads();
    }
  }
}

// Backward sweep: x_j = U^-1 (y_j - D'_j x_jp - E'_j x_jpp - B'_j xb), a thread
// per row and run of 32 columns.  RB: rows, at least n; RB / 32 runs.
// (The instances are held to 128 registers; those in FP64 spill 260 bytes.)
template <int RB, typename T>
__global__ void __launch_bounds__(RB * (RB / 32), RB == 32 ? 16 : RB == 64 ? 4 : 1) k_backward_big(SweepArgs<T> a) {
  constexpr int NH = RB / 32, NT = RB * NH;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int CH = min(a.nrhs, SWB_RHS);
  double(*xa)[RB] = reinterpret_cast<double(*)[RB]>(smem_raw);
  double(*xz)[RB] = xa + CH;
  double(*y)[RB] = xz + CH;
  double(*part)[NT] = reinterpret_cast<double(*)[NT]>(y + CH);
  const int tid = threadIdx.x, h = tid / RB, i = tid % RB, lane = tid & 31;
  const Dims d = a.d;
  const int n = d.n, n2 = 2 * n, nx = d.nx, nb = d.nblock, k = a.k;
  const bool qrp = a.sel == SEL_QRP;
  const size_t xb_off = (size_t)(nb + 1) * n + d.qx;
  const long np = pairs_at_level(nb, k);
  for (long q = blockIdx.x; q < np; q += gridDim.x) {
    const int j = k + (int)(2L * k * q), jp = j - k, jpp = min(j + k, nb);
    const T* Dj = a.D + (size_t)j * n * n;
    const T* Ej = a.E + (size_t)j * n * n;
    const T* Bj = a.B + (size_t)j * n * nx;
    const T* Tj = a.Tm + (size_t)j * szT(d);
    for (int col0 = 0; col0 < a.nrhs; col0 += SWB_RHS) {
      const int nc = min(SWB_RHS, a.nrhs - col0);
      T m[32];
      auto load = [&](const T* M, int ld, int first) {  // columns from `first` on
#pragma unroll
        for (int u = 0; u < 32; ++u) {
          const int c = 32 * h + u;
          m[u] = ld_batch(i < n && c < n && c >= first, M + (size_t)c * ld + i);
        }
      };
      load(Dj, n, 0);
      for (int e = tid; e < RB * nc; e += NT) {
        const int p = e % RB, c = e / RB;
        const double* xc = a.x + (size_t)(col0 + c) * a.ldx;
        const bool in = p < n;
        const double v0 = ld_batch(in, xc + (size_t)jp * n + p), v1 = ld_batch(in, xc + (size_t)jpp * n + p),
                     v2 = ld_batch(in, xc + (size_t)j * n + p);
        xa[c][p] = v0;
        xz[c][p] = v1;
        y[c][p] = v2;
      }
      __syncthreads();
      for (int c = 0; c < nc; ++c) part[c][tid] = dot32(m, &xa[c][32 * h]);
      load(Ej, n, 0);
      T bv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) bv[u] = ld_batch(i < n && h + NH * u < nx, Bj + (size_t)(h + NH * u) * n + i);
      for (int c = 0; c < nc; ++c) {
        const double* xb = a.x + (size_t)(col0 + c) * a.ldx + xb_off;
        double s = part[c][tid] + dot32(m, &xz[c][32 * h]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (h + NH * u < nx) s = fma(double(bv[u]), xb[h + NH * u], s);
        if constexpr (NH == 1) {
          // more than four border columns on one warp: eight loads in flight (one
          // after the other, 60 blocks of n = 17 with 14 of them took 86 us, now 79)
          for (int e0 = 4; e0 < nx; e0 += 8) {
            T bm[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) bm[u] = ld_batch(i < n && e0 + u < nx, Bj + (size_t)(e0 + u) * n + i);
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (e0 + u < nx) s = fma(double(bm[u]), xb[e0 + u], s);
          }
        } else {
          for (int e = h + NH * 4; e < nx; e += NH)
            if (i < n) s = fma(double(Bj[(size_t)e * n + i]), xb[e], s);
        }
        part[c][tid] = s;
      }
      load(Tj, n2, i);  // U, on and right of the diagonal
      __syncthreads();
      for (int c = h; c < nc; c += NH) {
        double s = 0.0;
#pragma unroll
        for (int g = 0; g < NH; ++g) s += part[c][g * RB + i];
        y[c][i] -= s;
      }
      double ud = 1.0;
#pragma unroll
      for (int u = 0; u < 32; ++u)
        if (u == lane) ud = double(m[u]);
      const double rdi = i < n && h == i / 32 ? 1.0 / ud : 0.0;
      __syncthreads();
      for (int b = (n - 1) / 32; b >= 0; --b) {
        if (h == b && i / 32 == b) {  // the warp of the diagonal block
          for (int c = 0; c < nc; ++c) {
            double v = y[c][i];
#pragma unroll
            for (int u = 31; u >= 0; --u) {
              const double xi = __shfl_sync(FULL, v * rdi, u);
              v = lane == u ? xi : fma(-double(m[u]), lane < u ? xi : 0.0, v);
            }
            y[c][i] = v;
          }
        }
        __syncthreads();
        if (h == b && i / 32 < b)
          for (int c = 0; c < nc; ++c) y[c][i] -= dot32(m, &y[c][32 * b]);
        __syncthreads();
      }
      for (int e = tid; e < RB * nc; e += NT) {
        const int p = e % RB, c = e / RB;
        if (p < n) {
          const int dst = qrp ? (int)a.P[(size_t)j * szP(d) + n2 + p] : p;
          a.x[(size_t)(col0 + c) * a.ldx + (size_t)j * n + dst] = y[c][p];
        }
      }
      __syncthreads();
    }
  }
}
