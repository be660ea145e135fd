// Large blocks, FP64 LU: blocked elimination of one pair (or of the last block)
// by one CTA of NT = 256 or 512 threads, included by bcr_kernels.cu.
//
// The panel goes in blocks of w <= 64 columns.  A block is factored in shared
// memory and turned into the operator G of its eliminations on the way:
//   rows that became pivots:  G = L11^-1  (w x w, unit lower),
//   the other rows:           G = -L21 L11^-1,
// both acting on the pivot rows as they were before the block, so that
// everything right of the block is ONE product of depth w,
//   row <- (pivot row: 0, other row: itself) + G * (pivot rows),
// with no triangular solve.  Each warp takes strips of 16 columns, keeps the
// strip's pivot rows as B fragments in registers and walks over all rows, 16 at
// a time (FP64 tensor cores; G in shared memory); no barrier is needed until
// the next block.  Rows of the work matrix never move; the rows left after a
// block are walked in ascending order, in which the reduced rows are also
// stored, so that the slab and the results are read and written in whole
// sectors.
//
// T_j and C_j hold the operator form, block by block (SweepArgs::op = columns
// per block): the forward sweep applies each block as a matrix-vector product.
//
// The columns right of the panel can be split over the CTAs of a cluster: each
// factors the panel for itself (the same arithmetic, so the same pivots) and
// updates its own slice of the columns; they meet once, after the loads,
// because the results overwrite the sources.
//
// What bounds it (n = 128, nr = nx = 16, cycles of a pair on one SM): the pivot
// steps, 179,000 (1,400 each, dependent integer and reduction latencies),
// and the products, 325,000 (8.6 M fused multiply-adds: 148,000 at the FP64
// rate; the fragment and accumulator traffic takes the L1 pipe nearly as long).
// 1,024 blocks of n = 128: the factorization's levels 8.8 -> 4.1 ms; a lone pair
// 670 -> 193 us with its columns over 8 CTAs.
//
// The last block (lub_square) takes the same panels 16 columns at a time, with L and
// a substitution in place of the operator: its L is less well conditioned.
#pragma once

#include "bcr_lub_plan.cuh"

template <int NT>
struct LubShared {
  int row[NT];              // live rows (not yet pivots), ascending
  int pos[NT];              // row -> position in getrf's order (settles ties)
  int list[LUB_W + NT];     // this block's pivots in order (padded to `depth` by
                            // -1), then the rows left, ascending: index | row << 10
  int4 hdr[2][NT / 32];     // candidate of each warp: |a| (two words), position and index
  double val[2][NT / 32][LUB_SB];  // its row: reciprocal of the pivot, then the columns to its right
  int wcnt[NT / 32];
  int info, nrest;
};

__device__ __forceinline__ void lub_bar(int threads) { asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory"); }

// A predicated load, 0 where p is false.  A conditional expression around a load
// becomes a branch, after which the loads of an unrolled batch wait for each
// other (the forward sweep of one pair at n = 128 took 50 us that way).
__device__ __forceinline__ double ldg_if(bool p, const double* a) {
  double v;
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f64 %0, 0d0000000000000000; @q ld.global.f64 %0, [%1]; }\n"
               : "=d"(v)
               : "l"(a), "r"((unsigned)p)
               : "memory");
  return v;
}
// Stores of one lane (p) without a branch: a candidate's header, and its row.
__device__ __forceinline__ void sts_candidate(bool p, unsigned hdr, unsigned hi, unsigned lo, unsigned z, unsigned val,
                                              double rc, const double (&v)[LUB_SB]) {
  static_assert(LUB_SB == 16, "stores below");
  asm volatile(
      "{ .reg .pred q; setp.ne.u32 q, %0, 0;\n"
      "@q st.shared.v4.u32 [%1], {%2, %3, %4, %4};\n"
      "@q st.shared.v2.f64 [%5], {%6, %7};\n"
      "@q st.shared.v2.f64 [%5 + 16], {%8, %9};\n"
      "@q st.shared.v2.f64 [%5 + 32], {%10, %11};\n"
      "@q st.shared.v2.f64 [%5 + 48], {%12, %13};\n"
      "@q st.shared.v2.f64 [%5 + 64], {%14, %15};\n"
      "@q st.shared.v2.f64 [%5 + 80], {%16, %17};\n"
      "@q st.shared.v2.f64 [%5 + 96], {%18, %19};\n"
      "@q st.shared.v2.f64 [%5 + 112], {%20, %21}; }\n" ::"r"((unsigned)p),
      "r"(hdr), "r"(hi), "r"(lo), "r"(z), "r"(val), "d"(rc), "d"(v[1]), "d"(v[2]), "d"(v[3]), "d"(v[4]), "d"(v[5]),
      "d"(v[6]), "d"(v[7]), "d"(v[8]), "d"(v[9]), "d"(v[10]), "d"(v[11]), "d"(v[12]), "d"(v[13]), "d"(v[14]), "d"(v[15])
      : "memory");
}

// Factors the w columns of Pb (column stride ld, nl live rows by index) with the
// getrf pivot rule among the rows below ncand and leaves, by row, U on and right
// of a pivot row's diagonal and the operator G left of it (rows that did not
// become pivots: G).  Fills list and nrest, updates pos.  kb: columns factored
// before.  Sets info (first zero pivot + 1).
//
// SQ (the last block, w <= 16): the columns come from W and go back there by
// original row, L\U; Pb keeps -L (the rows left, and the pivot rows left of their
// diagonal) in place of the operator.
//
// Sub-blocks of 16 columns, a row of them per thread in registers.  As in the
// warp-per-pair kernel the register of an eliminated column takes the operator
// row X (row = row at the sub-block's start + X times the pivot rows at its
// start), so the block's other columns, left and right, need no triangular
// solve either: every row adds X times the 16 pivot rows, on the tensor cores.
// (Sub-blocks of 8 moved the block through shared memory twice as often, which
// bound them: 730 of 1,630 cycles per column of a 272-row panel.)
// A pivot is found by three warp reductions (upper and lower word of |a|, then
// position and lane, which settles ties by getrf's rule), once within each
// warp and once over the warps' candidates, with one barrier between.  The
// steps are one rolled loop over rotating registers: unrolled, each step's code
// is fetched for a single use.
template <int NT, bool SQ = false>
__device__ void lub_panel(LubShared<NT>& sh, double* Pb, int ld, double* Xb, double* Ub, int nl, int kb, int w,
                          int ncand, int depth, double* Wc = nullptr, int ldw = 0) {
  constexpr unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwa = (nl + 31) / 32;  // warps with rows
  const bool act = tid < nl;
  const int row = act ? sh.row[tid] : 0;
  int mypos = act ? sh.pos[row] : -1;
  bool done = !act || row >= ncand;  // border rows are eliminated but never pivots
  bool used = false;                 // this row became a pivot
  for (int i = w + tid; i < depth; i += NT) sh.list[i] = -1;
  constexpr int SB = LUB_SB;
  for (int c0 = 0; c0 < w; c0 += SB) {
    if (warp < nwa) {
      const bool before = used;  // a pivot of an earlier sub-block
      int own = SB;
      const int pos_in = mypos;
      const bool done_in = done;
      double v[SB];
      const int steps = min(SB, w - c0);
      const unsigned hdr0 = (unsigned)__cvta_generic_to_shared(&sh.hdr[0][warp]);
      const unsigned val0 = (unsigned)__cvta_generic_to_shared(&sh.val[0][warp][0]);
      constexpr unsigned HS = sizeof(sh.hdr[0]), VS = sizeof(sh.val[0]);
      const int hl = lane < nwa ? lane : 0;
      // zero, tiny and huge pivots are only noted, and the sub-block run again with
      // their correctly rounded reciprocals (see tc_pair)
      for (int attempt = 0;; ++attempt) {
        bool bad = false;
#pragma unroll
        for (int c = 0; c < SB; ++c)
          v[c] = SQ ? ldg_if(act, Wc + (size_t)min(c, w - 1) * ldw + row) : Pb[(size_t)min(c0 + c, w - 1) * ld + tid];
#pragma unroll 1
      for (int i = 0; i < steps; ++i) {
        // v[0] is column i; a step moves every column one register down and the
        // eliminated one to the end
        const double v0 = v[0];
        const int gi = kb + c0 + i;
        const unsigned par = i & 1;
        unsigned hi, lo;
        double rc;
        tc_candidate(v0, done, hi, lo, rc);
        const unsigned hmax = __reduce_max_sync(FULL, hi);
        lo = hi == hmax ? lo : 0u;
        const unsigned lmax = __reduce_max_sync(FULL, lo);
        const bool in = hi == hmax && lo == lmax && !done;
        const unsigned best = __reduce_min_sync(FULL, in ? ((unsigned)mypos << 5) | lane : 0xffffffffu);
        if (attempt && hmax != 0u && !tc_plain_pivot<double>(hmax)) rc = v0 != 0.0 ? __drcp_rn(v0) : 0.0;
        // the warp's candidate; where none is left (hmax = 0, best all ones) lane 31
        // posts zeros
        sts_candidate((best & 31u) == (unsigned)lane, hdr0 + par * HS, hmax, lmax, (best >> 5 << 9) | tid,
                      val0 + par * VS, rc, v);
        lub_bar(nwa * 32);
        const int4 h = sh.hdr[par][hl];
        const unsigned bh = __reduce_max_sync(FULL, (unsigned)h.x);
        const unsigned bl = __reduce_max_sync(FULL, (unsigned)h.x == bh ? (unsigned)h.y : 0u);
        const unsigned pt =
            __reduce_min_sync(FULL, (unsigned)h.x == bh && (unsigned)h.y == bl ? (unsigned)h.z : 0xffffffffu);
        bad = bad || !tc_plain_pivot<double>(bh);
        const int p = (int)(pt & 511u), pmin = (int)(pt >> 9);
        const double* sv = sh.val[par][p >> 5];
        double u[SB];
#pragma unroll
        for (int c = 0; c < SB; c += 2) load2(&sv[c], u[c], u[c + 1]);
        mypos = mypos == gi ? pmin : mypos;
        if (tid == p) {
          if (attempt && v0 == 0.0 && sh.info == 0) sh.info = gi + 1;
          mypos = gi;
          done = used = true;
          own = i;
          sh.list[c0 + i] = tid | (row << 10);
        }
        const double l = used ? 0.0 : v0 * u[0];
        if (SQ && act && !used) Pb[(size_t)i * ld + tid] = -l;
#pragma unroll
        for (int c = 1; c < SB; ++c) v[c - 1] = fma(-l, u[c], v[c]);
        v[SB - 1] = used ? v0 : -l;
      }
        if (!bad || attempt) break;
        mypos = pos_in;
        done = done_in;
        used = before;
        own = SB;
        lub_bar(nwa * 32);  // the last step's readers of the candidates are done
      }
#pragma unroll 1
      for (int i = steps; i < SB; ++i) {  // a partial sub-block: the rest of the rotation
        const double v0 = v[0];
#pragma unroll
        for (int c = 1; c < SB; ++c) v[c - 1] = v[c];
        v[SB - 1] = v0;
      }
      if (act) {
#pragma unroll
        for (int c = 0; c < SB; ++c) {
          if constexpr (SQ) {
            if (c < w) Wc[(size_t)c * ldw + row] = c >= own ? v[c] : -Pb[(size_t)c * ld + tid];
            continue;
          }
          if (!before && c0 + c < w) Pb[(size_t)(c0 + c) * ld + tid] = v[c];
          Xb[(size_t)c * ld + tid] = !before && c < own && c0 + c < w ? v[c] : 0.0;
        }
      }
    }
    if (SQ || w <= SB) break;
    __syncthreads();
    // the sub-block's pivot rows in the block's other columns, as they are now
    for (int e = tid; e < w * SB; e += NT) {
      const int c = e / SB, m = e % SB;
      Ub[c * LUB_UB + m] = c0 + m < w ? Pb[(size_t)c * ld + (sh.list[c0 + m] & 1023)] : 0.0;
    }
    __syncthreads();
    // a row tile of 16 per warp, three column groups of 8 at a time; rows and
    // columns beyond the block are read (inside the buffers) and computed, each
    // only into itself, but not stored
    {
      constexpr int GT = 3;
      const int g = lane >> 2, q = lane & 3;
      const int own_g = min(SB, (w - c0 + 7) & ~7) / 8;  // groups of the sub-block itself
      const int tr = (nl + 15) / 16, tc = (w + 7) / 8 - own_g, ht = (tc + GT - 1) / GT;
      for (int t = warp; t < tr * ht; t += NT / 32) {
        const int h = t / tr, rb = (t - h * tr) * 16 + g;
        double x[GT][2][2];
        double* e0[GT];
        const double* ub[GT];
        int ca[GT];
#pragma unroll
        for (int i = 0; i < GT; ++i) {
          int cg = 8 * min(h * GT + i, tc - 1);
          if (cg >= c0) cg += 8 * own_g;
          ca[i] = cg + 2 * q;
          e0[i] = Pb + (size_t)ca[i] * ld + rb;
          ub[i] = Ub + (cg + g) * LUB_UB + q;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            x[i][u][0] = e0[i][8 * u];
            x[i][u][1] = e0[i][ld + 8 * u];
          }
        }
        const double* xa = Xb + (size_t)q * ld + rb;
#pragma unroll
        for (int ks = 0; ks < SB / 4; ++ks) {
          const double a0 = xa[(size_t)(4 * ks) * ld], a1 = xa[(size_t)(4 * ks) * ld + 8];
#pragma unroll
          for (int i = 0; i < GT; ++i) {
            const double b = ub[i][4 * ks];
            dmma_8x8x4(x[i][0][0], x[i][0][1], a0, b);
            dmma_8x8x4(x[i][1][0], x[i][1][1], a1, b);
          }
        }
#pragma unroll
        for (int i = 0; i < GT; ++i) {
          const bool ok = h * GT + i < tc;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const bool on = ok && rb + 8 * u < nl;
            if (on && ca[i] < w) e0[i][8 * u] = x[i][u][0];
            if (on && ca[i] + 1 < w) e0[i][ld + 8 * u] = x[i][u][1];
          }
        }
      }
    }
    __syncthreads();
  }
  if (act) sh.pos[row] = mypos;
  // the rows left, ascending
  const unsigned keep = __ballot_sync(FULL, act && !used);
  if (lane == 0) sh.wcnt[warp] = __popc(keep);
  __syncthreads();
  int base = 0;
  for (int o = 0; o < warp; ++o) base += sh.wcnt[o];
  if (act && !used) sh.list[depth + base + __popc(keep & ((1u << lane) - 1u))] = tid | (row << 10);
  if (tid == NT - 1) sh.nrest = base + __popc(keep);
}

// Pb <- the operator alone, for the products: the pivot rows' unit diagonal and
// zeros right of it, zero columns [w, depth)
template <int NT>
__device__ void lub_operator(const LubShared<NT>& sh, double* Pb, int ld, int nl, int w, int depth) {
  const int tid = threadIdx.x, lane = tid & 31;
  for (int c = tid >> 5; c < w; c += NT / 32)
    for (int i = lane; i <= c; i += 32) Pb[(size_t)c * ld + (sh.list[i] & 1023)] = i == c ? 1.0 : 0.0;
  for (int c = w + (tid >> 5); c < depth; c += NT / 32)
    for (int r = lane; r < nl; r += 32) Pb[(size_t)c * ld + r] = 0.0;
}

// Pb column c <- W column c0 + c (rows of W by row[]); one column per warp
template <int NT>
__device__ void lub_stage(const LubShared<NT>& sh, double* Pb, int ld, const double* W, int R, int nl, int c0, int w) {
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < w; c += NT / 32) {
    const double* col = W + (size_t)(c0 + c) * R;
    for (int l0 = lane; l0 < nl; l0 += 256) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = ldg_if(l0 + 32 * u < nl, col + sh.row[min(l0 + 32 * u, nl - 1)]);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (l0 + 32 * u < nl) Pb[(size_t)c * ld + l0 + 32 * u] = v[u];
    }
  }
}

// row[] <- the rows left after the block
template <int NT>
__device__ void lub_shrink(LubShared<NT>& sh, int depth) {
  const int t = threadIdx.x;
  if (t < sh.nrest) sh.row[t] = sh.list[depth + t] >> 10;
}

// A group of columns with one source and one set of destinations (all pointers
// to the group's first column):
//   src: current values by original row, rows [lo, hi) (zero elsewhere);
//   du:  the block's U rows, by order;
//   dc:  the other rows, by order among them (or by row: in place);
//   db:  the last rows (border), by number; db = dbs + value when dbs is given.
struct LubCols {
  int cols;
  const double* src;
  int ss, lo, hi;
  double* du;
  int us;
  double* dc;
  int cs, nb;          // nb: border rows kept apart (0: none)
  double* db;
  const double* dbs;
  int bs;
};

// Columns [cb, cb + 16) of the group, row tiles [t0, t1) of 16 (the first
// depth / 16 are the block's pivots).  c_byrow: the other rows by original row.
template <int NT, int NB>
__device__ __forceinline__ void lub_item(const LubShared<NT>& sh, const double* Pb, int ld, const LubCols& G,
                                         int cb, int t0, int t1, bool c_byrow) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  constexpr int PT = NB / 2;  // pivot tiles
  const int nrest = sh.nrest;
  double bf[2 * NB][2];
#pragma unroll
  for (int ks = 0; ks < 2 * NB; ++ks) {
    const int e = sh.list[4 * ks + q], r = e >> 10;
    const bool on = e >= 0 && r >= G.lo && r < G.hi;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int c = cb + 8 * v + g;
      bf[ks][v] = ldg_if(on && c < G.cols, G.src + (size_t)c * G.ss + r);
    }
  }
  double cur[2][2][2];
  int ent[2];
  auto fetch = [&](int t, double (&x)[2][2][2], int (&en)[2]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = t * 16 + u * 8 + g;
      const bool rest = t >= PT && t < t1 && e < 8 * NB + nrest;
      en[u] = t < t1 && (t < PT || rest) ? sh.list[e] : -1;
      const int r = en[u] >> 10;
      const bool on = rest && r >= G.lo && r < G.hi;
      const double* s = G.src + r;
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = cb + 8 * v + 2 * q + h;
          x[u][v][h] = ldg_if(on && c < G.cols, s + (size_t)c * G.ss);
        }
    }
  };
  fetch(t0, cur, ent);
  for (int t = t0; t < t1; ++t) {
    double nxt[2][2][2];
    int en[2];
    fetch(t + 1, nxt, en);
    const double* a0 = Pb + (size_t)q * ld + (ent[0] < 0 ? 0 : ent[0] & 1023);
    const double* a1 = Pb + (size_t)q * ld + (ent[1] < 0 ? 0 : ent[1] & 1023);
#pragma unroll
    for (int ks = 0; ks < 2 * NB; ++ks) {
      const double f0 = a0[(size_t)(4 * ks) * ld], f1 = a1[(size_t)(4 * ks) * ld];
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        dmma_8x8x4(cur[0][v][0], cur[0][v][1], f0, bf[ks][v]);
        dmma_8x8x4(cur[1][v][0], cur[1][v][1], f1, bf[ks][v]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (ent[u] < 0) continue;
      const int i = t * 16 + u * 8 + g, r = ent[u] >> 10;
      double* dst;
      int st;
      double add = 0.0;
      const double* as = nullptr;
      if (t < PT) {
        dst = G.du + i;
        st = G.us;
      } else {
        const int e = i - 8 * NB, b = e - (nrest - G.nb);
        if (b >= 0) {
          dst = G.db + b;
          st = G.bs;
          if (G.dbs) as = G.dbs + b;
        } else {
          dst = G.dc + (c_byrow ? r : e);
          st = G.cs;
        }
      }
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = cb + 8 * v + 2 * q + h;
          if (c < G.cols) {
            if (as) add = as[(size_t)c * st];
            dst[(size_t)c * st] = cur[u][v][h] + add;
          }
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      ent[u] = en[u];
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) cur[u][v][h] = nxt[u][v][h];
    }
  }
}

// Item `it` of the strips of 16 columns of ng groups, each split in `parts` row
// ranges; group(i) gives the columns of group i, make(i) its description.
template <int NB, int NT, typename Cols, typename Make>
__device__ __forceinline__ void lub_update(const LubShared<NT>& sh, const double* Pb, int ld, int ng,
                                           bool c_byrow, Cols cols, Make make) {
  const int warp = threadIdx.x >> 5, nw = NT / 32;
  int ns = 0;
  for (int i = 0; i < ng; ++i) ns += (cols(i) + 15) / 16;
  if (ns == 0) return;
  const int tiles = NB / 2 + (sh.nrest + 15) / 16;
  // rows split where the strips leave warps idle
  int parts = 1;
  const int rounds = (ns + nw - 1) / nw;  // of whole strips
  for (int p = 2; p <= 4; ++p)
    if ((ns * p + nw - 1) / nw * (tiles / p + 3) < rounds * (tiles + 3) * 9 / 10 && p <= tiles) parts = p;
  const int tp = (tiles + parts - 1) / parts;
  for (int it = warp; it < ns * parts; it += nw) {
    int s = it % ns, i = 0;
    while (s >= (cols(i) + 15) / 16) {
      s -= (cols(i) + 15) / 16;
      ++i;
    }
    const int t0 = it / ns * tp, t1 = t0 + tp < tiles ? t0 + tp : tiles;
    if (t0 < t1) lub_item<NT, NB>(sh, Pb, ld, make(i), 16 * s, t0, t1, c_byrow);
  }
}

__device__ __forceinline__ unsigned cluster_ctas() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;\n" : "=r"(v));
  return v;
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(v));
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}

// One pair per cluster of `cluster_ctas()` CTAs (1: per CTA, grid-stride).
template <int NT, int NB>
__global__ void __launch_bounds__(NT, 512 / NT) k_factor_lu_lub(FactorArgs<double> a, double* slab, size_t slab_elems,
                                                                int bw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LubShared<NT> sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = NT / 32, DEPTH = 8 * NB;
  const Dims d = a.d;
  const int n = d.n, nr = d.nr, nx = d.nx, nb = d.nblock;
  const int n2 = 2 * n, n3 = 3 * n, R = n2 + nr, NC = n3 + nx, ld = lub_ld(R);
  const size_t nn = (size_t)n * n, nnx = (size_t)n * nx, nrn = (size_t)nr * n, nrnx = (size_t)nr * nx;
  double* Pb = reinterpret_cast<double*>(smem_raw);    // [DEPTH][ld] the panel block
  double* Xb = Pb + (size_t)DEPTH * ld;                // [LUB_SB][ld] the sub-block's operator rows
  double* Ub = Xb + (size_t)LUB_SB * ld;               // [DEPTH][LUB_UB] its pivot rows
  double* W = slab + (size_t)blockIdx.x * slab_elems;  // [NC][R], by original row
  const int k = a.k;
  const long np = pairs_at_level(nb, k);
  const int slices = (int)cluster_ctas(), slice = (int)cluster_rank();
  const long first_pair = blockIdx.x / slices, pair_step = gridDim.x / slices;
  // this CTA's trailing columns, in multiples of 16
  const int trail = NC - n, per = ((trail + slices - 1) / slices + 15) & ~15;
  const int cl = min(n + slice * per, NC), ch = min(cl + per, NC);
  // the factor columns are written by the CTAs in turn (slices is a power of two)
  const auto mine = [&](int c) { return (c & (slices - 1)) == slice; };
  const bool direct = a.first != 0;  // the sources are not the results: read them in place
  const double* sD = direct ? a.D0 : a.D;
  const double* sE = direct ? a.E0 : a.E;
  const double* sB = direct ? a.B0 : a.B;
  const double* sC = direct ? a.C0 : a.C;
  for (long qp = first_pair; qp < np; qp += pair_step) {
    const int j = k + (int)(2L * k * qp), jp = j - k;
    const size_t oj = (size_t)j * nn, ojp = (size_t)jp * nn;
    const int w0 = n < bw ? n : bw;
    // ------------------------------------------------------------ load
    // the first block of the panel straight into shared memory, the other
    // panel columns and this CTA's trailing columns into the slab (not where
    // they can be read in place), one column per warp; the zeros of the
    // trailing columns are not stored
    for (int c = warp; c < n; c += NW) {
      const bool sp = !direct && n + c >= cl && n + c < ch, sq = !direct && n2 + c >= cl && n2 + c < ch;
      double* pc = c < w0 ? Pb + (size_t)c * ld : W + (size_t)c * R;
      double v[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = lane + 32 * u;
        const bool in = i < n;
        const size_t o = (size_t)c * n + i;
        v[u][0] = ldg_if(in, sE + ojp + o);
        v[u][1] = ldg_if(in, sD + oj + o);
        v[u][2] = ldg_if(in && sp, sD + ojp + o);
        v[u][3] = ldg_if(in && sq, sE + oj + o);
      }
      for (int r = lane; r < nr; r += 32) pc[n2 + r] = sC[(size_t)j * nrn + (size_t)c * nr + r];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = lane + 32 * u;
        if (i < n) {
          pc[i] = v[u][0];
          pc[n + i] = v[u][1];
          if (sp) W[(size_t)(n + c) * R + i] = v[u][2];
          if (sq) W[(size_t)(n2 + c) * R + n + i] = v[u][3];
        }
      }
    }
    for (int c = max(cl, n3) + warp; c < ch; c += NW)
      for (int i = lane; i < n; i += 32) {
        W[(size_t)c * R + i] = sB[(size_t)jp * nnx + (size_t)(c - n3) * n + i];
        W[(size_t)c * R + n + i] = sB[(size_t)j * nnx + (size_t)(c - n3) * n + i];
      }
    for (int r = tid; r < R; r += NT) sh.row[r] = sh.pos[r] = r;
    if (tid == 0) sh.info = 0;
    if (slices > 1) {
      __threadfence();
      cluster_barrier();  // the sources are read: the results may replace them
    }
    __syncthreads();
    // ------------------------------------------------- blocked elimination
    double* Tj = a.Tm + (size_t)j * szT(d);
    unsigned char* Pj = a.P + (size_t)j * szP(d);
    int nl = R, kb = 0;
    for (; kb < n; kb += bw) {
      const int w = n - kb < bw ? n - kb : bw, kbw = kb + w;
      const bool last = kbw >= n;
      if (kb > 0) {
        lub_stage(sh, Pb, ld, W, R, nl, kb, w);
        __syncthreads();
      }
      lub_panel(sh, Pb, ld, Xb, Ub, nl, kb, w, n2, DEPTH);
      __syncthreads();
      if (sh.info != 0) break;
      // this block's columns of T: the pivot rows, and the rows left where their
      // order is final; else kept in the slab.  C_j.
      const int nrest = sh.nrest;
      for (int c = warp; c < w; c += NW) {
        if (!mine(c)) continue;
        const double* pc = Pb + (size_t)c * ld;
        double* tcol = Tj + (size_t)(kb + c) * n2 + kb;
        for (int i = lane; i < w; i += 32) tcol[i] = pc[sh.list[i] & 1023];
        if (last) {
          for (int e = lane; e < nrest - nr; e += 32) tcol[w + e] = pc[sh.list[DEPTH + e] & 1023];
        } else {
          double* wcol = W + (size_t)(kb + c) * R;
          for (int e = lane; e < nrest - nr; e += 32) {
            const int en = sh.list[DEPTH + e];
            wcol[en >> 10] = pc[en & 1023];
          }
        }
        for (int e = nrest - nr + lane; e < nrest; e += 32)
          a.C[(size_t)j * nrn + (size_t)(kb + c) * nr + (e - (nrest - nr))] = pc[sh.list[DEPTH + e] & 1023];
      }
      if (slice == 0) {
        for (int i = tid; i < w; i += NT) Pj[kb + i] = (unsigned char)(sh.list[i] >> 10);
        if (last)
          for (int e = tid; e < n; e += NT) Pj[n + e] = (unsigned char)(sh.list[DEPTH + e] >> 10);
      }
      __syncthreads();
      lub_operator(sh, Pb, ld, nl, w, DEPTH);
      __syncthreads();
      // column groups: the panel's other columns, then this CTA's part of x_jp,
      // x_jpp and xb
      auto lo_of = [&](int i) { return i == 0 ? kbw : max(cl, i == 1 ? n : i == 2 ? n2 : n3); };
      auto hi_of = [&](int i) { return i == 0 ? n : min(ch, i == 1 ? n2 : i == 2 ? n3 : NC); };
      auto cols = [&](int i) { return max(hi_of(i) - lo_of(i), 0); };
      auto make = [&](int i) {
        LubCols G;
        const int c = lo_of(i);
        G.cols = cols(i);
        G.src = W + (size_t)c * R;
        G.ss = R;
        G.lo = 0;
        G.hi = R;
        if (kb == 0 && i > 0) {  // structure of the trailing columns: TOP, BOTTOM or both
          G.lo = i == 2 ? n : 0;
          G.hi = i == 1 ? n : n2;
          if (direct && i < 3) {
            G.src = i == 1 ? sD + ojp + (size_t)(c - n) * n : sE + oj + (size_t)(c - n2) * n - n;
            G.ss = n;
          }
        }
        G.us = n;
        if (i == 0) { G.du = Tj + (size_t)c * n2 + kb; G.us = n2; }
        else if (i == 1) G.du = a.D + oj + (size_t)(c - n) * n + kb;
        else if (i == 2) G.du = a.E + oj + (size_t)(c - n2) * n + kb;
        else G.du = a.B + (size_t)j * nnx + (size_t)(c - n3) * n + kb;
        G.dc = W + (size_t)c * R;
        G.cs = R;
        G.nb = 0;
        G.db = nullptr;
        G.dbs = nullptr;
        G.bs = nr;
        if (last && i > 0) {
          G.cs = n;
          G.nb = nr;
          if (i == 1) {
            G.dc = a.D + ojp + (size_t)(c - n) * n;
            G.db = a.C + (size_t)jp * nrn + (size_t)(c - n) * nr;
            G.dbs = sC + (size_t)jp * nrn + (size_t)(c - n) * nr;
          } else if (i == 2) {
            G.dc = a.E + ojp + (size_t)(c - n2) * n;
            G.db = a.Rbuf + (size_t)j * nrn + (size_t)(c - n2) * nr;
          } else {
            G.dc = a.B + (size_t)jp * nnx + (size_t)(c - n3) * n;
            G.db = a.Fbuf + (size_t)j * nrnx + (size_t)(c - n3) * nr;
          }
        }
        return G;
      };
      lub_update<NB>(sh, Pb, ld, 4, !last, cols, make);
      __syncthreads();
      if (!last) {
        lub_shrink(sh, DEPTH);
        nl -= w;
        __syncthreads();
      }
    }
    if (sh.info != 0) {
      if (tid == 0 && slice == 0) report(a.st, DEV_ZERO_PIVOT, j, sh.info, k);
    } else {
      // columns of the earlier blocks: rows whose order was not final then
      // (row[]: order -> row, from the row map)
      if (slice == 0)
        for (int i = tid; i < n; i += NT) Pj[n2 + i] = (unsigned char)i;
      const int kl = ((n - 1) / bw) * bw;  // first column of the last block
      if (kl > 0) {
        // order of each row: later pivots through pos, the rows left by the list
        for (int e = tid; e < n; e += NT) sh.pos[sh.list[DEPTH + e] >> 10] = n + e;
        __syncthreads();
        for (int r = tid; r < n2; r += NT) sh.row[sh.pos[r]] = r;
        __syncthreads();
        for (int c = warp; c < kl; c += NW) {
          const int cb = c / bw * bw, p0 = cb + bw;
          if (!mine(c - cb)) continue;
          const double* wcol = W + (size_t)c * R;
          double* tcol = Tj + (size_t)c * n2;
          for (int p = p0 + lane; p < n2; p += 256) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = ldg_if(p + 32 * u < n2, wcol + sh.row[min(p + 32 * u, n2 - 1)]);
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (p + 32 * u < n2) tcol[p + 32 * u] = v[u];
          }
        }
      }
    }
    __syncthreads();
  }
}

// Columns right of a block of 16 of the last block, a strip of 16 columns per warp,
// in place: the pivot rows' part by substitution with L11 (a quad holds a column's
// 16 rows; -L in Pb), then row -= L21 times it, the products summed from zero: they
// round at the element's size once per block and not once per product.  With L11^-1
// in place of the substitution, and summed onto the element, the solution's error
// was 1.4 times as large for blocks of 64 columns at order 288 (1.2 times for 16).
// Order 288: 360 us then, 340 now (it was 679 with the kernel before those).
template <int NT>
__device__ void lub_square_update(const LubShared<NT>& sh, const double* Pb, int ld, double* C, int N, int cols) {
  constexpr int W = 16;
  constexpr unsigned FULL = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int tiles = (sh.nrest + 15) / 16;
  const double* Lr[W / 4];
  int pr[W / 4];
#pragma unroll
  for (int ks = 0; ks < W / 4; ++ks) {
    const int e = sh.list[4 * ks + q];
    Lr[ks] = Pb + (e & 1023);
    pr[ks] = e >> 10;
  }
  for (int cb = 16 * warp; cb < cols; cb += 16 * (NT / 32)) {
    double bf[W / 4][2];
#pragma unroll
    for (int ks = 0; ks < W / 4; ++ks)
#pragma unroll
      for (int v = 0; v < 2; ++v) bf[ks][v] = ldg_if(cb + 8 * v + g < cols, C + (size_t)(cb + 8 * v + g) * N + pr[ks]);
#pragma unroll
    for (int i = 0; i < W - 1; ++i) {
      const double u0 = __shfl_sync(FULL, bf[i / 4][0], (lane & ~3) | (i & 3));
      const double u1 = __shfl_sync(FULL, bf[i / 4][1], (lane & ~3) | (i & 3));
#pragma unroll
      for (int ks = i / 4; ks < W / 4; ++ks)
        if (4 * ks + q > i) {
          const double l = Lr[ks][(size_t)i * ld];
          bf[ks][0] = fma(l, u0, bf[ks][0]);
          bf[ks][1] = fma(l, u1, bf[ks][1]);
        }
    }
#pragma unroll
    for (int ks = 0; ks < W / 4; ++ks)
#pragma unroll
      for (int v = 0; v < 2; ++v)
        if (cb + 8 * v + g < cols) C[(size_t)(cb + 8 * v + g) * N + pr[ks]] = bf[ks][v];
    for (int t = 0; t < tiles; ++t) {
      int ent[2];
      double cur[2][2][2], acc[2][2][2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int e = t * 16 + u * 8 + g;
        ent[u] = e < sh.nrest ? sh.list[W + e] : -1;
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = cb + 8 * v + 2 * q + h;
            cur[u][v][h] = ldg_if(ent[u] >= 0 && c < cols, C + (size_t)c * N + (ent[u] >> 10));
            acc[u][v][h] = 0.0;
          }
      }
      const double* a0 = Pb + (size_t)q * ld + (ent[0] < 0 ? 0 : ent[0] & 1023);
      const double* a1 = Pb + (size_t)q * ld + (ent[1] < 0 ? 0 : ent[1] & 1023);
#pragma unroll
      for (int ks = 0; ks < W / 4; ++ks) {
        const double f0 = a0[(size_t)(4 * ks) * ld], f1 = a1[(size_t)(4 * ks) * ld];
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          dmma_8x8x4(acc[0][v][0], acc[0][v][1], f0, bf[ks][v]);
          dmma_8x8x4(acc[1][v][0], acc[1][v][1], f1, bf[ks][v]);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = cb + 8 * v + 2 * q + h;
            if (ent[u] >= 0 && c < cols) C[(size_t)c * N + (ent[u] >> 10)] = cur[u][v][h] + acc[u][v][h];
          }
    }
  }
}

// Blocked LU of the N x N matrix W in place (rows not moved), blocks of 16 columns:
// L\U by original row, piv[position] = row.  Returns the LAPACK info.
template <int NT>
__device__ int lub_square(LubShared<NT>& sh, double* Pb, double* W, int N, int* piv) {
  constexpr int BW = LUB_LAST_W;
  const int tid = threadIdx.x, ld = lub_ld(N);
  for (int r = tid; r < N; r += NT) sh.row[r] = sh.pos[r] = r;
  if (tid == 0) sh.info = 0;
  __syncthreads();
  int nl = N;
  for (int kb = 0; kb < N; kb += BW) {
    const int w = N - kb < BW ? N - kb : BW;
    lub_panel<NT, true>(sh, Pb, ld, nullptr, nullptr, nl, kb, w, N, BW, W + (size_t)kb * N, N);
    __syncthreads();
    if (sh.info != 0) break;
    for (int i = tid; i < w; i += NT) piv[kb + i] = sh.list[i] >> 10;
    if (kb + w < N) lub_square_update(sh, Pb, ld, W + (size_t)(kb + w) * N, N, N - kb - w);  // w == BW
    __syncthreads();
    lub_shrink(sh, BW);
    nl -= w;
    __syncthreads();
  }
  return sh.info;
}
