// Device code of the FP64 and 128-thread ladder Bethe-Salpeter kernels (see bse.cu, whose host entry points launch them).
// The FP64 kernels are instantiated per thread count in bse_fp64_*.cu, so that they compile side by side.
#pragma once

#include "bse_core.cuh"
#include "lu_dmma.cuh"

namespace dga {

#ifndef DGA_MIXED_MIN_BLOCKS
#define DGA_MIXED_MIN_BLOCKS 3  // resident CTAs per SM the mixed-precision kernels are compiled for
#endif
constexpr int BSE_THREADS = 128;
constexpr int BSE_NB = 32;  // panel width (also the row-block of the triangular solves)
constexpr int BSE_TM = 32;  // trailing-update row tile
constexpr int BSE_TN = 64;  // trailing-update column strip
constexpr int BSE_MAX_N = 2048;
constexpr int MAX_RHS = 16;  // n2 <= 16 (up to 4 orbitals)

// ----------------------------------------------------------------------------------------------
// Block-wide arg-max of the pivot measure: larger value wins, ties go to the smaller row index.
// ----------------------------------------------------------------------------------------------
template <typename R>
__device__ int block_argmax(R v, int idx, R* s_val, int* s_idx) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    R ov = __shfl_down_sync(0xffffffffu, v, off);
    int oi = __shfl_down_sync(0xffffffffu, idx, off);
    argmax_merge(v, idx, ov, oi);
  }
  if (lane == 0) {
    s_val[warp] = v;
    s_idx[warp] = idx;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    v = lane < nw ? s_val[lane] : R(-1);
    idx = lane < nw ? s_idx[lane] : 0x7fffffff;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      R ov = __shfl_down_sync(0xffffffffu, v, off);
      int oi = __shfl_down_sync(0xffffffffu, idx, off);
      argmax_merge(v, idx, ov, oi);
    }
    if (lane == 0) {
      s_val[0] = v;
      s_idx[0] = idx;
    }
  }
  __syncthreads();
  int r = s_idx[0];
  __syncthreads();
  return r;
}

// ----------------------------------------------------------------------------------------------
// Shared-memory layout of one CTA: the GEMM tiles and the panel/triangular-solve buffers are never live at
// the same time, so they share storage.
// ----------------------------------------------------------------------------------------------
template <typename C>
struct BseSmem {
  union {
    struct {
      C Ls[BSE_NB][BSE_TM];      // L21 row tile (k, row)
      C Us[BSE_TN][BSE_NB + 1];  // U12 column strip (col, k), padded
    } g;
    struct {
      C L11[BSE_NB][BSE_NB + 1];
      C L11i[BSE_NB][BSE_NB + 1];  // inverse of the unit lower triangle of L11
      C A12[BSE_NB][BSE_NB + 1];   // A12 chunk of the U12 solve (col, k); solved block of the RHS solves
    } t;
  } u;
  C row[BSE_NB];
  double red_val[32];
  int red_idx[32];
  int flag;
};

// X = L^-1 for the unit lower triangular nb x nb block in L11 (column c of X by thread c):
// X[r][c] = -sum_{k=c}^{r-1} L[r][k] X[k][c] for r > c, X[c][c] = 1.
template <typename C>
__device__ void unit_lower_inverse(BseSmem<C>& sm, int nb) {
  using R = decltype(C::x);
  const int c = threadIdx.x;
  if (c < nb) {
    for (int r = 0; r < c; ++r) sm.u.t.L11i[r][c] = cmake<C>(R(0), R(0));
    sm.u.t.L11i[c][c] = cmake<C>(R(1), R(0));
    for (int r = c + 1; r < nb; ++r) {
      C acc = cmake<C>(R(0), R(0));
      for (int k = c; k < r; ++k) cfms(acc, sm.u.t.L11[r][k], sm.u.t.L11i[k][c]);
      sm.u.t.L11i[r][c] = acc;
    }
  }
}

// ----------------------------------------------------------------------------------------------
// LU with partial pivoting of the N x N column-major matrix A (leading dimension ld) in place.
// piv[j] receives the row exchanged with row j.  Returns true if an exact zero pivot was met.
// ----------------------------------------------------------------------------------------------
template <typename C>
__device__ bool lu_factor(C* __restrict__ A, int N, int ld, int* __restrict__ piv, BseSmem<C>& sm) {
  using R = decltype(C::x);
  const int tid = threadIdx.x, T = blockDim.x;
  bool singular = false;

  for (int k0 = 0; k0 < N; k0 += BSE_NB) {
    const int nb = min(BSE_NB, N - k0);
    // ---- panel factorisation (columns k0 .. k0+nb-1) ----
    // pivot candidates of the first panel column; later columns get theirs from the previous update
    R best = R(-1);
    int bidx = 0x7fffffff;
    for (int i = k0 + tid; i < N; i += T) {
      R v = cabs1(A[(size_t)k0 * ld + i]);
      if (v > best) {
        best = v;
        bidx = i;
      }
    }
    for (int jj = 0; jj < nb; ++jj) {
      const int j = k0 + jj;
      int p;
      {
        double dv = (double)best;  // reduce in double precision storage (R may be float)
        p = block_argmax<double>(dv, bidx, sm.red_val, sm.red_idx);
      }
      if (p >= N) p = j;  // cannot happen for j < N; keeps the index in range regardless
      if (tid == 0) piv[j] = p;
      if (p != j) {
        for (int c = tid; c < nb; c += T) {
          C* col = A + (size_t)(k0 + c) * ld;
          C t = col[j];
          col[j] = col[p];
          col[p] = t;
        }
      }
      __syncthreads();
      const C d = A[(size_t)j * ld + j];
      const bool zero = (d.x == R(0) && d.y == R(0));
      if (zero) singular = true;
      const C rinv = zero ? cmake<C>(R(0), R(0)) : crecip(d);
      const int ncols = nb - jj - 1;
      for (int c = tid; c < ncols; c += T) sm.row[c] = A[(size_t)(j + 1 + c) * ld + j];
      __syncthreads();
      best = R(-1);
      bidx = 0x7fffffff;
      for (int i = j + 1 + tid; i < N; i += T) {
        C l = A[(size_t)j * ld + i];
        if (!zero) l = cmul(l, rinv);
        A[(size_t)j * ld + i] = l;
        // batched loads: 8 independent loads in flight before the updates
        for (int c0 = 0; c0 < ncols; c0 += 8) {
          C v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (c0 + u < ncols) v[u] = A[(size_t)(j + 1 + c0 + u) * ld + i];
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (c0 + u < ncols) {
              cfms(v[u], l, sm.row[c0 + u]);
              A[(size_t)(j + 1 + c0 + u) * ld + i] = v[u];
            }
          if (c0 == 0) {  // column j+1 just updated: its pivot candidate (look-ahead)
            const R a = cabs1(v[0]);
            if (a > best) {
              best = a;
              bidx = i;
            }
          }
        }
      }
      __syncthreads();
    }
    // ---- L11 and its inverse in shared memory ----
    for (int e = tid; e < nb * nb; e += T) {
      const int r = e % nb, c = e / nb;
      sm.u.t.L11[r][c] = A[(size_t)(k0 + c) * ld + k0 + r];
    }
    __syncthreads();
    unit_lower_inverse(sm, nb);
    // ---- row interchanges on the columns outside the panel ----
    // When every pivot row lies below the panel and no two coincide, the interchanges are independent pairs
    // and are applied in parallel over (interchange, column); otherwise they run in order per column.
    const int k1 = k0 + nb;
    if (tid < 32) {
      bool ok = true;
      if (tid < nb) {
        const int p = piv[k0 + tid];
        if (p != k0 + tid) {
          if (p < k1) ok = false;
          for (int o = 0; o < nb; ++o)
            if (o != tid && piv[k0 + o] == p) ok = false;
        }
      }
      const unsigned all_ok = __all_sync(0xffffffffu, ok);
      if (tid == 0) sm.flag = all_ok ? 1 : 0;
    }
    __syncthreads();
    if (sm.flag) {
      const int ncol = N - nb;
      for (int e = tid; e < nb * ncol; e += T) {
        const int jj = e / ncol;
        int c = e - jj * ncol;
        c = c < k0 ? c : c + nb;  // skip the panel columns
        const int p = piv[k0 + jj];
        if (p != k0 + jj) {
          C* col = A + (size_t)c * ld;
          C t = col[k0 + jj];
          col[k0 + jj] = col[p];
          col[p] = t;
        }
      }
    } else {
      for (int c = tid; c < N; c += T) {
        if (c >= k0 && c < k1) continue;
        C* col = A + (size_t)c * ld;
        for (int jj = 0; jj < nb; ++jj) {
          const int p = piv[k0 + jj];
          if (p != k0 + jj) {
            C t = col[k0 + jj];
            col[k0 + jj] = col[p];
            col[p] = t;
          }
        }
      }
    }
    __syncthreads();
    // ---- U12 = L11^-1 A12, in chunks of 32 columns staged through shared memory ----
    for (int c0 = k1; c0 < N; c0 += BSE_NB) {
      const int cw = min(BSE_NB, N - c0);
      for (int e = tid; e < nb * cw; e += T) {
        const int c = e / nb, k = e % nb;
        sm.u.t.A12[c][k] = A[(size_t)(c0 + c) * ld + k0 + k];
      }
      __syncthreads();
      for (int e = tid; e < cw * (BSE_NB / 8); e += T) {
        const int c = e % cw, g = e / cw;  // 8-row groups
        C out[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) out[u] = cmake<C>(R(0), R(0));
        for (int k = 0; k < nb; ++k) {
          const C a = sm.u.t.A12[c][k];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int r = g * 8 + u;
            if (r < nb && k <= r) cfma(out[u], sm.u.t.L11i[r][k], a);
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int r = g * 8 + u;
          if (r < nb) A[(size_t)(c0 + c) * ld + k0 + r] = out[u];
        }
      }
      __syncthreads();
    }
    // ---- trailing update A22 -= L21 U12: column strips of BSE_TN, row tiles of BSE_TM ----
    const int nt = N - k1;
    if (nt > 0) {
      const int ty = tid % (BSE_TM / 4), tx = tid / (BSE_TM / 4);  // 8 x 16 thread grid, 4x4 outputs each
      for (int cs = k1; cs < N; cs += BSE_TN) {
        for (int e = tid; e < nb * BSE_TN; e += T) {
          const int c = e / nb, k = e % nb;
          sm.u.g.Us[c][k] = (cs + c < N) ? A[(size_t)(cs + c) * ld + k0 + k] : cmake<C>(R(0), R(0));
        }
        for (int rt = k1; rt < N; rt += BSE_TM) {
          C acc[4][4];
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int c = cs + tx + 16 * b;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              const int r = rt + ty + 8 * a;
              acc[a][b] = (c < N && r < N) ? A[(size_t)c * ld + r] : cmake<C>(R(0), R(0));
            }
          }
          for (int e = tid; e < nb * BSE_TM; e += T) {
            const int k = e / BSE_TM, r = e % BSE_TM;
            sm.u.g.Ls[k][r] = (rt + r < N) ? A[(size_t)(k0 + k) * ld + rt + r] : cmake<C>(R(0), R(0));
          }
          __syncthreads();
#pragma unroll 4
          for (int k = 0; k < nb; ++k) {
            C lv[4], uv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) lv[a] = sm.u.g.Ls[k][ty + 8 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) uv[b] = sm.u.g.Us[tx + 16 * b][k];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
              for (int b = 0; b < 4; ++b) cfms(acc[a][b], lv[a], uv[b]);
          }
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int c = cs + tx + 16 * b;
            if (c < N) {
              C* col = A + (size_t)c * ld;
#pragma unroll
              for (int a = 0; a < 4; ++a) {
                const int r = rt + ty + 8 * a;
                if (r < N) col[r] = acc[a][b];
              }
            }
          }
          __syncthreads();
        }
      }
    }
  }
  return singular;
}

// ----------------------------------------------------------------------------------------------
// Solves for the n_rhs columns of Y in place (column-major, leading dimension N), with the LU factors of lu_factor or
// lu_factor_dmma (unit lower L below the diagonal, U on and above): lu_forward_inplace Y = L^-1 Y, lu_backward_inplace
// Y = U^-1 Y.  Blocked by 32 rows: the diagonal
// block is solved by one warp per right-hand side (lane = row, the solved value broadcast by shuffle), the
// rest of the rows are updated from the block copy in shared memory.  L11: the diagonal block, yb: [n_rhs][32] the
// solved block, both in shared memory.
// ----------------------------------------------------------------------------------------------
template <typename C, typename CY, int NR>
__device__ void lu_forward_inplace(const C* __restrict__ A, int N, int ld, CY* __restrict__ Y,
                                 C (*__restrict__ L11)[BSE_NB + 1], CY* __restrict__ yb) {
  constexpr int n_rhs = NR;
  // factor elements a thread has in flight in the row updates: eight where each one feeds several right-hand
  // sides; with one to three the registers go to the factorisation around the solve instead
  constexpr int SOLVE_LOADS = NR >= 4 ? 8 : 1;
  using R = decltype(C::x);
  using RY = decltype(CY::x);
  const int tid = threadIdx.x, T = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarps = T >> 5;
  // forward: L z = b
  for (int b0 = 0; b0 < N; b0 += BSE_NB) {
    const int bn = min(BSE_NB, N - b0);
    for (int e = tid; e < bn * bn; e += T) {
      const int r = e % bn, c = e / bn;
      L11[r][c] = A[(size_t)(b0 + c) * ld + b0 + r];
    }
    __syncthreads();
    for (int s = warp; s < n_rhs; s += nwarps) {
      CY y = lane < bn ? Y[(size_t)s * N + b0 + lane] : cmake<CY>(RY(0), RY(0));
      for (int r = 0; r < bn; ++r) {
        CY yr;
        yr.x = __shfl_sync(0xffffffffu, y.x, r);
        yr.y = __shfl_sync(0xffffffffu, y.y, r);
        if (lane > r && lane < bn) {
          const C l = L11[lane][r];
          cfms(y, cmake<CY>((RY)l.x, (RY)l.y), yr);
        }
      }
      if (lane < bn) {
        Y[(size_t)s * N + b0 + lane] = y;
        yb[s * 32 + lane] = y;
      }
    }
    __syncthreads();
    // rows below the block: one thread per row, every right-hand side at once (each L element read once,
    // SOLVE_LOADS of them in flight; the products are summed in ascending r)
    for (int i = b0 + bn + tid; i < N; i += T) {
      CY acc[NR];
#pragma unroll
      for (int s = 0; s < NR; ++s) acc[s] = Y[(size_t)s * N + i];
      if constexpr (SOLVE_LOADS == 1) {
        for (int r = 0; r < bn; ++r) {
          const C l = A[(size_t)(b0 + r) * ld + i];
          const CY lw = cmake<CY>((RY)l.x, (RY)l.y);
#pragma unroll
          for (int s = 0; s < NR; ++s) cfms(acc[s], lw, yb[s * 32 + r]);
        }
      } else {
        for (int r0 = 0; r0 < bn; r0 += SOLVE_LOADS) {
          C l[SOLVE_LOADS];
#pragma unroll
          for (int u = 0; u < SOLVE_LOADS; ++u)
            l[u] = (r0 + u < bn) ? A[(size_t)(b0 + r0 + u) * ld + i] : cmake<C>(R(0), R(0));
#pragma unroll
          for (int u = 0; u < SOLVE_LOADS; ++u) {
            if (r0 + u >= bn) break;
            const CY lw = cmake<CY>((RY)l[u].x, (RY)l[u].y);
#pragma unroll
            for (int s = 0; s < NR; ++s) cfms(acc[s], lw, yb[s * 32 + r0 + u]);
          }
        }
      }
#pragma unroll
      for (int s = 0; s < NR; ++s) Y[(size_t)s * N + i] = acc[s];
    }
    __syncthreads();
  }
}

template <typename C, typename CY, int NR>
__device__ void lu_backward_inplace(const C* __restrict__ A, int N, int ld, CY* __restrict__ Y,
                                 C (*__restrict__ L11)[BSE_NB + 1], CY* __restrict__ yb) {
  constexpr int n_rhs = NR;
  // factor elements a thread has in flight in the row updates: eight where each one feeds several right-hand
  // sides; with one to three the registers go to the factorisation around the solve instead
  constexpr int SOLVE_LOADS = NR >= 4 ? 8 : 1;
  using R = decltype(C::x);
  using RY = decltype(CY::x);
  const int tid = threadIdx.x, T = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarps = T >> 5;
  const int nblk = (N + BSE_NB - 1) / BSE_NB;
  for (int blk = nblk - 1; blk >= 0; --blk) {
    const int b0 = blk * BSE_NB;
    const int bn = min(BSE_NB, N - b0);
    for (int e = tid; e < bn * bn; e += T) {
      const int r = e % bn, c = e / bn;
      L11[r][c] = A[(size_t)(b0 + c) * ld + b0 + r];
    }
    __syncthreads();
    for (int s = warp; s < n_rhs; s += nwarps) {
      CY y = lane < bn ? Y[(size_t)s * N + b0 + lane] : cmake<CY>(RY(0), RY(0));
      const C d = lane < bn ? L11[lane][lane] : cmake<C>(R(1), R(0));
      const double2 rd = crecip(make_double2((double)d.x, (double)d.y));  // every row's at once, not one after the other
      for (int r = bn - 1; r >= 0; --r) {
        if (lane == r) y = cmul_fma(y, rd);
        CY yr;
        yr.x = __shfl_sync(0xffffffffu, y.x, r);
        yr.y = __shfl_sync(0xffffffffu, y.y, r);
        if (lane < r) {
          const C u = L11[lane][r];
          cfms(y, cmake<CY>((RY)u.x, (RY)u.y), yr);
        }
      }
      if (lane < bn) {
        Y[(size_t)s * N + b0 + lane] = y;
        yb[s * 32 + lane] = y;
      }
    }
    __syncthreads();
    // rows above the block: one thread per row, every right-hand side at once (each U element read once,
    // SOLVE_LOADS of them in flight, summed in ascending r)
    for (int i = tid; i < b0; i += T) {
      CY acc[NR];
#pragma unroll
      for (int s = 0; s < NR; ++s) acc[s] = Y[(size_t)s * N + i];
      if constexpr (SOLVE_LOADS == 1) {
        for (int r = 0; r < bn; ++r) {
          const C u = A[(size_t)(b0 + r) * ld + i];
          const CY uw = cmake<CY>((RY)u.x, (RY)u.y);
#pragma unroll
          for (int s = 0; s < NR; ++s) cfms(acc[s], uw, yb[s * 32 + r]);
        }
      } else {
        for (int r0 = 0; r0 < bn; r0 += SOLVE_LOADS) {
          C uu[SOLVE_LOADS];
#pragma unroll
          for (int u = 0; u < SOLVE_LOADS; ++u)
            uu[u] = (r0 + u < bn) ? A[(size_t)(b0 + r0 + u) * ld + i] : cmake<C>(R(0), R(0));
#pragma unroll
          for (int u = 0; u < SOLVE_LOADS; ++u) {
            if (r0 + u >= bn) break;
            const CY uw = cmake<CY>((RY)uu[u].x, (RY)uu[u].y);
#pragma unroll
            for (int s = 0; s < NR; ++s) cfms(acc[s], uw, yb[s * 32 + r0 + u]);
          }
        }
      }
#pragma unroll
      for (int s = 0; s < NR; ++s) Y[(size_t)s * N + i] = acc[s];
    }
    __syncthreads();
  }
}

template <typename C, typename CY, int NR>
__device__ void lu_solve_inplace(const C* __restrict__ A, int N, int ld, CY* __restrict__ Y,
                                 C (*__restrict__ L11)[BSE_NB + 1], CY* __restrict__ yb) {
  lu_forward_inplace<C, CY, NR>(A, N, ld, Y, L11, yb);
  lu_backward_inplace<C, CY, NR>(A, N, ld, Y, L11, yb);
}

// perm[i] = the original row at position i after the interchanges in piv (both N ints in shared memory).  One warp looks
// for the rows that moved, 32 at a time, and swaps those in order.
inline __device__ void build_perm(int N, const int* __restrict__ piv, int* __restrict__ perm) {
  const int tid = threadIdx.x, T = blockDim.x;
  for (int i = tid; i < N; i += T) perm[i] = i;
  __syncthreads();
  if (tid < 32) {
    for (int i0 = 0; i0 < N; i0 += 32) {
      const int p = i0 + tid < N ? piv[i0 + tid] : i0 + tid;
      unsigned moved = __ballot_sync(0xffffffffu, p != i0 + tid);
      while (moved) {
        const int b = __ffs(moved) - 1, q = __shfl_sync(0xffffffffu, p, b);
        moved &= moved - 1;
        if (tid == 0) {
          const int t = perm[i0 + b];
          perm[i0 + b] = perm[q];
          perm[q] = t;
        }
      }
    }
  }
  __syncthreads();
}

// Y = P * S where S is the n2-column selector (S[j, s] = 1 if the orbital pair of row j is s) and P the
// row permutation recorded in piv.  perm is shared scratch of N ints.
template <typename CY>
__device__ void permuted_selector(CY* __restrict__ Y, int N, int nv, int n_rhs, const int* __restrict__ piv,
                                  int* __restrict__ perm) {
  using RY = decltype(CY::x);
  const int tid = threadIdx.x, T = blockDim.x;
  build_perm(N, piv, perm);
  for (int e = tid; e < N * n_rhs; e += T) {
    const int i = e % N, s = e / N;
    Y[(size_t)s * N + i] = cmake<CY>((perm[i] / nv == s) ? RY(1) : RY(0), RY(0));
  }
  __syncthreads();
}

constexpr int fp64_min_blocks(int NT) { return 512 / NT; }  // 128 registers a thread

// Shared memory of the FP64 kernels: the factorisation's and the solves' buffers are never live at the same time.  The
// pivots (N ints) follow it.
template <int NT>
struct Fp64Smem {
  union {
    LuSmem<NT, 16> lu16;
    LuSmem<NT, NT <= 64 ? 16 : 32> lu32;  // CTAs of one or two warps take no matrix beyond LU_SMALL_N
    struct {
      double2 yb[MAX_RHS * BSE_NB];
      double2 L11[NT <= 64 ? 1 : BSE_NB][BSE_NB + 1];
    } solve;
  };
  int flag;
};

// LU and backward substitution with the block width of N.
template <int NT>
__device__ __forceinline__ bool fp64_lu(double2* __restrict__ A, int N, int ncols, int* __restrict__ piv,
                                        Fp64Smem<NT>& sm) {
  if (NT <= 64 || N <= LU_SMALL_N) return lu_factor_dmma<NT, 16>(A, N, ncols, N, piv, sm.lu16);
  return lu_factor_dmma<NT, NT <= 64 ? 16 : 32>(A, N, ncols, N, piv, sm.lu32);
}
template <int NT>
__device__ __forceinline__ void fp64_backward(const double2* __restrict__ A, int N, double2* Y, int ncols,
                                              Fp64Smem<NT>& sm) {
  if (NT <= 64 || N <= LU_SMALL_N)
    lu_backward_dmma<NT, 16>(A, N, N, Y, N, ncols, sm.lu16);
  else
    lu_backward_dmma<NT, NT <= 64 ? 16 : 32>(A, N, N, Y, N, ncols, sm.lu32);
}

// Y = U^-1 Y for a few right-hand sides in a CTA of one or two warps: as lu_backward_inplace, but the diagonal block's
// columns come straight from L2, eight steps ahead of the chain, so that no shared memory limits the CTAs of an SM. (With
// eight warps the staged form is the faster one: 711 against 750 ms for the three-orbital pass's items, whose blocks come
// from HBM.)
template <int NR>
__device__ void lu_backward_direct(const double2* __restrict__ A, int N, double2* __restrict__ Y,
                                   double2* __restrict__ yb) {
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = T >> 5;
  for (int b0 = (N - 1) / 32 * 32; b0 >= 0; b0 -= 32) {
    const int bn = min(32, N - b0);
    for (int s = warp; s < NR; s += nwarps) {
      const double2* D = A + (size_t)b0 * N + b0 + min(lane, bn - 1);
      double2 y = lane < bn ? Y[(size_t)s * N + b0 + lane] : make_double2(0.0, 0.0);
      const double2 rd = crecip(D[(size_t)min(lane, bn - 1) * N]);  // every row's at once, not one after the other
      double2 u[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) u[k] = D[(size_t)min(24 + k, bn - 1) * N];
#pragma unroll 1
      for (int r0 = 24; r0 >= 0; r0 -= 8) {
        double2 n[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) n[k] = D[(size_t)min(max(r0 - 8, 0) + k, bn - 1) * N];
#pragma unroll
        for (int k = 7; k >= 0; --k) {
          const int r = r0 + k;
          if (r >= bn) continue;
          if (lane == r) y = cmul_fma(y, rd);
          double2 yr;
          yr.x = __shfl_sync(0xffffffffu, y.x, r);
          yr.y = __shfl_sync(0xffffffffu, y.y, r);
          if (lane < r) cfms(y, u[k], yr);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = n[k];
      }
      if (lane < bn) {
        Y[(size_t)s * N + b0 + lane] = y;
        yb[s * 32 + lane] = y;
      }
    }
    __syncthreads();
    // rows above the block: one thread per row, every right-hand side at once, eight factor elements in flight
    for (int i = tid; i < b0; i += T) {
      double2 acc[NR];
#pragma unroll
      for (int s = 0; s < NR; ++s) acc[s] = Y[(size_t)s * N + i];
      for (int r0 = 0; r0 < bn; r0 += 8) {
        double2 u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = A[(size_t)(b0 + min(r0 + k, bn - 1)) * N + i];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (r0 + k >= bn) break;
#pragma unroll
          for (int s = 0; s < NR; ++s) cfms(acc[s], u[k], yb[s * 32 + r0 + k]);
        }
      }
#pragma unroll
      for (int s = 0; s < NR; ++s) Y[(size_t)s * N + i] = acc[s];
    }
    __syncthreads();
  }
}

// The right-hand-side count is chosen per item (n2 = 1, 4, 9 or 16), which keeps one copy of the factorisation per kernel.
template <int NR, int NT>
__device__ __forceinline__ void lu_backward_rhs(const double2* __restrict__ A, int N, double2* __restrict__ Y,
                                                Fp64Smem<NT>& sm) {
  if constexpr (NT <= 64)
    lu_backward_direct<NR>(A, N, Y, sm.solve.yb);
  else
    lu_backward_inplace<double2, double2, NR>(A, N, N, Y, sm.solve.L11, sm.solve.yb);
}
template <int NT>
__device__ __forceinline__ void lu_backward_n2(int n2, const double2* __restrict__ A, int N, double2* __restrict__ Y,
                                               Fp64Smem<NT>& sm) {
  switch (n2) {
    case 1: lu_backward_rhs<1, NT>(A, N, Y, sm); break;
    case 4: lu_backward_rhs<4, NT>(A, N, Y, sm); break;
    case 9: lu_backward_rhs<9, NT>(A, N, Y, sm); break;
    default: lu_backward_rhs<16, NT>(A, N, Y, sm); break;
  }
}

// A work item's matrix, column-major with leading dimension N, formed eight columns at a time (eight loads of Gamma_r in
// flight per thread; one column at a time the loop waited for L2 once per column), and the n2 selector right-hand sides
// (S[j, s] = 1 if the orbital pair of row j is s) in the columns behind it.
template <typename Source>
__device__ void form_item_fp64(const Source& src, const WorkItem& wi, int N, int n2, int nv, double2* __restrict__ A) {
  const int tid = threadIdx.x, T = blockDim.x;
  for (int i = tid; i < N; i += T) {
    const int pr = i / nv, vr = i - pr * nv;
    int pc = 0, vc = 0;
    for (int j0 = 0; j0 < N; j0 += 8) {
      double2 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (j0 + u < N) v[u] = src.element(wi.ch, wi.q, wi.w, N, i, j0 + u, pr, vr, pc, vc);
        if (++vc == nv) {
          vc = 0;
          ++pc;
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (j0 + u < N) A[(size_t)(j0 + u) * N + i] = v[u];
    }
    for (int s = 0; s < n2; ++s) A[(size_t)(N + s) * N + i] = make_double2(pr == s ? 1.0 : 0.0, 0.0);
  }
}

// n_box further right-hand sides behind the selectors leave as L^-1 P B (the caller's backward substitution is left).
template <typename Source, int NT>
__device__ int solve_item_fp64(const Source& src, const WorkItem& wi, int N, int n2, int nv, double beta,
                               double2* __restrict__ o, double2* __restrict__ A, Fp64Smem<NT>& sm, int* piv,
                               int n_box = 0) {
  const int tid = threadIdx.x, T = blockDim.x;
  double2* Y = A + (size_t)N * N;
  form_item_fp64(src, wi, N, n2, nv, A);
  __syncthreads();
  const bool singular = fp64_lu<NT>(A, N, N + n2 + n_box, piv, sm);
  lu_backward_n2<NT>(n2, A, N, Y, sm);
  // X[i][s] = Y[i][s] / beta, finiteness check
  if (tid == 0) sm.flag = 0;
  __syncthreads();
  bool bad = false;
  for (int e = tid; e < N * n2; e += T) {
    const int i = e / n2, s = e - i * n2;
    double2 y = Y[(size_t)s * N + i];
    y.x = y.x / beta;
    y.y = y.y / beta;
    if (!cfinite(y)) bad = true;
    o[e] = y;
  }
  if (bad) atomicOr(&sm.flag, DGA_ITEM_NONFINITE);
  __syncthreads();
  const int st = (singular ? DGA_ITEM_SINGULAR : 0) | sm.flag;
  __syncthreads();
  return st;
}

// FP64 kernel: one CTA per work item, persistent over the list.
template <typename Source, int NT>
__global__ void __launch_bounds__(NT, fp64_min_blocks(NT))
    bse_solve_sum_fp64_kernel(Source src, const WorkItem* __restrict__ work, int n_items, int N, int n2,
                              int nv, int W, int Q, double beta, double2* __restrict__ out,
                              int* __restrict__ status, double2* __restrict__ scratch, size_t slot_elems,
                              int redo_only) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fp64Smem<NT>& sm = *reinterpret_cast<Fp64Smem<NT>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(Fp64Smem<NT>));
  double2* A = scratch + (size_t)blockIdx.x * slot_elems;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    // re-solve mode: only the items whose status says the mixed solve did not converge or was not finite
    if (redo_only && (status[item] & DGA_ITEM_REDO) == 0) continue;
    const WorkItem wi = work[item];
    double2* o = out + (((size_t)wi.ch * Q + wi.q) * W + wi.w) * (size_t)N * n2;
    const int st = solve_item_fp64<Source, NT>(src, wi, N, n2, nv, beta, o, A, sm, piv);
    if (threadIdx.x == 0 && status) status[item] = st;
  }
}

// ----------------------------------------------------------------------------------------------
// Mixed form: FP32 LU (same core, float2 storage, FP32 trailing updates) and FP64 iterative refinement.
//
//   Y0 = (LU)^-1 P S with the FP32 factors and FP64 accumulation of the triangular solves;
//   repeat: r = S - A Y with A formed on the fly in FP64 from Gamma_r, chi0^-1 and U_r + V_r^q,
//           d = (LU)^-1 P r,  Y += d,  until the correction, or the error left after it as estimated from the
//           observed contraction, is below tol max|Y| (refine_converged), or max_iter corrections.
//
// FP64 is used only for A in the residual, the residual accumulation and Y.  Items that do not reach the
// tolerance are flagged DGA_ITEM_NOCONVERGE (the host re-solves them with the FP64 kernel).
// ----------------------------------------------------------------------------------------------

// byte offset of the [n2][n2] column-sum block after the pivot and permutation arrays, 16-byte aligned
__host__ __device__ inline size_t mixed_colsum_offset(int N) {
  return (sizeof(BseSmem<float2>) + 2 * sizeof(int) * (size_t)N + 15) & ~(size_t)15;
}

// One work item in the mixed form (FP32 LU, FP64 refinement).  Returns the status bits; *iters = corrections.
template <int NR>
__device__ int solve_item_mixed(const StructuredSource& src, const WorkItem& wi, int N, int nv, double beta,
                                int max_iter, double tol, double2* __restrict__ o, float2* __restrict__ A,
                                double2* __restrict__ Y, double2* __restrict__ Rb, BseSmem<float2>& sm, int* piv,
                                int* perm, double2* colsum, int* iters) {
  const int tid = threadIdx.x, T = blockDim.x;
  {
    const int pr0 = tid / nv, vr0 = tid - pr0 * nv;
    const int qT = T / nv, rT = T - qT * nv;
    int pc = 0, vc = 0;
    for (int j = 0; j < N; ++j) {
      float2* col = A + (size_t)j * N;
      int pr = pr0, vr = vr0;
      for (int i = tid; i < N; i += T) {
        const double2 a = src.element(wi.ch, wi.q, wi.w, N, i, j, pr, vr, pc, vc);
        col[i] = make_float2((float)a.x, (float)a.y);
        pr += qT;
        vr += rT;
        if (vr >= nv) {
          vr -= nv;
          ++pr;
        }
      }
      if (++vc == nv) {
        vc = 0;
        ++pc;
      }
    }
  }
  __syncthreads();
  const bool singular = lu_factor<float2>(A, N, N, piv, sm);
  double2* yb = reinterpret_cast<double2*>(&sm.u.t.A12[0][0]);
  permuted_selector<double2>(Y, N, nv, NR, piv, perm);
  lu_solve_inplace<float2, double2, NR>(A, N, N, Y, sm.u.t.L11, yb);
  double prev = 0.0;
  for (int e = tid; e < N * NR; e += T) prev = fmax(prev, fmax(fabs(Y[e].x), fabs(Y[e].y)));
  prev = block_max(prev, sm.red_val);
  int it = 0;
  bool converged = false;
  for (; it < max_iter; ++it) {
    structured_residual_permuted<NR>(src, wi.ch, wi.q, wi.w, N, nv, Y, Rb, perm, colsum,
                                     reinterpret_cast<double2*>(&sm.u));
    lu_solve_inplace<float2, double2, NR>(A, N, N, Rb, sm.u.t.L11, yb);
    double dmax = 0.0, ymax = 0.0;
    for (int e = tid; e < N * NR; e += T) {
      const double2 d = Rb[e];
      const double2 y = cadd(Y[e], d);
      Y[e] = y;
      dmax = fmax(dmax, fmax(fabs(d.x), fabs(d.y)));
      ymax = fmax(ymax, fmax(fabs(y.x), fabs(y.y)));
    }
    dmax = block_max(dmax, sm.red_val);
    ymax = block_max(ymax, sm.red_val);
    if (isnan(dmax) || refine_converged(dmax, ymax, prev, tol)) {  // NaN is flagged below
      converged = !isnan(dmax);
      ++it;
      break;
    }
    prev = dmax;
  }
  if (tid == 0) sm.flag = 0;
  __syncthreads();
  bool bad = false;
  for (int e = tid; e < N * NR; e += T) {
    const int i = e / NR, sidx = e % NR;
    double2 y = Y[(size_t)sidx * N + i];
    y.x = y.x / beta;
    y.y = y.y / beta;
    if (!cfinite(y)) bad = true;
    o[e] = y;
  }
  if (bad) atomicOr(&sm.flag, DGA_ITEM_NONFINITE);
  __syncthreads();
  const int st = (singular ? DGA_ITEM_SINGULAR : 0) | sm.flag | (converged ? 0 : DGA_ITEM_NOCONVERGE);
  *iters = it;
  __syncthreads();
  return st;
}

template <int NR>
__global__ void __launch_bounds__(BSE_THREADS, DGA_MIXED_MIN_BLOCKS)
    bse_solve_sum_mixed_kernel(StructuredSource src, const WorkItem* __restrict__ work, int n_items, int N, int n2,
                               int nv, int W, int Q, double beta, int max_iter, double tol,
                               double2* __restrict__ out, int* __restrict__ status, int* __restrict__ iters,
                               unsigned char* __restrict__ scratch, size_t slot_bytes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BseSmem<float2>& sm = *reinterpret_cast<BseSmem<float2>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(BseSmem<float2>));
  int* perm = piv + N;
  double2* colsum = reinterpret_cast<double2*>(smem_raw + mixed_colsum_offset(N));
  unsigned char* slot = scratch + (size_t)blockIdx.x * slot_bytes;
  float2* A = reinterpret_cast<float2*>(slot);
  double2* Y = reinterpret_cast<double2*>(slot + (((size_t)N * N * sizeof(float2) + 255) & ~(size_t)255));
  double2* Rb = Y + (size_t)N * n2;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const WorkItem wi = work[item];
    double2* o = out + (((size_t)wi.ch * Q + wi.q) * W + wi.w) * (size_t)N * n2;
    int it = 0;
    const int st = solve_item_mixed<NR>(src, wi, N, nv, beta, max_iter, tol, o, A, Y, Rb, sm, piv, perm, colsum,
                                        &it);
    if (threadIdx.x == 0) {
      if (status) status[item] = st;
      if (iters) iters[item] = it;
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Heterogeneous batch: one persistent launch over the work items of several problems (requests) whose
// sizes differ (niv, niw, number of q points, beta, inputs) but which share the number of orbitals, so that
// the RHS count NR = n_orb^2 is a compile-time constant of the launch.  Each item names its problem, whose
// descriptor carries the sizes, the resident inputs and the output.  The per-item body is the same as the
// single-problem kernels.
// ----------------------------------------------------------------------------------------------
// A batch item's problem, from its descriptor.
struct MultiProblem {
  StructuredSource src;
  WorkItem wi;
  int N, n2, nv;
  double2* o;
  __device__ __forceinline__ MultiProblem(const dga_bse_problem& d, const MultiItem& mi) : wi{mi.ch, mi.q, mi.w} {
    n2 = d.n_orb * d.n_orb;
    nv = 2 * d.niv;
    N = n2 * nv;
    src.gamma_cm = (const double2*)d.gamma_cm;
    src.chi0_inv = (const double2*)d.chi0_inv;
    src.uv = (const double2*)d.uv;
    src.n2 = n2;
    src.nv = nv;
    src.W = d.niw_half;
    src.Q = d.n_q;
    src.inv_beta2 = d.inv_beta2;
    o = (double2*)d.out + (((size_t)wi.ch * d.n_q + wi.q) * d.niw_half + wi.w) * (size_t)N * n2;
  }
};

// FP64 batch; redo_only: the re-solve of the items a mixed launch flagged. Shared memory and the scratch slot are sized
// for the largest problem of the launch.
template <int NT>
__global__ void __launch_bounds__(NT, fp64_min_blocks(NT))
    bse_multi_fp64_kernel(const dga_bse_problem* __restrict__ probs, const MultiItem* __restrict__ work, int n_items,
                          int n_max, int* __restrict__ status, int* __restrict__ iters,
                          unsigned char* __restrict__ scratch, size_t slot_bytes, int redo_only) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fp64Smem<NT>& sm = *reinterpret_cast<Fp64Smem<NT>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(Fp64Smem<NT>));
  double2* A = reinterpret_cast<double2*>(scratch + (size_t)blockIdx.x * slot_bytes);
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    if (redo_only && (status[item] & DGA_ITEM_REDO) == 0) continue;
    const MultiItem mi = work[item];
    const dga_bse_problem d = probs[mi.prob];
    const MultiProblem pb(d, mi);
    const int st = solve_item_fp64<StructuredSource, NT>(pb.src, pb.wi, pb.N, pb.n2, pb.nv, d.beta, pb.o, A, sm, piv);
    __syncthreads();  // every thread has read status[item] before it is rewritten
    if (threadIdx.x == 0) {
      status[item] = st;
      if (iters && !redo_only) iters[item] = 0;
    }
  }
}

template <int NR>
__device__ __forceinline__ int multi_item_mixed(const dga_bse_problem& d, const MultiItem& mi, int n_max, int max_iter,
                                                double tol, unsigned char* slot, unsigned char* smem_raw, int* it) {
  const MultiProblem pb(d, mi);
  BseSmem<float2>& sm = *reinterpret_cast<BseSmem<float2>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(BseSmem<float2>));
  int* perm = piv + n_max;
  double2* colsum = reinterpret_cast<double2*>(smem_raw + mixed_colsum_offset(n_max));
  float2* A = reinterpret_cast<float2*>(slot);
  double2* Y = reinterpret_cast<double2*>(slot + (((size_t)pb.N * pb.N * sizeof(float2) + 255) & ~(size_t)255));
  double2* Rb = Y + (size_t)pb.N * pb.n2;
  return solve_item_mixed<NR>(pb.src, pb.wi, pb.N, pb.nv, d.beta, max_iter, tol, pb.o, A, Y, Rb, sm, piv, perm, colsum,
                              it);
}

// Mixed batch of problems of one orbital count (NR = n_orb^2 > 0), or (NR = 0) of problems that differ in it (the
// 2-orbital bilayer next to a 1-orbital lattice, say), with the right-hand-side count chosen per item.
template <int NR>
__global__ void __launch_bounds__(BSE_THREADS, DGA_MIXED_MIN_BLOCKS)
    bse_multi_mixed_kernel(const dga_bse_problem* __restrict__ probs, const MultiItem* __restrict__ work, int n_items,
                           int n_max, int max_iter, double tol, int* __restrict__ status, int* __restrict__ iters,
                           unsigned char* __restrict__ scratch, size_t slot_bytes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* slot = scratch + (size_t)blockIdx.x * slot_bytes;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const MultiItem mi = work[item];
    const dga_bse_problem d = probs[mi.prob];
    int it = 0, st = 0;
    if constexpr (NR > 0) {
      st = multi_item_mixed<NR>(d, mi, n_max, max_iter, tol, slot, smem_raw, &it);
    } else {
      switch (d.n_orb) {
        case 1: st = multi_item_mixed<1>(d, mi, n_max, max_iter, tol, slot, smem_raw, &it); break;
        case 2: st = multi_item_mixed<4>(d, mi, n_max, max_iter, tol, slot, smem_raw, &it); break;
        case 3: st = multi_item_mixed<9>(d, mi, n_max, max_iter, tol, slot, smem_raw, &it); break;
        default: st = multi_item_mixed<16>(d, mi, n_max, max_iter, tol, slot, smem_raw, &it); break;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      status[item] = st;
      if (iters) iters[item] = it;
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Eliashberg full vertex in the pp frequency box (one CTA per (channel, q, w) item):
//   F[(p,nu),(s,nu')] = beta^2 (delta_{nu nu'} c0(nu)[p][s] - sum_{m,m'} c0(nu)[p][m] chi*[(m,nu),(m',nu')] c0(nu')[m'][s])
//                       + (Z G3(nu) G3(nu'))[p][s],   Z = U_r - U_r chi_r U_r,  c0 = chi0^-1,  G3 = gamma_r
// for nu, nu' in the box [niv - P, niv + P) (eliashberg_solver.py:175-204).  chi* = A^-1 is never formed: the unit vectors
// of the box frequencies are right-hand sides of the LU (their forward substitution runs with the factorisation's block
// rows, all columns at once on the FP64 tensor pipe).
//   g3: [2][Q][W][nv][n2][n2]; chi_phys: [2][Q][W][n2][n2]; out: [2][Q][Wpp][Mb][Mb]
//   slot: A (N x N) | Y (N x Mb) | H (2P x n2 x n2) | Z (n2 x n2), complex128
// ----------------------------------------------------------------------------------------------
// The unit vectors of the box columns: column vb n2 + m' of Y has its one at row (m', off + vb).
inline __device__ void eli_box_columns(int N, int n2, int nv, int P, double2* __restrict__ Y) {
  const int off = nv / 2 - P, Mb = n2 * 2 * P;
  for (int e = threadIdx.x; e < N * Mb; e += blockDim.x) {
    const int i = e % N, col = e / N, vb = col / n2, mp = col - vb * n2;
    Y[e] = make_double2(i == mp * nv + off + vb ? 1.0 : 0.0, 0.0);
  }
}

// beta^2 (delta_{nu nu'} c0(nu)[p][s] - sum_{m,m'} c0(nu)[p][m] chi*[(m,nu),(m',nu')] c0(nu')[m'][s]) with chi* in the box
// columns Y.
__device__ __forceinline__ double2 eli_box_element(const StructuredSource& src, const WorkItem& wi, int W, int n2, int nv,
                                                   int N, int off, int P, double beta2, const double2* Y, int p, int vb,
                                                   int sidx, int vbp) {
  const int vr = off + vb, vc = off + vbp;
  const double2* c0r = src.chi0_inv + (((size_t)wi.q * W + wi.w) * nv + vr) * n2 * n2;
  const double2* c0c = src.chi0_inv + (((size_t)wi.q * W + wi.w) * nv + vc) * n2 * n2;
  double2 t = make_double2(0.0, 0.0);
  for (int m = 0; m < n2; ++m) {
    double2 inner = make_double2(0.0, 0.0);
    for (int mp = 0; mp < n2; ++mp) cfma(inner, Y[(size_t)(vbp * n2 + mp) * N + m * nv + vr], c0c[mp * n2 + sidx]);
    cfma(t, c0r[p * n2 + m], inner);
  }
  double2 f1 = make_double2(-t.x, -t.y);
  if (vb == vbp) f1 = cadd(f1, c0r[p * n2 + sidx]);
  return cscale(f1, beta2);
}

template <int NT>
__global__ void __launch_bounds__(NT, fp64_min_blocks(NT))
    eli_full_vertex_kernel(StructuredSource src, const WorkItem* __restrict__ work, int n_items, int N, int n2, int nv,
                           int W, int Q, int P, int Wpp, double beta, const double2* __restrict__ g3,
                           const double2* __restrict__ chi_phys, double2* __restrict__ out, int* __restrict__ status,
                           double2* __restrict__ scratch, size_t slot_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fp64Smem<NT>& sm = *reinterpret_cast<Fp64Smem<NT>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(Fp64Smem<NT>));
  double2* A = scratch + (size_t)blockIdx.x * slot_elems;
  double2* Y = A + (size_t)N * N;
  const int nvp = 2 * P, Mb = n2 * nvp, off = nv / 2 - P;
  double2* H = Y + (size_t)N * Mb;
  double2* Z = H + (size_t)nvp * n2 * n2;
  const int tid = threadIdx.x, T = blockDim.x;
  const double beta2 = beta * beta;

  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const WorkItem wi = work[item];
    form_item_fp64(src, wi, N, 0, nv, A);
    eli_box_columns(N, n2, nv, P, Y);
    __syncthreads();
    const bool singular = fp64_lu<NT>(A, N, N + Mb, piv, sm);
    fp64_backward<NT>(A, N, Y, Mb, sm);
    // Z = U_r - U_r chi_r U_r, then H(nu) = Z G3(nu) for the box frequencies
    const double2* uvq = src.uv + ((size_t)wi.ch * Q + wi.q) * n2 * n2;
    const double2* cp = chi_phys + (((size_t)wi.ch * Q + wi.q) * W + wi.w) * n2 * n2;
    for (int e = tid; e < n2 * n2; e += T) {
      const int p = e / n2, s = e - p * n2;
      double2 acc = uvq[e];
      for (int t = 0; t < n2; ++t) {
        double2 cu = make_double2(0.0, 0.0);
        for (int u = 0; u < n2; ++u) cfma(cu, cp[t * n2 + u], uvq[u * n2 + s]);
        cfms(acc, uvq[p * n2 + t], cu);
      }
      Z[e] = acc;
    }
    __syncthreads();
    const double2* g3q = g3 + ((((size_t)wi.ch * Q + wi.q) * W + wi.w) * nv) * n2 * n2;
    for (int e = tid; e < nvp * n2 * n2; e += T) {
      const int vb = e / (n2 * n2), ps = e - vb * n2 * n2, p = ps / n2, s = ps - p * n2;
      const double2* g = g3q + (size_t)(off + vb) * n2 * n2;
      double2 acc = make_double2(0.0, 0.0);
      for (int t = 0; t < n2; ++t) cfma(acc, Z[p * n2 + t], g[t * n2 + s]);
      H[e] = acc;
    }
    __syncthreads();
    double2* o = out + (((size_t)wi.ch * Q + wi.q) * Wpp + wi.w) * (size_t)Mb * Mb;
    for (int e = tid; e < Mb * Mb; e += T) {
      const int sidx = e % n2, vbp = (e / n2) % nvp, row = e / Mb;
      const int p = row / nvp, vb = row - p * nvp, vc = off + vbp;
      const double2 f1 = eli_box_element(src, wi, W, n2, nv, N, off, P, beta2, Y, p, vb, sidx, vbp);
      // (Z G3(nu)) G3(nu')
      const double2* hrow = H + (size_t)vb * n2 * n2 + p * n2;
      const double2* gcol = g3q + (size_t)vc * n2 * n2;
      double2 f2 = make_double2(0.0, 0.0);
      for (int u = 0; u < n2; ++u) cfma(f2, hrow[u], gcol[u * n2 + sidx]);
      o[(size_t)row * Mb + sidx * nvp + vbp] = cadd(f1, f2);
    }
    __syncthreads();
    if (tid == 0 && status) status[item] = singular ? DGA_ITEM_SINGULAR : 0;
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------------------------
// Dense batched LU and solves with many right-hand sides (the local Schwinger-Dyson equation's full inverses,
// numpy.linalg.inv behind LocalFourPoint.invert, local_four_point.py:298-310).  The factorisation is lu_factor_dmma
// (LAPACK's pivot order) with one CTA per matrix, lu_factor beyond N = 2048; the solves spread over (matrix, block of
// DENSE_COLS or DENSE_RHS right-hand sides) CTAs, each streaming the factors once for its block.
// ----------------------------------------------------------------------------------------------
constexpr int DENSE_RHS = 16;   // right-hand sides are padded to a multiple of this; columns a CTA solves by rows
constexpr int DENSE_COLS = 64;  // columns a CTA solves with 16 a warp

template <int NT>
__global__ void __launch_bounds__(NT, fp64_min_blocks(NT))
    dense_lu_kernel(double2* __restrict__ a, int N, int n_mat, long long mat_stride, int* __restrict__ piv_out,
                    int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fp64Smem<NT>& sm = *reinterpret_cast<Fp64Smem<NT>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(Fp64Smem<NT>));
  for (int m = blockIdx.x; m < n_mat; m += gridDim.x) {
    const bool singular = fp64_lu<NT>(a + (size_t)m * mat_stride, N, N, piv, sm);
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += NT) piv_out[(size_t)m * N + i] = piv[i];
    if (threadIdx.x == 0) status[m] = singular ? DGA_ITEM_SINGULAR : DGA_ITEM_OK;
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------------------------
// Eliashberg full vertex fused into the FP64 BSE (eliashberg_solver.py:175-204): an item with w < Wpp keeps its LU
// factors after the selector solve and solves the unit vectors of the pp box with them, writing
//   f1[(p,nu),(s,nu')] = beta^2 (delta_{nu nu'} c0(nu)[p][s] - sum_{m,m'} c0(nu)[p][m] chi*[(m,nu),(m',nu')] c0(nu')[m'][s])
// for nu, nu' in [niv - P, niv + P).  The ladder term (Z G3(nu) G3(nu'), which needs the lambda-corrected chi_r and
// the three-leg vertex of the whole pass) is added afterwards by eli_ladder_term_kernel; f1 + term is the sum
// eli_full_vertex_kernel forms, in the same order, from the same factors.
// ----------------------------------------------------------------------------------------------
// FP64 BSE (as bse_solve_sum_fp64_kernel) with the pp-box epilogue for items w < Wpp.  out_pp: [2][Q][Wpp][Mb][Mb].
template <int NT>
__global__ void __launch_bounds__(NT, fp64_min_blocks(NT))
    bse_fp64_eli_kernel(StructuredSource src, const WorkItem* __restrict__ work, int n_items, int N, int n2, int nv,
                        int W, int Q, double beta, double2* __restrict__ out, int P, int Wpp,
                        double2* __restrict__ out_pp, int* __restrict__ status, double2* __restrict__ scratch,
                        size_t slot_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fp64Smem<NT>& sm = *reinterpret_cast<Fp64Smem<NT>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(Fp64Smem<NT>));
  double2* A = scratch + (size_t)blockIdx.x * slot_elems;
  double2* Y = A + (size_t)N * (N + n2);
  const int nvp = 2 * P, Mb = n2 * nvp;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const WorkItem wi = work[item];
    double2* o = out + (((size_t)wi.ch * Q + wi.q) * W + wi.w) * (size_t)N * n2;
    const bool box = wi.w < Wpp;
    if (box) eli_box_columns(N, n2, nv, P, Y);
    const int st =
        solve_item_fp64<StructuredSource, NT>(src, wi, N, n2, nv, beta, o, A, sm, piv, box ? Mb : 0);
    if (box) {
      fp64_backward<NT>(A, N, Y, Mb, sm);
      double2* opp = out_pp + (((size_t)wi.ch * Q + wi.q) * Wpp + wi.w) * (size_t)Mb * Mb;
      for (int e = threadIdx.x; e < Mb * Mb; e += NT) {
        const int sidx = e % n2, vbp = (e / n2) % nvp, row = e / Mb;
        const int p = row / nvp, vb = row - p * nvp;
        opp[(size_t)row * Mb + sidx * nvp + vbp] =
            eli_box_element(src, wi, W, n2, nv, N, nv / 2 - P, P, beta * beta, Y, p, vb, sidx, vbp);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0 && status) status[item] = st;
  }
}


#define DGA_FP64_KERNELS(PREFIX, NT)                                                                                    \
  PREFIX __global__ void bse_solve_sum_fp64_kernel<StructuredSource, NT>(                                               \
      StructuredSource, const WorkItem* __restrict__, int, int, int, int, int, int, double, double2* __restrict__,      \
      int* __restrict__, double2* __restrict__, size_t, int);                                                           \
  PREFIX __global__ void bse_solve_sum_fp64_kernel<DenseSource, NT>(                                                    \
      DenseSource, const WorkItem* __restrict__, int, int, int, int, int, int, double, double2* __restrict__,           \
      int* __restrict__, double2* __restrict__, size_t, int);                                                           \
  PREFIX __global__ void bse_multi_fp64_kernel<NT>(const dga_bse_problem* __restrict__, const MultiItem* __restrict__,  \
                                                   int, int, int* __restrict__, int* __restrict__,                      \
                                                   unsigned char* __restrict__, size_t, int);                           \
  PREFIX __global__ void eli_full_vertex_kernel<NT>(                                                                    \
      StructuredSource, const WorkItem* __restrict__, int, int, int, int, int, int, int, int, double,                   \
      const double2* __restrict__, const double2* __restrict__, double2* __restrict__, int* __restrict__,               \
      double2* __restrict__, size_t);                                                                                   \
  PREFIX __global__ void dense_lu_kernel<NT>(double2* __restrict__, int, int, long long, int* __restrict__,             \
                                             int* __restrict__);                                                        \
  PREFIX __global__ void bse_fp64_eli_kernel<NT>(                                                                       \
      StructuredSource, const WorkItem* __restrict__, int, int, int, int, int, int, double, double2* __restrict__, int, \
      int, double2* __restrict__, int* __restrict__, double2* __restrict__, size_t);

}  // namespace dga
