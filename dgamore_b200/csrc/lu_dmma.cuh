// FP64 complex LU with partial pivoting of one matrix by one CTA, Crout order, products on the FP64 tensor pipe.
//
// The matrix is column-major in the CTA's scratch (or any global memory); the result has LAPACK's layout (unit lower L
// below the diagonal, U on and above, piv[j] = the row exchanged with row j) and its pivots (largest |re| + |im|, first
// index on ties), as lu_factor's.
//
// Why Crout order: a right-looking update reads and writes the whole trailing matrix once per 32 columns (2/3 N^3 / 32
// elements read and written, 248 MB at N = 720 with the factor tiles); here a block column and a block row are
// accumulated in registers over everything to their left and above and written once, so the same products cost
// reads only (62 MB by count at N = 720; a whole item of the BSE moves 123 MB of DRAM, 173 before), and a CTA needs no
// shared-memory tiles or barriers inside them.
//
// Why mma.sync f64: the FP64 tensor pipe and the FP64 vector pipe have the same peak (37 TFLOP/s measured for either),
// but an m16n8k4 product takes one warp instruction where the vector pipe takes 16, and its A and B fragments of an
// interleaved complex matrix are one 16-byte load per lane each (lane (g, t) holds row g and column t), so operands come
// straight from L2 and L1: four warps per SM already reach 35 TFLOP/s. The tcgen05 pipe has no FP64 kind.
//
// What bounds it: the products at N = 720 (592 factorisations in 28.1 ms, 21.0 TFLOP/s, two CTAs an SM), waits on HBM and
// L2 for the panels and the tiles' first elements below about N = 250 (14,208 of N = 120 in 6.8 ms, 9.6 TFLOP/s).
#pragma once

#include "dga_common.cuh"
#include "tc_tile.cuh"

namespace dga {

constexpr int LU_MAX_N = 2048;
constexpr int LU_RING = 4;  // steps of four columns a lane has in flight

// Block width by the matrix size alone, so that a matrix goes through the same operations whatever CTA it is given. 16 up
// to N = 192, where one or two warps take a matrix and 16 or 8 matrices share an SM (the shared memory of a 32-wide block
// would admit five): the panels' chains of dependent steps, not the products, are what the time goes to. 29,600
// factorisations of N = 40 take 1.45 ms, 2.79 in CTAs of 128 threads and 3.01 at 32 wide too; 9,472 of N = 160 8.2 against
// 9.2; with many right-hand sides the wider block is the faster one from N = 240 (154 against 162 ms for the
// bilayer pass with its pairing box).
constexpr int LU_SMALL_N = 192;

// Panel columns a thread can keep in registers with RPT rows (at most 16 complex values, 64 registers), and the columns
// that are factored at a time: by the matrix size and the rows left alone, within what every thread count can keep there.
template <int RPT>
struct LuPanelWidth {
  static constexpr int value = RPT <= 2 ? 8 : RPT <= 4 ? 4 : 2;
};
__device__ __forceinline__ int lu_panel_width(int N, int m) {
  const int rows = N <= LU_SMALL_N ? 64 : N <= 512 ? 128 : 256;  // the smallest thread count that takes N
  return m <= 2 * rows ? 8 : m <= 4 * rows ? 4 : 2;
}

constexpr int LU_WARP_BUF = LU_RING * 2 * 33;

template <int NT, int NB>
struct LuSmem {
  double2 L11i[NB][NB + 1];  // inverse of the diagonal block's triangle
  union {
    double2 L11[NB][NB + 1];  // the triangle itself, dead once it is inverted
    // per warp: each lane's fragments of the streamed factor on their way from HBM ([LU_RING][2][33]), then 8 columns of the
    // block row before the triangular solve ([8][NB + 1])
    double2 warp[NT / 32][LU_WARP_BUF];
  };
  double2 us[8][NB];               // panel: rows of U of the columns just factored
  double2 cand[2][NT / 32][10];    // panel: each warp's candidate pivot row, conj(pivot), 1 / |pivot|^2
  __align__(16) unsigned long long key[2][(NT / 32 + 1) / 2 * 2];
  int flag;
};

__device__ __forceinline__ void cp_async16(double2* smem, const double2* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}
// fill: 16 bytes of zeros in place of the source where false
__device__ __forceinline__ void cp_async16_or_zero(double2* smem, const double2* g, bool fill) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g),
               "r"(fill ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void prefetch_l1(const double2* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// c += a b for a 16 x 4 a (rows g, g + 8), 4 x 8 b, 16 x 8 c
__device__ __forceinline__ void dmma_16x8x4(double (&c)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// Complex 16 x 8 accumulator: element (g + 8 (i / 2), 2 t + i % 2) in re[i], im[i].
struct CAcc {
  double re[4], im[4];
};

// a b with one rounding order everywhere: left to the compiler, the contraction may differ between kernels that must give
// the same bits
__device__ __forceinline__ double2 cmul_fma(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}

// c[n] += a b[n] on complex fragments: the products with Re a first, then those with Im a (one negated copy)
template <int NTILE>
__device__ __forceinline__ void cdmma_row(CAcc* c, double2 a0, double2 a1, const double2* b) {
#pragma unroll
  for (int n = 0; n < NTILE; ++n) {
    dmma_16x8x4(c[n].re, a0.x, a1.x, b[n].x);
    dmma_16x8x4(c[n].im, a0.x, a1.x, b[n].y);
  }
  const double m0 = -a0.y, m1 = -a1.y;
#pragma unroll
  for (int n = 0; n < NTILE; ++n) {
    dmma_16x8x4(c[n].re, m0, m1, b[n].y);
    dmma_16x8x4(c[n].im, a0.y, a1.y, b[n].x);
  }
}

// Block column: A[j0.., j0 .. j0+nb) -= A[j0.., 0..j0) A[0..j0, j0 .. j0+nb). One warp per 16 rows x NB columns; rows and
// columns past the end read the last valid ones and are not stored. L streams from HBM (the matrices in flight are twice
// L2 at N = 120 and twenty times at N = 720): a lane copies the two elements it multiplies three steps later, 1,500 cycles of the FP64 pipe at NB = 32, into its own
// ring slot, so nothing has to be synchronised; U is shared by all warps and comes from L1, one step ahead.
template <int NT, int NB>
__device__ void lu_block_column(double2* __restrict__ A, int N, int ld, int j0, int nb, LuSmem<NT, NB>& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int tiles = (N - j0 + 15) / 16;
  double2(*ring)[2][33] = reinterpret_cast<double2(*)[2][33]>(sm.warp[warp]);
  constexpr int NTN = NB / 8;
  int ob[NTN];
#pragma unroll
  for (int nt = 0; nt < NTN; ++nt) ob[nt] = min(j0 + nt * 8 + g, N - 1) * ld + t;
  for (int tile = warp; tile < tiles; tile += NT / 32) {
    const int r0 = j0 + tile * 16 + g, r1 = r0 + 8;
    CAcc acc[NTN];
#pragma unroll
    for (int nt = 0; nt < NTN; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[nt].re[i] = acc[nt].im[i] = 0.0;
    const int d1 = min(r1, N - 1) - min(r0, N - 1), step = 4 * ld;
    const double2* pa = A + t * ld + min(r0, N - 1);
    // the tile itself, read after the products: 256 bytes a column, one 128-byte line a lane
    for (int e = lane; e < 2 * nb; e += 32) prefetch_l1(A + (size_t)(j0 + e / 2) * ld + min(j0 + tile * 16 + (e & 1) * 8, N - 1));
#pragma unroll
    for (int u = 0; u < LU_RING - 1; ++u) {  // j0 >= 16: at least four steps
      cp_async16(&ring[u][0][lane], pa);
      cp_async16(&ring[u][1][lane], pa + d1);
      cp_async_commit();
      pa += step;
    }
    double2 b[NTN];
#pragma unroll
    for (int nt = 0; nt < NTN; ++nt) b[nt] = A[ob[nt]];
    int slot = 0;
    for (int k = 0; k < j0; k += 4) {
      cp_async_wait<LU_RING - 2>();
      const double2 x0 = ring[slot][0][lane], x1 = ring[slot][1][lane];
      const int next = (slot + LU_RING - 1) % LU_RING;
      if (k + 4 * (LU_RING - 1) < j0) {
        cp_async16(&ring[next][0][lane], pa);
        cp_async16(&ring[next][1][lane], pa + d1);
        pa += step;
      }
      cp_async_commit();
      slot = (slot + 1) % LU_RING;
      double2 y[NTN];
#pragma unroll
      for (int nt = 0; nt < NTN; ++nt) y[nt] = b[nt];
      if (k + 4 < j0) {
#pragma unroll
        for (int nt = 0; nt < NTN; ++nt) b[nt] = A[ob[nt] + k + 4];
      }
      cdmma_row<NTN>(acc, x0, x1, y);
    }
#pragma unroll
    for (int nt = 0; nt < NTN; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = nt * 8 + 2 * t + (i & 1), r = i < 2 ? r0 : r1;
        if (c < nb && r < N) {
          double2* e = A + (size_t)(j0 + c) * ld + r;
          *e = make_double2(e->x - acc[nt].re[i], e->y - acc[nt].im[i]);
        }
      }
  }
}

// Block row of ncols columns Y (leading dimension ldy; the matrix's own to the right of the block, or right-hand sides):
//   Y[j0..j0+nb) = T^-1 (Y[j0..j0+nb) - A[j0..j0+nb, k0..k1) Y[k0..k1)),   T^-1 in sm.L11i.
// UPPER false: T = L11, k0 = 0, k1 = j0 (the factorisation's block row, forward substitution); UPPER true: T = U11,
// k0 = j0 + nb, k1 = N (backward substitution). One warp per NB rows x 16 columns: Y streams through the ring, the rows of
// A are shared by all warps and come from L1. Rows past nb count as zero, columns past ncols read the last one and are
// not stored.
template <int NT, int NB, bool UPPER>
__device__ void lu_block_row(const double2* __restrict__ A, int N, int ld, int j0, int nb, int k0, int k1, double2* Y,
                             int ldy, int ncols, LuSmem<NT, NB>& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  constexpr int MT = NB / 16;
  const int tiles = (ncols + 15) / 16, steps = (k1 - k0 + 3) / 4;
  for (int tile = warp; tile < tiles; tile += NT / 32) {
    const int c0 = tile * 16;
    CAcc acc[MT][2];  // [16-row half][8-column half]
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[mt][nt].re[i] = acc[mt][nt].im[i] = 0.0;
    if (steps > 0) {
      double2(*ring)[2][33] = reinterpret_cast<double2(*)[2][33]>(sm.warp[warp]);
      const double2* pb = Y + (size_t)min(c0 + g, ncols - 1) * ldy + k0 + t;
      const size_t d1 = (size_t)(min(c0 + 8 + g, ncols - 1) - min(c0 + g, ncols - 1)) * ldy;
      int left = k1 - k0 - t;  // rows of Y from this lane's on; past the end they count as zero
      __syncwarp();  // the ring shares its memory with the previous tile's columns
      // only what a step will wait for: a copy still on its way after the last step would land in the columns below
#pragma unroll
      for (int u = 0; u < LU_RING - 1; ++u) {
        if (u < steps) {
          const bool in = left > 0;
          cp_async16_or_zero(&ring[u][0][lane], in ? pb : Y, in);
          cp_async16_or_zero(&ring[u][1][lane], in ? pb + d1 : Y, in);
          pb += 4;
          left -= 4;
        }
        cp_async_commit();
      }
      int ra[2 * MT], ca = k0 + t;
#pragma unroll
      for (int u = 0; u < 2 * MT; ++u) ra[u] = min(j0 + g + u * 8, N - 1);
      double2 a[2 * MT];
#pragma unroll
      for (int u = 0; u < 2 * MT; ++u) a[u] = A[min(ca, N - 1) * ld + ra[u]];
      int slot = 0;
      for (int s = 0; s < steps; ++s) {
        cp_async_wait<LU_RING - 2>();
        const double2 y[2] = {ring[slot][0][lane], ring[slot][1][lane]};
        const int next = (slot + LU_RING - 1) % LU_RING;
        if (s + LU_RING - 1 < steps) {
          const bool in = left > 0;
          cp_async16_or_zero(&ring[next][0][lane], in ? pb : Y, in);
          cp_async16_or_zero(&ring[next][1][lane], in ? pb + d1 : Y, in);
          pb += 4;
          left -= 4;
        }
        cp_async_commit();
        slot = (slot + 1) % LU_RING;
        double2 x[2 * MT];
#pragma unroll
        for (int u = 0; u < 2 * MT; ++u) x[u] = a[u];
        if (s + 1 < steps) {
          ca += 4;
#pragma unroll
          for (int u = 0; u < 2 * MT; ++u) a[u] = A[min(ca, N - 1) * ld + ra[u]];
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) cdmma_row<2>(acc[mt], x[2 * mt], x[2 * mt + 1], y);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      double2(*w)[NB + 1] = reinterpret_cast<double2(*)[NB + 1]>(sm.warp[warp]);
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = min(c0 + nt * 8 + 2 * t + (i & 1), ncols - 1), r = mt * 16 + g + (i < 2 ? 0 : 8);
          double2 v = make_double2(0.0, 0.0);
          if (r < nb) {
            v = Y[(size_t)c * ldy + j0 + r];
            v = make_double2(v.x - acc[mt][nt].re[i], v.y - acc[mt][nt].im[i]);
          }
          w[2 * t + (i & 1)][r] = v;
        }
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        CAcc x[1];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[0].re[i] = x[0].im[i] = 0.0;
        const int from = UPPER ? mt * 16 : 0, to = UPPER ? NB : mt * 16 + 16;
#pragma unroll 2
        for (int k = from; k < to; k += 4) {
          const double2 y[1] = {w[g][k + t]};
          cdmma_row<1>(x, sm.L11i[mt * 16 + g][k + t], sm.L11i[mt * 16 + g + 8][k + t], y);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = c0 + nt * 8 + 2 * t + (i & 1), r = mt * 16 + g + (i < 2 ? 0 : 8);
          if (c < ncols && r < nb) Y[(size_t)c * ldy + j0 + r] = make_double2(x[0].re[i], x[0].im[i]);
        }
      }
    }
  }
}

// sum over k < n of a(k) b(k) in four partial sums (a quarter of the dependent chain)
template <typename FA, typename FB>
__device__ __forceinline__ double2 cdot4(int n, FA a, FB b) {
  double2 s[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) s[u] = make_double2(0.0, 0.0);
  for (int k = 0; k < n; k += 4)
#pragma unroll
    for (int u = 0; u < 4; ++u) cfma(s[u], a(k + u), b(k + u));
  return cadd(cadd(s[0], s[1]), cadd(s[2], s[3]));
}

constexpr unsigned long long LU_INF_BITS = 0x7ff0000000000000ull;

// Pivot candidates are compared as integers: the 64 bits of |re| + |im| (a non-negative double orders as an integer does)
// plus one, then the position, the first one largest, as LAPACK takes them. Integers keep the search off the FP64 pipe,
// where each comparison would wait behind the products of the other warps. 0: no candidate (a NaN is none).
__device__ __forceinline__ unsigned long long lu_key(double2 a) {
  const unsigned long long x = __double_as_longlong(cabs1(a));
  return x > LU_INF_BITS ? 0 : x + 1;
}

__device__ __forceinline__ int lu_cand_at(const double2* cand) { return __double2loint(cand[9].y); }

__device__ __forceinline__ unsigned long long warp_max(unsigned long long key) {
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)key : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

// Division by a pivot d: a conj(d) / |d|^2 with 1 / |d|^2 by two Newton-Raphson steps from a single-precision
// reciprocal (a chain of seven FP64 operations; Smith's quotient has about thirty), within a few ulp; pivots outside
// 2^-60 .. 2^60, whose square the seed could not hold, take Smith's reciprocal.
__device__ __forceinline__ void pivot_recip(double2 d, double2& c, double& s) {
  const int e = max((__double2hiint(d.x) >> 20) & 0x7ff, (__double2hiint(d.y) >> 20) & 0x7ff);
  const double q = fma(d.x, d.x, d.y * d.y);
  float seed;
  asm("rcp.approx.f32 %0, %1;" : "=f"(seed) : "f"((float)q));
  double r = (double)seed;
  r = fma(r, fma(-q, r, 1.0), r);
  s = fma(r, fma(-q, r, 1.0), r);
  c = make_double2(d.x, -d.y);
  if ((unsigned)(e - (1023 - 60)) >= 120u && (d.x != 0.0 || d.y != 0.0)) {
    s = 1.0;
    c = crecip(d);
  }
}

// y = L^-1 y for the leading n x n unit lower triangle at L (row pitch LD); a rotating loop, as in the panel
template <int PW, int LD>
__device__ __forceinline__ void unit_lower_solve(double2 (&y)[PW], int n, const double2* L) {
#pragma unroll 1
  for (int k = 0; k < PW; ++k) {
    const double2 yk = y[0];
#pragma unroll
    for (int r = 1; r < PW; ++r)
      if (k + r < n) cfms(y[r], L[(k + r) * LD + k], yk);
#pragma unroll
    for (int r = 0; r + 1 < PW; ++r) y[r] = y[r + 1];
    y[PW - 1] = yk;
  }
}

// sm.L11i = inverse of the unit lower NB x NB block in sm.L11 by doubling: its 8 x 8 diagonal blocks by substitution (one
// thread per column), then [A 0; B C]^-1 = [A^-1 0; -C^-1 B A^-1 C^-1] at 16 (and 32).
template <int NT, int NB>
__device__ void lu_unit_lower_inverse(LuSmem<NT, NB>& sm) {
  const int tid = threadIdx.x;
  for (int e = tid; e < NB * NB; e += NT) {
    const int r = e % NB, c = e / NB;
    if ((r ^ c) & ~7) sm.L11i[r][c] = make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (tid < NB) {
    const int o = tid & ~7, c = tid & 7;
    double2 y[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) y[r] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    unit_lower_solve<8, NB + 1>(y, 8, &sm.L11[o][o]);
#pragma unroll
    for (int r = 0; r < 8; ++r) sm.L11i[o + r][o + c] = y[r];
  }
  __syncthreads();
  double2* tmp = &sm.us[0][0];  // B A^-1, at most 16 x 16
#pragma unroll
  for (int h = 8; h < NB; h *= 2) {
    const int n = NB / 2 * h;
    for (int e = tid; e < n; e += NT) {
      const int b = e / (h * h), r = (e / h) % h, c = e % h, o = b * 2 * h;
      tmp[e] = cdot4(h, [&](int k) { return sm.L11[o + h + r][o + k]; }, [&](int k) { return sm.L11i[o + k][o + c]; });
    }
    __syncthreads();
    for (int e = tid; e < n; e += NT) {
      const int b = e / (h * h), r = (e / h) % h, c = e % h, o = b * 2 * h;
      const double2 v = cdot4(h, [&](int k) { return sm.L11i[o + h + r][o + h + k]; },
                              [&](int k) { return tmp[b * h * h + k * h + c]; });
      sm.L11i[o + h + r][o + c] = make_double2(-v.x, -v.y);
    }
    __syncthreads();
  }
}

// Panel: factors the columns [j0, j0 + nb) of the rows j0.. with partial pivoting, PW columns at a time in registers (a
// thread holds the rows j0 + tid + NT i). A row keeps its registers when it is exchanged; only its position changes, and
// the columns are written back at the new positions. One barrier per column: each warp offers its best row with its
// reciprocal already taken, every thread picks the winner. The PW columns are then applied to the rest of the block, whose
// interchanges are made here; the columns outside it follow in lu_interchange. Returns true if
// an exact zero pivot was met.
template <int NT, int NB, int RPT>
__device__ bool lu_panel(double2* __restrict__ A, int N, int ld, int j0, int nb, int* __restrict__ piv,
                         LuSmem<NT, NB>& sm) {
  constexpr int PW = LuPanelWidth<RPT>::value, NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool singular = false;
  const int width = lu_panel_width(N, N - j0);  // <= PW
  for (int p0 = 0; p0 < nb; p0 += width) {
    const int pw = min(width, nb - p0), jc = j0 + p0;
    double2* P = A + (size_t)jc * ld;
    double2 a[RPT][PW];
    int pos[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      pos[i] = j0 + tid + NT * i;
      if (pos[i] < jc) pos[i] = N;  // already a pivot row of this block
#pragma unroll
      for (int c = 0; c < PW; ++c)
        a[i][c] = (pos[i] < N && c < pw) ? P[(size_t)c * ld + pos[i]] : make_double2(0.0, 0.0);
    }
    bool exchanged = false;
    // One loop body serves every column, so that it stays in the instruction cache (unrolled, the fetches took longer than
    // the arithmetic): the registers rotate, the current column is always a[i][0], and after PW steps they are in place.
#pragma unroll 1
    for (int jj = 0; jj < PW; ++jj) {
      if (jj < pw) {
        const int j = jc + jj, buf = jj & 1;
        unsigned long long own = 0;
        int at = N;
        double2 d = make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const unsigned long long x = (pos[i] >= j && pos[i] < N) ? lu_key(a[i][0]) : 0;
          if (x > own || (x == own && pos[i] < at)) {
            own = x;
            at = pos[i];
            d = a[i][0];
          }
        }
        double2 rc;
        double rs;
        pivot_recip(d, rc, rs);
        unsigned long long key = warp_max(own);
        bool offer = own == key;
        if (__popc(__ballot_sync(0xffffffffu, offer)) > 1) {  // a tie: the first row (the whole warp takes the reduction)
          const unsigned first = __reduce_min_sync(0xffffffffu, offer ? (unsigned)at : 0xffffffffu);
          offer = (unsigned)at == first;
        }
        if (offer && key) {
#pragma unroll
          for (int i = 0; i < RPT; ++i)
            if (pos[i] == at) {
#pragma unroll
              for (int c = 0; c < PW; ++c) sm.cand[buf][warp][c] = a[i][c];
            }
          sm.cand[buf][warp][8] = rc;
          sm.cand[buf][warp][9] = make_double2(rs, __hiloint2double(0, at));
        }
        if (lane == 0) sm.key[buf][warp] = key;
        __syncthreads();
        int win = 0;
        if constexpr (NW > 1) {
          const ulonglong2* keys = reinterpret_cast<const ulonglong2*>(sm.key[buf]);
          key = 0;
          bool tie = false;
#pragma unroll
          for (int w = 0; w < NW / 2; ++w) {
            const ulonglong2 x = keys[w];
            const unsigned long long m = x.x > x.y ? x.x : x.y;
            const bool more = m > key;
            tie = more ? x.x == x.y : tie || m == key;
            win = more ? 2 * w + (x.y > x.x) : win;
            key = more ? m : key;
          }
          if (tie && key) {
#pragma unroll 1
            for (int w = win + 1; w < NW; ++w)
              if (sm.key[buf][w] == key && lu_cand_at(sm.cand[buf][w]) < lu_cand_at(sm.cand[buf][win])) win = w;
          }
        }
        int p = lu_cand_at(sm.cand[buf][win]);
        if (key == 0) {  // no comparable entry (every one is NaN): the diagonal row stays
          p = j;
          win = 0;
#pragma unroll
          for (int i = 0; i < RPT; ++i)
            if (pos[i] == p) {
#pragma unroll
              for (int c = 0; c < PW; ++c) sm.cand[buf][0][c] = a[i][c];
              sm.cand[buf][0][8] = make_double2(a[i][0].x, -a[i][0].y);  // NaN either way
              sm.cand[buf][0][9].x = 1.0;
            }
          __syncthreads();
        }
        const double2* row = sm.cand[buf][win];
        const double2 cd = row[8];
        const double cs = row[9].x;
        const bool zero = row[0].x == 0.0 && row[0].y == 0.0;
        singular |= zero;
        if (tid == 0) piv[j] = p;
        exchanged |= p != j;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          if (pos[i] == p)
            pos[i] = j;
          else if (pos[i] == j)
            pos[i] = p;
          if (pos[i] > j && pos[i] < N) {
            if (!zero) a[i][0] = cscale(cmul_fma(a[i][0], cd), cs);
#pragma unroll
            for (int c = 1; c < PW; ++c)
              if (c < PW - jj) cfms(a[i][c], a[i][0], row[c]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const double2 first = a[i][0];
#pragma unroll
        for (int c = 0; c + 1 < PW; ++c) a[i][c] = a[i][c + 1];
        a[i][PW - 1] = first;
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      if (pos[i] >= N) continue;
#pragma unroll
      for (int c = 0; c < PW; ++c)
        if (c < pw) P[(size_t)c * ld + pos[i]] = a[i][c];
      if (pos[i] < jc + pw) {
#pragma unroll
        for (int c = 0; c < PW; ++c)
          if (jc + c < pos[i]) sm.L11[pos[i] - j0][p0 + c] = a[i][c];
      }
    }
    __syncthreads();
    if (exchanged) {
      for (int c = tid; c < nb - pw; c += NT) {
        double2* col = A + (size_t)(j0 + (c < p0 ? c : c + pw)) * ld;
        for (int jj = 0; jj < pw; ++jj) {
          const int p = piv[jc + jj];
          if (p != jc + jj) {
            const double2 x = col[jc + jj];
            col[jc + jj] = col[p];
            col[p] = x;
          }
        }
      }
      __syncthreads();
    }
    const int rest = nb - p0 - pw;
    if (rest > 0) {
      // the pivot rows in the block's remaining columns: U = L^-1 A with the PW x PW unit lower triangle
      for (int c = tid; c < rest; c += NT) {
        double2* col = P + (size_t)(pw + c) * ld + jc;
        double2 y[PW];
#pragma unroll
        for (int r = 0; r < PW; ++r) y[r] = r < pw ? col[r] : make_double2(0.0, 0.0);
        unit_lower_solve<PW, NB + 1>(y, pw, &sm.L11[p0][p0]);
#pragma unroll
        for (int r = 0; r < PW; ++r)
          if (r < pw) {
            col[r] = y[r];
            sm.us[r][c] = y[r];
          }
      }
      __syncthreads();
      // and applied to the rows below, 16 rows x 8 columns at a time on the tensor pipe (row by row on the vector pipe the
      // update was a third of the panel: each of its many instructions waits behind the other matrices' products)
      const int first = jc + pw, tiles = (N - first + 15) / 16, g = lane >> 2, t = lane & 3;
      for (int tile = warp; tile < tiles; tile += NW) {
        const int r0 = first + tile * 16 + g, r1 = r0 + 8;
        const double2 *l0 = P + min(r0, N - 1), *l1 = P + min(r1, N - 1);
        double2 x0[2], x1[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const bool in = h * 4 + t < pw;
          x0[h] = in ? l0[(size_t)(h * 4 + t) * ld] : make_double2(0.0, 0.0);
          x1[h] = in ? l1[(size_t)(h * 4 + t) * ld] : make_double2(0.0, 0.0);
        }
#pragma unroll 1
        for (int c0 = 0; c0 < rest; c0 += 8) {
          double2 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int c = c0 + 2 * t + (i & 1), r = i < 2 ? r0 : r1;
            v[i] = (c < rest && r < N) ? P[(size_t)(pw + c) * ld + r] : make_double2(0.0, 0.0);
          }
          CAcc acc[1];
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[0].re[i] = acc[0].im[i] = 0.0;
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (h * 4 < pw) {
              const double2 y[1] = {h * 4 + t < pw ? sm.us[h * 4 + t][c0 + g] : make_double2(0.0, 0.0)};
              cdmma_row<1>(acc, x0[h], x1[h], y);
            }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int c = c0 + 2 * t + (i & 1), r = i < 2 ? r0 : r1;
            if (c < rest && r < N)
              P[(size_t)(pw + c) * ld + r] = make_double2(v[i].x - acc[0].re[i], v[i].y - acc[0].im[i]);
          }
        }
      }
      __syncthreads();
    }
  }
  return singular;
}

// sm.L11i = L11^-1 of the factored nb x nb diagonal block at j0, as an NB x NB unit lower triangle (identity past nb).
template <int NT, int NB>
__device__ void lu_invert_lower(const double2* __restrict__ A, int ld, int j0, int nb, LuSmem<NT, NB>& sm) {
  const int tid = threadIdx.x;
  for (int e = tid; e < NB * NB; e += NT) {
    const int r = e % NB, c = e / NB;
    if (r > c) sm.L11[r][c] = r < nb ? A[(size_t)(j0 + c) * ld + j0 + r] : make_double2(0.0, 0.0);
  }
  lu_unit_lower_inverse<NT, NB>(sm);
}

// sm.L11i = U11^-1 of the diagonal block (zero past nb): with D its diagonal, U11^-1 = ((D^-1 U11)^T)^-T D^-1, so that the
// same unit lower inverse serves.
template <int NT, int NB>
__device__ void lu_invert_upper(const double2* __restrict__ A, int ld, int j0, int nb, LuSmem<NT, NB>& sm) {
  const int tid = threadIdx.x;
  double2* dinv = &sm.cand[0][0][0];
  if (tid < NB) dinv[tid] = tid < nb ? crecip(A[(size_t)(j0 + tid) * ld + j0 + tid]) : make_double2(0.0, 0.0);
  __syncthreads();
  for (int e = tid; e < NB * NB; e += NT) {
    const int c = e % NB, r = e / NB;  // U11[c][r], c < r
    if (r > c) sm.L11[r][c] = r < nb ? cmul_fma(A[(size_t)(j0 + r) * ld + j0 + c], dinv[c]) : make_double2(0.0, 0.0);
  }
  lu_unit_lower_inverse<NT, NB>(sm);
  for (int e = tid; e < NB * NB; e += NT) {
    const int i = e % NB, j = e / NB;
    if (i < j) {
      sm.L11i[i][j] = cmul_fma(sm.L11i[j][i], dinv[j]);
      sm.L11i[j][i] = make_double2(0.0, 0.0);
    } else if (i == j) {
      sm.L11i[i][i] = dinv[i];
    }
  }
  __syncthreads();
}

// The block's row interchanges on the columns outside it, a thread per column: one interchange after the other over all
// columns when they are independent pairs (every pivot row below the block, no two alike), else all of a column's in turn;
// nothing to do when no row moved. (One loop in order for every case: 3,552 of N = 240 whose rows all move take 15.8 ms
// instead of 14.9; a thread per pair and column, four in flight: 82 of N = 720 13.6 instead of 12.9.)
template <int NT, int NB>
__device__ void lu_interchange(double2* __restrict__ A, int ncols, int ld, int j0, int nb, const int* __restrict__ piv,
                               LuSmem<NT, NB>& sm) {
  const int tid = threadIdx.x, k1 = j0 + nb;
  if (tid < 32) {
    bool alone = true, moved = false;
    if (tid < nb) {
      const int p = piv[j0 + tid];
      moved = p != j0 + tid;
      if (moved) {
        if (p < k1) alone = false;
        for (int o = 0; o < nb; ++o)
          if (o != tid && piv[j0 + o] == p) alone = false;
      }
    }
    const unsigned all_alone = __all_sync(0xffffffffu, alone), any = __any_sync(0xffffffffu, moved);
    if (tid == 0) sm.flag = !any ? 0 : all_alone ? 1 : 2;
  }
  __syncthreads();
  const int ncol = ncols - nb;
  if (sm.flag == 1) {
    for (int jj = 0; jj < nb; ++jj) {
      const int j = j0 + jj, p = piv[j];
      if (p == j) continue;
      for (int c = tid; c < ncol; c += NT) {
        double2* col = A + (size_t)(c < j0 ? c : c + nb) * ld;
        const double2 x = col[j];
        col[j] = col[p];
        col[p] = x;
      }
    }
  } else if (sm.flag == 2) {
    for (int c = tid; c < ncol; c += NT) {
      double2* col = A + (size_t)(c < j0 ? c : c + nb) * ld;
      for (int jj = 0; jj < nb; ++jj) {
        const int j = j0 + jj, p = piv[j];
        if (p != j) {
          const double2 x = col[j];
          col[j] = col[p];
          col[p] = x;
        }
      }
    }
  }
  __syncthreads();
}

// LU of the N x N column-major matrix A (leading dimension ld) in place, N <= 8 NT and N <= 2048. piv: N entries in shared
// memory. The columns N .. ncols - 1 are right-hand sides: they take the interchanges and the block rows with the matrix
// and leave as L^-1 P B, so that only the backward substitution is left. The result does not depend on NT: every element
// goes through the same operations in the same order.
template <int NT, int NB>
__device__ bool lu_factor_dmma(double2* __restrict__ A, int N, int ncols, int ld, int* __restrict__ piv,
                                            LuSmem<NT, NB>& sm) {
  bool singular = false;
  for (int j0 = 0; j0 < N; j0 += NB) {
    const int nb = min(NB, N - j0), m = N - j0, right = ncols - j0 - nb;
    if (j0 > 0) {
      lu_block_column<NT, NB>(A, N, ld, j0, nb, sm);
      __syncthreads();
    }
    if (m <= NT)
      singular |= lu_panel<NT, NB, 1>(A, N, ld, j0, nb, piv, sm);
    else if (m <= 2 * NT)
      singular |= lu_panel<NT, NB, 2>(A, N, ld, j0, nb, piv, sm);
    else if (m <= 4 * NT)
      singular |= lu_panel<NT, NB, 4>(A, N, ld, j0, nb, piv, sm);
    else
      singular |= lu_panel<NT, NB, 8>(A, N, ld, j0, nb, piv, sm);
    lu_interchange<NT, NB>(A, ncols, ld, j0, nb, piv, sm);
    if (right > 0) {
      lu_invert_lower<NT, NB>(A, ld, j0, nb, sm);
      lu_block_row<NT, NB, false>(A, N, ld, j0, nb, 0, j0, A + (size_t)(j0 + nb) * ld, ld, right, sm);
      __syncthreads();
    }
  }
  return singular;
}

// Y = L^-1 Y (rows already interchanged) for the ncols columns of Y, with the factors of lu_factor_dmma.
template <int NT, int NB>
__device__ void lu_forward_dmma(const double2* __restrict__ A, int N, int ld, double2* Y, int ldy, int ncols,
                                             LuSmem<NT, NB>& sm) {
  for (int j0 = 0; j0 < N; j0 += NB) {
    const int nb = min(NB, N - j0);
    lu_invert_lower<NT, NB>(A, ld, j0, nb, sm);
    lu_block_row<NT, NB, false>(A, N, ld, j0, nb, 0, j0, Y, ldy, ncols, sm);
    __syncthreads();
  }
}

// Y = U^-1 Y for the ncols columns of Y.
template <int NT, int NB>
__device__ void lu_backward_dmma(const double2* __restrict__ A, int N, int ld, double2* Y, int ldy,
                                              int ncols, LuSmem<NT, NB>& sm) {
  for (int j0 = (N - 1) / NB * NB; j0 >= 0; j0 -= NB) {
    const int nb = min(NB, N - j0);
    lu_invert_upper<NT, NB>(A, ld, j0, nb, sm);
    lu_block_row<NT, NB, true>(A, N, ld, j0, nb, j0 + nb, N, Y, ldy, ncols, sm);
    __syncthreads();
  }
}

}  // namespace dga
