// FP64 complex LU with partial pivoting of one matrix by one CTA, Crout order, products on the FP64 tensor pipe.
//
// The matrix is column-major in the CTA's scratch (or any global memory); the result has LAPACK's layout (unit lower L
// below the diagonal, U on and above, piv[j] = the row exchanged with row j) and its pivots (largest |re| + |im|, first
// index on ties), as lu_factor's.
//
// Why Crout order: a right-looking update reads and writes the whole trailing matrix once per 32 columns (2/3 N^3 / 32
// elements read and written, 248 MB at N = 720 with the factor tiles); here a block column and a block row are
// accumulated in registers over everything to their left and above and written once, so the same products cost
// reads only (62 MB at N = 720), and a CTA needs no shared-memory tiles or barriers inside them.
//
// Why mma.sync f64: the FP64 tensor pipe and the FP64 vector pipe have the same peak (37 TFLOP/s measured for either),
// but an m16n8k4 product takes one warp instruction where the vector pipe takes 16, and its A and B fragments of an
// interleaved complex matrix are one 16-byte load per lane each (lane (g, t) holds row g and column t), so operands come
// straight from L2 and L1: four warps per SM already reach 35 TFLOP/s. The tcgen05 pipe has no FP64 kind.
//
// What bounds it: the products at N = 720 (592 factorisations in 27.0 ms, 21.9 TFLOP/s, two CTAs an SM, three quarters of
// the time in the block columns and rows), the panels' dependent steps below about N = 200 (14,208 of N = 120 in 7.9 ms).
// Whole passes, from the right-looking vector-pipe form to this one: 1,130 to 762 ms for three orbitals on 32 x 32
// (N = 720), 103 to 72 ms for one orbital on 64 x 64 (N = 120), 0.85 to 0.62 ms on 16 x 16 (N = 40).
#pragma once

#include "dga_common.cuh"
#include "tc_tile.cuh"

namespace dga {

constexpr int LU_NB = 32;   // block width
constexpr int LU_MAX_N = 2048;
constexpr int LU_RING = 4;  // steps of four columns a lane has in flight
static_assert(LU_RING * 2 == 8, "a warp's ring and its 8-column tile share their memory");

// Rows a thread holds in the panel and panel columns it keeps in registers, for matrices of up to RPT * NT rows: at most
// RPT * PW = 16 complex values (64 registers).
template <int RPT>
struct LuPanelWidth {
  static constexpr int value = RPT <= 2 ? 8 : RPT <= 4 ? 4 : 2;
};

template <int NT>
struct LuSmem {
  double2 L11i[LU_NB][LU_NB + 1];  // inverse of the diagonal block's unit lower triangle
  union {
    double2 L11[LU_NB][LU_NB + 1];                    // the triangle itself, dead once it is inverted
    // (each warp's part is the same memory in both)
    double2 tile[NT / 32][8][LU_NB + 1];              // per warp: 8 columns of the block row before the triangular solve
    double2 ring[NT / 32][LU_RING][2][LU_NB + 1];     // per lane: fragments of the streamed factor on their way from HBM
  };
  double2 us[8][LU_NB];            // panel: rows of U of the columns just factored
  double2 cand[2][NT / 32][10];    // panel: each warp's candidate pivot row, conj(pivot), 1 / |pivot|^2
  __align__(16) unsigned long long key[2][NT / 32];
  int flag;
};

__device__ __forceinline__ void cp_async16(double2* smem, const double2* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}
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

// Block column: A[j0.., j0 .. j0+nb) -= A[j0.., 0..j0) A[0..j0, j0 .. j0+nb). One warp per 16 rows x 32 columns; rows and
// columns past the end read the last valid ones and are not stored. L streams from HBM (the matrices in flight are ten
// times L2): a lane copies the two elements it multiplies three steps later, 1,500 cycles of the FP64 pipe, into its own
// ring slot, so nothing has to be synchronised; U is shared by all warps and comes from L1, one step ahead.
template <int NT>
__device__ void lu_block_column(double2* __restrict__ A, int N, int ld, int j0, int nb, LuSmem<NT>& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int tiles = (N - j0 + 15) / 16;
  double2(*ring)[2][LU_NB + 1] = sm.ring[warp];
  int ob[4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) ob[nt] = min(j0 + nt * 8 + g, N - 1) * ld + t;
  for (int tile = warp; tile < tiles; tile += NT / 32) {
    const int r0 = j0 + tile * 16 + g, r1 = r0 + 8;
    CAcc acc[4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[nt].re[i] = acc[nt].im[i] = 0.0;
    const int d1 = min(r1, N - 1) - min(r0, N - 1), step = 4 * ld;
    const double2* pa = A + t * ld + min(r0, N - 1);
#pragma unroll
    for (int u = 0; u < LU_RING - 1; ++u) {  // j0 >= 32: at least eight steps
      cp_async16(&ring[u][0][lane], pa);
      cp_async16(&ring[u][1][lane], pa + d1);
      cp_async_commit();
      pa += step;
    }
    double2 b[4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) b[nt] = A[ob[nt]];
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
      double2 y[4];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) y[nt] = b[nt];
      if (k + 4 < j0) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) b[nt] = A[ob[nt] + k + 4];
      }
      cdmma_row<4>(acc, x0, x1, y);
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
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

// Block row: U[j0..j0+32, c] = L11^-1 (A[j0..j0+32, c] - A[j0..j0+32, 0..j0) A[0..j0, c]) for the columns c >= j0 + 32.
// One warp per 32 rows x 16 columns; the triangular solve is a product with the inverse in shared memory.
template <int NT>
__device__ void lu_block_row(double2* __restrict__ A, int N, int ld, int j0, LuSmem<NT>& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int c_first = j0 + LU_NB, tiles = (N - c_first + 15) / 16;
  for (int tile = warp; tile < tiles; tile += NT / 32) {
    const int c0 = c_first + tile * 16;
    CAcc acc[2][2];  // [16-row half][8-column half]
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[mt][nt].re[i] = acc[mt][nt].im[i] = 0.0;
    if (j0 > 0) {
      double2(*ring)[2][LU_NB + 1] = sm.ring[warp];
      int oa = t * ld + j0 + g;
      const double2* pb = A + (size_t)min(c0 + g, N - 1) * ld + t;
      const int d1 = (min(c0 + 8 + g, N - 1) - min(c0 + g, N - 1)) * ld, step = 4 * ld;
      __syncwarp();  // the ring shares its memory with the previous tile's columns
#pragma unroll
      for (int u = 0; u < LU_RING - 1; ++u) {
        cp_async16(&ring[u][0][lane], pb);
        cp_async16(&ring[u][1][lane], pb + d1);
        cp_async_commit();
        pb += 4;
      }
      double2 a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = A[oa + u * 8];
      int slot = 0;
      for (int k = 0; k < j0; k += 4) {
        cp_async_wait<LU_RING - 2>();
        const double2 y[2] = {ring[slot][0][lane], ring[slot][1][lane]};
        const int next = (slot + LU_RING - 1) % LU_RING;
        if (k + 4 * (LU_RING - 1) < j0) {
          cp_async16(&ring[next][0][lane], pb);
          cp_async16(&ring[next][1][lane], pb + d1);
          pb += 4;
        }
        cp_async_commit();
        slot = (slot + 1) % LU_RING;
        double2 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = a[u];
        if (k + 4 < j0) {
          oa += step;
#pragma unroll
          for (int u = 0; u < 4; ++u) a[u] = A[oa + u * 8];
        }
        cdmma_row<2>(acc[0], x[0], x[1], y);
        cdmma_row<2>(acc[1], x[2], x[3], y);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      double2(&w)[8][LU_NB + 1] = sm.tile[warp];
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = min(c0 + nt * 8 + 2 * t + (i & 1), N - 1), r = mt * 16 + g + (i < 2 ? 0 : 8);
          const double2 v = A[(size_t)c * ld + j0 + r];
          w[2 * t + (i & 1)][r] = make_double2(v.x - acc[mt][nt].re[i], v.y - acc[mt][nt].im[i]);
        }
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        CAcc x[1];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[0].re[i] = x[0].im[i] = 0.0;
#pragma unroll 2
        for (int k = 0; k < mt * 16 + 16; k += 4) {
          const double2 y[1] = {w[g][k + t]};
          cdmma_row<1>(x, sm.L11i[mt * 16 + g][k + t], sm.L11i[mt * 16 + g + 8][k + t], y);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = c0 + nt * 8 + 2 * t + (i & 1), r = j0 + mt * 16 + g + (i < 2 ? 0 : 8);
          if (c < N) A[(size_t)c * ld + r] = make_double2(x[0].re[i], x[0].im[i]);
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

// Inverse of the unit lower 32 x 32 block in sm.L11 by doubling, from the inverses of its 8 x 8 diagonal blocks in
// sm.L11i: [A 0; B C]^-1 = [A^-1 0; -C^-1 B A^-1 C^-1] at 16 and 32.
template <int NT>
__device__ void lu_unit_lower_inverse(LuSmem<NT>& sm) {
  const int tid = threadIdx.x;
  double2* tmp = &sm.us[0][0];  // B A^-1, at most 16 x 16
#pragma unroll
  for (int h = 8; h <= 16; h *= 2) {
    const int n = LU_NB / 2 * h;
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

constexpr unsigned long long LU_INF_BITS = 0x7ff0000000000000ull;

// Pivot candidates are compared as one 64-bit integer: the high 48 bits of |re| + |im| (a non-negative double orders as
// an integer does), then the position, the first one largest, then the warp that offers it. Integers keep the search off
// the FP64 pipe, where each comparison would wait behind the products of the other warps; entries that agree to 2^-36 are
// tied and the first of them is taken. 0: no candidate (a NaN is none).
__device__ __forceinline__ unsigned long long lu_key(double2 a, int pos, int warp) {
  const unsigned long long x = __double_as_longlong(cabs1(a));
  return x > LU_INF_BITS ? 0 : (x & ~0xffffull) | (unsigned)((2048 - pos) << 4) | (unsigned)warp;
}

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

// y = L^-1 y for the leading n x n unit lower triangle at L in sm.L11's row pitch; a rotating loop, as in the panel
template <int PW>
__device__ __forceinline__ void unit_lower_solve(double2 (&y)[PW], int n, const double2* L) {
#pragma unroll 1
  for (int k = 0; k < PW; ++k) {
    const double2 yk = y[0];
#pragma unroll
    for (int r = 1; r < PW; ++r)
      if (k + r < n) cfms(y[r], L[(k + r) * (LU_NB + 1) + k], yk);
#pragma unroll
    for (int r = 0; r + 1 < PW; ++r) y[r] = y[r + 1];
    y[PW - 1] = yk;
  }
}

// Panel: factors the columns [j0, j0 + nb) of the rows j0.. with partial pivoting, PW columns at a time in registers (a
// thread holds the rows j0 + tid + NT i). A row keeps its registers when it is exchanged; only its position changes, and
// the columns are written back at the new positions. One barrier per column: each warp offers its best row with its
// reciprocal already taken, every thread picks the winner. The PW columns are then applied to the rest of the block, whose
// interchanges are made here; the columns outside it follow in lu_interchange. Returns true if
// an exact zero pivot was met.
template <int NT, int RPT>
__device__ bool lu_panel(double2* __restrict__ A, int N, int ld, int j0, int nb, int* __restrict__ piv,
                         LuSmem<NT>& sm) {
  constexpr int PW = LuPanelWidth<RPT>::value, NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool singular = false;
  for (int p0 = 0; p0 < nb; p0 += PW) {
    const int pw = min(PW, nb - p0), jc = j0 + p0;
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
        double2 d = make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const unsigned long long x = (pos[i] >= j && pos[i] < N) ? lu_key(a[i][0], pos[i], warp) : 0;
          if (x > own) {
            own = x;
            d = a[i][0];
          }
        }
        double2 rc;
        double rs;
        pivot_recip(d, rc, rs);
        unsigned long long key = warp_max(own);
        if (own == key && key) {
          const int p = 2048 - (int)((key >> 4) & 0xfff);
#pragma unroll
          for (int i = 0; i < RPT; ++i)
            if (pos[i] == p) {
#pragma unroll
              for (int c = 0; c < PW; ++c) sm.cand[buf][warp][c] = a[i][c];
            }
          sm.cand[buf][warp][8] = rc;
          sm.cand[buf][warp][9].x = rs;
        }
        if (lane == 0) sm.key[buf][warp] = key;
        __syncthreads();
        if constexpr (NW > 1) {
          const ulonglong2* keys = reinterpret_cast<const ulonglong2*>(sm.key[buf]);
          key = 0;
#pragma unroll
          for (int w = 0; w < NW / 2; ++w) {
            const ulonglong2 x = keys[w];
            const unsigned long long m = x.x > x.y ? x.x : x.y;
            key = m > key ? m : key;
          }
        }
        int p = 2048 - (int)((key >> 4) & 0xfff), win = (int)(key & 15);
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
            if (!zero) a[i][0] = cscale(cmul(a[i][0], cd), cs);
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
        unit_lower_solve<PW>(y, pw, &sm.L11[p0][p0]);
#pragma unroll
        for (int r = 0; r < PW; ++r)
          if (r < pw) {
            col[r] = y[r];
            sm.us[r][c] = y[r];
          }
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        if (pos[i] < jc + pw || pos[i] >= N) continue;
        double2* row = P + (size_t)pw * ld + pos[i];
        double2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = u < rest ? row[(size_t)u * ld] : make_double2(0.0, 0.0);
#pragma unroll 1
        for (int c = 0; c < rest; c += 4) {  // four columns at a time, the next four on their way
          double2 n[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            n[u] = c + 4 + u < rest ? row[(size_t)(c + 4 + u) * ld] : make_double2(0.0, 0.0);
#pragma unroll
          for (int k = 0; k < PW; ++k)
            if (k < pw) {
#pragma unroll
              for (int u = 0; u < 4; ++u) cfms(v[u], a[i][k], sm.us[k][c + u]);
            }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (c + u < rest) row[(size_t)(c + u) * ld] = v[u];
            v[u] = n[u];
          }
        }
      }
      __syncthreads();
    }
  }
  return singular;
}

// The unit lower triangle of the factored 32 x 32 diagonal block in sm.L11, and the inverses of its 8 x 8 diagonal blocks
// (one thread per column) in sm.L11i, zero elsewhere.
template <int NT>
__device__ void lu_load_l11(const double2* __restrict__ A, int ld, int j0, LuSmem<NT>& sm) {
  const int tid = threadIdx.x;
  for (int e = tid; e < LU_NB * LU_NB; e += NT) {
    const int r = e % LU_NB, c = e / LU_NB;
    if (r > c) sm.L11[r][c] = A[(size_t)(j0 + c) * ld + j0 + r];
    if ((r ^ c) & ~7) sm.L11i[r][c] = make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (tid < LU_NB) {
    const int o = tid & ~7, c = tid & 7;
    double2 y[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) y[r] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    unit_lower_solve<8>(y, 8, &sm.L11[o][o]);
#pragma unroll
    for (int r = 0; r < 8; ++r) sm.L11i[o + r][o + c] = y[r];
  }
  __syncthreads();
}

// The block's row interchanges on the columns outside it: in parallel over (interchange, column) when they are
// independent pairs (every pivot row below the block, no two alike), else in order per column; nothing to do when no
// row moved.
template <int NT>
__device__ void lu_interchange(double2* __restrict__ A, int N, int ld, int j0, int nb, const int* __restrict__ piv,
                               LuSmem<NT>& sm) {
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
  const int ncol = N - nb;
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
// memory. The result does not depend on NT: every element goes through the same operations in the same order.
template <int NT>
__device__ __noinline__ bool lu_factor_dmma(double2* __restrict__ A, int N, int ld, int* __restrict__ piv, LuSmem<NT>& sm) {
  bool singular = false;
  for (int j0 = 0; j0 < N; j0 += LU_NB) {
    const int nb = min(LU_NB, N - j0), m = N - j0;
    if (j0 > 0) {
      lu_block_column<NT>(A, N, ld, j0, nb, sm);
      __syncthreads();
    }
    if (m <= NT)
      singular |= lu_panel<NT, 1>(A, N, ld, j0, nb, piv, sm);
    else if (m <= 2 * NT)
      singular |= lu_panel<NT, 2>(A, N, ld, j0, nb, piv, sm);
    else if (m <= 4 * NT)
      singular |= lu_panel<NT, 4>(A, N, ld, j0, nb, piv, sm);
    else
      singular |= lu_panel<NT, 8>(A, N, ld, j0, nb, piv, sm);
    lu_interchange<NT>(A, N, ld, j0, nb, piv, sm);
    if (j0 + nb < N) {
      lu_load_l11<NT>(A, ld, j0, sm);
      lu_unit_lower_inverse<NT>(sm);
      lu_block_row<NT>(A, N, ld, j0, sm);
      __syncthreads();
    }
  }
  return singular;
}

}  // namespace dga
