// Batched ladder Bethe-Salpeter solve for every (channel, q, w) work item.
//
// For one item the compound-index matrix (row (o1,o2,nu), column (o4,o3,nu'), N = n^2 * 2 niv) is
//
//     A = (blockdiag_nu chi0^-1(q,w,nu) + Gamma_r(w) / beta^2) - (U_r + V_r^q) / beta^2
//
// (dgamore/nonlocal_sde.py:85-96 assembled through FourPoint.add, four_point.py:332-430), and the result is
//
//     X[(o1,o2,nu), (o4,o3)] = sum_nu' (A^-1)[(o1,o2,nu), (o4,o3,nu')] / beta
//
// (four_point.py:620-642; equivalently the solve against the n^2 selector right-hand sides of
// four_point.py:644-684).  Each CTA owns one item at a time (persistent loop over a device work list):
//
//   1. form A column-major in the CTA's scratch slot (Gamma_r is pre-permuted to the same column-major
//      compound layout once per request, so this is a coalesced stream plus a block-diagonal add);
//   2. LU with partial pivoting, LAPACK's pivot measure |re|+|im| and first-index ties (izamax): in FP64 the Crout form
//      of lu_dmma.cuh on the FP64 tensor pipe; in FP32 (lu_factor below) a right-looking form, panel width NB, the
//      trailing matrix updated by a tiled complex GEMM from shared memory;
//   3. the permuted selector right-hand side is solved by blocked forward and back substitution and
//      written out divided by beta.
//
// The mixed form factors in FP32 (FP64 residuals and refinement; see solve_item_mixed below); dense matrices beyond the
// Crout form's size also take lu_factor.
#include "bse_kernels.cuh"

#include <stdio.h>

#include <type_traits>

namespace dga {

DGA_FP64_KERNELS(extern template, 32)
DGA_FP64_KERNELS(extern template, 64)
DGA_FP64_KERNELS(extern template, 128)
DGA_FP64_KERNELS(extern template, 256)

// The same for N > LU_MAX_N, by the right-looking form.
__global__ void __launch_bounds__(BSE_THREADS, 3)
    dense_lu_large_kernel(double2* __restrict__ a, int N, int n_mat, long long mat_stride, int* __restrict__ piv_out,
                          int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BseSmem<double2>& sm = *reinterpret_cast<BseSmem<double2>*>(smem_raw);
  int* piv = reinterpret_cast<int*>(smem_raw + sizeof(BseSmem<double2>));
  for (int m = blockIdx.x; m < n_mat; m += gridDim.x) {
    const bool singular = lu_factor<double2>(a + (size_t)m * mat_stride, N, N, piv, sm);
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += blockDim.x) piv_out[(size_t)m * N + i] = piv[i];
    if (threadIdx.x == 0) status[m] = singular ? DGA_ITEM_SINGULAR : DGA_ITEM_OK;
    __syncthreads();
  }
}

// out_m[:, k] = A_m^-1 B_m[:, k] for k < n_rhs, column-major with leading dimension N, COLS
// columns a CTA (columns n_rhs .. of the last 16 are solved for zero right-hand sides): substitution by 32-row blocks.
// DENSE_COLS: 16 columns a warp, each block accumulated on the FP64 tensor pipe over all solved blocks, with the diagonal
// blocks inverted.  DENSE_RHS: 16 columns a CTA, whose threads split the rows under (over) each solved block
// (dense_rows_form has the rule).  B_m(r, k) =
// b[m b_sm + r b_sr + k b_sk], or the identity when b is null.  A non-finite solution element sets
// DGA_ITEM_NONFINITE in status[m].
template <int COLS>
__global__ void __launch_bounds__(BSE_THREADS, COLS == DENSE_RHS ? 3 : fp64_min_blocks(BSE_THREADS))
    dense_solve_kernel(const double2* __restrict__ lu, const int* __restrict__ piv, int N, int n_mat,
                       long long lu_stride, const double2* __restrict__ b, long long b_sm, long long b_sr,
                       long long b_sk, int n_rhs, double2* __restrict__ out, long long out_stride,
                       int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fp64Smem<BSE_THREADS>& sm = *reinterpret_cast<Fp64Smem<BSE_THREADS>*>(smem_raw);
  int* perm = reinterpret_cast<int*>(smem_raw + sizeof(Fp64Smem<BSE_THREADS>));
  const int tid = threadIdx.x, T = blockDim.x;
  const int cols = (n_rhs + DENSE_RHS - 1) / DENSE_RHS * DENSE_RHS, n_blk = (cols + COLS - 1) / COLS;
  for (int t = blockIdx.x; t < n_mat * n_blk; t += gridDim.x) {
    const int m = t / n_blk, k0 = (t - m * n_blk) * COLS, nc = min(COLS, cols - k0);
    const int* pv = piv + (size_t)m * N;
    build_perm(N, pv, perm);
    double2* Y = out + (size_t)m * out_stride + (size_t)k0 * N;
    for (int e = tid; e < N * nc; e += T) {
      const int i = e % N, k = e / N, col = k0 + k;
      double2 v = make_double2(0.0, 0.0);
      if (col < n_rhs) {
        const int r = perm[i];
        if (b)
          v = b[m * b_sm + r * b_sr + col * b_sk];
        else if (r == col)
          v.x = 1.0;
      }
      Y[(size_t)k * N + i] = v;
    }
    __syncthreads();
    const double2* f = lu + (size_t)m * lu_stride;
    if constexpr (COLS == DENSE_RHS) {
      lu_solve_inplace<double2, double2, DENSE_RHS>(f, N, N, Y, sm.solve.L11, sm.solve.yb);
    } else {
      lu_forward_dmma<BSE_THREADS, 32>(f, N, N, Y, N, nc, sm.lu32);
      lu_backward_dmma<BSE_THREADS, 32>(f, N, N, Y, N, nc, sm.lu32);
    }
    int bad = 0;
    for (int e = tid; e < N * nc; e += T) {
      const double2 v = Y[e];
      bad |= !(isfinite(v.x) && isfinite(v.y));
    }
    if (__syncthreads_or(bad) && tid == 0) atomicOr(status + m, DGA_ITEM_NONFINITE);
    __syncthreads();
  }
}

// f[ch][q][w] += (Z G3(nu)) G3(nu') over the pp box, Z = U_r - U_r chi_r U_r (the second term of the full vertex,
// eliashberg_solver.py:175-204); one CTA per (ch, q, w < Wpp), Z and H(nu) = Z G3(nu) in shared memory.
//   g3: [2][Q][W][nv][n2][n2]; chi_phys: [2][Q][W][n2][n2]; uv: [2][Q][n2][n2]; f: [2][Q][Wpp][Mb][Mb]
__global__ void eli_ladder_term_kernel(const double2* __restrict__ uv, const double2* __restrict__ g3,
                                       const double2* __restrict__ chi_phys, int n2, int nv, int W, int Q, int P,
                                       int Wpp, double2* __restrict__ f) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* Z = reinterpret_cast<double2*>(smem_raw);
  double2* H = Z + n2 * n2;
  const int wq = blockIdx.x, w = wq % Wpp, q = (wq / Wpp) % Q, ch = wq / (Wpp * Q);
  const int tid = threadIdx.x, T = blockDim.x;
  const int nvp = 2 * P, Mb = n2 * nvp, off = nv / 2 - P;
  const double2* uvq = uv + ((size_t)ch * Q + q) * n2 * n2;
  const double2* cp = chi_phys + (((size_t)ch * Q + q) * W + w) * n2 * n2;
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
  const double2* g3q = g3 + ((((size_t)ch * Q + q) * W + w) * nv) * n2 * n2;
  for (int e = tid; e < nvp * n2 * n2; e += T) {
    const int vb = e / (n2 * n2), ps = e - vb * n2 * n2, p = ps / n2, s = ps - p * n2;
    const double2* g = g3q + (size_t)(off + vb) * n2 * n2;
    double2 acc = make_double2(0.0, 0.0);
    for (int t = 0; t < n2; ++t) cfma(acc, Z[p * n2 + t], g[t * n2 + s]);
    H[e] = acc;
  }
  __syncthreads();
  double2* o = f + (size_t)wq * Mb * Mb;
  for (int e = tid; e < Mb * Mb; e += T) {
    const int row = e / Mb, colx = e - row * Mb;  // column index sidx * nvp + vbp
    const int sidx = colx / nvp, vbp = colx - sidx * nvp;
    const int p = row / nvp, vb = row - p * nvp;
    const double2* hrow = H + (size_t)vb * n2 * n2 + p * n2;
    const double2* gcol = g3q + (size_t)(off + vbp) * n2 * n2;
    double2 f2 = make_double2(0.0, 0.0);
    for (int u = 0; u < n2; ++u) cfma(f2, hrow[u], gcol[u * n2 + sidx]);
    o[e] = cadd(o[e], f2);
  }
}

// Threads of an FP64 CTA: one warp up to N = 64 (29,600 factorisations of N = 40: 1.45 ms, 1.79 with two warps), two up to
// N = 192 (14,208 of N = 120: 6.8 ms, 7.6 with four), four up to N = 512 (1,184 of N = 480: 18.4 ms, 19.6 with eight), eight
// above (592 of N = 720: 27.9 ms). Where the items would fill less than half of the SMs' threads that way, each gets more,
// up to two rows a thread (441 items of N = 200: 1.8 ms with four warps, 2.5 with two). at_once: the items, or where the
// launch has room for fewer CTAs (scratch slots, a limit of the caller's), as many as it has room for.
static int fp64_threads(int N, int at_once) {
  int nt = N <= 64 ? 32 : N <= LU_SMALL_N ? 64 : N <= 512 ? 128 : 256;
  while (nt < 256 && nt < N && (long)at_once * nt <= (long)device_sm_count() * 256) nt *= 2;
  return nt;
}
}  // namespace dga

using namespace dga;

// Calls f with the FP64 kernels' thread count for sizes up to N (fp64_threads) as a compile-time constant, and their
// dynamic shared memory.
template <typename F>
static auto with_fp64_threads(int N, int at_once, F f) {
  const size_t piv = sizeof(int) * (size_t)N;
  switch (fp64_threads(N, at_once)) {
    case 32: return f(std::integral_constant<int, 32>{}, sizeof(Fp64Smem<32>) + piv);
    case 64: return f(std::integral_constant<int, 64>{}, sizeof(Fp64Smem<64>) + piv);
    case 128: return f(std::integral_constant<int, 128>{}, sizeof(Fp64Smem<128>) + piv);
    default: return f(std::integral_constant<int, 256>{}, sizeof(Fp64Smem<256>) + piv);
  }
}

// Resident CTAs of the kernel per SM at this much dynamic shared memory, with the kernel's limits set for it. Without the
// carve-out the driver may size shared memory for fewer CTAs than fit (six of eight for the two-warp FP64 kernel).
template <typename K>
static int prepare_kernel(K kernel, size_t smem, int threads) {
  allow_shared_memory(kernel, smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (per_sm < 1) per_sm = 1;
  const size_t used = (size_t)per_sm * (smem + 1024);  // 1 KB of each CTA is the system's
  const int percent = (int)((used * 100 + 228 * 1024 - 1) / (228 * 1024));
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent < 100 ? percent : 100);
  return per_sm;
}

template <typename K>
static int grid_for(K kernel, int n_items, size_t smem, int threads = BSE_THREADS) {
  const int g = device_sm_count() * prepare_kernel(kernel, smem, threads);
  return n_items < g ? n_items : g;
}

// An FP64 launch over n_items items by at most `limit` CTAs.
struct Fp64Run {
  int at_once, grid;
};

static Fp64Run bse_run(int N, int n_items, size_t limit = (size_t)-1) {
  const int at_once = (size_t)n_items < limit ? n_items : (int)limit;
  return {at_once, with_fp64_threads(N, at_once, [&](auto nt, size_t smem) {
            return grid_for(bse_solve_sum_fp64_kernel<StructuredSource, nt.value>, at_once, smem, nt.value);
          })};
}

static bool supported_rhs(int n2) { return n2 == 1 || n2 == 4 || n2 == 9 || n2 == 16; }

template <typename Source>
static void launch_fp64(int n2, Fp64Run run, cudaStream_t stream, const Source& src, const WorkItem* work, int n_items,
                        int N, int nv, int W, int Q, double beta, double2* out, int* status, double2* scratch,
                        size_t slot, int redo) {
  with_fp64_threads(N, run.at_once, [&](auto nt, size_t smem) {
    auto kernel = bse_solve_sum_fp64_kernel<Source, nt.value>;
    // bse_run has set the structured kernel's limits
    if constexpr (!std::is_same_v<Source, StructuredSource>) prepare_kernel(kernel, smem, nt.value);
    kernel<<<run.grid, nt.value, smem, stream>>>(src, work, n_items, N, n2, nv, W, Q, beta, out, status, scratch, slot,
                                                 redo);
  });
}

extern "C" {

// Scratch bytes the FP64 BSE entry points need for a launch over n_items items of compound size N with
// n2 right-hand sides: one N x N matrix plus N x n2 solution per resident CTA.
size_t dga_bse_scratch_bytes(int N, int n2, int n_items) {
  if (N <= 0 || n2 <= 0 || n_items <= 0) return 0;
  return (size_t)bse_run(N, n_items).grid * ((size_t)N * N + (size_t)N * n2) * sizeof(double2);
}

int dga_bse_solve_sum_c128(int n_orb, int niv, int niw_half, int n_q, int n_ch, double beta, double inv_beta2,
                           const void* gamma_cm, const void* chi0_inv, const void* uv, const int* work,
                           int n_items, void* out, int* status, void* scratch, size_t scratch_bytes,
                           cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_ch <= 0 || n_items <= 0 || N > BSE_MAX_N) {
    dga_set_error("dga_bse_solve_sum_c128: invalid sizes (n_orb=%d niv=%d niw_half=%d n_q=%d n_ch=%d items=%d)",
                  n_orb, niv, niw_half, n_q, n_ch, n_items);
    return DGA_ERR_ARG;
  }
  if (!gamma_cm || !chi0_inv || !uv || !work || !out || !scratch) {
    dga_set_error("dga_bse_solve_sum_c128: null pointer argument");
    return DGA_ERR_ARG;
  }
  const Fp64Run run = bse_run(N, n_items);
  const size_t slot = (size_t)N * N + (size_t)N * n2;
  if (scratch_bytes < (size_t)run.grid * slot * sizeof(double2)) {
    dga_set_error("dga_bse_solve_sum_c128: scratch too small (%zu < %zu)", scratch_bytes,
                  (size_t)run.grid * slot * sizeof(double2));
    return DGA_ERR_SCRATCH;
  }
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  launch_fp64(n2, run, stream, src, (const WorkItem*)work, n_items, N, nv, niw_half, n_q, beta,
              (double2*)out, status, (double2*)scratch, slot, 0);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_solve_sum_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

// FP64 re-solve of the items a mixed launch flagged (status & (NOCONVERGE | NONFINITE)); other items are left
// untouched.  Same arguments as dga_bse_solve_sum_c128 with `status` read and rewritten for the re-solved items;
// the scratch may be sized for a smaller grid (grid_limit CTAs).
int dga_bse_resolve_fp64_c128(int n_orb, int niv, int niw_half, int n_q, int n_ch, double beta, double inv_beta2,
                              const void* gamma_cm, const void* chi0_inv, const void* uv, const int* work, int n_items,
                              void* out, int* status, int grid_limit, void* scratch, size_t scratch_bytes,
                              cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_ch <= 0 || n_items <= 0 || N > BSE_MAX_N ||
      grid_limit <= 0 || !gamma_cm || !chi0_inv || !uv || !work || !out || !status || !scratch) {
    dga_set_error("dga_bse_resolve_fp64_c128: invalid arguments");
    return DGA_ERR_ARG;
  }
  const Fp64Run run = bse_run(N, n_items, (size_t)grid_limit);
  const size_t slot = (size_t)N * N + (size_t)N * n2;
  if (scratch_bytes < (size_t)run.grid * slot * sizeof(double2)) {
    dga_set_error("dga_bse_resolve_fp64_c128: scratch too small");
    return DGA_ERR_SCRATCH;
  }
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  launch_fp64(n2, run, stream, src, (const WorkItem*)work, n_items, N, nv, niw_half, n_q, beta,
              (double2*)out, status, (double2*)scratch, slot, 1);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_resolve_fp64_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

// Generic FourPoint.invert_and_sum_over_last_vn (four_point.py:620-642): the matrix is given explicitly in
// the FourPoint layout [q][o1][o2][o3][o4][w][nu][nu'] (half w range); out is [q][w][N][n2].
int dga_invert_sum_dense_c128(int n_orb, int niv, int niw_half, int n_q, double beta, const void* mat,
                              const int* work, int n_items, void* out, int* status, void* scratch,
                              size_t scratch_bytes, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_items <= 0 || N > BSE_MAX_N || !mat || !work ||
      !out || !scratch) {
    dga_set_error("dga_invert_sum_dense_c128: invalid arguments");
    return DGA_ERR_ARG;
  }
  const Fp64Run run = bse_run(N, n_items);
  const size_t slot = (size_t)N * N + (size_t)N * n2;
  if (scratch_bytes < (size_t)run.grid * slot * sizeof(double2)) {
    dga_set_error("dga_invert_sum_dense_c128: scratch too small");
    return DGA_ERR_SCRATCH;
  }
  DenseSource src;
  src.mat = (const double2*)mat;
  src.nb = n_orb;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  launch_fp64(n2, run, stream, src, (const WorkItem*)work, n_items, N, nv, niw_half, n_q, beta,
              (double2*)out, status, (double2*)scratch, slot, 0);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_invert_sum_dense_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"


static size_t mixed_smem_bytes(int N, int n2) { return mixed_colsum_offset(N) + (size_t)n2 * n2 * sizeof(double2); }

static size_t mixed_slot_bytes(int N, int n2) {
  return (((size_t)N * N * sizeof(float2) + 255) & ~(size_t)255) + 2 * (size_t)N * n2 * sizeof(double2);
}
// Default launch of the mixed form: the block-form kernel (4) wherever its solve phase fits shared memory (it is
// the fastest of the mixed kernels at every size measured, N = 40 to 720; the FP64 form is the faster one for one orbital
// at N = 40 and 120); else, from N = 320, the shared-memory-panel kernel with tensor-core trailing tiles (3) or FP32
// tiles (1), else the 128-thread kernel (2).
static int default_mixed_kernel(int N, int n2) {
  if (dga_block_supported(N, n2)) return 4;
  if (N < 320) return 2;
  if (dga_panel_supported(N, n2, true)) return 3;
  if (dga_panel_supported(N, n2)) return 1;
  return 2;
}

// Grid and scratch slot of the mixed kernels that own their launch geometry (1, 3: panel; 4: block form).
static int owned_grid(int kernel, int n2, int N, int n_items) {
  return kernel == 4 ? dga_block_grid(n2, n_items) : dga_panel_grid(n2, N, n_items, kernel == 3);
}
static size_t owned_slot(int kernel, int N, int n2) {
  return kernel == 4 ? dga_block_slot_bytes(N, n2) : dga_panel_slot_bytes(N, n2);
}

static int mixed_grid(int n_items, size_t smem) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  (void)sms;
  return grid_for(bse_solve_sum_mixed_kernel<9>, n_items, smem);
}

extern "C" {

// Scratch bytes of dga_bse_solve_sum_mixed_c128: one N x N complex64 matrix and two N x n2 complex128
// blocks per resident CTA.
size_t dga_bse_mixed_scratch_bytes(int N, int n2, int n_items) {
  if (N <= 0 || n2 <= 0 || n_items <= 0) return 0;
  const int kernel = default_mixed_kernel(N, n2);
  if (kernel != 2) return (size_t)owned_grid(kernel, n2, N, n_items) * owned_slot(kernel, N, n2);
  const size_t smem = mixed_smem_bytes(N, n2);
  return (size_t)mixed_grid(n_items, smem) * mixed_slot_bytes(N, n2);
}

// Mixed-precision ladder BSE: same inputs and output as dga_bse_solve_sum_c128; FP32 LU, FP64 residuals and
// refinement to tol (refine_converged) within max_iter corrections.  iters: per-item corrections (optional).
int dga_bse_solve_sum_mixed_c128(int n_orb, int niv, int niw_half, int n_q, int n_ch, double beta, double inv_beta2,
                                 const void* gamma_cm, const void* chi0_inv, const void* uv, const int* work,
                                 int n_items, int max_iter, double tol, void* out, int* status, int* iters,
                                 void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_ch <= 0 || n_items <= 0 || N > BSE_MAX_N ||
      n2 > MAX_RHS || max_iter < 0) {
    dga_set_error("dga_bse_solve_sum_mixed_c128: invalid sizes (n_orb=%d niv=%d niw_half=%d n_q=%d n_ch=%d items=%d)",
                  n_orb, niv, niw_half, n_q, n_ch, n_items);
    return DGA_ERR_ARG;
  }
  if (!gamma_cm || !chi0_inv || !uv || !work || !out || !scratch) {
    dga_set_error("dga_bse_solve_sum_mixed_c128: null pointer argument");
    return DGA_ERR_ARG;
  }
  const int kernel = default_mixed_kernel(N, n2);
  const bool panel = kernel != 2;
  const size_t smem = mixed_smem_bytes(N, n2);
  const int grid = panel ? owned_grid(kernel, n2, N, n_items) : mixed_grid(n_items, smem);
  const size_t slot = panel ? owned_slot(kernel, N, n2) : mixed_slot_bytes(N, n2);
  if (scratch_bytes < (size_t)grid * slot) {
    dga_set_error("dga_bse_solve_sum_mixed_c128: scratch too small (%zu < %zu)", scratch_bytes, (size_t)grid * slot);
    return DGA_ERR_SCRATCH;
  }
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  if (panel) {
    // from N = 320: the block-form kernel (bse_block.cu, two 256-thread CTAs per SM), or where it does not fit the
    // shared-memory panel (bse_panel.cu, one 512-thread CTA per SM)
    cudaError_t err =
        kernel == 4 ? dga_block_launch(grid, src, (const WorkItem*)work, n_items, N, n2, nv, niw_half, n_q, beta,
                                       max_iter, tol, (double2*)out, status, iters, (unsigned char*)scratch, slot,
                                       stream)
                    : dga_panel_launch(grid, src, (const WorkItem*)work, n_items, N, n2, nv, niw_half, n_q, beta,
                                       max_iter, tol, (double2*)out, status, iters, (unsigned char*)scratch, slot,
                                       stream, kernel == 3);
    if (err != cudaSuccess) {
      dga_set_error("dga_bse_solve_sum_mixed_c128: launch failed: %s", cudaGetErrorString(err));
      return DGA_ERR_LAUNCH;
    }
    return DGA_OK;
  }
#define DGA_MIXED_CASE(NRV)                                                                                       \
  case NRV:                                                                                                       \
    allow_shared_memory(bse_solve_sum_mixed_kernel<NRV>, smem);                                                    \
    bse_solve_sum_mixed_kernel<NRV><<<grid, BSE_THREADS, smem, stream>>>(                                          \
        src, (const WorkItem*)work, n_items, N, NRV, nv, niw_half, n_q, beta, max_iter, tol, (double2*)out, status, \
        iters, (unsigned char*)scratch, slot);                                                                    \
    break;
  switch (n2) {
    DGA_MIXED_CASE(1)
    DGA_MIXED_CASE(4)
    DGA_MIXED_CASE(9)
    DGA_MIXED_CASE(16)
    default:
      break;
  }
#undef DGA_MIXED_CASE
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_solve_sum_mixed_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"


// ------------------------------------------------------------------------------------------------
// Eliashberg full vertex (host side)
// ------------------------------------------------------------------------------------------------
static int eli_vertex_grid(int N, int n_items) {
  return with_fp64_threads(N, n_items, [&](auto nt, size_t smem) {
    return grid_for(eli_full_vertex_kernel<nt.value>, n_items, smem, nt.value);
  });
}

static size_t eli_slot_elems(int N, int n2, int P) {
  return (size_t)N * N + (size_t)N * 2 * P * n2 + (size_t)2 * P * n2 * n2 + (size_t)n2 * n2;
}

extern "C" {

// Scratch bytes of dga_eli_full_vertex_c128 for n_items items.
size_t dga_eli_vertex_scratch_bytes(int n_orb, int niv, int niv_pp, int n_items) {
  const int n2 = n_orb * n_orb, N = n2 * 2 * niv;
  if (!supported_rhs(n2) || n_items <= 0) return 0;
  const int grid = eli_vertex_grid(N, n_items);
  return (size_t)grid * eli_slot_elems(N, n2, niv_pp) * sizeof(double2);
}

// Full ladder vertex of both channels in the pp box (eliashberg_solver.py:175-204) for the work items
// (ch, q, w) with w < w_pp; inputs as dga_bse_solve_sum_c128 plus gamma_r (g3 [2][Q][W][nv][n2][n2]) and the
// physical susceptibility (chi_phys [2][Q][W][n2][n2]); out: [2][Q][w_pp][Mb][Mb], Mb = n2 * 2 niv_pp.
int dga_eli_full_vertex_c128(int n_orb, int niv, int niw_half, int n_q, int niv_pp, int w_pp, double beta,
                             double inv_beta2, const void* gamma_cm, const void* chi0_inv, const void* uv,
                             const void* g3, const void* chi_phys, const int* work, int n_items, void* out,
                             int* status, void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || niv_pp <= 0 || niv_pp > niv ||
      w_pp <= 0 || w_pp > niw_half || n_items <= 0 || N > BSE_MAX_N || !gamma_cm || !chi0_inv || !uv || !g3 ||
      !chi_phys || !work || !out || !scratch) {
    dga_set_error("dga_eli_full_vertex_c128: invalid arguments");
    return DGA_ERR_ARG;
  }
  const int grid = eli_vertex_grid(N, n_items);
  const size_t slot = eli_slot_elems(N, n2, niv_pp);
  if (scratch_bytes < (size_t)grid * slot * sizeof(double2)) {
    dga_set_error("dga_eli_full_vertex_c128: scratch too small");
    return DGA_ERR_SCRATCH;
  }
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  with_fp64_threads(N, n_items, [&](auto nt, size_t smem) {
    eli_full_vertex_kernel<nt.value><<<grid, nt.value, smem, stream>>>(
        src, (const WorkItem*)work, n_items, N, n2, nv, niw_half, n_q, niv_pp, w_pp, beta, (const double2*)g3,
        (const double2*)chi_phys, (double2*)out, status, (double2*)scratch, slot);
  });
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_eli_full_vertex_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"


// ------------------------------------------------------------------------------------------------
// Heterogeneous batch (host side)
// ------------------------------------------------------------------------------------------------
// Launch geometry of a batch.  In the mixed form every request must have the same default kernel as when it runs
// alone (default_mixed_kernel), so that a request's results are the same in a batch and alone; *kernel receives
// it (1, 3: shared-memory panel, 4: block form, 2: 128-thread kernel; always 2 in FP64).  Returns false for an
// invalid batch.  Problems may differ in orbital count (*n2_max receives the largest n_orb^2, *hetero whether they
// differ); such a batch runs kernels that choose the right-hand-side count per item: the 128-thread kernels, or
// the block-form kernel for orbital counts 1 to 3 (the 4-orbital block kernel is compiled alone).  The
// shared-memory-panel kernels take one orbital count per launch.
static bool batch_dims(const dga_bse_problem* probs, int n_prob, int mixed, int* n_max, size_t* slot, int* kernel,
                       int* n2_max = nullptr, bool* hetero = nullptr) {
  *n_max = 0;
  *slot = 0;
  *kernel = 2;
  if (n_prob <= 0) return false;
  int n2m = 0;
  bool het = false;
  for (int p = 0; p < n_prob; ++p) {
    const int n2 = probs[p].n_orb * probs[p].n_orb;
    const int N = n2 * 2 * probs[p].niv;
    if (probs[p].n_orb <= 0 || !supported_rhs(n2) || probs[p].niv <= 0 || N > BSE_MAX_N) return false;
    het |= probs[p].n_orb != probs[0].n_orb;
    if (mixed) {
      const int k = default_mixed_kernel(N, n2);
      if (p == 0) *kernel = k;
      if (k != *kernel) return false;
    }
    if (N > *n_max) *n_max = N;
    if (n2 > n2m) n2m = n2;
  }
  const bool panel = *kernel != 2;
  if (het && panel && (*kernel != 4 || n2m > 9)) return false;
  for (int p = 0; p < n_prob; ++p) {
    const int n2 = probs[p].n_orb * probs[p].n_orb;
    const int N = n2 * 2 * probs[p].niv;
    const size_t sl = panel ? owned_slot(*kernel, N, n2)
                      : mixed ? mixed_slot_bytes(N, n2)
                              : ((size_t)N * N + (size_t)N * n2) * sizeof(double2);
    if (sl > *slot) *slot = sl;
  }
  *slot = (*slot + 255) & ~(size_t)255;
  if (n2_max) *n2_max = n2m;
  if (hetero) *hetero = het;
  return true;
}

static size_t batch_smem(int n_max, int n2, int mixed) {
  return mixed ? mixed_smem_bytes(n_max, n2) : 0;  // the FP64 kernels' own: with_fp64_threads
}

// The batch kernels' grids for requests of sizes up to n_max (n2 = 0: of several orbital counts); at_once: the items or the
// scratch slots, whichever are fewer.
static int batch_grid(int mixed, int n2, int n_max, int at_once, size_t smem) {
  if (!mixed)
    return with_fp64_threads(n_max, at_once, [&](auto nt, size_t smem64) {
      return grid_for(bse_multi_fp64_kernel<nt.value>, at_once, smem64, nt.value);
    });
  switch (n2) {
    case 0: return grid_for(bse_multi_mixed_kernel<0>, at_once, smem);
    case 1: return grid_for(bse_multi_mixed_kernel<1>, at_once, smem);
    case 4: return grid_for(bse_multi_mixed_kernel<4>, at_once, smem);
    case 9: return grid_for(bse_multi_mixed_kernel<9>, at_once, smem);
    case 16: return grid_for(bse_multi_mixed_kernel<16>, at_once, smem);
    default: return 0;
  }
}

extern "C" {

// Scratch bytes of dga_bse_solve_sum_batch_c128 (probs is a HOST array here); 0 for an invalid batch.
size_t dga_bse_batch_scratch_bytes(const dga_bse_problem* probs, int n_prob, int n_items, int mode) {
  int n_max = 0, kernel = 2, n2_max = 0;
  size_t slot = 0;
  bool hetero = false;
  const int mixed = mode == 1;
  if (!probs || n_items <= 0 || mode < 0 || mode > 2 ||
      !batch_dims(probs, n_prob, mixed, &n_max, &slot, &kernel, &n2_max, &hetero))
    return 0;
  const int n2 = probs[0].n_orb * probs[0].n_orb;
  const bool panel = kernel != 2;
  if (panel)
    return (size_t)(kernel == 4 ? dga_block_grid(hetero ? 0 : n2, n_items)
                                : dga_panel_batch_grid(n2, n_max, n_items, kernel == 3)) *
           slot;
  return (size_t)batch_grid(mixed, hetero ? 0 : n2, n_max, n_items, batch_smem(n_max, hetero ? n2_max : n2, mixed)) *
         slot;
}

// One persistent launch over the (problem, ch, q, w) items of several problems of the same orbital count whose
// frequency boxes, q sets, beta and inputs differ.
//   probs_host: the descriptors (read on the host for the launch geometry); probs_dev: the same array in device
//   memory (read by the kernel); work: [n_items][4] ints (problem, channel, q, w) in device memory; mode: 0 =
//   FP64 LU, 1 = FP32 LU + FP64 refinement (max_iter, tol), 2 = FP64 re-solve of the items whose status holds
//   NOCONVERGE or NONFINITE; status / iters: [n_items] (iters may be null).  The grid is the smaller of the
//   resident CTAs, n_items and scratch_bytes / slot: a smaller scratch buffer caps the launch's HBM footprint.
int dga_bse_solve_sum_batch_c128(const dga_bse_problem* probs_host, const void* probs_dev, int n_prob, const int* work,
                                 int n_items, int mode, int max_iter, double tol, int* status, int* iters,
                                 void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  int n_max = 0, kernel = 2, n2_max = 0;
  size_t slot = 0;
  bool hetero = false;
  const int mixed = mode == 1;
  if (!probs_host || !probs_dev || !work || !scratch || !status || n_items <= 0 || max_iter < 0 || mode < 0 ||
      mode > 2 || !batch_dims(probs_host, n_prob, mixed, &n_max, &slot, &kernel, &n2_max, &hetero)) {
    dga_set_error("dga_bse_solve_sum_batch_c128: invalid arguments (n_orb in {1,2,3,4}; in the mixed form all "
                  "problems take the same default kernel, and problems of different n_orb take the block-form or "
                  "the 128-thread kernel with n_orb at most 3)");
    return DGA_ERR_ARG;
  }
  for (int p = 0; p < n_prob; ++p) {
    const dga_bse_problem& d = probs_host[p];
    if (!d.gamma_cm || !d.chi0_inv || !d.uv || !d.out || d.niw_half <= 0 || d.n_q <= 0) {
      dga_set_error("dga_bse_solve_sum_batch_c128: problem %d has a null pointer or empty size", p);
      return DGA_ERR_ARG;
    }
  }
  const int n2 = probs_host[0].n_orb * probs_host[0].n_orb;
  const size_t smem = batch_smem(n_max, hetero ? n2_max : n2, mixed);
  const bool panel = kernel != 2;
  if (scratch_bytes < slot) {
    dga_set_error("dga_bse_solve_sum_batch_c128: scratch too small (%zu < one slot of %zu)", scratch_bytes, slot);
    return DGA_ERR_SCRATCH;
  }
  const int at_once = (size_t)n_items < scratch_bytes / slot ? n_items : (int)(scratch_bytes / slot);
  int grid = panel    ? (kernel == 4 ? dga_block_grid(hetero ? 0 : n2, n_items)
                                     : dga_panel_batch_grid(n2, n_max, n_items, kernel == 3))
                      : batch_grid(mixed, hetero ? 0 : n2, n_max, at_once, smem);
  if (grid > at_once) grid = at_once;
  const int redo = mode == 2;
  const dga_bse_problem* pd = (const dga_bse_problem*)probs_dev;
  const MultiItem* wk = (const MultiItem*)work;
  unsigned char* sc = (unsigned char*)scratch;
  if (panel) {
    cudaError_t err =
        kernel == 4 ? dga_block_batch_launch(grid, hetero ? 0 : n2, pd, wk, n_items, n_max, max_iter, tol, status,
                                             iters, sc, slot, stream)
                    : dga_panel_batch_launch(grid, n2, pd, wk, n_items, n_max, max_iter, tol, status, iters, sc, slot,
                                             stream, kernel == 3);
    if (err != cudaSuccess) {
      dga_set_error("dga_bse_solve_sum_batch_c128: launch failed: %s", cudaGetErrorString(err));
      return DGA_ERR_LAUNCH;
    }
    return DGA_OK;
  }
  if (mixed) {
    const auto go = [&](auto kernel) {
      kernel<<<grid, BSE_THREADS, smem, stream>>>(pd, wk, n_items, n_max, max_iter, tol, status, iters, sc, slot);
    };
    switch (hetero ? 0 : n2) {
      case 0: go(bse_multi_mixed_kernel<0>); break;
      case 1: go(bse_multi_mixed_kernel<1>); break;
      case 4: go(bse_multi_mixed_kernel<4>); break;
      case 9: go(bse_multi_mixed_kernel<9>); break;
      case 16: go(bse_multi_mixed_kernel<16>); break;
    }
  } else {
    with_fp64_threads(n_max, at_once, [&](auto nt, size_t smem64) {
      bse_multi_fp64_kernel<nt.value><<<grid, nt.value, smem64, stream>>>(pd, wk, n_items, n_max, status, iters, sc, slot,
                                                                        redo);
    });
  }
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_solve_sum_batch_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"

// Loads the code of a batch's kernels ahead of their first launch (see include/dga_b200.h): the block form's and the FP64
// kernels of every thread count, since which of them a batch takes changes with its sizes (2.4 to 10 ms at a first use).
extern "C" int dga_bse_preload(void) {
  cudaFuncAttributes a;
  int bad = dga_block_preload();
  bad |= cudaFuncGetAttributes(&a, bse_multi_fp64_kernel<32>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, bse_multi_fp64_kernel<64>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, bse_multi_fp64_kernel<128>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, bse_multi_fp64_kernel<256>) != cudaSuccess;
  if (bad) {
    dga_set_error("dga_bse_preload: a kernel could not be loaded: %s", cudaGetErrorString(cudaGetLastError()));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

extern "C" int dga_bse_default_kernel(int n_orb, int niv, int mixed) {
  const int n2 = n_orb * n_orb, N = n2 * 2 * niv;
  if (n_orb <= 0 || niv <= 0 || !supported_rhs(n2) || N > BSE_MAX_N) return -1;
  return mixed ? default_mixed_kernel(N, n2) : 2;
}

// ------------------------------------------------------------------------------------------------
// Tuned entry: the same solves with an explicit kernel choice and CTAs per SM (the autotuner's knobs)
// ------------------------------------------------------------------------------------------------
static int sm_count() { return device_sm_count(); }

// 1 = panel kernel, 2 = 128-thread kernel, 3 = panel kernel with tensor-core trailing tiles,
// -1 = the requested kernel cannot run this size
static int tuned_kernel(int mixed, int N, int n2, const dga_bse_tuning* t) {
  const int k = t ? t->kernel : 0;
  if (k < 0 || k > 4) return -1;
  if (!mixed) return (k == 1 || k == 3 || k == 4) ? -1 : 2;
  if (k == 0) return default_mixed_kernel(N, n2);
  if (k == 1 && !dga_panel_supported(N, n2)) return -1;
  if (k == 3 && !dga_panel_supported(N, n2, true)) return -1;
  if (k == 4 && !dga_block_supported(N, n2)) return -1;
  return k;
}

// run: the FP64 form's threads and grid (the returned grid again)
static int tuned_grid(int kernel, int mixed, int N, int n2, int n_items, const dga_bse_tuning* t, size_t* slot,
                      size_t* smem, Fp64Run* run) {
  if (kernel == 1 || kernel == 3) {
    *slot = dga_panel_slot_bytes(N, n2);
    *smem = 0;
    return dga_panel_grid(n2, N, n_items, kernel == 3);
  }
  if (kernel == 4) {
    *slot = dga_block_slot_bytes(N, n2);
    *smem = 0;
    return dga_block_grid(n2, n_items);
  }
  const int cps = t ? t->ctas_per_sm : 0;
  const size_t cap = cps > 0 ? (size_t)sm_count() * cps : (size_t)-1;
  if (!mixed) {
    *smem = 0;  // with_fp64_threads
    *slot = ((size_t)N * N + (size_t)N * n2) * sizeof(double2);
    *run = bse_run(N, n_items, cap);
    return run->grid;
  }
  *smem = mixed_smem_bytes(N, n2);
  *slot = mixed_slot_bytes(N, n2);
  const int grid = mixed_grid(n_items, *smem);
  return (size_t)grid > cap ? (int)cap : grid;
}

extern "C" {

size_t dga_bse_tuned_scratch_bytes(int N, int n2, int n_items, int mixed, const dga_bse_tuning* t) {
  if (N <= 0 || !supported_rhs(n2) || n_items <= 0 || N > BSE_MAX_N) return 0;
  const int kernel = tuned_kernel(mixed, N, n2, t);
  if (kernel < 0) return 0;
  size_t slot = 0, smem = 0;
  Fp64Run run{};
  const int grid = tuned_grid(kernel, mixed, N, n2, n_items, t, &slot, &smem, &run);
  return (size_t)grid * slot;
}

int dga_bse_solve_sum_tuned_c128(int n_orb, int niv, int niw_half, int n_q, int n_ch, double beta, double inv_beta2,
                                 const void* gamma_cm, const void* chi0_inv, const void* uv, const int* work,
                                 int n_items, int mixed, int max_iter, double tol, void* out, int* status, int* iters,
                                 const dga_bse_tuning* t, void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_ch <= 0 || n_items <= 0 ||
      N > BSE_MAX_N || max_iter < 0 || (mixed != 0 && mixed != 1)) {
    dga_set_error("dga_bse_solve_sum_tuned_c128: invalid sizes (n_orb=%d niv=%d niw_half=%d n_q=%d items=%d)", n_orb,
                  niv, niw_half, n_q, n_items);
    return DGA_ERR_ARG;
  }
  if (!gamma_cm || !chi0_inv || !uv || !work || !out || !scratch || (mixed && !status)) {
    dga_set_error("dga_bse_solve_sum_tuned_c128: null pointer argument");
    return DGA_ERR_ARG;
  }
  const int kernel = tuned_kernel(mixed, N, n2, t);
  if (kernel < 0) {
    dga_set_error("dga_bse_solve_sum_tuned_c128: kernel %d cannot run N=%d in this precision", t ? t->kernel : 0, N);
    return DGA_ERR_ARG;
  }
  size_t slot = 0, smem = 0;
  Fp64Run run{};
  const int grid = tuned_grid(kernel, mixed, N, n2, n_items, t, &slot, &smem, &run);
  if (scratch_bytes < (size_t)grid * slot) {
    dga_set_error("dga_bse_solve_sum_tuned_c128: scratch too small (%zu < %zu)", scratch_bytes, (size_t)grid * slot);
    return DGA_ERR_SCRATCH;
  }
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  cudaError_t err;
  if (kernel == 1 || kernel == 3) {
    err = dga_panel_launch(grid, src, (const WorkItem*)work, n_items, N, n2, nv, niw_half, n_q, beta, max_iter, tol,
                           (double2*)out, status, iters, (unsigned char*)scratch, slot, stream, kernel == 3,
                           t ? t->wait_limit : 0);
  } else if (kernel == 4) {
    err = dga_block_launch(grid, src, (const WorkItem*)work, n_items, N, n2, nv, niw_half, n_q, beta, max_iter, tol,
                           (double2*)out, status, iters, (unsigned char*)scratch, slot, stream, t ? t->wait_limit : 0);
  } else if (mixed) {
#define DGA_TUNED_MIXED_CASE(NRV)                                                                                    \
  case NRV:                                                                                                          \
    allow_shared_memory(bse_solve_sum_mixed_kernel<NRV>, smem);                                                      \
    bse_solve_sum_mixed_kernel<NRV><<<grid, BSE_THREADS, smem, stream>>>(                                            \
        src, (const WorkItem*)work, n_items, N, NRV, nv, niw_half, n_q, beta, max_iter, tol, (double2*)out, status,  \
        iters, (unsigned char*)scratch, slot);                                                                       \
    break;
    switch (n2) {
      DGA_TUNED_MIXED_CASE(1)
      DGA_TUNED_MIXED_CASE(4)
      DGA_TUNED_MIXED_CASE(9)
      DGA_TUNED_MIXED_CASE(16)
    }
#undef DGA_TUNED_MIXED_CASE
    err = cudaGetLastError();
  } else {
    launch_fp64(n2, run, stream, src, (const WorkItem*)work, n_items, N, nv, niw_half, n_q, beta,
                (double2*)out, status, (double2*)scratch, slot / sizeof(double2), 0);
    err = cudaGetLastError();
  }
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_solve_sum_tuned_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Allocation-free variant of dga_bse_solve_sum_c128.
//
// Some callers of this library cannot call cudaMalloc: a host program that binds only this C ABI and has no
// device allocator of its own, or a steady-state serving loop that must never trigger cudaMalloc's implicit
// device-wide synchronisation.  For them the per-CTA working matrices live in the fixed array below, which is
// part of this library's device image: every GPU that loads the library holds these 64 MiB until the process
// exits.  In host code `g_bse_noalloc_scratch` is only a host-side stand-in for the array, not a device
// address, so the device address is looked up once per device with cudaGetSymbolAddress and cached.
// ------------------------------------------------------------------------------------------------

#include <mutex>

#define DGA_BSE_NOALLOC_SCRATCH_BYTES (64ull << 20)
#define DGA_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) double2 g_bse_noalloc_scratch[DGA_BSE_NOALLOC_SCRATCH_BYTES / sizeof(double2)];

static std::mutex g_noalloc_mutex;
static void* g_noalloc_ptr[DGA_NOALLOC_MAX_DEVICES] = {nullptr};

// Device address of the scratch array on the current device (looked up on the first call per device).
static int noalloc_scratch_ptr(void** out) {
  int dev = -1;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess || dev < 0 || dev >= DGA_NOALLOC_MAX_DEVICES) {
    dga_set_error("dga_bse_solve_sum_noalloc_c128: no usable current device (%s)", cudaGetErrorString(err));
    return DGA_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    err = cudaGetSymbolAddress(&p, g_bse_noalloc_scratch);
    if (err != cudaSuccess || !p) {
      dga_set_error("dga_bse_solve_sum_noalloc_c128: cudaGetSymbolAddress failed: %s", cudaGetErrorString(err));
      return DGA_ERR_CUDA;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return DGA_OK;
}

extern "C" {

// Same result as dga_bse_solve_sum_c128 without a caller scratch buffer.  At most
// DGA_BSE_NOALLOC_SCRATCH_BYTES (64 MiB) of working matrices are used: as many CTAs run as there are
// (N*N + N*n2)*16-byte slots in it (at least one), so a compound size N above about 2040 is rejected.
// The first call on a device looks up the array's device address (this can load the module); make that first
// call before any stream capture.  Calls share the array, so calls that overlap on the GPU (different streams
// or threads without ordering between them) race; calls on one stream are ordered and safe.  Each item
// rewrites its slot completely before reading it, so nothing has to be cleared between calls.
int dga_bse_solve_sum_noalloc_c128(int n_orb, int niv, int niw_half, int n_q, int n_ch, double beta,
                                   double inv_beta2, const void* gamma_cm, const void* chi0_inv, const void* uv,
                                   const int* work, int n_items, void* out, int* status, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_ch <= 0 || n_items <= 0) {
    dga_set_error("dga_bse_solve_sum_noalloc_c128: invalid sizes (n_orb=%d niv=%d niw_half=%d n_q=%d n_ch=%d "
                  "items=%d)", n_orb, niv, niw_half, n_q, n_ch, n_items);
    return DGA_ERR_ARG;
  }
  const size_t slot = (size_t)N * N + (size_t)N * n2;
  const size_t capacity_slots = DGA_BSE_NOALLOC_SCRATCH_BYTES / (slot * sizeof(double2));
  if (N > BSE_MAX_N || capacity_slots < 1) {
    dga_set_error("dga_bse_solve_sum_noalloc_c128: compound size N=%d needs %zu bytes per matrix, more than the "
                  "fixed %llu-byte scratch; use dga_bse_solve_sum_c128 with a caller buffer", N,
                  slot * sizeof(double2), (unsigned long long)DGA_BSE_NOALLOC_SCRATCH_BYTES);
    return DGA_ERR_SCRATCH;
  }
  if (!gamma_cm || !chi0_inv || !uv || !work || !out) {
    dga_set_error("dga_bse_solve_sum_noalloc_c128: null pointer argument");
    return DGA_ERR_ARG;
  }
  void* scratch = nullptr;
  int rc = noalloc_scratch_ptr(&scratch);
  if (rc != DGA_OK) return rc;
  const Fp64Run run = bse_run(N, n_items, capacity_slots);
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  launch_fp64(n2, run, stream, src, (const WorkItem*)work, n_items, N, nv, niw_half, n_q, beta,
              (double2*)out, status, (double2*)scratch, slot, 0);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_solve_sum_noalloc_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"

extern "C" {

// Batched dense LU with partial pivoting of n_mat N x N column-major matrices a + m*mat_stride (in place).
int dga_lu_batched_c128(void* a, int N, int n_mat, long long mat_stride, int* piv, int* status, cudaStream_t stream) {
  if (!a || !piv || !status || N <= 0 || N > DGA_DENSE_MAX_N || n_mat <= 0 || mat_stride < (long long)N * N) {
    dga_set_error("dga_lu_batched_c128: invalid arguments (N=%d n_mat=%d)", N, n_mat);
    return DGA_ERR_ARG;
  }
  if (N <= LU_MAX_N) {
    with_fp64_threads(N, n_mat, [&](auto nt, size_t smem) {
      const int grid = grid_for(dense_lu_kernel<nt.value>, n_mat, smem, nt.value);
      dense_lu_kernel<nt.value><<<grid, nt.value, smem, stream>>>((double2*)a, N, n_mat, mat_stride, piv, status);
    });
  } else {
    const size_t smem = sizeof(BseSmem<double2>) + sizeof(int) * (size_t)N;
    const int grid = grid_for(dense_lu_large_kernel, n_mat, smem);
    dense_lu_large_kernel<<<grid, BSE_THREADS, smem, stream>>>((double2*)a, N, n_mat, mat_stride, piv, status);
  }
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_lu_batched_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

// Whether 16 columns get a CTA (true) or a warp. A warp's chain of products over the solved rows is the longer one from about
// N = 400, as long as all CTAs of the first kind are resident at once, three an SM: 21 matrices of N = 720 with 64 columns
// 2.5 against 3.7 ms, one with 720 columns 2.0 against 2.6, 82 with 96 columns (492 CTAs) 5.4 against 4.0; N = 400 with 64
// columns 0.92 against 0.93, N = 320 0.69 against 0.61. With a single warp in each CTA and factors that do not stay in
// L2, HBM's latency adds to the chain: 82 matrices with 16 columns 0.98 against 1.07 ms at N = 360, 0.81 either way at 320.
static bool dense_rows_form(int N, int n_mat, long long cols) {
  if (n_mat * (cols / DENSE_RHS) > 3LL * device_sm_count()) return false;
  const bool from_hbm = cols == DENSE_RHS && (size_t)n_mat * N * N * sizeof(double2) > ((size_t)126 << 20);
  return N > (from_hbm ? 320 : 400);
}

// Solves with the factors of dga_lu_batched_c128 for n_rhs right-hand sides (b null: the identity).
int dga_lu_solve_batched_c128(const void* lu, const int* piv, int N, int n_mat, long long lu_stride, const void* b,
                              long long b_stride_m, long long b_stride_r, long long b_stride_k, int n_rhs, void* out,
                              long long out_stride, int* status, cudaStream_t stream) {
  const long long cols = ((long long)n_rhs + DENSE_RHS - 1) / DENSE_RHS * DENSE_RHS;
  if (!lu || !piv || !out || !status || N <= 0 || N > DGA_DENSE_MAX_N || n_mat <= 0 || n_rhs <= 0 ||
      lu_stride < (long long)N * N || out_stride < cols * N || (!b && n_rhs > N)) {
    dga_set_error("dga_lu_solve_batched_c128: invalid arguments (N=%d n_mat=%d n_rhs=%d)", N, n_mat, n_rhs);
    return DGA_ERR_ARG;
  }
  const size_t smem = sizeof(Fp64Smem<BSE_THREADS>) + sizeof(int) * (size_t)N;
  const bool rows = dense_rows_form(N, n_mat, cols);
  const int per_cta = rows ? DENSE_RHS : DENSE_COLS;
  const long long n_tasks = (long long)n_mat * ((cols + per_cta - 1) / per_cta);
  if (n_tasks > 0x7fffffffLL) {
    dga_set_error("dga_lu_solve_batched_c128: too many right-hand-side blocks");
    return DGA_ERR_ARG;
  }
  const auto go = [&](auto kernel) {
    const int grid = grid_for(kernel, (int)n_tasks, smem);
    kernel<<<grid, BSE_THREADS, smem, stream>>>((const double2*)lu, piv, N, n_mat, lu_stride, (const double2*)b,
                                                b_stride_m, b_stride_r, b_stride_k, n_rhs, (double2*)out, out_stride,
                                                status);
  };
  if (rows)
    go(dense_solve_kernel<DENSE_RHS>);
  else
    go(dense_solve_kernel<DENSE_COLS>);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_lu_solve_batched_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"

// Scratch of one CTA of the fused form: the matrix, the selectors and the box columns.
static size_t eli_fused_slot(int N, int n2, int niv_pp) { return (size_t)N * (N + n2 + (size_t)n2 * 2 * niv_pp); }

static int eli_grid(int N, int n_items) {
  return with_fp64_threads(N, n_items, [&](auto nt, size_t smem) {
    return grid_for(bse_fp64_eli_kernel<nt.value>, n_items, smem, nt.value);
  });
}

extern "C" {

// Scratch bytes of dga_bse_solve_sum_eli_c128 for n_items items of size N with a box of niv_pp frequencies.
size_t dga_bse_eli_box_scratch_bytes(int N, int n2, int niv_pp, int n_items) {
  if (N <= 0 || !supported_rhs(n2) || niv_pp <= 0 || n_items <= 0) return 0;
  return (size_t)eli_grid(N, n_items) * eli_fused_slot(N, n2, niv_pp) * sizeof(double2);
}

// The same for the largest box (niv_pp = niv, N columns).
size_t dga_bse_eli_scratch_bytes(int N, int n2, int n_items) {
  if (N <= 0 || !supported_rhs(n2) || n_items <= 0) return 0;
  return dga_bse_eli_box_scratch_bytes(N, n2, (N + 2 * n2 - 1) / (2 * n2), n_items);
}

// dga_bse_solve_sum_c128 whose items with w < w_pp also write the chi* part of the Eliashberg full vertex in the pp
// box (niv_pp) from the same LU factors: out_pp [2][Q][w_pp][Mb][Mb], Mb = n2 * 2 niv_pp; dga_eli_ladder_term_c128
// completes it to the vertex dga_eli_full_vertex_c128 computes.
int dga_bse_solve_sum_eli_c128(int n_orb, int niv, int niw_half, int n_q, int n_ch, double beta, double inv_beta2,
                               const void* gamma_cm, const void* chi0_inv, const void* uv, const int* work,
                               int n_items, int niv_pp, int w_pp, void* out, void* out_pp, int* status, void* scratch,
                               size_t scratch_bytes, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv, N = n2 * nv;
  if (!supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 || n_ch != 2 || n_items <= 0 ||
      N > BSE_MAX_N || niv_pp <= 0 || niv_pp > niv || w_pp <= 0 || w_pp > niw_half || !gamma_cm || !chi0_inv ||
      !uv || !work || !out || !out_pp || !scratch) {
    dga_set_error("dga_bse_solve_sum_eli_c128: invalid arguments");
    return DGA_ERR_ARG;
  }
  const size_t slot = eli_fused_slot(N, n2, niv_pp);
  const int grid = eli_grid(N, n_items);
  if (scratch_bytes < (size_t)grid * slot * sizeof(double2)) {
    dga_set_error("dga_bse_solve_sum_eli_c128: scratch too small");
    return DGA_ERR_SCRATCH;
  }
  StructuredSource src;
  src.gamma_cm = (const double2*)gamma_cm;
  src.chi0_inv = (const double2*)chi0_inv;
  src.uv = (const double2*)uv;
  src.n2 = n2;
  src.nv = nv;
  src.W = niw_half;
  src.Q = n_q;
  src.inv_beta2 = inv_beta2;
  with_fp64_threads(N, n_items, [&](auto nt, size_t smem) {
    bse_fp64_eli_kernel<nt.value><<<grid, nt.value, smem, stream>>>(
        src, (const WorkItem*)work, n_items, N, n2, nv, niw_half, n_q, beta, (double2*)out, niv_pp, w_pp,
        (double2*)out_pp, status, (double2*)scratch, slot);
  });
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_bse_solve_sum_eli_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

// f += (Z G3(nu)) G3(nu') over the pp box for every (ch, q, w < w_pp), Z = U_r - U_r chi_r U_r: completes the
// out_pp of dga_bse_solve_sum_eli_c128 to the full vertex (g3 [2][Q][W][nv][n2][n2], chi_phys [2][Q][W][n2][n2]
// lambda-corrected, uv [2][Q][n2][n2]).
int dga_eli_ladder_term_c128(const void* uv, const void* g3, const void* chi_phys, int n_orb, int niv, int niw_half,
                             int n_q, int niv_pp, int w_pp, void* f, cudaStream_t stream) {
  const int n2 = n_orb * n_orb, nv = 2 * niv;
  if (!uv || !g3 || !chi_phys || !f || !supported_rhs(n2) || n_orb <= 0 || niv <= 0 || niw_half <= 0 || n_q <= 0 ||
      niv_pp <= 0 || niv_pp > niv || w_pp <= 0 || w_pp > niw_half) {
    dga_set_error("dga_eli_ladder_term_c128: invalid arguments");
    return DGA_ERR_ARG;
  }
  const size_t smem = ((size_t)n2 * n2 + (size_t)2 * niv_pp * n2 * n2) * sizeof(double2);
  allow_shared_memory(eli_ladder_term_kernel, smem);
  eli_ladder_term_kernel<<<2 * n_q * w_pp, 256, smem, stream>>>((const double2*)uv, (const double2*)g3,
                                                              (const double2*)chi_phys, n2, nv, niw_half, n_q,
                                                              niv_pp, w_pp, (double2*)f);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    dga_set_error("dga_eli_ladder_term_c128: launch failed: %s", cudaGetErrorString(err));
    return DGA_ERR_LAUNCH;
  }
  return DGA_OK;
}

}  // extern "C"
