// Dense-MPO channel environments, two-point correlators and the entanglement
// spectrum on the device:
//   dominant_env          envs.jl:34-99 (identity or dense-MPO transfer matrix of one
//                         unit cell, :LM Arnoldi from v0 = ones, unit norm)
//   envs_build_dense      DMRGCache(psi, ::DenseIMPO), envs.jl:284-304, with
//                         normalize_envs! (envs.jl:559-584)
//   energy_dense          expectationvalue(psi, ::DenseIMPO, envs), expval.jl:60-79
//   correlator            correlators.jl:13-42
//   entanglement_spectrum toolbox.jl:9-14: singular values of C[loc] by one-sided
//                         (Hestenes) Jacobi rotations, all column pairs of a round
//                         rotated in parallel (round-robin schedule), one CTA per pair
#include "observables.h"

#include <algorithm>
#include <cmath>

#include "gauge.h"

namespace imps {
namespace {

constexpr int kJacThreads = 256;

__device__ __forceinline__ double block_sum256(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double r = 0.0;
  for (int q = 0; q < kJacThreads / 32; ++q) r += sh[q];
  __syncthreads();
  return r;
}

// Player at position `pos` of round `r` in the round-robin schedule of P (even)
// players: position 0 is fixed, the other P-1 rotate by one per round.
__device__ __forceinline__ int rr_player(int pos, int r, int P) {
  return pos == 0 ? 0 : ((pos - 1 + r) % (P - 1)) + 1;
}

// One round of one-sided Jacobi: CTA k orthogonalises columns (a, b) = players at
// positions k and P-1-k.  Columns >= ncol are zero padding (never rotated).  With
// gamma = u_a^H u_b = |gamma| e^{i phi}, the real Jacobi rotation of the Gram matrix
// [[alpha, |gamma|], [|gamma|, beta]] applied to (u_a, e^{-i phi} u_b) makes them
// orthogonal.  *rot counts the rotations performed (the convergence test of a sweep).
__global__ void __launch_bounds__(kJacThreads) k_jacobi_round(int n, int ncol, int P, int r, dcplx* __restrict__ U,
                                                          int64_t ldu, double tol, int* __restrict__ rot,
                                                          dcplx* __restrict__ V, int nv, int64_t ldv) {
  grid_enter();
  __shared__ double sh[kJacThreads / 32];
  const int k = blockIdx.x;
  int a = rr_player(k, r, P), b = rr_player(P - 1 - k, r, P);
  if (a > b) {
    const int t = a;
    a = b;
    b = t;
  }
  if (b >= ncol) return;
  dcplx* ua = U + ldu * (int64_t)a;
  dcplx* ub = U + ldu * (int64_t)b;
  double al = 0.0, be = 0.0, gr = 0.0, gi = 0.0;
  for (int i = threadIdx.x; i < n; i += kJacThreads) {
    const dcplx x = ua[i], y = ub[i];
    al = fma(x.x, x.x, fma(x.y, x.y, al));
    be = fma(y.x, y.x, fma(y.y, y.y, be));
    gr = fma(x.x, y.x, fma(x.y, y.y, gr));   // Re conj(x) y
    gi = fma(x.x, y.y, fma(-x.y, y.x, gi));  // Im conj(x) y
  }
  al = block_sum256(al, sh);
  be = block_sum256(be, sh);
  gr = block_sum256(gr, sh);
  gi = block_sum256(gi, sh);
  const double g = hypot(gr, gi);
  if (!(g > tol * sqrt(al * be)) || g == 0.0) return;
  const double zeta = (be - al) / (2.0 * g);
  const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
  const double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
  const double er = gr / g, ei = gi / g;  // e^{i phi}
  for (int i = threadIdx.x; i < n; i += kJacThreads) {
    const dcplx x = ua[i], y = ub[i];
    // y' = e^{-i phi} y
    const double ypr = er * y.x + ei * y.y, ypi = er * y.y - ei * y.x;
    const double nxr = c * x.x - s * ypr, nxi = c * x.y - s * ypi;
    const double nyr = s * x.x + c * ypr, nyi = s * x.y + c * ypi;
    ua[i] = make_double2(nxr, nxi);
    // back to the original phase of column b: e^{i phi} y''
    ub[i] = make_double2(er * nyr - ei * nyi, er * nyi + ei * nyr);
  }
  // the same rotation on the columns of V (right singular vectors), if requested
  if (V) {
    dcplx* va = V + ldv * (int64_t)a;
    dcplx* vb = V + ldv * (int64_t)b;
    for (int i = threadIdx.x; i < nv; i += kJacThreads) {
      const dcplx x = va[i], y = vb[i];
      const double ypr = er * y.x + ei * y.y, ypi = er * y.y - ei * y.x;
      const double nxr = c * x.x - s * ypr, nxi = c * x.y - s * ypi;
      const double nyr = s * x.x + c * ypr, nyi = s * x.y + c * ypi;
      va[i] = make_double2(nxr, nxi);
      vb[i] = make_double2(er * nyr - ei * nyi, er * nyi + ei * nyr);
    }
  }
  if (threadIdx.x == 0) atomicAdd(rot, 1);
}

// Block form of the round for values only: the columns are taken in blocks of 8, CTA k
// orthogonalises the 16 columns of blocks (a, b) of the round-robin schedule of blocks in
// shared memory (round 0 also the pairs inside each block), a warp per pair.  A warp keeps
// its column of block a in registers while the 8 columns of block b come to it in turn, so a
// sweep is nblk - 1 launches of 8 steps instead of 8 nblk - 1 launches of one.
// n <= 32 EPL rows; the columns past the last one are zero (never rotated).  Bound by the
// latency of a step (two sums over the warp, two square roots, two divisions): 10 us a launch
// of 16 CTAs at n = 256, against 24 us for 8 rounds of k_jacobi_round.
constexpr int kJacBlk = 8;

// Orthogonalises x, y (a row i = lane + 32 u of each per register); true when it rotated.
template <int EPL>
__device__ __forceinline__ bool jacobi_pair(dcplx (&x)[EPL], dcplx (&y)[EPL], double tol2, int lane) {
  double v[4] = {0.0, 0.0, 0.0, 0.0};   // ||x||^2, ||y||^2, x^H y
#pragma unroll
  for (int u = 0; u < EPL; ++u) {
    v[0] = fma(x[u].x, x[u].x, fma(x[u].y, x[u].y, v[0]));
    v[1] = fma(y[u].x, y[u].x, fma(y[u].y, y[u].y, v[1]));
    v[2] = fma(x[u].x, y[u].x, fma(x[u].y, y[u].y, v[2]));
    v[3] = fma(x[u].x, y[u].y, fma(-x[u].y, y[u].x, v[3]));
  }
  // lanes of the upper half keep v[2..3], then every quarter one sum
#pragma unroll
  for (int o = 16, half = 2; half >= 1; o >>= 1, half >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int q = 0; q < half; ++q) {
      const double send = up ? v[q] : v[q + half], keep = up ? v[q + half] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  const double al = __shfl_sync(0xffffffffu, v[0], 0), be = __shfl_sync(0xffffffffu, v[0], 8);
  const double gr = __shfl_sync(0xffffffffu, v[0], 16), gi = __shfl_sync(0xffffffffu, v[0], 24);
  const double g2 = gr * gr + gi * gi;
  if (!(g2 > tol2 * al * be)) return false;
  // tan of the rotation that annihilates the off-diagonal of [[al, g], [g, be]], g = |x^H y|
  const double g = sqrt(g2), d = be - al;
  const double t = copysign(2.0 * g / (fabs(d) + sqrt(fma(d, d, 4.0 * g2))), d);
  const double c = 1.0 / sqrt(fma(t, t, 1.0)), s = c * t, ig = 1.0 / g;
  const double er = gr * ig, ei = gi * ig;
  const double sr = s * er, si = s * ei;
#pragma unroll
  for (int u = 0; u < EPL; ++u) {
    const dcplx a = x[u], b = y[u];
    // x' = c x - s e^{-i phi} y,  y' = s e^{i phi} x + c y
    x[u] = make_double2(c * a.x - (sr * b.x + si * b.y), c * a.y - (sr * b.y - si * b.x));
    y[u] = make_double2((sr * a.x - si * a.y) + c * b.x, (sr * a.y + si * a.x) + c * b.y);
  }
  return true;
}

template <int EPL>
__global__ void __launch_bounds__(32 * kJacBlk) k_jacobi_block(int n, int nblk, int r, dcplx* __restrict__ U,
                                                               int64_t ldu, double tol2, int* __restrict__ rot) {
  grid_enter();
  extern __shared__ dcplx cols[];   // [16][32 EPL]
  constexpr int LDC = 32 * EPL;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = blockIdx.x;
  const int ba = rr_player(k, r, nblk) * kJacBlk, bb = rr_player(nblk - 1 - k, r, nblk) * kJacBlk;
  dcplx x[EPL], y[EPL];
  int cnt = 0;
  auto global_col = [&](int q) { return U + ldu * (int64_t)((q < kJacBlk ? ba : bb - kJacBlk) + q); };
  auto get = [&](const dcplx* p, dcplx (&z)[EPL]) {
#pragma unroll
    for (int u = 0; u < EPL; ++u) z[u] = p[lane + 32 * u];
  };
  auto put = [&](dcplx* p, const dcplx (&z)[EPL]) {
#pragma unroll
    for (int u = 0; u < EPL; ++u) p[lane + 32 * u] = z[u];
  };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const dcplx* src = global_col(w + kJacBlk * h);
#pragma unroll
    for (int u = 0; u < EPL; ++u)
      cols[(w + kJacBlk * h) * LDC + lane + 32 * u] = lane + 32 * u < n ? src[lane + 32 * u] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (r == 0) {
    const int off = w < 4 ? 0 : kJacBlk, q = w & 3;
    for (int s = 0; s < kJacBlk - 1; ++s) {
      dcplx* px = cols + (off + rr_player(q, s, kJacBlk)) * LDC;
      dcplx* py = cols + (off + rr_player(kJacBlk - 1 - q, s, kJacBlk)) * LDC;
      get(px, x);
      get(py, y);
      if (jacobi_pair<EPL>(x, y, tol2, lane)) {
        ++cnt;
        put(px, x);
        put(py, y);
      }
      __syncthreads();
    }
  }
  get(cols + w * LDC, x);
  for (int s = 0; s < kJacBlk; ++s) {
    dcplx* py = cols + (kJacBlk + ((w + s) & (kJacBlk - 1))) * LDC;
    get(py, y);
    if (jacobi_pair<EPL>(x, y, tol2, lane)) {
      ++cnt;
      put(py, y);
    }
    __syncthreads();
  }
  if (!__syncthreads_or(cnt)) return;
  if (lane == 0 && cnt) atomicAdd(rot, cnt);
  dcplx* da = global_col(w);
  dcplx* db = global_col(w + kJacBlk);
  get(cols + (w + kJacBlk) * LDC, y);
#pragma unroll
  for (int u = 0; u < EPL; ++u) {
    const int i = lane + 32 * u;
    if (i < n) {
      da[i] = x[u];
      db[i] = y[u];
    }
  }
}

template <int EPL>
void jacobi_block_round(Context* ctx, int n, int nblk, int r, dcplx* U, double tol, int* rot) {
  constexpr int SMEM = 2 * kJacBlk * 32 * EPL * (int)sizeof(dcplx);
  static DeviceOnce attr;
  attr.run(ctx->device, [] {
    IMPS_CUDA(cudaFuncSetAttribute(k_jacobi_block<EPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
  });
  launch_kernel(ctx, k_jacobi_block<EPL>, nblk / 2, 32 * kJacBlk, SMEM, n, nblk, r, U, n, tol * tol, rot);
}

// out[:, j] = scale_j * in[:, perm[j]] for j < k (column gather with optional scaling)
__global__ void k_gather_cols(int rows, int k, const dcplx* __restrict__ in, int64_t ldi, const int* __restrict__ perm,
                              const double* __restrict__ scale, dcplx* __restrict__ out, int64_t ldo) {
  grid_enter();
  const int64_t tot = (int64_t)rows * k;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot; t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % rows), j = (int)(t / rows);
    const dcplx v = in[i + ldi * (int64_t)perm[j]];
    const double f = scale ? scale[j] : 1.0;
    out[i + ldo * (int64_t)j] = make_double2(v.x * f, v.y * f);
  }
}

__global__ void k_col_norms2(int n, int ncol, const dcplx* __restrict__ U, int64_t ldu, double* __restrict__ out) {
  grid_enter();
  __shared__ double sh[kJacThreads / 32];
  const int j = blockIdx.x;
  if (j >= ncol) return;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kJacThreads) {
    const dcplx x = U[i + ldu * (int64_t)j];
    s = fma(x.x, x.x, fma(x.y, x.y, s));
  }
  s = block_sum256(s, sh);
  if (threadIdx.x == 0) out[j] = s;
}

void check(Context* ctx) {
  ctx->n_kernels++;
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) throw Error(IMPS_CUDA_ERROR, std::string("observables launch: ") + cudaGetErrorString(e));
}

}  // namespace

// Jacobi sweeps over the columns of U (n rows, ncol columns, room for an even number of them, or
// with `blocks` for a multiple of 16) until no pair rotates.
static void jacobi_sweeps(Context* ctx, int n, int ncol, dcplx* U, bool blocks) {
  DevBuf& flag = ctx->buf("jac_flag", 64);
  int* rot = static_cast<int*>(flag.ptr);
  const double tol = 1e-15 * std::sqrt((double)n);
  const int P = ncol + (ncol & 1), nblk = (ncol + 2 * kJacBlk - 1) / (2 * kJacBlk) * 2;
  for (int sweep = 0; sweep < 60; ++sweep) {
    IMPS_CUDA(cudaMemsetAsync(rot, 0, sizeof(int), ctx->stream));
    if (blocks) {
      for (int r = 0; r < nblk - 1; ++r) {
        if (n <= 128) jacobi_block_round<4>(ctx, n, nblk, r, U, tol, rot);
        else if (n <= 256) jacobi_block_round<8>(ctx, n, nblk, r, U, tol, rot);
        else jacobi_block_round<16>(ctx, n, nblk, r, U, tol, rot);
        check(ctx);
      }
    } else {
      for (int r = 0; r < P - 1; ++r) {
        launch_kernel(ctx, k_jacobi_round, P / 2, kJacThreads, 0, n, ncol, P, r, U, n, tol, rot, nullptr, 0, 0);
        check(ctx);
      }
    }
    int done = 0;
    download(ctx, &done, rot, sizeof(int));
    if (done == 0) break;
  }
}

// The squared singular values of the D x D matrix A, descending, divided by a power of four so
// that the largest is of order one (their own squares, up to 4^1024, need not be doubles).
// One-sided Jacobi on A itself
// takes many sweeps when A's columns are far from orthogonal (34 for a bond matrix in a
// general basis, D = 256: 34 ms); on the conjugate transpose of the R factor of A with its
// columns by descending norm, whose columns are graded and nearly orthogonal, it takes 11,
// in blocks (5.2 ms with the QR).  With a workspace cap A is taken as it is, and in blocks only
// where the padding to whole blocks fits as well.
std::vector<double> singular_values_sq(Context* ctx, int D, const dcplx* A, int64_t lda) {
  IMPS_REQUIRE(D > 0, IMPS_INVALID_ARG, "singular values: empty matrix");
  // blocks: 16 columns fit in a CTA's shared memory and registers
  bool blocks = D <= 512;
  int P = D + (D & 1);
  if (blocks) {
    try {
      const int padded = (D + 2 * kJacBlk - 1) / (2 * kJacBlk) * (2 * kJacBlk);
      ctx->buf("jac_norms", (size_t)padded * sizeof(double));
      ctx->buf("jac_flag", 64);
      ctx->buf("jac_u", (size_t)D * padded * sizeof(dcplx));
      P = padded;
    } catch (const Error& err) {
      if (err.status != IMPS_OOM) throw;
      cudaGetLastError();
      blocks = false;
      ctx->scratch.erase("jac_norms");   // (its padding may be what is missing)
    }
  }
  DevBuf& U = ctx->buf("jac_u", (size_t)D * P * sizeof(dcplx));
  DevBuf& nr = ctx->buf("jac_norms", (size_t)P * sizeof(double));
  ScopedTimer tm(ctx, "jacobi_svd", 0.0);
  zfill(ctx, (int64_t)D * P, 0.0, U.z());
  std::vector<double> s2(D);
  auto norms = [&] {
    launch_kernel(ctx, k_col_norms2, D, kJacThreads, 0, D, D, U.z(), D, nr.d());
    check(ctx);
    download(ctx, s2.data(), nr.ptr, D * sizeof(double));
  };
  zcopy2d(ctx, D, D, A, lda, U.z(), D);
  norms();
  const double top = *std::max_element(s2.begin(), s2.end());
  bool finite = true;
  for (double v : s2) finite = finite && std::isfinite(v);
  if (finite && top > 0.0) {   // an exact scale that keeps the squares' squares in range
    int e;
    std::frexp(std::sqrt(top), &e);
    zscal(ctx, (int64_t)D * D, std::ldexp(1.0, -e), U.z());
  }
  if (finite && top > 0.0 && ctx->workspace_limit == 0 && D <= 32768) {
    try {
      std::vector<int> perm(D);
      for (int j = 0; j < D; ++j) perm[j] = j;
      std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return s2[a] > s2[b]; });
      DevBuf& W = ctx->buf("jac_w", (size_t)D * D * sizeof(dcplx));
      DevBuf& R = ctx->buf("jac_r", (size_t)D * D * sizeof(dcplx));
      int* pd = static_cast<int*>(ctx->buf("jac_perm", (size_t)D * sizeof(int)).ptr);
      upload(ctx, pd, perm.data(), (size_t)D * sizeof(int));
      launch_kernel(ctx, k_gather_cols, 148 * 8, 256, 0, D, D, U.z(), D, pd, nullptr, W.z(), D);
      check(ctx);
      qr_factor(ctx, D, D, W.z(), D, R.z(), "qr");
      zconj_transpose(ctx, D, D, R.z(), D, U.z(), D);
    } catch (const Error& err) {
      if (err.status != IMPS_OOM) throw;
      cudaGetLastError();   // U still holds A
    }
  }
  jacobi_sweeps(ctx, D, D, U.z(), blocks);
  norms();
  std::sort(s2.begin(), s2.end(), [](double x, double y) { return x > y; });
  return s2;
}

int svd_thin(Context* ctx, int m, int n, const dcplx* A, int64_t lda, int kmax, double cutoff, dcplx* U,
             std::vector<double>& s, dcplx* V) {
  IMPS_REQUIRE(m > 0 && n > 0, IMPS_INVALID_ARG, "svd: empty matrix");
  if (m < n) {
    // A = (A^H)^H: the SVD of A^H with the roles of U and V exchanged
    DevBuf& AH = ctx->buf("svd_ah", (size_t)m * n * sizeof(dcplx));
    zconj_transpose(ctx, m, n, A, lda, AH.z(), n);
    DevBuf& Ut = ctx->buf("svd_ut", (size_t)n * std::min(m, kmax > 0 ? kmax : m) * sizeof(dcplx));
    const int k = svd_thin(ctx, n, m, AH.z(), n, kmax, cutoff, Ut.z(), s, U);
    // V = U' (n x k) of the transposed problem
    zcopy2d(ctx, n, k, Ut.z(), n, V, n);
    return k;
  }
  const int P = n + (n & 1);
  DevBuf& W = ctx->buf("svd_w", (size_t)m * P * sizeof(dcplx));
  DevBuf& Vw = ctx->buf("svd_v", (size_t)n * P * sizeof(dcplx));
  DevBuf& flag = ctx->buf("jac_flag", 64);
  DevBuf& nr = ctx->buf("jac_norms", (size_t)P * sizeof(double));
  zcopy2d(ctx, m, n, A, lda, W.z(), m);
  zset_identity(ctx, n, Vw.z(), n, 1.0);
  ScopedTimer tm(ctx, "jacobi_svd", 0.0);
  const double tol = 1e-15 * std::sqrt((double)m);
  for (int sweep = 0; sweep < 60; ++sweep) {
    IMPS_CUDA(cudaMemsetAsync(flag.ptr, 0, sizeof(int), ctx->stream));
    for (int r = 0; r < P - 1; ++r) {
      launch_kernel(ctx, k_jacobi_round, P / 2, kJacThreads, 0, m, n, P, r, W.z(), m, tol, static_cast<int*>(flag.ptr),
                                                             Vw.z(), n, n);
      check(ctx);
    }
    int rot = 0;
    download(ctx, &rot, flag.ptr, sizeof(int));
    if (rot == 0) break;
  }
  launch_kernel(ctx, k_col_norms2, n, kJacThreads, 0, m, n, W.z(), m, nr.d());
  check(ctx);
  std::vector<double> n2(n);
  download(ctx, n2.data(), nr.ptr, n * sizeof(double));
  std::vector<int> perm(n);
  for (int j = 0; j < n; ++j) perm[j] = j;
  std::stable_sort(perm.begin(), perm.end(), [&](int x, int y) { return n2[x] > n2[y]; });
  int k = kmax > 0 ? std::min(kmax, n) : n;
  while (k > 1 && std::sqrt(std::max(n2[perm[k - 1]], 0.0)) <= cutoff) --k;
  s.resize(k);
  std::vector<double> inv(k);
  for (int j = 0; j < k; ++j) {
    s[j] = std::sqrt(std::max(n2[perm[j]], 0.0));
    inv[j] = s[j] > 0.0 ? 1.0 / s[j] : 0.0;
  }
  // the doubles first: an int array of odd length before them would misalign them
  DevBuf& pb = ctx->buf("svd_perm", (size_t)k * (sizeof(int) + sizeof(double)));
  double* sd = static_cast<double*>(pb.ptr);
  int* pd = reinterpret_cast<int*>(static_cast<char*>(pb.ptr) + (size_t)k * sizeof(double));
  upload(ctx, pd, perm.data(), (size_t)k * sizeof(int));
  upload(ctx, sd, inv.data(), (size_t)k * sizeof(double));
  auto grid = [](int64_t t) { return (int)std::max<int64_t>(1, std::min<int64_t>((t + 255) / 256, 148 * 8)); };
  // U = W[:, perm] / s (columns of exactly zero singular value stay zero), V = Vw[:, perm]
  launch_kernel(ctx, k_gather_cols, grid((int64_t)m * k), 256, 0, m, k, W.z(), m, pd, sd, U, m);
  check(ctx);
  launch_kernel(ctx, k_gather_cols, grid((int64_t)n * k), 256, 0, n, k, Vw.z(), n, pd, nullptr, V, n);
  check(ctx);
  return k;
}

std::vector<double> entanglement_spectrum(Context* ctx, imps_state* st, int bond) {
  Fp64Scope fp64(ctx);
  const int b = ((bond % st->N) + st->N) % st->N;
  const int D = st->Dr(b);
  std::vector<double> p = singular_values_sq(ctx, D, st->C[b].z(), D);
  double tot = 0.0;
  for (double v : p) tot += v;
  IMPS_REQUIRE(tot > 0.0, IMPS_INVALID_ARG, "entanglement spectrum: zero center matrix");
  for (double& v : p) v /= tot;
  return p;
}

KrylovResult dominant_env(Context* ctx, imps_state* st, const imps_mpo* mpo, int side, double tol, int krylovdim,
                          int maxiter, dcplx* out) {
  Fp64Scope fp64(ctx);
  const int N = st->N;
  const int D = st->Dl(0);
  const int w = mpo ? mpo->sites[0].m : 1;
  const int64_t n = (int64_t)D * w * D;
  DevBuf& a = ctx->buf("domenv_a", (size_t)n * sizeof(dcplx));
  DevBuf& b = ctx->buf("domenv_b", (size_t)n * sizeof(dcplx));
  DevBuf& v0 = ctx->buf("domenv_v0", (size_t)n * sizeof(dcplx));
  LinOp op = [&](const dcplx* v, dcplx* o) {
    const dcplx* cur = v;
    for (int k = 0; k < N; ++k) {
      const int l = side == 0 ? k : N - 1 - k;
      dcplx* dst = (k == N - 1) ? o : ((k % 2 == 0) ? a.z() : b.z());
      const int Dl = st->Dl(l), d = st->d[l], Dr = st->Dr(l);
      if (!mpo) {
        if (side == 0) push_left_id(ctx, Dl, d, Dr, cur, st->AL[l].z(), st->AL[l].z(), dst);
        else push_right_id(ctx, Dl, d, Dr, cur, st->AR[l].z(), st->AR[l].z(), dst);
      } else {
        const MpoSite& W = mpo->sites[l % mpo->N];
        if (side == 0) push_mpo_left(ctx, W, Dl, d, Dr, cur, st->AL[l].z(), dst);
        else push_mpo_right(ctx, W, Dl, d, Dr, cur, st->AR[l].z(), dst);
      }
      cur = dst;
    }
  };
  zfill(ctx, n, cplx(1.0, 0.0), v0.z());
  KrylovResult r = arnoldi_dominant(ctx, n, op, v0.z(), out, tol, krylovdim, maxiter, true);
  const double nv = dznrm2(ctx, n, out);
  zscal(ctx, n, 1.0 / nv, out);
  return r;
}

KrylovResult envs_build_dense(Context* ctx, imps_envs* envs, imps_state* st, const imps_mpo* mpo, double tol,
                              int krylovdim, int maxiter) {
  Fp64Scope fp64(ctx);
  const int N = st->N;
  IMPS_REQUIRE(envs->N == N && mpo->N > 0 && N % mpo->N == 0, IMPS_DIM_MISMATCH,
               "dense environments: unit cells of state, MPO and environments differ");
  KrylovResult rl = dominant_env(ctx, st, mpo, 0, tol, krylovdim, maxiter, envs->lefts[0].z());
  KrylovResult rr = dominant_env(ctx, st, mpo, 1, tol, krylovdim, maxiter, envs->rights[N - 1].z());
  for (int l = 1; l < N; ++l)
    push_mpo_left(ctx, mpo->sites[(l - 1) % mpo->N], st->Dl(l - 1), st->d[l - 1], st->Dr(l - 1),
                  envs->lefts[l - 1].z(), st->AL[l - 1].z(), envs->lefts[l].z());
  for (int l = N - 2; l >= 0; --l)
    push_mpo_right(ctx, mpo->sites[(l + 1) % mpo->N], st->Dl(l + 1), st->d[l + 1], st->Dr(l + 1),
                   envs->rights[l + 1].z(), st->AR[l + 1].z(), envs->rights[l].z());
  for (int l = 0; l < N; ++l) envs->GLp_valid[l] = false;
  // normalize_envs!: unit-norm right environments, lefts[i+1] /= <C_i, H_C(i) C_i>
  for (int i = 0; i < N; ++i) {
    const int64_t nr = (int64_t)envs->Dr[i] * envs->nr[i] * envs->Dr[i];
    const double rn = dznrm2(ctx, nr, envs->rights[i].z());
    if (rn > 0) zscal(ctx, nr, 1.0 / rn, envs->rights[i].z());
    const int D = st->Dr(i);
    DevBuf& hc = ctx->buf("dense_hc", (size_t)D * D * sizeof(dcplx));
    c_apply(ctx, envs, i, st->C[i].z(), hc.z());
    const cplx lam = zdotc(ctx, (int64_t)D * D, st->C[i].z(), hc.z());
    if (std::abs(lam) > 0) {
      const int l1 = (i + 1) % N;
      const int64_t nl = (int64_t)envs->Dl[l1] * envs->ml[l1] * envs->Dl[l1];
      zscal(ctx, nl, 1.0 / lam, envs->lefts[l1].z());
      envs->GLp_valid[l1] = false;
    }
  }
  envs->version++;
  KrylovResult r;
  r.converged = rl.converged && rr.converged;
  r.numops = rl.numops + rr.numops;
  r.numiter = rl.numiter + rr.numiter;
  r.normres = std::max(rl.normres, rr.normres);
  r.value = rl.value;
  return r;
}

cplx energy_dense(Context* ctx, imps_envs* envs, const imps_mpo* mpo, imps_state* st) {
  Fp64Scope fp64(ctx);
  cplx E = 0.0;
  for (int i = 0; i < st->N; ++i) {
    const int64_t n = st->site_elems(i);
    DevBuf& y = ctx->buf("dense_e", (size_t)n * sizeof(dcplx));
    ac_apply(ctx, envs, mpo, i, st->AC[i].z(), y.z());
    E += zdotc(ctx, n, st->AC[i].z(), y.z());
  }
  return E / state_dot(ctx, st);
}

void apply_local(Context* ctx, int Dl, int d, int Dr, const dcplx* O_dev, const dcplx* A, dcplx* out) {
  // out[:, :, b] = A[:, :, b] O^T  (out[a, u, b] = sum_s O[u, s] A[a, s, b])
  zgemm_fp64(ctx, OP_N, OP_T, Dl, d, d, 1.0, A, Dl, (int64_t)Dl * d, O_dev, d, 0, 0.0, out, Dl, (int64_t)Dl * d, Dr);
}

std::vector<cplx> correlator(Context* ctx, imps_state* st, const cplx* O1, const cplx* O2, int i,
                             const std::vector<int>& js) {
  Fp64Scope fp64(ctx);
  const int N = st->N;
  IMPS_REQUIRE(!js.empty() && js[0] > i, IMPS_INVALID_ARG, "correlator: i should be smaller than j");
  for (size_t k = 1; k < js.size(); ++k)
    IMPS_REQUIRE(js[k] > js[k - 1], IMPS_INVALID_ARG, "correlator: js must increase");
  auto site = [&](int l) { return ((l - 1) % N + N) % N; };  // 1-based -> 0-based periodic
  const int si = site(i);
  const int dmax = *std::max_element(st->d.begin(), st->d.end());
  DevBuf& Od = ctx->buf("corr_o", (size_t)2 * dmax * dmax * sizeof(dcplx));
  const int d1 = st->d[si];
  upload(ctx, Od.ptr, O1, (size_t)d1 * d1 * sizeof(dcplx));
  size_t mx = 0;
  int Dmax = 0;
  for (int l = 0; l < N; ++l) {
    mx = std::max(mx, st->site_elems(l));
    Dmax = std::max(Dmax, std::max(st->Dl(l), st->Dr(l)));
  }
  DevBuf& OA = ctx->buf("corr_oa", mx * sizeof(dcplx));
  DevBuf& Va = ctx->buf("corr_va", (size_t)Dmax * Dmax * sizeof(dcplx));
  DevBuf& Vb = ctx->buf("corr_vb", (size_t)Dmax * Dmax * sizeof(dcplx));
  DevBuf& Ib = ctx->buf("corr_id", (size_t)Dmax * Dmax * sizeof(dcplx));
  DevBuf& E = ctx->buf("corr_e", (size_t)Dmax * Dmax * sizeof(dcplx));
  // V = push_env_left(I, O1 AC_i, AC_i)
  {
    const int Dl = st->Dl(si), Dr = st->Dr(si);
    zset_identity(ctx, Dl, Ib.z(), Dl, 1.0);
    apply_local(ctx, Dl, d1, Dr, Od.z(), st->AC[si].z(), OA.z());
    push_left_id(ctx, Dl, d1, Dr, Ib.z(), OA.z(), st->AC[si].z(), Va.z());
  }
  dcplx* V = Va.z();
  dcplx* Vn = Vb.z();
  std::vector<cplx> out(js.size());
  int ctr = i;
  for (size_t k = 0; k < js.size(); ++k) {
    const int j = js[k];
    for (int l = ctr + 1; l <= j - 1; ++l) {
      const int s = site(l);
      push_left_id(ctx, st->Dl(s), st->d[s], st->Dr(s), V, st->AR[s].z(), st->AR[s].z(), Vn);
      std::swap(V, Vn);
    }
    const int sj = site(j);
    const int Dl = st->Dl(sj), d = st->d[sj], Dr = st->Dr(sj);
    upload(ctx, Od.z() + dmax * dmax, O2, (size_t)d * d * sizeof(dcplx));
    apply_local(ctx, Dl, d, Dr, Od.z() + dmax * dmax, st->AR[sj].z(), OA.z());
    push_left_id(ctx, Dl, d, Dr, V, OA.z(), st->AR[sj].z(), E.z());
    zset_identity(ctx, Dr, Ib.z(), Dr, 1.0);
    out[k] = ztrace_prod(ctx, Dr, E.z(), Dr, Ib.z(), Dr);
    ctr = j;  // as the reference (correlators.jl:34): the next j transfers from ctr + 1
  }
  const cplx nrm = state_dot(ctx, st);
  for (auto& v : out) v /= nrm;
  return out;
}

}  // namespace imps
