// Context, transfers, timing and the memory-bound vector kernels (Krylov
// orthogonalisation, norms, axpy, transposes).  Reductions are two-pass and
// deterministic: per-block partials in a fixed order, then one final block.
#include "imps_internal.h"

#include <algorithm>
#include <vector>
#include <cmath>
#include <cstring>
#include <array>
#include <atomic>
#include <map>
#include <system_error>
#include <thread>

namespace imps {

namespace {
constexpr int kRedThreads = 256;
constexpr int kMaxRedBlocks = 1184;  // 8 x 148 SMs

__device__ __forceinline__ dcplx cmul(dcplx a, dcplx b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ dcplx cmulc(dcplx a, dcplx b) {  // conj(a) * b
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.x, b.y, -a.y * b.x));
}

int red_blocks(int64_t n) {
  int64_t b = (n + kRedThreads - 1) / kRedThreads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, kMaxRedBlocks));
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NT / 32; ++i) r += sh[i];
  }
  __syncthreads();
  return r;
}

__global__ void k_nrm2_partial(int64_t n, const dcplx* __restrict__ x, double* __restrict__ part) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx v = x[i];
    s = fma(v.x, v.x, fma(v.y, v.y, s));
  }
  double r = block_sum<kRedThreads>(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = r;
}

__global__ void k_dotc_partial(int64_t n, const dcplx* __restrict__ x, const dcplx* __restrict__ y,
                               double* __restrict__ part) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  double sr = 0.0, si = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx p = cmulc(x[i], y[i]);
    sr += p.x;
    si += p.y;
  }
  double r = block_sum<kRedThreads>(sr, sh);
  double q = block_sum<kRedThreads>(si, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = r;
    part[2 * blockIdx.x + 1] = q;
  }
}

// Sum `ncol` columns of partials (each `nb` long, stride ld) in a fixed order.
__global__ void k_final_sum(int nb, int ncol, const double* __restrict__ part, int64_t ld, double* __restrict__ out) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  for (int c = 0; c < ncol; ++c) {
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) s += part[i + ld * c];
    double r = block_sum<kRedThreads>(s, sh);
    if (threadIdx.x == 0) out[c] = r;
  }
}

// One block per column: out[c] = sum_i part[i + ld c] (same order as k_final_sum).
__global__ void k_final_sum_cols(int nb, const double* __restrict__ part, int64_t ld, double* __restrict__ out) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  const int c = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) s += part[i + ld * c];
  double r = block_sum<kRedThreads>(s, sh);
  if (threadIdx.x == 0) out[c] = r;
}

// Projection pass, step 1: partials of h_j = <V_j, w> for a chunk of up to CH
// vectors (columns 2 j0 + 2 j, +1 of `part`) and, when norm_col >= 0, of ||w||^2.
template <int CH>
__global__ void k_proj_dots(int64_t n, int nv, const dcplx* __restrict__ V, int64_t ldv, const dcplx* __restrict__ w,
                            double* __restrict__ part, int64_t ldp, int col0, int norm_col) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  double ar[CH], ai[CH], nn = 0.0;
#pragma unroll
  for (int j = 0; j < CH; ++j) { ar[j] = 0.0; ai[j] = 0.0; }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const dcplx wi = w[i];
    nn = fma(wi.x, wi.x, fma(wi.y, wi.y, nn));
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      if (j < nv) {
        const dcplx p = cmulc(V[i + ldv * j], wi);
        ar[j] += p.x;
        ai[j] += p.y;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < CH; ++j) {
    if (j < nv) {
      const double r = block_sum<kRedThreads>(ar[j], sh);
      const double q = block_sum<kRedThreads>(ai[j], sh);
      if (threadIdx.x == 0) {
        part[blockIdx.x + ldp * (col0 + 2 * j)] = r;
        part[blockIdx.x + ldp * (col0 + 2 * j + 1)] = q;
      }
    }
  }
  if (norm_col >= 0) {
    const double r = block_sum<kRedThreads>(nn, sh);
    if (threadIdx.x == 0) part[blockIdx.x + ldp * norm_col] = r;
  }
}

// Projection pass, step 2: w -= sum_j h_j V_j for up to 32 vectors, h read from the
// device (interleaved re/im at hdev[2 j0 ..]); on the last chunk also the partials
// of the new ||w||^2 (one per block) go to `npart`.
__global__ void k_proj_update(int64_t n, int nv, const dcplx* __restrict__ V, int64_t ldv,
                              const double* __restrict__ hdev, dcplx* __restrict__ w, double* __restrict__ npart) {
  grid_enter();
  __shared__ double2 c[32];
  __shared__ double sh[kRedThreads / 32];
  if (threadIdx.x < nv) c[threadIdx.x] = make_double2(-hdev[2 * threadIdx.x], -hdev[2 * threadIdx.x + 1]);
  __syncthreads();
  double nn = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx acc = w[i];
    for (int j = 0; j < nv; ++j) {
      const dcplx p = cmul(c[j], V[i + ldv * j]);
      acc.x += p.x;
      acc.y += p.y;
    }
    w[i] = acc;
    nn = fma(acc.x, acc.x, fma(acc.y, acc.y, nn));
  }
  if (npart) {
    const double r = block_sum<kRedThreads>(nn, sh);
    if (threadIdx.x == 0) npart[blockIdx.x] = r;
  }
}

// Gram-Schmidt projections against a basis of nv <= NV columns, one kernel per pass.
// The rows are taken in chunks of GS_ROWS.  A GS_STAGES-deep cp.async ring stages each
// chunk of V[chunk, 0:nv] and w[chunk] from HBM into shared memory (coalesced: 64
// consecutive rows per column), so several chunks are in flight per block while the
// current one is used: the pending update w <- w - V h (the column partial sums of a row
// combined through shared memory), then the chunk's contribution to h'_j = <V_j, w> for
// every column, GS_THREADS / NV threads per column.  Few registers per thread.
// Partials: part[blockIdx.x + ldp k], k < 2 nv the dots (re, im), k = 2 nv the norm^2
// of w (after the update).
constexpr int GS_THREADS = 256;
constexpr int GS_ROWS = 64;
constexpr int GS_QP = GS_THREADS / GS_ROWS;
constexpr int GS_STAGES = 3;

template <int NV>
constexpr size_t gs_smem_bytes() {
  return (size_t)GS_STAGES * (NV + 1) * GS_ROWS * sizeof(dcplx);
}

__device__ __forceinline__ void gs_cp16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int NV, bool UPDATE>
__global__ void __launch_bounds__(GS_THREADS) k_gs_pass(int64_t n, int nv, const dcplx* __restrict__ V, int64_t ldv,
                                                       const double* __restrict__ hdev, dcplx* __restrict__ w,
                                                       double* __restrict__ part, int64_t ldp) {
  grid_enter();
  constexpr int TPC = GS_THREADS / NV;   // threads per column in the dot phase
  constexpr int RPD = GS_ROWS / TPC;     // rows per thread in the dot phase
  constexpr int STAGE = (NV + 1) * GS_ROWS;
  extern __shared__ __align__(16) dcplx gs_sm[];   // [stage][NV + 1][GS_ROWS]: columns, then w
  __shared__ dcplx as[GS_ROWS];
  __shared__ dcplx apart[UPDATE ? GS_QP : 1][GS_ROWS];
  __shared__ dcplx cs[NV];
  __shared__ double nred[GS_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31;
  if (UPDATE && tid < NV)
    cs[tid] = tid < nv ? make_double2(-hdev[2 * tid], -hdev[2 * tid + 1]) : make_double2(0.0, 0.0);
  const int r1 = tid % GS_ROWS, q = tid / GS_ROWS;   // load / update phase: row r1, columns q + GS_QP u
  const int jd = tid / TPC, sd = tid % TPC;          // dot phase: column jd, rows sd + TPC u
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(gs_sm));
  const int64_t nchunks = (n + GS_ROWS - 1) / GS_ROWS;
  auto issue = [&](int stage, int64_t chunk) {
    const int64_t i = chunk * GS_ROWS + r1;
    const bool ok = i < n;
#pragma unroll
    for (int u = 0; u < NV / GS_QP; ++u) {
      const int j = q + GS_QP * u;
      const bool live = ok && j < nv;
      gs_cp16(sbase + 16u * (uint32_t)(stage * STAGE + j * GS_ROWS + r1), live ? (const void*)(V + i + ldv * j) : V,
              live ? 16 : 0);
    }
    if (q == 0) gs_cp16(sbase + 16u * (uint32_t)(stage * STAGE + NV * GS_ROWS + r1), ok ? (const void*)(w + i) : w,
                        ok ? 16 : 0);
  };
  // chunk t of this block is blockIdx.x + t gridDim.x
  int64_t t_issue = 0;
#pragma unroll
  for (int st = 0; st < GS_STAGES - 1; ++st) {
    const int64_t c = blockIdx.x + t_issue * gridDim.x;
    if (c < nchunks) issue(st, c);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    ++t_issue;
  }
  double dre = 0.0, dim = 0.0, nrm = 0.0;
  for (int64_t t = 0;; ++t) {
    const int64_t chunk = blockIdx.x + t * gridDim.x;
    if (chunk >= nchunks) break;
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GS_STAGES - 2) : "memory");
    __syncthreads();
    {
      const int64_t c = blockIdx.x + t_issue * gridDim.x;
      if (c < nchunks) issue((int)(t_issue % GS_STAGES), c);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      ++t_issue;
    }
    const dcplx* Vs = gs_sm + (t % GS_STAGES) * STAGE;
    const dcplx* ws = Vs + NV * GS_ROWS;
    const int64_t i = chunk * GS_ROWS + r1;
    const dcplx* arow = ws;
    if (UPDATE) {
      double ar = 0.0, ai = 0.0;
#pragma unroll
      for (int u = 0; u < NV / GS_QP; ++u) {
        const int j = q + GS_QP * u;
        const dcplx c = cs[j], v = Vs[j * GS_ROWS + r1];
        ar = fma(c.x, v.x, fma(-c.y, v.y, ar));
        ai = fma(c.x, v.y, fma(c.y, v.x, ai));
      }
      apart[q][r1] = make_double2(ar, ai);
      __syncthreads();
      if (tid < GS_ROWS) {
        dcplx wi = ws[tid];
#pragma unroll
        for (int k = 0; k < GS_QP; ++k) {
          wi.x += apart[k][tid].x;
          wi.y += apart[k][tid].y;
        }
        if (i < n) w[i] = wi;
        as[tid] = wi;
        nrm = fma(wi.x, wi.x, fma(wi.y, wi.y, nrm));
      }
      __syncthreads();
      arow = as;
    } else if (tid < GS_ROWS) {
      const dcplx wi = ws[tid];
      nrm = fma(wi.x, wi.x, fma(wi.y, wi.y, nrm));
    }
    if (jd < nv) {
#pragma unroll
      for (int u = 0; u < RPD; ++u) {
        const int r = sd + TPC * u;
        const dcplx v = Vs[jd * GS_ROWS + r], a = arow[r];
        dre = fma(v.x, a.x, fma(v.y, a.y, dre));
        dim = fma(v.x, a.y, fma(-v.y, a.x, dim));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int o = TPC / 2; o >= 1; o >>= 1) {
    dre += __shfl_xor_sync(0xffffffffu, dre, o);
    dim += __shfl_xor_sync(0xffffffffu, dim, o);
  }
  if (sd == 0 && jd < nv) {
    part[blockIdx.x + ldp * (2 * jd)] = dre;
    part[blockIdx.x + ldp * (2 * jd + 1)] = dim;
  }
  for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
  if (lane == 0) nred[tid >> 5] = nrm;
  __syncthreads();
  if (tid == 0) {
    double tsum = 0.0;
    for (int k = 0; k < GS_THREADS / 32; ++k) tsum += nred[k];
    part[blockIdx.x + ldp * (2 * nv)] = tsum;
  }
}

struct CoefPack {
  double2 c[32];
};

__global__ void k_gemv_acc(int64_t n, int nv, const dcplx* __restrict__ V, int64_t ldv, CoefPack coef,
                           dcplx* __restrict__ w, int set) {
  grid_enter();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx acc = set ? make_double2(0.0, 0.0) : w[i];
    for (int j = 0; j < nv; ++j) {
      dcplx p = cmul(coef.c[j], V[i + ldv * j]);
      acc.x += p.x;
      acc.y += p.y;
    }
    w[i] = acc;
  }
}

__global__ void k_scal(int64_t n, double2 a, dcplx* x) {
  grid_enter();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = cmul(a, x[i]);
}
__global__ void k_axpby(int64_t n, double2 a, const dcplx* __restrict__ x, double2 b, dcplx* __restrict__ y,
                        int use_b) {
  grid_enter();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx v = cmul(a, x[i]);
    if (use_b) {
      dcplx u = cmul(b, y[i]);
      v.x += u.x;
      v.y += u.y;
    }
    y[i] = v;
  }
}
__global__ void k_axpy(int64_t n, double2 a, const dcplx* __restrict__ x, dcplx* __restrict__ y) {
  grid_enter();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx v = cmul(a, x[i]);
    dcplx u = y[i];
    y[i] = make_double2(u.x + v.x, u.y + v.y);
  }
}
__global__ void k_fill(int64_t n, double2 v, dcplx* x) {
  grid_enter();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = v;
}
__global__ void k_set_identity(int D, dcplx* X, int64_t ld, double2 diag) {
  grid_enter();
  int64_t total = (int64_t)D * D;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    int a = (int)(t % D), b = (int)(t / D);
    X[a + ld * b] = (a == b) ? diag : make_double2(0.0, 0.0);
  }
}

// 32 x 32 tiled conjugate transpose: Y[j + ldy i] = conj(X[i + ldx j]).
__global__ void k_conj_transpose(int m, int n, const dcplx* __restrict__ X, int64_t ldx, dcplx* __restrict__ Y,
                                 int64_t ldy) {
  grid_enter();
  __shared__ dcplx tile[32][33];
  int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int i = i0 + threadIdx.x, j = j0 + r;
    if (i < m && j < n) tile[r][threadIdx.x] = X[i + ldx * j];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int j = j0 + threadIdx.x, i = i0 + r;
    if (i < m && j < n) {
      dcplx v = tile[threadIdx.x][r];
      Y[j + ldy * i] = make_double2(v.x, -v.y);
    }
  }
}

// partials of sum_{a,b} L[a,b] V[b,a]
__global__ void k_trace_prod_partial(int D, const dcplx* __restrict__ L, int64_t ldl, const dcplx* __restrict__ V,
                                     int64_t ldv, double* __restrict__ part) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  double sr = 0.0, si = 0.0;
  int64_t total = (int64_t)D * D;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    int a = (int)(t % D), b = (int)(t / D);
    dcplx p = cmul(L[a + ldl * b], V[b + ldv * a]);
    sr += p.x;
    si += p.y;
  }
  double r = block_sum<kRedThreads>(sr, sh);
  double q = block_sum<kRedThreads>(si, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = r;
    part[2 * blockIdx.x + 1] = q;
  }
}

// X -= tr(rho X) I in one launch: the partial sums of k_trace_prod_partial, added in block
// order by the last block to finish (so the value does not depend on timing), which then
// corrects the diagonal; no trip to the host.  The counter is left at zero.
__global__ void k_regularize(int D, const dcplx* __restrict__ L, int64_t ldl, dcplx* __restrict__ V, int64_t ldv,
                             double* __restrict__ part, unsigned* __restrict__ counter) {
  grid_enter();
  __shared__ double sh[kRedThreads / 32];
  __shared__ double all[2 * kMaxRedBlocks];
  __shared__ double tr[2];
  __shared__ bool last;
  double sr = 0.0, si = 0.0;
  const int64_t total = (int64_t)D * D;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(t % D), b = (int)(t / D);
    const dcplx p = cmul(L[a + ldl * b], V[b + ldv * a]);
    sr += p.x;
    si += p.y;
  }
  const double r = block_sum<kRedThreads>(sr, sh), q = block_sum<kRedThreads>(si, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = r;
    part[2 * blockIdx.x + 1] = q;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = threadIdx.x; i < 2 * (int)gridDim.x; i += blockDim.x) all[i] = __ldcg(&part[i]);
  __syncthreads();
  if (threadIdx.x < 2) {
    double s = 0.0;
#pragma unroll 16
    for (int i = 0; i < (int)gridDim.x; ++i) s += all[2 * i + threadIdx.x];
    tr[threadIdx.x] = s;
  }
  if (threadIdx.x == 0) *counter = 0u;
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const dcplx u = V[i + ldv * i];
    V[i + ldv * i] = make_double2(u.x - tr[0], u.y - tr[1]);
  }
}

__global__ void k_copy2d(int rows, int cols, const dcplx* __restrict__ X, int64_t ldx, dcplx* __restrict__ Y,
                         int64_t ldy, int add) {
  grid_enter();
  int64_t total = (int64_t)rows * cols;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(t % rows), c = (int)(t / rows);
    dcplx v = X[r + ldx * c];
    if (add) {
      dcplx u = Y[r + ldy * c];
      v.x += u.x;
      v.y += u.y;
    }
    Y[r + ldy * c] = v;
  }
}

__global__ void k_add_diag(int D, dcplx* X, int64_t ld, double2 v) {
  grid_enter();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < D; i += gridDim.x * blockDim.x) {
    dcplx u = X[i + ld * i];
    X[i + ld * i] = make_double2(u.x + v.x, u.y + v.y);
  }
}
__global__ void k_fill2d(int rows, int cols, dcplx* Y, int64_t ldy, double2 v) {
  grid_enter();
  int64_t total = (int64_t)rows * cols;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(t % rows), c = (int)(t / rows);
    Y[r + ldy * c] = v;
  }
}

int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 16));
}

inline double2 d2(cplx z) { return make_double2(z.real(), z.imag()); }

void check_launch(Context* ctx) {
  ctx->n_kernels++;
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) throw Error(IMPS_CUDA_ERROR, std::string("kernel launch: ") + cudaGetErrorString(e));
}

}  // namespace

namespace {
// never destroyed: a context may go after the library's statics
std::mutex& pools_mu() {
  static auto* m = new std::mutex;
  return *m;
}
std::set<BlockPool*>& pools() {
  static auto* s = new std::set<BlockPool*>;
  return *s;
}
}  // namespace

BlockPool::BlockPool() {
  std::lock_guard<std::mutex> lock(pools_mu());
  pools().insert(this);
}
BlockPool::~BlockPool() {
  {
    std::lock_guard<std::mutex> lock(pools_mu());
    pools().erase(this);
  }
  trim();
}
void* BlockPool::take(size_t bytes) {
  std::lock_guard<std::mutex> lock(mu_);
  auto it = idle_.find(bytes);
  if (it == idle_.end()) return nullptr;
  void* p = it->second;
  idle_.erase(it);
  held_ -= bytes;
  return p;
}
bool BlockPool::give(void* ptr, size_t bytes) {
  std::lock_guard<std::mutex> lock(mu_);
  if (!open_ || held_ + bytes > kMost) return false;
  idle_.emplace(bytes, ptr);
  held_ += bytes;
  return true;
}
void BlockPool::trim() {
  std::lock_guard<std::mutex> lock(mu_);
  for (auto& kv : idle_) cudaFree(kv.second);
  idle_.clear();
  held_ = 0;
}
void BlockPool::keep(bool on) {
  {
    std::lock_guard<std::mutex> lock(mu_);
    open_ = on;
  }
  if (!on) trim();
}
size_t BlockPool::held() {
  std::lock_guard<std::mutex> lock(mu_);
  return held_;
}
void BlockPool::trim_all() {
  std::lock_guard<std::mutex> lock(pools_mu());
  for (BlockPool* p : pools()) p->trim();
}

static thread_local Context* g_running = nullptr;
RunningCall::RunningCall(Context* c) : ctx(c), old(g_running) {
  if (ctx) {
    ctx->call_mu.lock();
    ctx->calls++;
  }
  g_running = ctx;
}
RunningCall::~RunningCall() {
  g_running = old;
  if (ctx) {
    ctx->calls--;
    ctx->call_mu.unlock();
  }
}

static std::set<Context*>& contexts() {   // under pools_mu
  static auto* s = new std::set<Context*>;
  return *s;
}
void register_context(Context* ctx) {
  std::lock_guard<std::mutex> lock(pools_mu());
  contexts().insert(ctx);
}
void unregister_context(Context* ctx) {
  std::lock_guard<std::mutex> lock(pools_mu());
  contexts().erase(ctx);
}

void give_back_idle() {
  BlockPool::trim_all();
  Context* c = g_running;
  if (c && c->no_scratch == 0 && !c->optional.empty() && !c->capturing()) c->release_optional();
  std::lock_guard<std::mutex> lock(pools_mu());
  for (Context* o : contexts()) {
    if (o == c || !o->call_mu.try_lock()) continue;
    if (o->calls == 0 && !o->optional.empty() && !o->capturing()) o->release_optional();
    o->call_mu.unlock();
  }
}

double* Context::pinned(size_t bytes) {
  if (bytes > host_pinned_bytes) {
    if (host_pinned) cudaFreeHost(host_pinned);
    host_pinned = nullptr;
    size_t b = std::max<size_t>(bytes, 1 << 16);
    IMPS_CUDA(cudaMallocHost((void**)&host_pinned, b));
    host_pinned_bytes = b;
  }
  return host_pinned;
}

static cudaEvent_t pooled_event(Context* ctx) {
  if (!ctx->event_pool.empty()) {
    cudaEvent_t e = ctx->event_pool.back();
    ctx->event_pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  cudaEventCreate(&e);
  return e;
}

ScopedTimer::ScopedTimer(Context* c, const char* n, double f) : ctx(c), flops(f) {
  if (!ctx->profile) return;
  if (!ctx->profile_only.empty() && ctx->profile_only.count(n) == 0) return;
  name = n;
  if (ctx->prof_tag && ctx->prof_tag[0]) name = name + "@" + ctx->prof_tag;
  e0 = pooled_event(ctx);
  e1 = pooled_event(ctx);
  cudaEventRecord(e0, ctx->stream);
}
ScopedTimer::~ScopedTimer() {
  if (e0) {
    cudaEventRecord(e1, ctx->stream);
    ctx->pending.push_back({name, {e0, e1}});
    ctx->pending_flops.push_back(flops);
  }
}

// The error flag rides along with a synchronisation that happens anyway.
static void err_copy(Context* ctx) {
  if (ctx->err_armed || ctx->err_later)
    IMPS_CUDA(cudaMemcpyAsync(ctx->err_host, ctx->err_dev, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
}
static void err_after_sync(Context* ctx) {
  if (!ctx->err_armed && !ctx->err_later) return;
  ctx->err_armed = ctx->err_later = false;
  if (ctx->err_host[0] != 0) {
    ctx->err_host[0] = 0;
    IMPS_CUDA(cudaMemsetAsync(ctx->err_dev, 0, sizeof(int), ctx->stream));
    throw Error(IMPS_TIMEOUT, "a bounded device wait of a GEMM pipeline ran out");
  }
}
void check_device_errors(Context* ctx, bool all) {
  if (ctx->err_armed || (all && ctx->err_later)) synchronize(ctx);
}
void synchronize(Context* ctx) {
  err_copy(ctx);
  IMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  err_after_sync(ctx);
}

namespace {
// Large arrays of the caller's pageable memory go through page-locked chunks, filled or emptied
// by a few threads: one thread's copies (and, into a fresh array, its page faults) take longer
// than the transfer.  The calling thread issues every transfer and event on the context's
// stream, whose handle may name another stream in another thread (cudaStreamPerThread); the
// others move host memory and make no CUDA calls, whose first one in a thread costs some 100
// us.  One staging area per process; a second context that finds it taken, small arrays and
// page-locked ones use the plain copy.
constexpr size_t kStageThreads = 4;   // with the calling one
constexpr size_t kStageSlots = 2 * kStageThreads, kStageChunk = (size_t)1 << 20, kStageMin = (size_t)4 << 20;

struct Staging {
  std::mutex mu;
  char* mem = nullptr;   // kStageSlots chunks
  std::map<int, std::array<cudaEvent_t, kStageSlots>> events;   // of each device
};
Staging& staging() {
  static auto* s = new Staging;   // as long as the process, like the driver's own
  return *s;
}

bool page_locked(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;   // leave it to the plain copy
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// One array's way through the slots.  Thread t moves the t-th contiguous part in host memory
// (its own pages and its own two slots); chunk i is the (i / kStageThreads)-th of part
// i % kStageThreads and uses slot i % kStageSlots, and the transfers go in the order of i.
struct StagedCopy {
  char *dev, *host, *slots;
  size_t bytes, part, n;
  bool to_device;
  cudaStream_t stream;
  cudaEvent_t* ev;
  std::atomic<size_t> limit{0};                  // chunks below may be moved: their slot is free (or full)
  std::atomic<size_t> moved[kStageSlots] = {};   // 1 + the last chunk of the slot that was moved
  std::atomic<bool> stop{false};                 // all is done, or a transfer failed
  cudaError_t error = cudaSuccess;               // (the calling thread's from here)
  size_t issued = 0, done = 0;                   // transfers queued and completed
  size_t mine = 0;                               // the calling thread's next chunk

  size_t offset(size_t i) const { return i % kStageThreads * part + i / kStageThreads * kStageChunk; }
  size_t len(size_t i) const {
    const size_t end = std::min(bytes, (i % kStageThreads + 1) * part), o = offset(i);
    return o < end ? std::min(kStageChunk, end - o) : 0;
  }
  char* slot(size_t i) const { return slots + i % kStageSlots * kStageChunk; }
  void move(size_t i) {
    if (const size_t k = len(i)) {
      if (to_device) std::memcpy(slot(i), host + offset(i), k);
      else std::memcpy(host + offset(i), slot(i), k);
    }
    moved[i % kStageSlots].store(i + 1);
  }
  void work(size_t t) {
    for (size_t i = t; i < n; i += kStageThreads) {
      while (limit.load() <= i) {
        if (stop.load()) return;
        std::this_thread::yield();
      }
      move(i);
    }
    // A core that goes idle with the chunks in its cache makes their transfer wait for it (4 MiB
    // to the device 750 us, 250 with the threads kept until the transfers are done)
    while (!stop.load()) std::this_thread::yield();
  }
  bool ok(cudaError_t e) {
    if (e == cudaSuccess) return true;
    error = e;
    stop.store(true);
    return false;
  }
  void issue() {
    const size_t i = issued, k = len(i);
    char* d = dev + offset(i);
    if (k && !ok(to_device ? cudaMemcpyAsync(d, slot(i), k, cudaMemcpyHostToDevice, stream)
                           : cudaMemcpyAsync(slot(i), d, k, cudaMemcpyDeviceToHost, stream)))
      return;
    if (ok(cudaEventRecord(ev[i % kStageSlots], stream))) ++issued;
  }
  // notes the transfers that have completed
  void poll() {
    while (done < issued) {
      const cudaError_t e = cudaEventQuery(ev[done % kStageSlots]);
      if (e == cudaErrorNotReady) {
        cudaGetLastError();
        break;
      }
      if (!ok(e)) return;
      ++done;
    }
    limit.store(to_device ? done + kStageSlots : done);
  }
  // The calling thread: transfers whose host side is ready, its own part, completions.
  void run(size_t first_missing) {
    limit.store(to_device ? kStageSlots : 0);
    size_t left = 0;   // chunks of the calling thread (and of threads that did not start)
    auto own = [&](size_t i) { return i % kStageThreads == 0 || i % kStageThreads >= first_missing; };
    for (size_t i = 0; i < n; ++i) left += own(i);
    while (error == cudaSuccess && (issued < n || left > 0)) {
      const size_t ready = to_device ? issued + 1 : (issued < kStageSlots ? 0 : issued - kStageSlots + 1);
      if (issued < n && moved[issued % kStageSlots].load() == ready) {
        issue();
        continue;
      }
      poll();
      while (mine < n && !own(mine)) ++mine;
      if (mine < n && mine < limit.load()) {
        move(mine++);
        --left;
      } else {
        std::this_thread::yield();
      }
    }
    while (error == cudaSuccess && done < n) poll();
    for (size_t t = 1; t < first_missing && !to_device && error == cudaSuccess; ++t)   // the others' last chunks
      while (moved[(n - kStageThreads + t) % kStageSlots].load() != n - kStageThreads + t + 1) std::this_thread::yield();
    stop.store(true);
  }
};

// false: not staged, nothing done
bool staged_copy(Context* ctx, void* dev, void* host, size_t bytes, bool to_device) {
  if (bytes < kStageMin || std::thread::hardware_concurrency() < 2 * kStageThreads || page_locked(host)) return false;
  Staging& s = staging();
  std::unique_lock<std::mutex> lock(s.mu, std::try_to_lock);
  if (!lock.owns_lock()) return false;
  if (!s.mem && cudaHostAlloc((void**)&s.mem, kStageSlots * kStageChunk, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    s.mem = nullptr;
    return false;
  }
  auto known = s.events.find(ctx->device);
  if (known == s.events.end()) {
    std::array<cudaEvent_t, kStageSlots> ev{};
    for (auto& e : ev) IMPS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    known = s.events.emplace(ctx->device, ev).first;
  }
  StagedCopy c;
  c.dev = static_cast<char*>(dev);
  c.host = static_cast<char*>(host);
  c.slots = s.mem;
  c.ev = known->second.data();
  c.bytes = bytes;
  c.part = ((bytes + kStageThreads - 1) / kStageThreads + 4095) / 4096 * 4096;
  c.n = kStageThreads * ((c.part + kStageChunk - 1) / kStageChunk);
  c.to_device = to_device;
  c.stream = ctx->stream;
  std::thread th[kStageThreads];
  size_t started = 1;
  for (; started < kStageThreads; ++started) {
    try {
      th[started] = std::thread(&StagedCopy::work, &c, started);
    } catch (const std::system_error&) {
      break;   // no thread to be had: the calling one takes the part
    }
  }
  c.run(started);
  for (auto& t : th)
    if (t.joinable()) t.join();
  // (without an error every transfer is done and has left the slots)
  if (c.error != cudaSuccess) cudaStreamSynchronize(ctx->stream);
  IMPS_CUDA(c.error);
  return true;
}
}  // namespace

void upload(Context* ctx, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  if (!staged_copy(ctx, dst, const_cast<void*>(src), bytes, true))
    IMPS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
  err_copy(ctx);
  IMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  err_after_sync(ctx);
}
void download(Context* ctx, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  // a solver's scalars through page-locked memory: half the latency of a pageable copy
  void* to = bytes <= 65536 ? (void*)ctx->pinned(bytes) : dst;
  if (!staged_copy(ctx, const_cast<void*>(src), dst, bytes, false))
    IMPS_CUDA(cudaMemcpyAsync(to, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  err_copy(ctx);
  IMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  if (to != dst) std::memcpy(dst, to, bytes);
  err_after_sync(ctx);
}

void zcopy(Context* ctx, int64_t n, const dcplx* x, dcplx* y) {
  if (n <= 0 || x == y) return;
  IMPS_CUDA(cudaMemcpyAsync(y, x, n * sizeof(dcplx), cudaMemcpyDeviceToDevice, ctx->stream));
}
void zscal(Context* ctx, int64_t n, cplx a, dcplx* x) {
  if (n <= 0) return;
  launch_kernel(ctx, k_scal, grid_for(n), 256, 0, n, d2(a), x);
  check_launch(ctx);
}
void zaxpy(Context* ctx, int64_t n, cplx a, const dcplx* x, dcplx* y) {
  if (n <= 0) return;
  launch_kernel(ctx, k_axpy, grid_for(n), 256, 0, n, d2(a), x, y);
  check_launch(ctx);
}
void zaxpby(Context* ctx, int64_t n, cplx a, const dcplx* x, cplx b, dcplx* y) {
  if (n <= 0) return;
  launch_kernel(ctx, k_axpby, grid_for(n), 256, 0, n, d2(a), x, d2(b), y, b != cplx(0.0, 0.0));
  check_launch(ctx);
}
void zfill(Context* ctx, int64_t n, cplx v, dcplx* x) {
  if (n <= 0) return;
  launch_kernel(ctx, k_fill, grid_for(n), 256, 0, n, d2(v), x);
  check_launch(ctx);
}
void zset_identity(Context* ctx, int D, dcplx* X, int64_t ld, cplx diag) {
  if (D <= 0) return;
  launch_kernel(ctx, k_set_identity, grid_for((int64_t)D * D), 256, 0, D, X, ld, d2(diag));
  check_launch(ctx);
}

double dznrm2(Context* ctx, int64_t n, const dcplx* x) {
  if (n <= 0) return 0.0;
  int nb = red_blocks(n);
  DevBuf& red = ctx->buf("red_part", (size_t)(nb + 8) * sizeof(double));
  DevBuf& out = ctx->buf("red_out", 64 * sizeof(double));
  ScopedTimer t(ctx, "blas1", (double)n * 16);
  launch_kernel(ctx, k_nrm2_partial, nb, kRedThreads, 0, n, x, red.d());
  check_launch(ctx);
  launch_kernel(ctx, k_final_sum, 1, kRedThreads, 0, nb, 1, red.d(), nb, out.d());
  check_launch(ctx);
  double h;
  download(ctx, &h, out.d(), sizeof(double));
  return std::sqrt(h);
}

cplx zdotc(Context* ctx, int64_t n, const dcplx* x, const dcplx* y) {
  if (n <= 0) return cplx(0.0, 0.0);
  int nb = red_blocks(n);
  DevBuf& red = ctx->buf("red_part", (size_t)(2 * nb + 8) * sizeof(double));
  DevBuf& out = ctx->buf("red_out", 64 * sizeof(double));
  ScopedTimer t(ctx, "blas1", (double)n * 32);
  (void)out;
  launch_kernel(ctx, k_dotc_partial, nb, kRedThreads, 0, n, x, y, red.d());
  check_launch(ctx);
  double h[2];
  {
    // per-block (re, im) partials summed on the host in block order (deterministic)
    std::vector<double> p(2 * nb);
    download(ctx, p.data(), red.d(), p.size() * sizeof(double));
    double sr = 0.0, si = 0.0;
    for (int i = 0; i < nb; ++i) { sr += p[2 * i]; si += p[2 * i + 1]; }
    h[0] = sr;
    h[1] = si;
  }
  return cplx(h[0], h[1]);
}

static void gemv_common(Context* ctx, int64_t n, int nv, const dcplx* V, int64_t ldv, const cplx* coef, dcplx* w,
                        int set) {
  ScopedTimer t(ctx, "orth", (double)n * 16 * (nv + 2));
  int done = 0;
  bool first = true;
  while (done < nv || (first && set)) {
    int cnt = std::min(32, nv - done);
    CoefPack p;
    for (int j = 0; j < cnt; ++j) p.c[j] = d2(coef[done + j]);
    launch_kernel(ctx, k_gemv_acc, grid_for(n), 256, 0, n, cnt, V + ldv * (int64_t)done, ldv, p, w,
                                                      (first && set) ? 1 : 0);
    check_launch(ctx);
    done += cnt;
    first = false;
    if (cnt == 0) break;
  }
}

void zgemv_acc(Context* ctx, int64_t n, int nv, const dcplx* V, int64_t ldv, const cplx* coef, dcplx* w) {
  if (nv <= 0) return;
  gemv_common(ctx, n, nv, V, ldv, coef, w, 0);
}
void zgemv_set(Context* ctx, int64_t n, int nv, const dcplx* V, int64_t ldv, const cplx* coef, dcplx* y) {
  gemv_common(ctx, n, nv, V, ldv, coef, y, 1);
}

double proj_pass(Context* ctx, int64_t n, int nv, const dcplx* V, int64_t ldv, dcplx* w, cplx* h_host,
                 double* nw_old2) {
  // columns of the partials: 2 nv dot columns, then ||w_old||^2, then ||w_new||^2
  const int nb = std::min(red_blocks(n), 592);
  constexpr int CH = 8;
  const int ncol = 2 * nv + 2;
  DevBuf& red = ctx->buf("proj_part", (size_t)nb * ncol * sizeof(double));
  DevBuf& out = ctx->buf("proj_out", (size_t)ncol * sizeof(double));
  ScopedTimer t(ctx, "orth", (double)n * 16 * (2 * nv + 3));
  const int norm_col = nw_old2 ? 2 * nv : -1;
  if (nv == 0 && nw_old2) {
    launch_kernel(ctx, k_proj_dots<CH>, nb, kRedThreads, 0, n, 0, V, ldv, w, red.d(), nb, 0, norm_col);
    check_launch(ctx);
  }
  for (int c0 = 0; c0 < nv; c0 += CH) {
    const int nvc = std::min(CH, nv - c0);
    launch_kernel(ctx, k_proj_dots<CH>, nb, kRedThreads, 0, n, nvc, V + ldv * (int64_t)c0, ldv, w, red.d(), nb, 2 * c0,
                                                         c0 == 0 ? norm_col : -1);
    check_launch(ctx);
  }
  const int ndots = 2 * nv + (nw_old2 ? 1 : 0);
  if (ndots > 0) {
    launch_kernel(ctx, k_final_sum_cols, ndots, kRedThreads, 0, nb, red.d(), nb, out.d());
    check_launch(ctx);
  }
  for (int c0 = 0; c0 < nv || (nv == 0 && c0 == 0); c0 += 32) {
    const int cnt = std::min(32, nv - c0);
    const bool last = c0 + 32 >= nv;
    launch_kernel(ctx, k_proj_update, nb, kRedThreads, 0, n, cnt, V + ldv * (int64_t)c0, ldv, out.d() + 2 * c0, w,
                                                       last ? red.d() + (size_t)nb * (2 * nv + 1) : nullptr);
    check_launch(ctx);
    if (nv == 0) break;
  }
  launch_kernel(ctx, k_final_sum_cols, 1, kRedThreads, 0, nb, red.d() + (size_t)nb * (2 * nv + 1), nb,
                                                       out.d() + 2 * nv + 1);
  check_launch(ctx);
  std::vector<double> hv(ncol);
  download(ctx, hv.data(), out.d(), hv.size() * sizeof(double));
  for (int j = 0; j < nv; ++j) h_host[j] = cplx(hv[2 * j], hv[2 * j + 1]);
  if (nw_old2) *nw_old2 = hv[2 * nv];
  return hv[2 * nv + 1];
}

namespace {
template <int NV>
int gs_blocks_for(int64_t n) {
  // resident blocks per SM by shared memory (the ring plus the static arrays), at most 8
  const int per_sm = std::max(1, std::min(8, (int)((220 * 1024) / (gs_smem_bytes<NV>() + 8 * 1024))));
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + GS_ROWS - 1) / GS_ROWS, (int64_t)148 * per_sm));
}
template <int NV, bool UPDATE>
void launch_gs_kernel(Context* ctx, int nb, int64_t n, int nv, const dcplx* V, int64_t ldv, const double* hdev,
                      dcplx* w, double* part, int64_t ldp) {
  static DeviceOnce attr;
  attr.run(ctx->device, [] {
    IMPS_CUDA(cudaFuncSetAttribute(k_gs_pass<NV, UPDATE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)gs_smem_bytes<NV>()));
  });
  launch_kernel(ctx, k_gs_pass<NV, UPDATE>, nb, GS_THREADS, gs_smem_bytes<NV>(), n, nv, V, ldv, hdev, w, part, ldp);
}
int gs_pass_blocks(int64_t n, int nv) {
  return nv <= 8 ? gs_blocks_for<8>(n) : nv <= 16 ? gs_blocks_for<16>(n) : gs_blocks_for<32>(n);
}
void gs_pass(Context* ctx, bool update, int64_t n, int nv, const dcplx* V, int64_t ldv, const double* hdev, dcplx* w,
             double* part, int64_t ldp, double* out) {
  const int nb = gs_pass_blocks(n, nv);
  if (nv <= 8) {
    if (update) launch_gs_kernel<8, true>(ctx, nb, n, nv, V, ldv, hdev, w, part, ldp);
    else launch_gs_kernel<8, false>(ctx, nb, n, nv, V, ldv, hdev, w, part, ldp);
  } else if (nv <= 16) {
    if (update) launch_gs_kernel<16, true>(ctx, nb, n, nv, V, ldv, hdev, w, part, ldp);
    else launch_gs_kernel<16, false>(ctx, nb, n, nv, V, ldv, hdev, w, part, ldp);
  } else {
    if (update) launch_gs_kernel<32, true>(ctx, nb, n, nv, V, ldv, hdev, w, part, ldp);
    else launch_gs_kernel<32, false>(ctx, nb, n, nv, V, ldv, hdev, w, part, ldp);
  }
  check_launch(ctx);
  launch_kernel(ctx, k_final_sum_cols, 2 * nv + 1, kRedThreads, 0, nb, part, ldp, out);
  check_launch(ctx);
}
const char* kNonFinite =
    "non-finite value (NaN or Inf) in the Krylov iteration: the operator or the start vector holds one";
}  // namespace

double gs_project(Context* ctx, int64_t n, int nv, const dcplx* V, int64_t ldv, dcplx* w, std::vector<cplx>& h) {
  h.assign(nv, cplx(0.0, 0.0));
  if (nv <= 0) {
    const double nw = dznrm2(ctx, n, w);
    IMPS_REQUIRE(std::isfinite(nw), IMPS_INVALID_ARG, kNonFinite);
    return nw;
  }
  if (nv > 32) {
    // wide bases: the chunked two-kernel projection
    std::vector<cplx> h1(nv);
    double nw0 = 0.0;
    double nw1 = proj_pass(ctx, n, nv, V, ldv, w, h1.data(), &nw0);
    IMPS_REQUIRE(std::isfinite(nw0) && std::isfinite(nw1), IMPS_INVALID_ARG, kNonFinite);
    for (int j = 0; j < nv; ++j) h[j] += h1[j];
    for (int pass = 1; pass < 3 && nw1 < 0.5 * nw0; ++pass) {
      nw0 = nw1;
      nw1 = proj_pass(ctx, n, nv, V, ldv, w, h1.data(), nullptr);
      for (int j = 0; j < nv; ++j) h[j] += h1[j];
    }
    return std::sqrt(std::max(nw1, 0.0));
  }
  const int nb = gs_pass_blocks(n, nv);
  const int ncol = 2 * nv + 1;
  DevBuf& part = ctx->buf("gs_part", (size_t)nb * ncol * sizeof(double));
  DevBuf& outb = ctx->buf("gs_out", (size_t)3 * ncol * sizeof(double));
  double* out[3] = {outb.d(), outb.d() + ncol, outb.d() + 2 * ncol};
  ScopedTimer t(ctx, "orth", (double)n * 16 * (nv + 1));
  // projection 1 (dots of w), then its update fused with the dots of projection 2
  gs_pass(ctx, false, n, nv, V, ldv, nullptr, w, part.d(), nb, out[0]);
  gs_pass(ctx, true, n, nv, V, ldv, out[0], w, part.d(), nb, out[1]);
  std::vector<double> hv(2 * ncol);
  download(ctx, hv.data(), out[0], hv.size() * sizeof(double));
  double nw0 = hv[2 * nv], nw1 = hv[ncol + 2 * nv];
  IMPS_REQUIRE(std::isfinite(nw0) && std::isfinite(nw1), IMPS_INVALID_ARG, kNonFinite);
  for (int j = 0; j < nv; ++j) h[j] = cplx(hv[2 * j], hv[2 * j + 1]);
  // iterative refinement (KrylovKit's ClassicalGramSchmidtIR, eta = 1/sqrt(2)): apply the
  // pending projection while the last one shrank ||w|| below eta of its previous value,
  // at most three projections in all
  int cur = 1;
  std::vector<double> hn(hv.begin() + ncol, hv.end());
  for (int pass = 1; pass < 3 && nw1 < 0.5 * nw0; ++pass) {
    const int nxt = cur == 1 ? 2 : 1;
    gs_pass(ctx, true, n, nv, V, ldv, out[cur], w, part.d(), nb, out[nxt]);
    for (int j = 0; j < nv; ++j) h[j] += cplx(hn[2 * j], hn[2 * j + 1]);
    download(ctx, hn.data(), out[nxt], ncol * sizeof(double));
    nw0 = nw1;
    nw1 = hn[2 * nv];
    IMPS_REQUIRE(std::isfinite(nw1), IMPS_INVALID_ARG, kNonFinite);
    cur = nxt;
  }
  return std::sqrt(std::max(nw1, 0.0));
}

void zconj_transpose(Context* ctx, int m, int n, const dcplx* X, int64_t ldx, dcplx* Y, int64_t ldy) {
  if (m <= 0 || n <= 0) return;
  dim3 grid((m + 31) / 32, (n + 31) / 32), block(32, 8);
  ScopedTimer t(ctx, "permute", (double)m * n * 32);
  launch_kernel(ctx, k_conj_transpose, grid, block, 0, m, n, X, ldx, Y, ldy);
  check_launch(ctx);
}

cplx ztrace_prod(Context* ctx, int D, const dcplx* L, int64_t ldl, const dcplx* V, int64_t ldv) {
  int64_t n = (int64_t)D * D;
  int nb = red_blocks(n);
  DevBuf& red = ctx->buf("red_part", (size_t)(2 * nb + 8) * sizeof(double));
  launch_kernel(ctx, k_trace_prod_partial, nb, kRedThreads, 0, D, L, ldl, V, ldv, red.d());
  check_launch(ctx);
  std::vector<double> p(2 * nb);
  download(ctx, p.data(), red.d(), p.size() * sizeof(double));
  double sr = 0.0, si = 0.0;
  for (int i = 0; i < nb; ++i) { sr += p[2 * i]; si += p[2 * i + 1]; }
  return cplx(sr, si);
}

void zregularize(Context* ctx, int D, const dcplx* rho, int64_t ldr, dcplx* X, int64_t ldx) {
  const int nb = red_blocks((int64_t)D * D);
  DevBuf& red = ctx->buf("red_part", (size_t)(2 * nb + 8) * sizeof(double));
  launch_kernel(ctx, k_regularize, nb, kRedThreads, 0, D, rho, ldr, X, ldx, red.d(), ctx->counters);
  check_launch(ctx);
}

void zcopy2d(Context* ctx, int rows, int cols, const dcplx* X, int64_t ldx, dcplx* Y, int64_t ldy) {
  if (rows <= 0 || cols <= 0) return;
  launch_kernel(ctx, k_copy2d, grid_for((int64_t)rows * cols), 256, 0, rows, cols, X, ldx, Y, ldy, 0);
  check_launch(ctx);
}

void zadd_diag(Context* ctx, int D, dcplx* X, int64_t ld, cplx v) {
  if (D <= 0) return;
  launch_kernel(ctx, k_add_diag, grid_for(D), 256, 0, D, X, ld, d2(v));
  check_launch(ctx);
}
void zfill2d(Context* ctx, int rows, int cols, cplx v, dcplx* Y, int64_t ldy) {
  if (rows <= 0 || cols <= 0) return;
  launch_kernel(ctx, k_fill2d, grid_for((int64_t)rows * cols), 256, 0, rows, cols, Y, ldy, d2(v));
  check_launch(ctx);
}

}  // namespace imps
