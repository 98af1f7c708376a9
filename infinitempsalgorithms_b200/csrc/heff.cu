// Effective Hamiltonians and transfer pushes as GEMM -> level mix -> GEMM.
//
//   AC:  T1 = GL (Dl m x Dl) x (Dl x d Dr)            [effective.jl:90-102]
//        T2[b,u,c,j] = sum_{i,s} W[i,u,j,s] T1[b,i,s,c] (block-sparse level mix)
//        y  = T2 (Dl d x Dr n) GR (Dr n x Dr)
//   C:   U  = x (D x D) GR (D x n D);  y = GLp (D x D n) U (D n x D)   [effective.jl:72-76]
//   pushes: the same two-GEMM pattern with conj(A) on one side    [transfermatrix.jl, envs.jl:104-231]
#include "imps_internal.h"

#include <algorithm>

namespace imps {
namespace {

constexpr int kMaxNz = 256;
constexpr int kMaxQ = 64;

struct MixArgs {
  int Db, R, P, Q, S, Cn;
  int64_t in_r, in_s, in_c, out_p, out_q, out_c;
  double2 scale;
  int nq;
  short qval[kMaxQ];
  short qstart[kMaxQ + 1];
  short rval[kMaxNz];
  unsigned long long* row_max;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// MAX: also the rows' maxima for the split engine that takes `out` next (it would read all of
// `out` again for them).  Only their exponents count there, so the upper words are compared
// as integers (FP64 maxima made the kernel slower than the extra read); a NaN is ignored, as
// a maximum of doubles would.
__device__ __forceinline__ uint32_t upper_word(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
  return h > 0x7ff00000u ? 0u : h;
}
template <int P, bool MAX>
__global__ void __launch_bounds__(128) k_level_mix(const MixArgs a, const double2* __restrict__ M,
                                                   const double2* __restrict__ in, double2* __restrict__ out) {
  grid_enter();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= a.Db) return;
  uint32_t top[MAX ? P : 1];
#pragma unroll
  for (int p = 0; p < (MAX ? P : 1); ++p) top[p] = 0u;
  for (int c = blockIdx.y; c < a.Cn; c += gridDim.y) {
    const double2* inb = in + b + a.in_c * c;
    double2* outb = out + b + a.out_c * c;
    for (int iq = 0; iq < a.nq; ++iq) {
      const int q = a.qval[iq];
      double2 acc[P];
#pragma unroll
      for (int p = 0; p < P; ++p) acc[p] = make_double2(0.0, 0.0);
      for (int t = a.qstart[iq]; t < a.qstart[iq + 1]; ++t) {
        const int r = a.rval[t];
        for (int s = 0; s < a.S; ++s) {
          const double2 v = inb[a.in_r * r + a.in_s * s];
#pragma unroll
          for (int p = 0; p < P; ++p) {
            const double2 w = __ldg(&M[r + (int64_t)a.R * (p + (int64_t)P * (q + (int64_t)a.Q * s))]);
            acc[p].x = fma(w.x, v.x, fma(-w.y, v.y, acc[p].x));
            acc[p].y = fma(w.x, v.y, fma(w.y, v.x, acc[p].y));
          }
        }
      }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const double2 v = cmul(a.scale, acc[p]);
        outb[a.out_p * p + a.out_q * q] = v;
        if (MAX) top[p] = max(top[p], max(upper_word(v.x), upper_word(v.y)));
      }
    }
  }
  if (MAX) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const unsigned long long bits = (unsigned long long)top[p] << 32;
      unsigned long long* slot = &a.row_max[b + a.Db * p];
      if (bits > *(volatile unsigned long long*)slot) atomicMax(slot, bits);
    }
  }
}

// The whole AC application of a small state in one launch (GEMM, level mix, GEMM as above), a
// cluster of 8 CTAs: CTA r takes columns [Dr r / 8, Dr (r + 1) / 8) of x through both steps,
//   T1 = GL x,  T2 = W T1,  y_r = T2 GR  (its share of the sum over c),
// and then adds element block r of the eight partial results in rank order.  All operands
// and intermediates in shared memory; a thread forms 4 columns of a row of a product.  Bound by
// launch and shared-memory latency: TFIM D = 16 8.2 us a call, 16.4 us in three
// launches; the two meet near 7e5 complex multiply-adds (XXZ D = 32 18.5 and 20 us, TFIM
// D = 40 22.5 and 19 us).
constexpr int kSmallCl = 8, kSmallNt = 256;

struct SmallShape {
  int Dl, Dr, m, d;
  int64_t gr_ld;
  int wsz;       // elements of the MPO tensor
};
struct SmallLayout {   // offsets into shared memory, in elements
  int gl, x, gr, w, t1, t2, y, total;
};
__host__ __device__ inline SmallLayout small_layout(const SmallShape& h, int nq) {
  const int nc = (h.Dr + kSmallCl - 1) / kSmallCl;
  SmallLayout o;
  o.gl = 0;
  o.x = o.gl + h.Dl * h.m * h.Dl;
  o.gr = o.x + h.Dl * h.d * nc;
  o.w = o.gr + nc * nq * h.Dr;
  o.t1 = o.w + h.wsz;
  o.t2 = o.t1 + h.Dl * h.m * h.d * nc;
  o.y = o.t2 + h.Dl * h.d * nc * nq;
  o.total = o.y + h.Dl * h.d * h.Dr;
  return o;
}

// out[r + rows c] = sum_k A[r + rows k] B[c, k], 4 columns c a thread; B(c, k) = b[c cs + k ks]
__device__ __forceinline__ void small_gemm(int rows, int cols, int K, const double2* a, const double2* b, int cs, int ks,
                                           double2* out) {
  const int groups = (cols + 3) / 4;
  for (int t = threadIdx.x; t < rows * groups; t += kSmallNt) {
    const int r = t % rows, c0 = t / rows * 4;
    double2 acc[4];
    const double2* bp[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[j] = make_double2(0.0, 0.0);
      bp[j] = b + min(c0 + j, cols - 1) * cs;
    }
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      const double2 v = a[r + rows * k];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 w = bp[j][k * ks];
        acc[j].x = fma(v.x, w.x, fma(-v.y, w.y, acc[j].x));
        acc[j].y = fma(v.x, w.y, fma(v.y, w.x, acc[j].y));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c0 + j < cols) out[r + rows * (c0 + j)] = acc[j];
  }
}

__global__ void __cluster_dims__(kSmallCl, 1, 1) __launch_bounds__(kSmallNt)
    k_ac_small(const SmallShape h, const MixArgs mx, const double2* __restrict__ GL, const double2* __restrict__ GR,
               const double2* __restrict__ W, const double2* __restrict__ x, double2* __restrict__ y) {
  grid_enter();
  extern __shared__ __align__(16) double2 sm[];
  const SmallLayout o = small_layout(h, mx.nq);
  const int tid = threadIdx.x;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int c0 = h.Dr * (int)rank / kSmallCl, nc = h.Dr * ((int)rank + 1) / kSmallCl - c0;
  const int rows1 = h.Dl * h.m, rowsY = h.Dl * h.d, nk = nc * mx.nq;
  for (int e = tid; e < rows1 * h.Dl; e += kSmallNt) sm[o.gl + e] = GL[e];
  for (int e = tid; e < rowsY * nc; e += kSmallNt) sm[o.x + e] = x[(int64_t)rowsY * c0 + e];
  for (int e = tid; e < nk * h.Dr; e += kSmallNt) {
    const int k = e % nk, c = e / nk;   // k = cl + nc iq
    sm[o.gr + e] = GR[c0 + k % nc + h.Dr * mx.qval[k / nc] + h.gr_ld * c];
  }
  for (int e = tid; e < h.wsz; e += kSmallNt) sm[o.w + e] = W[e];
  __syncthreads();
  // T1[(b, i), (s, c)]
  if (nc > 0) small_gemm(rows1, h.d * nc, h.Dl, sm + o.gl, sm + o.x, h.Dl, 1, sm + o.t1);
  __syncthreads();
  // T2[(b, u), (c, iq)]
  for (int t = tid; t < rowsY * nk; t += kSmallNt) {
    const int b = t % h.Dl, u = t / h.Dl % h.d, k = t / rowsY, cl = k % nc, iq = k / nc;
    double2 acc = make_double2(0.0, 0.0);
    for (int e = mx.qstart[iq]; e < mx.qstart[iq + 1]; ++e) {
      const int r = mx.rval[e];
      for (int s = 0; s < h.d; ++s) {
        const double2 v = sm[o.t1 + b + h.Dl * r + rows1 * (s + h.d * cl)];
        const double2 w = sm[o.w + r + mx.R * (u + h.d * (mx.qval[iq] + mx.Q * s))];
        acc.x = fma(w.x, v.x, fma(-w.y, v.y, acc.x));
        acc.y = fma(w.x, v.y, fma(w.y, v.x, acc.y));
      }
    }
    sm[o.t2 + t] = acc;
  }
  __syncthreads();
  small_gemm(rowsY, h.Dr, nk, sm + o.t2, sm + o.gr, nk, 1, sm + o.y);
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int ny = rowsY * h.Dr, e0 = (int)((int64_t)ny * rank / kSmallCl), e1 = (int)((int64_t)ny * (rank + 1) / kSmallCl);
  for (int e = e0 + tid; e < e1; e += kSmallNt) {
    const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(sm + o.y + e));
    double2 v[kSmallCl];
#pragma unroll
    for (uint32_t q = 0; q < kSmallCl; ++q) {
      uint32_t a;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(q));
      asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[q].x), "=d"(v[q].y) : "r"(a) : "memory");
    }
    double2 acc = v[0];
#pragma unroll
    for (int q = 1; q < kSmallCl; ++q) {
      acc.x += v[q].x;
      acc.y += v[q].y;
    }
    y[e] = acc;
  }
  // no CTA leaves while a peer can still read its shared memory
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void k_scale_cols_rows(int m, int n, int k, dcplx* Q, int64_t ldq, dcplx* R, int64_t ldr,
                                  const dcplx* __restrict__ ph) {
  grid_enter();
  // Q[:, i] *= ph[i] (m x k), R[i, :] *= conj(ph[i]) (k x n)
  int64_t tq = (int64_t)m * k, tr = (int64_t)k * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tq + tr; t += (int64_t)gridDim.x * blockDim.x) {
    if (t < tq) {
      int r = (int)(t % m), c = (int)(t / m);
      Q[r + ldq * c] = cmul(ph[c], Q[r + ldq * c]);
    } else {
      int64_t u = t - tq;
      int r = (int)(u % k), c = (int)(u / k);
      double2 p = ph[r];
      R[r + ldr * c] = cmul(make_double2(p.x, -p.y), R[r + ldr * c]);
    }
  }
}

}  // namespace

static void mix_args(const MixPlan& plan, const std::pair<int, int>* nz_in, int nnz, MixArgs& a) {
  a.Db = plan.Db; a.R = plan.R; a.P = plan.P; a.Q = plan.Q; a.S = plan.S; a.Cn = plan.C;
  a.in_r = plan.in_r; a.in_s = plan.in_s; a.in_c = plan.in_c;
  a.out_p = plan.out_p; a.out_q = plan.out_q; a.out_c = plan.out_c;
  a.scale = make_double2(plan.scale.real(), plan.scale.imag());
  a.row_max = plan.row_max;
  IMPS_REQUIRE(nnz <= kMaxNz, IMPS_INVALID_ARG, "level_mix: too many MPO blocks");
  // group the nonzero (r, q) blocks by q (insertion sort into a fixed array: no heap use)
  std::pair<int, int> nz[kMaxNz];
  for (int t = 0; t < nnz; ++t) {
    std::pair<int, int> v = nz_in[t];
    int u = t;
    while (u > 0 && (nz[u - 1].second > v.second || (nz[u - 1].second == v.second && nz[u - 1].first > v.first))) {
      nz[u] = nz[u - 1];
      --u;
    }
    nz[u] = v;
  }
  a.nq = 0;
  for (int t = 0; t < nnz; ++t) {
    if (a.nq == 0 || a.qval[a.nq - 1] != nz[t].second) {
      IMPS_REQUIRE(a.nq < kMaxQ, IMPS_INVALID_ARG, "level_mix: too many MPO levels");
      a.qval[a.nq] = (short)nz[t].second;
      a.qstart[a.nq] = (short)t;
      a.nq++;
    }
    a.rval[t] = (short)nz[t].first;
  }
  a.qstart[a.nq] = (short)nnz;
}

void level_mix_nz(Context* ctx, const MixPlan& plan, const std::pair<int, int>* nz_in, int nnz, const dcplx* in,
                  dcplx* out) {
  MixArgs a;
  mix_args(plan, nz_in, nnz, a);
  if (a.nq == 0 || plan.Db <= 0 || plan.C <= 0) return;
  dim3 block(128);
  dim3 grid((plan.Db + 127) / 128, std::min(plan.C, 65535));
  if (plan.row_max)   // several columns a block: fewer meetings at the maxima
    grid.y = std::min<unsigned>(grid.y, std::max(1u, (unsigned)(ctx->num_sms * 16) / grid.x));
  double bytes = 16.0 * plan.Db * (double)plan.C * (plan.R * plan.S + plan.P * a.nq);
  ScopedTimer t(ctx, "level_mix", bytes);
  switch (plan.P) {
#define IMPS_MIX_CASE(PP) \
  case PP:                                                                                  \
    if (plan.row_max) launch_kernel(ctx, k_level_mix<PP, true>, grid, block, 0, a, plan.M, in, out); \
    else launch_kernel(ctx, k_level_mix<PP, false>, grid, block, 0, a, plan.M, in, out);             \
    break;
    IMPS_MIX_CASE(1) IMPS_MIX_CASE(2) IMPS_MIX_CASE(3) IMPS_MIX_CASE(4)
    IMPS_MIX_CASE(5) IMPS_MIX_CASE(6) IMPS_MIX_CASE(7) IMPS_MIX_CASE(8)
#undef IMPS_MIX_CASE
    default: throw Error(IMPS_INVALID_ARG, "level_mix: physical dimension above 8 is not supported");
  }
  ctx->n_kernels++;
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) throw Error(IMPS_CUDA_ERROR, std::string("level_mix launch: ") + cudaGetErrorString(e));
}

void level_mix(Context* ctx, const MixPlan& plan, const dcplx* in, dcplx* out) {
  level_mix_nz(ctx, plan, plan.nz.data(), (int)plan.nz.size(), in, out);
}

// Phase fix shared by qrpos/lqpos (see linalg.cu)
void scale_q_r(Context* ctx, int m, int n, int k, dcplx* Q, int64_t ldq, dcplx* R, int64_t ldr, const dcplx* ph) {
  int64_t tot = (int64_t)m * k + (int64_t)k * n;
  int g = (int)std::min<int64_t>((tot + 255) / 256, 148 * 16);
  launch_kernel(ctx, k_scale_cols_rows, std::max(g, 1), 256, 0, m, n, k, Q, ldq, R, ldr, ph);
  ctx->n_kernels++;
}

// ---------------------------------------------------------------------------
// AC / C effective Hamiltonians
// ---------------------------------------------------------------------------
void ac_apply(Context* ctx, const imps_envs* envs, const imps_mpo* mpo, int site, const dcplx* x, dcplx* y,
              const MpoSite* Wover, const dcplx* GRover, int64_t GRover_ld) {
  const MpoSite& W = Wover ? *Wover : mpo->sites[site % mpo->N];
  const int Dl = envs->Dl[site], Dr = envs->Dr[site];
  const int m = W.m, d = W.d, n = W.n;
  IMPS_REQUIRE(m == envs->ml[site], IMPS_DIM_MISMATCH, "ac_apply: MPO left levels != environment levels");
  const dcplx* GL = envs->lefts[site].z();
  const dcplx* GR = GRover ? GRover : envs->rights[site].z();
  IMPS_REQUIRE(GRover || n == envs->nr[site], IMPS_DIM_MISMATCH, "ac_apply: MPO right levels != environment");
  const int64_t gr_ld = GRover ? GRover_ld : (int64_t)Dr * n;
  ctx->n_ac_apply++;
  const int64_t t1n = (int64_t)Dl * m * d * Dr, t2n = (int64_t)Dl * d * Dr * n;
  MixPlan pl;
  pl.Db = Dl; pl.R = m; pl.P = d; pl.Q = n; pl.S = d; pl.C = Dr;
  pl.in_r = Dl; pl.in_s = (int64_t)Dl * m; pl.in_c = (int64_t)Dl * m * d;
  pl.out_p = Dl; pl.out_q = (int64_t)Dl * d * Dr; pl.out_c = (int64_t)Dl * d;
  pl.M = W.Wdev.z();
  pl.nz = W.nz;
  // Small states in one launch while its 1/8 of the products per SM (16 complex multiply-adds
  // a clock) stays below the three launches' time, everything fits in shared memory and every
  // level is written (a level without blocks is multiplied as a zero by the general path).
  // The split engine never takes products this small.
  const double macs = (double)Dl * m * d * Dr * Dl + (double)Dl * d * Dr * Dr * n;
  if (macs <= 7e5 && !ctx->ordered_sums() && ctx->fp64_engine != 1 && (int)W.nz.size() <= kMaxNz && n <= kMaxQ) {
    MixArgs a;
    mix_args(pl, pl.nz.data(), (int)pl.nz.size(), a);
    const SmallShape h{Dl, Dr, m, d, gr_ld, m * d * n * d};
    const size_t bytes = (size_t)small_layout(h, a.nq).total * sizeof(dcplx);
    if (a.nq == n && bytes <= 220 * 1024) {
      static DeviceOnce attr;
      attr.run(ctx->device, [] {
        IMPS_CUDA(cudaFuncSetAttribute(k_ac_small, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
      });
      ScopedTimer t(ctx, "ac_small", 8.0 * macs);
      ctx->gemm_flops += 8.0 * macs;
      launch_kernel(ctx, k_ac_small, kSmallCl, kSmallNt, bytes, h, a, GL, GR, W.Wdev.z(), x, y);
      ctx->n_kernels++;
      cudaError_t e = cudaPeekAtLastError();
      if (e != cudaSuccess) throw Error(IMPS_CUDA_ERROR, std::string("ac_small launch: ") + cudaGetErrorString(e));
      return;
    }
  }
  DevBuf& T1 = ctx->buf("ac_t1", t1n * sizeof(dcplx));
  DevBuf& T2 = ctx->buf("ac_t2", t2n * sizeof(dcplx));
  zgemm(ctx, OP_N, OP_N, Dl * m, d * Dr, Dl, 1.0, GL, (int64_t)Dl * m, 0, x, Dl, 0, 0.0, T1.z(), (int64_t)Dl * m, 0, 1);
  // levels q without any nonzero block must read as zero in the second GEMM
  {
    std::vector<bool> hit(n, false);
    for (auto& b : W.nz) hit[b.second] = true;
    for (int q = 0; q < n; ++q)
      if (!hit[q]) zfill(ctx, (int64_t)Dl * d * Dr, 0.0, T2.z() + (int64_t)Dl * d * Dr * q);
  }
  struct Forget {   // the maxima are for this product only, whatever becomes of it
    Context* ctx;
    ~Forget() { ctx->max_ready = nullptr; }
  } forget{ctx};
  pl.row_max = split_collect_max(ctx, T2.z(), Dl * d, Dr, Dr * n);
  level_mix(ctx, pl, T1.z(), T2.z());
  zgemm(ctx, OP_N, OP_N, Dl * d, Dr, Dr * n, 1.0, T2.z(), (int64_t)Dl * d, 0, GR, gr_ld, 0, 0.0, y,
        (int64_t)Dl * d, 0, 1);
}

void ensure_GLp(Context* ctx, imps_envs* envs, int l) {
  if (envs->GLp_valid[l]) return;
  const int D = envs->Dl[l], w = envs->ml[l];
  envs->GLp[l].ensure((size_t)D * D * w * sizeof(dcplx));
  // GLp[a + D (a' + D w)] = GL[a, w, a'] via the level mix with an identity level map
  DevBuf& Id = ctx->buf("glp_id", (size_t)w * w * sizeof(dcplx));
  std::vector<cplx> idh((size_t)w * w, cplx(0.0, 0.0));
  for (int i = 0; i < w; ++i) idh[i + (size_t)w * i] = 1.0;
  upload(ctx, Id.ptr, idh.data(), idh.size() * sizeof(dcplx));
  MixPlan pl;
  pl.Db = D; pl.R = w; pl.P = 1; pl.Q = w; pl.S = 1; pl.C = D;
  pl.in_r = D; pl.in_s = 0; pl.in_c = (int64_t)D * w;
  pl.out_p = 0; pl.out_q = (int64_t)D * D; pl.out_c = D;
  pl.M = Id.z();
  for (int i = 0; i < w; ++i) pl.nz.push_back({i, i});
  level_mix(ctx, pl, envs->lefts[l].z(), envs->GLp[l].z());
  envs->GLp_valid[l] = true;
}

void c_apply(Context* ctx, imps_envs* envs, int site, const dcplx* x, dcplx* y) {
  const int N = envs->N;
  const int l1 = (site + 1) % N;
  const int D = envs->Dr[site];
  const int w = envs->nr[site];
  IMPS_REQUIRE(envs->Dl[l1] == D && envs->ml[l1] == w, IMPS_DIM_MISMATCH, "c_apply: environment shapes disagree");
  ensure_GLp(ctx, envs, l1);
  ctx->n_c_apply++;
  DevBuf& U = ctx->buf("c_u", (size_t)D * D * w * sizeof(dcplx));
  zgemm(ctx, OP_N, OP_N, D, w * D, D, 1.0, x, D, 0, envs->rights[site].z(), D, 0, 0.0, U.z(), D, 0, 1);
  zgemm(ctx, OP_N, OP_N, D, D, D * w, 1.0, envs->GLp[l1].z(), D, 0, U.z(), (int64_t)D * w, 0, 0.0, y, D, 0, 1);
}

// ---------------------------------------------------------------------------
// Transfer pushes
// ---------------------------------------------------------------------------
void push_left_id(Context* ctx, int Dl, int d, int Dr, const dcplx* L, const dcplx* above, const dcplx* below,
                  dcplx* out) {
  ctx->n_push++;
  DevBuf& Y = ctx->buf("push_y", (size_t)Dl * d * Dr * sizeof(dcplx));
  zgemm(ctx, OP_N, OP_N, Dl, d * Dr, Dl, 1.0, L, Dl, 0, above, Dl, 0, 0.0, Y.z(), Dl, 0, 1);
  zgemm(ctx, OP_C, OP_N, Dr, Dr, Dl * d, 1.0, below, (int64_t)Dl * d, 0, Y.z(), (int64_t)Dl * d, 0, 0.0, out, Dr, 0, 1);
}

void push_right_id(Context* ctx, int Dl, int d, int Dr, const dcplx* R, const dcplx* above, const dcplx* below,
                   dcplx* out) {
  ctx->n_push++;
  DevBuf& Y = ctx->buf("push_y", (size_t)Dl * d * Dr * sizeof(dcplx));
  zgemm(ctx, OP_N, OP_N, Dl * d, Dr, Dr, 1.0, above, (int64_t)Dl * d, 0, R, Dr, 0, 0.0, Y.z(), (int64_t)Dl * d, 0, 1);
  zgemm(ctx, OP_N, OP_C, Dl, Dl, d * Dr, 1.0, Y.z(), Dl, 0, below, Dl, 0, 0.0, out, Dl, 0, 1);
}

void push_left_levels(Context* ctx, const MpoSite& W, int Dl, int d, int Dr, const dcplx* L, int64_t L_level_stride,
                      int64_t L_ld, const std::vector<std::pair<int, int>>& blocks, int q_count,
                      const std::vector<int>& q_targets, const dcplx* A, dcplx* out, int64_t out_level_stride,
                      int64_t out_ld, bool accumulate) {
  (void)q_count;
  if (blocks.empty()) return;
  ctx->n_push++;
  std::vector<int> ls;
  for (auto& b : blocks) ls.push_back(b.first);
  std::sort(ls.begin(), ls.end());
  ls.erase(std::unique(ls.begin(), ls.end()), ls.end());
  const int64_t ysz = (int64_t)Dl * d * Dr;
  DevBuf& Y = ctx->buf("pushl_y", (size_t)ysz * W.m * sizeof(dcplx));
  DevBuf& Z = ctx->buf("pushl_z", (size_t)ysz * W.n * sizeof(dcplx));
  for (int l : ls)
    zgemm(ctx, OP_N, OP_N, Dl, d * Dr, Dl, 1.0, L + L_level_stride * l, L_ld, 0, A, Dl, 0, 0.0, Y.z() + ysz * l, Dl,
          0, 1);
  MixPlan pl;
  pl.Db = Dl; pl.R = W.m; pl.P = d; pl.Q = W.n; pl.S = d; pl.C = Dr;
  pl.in_r = ysz; pl.in_s = Dl; pl.in_c = (int64_t)Dl * d;
  pl.out_p = Dl; pl.out_q = ysz; pl.out_c = (int64_t)Dl * d;
  pl.M = W.Wdev.z();
  pl.nz = blocks;
  level_mix(ctx, pl, Y.z(), Z.z());
  for (int q : q_targets) {
    bool any = false;
    for (auto& b : blocks) any |= (b.second == q);
    if (!any) continue;
    zgemm(ctx, OP_C, OP_N, Dr, Dr, Dl * d, 1.0, A, (int64_t)Dl * d, 0, Z.z() + ysz * q, (int64_t)Dl * d, 0,
          accumulate ? 1.0 : 0.0, out + out_level_stride * q, out_ld, 0, 1);
  }
}

void push_right_levels(Context* ctx, const MpoSite& W, int Dl, int d, int Dr, const dcplx* R,
                       int64_t R_level_stride, int64_t R_ld, const std::vector<std::pair<int, int>>& blocks,
                       const std::vector<int>& q_targets, const dcplx* A, dcplx* out, int64_t out_level_stride,
                       int64_t out_ld, bool accumulate) {
  // out_i = sum_{(i,l)} push_slice_right(R_l, W[i,:,l,:], A); blocks are (i, l) pairs
  if (blocks.empty()) return;
  ctx->n_push++;
  std::vector<int> ls;
  for (auto& b : blocks) ls.push_back(b.second);
  std::sort(ls.begin(), ls.end());
  ls.erase(std::unique(ls.begin(), ls.end()), ls.end());
  const int64_t ysz = (int64_t)Dl * d * Dr;
  DevBuf& Y = ctx->buf("pushr_y", (size_t)ysz * W.n * sizeof(dcplx));
  DevBuf& Z = ctx->buf("pushr_z", (size_t)ysz * W.m * sizeof(dcplx));
  for (int l : ls)
    zgemm(ctx, OP_N, OP_N, Dl * d, Dr, Dr, 1.0, A, (int64_t)Dl * d, 0, R + R_level_stride * l, R_ld, 0, 0.0,
          Y.z() + ysz * l, (int64_t)Dl * d, 0, 1);
  // Z_i[a', u, b] = sum_{l, s} W[i, u, l, s] Y_l[a', s, b]: mixing over the transposed tensor
  MixPlan pl;
  pl.Db = Dl; pl.R = W.n; pl.P = d; pl.Q = W.m; pl.S = d; pl.C = Dr;
  pl.in_r = ysz; pl.in_s = Dl; pl.in_c = (int64_t)Dl * d;
  pl.out_p = Dl; pl.out_q = ysz; pl.out_c = (int64_t)Dl * d;
  pl.M = W.Wdev.z() + (int64_t)W.m * W.d * W.n * W.d;  // transposed copy Wt[j,u,i,s] = W[i,u,j,s]
  for (auto& b : blocks) pl.nz.push_back({b.second, b.first});
  level_mix(ctx, pl, Y.z(), Z.z());
  for (int q : q_targets) {
    bool any = false;
    for (auto& b : blocks) any |= (b.first == q);
    if (!any) continue;
    zgemm(ctx, OP_N, OP_C, Dl, Dl, d * Dr, 1.0, Z.z() + ysz * q, Dl, 0, A, Dl, 0, accumulate ? 1.0 : 0.0,
          out + out_level_stride * q, out_ld, 0, 1);
  }
}

void push_mpo_left(Context* ctx, const MpoSite& W, int Dl, int d, int Dr, const dcplx* L, const dcplx* A, dcplx* out) {
  ctx->n_push++;
  const int m = W.m, n = W.n;
  DevBuf& Y = ctx->buf("ac_t1", (size_t)Dl * m * d * Dr * sizeof(dcplx));
  DevBuf& Z = ctx->buf("ac_t2", (size_t)Dl * d * n * Dr * sizeof(dcplx));
  zgemm(ctx, OP_N, OP_N, Dl * m, d * Dr, Dl, 1.0, L, (int64_t)Dl * m, 0, A, Dl, 0, 0.0, Y.z(), (int64_t)Dl * m, 0, 1);
  MixPlan pl;
  pl.Db = Dl; pl.R = m; pl.P = d; pl.Q = n; pl.S = d; pl.C = Dr;
  pl.in_r = Dl; pl.in_s = (int64_t)Dl * m; pl.in_c = (int64_t)Dl * m * d;
  pl.out_p = Dl; pl.out_q = (int64_t)Dl * d; pl.out_c = (int64_t)Dl * d * n;
  pl.M = W.Wdev.z();
  pl.nz = W.nz;
  std::vector<bool> hit(n, false);
  for (auto& b : W.nz) hit[b.second] = true;
  bool any_missing = false;
  for (int q = 0; q < n; ++q) any_missing |= !hit[q];
  if (any_missing) zfill(ctx, (int64_t)Dl * d * n * Dr, 0.0, Z.z());
  level_mix(ctx, pl, Y.z(), Z.z());
  zgemm(ctx, OP_C, OP_N, Dr, n * Dr, Dl * d, 1.0, A, (int64_t)Dl * d, 0, Z.z(), (int64_t)Dl * d, 0, 0.0, out, Dr, 0, 1);
}

void push_mpo_right(Context* ctx, const MpoSite& W, int Dl, int d, int Dr, const dcplx* R, const dcplx* A,
                    dcplx* out) {
  ctx->n_push++;
  const int m = W.m, n = W.n;
  DevBuf& Y = ctx->buf("ac_t1", (size_t)Dl * d * n * Dr * sizeof(dcplx));
  DevBuf& Z = ctx->buf("ac_t2", (size_t)Dl * m * d * Dr * sizeof(dcplx));
  zgemm(ctx, OP_N, OP_N, Dl * d, n * Dr, Dr, 1.0, A, (int64_t)Dl * d, 0, R, Dr, 0, 0.0, Y.z(), (int64_t)Dl * d, 0, 1);
  MixPlan pl;
  pl.Db = Dl; pl.R = n; pl.P = d; pl.Q = m; pl.S = d; pl.C = Dr;
  pl.in_r = (int64_t)Dl * d; pl.in_s = Dl; pl.in_c = (int64_t)Dl * d * n;
  pl.out_p = (int64_t)Dl * m; pl.out_q = Dl; pl.out_c = (int64_t)Dl * m * d;
  pl.M = W.Wdev.z() + (int64_t)W.m * W.d * W.n * W.d;
  for (auto& b : W.nz) pl.nz.push_back({b.second, b.first});
  std::vector<bool> hit(m, false);
  for (auto& b : W.nz) hit[b.first] = true;
  bool any_missing = false;
  for (int q = 0; q < m; ++q) any_missing |= !hit[q];
  if (any_missing) zfill(ctx, (int64_t)Dl * m * d * Dr, 0.0, Z.z());
  level_mix(ctx, pl, Y.z(), Z.z());
  zgemm(ctx, OP_N, OP_C, Dl * m, Dl, d * Dr, 1.0, Z.z(), (int64_t)Dl * m, 0, A, Dl, 0, 0.0, out, (int64_t)Dl * m, 0, 1);
}

}  // namespace imps
