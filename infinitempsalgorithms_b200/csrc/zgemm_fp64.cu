// FP64 complex GEMM engine (the plain method).  Column-major, op(A) in
// {N, T, C}, op(B) in {N, T, C}, strided batches.
//
// Tiling: 64 x 64 complex output tile per CTA of 256 threads, 4 x 4 complex
// accumulators per thread (strided by 16 so shared-memory reads of a warp hit
// consecutive addresses), K tile of 8 staged through shared memory with a
// register prefetch of the next tile.  Each complex MAC is 4 DFMA.
#include "gemm_modular.h"
#include "imps_internal.h"
#include "split_gemm.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace imps {
namespace {

constexpr int BM = 64, BN = 64, BK = 8, NT = 256;

__device__ __forceinline__ double2 conj2(double2 v) { return make_double2(v.x, -v.y); }

template <int OPA, int OPB, bool BETA>
__global__ void __launch_bounds__(NT, 2)
    k_zgemm(int M, int N, int K, double2 alpha, const double2* __restrict__ A, int64_t lda, int64_t sA,
            const double2* __restrict__ B, int64_t ldb, int64_t sB, double2 beta, double2* __restrict__ C,
            int64_t ldc, int64_t sC) {
  grid_enter();
  __shared__ double2 As[2][BK][BM + 1];
  __shared__ double2 Bs[2][BK][BN + 1];
  const int bz = blockIdx.z;
  A += sA * bz;
  B += sB * bz;
  C += sC * bz;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;

  // global-load coordinates: 2 A elements and 2 B elements per thread per K tile
  int am[2], ak[2], bk[2], bn[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (OPA == OP_N) { am[r] = tid & 63; ak[r] = (tid >> 6) + 4 * r; }
    else { ak[r] = tid & 7; am[r] = (tid >> 3) + 32 * r; }
    if (OPB == OP_N) { bk[r] = tid & 7; bn[r] = (tid >> 3) + 32 * r; }
    else { bn[r] = tid & 63; bk[r] = (tid >> 6) + 4 * r; }
  }
  double2 ra[2], rb[2];
  auto load_tile = [&](int k0) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int gm = m0 + am[r], gk = k0 + ak[r];
      double2 v = make_double2(0.0, 0.0);
      if (gm < M && gk < K) {
        v = (OPA == OP_N) ? A[gm + lda * gk] : A[gk + lda * gm];
        if (OPA == OP_C) v = conj2(v);
      }
      ra[r] = v;
      int gn = n0 + bn[r], gk2 = k0 + bk[r];
      double2 u = make_double2(0.0, 0.0);
      if (gn < N && gk2 < K) {
        u = (OPB == OP_N) ? B[gk2 + ldb * gn] : B[gn + ldb * gk2];
        if (OPB == OP_C) u = conj2(u);
      }
      rb[r] = u;
    }
  };
  auto store_tile = [&](int buf) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      As[buf][ak[r]][am[r]] = ra[r];
      Bs[buf][bk[r]][bn[r]] = rb[r];
    }
  };

  double2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_double2(0.0, 0.0);

  const int ktiles = (K + BK - 1) / BK;
  load_tile(0);
  store_tile(0);
  __syncthreads();
  for (int kt = 0; kt < ktiles; ++kt) {
    const int buf = kt & 1;
    if (kt + 1 < ktiles) load_tile((kt + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      double2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[buf][kk][tx + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[buf][kk][ty + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j].x = fma(a[i].x, b[j].x, acc[i][j].x);
          acc[i][j].x = fma(-a[i].y, b[j].y, acc[i][j].x);
          acc[i][j].y = fma(a[i].x, b[j].y, acc[i][j].y);
          acc[i][j].y = fma(a[i].y, b[j].x, acc[i][j].y);
        }
    }
    if (kt + 1 < ktiles) {
      store_tile(buf ^ 1);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + tx + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + ty + 16 * j;
      if (gn >= N) continue;
      double2 v = acc[i][j];
      double2 o = make_double2(alpha.x * v.x - alpha.y * v.y, alpha.x * v.y + alpha.y * v.x);
      if (BETA) {
        double2 c = C[gm + ldc * gn];
        o.x += beta.x * c.x - beta.y * c.y;
        o.y += beta.x * c.y + beta.y * c.x;
      }
      C[gm + ldc * gn] = o;
    }
  }
}

// ---------------------------------------------------------------------------
// FP64 tensor-core variant: mma.sync m8n8k4 f64 (DMMA).  64 x 64 complex output tile per
// CTA of 8 warps (2 x 4 warps of 32 x 16), two CTAs per SM, or for small grids 32 x 32 per
// CTA of 4 warps (2 x 2 of 16 x 16); a K stage of 16 complex, a 3-stage cp.async ring
// (zero-filled at the matrix edges).  A complex product is four real
// DMMAs per 8 x 8 block: re += ar br - ai bi, im += ar bi + ai br; the conjugate of an
// operand only flips the sign of its imaginary fragment.
// Shared tiles are k-major rows of double2.  A fragment read takes 4 k x 2 m (or n)
// consecutive elements per 8-lane phase, so a row stride of 2 mod 8 elements is free of
// bank conflicts; the loads of a transposed operand walk 4 k x 2 m per phase for the same
// reason.  Bound by the FP64 tensor pipe: four warps a scheduler (two CTAs) hide the
// fragment reads and the stage barriers behind the MMAs.  Measured (B200, N x N):
// 6144 x 4096 x 1024 6.50 ms and 4096 x 1024 x 6144 6.57 ms, 31.5 TFLOP/s (6.88 and 7.81 ms
// with 128 x 64 tiles of 32 x 32 warps and 2-way conflicts in the fragment reads); with the
// K stages shared (split_k) 502 x 251 x 1255 55 us (was 239) and 256 x 256 x 1024 (C x N)
// 32 us (was 210).
// ---------------------------------------------------------------------------
namespace dm {
constexpr int BK = 16, STAGES = 3;
template <int T>
struct Tile {
  static constexpr int NT = 4 * T;                // threads: 2 x T / 16 warps of T / 2 x 16
  static constexpr int MI = T / 16, NJ = 2;       // 8 x 8 blocks of a warp
  static constexpr int LD = T + 2;
  static constexpr int TILE = BK * LD;            // elements of one operand's stage
  static constexpr int SMEM = STAGES * 2 * TILE * 16;
};
}  // namespace dm

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// SPLITK: nsplit CTAs (along x) share one output tile, each summing its part of the K
// stages; CTA r writes its plain partial sums to part[r] (M x N each), which
// k_sum_split adds in order (so the result does not depend on timing).
template <int OPA, int OPB, bool BETA, bool SPLITK, int T>
__global__ void __launch_bounds__(4 * T, T == 64 ? 2 : 4)
    k_zgemm_dmma(int M, int N, int K, double2 alpha, const double2* __restrict__ A, int64_t lda, int64_t sA,
                 const double2* __restrict__ B, int64_t ldb, int64_t sB, double2 beta, double2* __restrict__ C,
                 int64_t ldc, int64_t sC, int nsplit, double2* __restrict__ part) {
  grid_enter();
  using D = dm::Tile<T>;
  extern __shared__ __align__(16) double2 smem_dm[];   // [STAGES][A tile, B tile][BK][LD]
  const int bz = blockIdx.z;
  A += sA * bz;
  B += sB * bz;
  C += sC * bz;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1;  // warp tile origin (T / 2 wm, 16 wn)
  const int rank = SPLITK ? (int)(blockIdx.x % nsplit) : 0;
  const int m0 = (int)(SPLITK ? blockIdx.x / nsplit : blockIdx.x) * T, n0 = blockIdx.y * T;
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dm));

  // Load coordinates.  An operand whose line index (m or n) is contiguous: line tid % T,
  // k = tid / T + 4 r; one contiguous in k: k from bits 0, 1, 3, 4 of tid, line from bit 2
  // and the warp, + T / 4 r.
  constexpr bool AK = OPA != OP_N, BKc = OPB == OP_N;   // contiguous along k
  const int kc = (tid & 3) | ((tid >> 1) & 12), lc = ((tid >> 2) & 1) | (warp << 1);
  const int ll = tid % T, kl = tid / T;
  const int am = AK ? lc : ll, ak = AK ? kc : kl;
  const int bn = BKc ? lc : ll, bk = BKc ? kc : kl;
  const int64_t a_r = AK ? T / 4 * lda : 4 * lda, b_r = BKc ? T / 4 * ldb : 4 * ldb;   // step of r
  const int64_t a_s = AK ? dm::BK : dm::BK * lda, b_s = BKc ? dm::BK : dm::BK * ldb;   // step of a stage
  // this CTA's K stages
  const int kall = (K + dm::BK - 1) / dm::BK;
  const int kt0 = SPLITK ? (int)((int64_t)kall * rank / nsplit) : 0;
  const int ktiles = (SPLITK ? (int)((int64_t)kall * (rank + 1) / nsplit) : kall) - kt0;
  const double2* pa = A + (AK ? ak + lda * (int64_t)(m0 + am) : (m0 + am) + lda * (int64_t)ak) + a_s * kt0;
  const double2* pb = B + (BKc ? bk + ldb * (int64_t)(n0 + bn) : (n0 + bn) + ldb * (int64_t)bk) + b_s * kt0;
  const uint32_t da = sbase + 16u * (ak * D::LD + am), db = sbase + 16u * (D::TILE + bk * D::LD + bn);
  constexpr uint32_t DA_R = 16u * (AK ? T / 4 : 4 * D::LD), DB_R = 16u * (BKc ? T / 4 : 4 * D::LD);

  auto issue = [&](int stage, int kt) {
    const int k0 = (kt0 + kt) * dm::BK;
    const double2* qa = pa + a_s * kt;
    const double2* qb = pb + b_s * kt;
    const uint32_t so = 16u * (uint32_t)(stage * 2 * D::TILE);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const bool ok = AK ? (m0 + am + T / 4 * r < M && k0 + ak < K) : (m0 + am < M && k0 + ak + 4 * r < K);
      cp_async16(da + so + DA_R * r, ok ? qa + a_r * r : A, ok ? 16 : 0);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const bool ok = BKc ? (n0 + bn + T / 4 * r < N && k0 + bk < K) : (n0 + bn < N && k0 + bk + 4 * r < K);
      cp_async16(db + so + DB_R * r, ok ? qb + b_r * r : B, ok ? 16 : 0);
    }
  };

  double cre[D::MI][2][2], cim[D::MI][2][2];
#pragma unroll
  for (int i = 0; i < D::MI; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) cre[i][j][0] = cre[i][j][1] = cim[i][j][0] = cim[i][j][1] = 0.0;

#pragma unroll
  for (int st = 0; st < dm::STAGES - 1; ++st) {
    if (st < ktiles) issue(st, st);
    cp_async_commit();
  }
  const int fr = lane >> 2, fk = lane & 3;  // fragment row/col (A: row m, col k; B: col n, row k)
  const int fa = fk * D::LD + T / 2 * wm + fr, fb = D::TILE + fk * D::LD + 16 * wn + fr;
  int stage = 0, nstage = dm::STAGES - 1;
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_async_wait<dm::STAGES - 2>();
    __syncthreads();
    if (kt + dm::STAGES - 1 < ktiles) issue(nstage, kt + dm::STAGES - 1);
    cp_async_commit();
    const double2* ss = smem_dm + stage * 2 * D::TILE;
#pragma unroll
    for (int kb = 0; kb < dm::BK; kb += 4) {
      double ar[D::MI], ai[D::MI], br[2], bi[2];
#pragma unroll
      for (int i = 0; i < D::MI; ++i) {
        const double2 v = ss[kb * D::LD + fa + 8 * i];
        ar[i] = v.x;
        ai[i] = (OPA == OP_C) ? -v.y : v.y;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const double2 v = ss[kb * D::LD + fb + 8 * j];
        br[j] = v.x;
        bi[j] = (OPB == OP_C) ? -v.y : v.y;
      }
      // the two updates of one accumulator are 4 MI MMAs apart
#pragma unroll
      for (int i = 0; i < D::MI; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dmma(cre[i][j][0], cre[i][j][1], ar[i], br[j]);
          dmma(cim[i][j][0], cim[i][j][1], ar[i], bi[j]);
        }
#pragma unroll
      for (int i = 0; i < D::MI; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dmma(cre[i][j][0], cre[i][j][1], -ai[i], bi[j]);
          dmma(cim[i][j][0], cim[i][j][1], ai[i], br[j]);
        }
    }
    stage = stage + 1 == dm::STAGES ? 0 : stage + 1;
    nstage = nstage + 1 == dm::STAGES ? 0 : nstage + 1;
  }
  cp_async_wait<0>();
  // D fragment: row = lane >> 2, cols 2 (lane & 3) + {0, 1} of each 8 x 8 block
  double2* P = SPLITK ? part + ((int64_t)bz * nsplit + rank) * M * (int64_t)N : nullptr;
#pragma unroll
  for (int i = 0; i < D::MI; ++i) {
    const int gm = m0 + T / 2 * wm + 8 * i + fr;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int gn = n0 + 16 * wn + 8 * j + 2 * fk + e;
        if (gn >= N) continue;
        const double vr = cre[i][j][e], vi = cim[i][j][e];
        if (SPLITK) {
          P[gm + M * (int64_t)gn] = make_double2(vr, vi);
          continue;
        }
        double2 o = make_double2(alpha.x * vr - alpha.y * vi, alpha.x * vi + alpha.y * vr);
        double2* p = C + gm + ldc * (int64_t)gn;
        if (BETA) {
          const double2 c = *p;
          o.x += beta.x * c.x - beta.y * c.y;
          o.y += beta.x * c.y + beta.y * c.x;
        }
        *p = o;
      }
  }
}

// C = alpha sum_r part[r] + beta C, the nsplit partial products of each batch entry in order
template <bool BETA>
__global__ void __launch_bounds__(256) k_sum_split(int M, int N, int nsplit, const double2* __restrict__ part,
                                                   double2 alpha, double2 beta, double2* __restrict__ C, int64_t ldc,
                                                   int64_t sC) {
  grid_enter();
  const int64_t len = (int64_t)M * N;
  part += (int64_t)blockIdx.y * nsplit * len;
  C += sC * blockIdx.y;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x) {
    double vr = 0.0, vi = 0.0;
    int q = 0;
    for (; q + 4 <= nsplit; q += 4) {  // four loads in flight
      double2 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(&part[i + len * (q + u)]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        vr += v[u].x;
        vi += v[u].y;
      }
    }
    for (; q < nsplit; ++q) {
      const double2 v = __ldg(&part[i + len * q]);
      vr += v.x;
      vi += v.y;
    }
    double2 o = make_double2(alpha.x * vr - alpha.y * vi, alpha.x * vi + alpha.y * vr);
    double2* p = C + i % M + ldc * (i / M);
    if (BETA) {
      const double2 c = *p;
      o.x += beta.x * c.x - beta.y * c.y;
      o.y += beta.x * c.y + beta.y * c.x;
    }
    *p = o;
  }
}

template <int OPA, int OPB, bool BETA, bool SPLITK, int T>
void launch_dmma(Context* ctx, int nsplit, double2* part, int M, int N, int K, double2 alpha, const dcplx* A,
                 int64_t lda, int64_t sA, const dcplx* B, int64_t ldb, int64_t sB, double2 beta, dcplx* C, int64_t ldc,
                 int64_t sC, int batch) {
  using D = dm::Tile<T>;
  auto kern = k_zgemm_dmma<OPA, OPB, BETA, SPLITK, T>;
  static DeviceOnce attr;  // the dynamic shared-memory opt-in
  attr.run(ctx->device, [&] {
    IMPS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, D::SMEM));
  });
  const dim3 grid((M + T - 1) / T * nsplit, (N + T - 1) / T, batch);
  launch_kernel(ctx, kern, grid, D::NT, D::SMEM, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, nsplit, part);
}

// Tile size and CTAs that share a tile's K stages (1: none): the smallest time of a model of
// the grid.  Measured on a B200: a K stage of a 64 x 64 tile takes 3.3 us alone on its SM and
// 2.46 us of the SM when others run beside it, one of a 32 x 32 tile 0.85 and 0.68 us; partial
// products cost one more launch (2.2 us and 0.1 us each) and their bytes at 3 TB/s.  Small
// tiles give 64 x 64 x 64 5.2 us (64 x 64 tiles: 13.2, shared 7.7), 448 x 448 x 64 7.1 us (12.4)
// and, where the sums are ordered and may not be shared, 384 x 384 x 1536 103 us (300).
struct DmmaPlan {
  int tile, nsplit;
  double us;
};
DmmaPlan dmma_plan(const Context* ctx, int M, int N, int K, int batch, bool share) {
  const int kall = (K + dm::BK - 1) / dm::BK;
  DmmaPlan best{64, 1, 1e300};
  for (int T : {64, 32}) {
    const int64_t tiles = (int64_t)((M + T - 1) / T) * ((N + T - 1) / T) * batch;
    if (T == 32 && (N + 31) / 32 > 65535) continue;   // grid limit
    const double alone = T == 64 ? 3.3 : 0.85, shared = T == 64 ? 2.46 : 0.68;
    for (int s = 1; s <= kall && s <= (share ? 64 : 1); ++s) {
      const double per_sm = (double)((tiles * s + ctx->num_sms - 1) / ctx->num_sms);
      double t = ((kall + s - 1) / s) * std::max(alone, shared * per_sm);
      if (s > 1) t += 2.2 + 0.1 * s + (double)tiles * s * (T * T * 16 / 3e6);
      if (t < best.us) best = {T, s, t};
    }
  }
  return best;
}

template <int OPA, int OPB>
void launch(Context* ctx, int M, int N, int K, double2 alpha, const dcplx* A, int64_t lda, int64_t sA,
            const dcplx* B, int64_t ldb, int64_t sB, double2 beta, dcplx* C, int64_t ldc, int64_t sC, int batch,
            bool use_beta) {
  if (ctx->fp64_engine == 1) {
    dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN, batch);
    if (use_beta)
      launch_kernel(ctx, k_zgemm<OPA, OPB, true>, grid, NT, 0, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC);
    else
      launch_kernel(ctx, k_zgemm<OPA, OPB, false>, grid, NT, 0, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc,
                                                              sC);
    return;
  }
  auto go = [&](auto beta_tag) {
    constexpr bool BETA = decltype(beta_tag)::value;
    // small tiles, and the K stages of a tile shared by several CTAs, where 64 x 64 tiles alone
    // would leave SMs idle (the long-K products of the pushes and of the QR, every product of
    // a small state)
    DmmaPlan plan = dmma_plan(ctx, M, N, K, batch, !ctx->ordered_sums());
    const int s = plan.nsplit;
    const int64_t len = (int64_t)M * N;
    double2* part = nullptr;
    if (s > 1) part = static_cast<double2*>(ctx->optional_buf("gemm_part", (size_t)len * s * batch * sizeof(double2)));
    if (s > 1 && !part) plan = dmma_plan(ctx, M, N, K, batch, false);
    auto run = [&](auto split_tag, auto tile_tag) {
      launch_dmma<OPA, OPB, BETA, decltype(split_tag)::value, decltype(tile_tag)::value>(
          ctx, part ? s : 1, part, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
    };
    using Big = std::integral_constant<int, 64>;
    using Small = std::integral_constant<int, 32>;
    if (!part) {
      if (plan.tile == 64) run(std::false_type{}, Big{});
      else run(std::false_type{}, Small{});
      return;
    }
    if (plan.tile == 64) run(std::true_type{}, Big{});
    else run(std::true_type{}, Small{});
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((len + 255) / 256, ctx->num_sms * 8 / batch));
    launch_kernel(ctx, k_sum_split<BETA>, dim3(g, batch), 256, 0, M, N, s, part, alpha, beta, C, ldc, sC);
    ctx->n_kernels++;
  };
  if (use_beta) go(std::true_type{});
  else go(std::false_type{});
}

}  // namespace

void zgemm_fp64(Context* ctx, Op opA, Op opB, int M, int N, int K, cplx alpha, const dcplx* A, int64_t lda,
                int64_t strideA, const dcplx* B, int64_t ldb, int64_t strideB, cplx beta, dcplx* C, int64_t ldc,
                int64_t strideC, int batch) {
  if (M <= 0 || N <= 0 || batch <= 0) return;
  IMPS_REQUIRE(batch <= 65535, IMPS_INVALID_ARG, "zgemm: batch too large");
  IMPS_REQUIRE((N + 31) / 32 <= 65535 * 2, IMPS_INVALID_ARG, "zgemm: N too large");
  if (K <= 0) {
    // C = beta C
    for (int b = 0; b < batch; ++b) {
      for (int n = 0; n < N; ++n) {
        if (beta == cplx(0.0, 0.0)) zfill(ctx, M, cplx(0.0, 0.0), C + strideC * b + ldc * n);
        else zscal(ctx, M, beta, C + strideC * b + ldc * n);
      }
    }
    return;
  }
  // products large enough: residue arithmetic on the int8 tensor cores
  if (batch == 1 && ctx->fp64_engine == 0 && !ctx->ordered_sums() &&
      zgemm_modular(ctx, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, dmma_plan(ctx, M, N, K, 1, true).us))
    return;
  double2 a = make_double2(alpha.real(), alpha.imag()), bt = make_double2(beta.real(), beta.imag());
  bool use_beta = beta != cplx(0.0, 0.0);
  ScopedTimer t(ctx, "zgemm_fp64", 8.0 * M * (double)N * K * batch);
  ctx->n_gemm++;
  ctx->n_kernels++;
#define IMPS_GEMM_CASE(OA, OB)                                                                              \
  if (opA == OA && opB == OB) {                                                                             \
    launch<OA, OB>(ctx, M, N, K, a, A, lda, strideA, B, ldb, strideB, bt, C, ldc, strideC, batch, use_beta); \
  }
  IMPS_GEMM_CASE(OP_N, OP_N)
  IMPS_GEMM_CASE(OP_N, OP_T)
  IMPS_GEMM_CASE(OP_N, OP_C)
  IMPS_GEMM_CASE(OP_T, OP_N)
  IMPS_GEMM_CASE(OP_C, OP_N)
  IMPS_GEMM_CASE(OP_T, OP_T)
  IMPS_GEMM_CASE(OP_C, OP_C)
  IMPS_GEMM_CASE(OP_T, OP_C)
  IMPS_GEMM_CASE(OP_C, OP_T)
#undef IMPS_GEMM_CASE
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) throw Error(IMPS_CUDA_ERROR, std::string("zgemm launch: ") + cudaGetErrorString(e));
}

int slices_for_tol(double tol) {
  // the truncation error of s slices is below 2^-7s of the row/column scales; keep
  // a 2^4 margin for the sum over K and the spread inside a row
  if (!(tol > 0)) return 8;
  int s = (int)std::ceil((-std::log2(tol) + 4.0) / 7.0);
  return std::min(8, std::max(2, s));
}

int active_slices(const Context* ctx) {
  if (ctx->precision != PREC_SPLIT_I8 || ctx->force_fp64 > 0) return 0;
  if (!ctx->adaptive_slices) return ctx->nslices;  // a fixed count is used as given
  // adaptive: beyond max_adaptive_slices (6 unless a scope raises it) the FP64 engine
  const int s = slices_for_tol(ctx->split_tol);
  return s > ctx->max_adaptive_slices ? 0 : s;
}

double split_floor(const Context* ctx) {
  const int s = active_slices(ctx);
  return s == 0 ? 0.0 : 16.0 * std::ldexp(1.0, -7 * s);
}

static std::shared_ptr<SplitOperand> get_split(Context* ctx, int side, Op op, int rows, int K, const dcplx* X,
                                               int64_t ld, int s) {
  const bool constant = ctx->const_ptrs.count(X) > 0;
  SplitKey key{X, side, (int)op, rows, K, ld, s};
  if (constant) {
    auto it = ctx->split_cache.find(key);
    if (it != ctx->split_cache.end()) {
      ctx->split_cache_hits++;
      return it->second;
    }
  }
  std::shared_ptr<SplitOperand> S;
  if (constant) {
    // reuse a pooled operand: the smallest whose planes already fit, else the largest
    auto rup = [](int64_t x) { return (x + 127) / 128 * 128; };
    const size_t need = (size_t)(side == 0 ? rup(2 * (int64_t)rows) : rup(rows)) * rup(2 * (int64_t)K) * s;
    int best = -1;
    for (int i = 0; i < (int)ctx->split_pool.size(); ++i) {
      const size_t have = ctx->split_pool[i]->data.bytes;
      if (best < 0) { best = i; continue; }
      const size_t cur = ctx->split_pool[best]->data.bytes;
      const bool fits = have >= need, cur_fits = cur >= need;
      if ((fits && (!cur_fits || have < cur)) || (!fits && !cur_fits && have > cur)) best = i;
    }
    if (best >= 0) {
      S = ctx->split_pool[best];
      ctx->split_pool.erase(ctx->split_pool.begin() + best);
    } else {
      S = std::make_shared<SplitOperand>();
    }
  } else {
    // transient operand: reuse one scratch object per side of this context
    if (!ctx->split_scratch[side]) ctx->split_scratch[side] = std::make_shared<SplitOperand>();
    S = ctx->split_scratch[side];
  }
  const bool have_max = side == 0 && !constant && ctx->max_ready == X;   // (in the scratch operand)
  ctx->max_ready = nullptr;
  if (side == 0) split_operand_a(ctx, *S, op, rows, K, X, ld, s, have_max);
  else split_operand_b(ctx, *S, op, K, rows, X, ld, s);
  if (constant) ctx->split_cache[key] = S;
  return S;
}

bool zgemm_splits(const Context* ctx, Op opA, Op opB, int M, int N, int K) {
  return active_slices(ctx) > 0 && opA != OP_T && opB != OP_T && M >= 64 && N >= 64 && K >= 32 &&
         (double)M * N * K >= 33554432.0;
}

unsigned long long* split_collect_max(Context* ctx, const dcplx* A, int M, int N, int K) {
  if (!zgemm_splits(ctx, OP_N, OP_N, M, N, K) || ctx->const_ptrs.count(A) > 0) return nullptr;
  if (!ctx->split_scratch[0]) ctx->split_scratch[0] = std::make_shared<SplitOperand>();
  ctx->max_ready = A;
  return split_line_max(ctx, *ctx->split_scratch[0], M);
}

void zgemm(Context* ctx, Op opA, Op opB, int M, int N, int K, cplx alpha, const dcplx* A, int64_t lda,
           int64_t strideA, const dcplx* B, int64_t ldb, int64_t strideB, cplx beta, dcplx* C, int64_t ldc,
           int64_t strideC, int batch, bool allow_split) {
  ctx->gemm_flops += 8.0 * (double)M * (double)N * (double)K * (double)batch;
  const int s = active_slices(ctx);
  const bool split = allow_split && alpha.imag() == 0.0 && (beta == cplx(0.0, 0.0) || beta == cplx(1.0, 0.0)) &&
                     zgemm_splits(ctx, opA, opB, M, N, K);
  if (!split) {
    zgemm_fp64(ctx, opA, opB, M, N, K, alpha, A, lda, strideA, B, ldb, strideB, beta, C, ldc, strideC, batch);
    return;
  }
  for (int b = 0; b < batch; ++b) {
    const dcplx* Ab = A + strideA * b;
    const dcplx* Bb = B + strideB * b;
    auto SA = get_split(ctx, 0, opA, M, K, Ab, lda, s);
    auto SB = get_split(ctx, 1, opB, N, K, Bb, ldb, s);
    ctx->split_calls++;
    split_gemm(ctx, *SA, *SB, s, alpha.real(), beta == cplx(1.0, 0.0), C + strideC * b, ldc);
  }
}

}  // namespace imps
