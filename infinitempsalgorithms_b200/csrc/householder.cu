// QRpos / LQpos on the device by blocked Householder QR, written here (no
// vendor solver library): FiniteMPSAlgorithms' `leftorth(.; alg = QRpos())` and
// `rightorth(.; alg = LQpos())` as used in src/states/ortho.jl:150, 188, 214-225.
//
// M (m x n) = Q R with Q (m x k) isometric, R (k x n) upper trapezoidal with a real
// non-negative diagonal, k = min(m, n).  The reflectors follow LAPACK's zgeqr2
// convention (H = I - tau v v^H with v[0] = 1 and beta = -sign(Re alpha) ||x|| real,
// the trailing columns updated with H^H), so R and Q agree with a LAPACK QR up to
// the final phase fix Q[:, i] *= ph_i, R[i, :] *= conj(ph_i), ph_i = R_ii / |R_ii|.
//
// Two-level blocked right-looking algorithm:
//  * k_qr_panel: one CTA or thread-block cluster (up to QR_CL CTAs, by the rows) factors
//    the panel A[p:m, p:p+b] (b <= 16), the panel rows held in registers.  Per column a
//    single reduction (distributed shared memory after one cluster barrier) gives ||x||^2, the inner products with the trailing panel columns and those with
//    the earlier reflectors needed for the compact-WY factor T (LAPACK zlarft,
//    T[0:c, c] = -tau_c T[0:c, 0:c] V^H v_c).  The kernel writes R (upper part of A),
//    V (explicit, unit diagonal, zeros above), tau and T.
//  * inner panels update only the rest of their outer block of QR_NBO columns; the
//    outer block's T is merged from the panels' factors (k_merge_t, with G = V^H V),
//    and the trailing matrix A2 <- (I - V T V^H)^H A2 = A2 - (V T^H) (A2^H V)^H is updated
//    once per outer block by FP64 GEMMs on the DMMA engine (the long-K product A2^H V
//    split into row chunks, one batched GEMM, summed in a fixed order).
//  * Q = H_1 ... H_k [I; 0] by the outer block reflectors applied backwards:
//    Q[P:m, P:k] <- (I - V T V^H) Q[P:m, P:k].
// LQpos is QRpos of the conjugate transpose.
#include <algorithm>

#include "imps_internal.h"

namespace imps {

void scale_q_r(Context* ctx, int m, int n, int k, dcplx* Q, int64_t ldq, dcplx* R, int64_t ldr, const dcplx* ph);

namespace {

constexpr int QR_CL = 8;     // most CTAs per cluster (portable cluster size)
constexpr int QR_NT = 512;   // threads per CTA
constexpr int QR_G = QR_CL * QR_NT;
constexpr int QR_NBMAX = 16;
constexpr int QR_NBO = 64;   // outer block: columns per compact-WY trailing update
constexpr int QR_MAXCHUNK = 32;  // most row chunks of a split-K X^H V product

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// all threads of every CTA of the cluster; release / acquire order the shared
// (and global) writes before the barrier with the reads after it
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
// store v into the same shared variable of CTA `rank` of the cluster (made visible to
// that CTA by the next cluster barrier's release / acquire).  Defined only once that CTA
// runs: a cluster barrier has to lie between the kernel's start and the first one.
__device__ __forceinline__ void st_peer(double* local, uint32_t rank, double v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(local)), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ dcplx cmul(dcplx a, dcplx b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ dcplx cmulc(dcplx a, dcplx b) {  // conj(a) * b
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.x, b.y, -a.y * b.x));
}

// Sum of val[s] over the 32 lanes of a warp for NV slots by a reduce-scatter: log2(NV)
// exchange rounds of halving width (NV - 1 shuffles in all), then plain rounds over the
// lanes that share a slot.  Returns the warp total of slot lane / (32 / NV).
template <int NV>
__device__ __forceinline__ double warp_reduce_scatter(double (&val)[NV], int lane) {
  int half = NV;
#pragma unroll
  for (int o = 16; o >= 32 / NV; o >>= 1) {
    half >>= 1;
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int v = 0; v < NV / 2; ++v) {
      if (v < half) {
        const double send = up ? val[v] : val[v + half];
        const double keep = up ? val[v + half] : val[v];
        val[v] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
  double r = val[0];
#pragma unroll
  for (int o = 32 / NV / 2; o >= 1; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

// Householder factorization of the panel A[0:R, 0:b] (lda), b <= NB, by a cluster of CL
// CTAs of NT threads.  Row il of the panel belongs to cluster thread g = rank * NT + tid with
// il = g + k CL NT, k < RPT, and lives in that thread's registers (NB RPT = 16 complex).
// The columns rotate through them: at column c register column q holds panel column
// (c + q) mod NB, so position 0 is the current one, the next ones the trailing columns and
// the last c the finished reflectors, and the column loop needs no unrolling.
// One reduction per column: ||x_c below||^2, d_j = x_c^H x_j (j > c, trailing panel columns)
// and e_l = V_l^H x_c (l < c, for T), all over the rows below c, together with row c of the
// panel (held by thread c of CTA 0).  With v = [1; scale x_c below]:
//   v^H x_j = x_j[c] + conj(scale) d_j,   V_l^H v = conj(V_l[c]) + scale e_l.
// Warp 0 alone takes the reflector's square root and divisions and the NB - 1 inner
// products; the last warp extends T while the others update their rows.
// The sums run over the 16 warps of every 512 rows in order, then over these groups, however
// the rows are spread (CTAs of fewer threads push their warps' sums themselves), so a
// panel's result does not depend on CL and NT.
// Bound by latency: a column costs one CTA of 512 rows about 2.9 us (its instructions about
// 1.9 us, the rest the reflector's divisions and the barriers), a cluster barrier 0.65 us
// more; so up to 256 rows take one CTA, more rows eight CTAs of as few threads as hold them.
// 16 columns of 512 rows: 66 us with eight CTAs of 512 threads and the rows in shared memory,
// 48 us on one CTA with the rows in registers, 38 us on eight CTAs of 64 threads; 2048 rows
// 69 us, 58 us (four CTAs of 512) and 45 us (eight of 256).
// Outputs: A (R above/on the diagonal, v below), V (R x b, ldv: v with unit diagonal and
// zeros above; the zabove rows before row 0 are zeroed too), tau[0:b], T (b x b, ldt).
template <int NB, int RPT, int CL, int NT>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(NT, 1)
    k_qr_panel(int R, int b, int zabove, dcplx* __restrict__ A, int64_t lda, dcplx* __restrict__ V, int64_t ldv,
               dcplx* __restrict__ tau, dcplx* __restrict__ T, int ldt) {
  // every CTA of the cluster runs before the first store into a peer's shared memory (a CTA
  // without rows gets there at once); the wait comes behind the panel's loads
  if constexpr (CL > 1) cluster_arrive();
  grid_enter();
  constexpr int NV = 2 * NB;             // reduction slots: [0] ||x||^2, [2q - 1, 2q] position q
  constexpr int NW = NT / 32;
  constexpr bool WARPS = CL > 1 && NT < QR_NT;   // the warps' sums travel, not the CTAs'
  constexpr int NGRP = WARPS ? CL * NT / QR_NT : 1, GW = QR_NT / 32;   // groups of 512 rows, their warps
  static_assert(!WARPS || CL * NT % QR_NT == 0, "whole groups");
  constexpr int HV = NV > 16 ? 16 : NV;  // slots reduced at a time (registers)
  constexpr int SPL = 32 / HV;           // lanes per slot after the reduce-scatter
  constexpr int G = CL * NT;
  __shared__ double wsum[NW][NV];
  __shared__ double red[2][WARPS ? 1 : CL][NV];   // partials pushed by every CTA of the cluster
  __shared__ double redw[2][NGRP][WARPS ? GW : 1][NV];   // or by every warp
  __shared__ dcplx rowl[NB];             // row c of the panel, written by its thread
  __shared__ double rowc[2][2 * NB];     // the same, pushed by CTA 0
  __shared__ dcplx sc[3];                // conj(tau), scale, beta
  __shared__ dcplx wv[NB], zs[NB];
  __shared__ dcplx Tsh[NB][NB + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = CL > 1 ? cluster_rank() : 0u;
  const int g = (int)rank * NT + tid;

  dcplx x[RPT][NB];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int il = g + k * G;
#pragma unroll
    for (int j = 0; j < NB; ++j) x[k][j] = (il < R && j < b) ? A[il + lda * (int64_t)j] : make_double2(0.0, 0.0);
  }
  if (rank == 0)
    for (int e = tid; e < NB * (NB + 1); e += NT) Tsh[e / (NB + 1)][e % (NB + 1)] = make_double2(0.0, 0.0);
  if constexpr (CL > 1) cluster_wait();

#pragma unroll 1
  for (int c = 0; c < b; ++c) {
    const int par = c & 1;
    const int nt = NB - c;   // positions below nt are trailing columns, the others reflectors
#pragma unroll
    for (int h = 0; h < NV / HV; ++h) {
      double val[HV];
#pragma unroll
      for (int s = 0; s < HV; ++s) val[s] = 0.0;
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const int il = g + k * G;
        if (il > c && il < R) {
          const dcplx xc = x[k][0];
          if (h == 0) val[0] = k == 0 ? fma(xc.x, xc.x, xc.y * xc.y) : fma(xc.x, xc.x, fma(xc.y, xc.y, val[0]));
#pragma unroll
          for (int s = 0; s < HV; ++s) {
            const int slot = h * HV + s, q = (slot + 1) >> 1;
            if (slot == 0) continue;
            const dcplx y = x[k][q];
            double p;
            if (slot & 1) p = fma(xc.x, y.x, xc.y * y.y);
            else p = q < nt ? fma(xc.x, y.y, -xc.y * y.x) : fma(y.x, xc.y, -y.y * xc.x);
            val[s] = k == 0 ? p : val[s] + p;
          }
        }
      }
      const double wvl = warp_reduce_scatter<HV>(val, lane);
      if constexpr (WARPS) {
        // the lanes of a slot share the peers
        const int wg = (int)rank * NW + warp;
#pragma unroll
        for (int q = 0; q < CL; q += SPL)
          st_peer(&redw[par][wg / GW][wg % GW][h * HV + lane / SPL], (uint32_t)(q + lane % SPL), wvl);
      } else if (lane % SPL == 0) {
        wsum[warp][h * HV + lane / SPL] = wvl;
      }
    }
    if (rank == 0 && tid == c) {
#pragma unroll
      for (int q = 0; q < NB; ++q) rowl[q] = x[0][q];
    }
    if constexpr (WARPS) {
      if (rank == 0 && warp == 0) {   // row c to every CTA, a component a lane
        __syncwarp();
        if (lane < 2 * NB) {
          const dcplx y = rowl[lane >> 1];
#pragma unroll
          for (uint32_t q = 0; q < CL; ++q) st_peer(&rowc[par][lane], q, (lane & 1) ? y.y : y.x);
        }
      }
      cluster_sync();
    } else {
      __syncthreads();
    }
    if constexpr (CL > 1 && !WARPS) {
      // push this CTA's partials (and, from CTA 0, row c) into every CTA; no remote loads
      if (tid < NV) {
        double t = 0.0;
        for (int q = 0; q < NW; ++q) t += wsum[q][tid];
#pragma unroll
        for (uint32_t q = 0; q < CL; ++q) st_peer(&red[par][rank][tid], q, t);
      } else if (rank == 0 && tid < NV + 2 * NB * CL) {
        const int e = tid - NV, slot = e % (2 * NB), dst = e / (2 * NB);
        const dcplx y = rowl[slot >> 1];
        st_peer(&rowc[par][slot], (uint32_t)dst, (slot & 1) ? y.y : y.x);
      }
      cluster_sync();
    }
    if (warp == 0) {
      double t = 0.0;
      if (lane < NV) {
        if constexpr (WARPS) {
          double tg[NGRP];
#pragma unroll
          for (int q = 0; q < NGRP; ++q) tg[q] = 0.0;
#pragma unroll
          for (int w = 0; w < GW; ++w)
#pragma unroll
            for (int q = 0; q < NGRP; ++q) tg[q] += redw[par][q][w][lane];
#pragma unroll
          for (int q = 0; q < NGRP; ++q) t += tg[q];
        } else if constexpr (CL > 1) {
#pragma unroll
          for (int q = 0; q < CL; ++q) t += red[par][q][lane];
        } else {
#pragma unroll
          for (int q = 0; q < NW; ++q) t += wsum[q][lane];
        }
      }
      // lane q serves position q
      const int q = lane < NB ? lane : 0;
      const double xsq = __shfl_sync(0xffffffffu, t, 0);
      const double dx = __shfl_sync(0xffffffffu, t, (2 * q - 1) & 31), dy = __shfl_sync(0xffffffffu, t, 2 * q);
      dcplx al, rq;
      if constexpr (CL > 1) {
        al = make_double2(rowc[par][0], rowc[par][1]);
        rq = make_double2(rowc[par][2 * q], rowc[par][2 * q + 1]);
      } else {
        al = rowl[0];
        rq = rowl[q];
      }
      // the reflector (LAPACK zlarfg); the four quotients of tau = (beta - alpha) / beta and
      // scale = 1 / (alpha - beta) in one division, a lane each
      dcplx tc, scale;
      double beta;
      if (xsq == 0.0 && al.y == 0.0) {
        tc = make_double2(0.0, 0.0);
        scale = make_double2(0.0, 0.0);
        beta = al.x;
      } else {
        beta = -copysign(sqrt(al.x * al.x + al.y * al.y + xsq), al.x);
        const double dr = al.x - beta, di = al.y, den = dr * dr + di * di;
        const int w = lane & 3;
        const double num = w == 0 ? beta - al.x : (w == 1 ? -al.y : (w == 2 ? dr : -di));
        const double quot = num / (w < 2 ? beta : den);
        tc = make_double2(__shfl_sync(0xffffffffu, quot, 0), __shfl_sync(0xffffffffu, quot, 1));
        scale = make_double2(__shfl_sync(0xffffffffu, quot, 2), __shfl_sync(0xffffffffu, quot, 3));
      }
      const dcplx dq = make_double2(dx, dy);
      if (lane >= 1 && lane < NB) {
        if (lane < nt) {
          const dcplx p = cmul(make_double2(scale.x, -scale.y), dq);
          wv[lane] = make_double2(rq.x + p.x, rq.y + p.y);
        } else {
          const dcplx se = cmul(scale, dq);
          zs[lane - nt] = make_double2(rq.x + se.x, -rq.y + se.y);
        }
      }
      if (lane == 0) {
        sc[0] = make_double2(tc.x, -tc.y);
        sc[1] = scale;
        sc[2] = make_double2(beta, 0.0);
        if (rank == 0) tau[c] = tc;
      }
    }
    __syncthreads();
    // v into column c, R diagonal, trailing panel columns x_j -= conj(tau) v (v^H x_j); every
    // column moves one position down, column c to the last
    {
      const dcplx ctc = sc[0], scale = sc[1];
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const int il = g + k * G;
        dcplx v = x[k][0], keep = x[k][0];
        const bool live = il >= c && il < R;
        if (il == c) {
          v = make_double2(1.0, 0.0);
          keep = sc[2];
        } else if (live) {
          v = cmul(v, scale);
          keep = v;
        }
        const dcplx cv = cmul(ctc, v);
#pragma unroll
        for (int q = 1; q < NB; ++q) {
          dcplx y = x[k][q];
          if (live && q < nt) {
            const dcplx p = cmul(cv, wv[q]);
            y.x -= p.x;
            y.y -= p.y;
          }
          x[k][q - 1] = y;
        }
        x[k][NB - 1] = keep;
      }
    }
    // T[0:c, c] = -tau T[0:c, 0:c] z with z_l = V_l^H v = conj(V_l[c]) + scale e_l (LAPACK zlarft)
    if (rank == 0 && warp == NW - 1) {
      const dcplx tc = make_double2(sc[0].x, -sc[0].y);
      if (lane < c) {
        dcplx sacc = make_double2(0.0, 0.0);
        for (int l = lane; l < c; ++l) {
          const dcplx p = cmul(Tsh[lane][l], zs[l]);
          sacc.x += p.x;
          sacc.y += p.y;
        }
        const dcplx t = cmul(tc, sacc);
        Tsh[lane][c] = make_double2(-t.x, -t.y);
      }
      if (lane == 0) Tsh[c][c] = tc;
      __syncwarp();
    }
  }
  // write back: the panel (R above the diagonal, v below) and the explicit V; column j is at
  // position j + NB - b
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int il = g + k * G;
    if (il >= R) continue;
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int j = q - (NB - b);
      if (j >= 0) {
        const dcplx y = x[k][q];
        A[il + lda * (int64_t)j] = y;
        V[il + ldv * (int64_t)j] = il > j ? y : (il == j ? make_double2(1.0, 0.0) : make_double2(0.0, 0.0));
      }
    }
  }
  for (int r = g; r < zabove; r += G)
    for (int j = 0; j < b; ++j) V[(int64_t)(r - zabove) + ldv * (int64_t)j] = make_double2(0.0, 0.0);
  if (rank == 0) {
    __syncthreads();
    for (int e = tid; e < b * b; e += NT) {
      const int i = e % b, j = e / b;
      T[i + (int64_t)ldt * j] = Tsh[i][j];
    }
  }
  // no CTA may leave while a peer can still write its shared memory
  if constexpr (CL > 1) cluster_sync();
}

// Compact-WY factor of an outer block from the factors of its inner panels (LAPACK
// zlarft, block form): T = [[T1, -T1 (V1^H V2) T2], [0, T2]] applied panel by panel,
// with G = V^H V of the whole outer block.  One CTA; T is bo x bo (ld bo).
struct PanelList {
  int n;
  short off[QR_NBO / 2 + 1];
  short w[QR_NBO / 2];
};

// T, G and the panels' products live in shared memory for the whole merge (one CTA), T and G
// in one array: the block of G above a panel's factor is read in that panel's step and then
// replaced by T's.  Bound by the latency of the sums' chains.
constexpr size_t QR_MERGE_SMEM = (size_t)QR_NBO * (QR_NBO + 1) * sizeof(dcplx);

constexpr int QR_MERGE_NT = 1024;   // one thread per output of a panel's step: 18 us (31 us with 256 threads)

__global__ void __launch_bounds__(QR_MERGE_NT) k_merge_t(int bo, PanelList pl, const dcplx* __restrict__ Tin,
                                                 const dcplx* __restrict__ G, dcplx* __restrict__ Tb) {
  grid_enter();
  extern __shared__ __align__(16) dcplx msm[];
  const int ld = bo + 1;
  dcplx* Ts = msm;                            // Ts[r + ld c]
  __shared__ dcplx Xs[QR_NBO][QR_NBMAX + 1];   // odd stride: no bank conflicts along r
  const int tid = threadIdx.x;
  for (int e = tid; e < bo * bo; e += blockDim.x) {
    const int r = e % bo, c = e / bo;
    int t = 0;
    while (t + 1 < pl.n && pl.off[t + 1] <= c) ++t;
    const int o = pl.off[t];
    dcplx v = make_double2(0.0, 0.0);
    if (r >= o && r < o + pl.w[t]) v = Tin[(size_t)t * QR_NBMAX * QR_NBMAX + (r - o) + QR_NBMAX * (c - o)];
    else if (r < o) v = G[r + (int64_t)bo * c];
    Ts[r + ld * c] = v;
  }
  __syncthreads();
  for (int t = 1; t < pl.n; ++t) {
    const int c0 = pl.off[t], bt = pl.w[t];
    const dcplx* Tt = Ts + c0 + ld * c0;   // the panel's own factor: Tt[v + ld u]
    for (int e = tid; e < c0 * bt; e += blockDim.x) {
      const int r = e % c0, u = e / c0;
      dcplx sacc = make_double2(0.0, 0.0);
      for (int l = r; l < c0; ++l) {
        const dcplx p = cmul(Ts[r + ld * l], Ts[l + ld * (c0 + u)]);
        sacc.x += p.x;
        sacc.y += p.y;
      }
      Xs[r][u] = sacc;
    }
    __syncthreads();
    for (int e = tid; e < c0 * bt; e += blockDim.x) {
      const int r = e % c0, u = e / c0;
      dcplx sacc = make_double2(0.0, 0.0);
      for (int v = 0; v <= u; ++v) {
        const dcplx p = cmul(Xs[r][v], Tt[v + ld * u]);
        sacc.x += p.x;
        sacc.y += p.y;
      }
      Ts[r + ld * (c0 + u)] = make_double2(-sacc.x, -sacc.y);
    }
    __syncthreads();
  }
  for (int e = tid; e < bo * bo; e += blockDim.x) Tb[e] = Ts[(e % bo) + ld * (e / bo)];
}

__global__ void k_extract_r(int k, int n, const dcplx* __restrict__ A, int64_t lda, dcplx* __restrict__ R,
                            int64_t ldr, dcplx* __restrict__ ph) {
  grid_enter();
  int64_t tot = (int64_t)k * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot; t += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(t % k), c = (int)(t / k);
    dcplx v = (r <= c) ? A[r + lda * c] : make_double2(0.0, 0.0);
    R[r + ldr * c] = v;
    if (r == c) {
      double a = hypot(v.x, v.y);
      ph[r] = (a > 0.0) ? make_double2(v.x / a, v.y / a) : make_double2(1.0, 0.0);
    }
  }
}

// out[i] = sum_c part[i + stride c] over nc partials, in a fixed order
__global__ void k_sum_partials(int64_t len, int nc, const dcplx* __restrict__ part, int64_t stride,
                               dcplx* __restrict__ out) {
  grid_enter();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x) {
    dcplx s = make_double2(0.0, 0.0);
    for (int c = 0; c < nc; ++c) {
      const dcplx v = part[i + stride * c];
      s.x += v.x;
      s.y += v.y;
    }
    out[i] = s;
  }
}

template <int NB, int RPT, int CL, int NT>
void launch_panel(Context* ctx, int R, int b, int zabove, dcplx* A, int64_t lda, dcplx* V, int64_t ldv, dcplx* tau,
                  dcplx* T, int ldt) {
  static_assert(NB * RPT == QR_NBMAX, "a thread holds 16 complex numbers");
  launch_kernel(ctx, k_qr_panel<NB, RPT, CL, NT>, CL, NT, 0, R, b, zabove, A, lda, V, ldv, tau, T, ldt);
  ctx->n_kernels++;
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) throw Error(IMPS_CUDA_ERROR, std::string("qr panel launch: ") + cudaGetErrorString(e));
}

// Panel width for a panel of R rows: the registers of a thread hold RPT rows x NB columns.
int panel_width(int R) {
  if (R <= QR_G) return 16;
  if (R <= 2 * QR_G) return 8;
  if (R <= 4 * QR_G) return 4;
  return 2;
}

// Small-product path for the updates inside an outer block (N <= 48 columns against
// b <= 16 reflectors): on these shapes a DMMA GEMM launch is all pipeline fill, so one
// kernel forms the long-K product and a second applies it.
constexpr int XS_NT = 256;   // threads of the X^H V kernel
constexpr int XS_ROWS = 64;  // rows staged in shared memory per step (one step per CTA)
constexpr int XS_COLS = 16;  // columns of X per CTA, one output (n, l) per thread
constexpr int XS_LD = XS_ROWS + 1;

// Wh (N x b, ld N) = X^H V over K rows, X (K x N) and V (K x b) with leading dimension ld.
// CTA (g, h) sums rows [g kc, (g + 1) kc) of columns [16 h, 16 h + 16) into part[g]; the last
// CTA of a column group to finish (counter[h]) adds the partials in CTA order, so the result
// does not depend on scheduling, resets the counter and, when T is given, forms its columns
// of Z (b x N, ld b) = op(T) Wh^H (op = C or N).  Bound by latency and shared-memory reads:
// column groups of 16 give three times the CTAs of one group of all columns (48 x 16 outputs
// over 512 rows: 8 us, 17 us in one group).
__global__ void __launch_bounds__(XS_NT) k_xhv_small(int K, int N, int b, int kc, const dcplx* __restrict__ X,
                                                      const dcplx* __restrict__ Vm, int64_t ld,
                                                      dcplx* __restrict__ part, unsigned* __restrict__ counter,
                                                      dcplx* __restrict__ Wh, const dcplx* __restrict__ T, int ldt,
                                                      int conjT, dcplx* __restrict__ Z) {
  grid_enter();
  __shared__ dcplx sh[(XS_COLS + QR_NBMAX) * XS_LD];  // [16 columns of X, b of V][XS_LD rows], later the summed Wh
  __shared__ dcplx Ts[QR_NBMAX][QR_NBMAX + 1];
  __shared__ bool last;
  const int nb = N * b, tid = threadIdx.x;
  const int n0 = blockIdx.y * XS_COLS, nn = min(XS_COLS, N - n0);
  const int k0 = blockIdx.x * kc, k1 = min(K, k0 + kc);
  const int nl = tid % XS_COLS, l = tid / XS_COLS;
  const bool live = nl < nn && l < b;
  dcplx acc = make_double2(0.0, 0.0);
  if (Z && tid < b * b) {   // op(T), read while the rows are on their way
    const int i = tid % b, j = tid / b;
    dcplx t = conjT ? T[j + (int64_t)ldt * i] : T[i + (int64_t)ldt * j];
    if (conjT) t.y = -t.y;
    Ts[i][j] = t;
  }
  for (int r0 = k0; r0 < k1; r0 += XS_ROWS) {
    const int nr = min(XS_ROWS, k1 - r0);
    __syncthreads();
#pragma unroll
    for (int e = tid; e < XS_ROWS * (XS_COLS + QR_NBMAX); e += XS_NT) {
      const int r = e % XS_ROWS, col = e / XS_ROWS;  // consecutive threads walk rows: coalesced
      dcplx v = make_double2(0.0, 0.0);
      if (r < nr) {
        if (col < XS_COLS) {
          if (col < nn) v = X[(int64_t)(r0 + r) + ld * (n0 + col)];
        } else if (col - XS_COLS < b) {
          v = Vm[(int64_t)(r0 + r) + ld * (col - XS_COLS)];
        }
      }
      sh[r + XS_LD * col] = v;
    }
    __syncthreads();
    if (live) {
      const dcplx* xc = sh + XS_LD * nl;
      const dcplx* vc = sh + XS_LD * (XS_COLS + l);
      for (int r = 0; r < nr; ++r) {
        const dcplx x = xc[r], v = vc[r];
        acc.x = fma(x.x, v.x, fma(x.y, v.y, acc.x));
        acc.y = fma(x.x, v.y, fma(-x.y, v.x, acc.y));
      }
    }
  }
  const int o = n0 + nl + N * l;
  if (live) part[(int64_t)blockIdx.x * nb + o] = acc;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = (atomicAdd(&counter[blockIdx.y], 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (live) {
    dcplx t = make_double2(0.0, 0.0);
    int g = 0;
    for (; g + 4 <= (int)gridDim.x; g += 4) {  // four loads in flight, added in CTA order
      const dcplx v0 = __ldcg(&part[(int64_t)g * nb + o]), v1 = __ldcg(&part[(int64_t)(g + 1) * nb + o]);
      const dcplx v2 = __ldcg(&part[(int64_t)(g + 2) * nb + o]), v3 = __ldcg(&part[(int64_t)(g + 3) * nb + o]);
      t.x += v0.x; t.y += v0.y;
      t.x += v1.x; t.y += v1.y;
      t.x += v2.x; t.y += v2.y;
      t.x += v3.x; t.y += v3.y;
    }
    for (; g < (int)gridDim.x; ++g) {
      const dcplx v = __ldcg(&part[(int64_t)g * nb + o]);
      t.x += v.x;
      t.y += v.y;
    }
    Wh[o] = t;
    sh[nl + XS_COLS * l] = t;
  }
  if (tid == 0) counter[blockIdx.y] = 0u;
  if (!Z) return;
  __syncthreads();
  // Z[i, n] = sum_l op(T)[i, l] conj(Wh[n, l])
  const int i = tid % QR_NBMAX, n = tid / QR_NBMAX;
  if (i < b && n < nn) {
    dcplx z = make_double2(0.0, 0.0);
    for (int q = 0; q < b; ++q) {
      const dcplx t = Ts[i][q], w = sh[n + XS_COLS * q];  // conj(w) below
      z.x += t.x * w.x + t.y * w.y;
      z.y += t.y * w.x - t.x * w.y;
    }
    Z[i + b * (n0 + n)] = z;
  }
}

// A2 (R x N, lda) -= V (R x b, ldv) Z (b x N), b <= 16, N <= 64: a thread per element,
// 64 rows x 4 columns per CTA (row loads coalesced, V rows shared through L1).  FULL: b = 16,
// all loads issued ahead of the sum.
template <bool FULL>
__global__ void __launch_bounds__(256) k_apply_small(int R, int N, int b, const dcplx* __restrict__ Vm, int64_t ldv,
                                                     const dcplx* __restrict__ Z, dcplx* __restrict__ A2,
                                                     int64_t lda) {
  grid_enter();
  const int r = blockIdx.x * 64 + (threadIdx.x & 63);
  const int n = blockIdx.y * 4 + (threadIdx.x >> 6);
  if (r >= R || n >= N) return;
  dcplx a = A2[r + lda * n];
  dcplx v[QR_NBMAX];
#pragma unroll
  for (int i = 0; i < QR_NBMAX; ++i)
    if (FULL || i < b) v[i] = Vm[r + ldv * i];
#pragma unroll
  for (int i = 0; i < QR_NBMAX; ++i) {
    if (FULL || i < b) {
      const dcplx z = __ldg(&Z[i + b * n]);
      a.x -= fma(v[i].x, z.x, -(v[i].y * z.y));
      a.y -= fma(v[i].x, z.y, v[i].y * z.x);
    }
  }
  A2[r + lda * n] = a;
}

// Wh = X^H V (and Z = op(T) Wh^H when T is given) by k_xhv_small.
void xhv_small(Context* ctx, int N, int b, int K, const dcplx* X, const dcplx* Vm, int64_t ld, dcplx* part,
               dcplx* Wh, const dcplx* T, int ldt, bool conjT, dcplx* Z) {
  IMPS_REQUIRE(N <= QR_NBO && b <= QR_NBMAX, IMPS_INVALID_ARG, "xhv_small: shape");
  DevBuf& cnt = ctx->buf("qr_xhv_count", 256);
  if (ctx->qr_count_ptr != cnt.ptr) {  // new counters start at zero; each launch leaves them at zero
    IMPS_CUDA(cudaMemsetAsync(cnt.ptr, 0, 256, ctx->stream));
    ctx->qr_count_ptr = cnt.ptr;
  }
  // one staged chunk of XS_ROWS rows per CTA, at most 64 partials (more rows per CTA past
  // that): the last CTA of a column group sums g values per output
  int g = std::max(1, std::min(64, (K + XS_ROWS - 1) / XS_ROWS));
  const int kc = (K + g - 1) / g;
  g = (K + kc - 1) / kc;
  ScopedTimer tm(ctx, "qr_small", 8.0 * N * b * (double)K);
  launch_kernel(ctx, k_xhv_small, dim3(g, (N + XS_COLS - 1) / XS_COLS), XS_NT, 0, K, N, b, kc, X, Vm, ld, part,
                static_cast<unsigned*>(cnt.ptr), Wh, T, ldt, conjT ? 1 : 0, Z);
  ctx->n_kernels++;
  IMPS_CUDA(cudaPeekAtLastError());
}

void apply_small(Context* ctx, int R, int N, int b, const dcplx* Vm, int64_t ldv, const dcplx* Z, dcplx* A2,
                 int64_t lda) {
  IMPS_REQUIRE(b <= QR_NBMAX && N <= QR_NBO, IMPS_INVALID_ARG, "apply_small: shape");
  ScopedTimer tm(ctx, "qr_small", 8.0 * R * N * (double)b);
  const dim3 grid((R + 63) / 64, (N + 3) / 4);
  if (b == QR_NBMAX) launch_kernel(ctx, k_apply_small<true>, grid, 256, 0, R, N, b, Vm, ldv, Z, A2, lda);
  else launch_kernel(ctx, k_apply_small<false>, grid, 256, 0, R, N, b, Vm, ldv, Z, A2, lda);
  ctx->n_kernels++;
  IMPS_CUDA(cudaPeekAtLastError());
}

// Wh (N x b, ld N) = X^H V with X (K x N) and V (K x b) sharing the leading dimension ld
// and a long K.  The long side N goes on the GEMM's 128-row output tile; K is split into
// row chunks (one batched GEMM over the full chunks and one for the remainder) so that
// about two CTAs per SM are busy, then the partial products are summed in a fixed order.
void gemm_xhv(Context* ctx, int N, int b, int K, const dcplx* X, const dcplx* Vm, int64_t ld, dcplx* part,
              dcplx* Wh) {
  const int tiles = ((N + 127) / 128) * ((b + 63) / 64);
  int nc = std::max(1, std::min({(2 * 148 + tiles - 1) / tiles, QR_MAXCHUNK, K / 64}));
  int kc = (K + nc - 1) / nc;
  kc = (kc + 15) / 16 * 16;
  nc = (K + kc - 1) / kc;
  // (zgemm_fp64 shares the K stages itself where the order of the sum is free)
  if (nc == 1 || !ctx->ordered_sums()) {
    zgemm_fp64(ctx, OP_C, OP_N, N, b, K, 1.0, X, ld, 0, Vm, ld, 0, 0.0, Wh, N, 0, 1);
    return;
  }
  const int nfull = K / kc, rem = K - nfull * kc;
  const int64_t pstride = (int64_t)N * b;
  if (nfull > 0)
    zgemm_fp64(ctx, OP_C, OP_N, N, b, kc, 1.0, X, ld, kc, Vm, ld, kc, 0.0, part, N, pstride, nfull);
  if (rem > 0)
    zgemm_fp64(ctx, OP_C, OP_N, N, b, rem, 1.0, X + (int64_t)nfull * kc, ld, 0, Vm + (int64_t)nfull * kc, ld, 0,
               0.0, part + pstride * nfull, N, 0, 1);
  const int g = (int)std::min<int64_t>((pstride + 255) / 256, 148 * 8);
  launch_kernel(ctx, k_sum_partials, std::max(g, 1), 256, 0, pstride, nc, part, pstride, Wh);
  ctx->n_kernels++;
}

// A2 (R x N) <- A2 - Y Wh^H with Y = V op(T) (R x b): one block-reflector application
// given Wh = A2^H V (op = C: A2 <- (I - V T V^H)^H A2; op = N: A2 <- (I - V T V^H) A2).
void apply_block(Context* ctx, int R, int N, int b, const dcplx* Vp, int64_t ldv, const dcplx* Tp, int ldt, Op opT,
                 const dcplx* Wh, dcplx* Y, dcplx* A2, int64_t lda) {
  zgemm_fp64(ctx, OP_N, opT, R, b, b, 1.0, Vp, ldv, 0, Tp, ldt, 0, 0.0, Y, R, 0, 1);
  zgemm_fp64(ctx, OP_N, OP_C, R, N, b, -1.0, Y, R, 0, Wh, N, 0, 1.0, A2, lda, 0, 1);
}

}  // namespace

// Factorisation half of QRpos: A = H_1 ... H_k [R; 0].  The explicit reflectors V, the
// compact-WY factor of every outer block and the diagonal phases stay in the slot's
// buffers (`<slot>_v`, `<slot>_t`, `<slot>_ph`) until the next factorisation into the
// same slot, so that Q can be formed later (qr_form_q) or not at all.  R gets the
// positive-diagonal phase fix.
void qr_factor(Context* ctx, int m, int n, const dcplx* M, int64_t ldm, dcplx* R, const char* slot) {
  IMPS_REQUIRE(m > 0 && n > 0, IMPS_INVALID_ARG, "qrpos: empty matrix");
  IMPS_REQUIRE(m <= 8 * QR_G, IMPS_INVALID_ARG, "qrpos: more than 32768 rows is not supported");
  ctx->n_qr++;
  const int k = std::min(m, n);
  const double qf = 8.0 * (2.0 * m * (double)n * k - 2.0 / 3.0 * k * (double)k * k);
  ctx->qr_flops += qf;
  ScopedTimer t(ctx, "qr", qf);
  const std::string sl(slot);
  const int nob = (k + QR_NBO - 1) / QR_NBO;
  const int wmax = std::max({n, k, QR_NBO});
  DevBuf& Ab = ctx->buf("qr_a", (size_t)m * n * sizeof(dcplx));
  DevBuf& Vb = ctx->buf(sl + "_v", (size_t)m * k * sizeof(dcplx));
  DevBuf& Tin = ctx->buf("qr_tin", (size_t)(QR_NBO / 2) * QR_NBMAX * QR_NBMAX * sizeof(dcplx));
  DevBuf& Tbig = ctx->buf(sl + "_t", (size_t)nob * QR_NBO * QR_NBO * sizeof(dcplx));
  DevBuf& Gb = ctx->buf("qr_g", (size_t)QR_NBO * QR_NBO * sizeof(dcplx));
  DevBuf& taub = ctx->buf("qr_tau", (size_t)k * sizeof(dcplx));
  DevBuf& ph = ctx->buf(sl + "_ph", (size_t)k * sizeof(dcplx));
  DevBuf& Wb = ctx->buf("qr_w", (size_t)QR_NBO * wmax * sizeof(dcplx));
  DevBuf& Yb = ctx->buf("qr_y", (size_t)QR_NBO * m * sizeof(dcplx));
  // partial products: the split-K GEMMs' chunks, or k_xhv_small's (up to 2 CTAs per SM)
  DevBuf& Pb = ctx->buf("qr_part", std::max((size_t)QR_NBO * wmax * QR_MAXCHUNK,
                                            (size_t)2 * ctx->num_sms * QR_NBO * QR_NBO) * sizeof(dcplx));
  DevBuf& Zb = ctx->buf("qr_z", (size_t)QR_NBMAX * QR_NBO * sizeof(dcplx));
  zcopy2d(ctx, m, n, M, ldm, Ab.z(), m);
  dcplx* A = Ab.z();
  int nblk = 0;
  for (int P = 0; P < k;) {
    const int bo = std::min(QR_NBO, k - P);
    PanelList pl;
    pl.n = 0;
    // inner panels; each also updates the rest of its outer block
    for (int p = P; p < P + bo;) {
      const int Rr = m - p;
      const int b = std::min(panel_width(Rr), P + bo - p);
      dcplx* Ap = A + p + (int64_t)m * p;
      dcplx* Vp = Vb.z() + p + (int64_t)m * p;
      dcplx* Tp = Tin.z() + (size_t)pl.n * QR_NBMAX * QR_NBMAX;
      switch (panel_width(Rr)) {
        case 16:
          if (Rr <= 128) launch_panel<16, 1, 1, 128>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX);
          else if (Rr <= 256) launch_panel<16, 1, 1, 256>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX);
          else if (Rr <= 512) launch_panel<16, 1, 8, 64>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX);
          else if (Rr <= 1024) launch_panel<16, 1, 8, 128>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX);
          else if (Rr <= 2048) launch_panel<16, 1, 8, 256>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX);
          else launch_panel<16, 1, 8, 512>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX);
          break;
        case 8: launch_panel<8, 2, 8, 512>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX); break;
        case 4: launch_panel<4, 4, 8, 512>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX); break;
        default: launch_panel<2, 8, 8, 512>(ctx, Rr, b, p - P, Ap, m, Vp, m, taub.z() + p, Tp, QR_NBMAX); break;
      }
      pl.off[pl.n] = (short)(p - P);
      pl.w[pl.n] = (short)b;
      pl.n++;
      const int n2in = P + bo - (p + b);
      if (n2in > 0) {
        // A2 <- A2 - V T^H (A2^H V)^H for the rest of the outer block
        dcplx* A2 = A + p + (int64_t)m * (p + b);
        xhv_small(ctx, n2in, b, Rr, A2, Vp, m, Pb.z(), Wb.z(), Tp, QR_NBMAX, true, Zb.z());
        apply_small(ctx, Rr, n2in, b, Vp, m, Zb.z(), A2, m);
      }
      p += b;
    }
    pl.off[pl.n] = (short)bo;
    // compact-WY factor of the outer block, then its trailing update
    const int RrB = m - P;
    dcplx* Vblk = Vb.z() + P + (int64_t)m * P;
    dcplx* Tb = Tbig.z() + (size_t)nblk * QR_NBO * QR_NBO;
    if (pl.n > 1) gemm_xhv(ctx, bo, bo, RrB, Vblk, Vblk, m, Pb.z(), Gb.z());
    static DeviceOnce merge_attr;
    merge_attr.run(ctx->device, [] {
      IMPS_CUDA(cudaFuncSetAttribute(k_merge_t, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QR_MERGE_SMEM));
    });
    launch_kernel(ctx, k_merge_t, 1, QR_MERGE_NT, QR_MERGE_SMEM, bo, pl, Tin.z(), Gb.z(), Tb);
    ctx->n_kernels++;
    const int n2 = n - (P + bo);
    if (n2 > 0) {
      dcplx* A2 = A + P + (int64_t)m * (P + bo);
      gemm_xhv(ctx, n2, bo, RrB, A2, Vblk, m, Pb.z(), Wb.z());
      apply_block(ctx, RrB, n2, bo, Vblk, m, Tb, bo, OP_C, Wb.z(), Yb.z(), A2, m);
    }
    ++nblk;
    P += bo;
  }
  {
    int64_t tot = (int64_t)k * n;
    int g = (int)std::min<int64_t>((tot + 255) / 256, 148 * 16);
    launch_kernel(ctx, k_extract_r, std::max(g, 1), 256, 0, k, n, A, m, R, k, ph.z());
    ctx->n_kernels++;
  }
  scale_q_r(ctx, 0, n, k, nullptr, 1, R, k, ph.z());  // R rows by conj(phase)
}

// Q (m x k, ld m) of the last qr_factor(m, n, ...) into `slot`:
// Q = H_1 ... H_k [I; 0] with the outer blocks applied from the last back, then the
// columns scaled by the diagonal phases (the positive-diagonal convention of QRpos).
void qr_form_q(Context* ctx, int m, int n, dcplx* Q, const char* slot) {
  const int k = std::min(m, n);
  const double qf = 8.0 * (2.0 * m * (double)n * k - 2.0 / 3.0 * k * (double)k * k);
  ctx->qr_flops += qf;
  ScopedTimer t(ctx, "qr", qf);
  const std::string sl(slot);
  const int nob = (k + QR_NBO - 1) / QR_NBO;
  const int wmax = std::max({n, k, QR_NBO});
  DevBuf& Vb = ctx->buf(sl + "_v", (size_t)m * k * sizeof(dcplx));
  DevBuf& Tbig = ctx->buf(sl + "_t", (size_t)nob * QR_NBO * QR_NBO * sizeof(dcplx));
  DevBuf& ph = ctx->buf(sl + "_ph", (size_t)k * sizeof(dcplx));
  DevBuf& Wb = ctx->buf("qr_w", (size_t)QR_NBO * wmax * sizeof(dcplx));
  DevBuf& Yb = ctx->buf("qr_y", (size_t)QR_NBO * m * sizeof(dcplx));
  DevBuf& Pb = ctx->buf("qr_part", (size_t)QR_NBO * wmax * QR_MAXCHUNK * sizeof(dcplx));
  zfill2d(ctx, m, k, 0.0, Q, m);
  zadd_diag(ctx, k, Q, m, 1.0);
  for (int t = nob - 1; t >= 0; --t) {
    const int P = t * QR_NBO, bo = std::min(QR_NBO, k - P);
    const int RrB = m - P, nc = k - P;
    dcplx* Vblk = Vb.z() + P + (int64_t)m * P;
    dcplx* Tb = Tbig.z() + (size_t)t * QR_NBO * QR_NBO;
    dcplx* Qs = Q + P + (int64_t)m * P;
    gemm_xhv(ctx, nc, bo, RrB, Qs, Vblk, m, Pb.z(), Wb.z());
    apply_block(ctx, RrB, nc, bo, Vblk, m, Tb, bo, OP_N, Wb.z(), Yb.z(), Qs, m);
  }
  scale_q_r(ctx, m, 0, k, Q, m, nullptr, k, ph.z());  // Q columns by phase
}

void qrpos(Context* ctx, int m, int n, const dcplx* M, int64_t ldm, dcplx* Q, dcplx* R) {
  qr_factor(ctx, m, n, M, ldm, R, "qr");
  if (Q) qr_form_q(ctx, m, n, Q, "qr");
}

// M (m x n) = L Q  <=>  M^H = Q^H L^H : QRpos of M^H (n x m) gives Q' (n x k), R' (k x m)
void lq_factor(Context* ctx, int m, int n, const dcplx* M, int64_t ldm, dcplx* L, const char* slot) {
  const int k = std::min(m, n);
  DevBuf& MH = ctx->buf("lq_mh", (size_t)m * n * sizeof(dcplx));
  DevBuf& Rp = ctx->buf("lq_r", (size_t)k * m * sizeof(dcplx));
  zconj_transpose(ctx, m, n, M, ldm, MH.z(), n);
  qr_factor(ctx, n, m, MH.z(), n, Rp.z(), slot);
  zconj_transpose(ctx, k, m, Rp.z(), k, L, m);  // L = R'^H  (m x k)
}

void lq_form_q(Context* ctx, int m, int n, dcplx* Q, const char* slot) {
  const int k = std::min(m, n);
  DevBuf& Qp = ctx->buf("lq_q", (size_t)n * k * sizeof(dcplx));
  qr_form_q(ctx, n, m, Qp.z(), slot);
  zconj_transpose(ctx, n, k, Qp.z(), n, Q, k);  // Q = Q'^H  (k x n)
}

void lqpos(Context* ctx, int m, int n, const dcplx* M, int64_t ldm, dcplx* L, dcplx* Q) {
  lq_factor(ctx, m, n, M, ldm, L, "qr");
  if (Q) lq_form_q(ctx, m, n, Q, "qr");
}

}  // namespace imps
