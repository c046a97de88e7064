// Unpreconditioned CG of one 2D scene inside one thread-block cluster.
//
// GridCg runs 2D scenes without a preconditioner (conjugategrad.cpp:
// 315-321): hundreds of iterations over a few thousand to a few hundred
// thousand cells.  As grid launches an iteration is four kernels whose work
// takes a microsecond or two and whose launches and cold starts take 27
// (96 x 128 cells, 377 iterations: 10.2 ms).  The scene's four vectors fit in
// the shared memory and registers of a cluster, so here one launch runs the
// whole solve and nothing but the result goes back to memory: 0.95 ms for the
// same solve, 2.5 us per iteration, most of it the latency of the two sums.
// Four steps of a batch of twelve 2D scenes (65^2 to 413^2, up to 950
// iterations) and four 3D ones went from 236 to 63 ms.
//
//  * CTA k of the cluster owns a strip of whole rows; thread t of T holds the
//    strip's cells t, t + T, ... (K of them): residual, A s and, up to 16
//    cells per thread, search value and pressure in registers.  The search
//    vector is also in shared memory for the neighbours, with one halo row on
//    each side.
//  * An iteration has two cluster-wide sums: (A s, s), and (r, r) with
//    max|r|.  A CTA's share goes into a slot of its own in the shared memory
//    of every CTA before a cluster barrier, and each then adds the slots in
//    rank order, so all CTAs hold the same bits and take the same branches
//    without a second exchange.
//  * The neighbours' edge rows of the residual travel with the second sum;
//    each CTA forms its halo rows of the search vector from them with the
//    owner's own arithmetic.  That saves a third barrier per iteration.
//
// Every cell's float operations are those of the grid kernels (pressure.cu),
// a thread sums its cells' products as theirs do, and the threads' sums are
// added up with more bits than their doubles have.  (Three floats to a sum cost
// instructions: with two, 48 bits, a 96 x 128 step takes 0.94 ms instead of 1.03.
// In double it is more: the FP64 pipe does two lanes a cycle.)
// The split depends on the scene's size alone, so a scene computes the same
// alone and in any batch.
#include <cfloat>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "mg_common.cuh"
#include "mg_kernels.h"
#include "mg_reduce.cuh"

namespace cg = cooperative_groups;

namespace mgpu {

namespace {

constexpr int kCcThreads = 512;     // of a CTA with a long strip
constexpr int kCcSmall = 256;       // of one with up to kCcStrip cells
constexpr int kCcStrip = 2048;
constexpr int kCcMaxCta = 16;
constexpr int kCcMaxK = 32;
static_assert(kCcStrip <= 8 * kCcSmall && kCcStrip >= 4 * kCcThreads, "the cells per thread that kernel_of has");
constexpr size_t kCcMaxSmem = 220 * 1024;

// a warp's share of a cluster sum: the sum and the largest |r| (as the float's
// bits; negative: none)
struct __align__(16) Share {
  TSum s;
  int mx;
};
template <int T>
struct SumSmem {
  static constexpr int kAdd = T / 128;  // warps that add up
  float2 part[T];
  int wmx[T / 32];
  Share share[2][kCcMaxCta * kAdd];  // of every CTA's adding warps, by sum
  float sum;
  int mx;
};

__device__ __forceinline__ TSum across(const TSum& a, int o) {
  return TSum{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o), __shfl_xor_sync(0xffffffffu, a.m, o)};
}

// The sum of the threads' sums over the cluster, rounded to float, and the
// maximum of mx, the same bits in every thread of every CTA.  Sums in three
// floats take instructions, so a quarter of a CTA's warps add up four threads
// each.  The cluster's shares are added up by every warp of a small CTA, by one
// of a large one (the other way about, steps of 96 x 128 and 150 x 170 cells are
// 3 % slower, those of 200 x 200 to 400 x 400 cells 5 %).
template <int T, bool MX>
__device__ __forceinline__ float cluster_sum(cg::cluster_group& cl, int ncta, SumSmem<T>& sm, int which, const FSum& own, int& mx) {
  constexpr int kAdd = SumSmem<T>::kAdd;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  sm.part[t] = make_float2(own.h, own.l);
  if (MX) {
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) sm.wmx[wid] = mx;
  }
  __syncthreads();
  if (wid < kAdd) {
    Share v{TSum{}, -1};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 p = sm.part[t + q * (T / 4)];
      if (q == 0) v.s = TSum{p.x, p.y, 0.f};
      else v.s.add(TSum{p.x, p.y, 0.f});
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v.s.add(across(v.s, o));
    if (MX) v.mx = __reduce_max_sync(0xffffffffu, sm.wmx[lane & (T / 32 - 1)]);
    if (ncta == 1) {
      if (lane == 0) sm.share[which][wid] = v;
    } else if (lane < ncta) {
      *cl.map_shared_rank(&sm.share[which][cl.block_rank() * kAdd + wid], lane) = v;
    }
  }
  if (ncta == 1) __syncthreads();
  else cl.sync();
  const int n = ncta * kAdd, lanes = min(n, 32);  // powers of two
  float sum = 0.f;
  if (T == kCcSmall || wid == 0) {
    Share v = sm.share[which][lane & (lanes - 1)];
    if (n > 32) {
      const Share u = sm.share[which][lane + 32];
      v.s.add(u.s);
      v.mx = max(v.mx, u.mx);
    }
    for (int o = lanes / 2; o > 0; o >>= 1) v.s.add(across(v.s, o));
    if (MX) mx = __reduce_max_sync(0xffffffffu, v.mx);
    sum = v.s.rounded();
  }
  if (T == kCcSmall) return sum;
  if (threadIdx.x == 0) {
    sm.sum = sum;
    sm.mx = mx;
  }
  __syncthreads();
  if (MX) mx = sm.mx;
  return sm.sum;
}

// the 2D part of a stencil code in a byte: A0 (bits 0-2), then the links
// -x, -y, +x, +y (bits 4-7).  A cell outside the fluid has the identity row:
// A0 = 1 and no links.
__device__ __forceinline__ unsigned pack_code(int c) {
  if (!(c & kCodeFluid)) return 1u;
  return (unsigned)((c & 7) | (c & (kLowX | kLowY)) | ((c & (kHighX | kHighY)) >> 1));
}
constexpr unsigned kBLowX = 16, kBLowY = 32, kBHighX = 64, kBHighY = 128;

template <int K, int T, bool A0>
__global__ void __launch_bounds__(T, 1) k_cg_cluster(const CgClusterScene* tab, CgClusterScene one) {
  extern __shared__ __align__(16) float smem[];
  __shared__ SumSmem<T> s_sum;
  constexpr bool kRegs = K <= 16;  // search and pressure values in registers
  cg::cluster_group cl = cg::this_cluster();
  const int ncta = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const CgClusterScene S = tab ? tab[blockIdx.x / ncta] : one;
  CgScalars* g = S.sc;
  if (g->done) return;  // the same for every CTA of the cluster
  const int tid = threadIdx.x;
  const int nx = S.nx, y0 = min(rank * S.rows, S.ny), R = min(S.rows, S.ny - y0);
  const int cells = R * nx, cap = S.rows * nx;
  const long long base = (long long)y0 * nx;
  const bool low = R > 0 && y0 > 0, high = R > 0 && y0 + R < S.ny;
  float* s_s = smem + nx;             // search: a halo row, the strip, a halo row
  float* s_rlo = smem + 2 * nx + cap; // residual of the neighbours' edge rows
  float* s_rhi = s_rlo + nx;
  float* s_p = s_rhi + nx;            // pressure (K > 16)
  float* s_a = s_p + (kRegs ? 0 : cap);  // diagonal (A0)
  const float accuracy = g->accuracy;
  const int maxIter = g->maxIter;

  float r[K], t[K], sv[kRegs ? K : 1], p[kRegs ? K : 1];
  unsigned code[(K + 3) / 4];
  int mx = -1;
  FSum acc;
#pragma unroll
  for (int q = 0; q < (K + 3) / 4; q++) code[q] = 0;
#pragma unroll
  for (int q = 0; q < K; q++) {
    const int e = tid + T * q;
    r[q] = 0.f;
    t[q] = 0.f;
    if (kRegs) sv[q] = p[q] = 0.f;
    if (e < cells) {
      const float v = S.rhs[base + e];
      r[q] = v;
      if (kRegs) sv[q] = v;
      else s_p[e] = 0.f;
      s_s[e] = v;
      const int c = S.code[base + e];
      code[q >> 2] |= pack_code(c) << (8 * (q & 3));
      if (A0) s_a[e] = (c & kCodeFluid) ? S.A0f[base + e] : 1.f;
      acc.add(v * v);
    }
  }
  for (int x = tid; x < nx; x += T) {
    smem[x] = low ? S.rhs[base - nx + x] : 0.f;
    if (R > 0) s_s[cells + x] = high ? S.rhs[base + cells + x] : 0.f;
    s_rlo[x] = s_rhi[x] = 0.f;
  }
  // no CTA stores into another's shared memory before that one has set it up
  if (ncta == 1) __syncthreads();
  else cl.sync();
  float* const rloUp = high ? cl.map_shared_rank(s_rlo, rank + 1) : s_rlo;   // where the next strip keeps my last row
  float* const rhiDown = low ? cl.map_shared_rank(s_rhi, rank - 1) : s_rhi;  // where the previous one keeps my first
  float sigma = cluster_sum<T, false>(cl, ncta, s_sum, 1, acc, mx);
  float alpha = 0.f, beta = 0.f, dp = 0.f, res = g->resNorm;
  int it = 0, done = 0, status = 0;

  while (it < maxIter) {
    // A s and (A s, s): ApplyMatrix2D (conjugategrad.h:137-151)
    acc = FSum();
#pragma unroll
    for (int q = 0; q < K; q++) {
      const int e = tid + T * q;
      if (e < cells) {
        const unsigned c = code[q >> 2] >> (8 * (q & 3));
        const float xc = kRegs ? sv[q] : s_s[e];
        float v = xc * (A0 ? s_a[e] : (float)(c & 7u));
        const float xl = s_s[e - 1], xr = s_s[e + 1], yl = s_s[e - nx], yr = s_s[e + nx];
        if (c & kBLowX) v = v - xl;
        if (c & kBHighX) v = v - xr;
        if (c & kBLowY) v = v - yl;
        if (c & kBHighY) v = v - yr;
        t[q] = v;
        acc.add(v * xc);
      }
    }
    dp = cluster_sum<T, false>(cl, ncta, s_sum, 0, acc, mx);
    alpha = fabsf(dp) > 0.f ? sigma / dp : 0.f;
    const float na = -alpha;
    // p += alpha s, r -= alpha A s; (r, r) and max|r|
    acc = FSum();
    mx = __float_as_int(-1.f);
#pragma unroll
    for (int q = 0; q < K; q++) {
      const int e = tid + T * q;
      if (e < cells) {
        if (kRegs) p[q] = p[q] + alpha * sv[q];
        else s_p[e] = s_p[e] + alpha * s_s[e];
        const float rv = r[q] + na * t[q];
        r[q] = rv;
        if (low && e < nx) rhiDown[e] = rv;
        if (high && e >= cells - nx) rloUp[e - (cells - nx)] = rv;
        acc.add(rv * rv);
        if (rv == rv) mx = max(mx, __float_as_int(fabsf(rv)));  // NaN takes no part, as in fmaxf
      }
    }
    const float sigmaNew = cluster_sum<T, true>(cl, ncta, s_sum, 1, acc, mx);
    it++;
    res = __int_as_float(mx);
    if (res < 0.f) res = S.nanNorm;
    if (res < accuracy) {
      sigma = res;
      done = 1;
      break;
    }
    beta = sigmaNew / sigma;
    sigma = sigmaNew;
    if (!(res < 1e35f)) {
      status = 2;
      done = 1;
      break;
    }
    // s = r + beta s (UpdateSearchVec), the halo rows with their owners' values
#pragma unroll
    for (int q = 0; q < K; q++) {
      const int e = tid + T * q;
      if (e < cells) {
        const float v = r[q] + beta * (kRegs ? sv[q] : s_s[e]);
        if (kRegs) sv[q] = v;
        s_s[e] = v;
      }
    }
    for (int x = tid; x < nx; x += T) {
      if (low) smem[x] = s_rlo[x] + beta * smem[x];
      if (high) s_s[cells + x] = s_rhi[x] + beta * s_s[cells + x];
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < K; q++) {
    const int e = tid + T * q;
    if (e < cells) S.p[base + e] = kRegs ? p[q] : s_p[e];
  }
  if (rank == 0 && tid == 0) {
    g->sigma = sigma;
    g->alpha = alpha;
    g->beta = beta;
    g->dp = dp;
    g->resNorm = res;
    g->iterations = it;
    g->status = status;
    g->done = done;
  }
}

typedef void (*CgClusterKernel)(const CgClusterScene*, CgClusterScene);
template <bool A0>
CgClusterKernel kernel_of(int threads, int k) {
  if (threads == kCcSmall) switch (k) {
    case 1: return k_cg_cluster<1, kCcSmall, A0>;
    case 2: return k_cg_cluster<2, kCcSmall, A0>;
    case 4: return k_cg_cluster<4, kCcSmall, A0>;
    default: return k_cg_cluster<8, kCcSmall, A0>;
  }
  switch (k) {
    case 8: return k_cg_cluster<8, kCcThreads, A0>;
    case 16: return k_cg_cluster<16, kCcThreads, A0>;
    default: return k_cg_cluster<32, kCcThreads, A0>;
  }
}
CgClusterKernel kernel_of(int threads, int k, bool a0) { return a0 ? kernel_of<true>(threads, k) : kernel_of<false>(threads, k); }

int g_ccMaxCta = 0;

size_t cc_smem(int nx, int rows, int k, bool a0) {
  const size_t cap = (size_t)nx * rows;
  return sizeof(float) * (4 * (size_t)nx + cap * (1 + (k > 16 ? 1 : 0) + (a0 ? 1 : 0)));
}

cudaLaunchConfig_t cc_config(int ctas, int threads, int scenes, size_t smem, cudaLaunchAttribute* at, cudaStream_t s) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = ctas;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctas * scenes));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace

int cg_cluster_prepare() {
  for (int k = 1; k <= kCcMaxK; k *= 2)
    for (int a = 0; a < 4; a++) {
      const CgClusterKernel f = kernel_of(a & 2 ? kCcThreads : kCcSmall, k, (a & 1) != 0);
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCcMaxSmem) != cudaSuccess ||
          cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return 1;
    }
  // the largest cluster the GPU co-schedules with a CTA's full shared memory
  g_ccMaxCta = 0;
  for (int c = kCcMaxCta; c >= 1 && !g_ccMaxCta; c /= 2) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = cc_config(c, kCcThreads, 1, kCcMaxSmem, at, nullptr);
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, kernel_of(kCcThreads, kCcMaxK, true), &cfg) == cudaSuccess && nc >= 1) g_ccMaxCta = c;
  }
  cudaGetLastError();
  return 0;
}

// Strips of about 2048 cells: an iteration's arithmetic and its two barriers
// then take about as long.  Up to there 256 threads of 8 cells, whose sums take
// half the instructions of 512 of 4 (steps of 64 x 64, 96 x 128 and 150 x 170
// cells 0.55, 1.06 and 1.48 ms instead of 0.59, 1.17 and 1.61); the largest scenes take every CTA of the
// largest cluster and up to 32 cells per thread.
bool cg_cluster_plan(const Dims& d, bool a0, CgClusterPlan* pl) {
  if (d.is3d || !g_ccMaxCta) return false;
  int c = 1;
  auto rows = [&](int ctas) { return (d.ny + ctas - 1) / ctas; };
  while (c < g_ccMaxCta && (long long)rows(c) * d.nx > kCcStrip) c *= 2;
  const long long strip = (long long)rows(c) * d.nx;
  if (strip > (long long)kCcThreads * kCcMaxK) return false;
  pl->threads = strip <= kCcStrip ? kCcSmall : kCcThreads;
  int k = pl->threads == kCcSmall ? 1 : 8;
  while ((long long)pl->threads * k < strip) k *= 2;
  pl->ctas = c;
  pl->k = k;
  pl->rows = rows(c);
  pl->smem = cc_smem(d.nx, pl->rows, k, a0);
  return pl->smem <= kCcMaxSmem;
}

cudaError_t launch_cg_cluster(const CgClusterPlan& pl, const CgClusterScene* tab, const CgClusterScene& one, int scenes,
                              bool a0, cudaStream_t s) {
  count_launch();
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t cfg = cc_config(pl.ctas, pl.threads, scenes, pl.smem, at, s);
  return cudaLaunchKernelEx(&cfg, kernel_of(pl.threads, pl.k, a0), tab, one);
}

}  // namespace mgpu
