// Particle systems and the FLIP grid transfers (plugin/flip.cpp:549-673):
// mapPartsToMAC, mapMACToParts, flipVelocityUpdate, mapPartsToGrid(Vec3),
// mapGridToParts(Vec3).
//
// Layout: a BasicParticleSystem (particle.h:182-193) is kept as four device
// arrays -- x, y, z, flag -- and a ParticleDataImpl<Real|Vec3|int>
// (particle.h:306) as one or three; the host side keeps the reference's
// records (16-byte {Vec3 pos; int flag;}, 12-byte Vec3) and uploads and
// downloads transpose them on the GPU.
//
// Grid-to-particle transfers are one thread per particle.  Particle-to-grid
// transfers (the reference's single-threaded setInterpolated loops,
// knMapLinearVec3ToMACGrid and knMapLinear) add every particle's weighted
// value into the 8 faces or cells around it, in particle order, so a face's
// float sums depend on that order.  The results here are the reference's bit
// for bit:
//
//  * MAC faces in 3D (mapPartsToMAC): the particles are listed, in particle
//    order, by the tiles of 4^3 or 8^3 cells they reach, and one warp per tile
//    adds them up one after another, a particle's 24 faces at a time, in
//    shared memory (k_tile_*).
//  * Cells (mapPartsToGrid), 2D, and systems too large for the lists: the
//    particles are sorted, stably, by the cell their interpolation stencil
//    starts at (one LSD radix sort per MAC component), and each face or cell
//    merges the up to 8 sorted buckets that reach it by particle index.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <set>
#include <string>

#include "../../include/mantagpu.h"
#include "mg_batch.h"
#include "mg_common.cuh"
#include "mg_f32x2.cuh"
#include "mg_kernels.h"

using namespace mgpu;

namespace {

constexpr int kPDelete = 1 << 10;  // ParticleBase::PDELETE (particle.h:41)
constexpr float kVecEps = 1e-6f;   // VECTOR_EPSILON of the float build (util/vectorbase.h:52)
constexpr int kRsThreads = 256, kRsItems = 8, kRsTile = kRsThreads * kRsItems;

// ---------------------------------------------------------------- records
__global__ void k_parts_unpack(long long n, const float4* __restrict__ rec, float* x, float* y, float* z, int* flag) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float4 r = rec[i];
    x[i] = r.x;
    y[i] = r.y;
    z[i] = r.z;
    flag[i] = __float_as_int(r.w);
  }
}
__global__ void k_parts_pack(long long n, float4* rec, const float* __restrict__ x, const float* __restrict__ y,
                             const float* __restrict__ z, const int* __restrict__ flag) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    rec[i] = make_float4(x[i], y[i], z[i], __int_as_float(flag[i]));
}
// Vec3 records <-> three planes (dir 0: unpack, 1: pack)
__global__ void k_vec_transpose(long long n, float* rec, float* a, float* b, float* c, int dir) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (dir == 0) {
      a[i] = rec[3 * i];
      b[i] = rec[3 * i + 1];
      c[i] = rec[3 * i + 2];
    } else {
      rec[3 * i] = a[i];
      rec[3 * i + 1] = b[i];
      rec[3 * i + 2] = c[i];
    }
  }
}

// -------------------------------------------------------- stencil buckets
// The first cell of a particle's interpolation stencil: BUILD_INDEX
// (util/interpol.h:50-66) for cell-centred grids (comp -1), BUILD_INDEX_SHIFT
// (:116-130) with component comp shifted for MAC faces.  In 2D the z index
// is 0 for every particle of the slab z in [0,1) (the reference's 2D
// particles sit at z = 0.5); it is taken as 0 for any other z as well.
// Particles that are deleted, or whose type matches exclude, get the key
// ncells, past every bucket.
struct PartView {
  const float* x;
  const float* y;
  const float* z;
  const int* flag;
  const int* ptype;  // may be null
  int exclude;
};

__device__ __forceinline__ bool part_skip(const PartView& p, long long i) {
  return (p.flag[i] & kPDelete) != 0 || (p.ptype && (p.ptype[i] & p.exclude) != 0);
}

__global__ void k_stencil_keys(Dims d, PartView p, long long n, int comp, unsigned* keys, unsigned* vals) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned key = (unsigned)d.n;
  if (!part_skip(p, i)) {
    const float px = p.x[i], py = p.y[i], pz = p.z[i];
    const Wts w = build_index<false>(d, px, py, pz);
    int xi = w.xi, yi = w.yi, zi = w.zi;
    if (comp >= 0) {
      const Wts s = build_index<true>(d, px, py, pz);
      if (comp == 0) xi = s.xi;
      if (comp == 1) yi = s.yi;
      if (comp == 2) zi = s.zi;
    }
    if (!d.is3d) zi = 0;
    key = (unsigned)(xi + d.nx * (yi + d.ny * zi));
  }
  keys[i] = key;
  vals[i] = (unsigned)i;
}

// -------------------------------------------------------------- radix sort
// One stable pass of an LSD radix sort on 8-bit digits.  A CTA owns a tile
// of 2048 consecutive elements; counts are stored digit-major (digit x
// tiles), so their exclusive scan gives every (digit, tile) its first output
// slot in digit order, then tile order.
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const unsigned* __restrict__ keys, long long n, int shift,
                                                        unsigned* hist, int tiles) {
  __shared__ unsigned h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kRsTile;
  for (int r = 0; r < kRsItems; r++) {
    const long long i = base + r * kRsThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[(size_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Within a tile, elements are placed in index order: rounds of 256 in turn,
// warps in turn within a round, lanes in turn within a warp (a lane's rank
// among the lanes holding its digit comes from __match_any_sync).
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const unsigned* __restrict__ kin,
                                                           const unsigned* __restrict__ vin, unsigned* kout,
                                                           unsigned* vout, long long n, int shift,
                                                           const unsigned* __restrict__ offs, int tiles) {
  __shared__ unsigned run[256];
  __shared__ unsigned wc[kRsThreads / 32][256];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  run[t] = offs[(size_t)t * tiles + blockIdx.x];
  const long long base = (long long)blockIdx.x * kRsTile;
  for (int r = 0; r < kRsItems; r++) {
#pragma unroll
    for (int q = 0; q < kRsThreads / 32; q++) wc[q][t] = 0;
    __syncthreads();
    const long long i = base + r * kRsThreads + t;
    const bool ok = i < n;
    unsigned key = 0, val = 0, dig = 0, rank = 0;
    const unsigned act = __ballot_sync(0xffffffffu, ok);
    if (ok) {
      key = kin[i];
      val = vin[i];
      dig = (key >> shift) & 255u;
      const unsigned peers = __match_any_sync(act, dig);
      rank = __popc(peers & ((1u << lane) - 1u));
      if (rank == 0) wc[w][dig] = __popc(peers);
    }
    __syncthreads();
    // thread t owns digit t: exclusive prefix over the warps, after the
    // slots taken by earlier rounds
    unsigned acc = run[t];
#pragma unroll
    for (int q = 0; q < kRsThreads / 32; q++) {
      const unsigned c = wc[q][t];
      wc[q][t] = acc;
      acc += c;
    }
    run[t] = acc;
    __syncthreads();
    if (ok) {
      const unsigned dst = wc[w][dig] + rank;
      kout[dst] = key;
      vout[dst] = val;
    }
    __syncthreads();
  }
}

// exclusive scan of n unsigned values in place: per-block scans of 2048,
// one CTA scanning the block totals, then the block offsets added
__device__ __forceinline__ unsigned block_excl_scan(unsigned v, unsigned* sh, unsigned* total) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    unsigned s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < (int)(blockDim.x >> 5)) sh[lane] = s;
  }
  __syncthreads();
  const unsigned before = (w > 0 ? sh[w - 1] : 0u) + x - v;
  *total = sh[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before;
}

__global__ void __launch_bounds__(kRsThreads) k_scan_tiles(unsigned* a, long long n, unsigned* sums) {
  __shared__ unsigned sh[32];
  const long long base = (long long)blockIdx.x * kRsTile + (long long)threadIdx.x * kRsItems;
  unsigned v[kRsItems], tot = 0;
#pragma unroll
  for (int q = 0; q < kRsItems; q++) {
    v[q] = base + q < n ? a[base + q] : 0u;
    tot += v[q];
  }
  unsigned blockTotal;
  unsigned run = block_excl_scan(tot, sh, &blockTotal);
#pragma unroll
  for (int q = 0; q < kRsItems; q++) {
    if (base + q < n) a[base + q] = run;
    run += v[q];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = blockTotal;
}

__global__ void __launch_bounds__(kRsThreads) k_scan_sums(unsigned* sums, int m) {
  __shared__ unsigned sh[32];
  unsigned carry = 0;
  for (int b0 = 0; b0 < m; b0 += kRsThreads) {
    const int i = b0 + threadIdx.x;
    const unsigned v = i < m ? sums[i] : 0u;
    unsigned tot;
    const unsigned ex = block_excl_scan(v, sh, &tot);
    if (i < m) sums[i] = carry + ex;
    carry += tot;
  }
}

__global__ void k_scan_add(unsigned* a, long long n, const unsigned* __restrict__ sums) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) a[i] += sums[i / kRsTile];
}

// starts[b] = first position of key >= b in the sorted keys (b = 0..ncells)
__global__ void k_bucket_starts(const unsigned* __restrict__ keys, long long n, long long ncells, unsigned* starts) {
  const long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (b > ncells) return;
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if ((long long)keys[mid] < b)
      lo = mid + 1;
    else
      hi = mid;
  }
  starts[b] = (unsigned)lo;
}

}  // namespace

namespace {

// ----------------------------------------------------- particle -> grid
// Positions and values copied into bucket order after a sort, so that the
// faces' merges read them in sequence instead of gathering each particle
// from its own index (every particle is read by up to 8 faces per sort).
struct SortedParts {
  const float* x;
  const float* y;
  const float* z;
  const float* v[3];
};
__global__ void k_sorted_copy(long long n, const unsigned* __restrict__ sorted, PartView p, const float* __restrict__ v0,
                              const float* __restrict__ v1, const float* __restrict__ v2, float* sx, float* sy,
                              float* sz, float* s0, float* s1, float* s2) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned k = sorted[i];
  sx[i] = p.x[k];
  sy[i] = p.y[k];
  sz[i] = p.z[k];
  s0[i] = __ldg(v0 + k);
  if (v1) {
    s1[i] = __ldg(v1 + k);
    s2[i] = __ldg(v2 + k);
  }
}

// The weights setInterpol / setInterpolMAC give the stencil corner (dx, dy,
// dz) of a particle: T[dy] * (S[dx] * F[dz]) (util/interpol.h:93-112,
// 159-195), with the axis of MAC component comp shifted.
struct CornerW {
  float S[2], T[2], F[2];
};
// One axis of BUILD_INDEX / BUILD_INDEX_SHIFT: the weights of the lower and
// upper sample for the coordinate q (already shifted by -0.5 or not), with
// the border clamps (the upper one only where the axis has more than one
// cell).  The same operations as build_index, one axis at a time, so a
// component's weights take three axes instead of both full variants.
__device__ __forceinline__ void axis_weights(float q, int n, bool clampHigh, float* w) {
  const int i = (int)q;
  float w1 = q - (float)i, w0 = 1.f - w1;
  if (q < 0.f) {
    w0 = 1.f;
    w1 = 0.f;
  }
  if (clampHigh && i >= n - 1) {
    w0 = 0.f;
    w1 = 1.f;
  }
  w[0] = w0;
  w[1] = w1;
}
__device__ __forceinline__ CornerW corner_weights(const Dims& d, float px, float py, float pz, int comp) {
  CornerW c;
  axis_weights(comp == 0 ? px : px - 0.5f, d.nx, true, c.S);
  axis_weights(comp == 1 ? py : py - 0.5f, d.ny, true, c.T);
  axis_weights(comp == 2 ? pz : pz - 0.5f, d.nz, d.nz > 1, c.F);
  return c;
}

// One thread per face (comp >= 0, MAC component comp) or cell (comp -1):
// merge the sorted buckets of the up to 8 stencil origins that reach it by
// particle index and add each particle's weight and weighted value in that
// order.  In 2D the z stride is 0, so the reference adds both z layers of a
// particle's stencil to the same face: the z = 1 layer first, except for the
// MAC z component, which adds its z = 0 layer first.
// Then, for MAC faces (mapPartsToMAC, flip.cpp:585-594): weights below
// VECTOR_EPSILON are stomped to 0 and the sum divided by a non-zero weight
// (safeDivide, general.h:150); vel, velOld and the optional weight grid are
// written.  For cells (mapPartsToGrid, knSafeDivReal, flip.cpp:549-557):
// weights below VECTOR_EPSILON give 0, others divide.
template <int kComps>
__global__ void __launch_bounds__(256) k_p2g_gather(Dims d, int comp, SortedParts sp,
                                                    const unsigned* __restrict__ sorted,
                                                    const unsigned* __restrict__ starts, float* o0, float* o1,
                                                    float* o2, float* old, float* wout) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i >= d.nx || j >= d.ny) return;
  constexpr unsigned kEnd = 0xffffffffu;
  unsigned cur[8], end[8], head[8];
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int bi = i - (q & 1), bj = j - ((q >> 1) & 1), bk = k - (q >> 2);
    const bool ok = bi >= 0 && bi <= d.nx - 2 && bj >= 0 && bj <= d.ny - 2 &&
                    (d.is3d ? (bk >= 0 && bk <= d.nz - 2) : (q >> 2) == 0);
    cur[q] = end[q] = 0;
    if (ok) {
      const long long key = bi + (long long)d.nx * (bj + (long long)d.ny * (d.is3d ? bk : 0));
      cur[q] = starts[key];
      end[q] = starts[key + 1];
    }
    head[q] = cur[q] < end[q] ? sorted[cur[q]] : kEnd;
  }
  const bool zFirst0 = comp == 2;  // 2D: which z layer the reference adds first
  float sum = 0.f, r0 = 0.f, r1 = 0.f, r2 = 0.f;
  for (;;) {
    unsigned best = head[0];
    int bq = 0;
#pragma unroll
    for (int q = 1; q < 8; q++)
      if (head[q] < best) {
        best = head[q];
        bq = q;
      }
    if (best == kEnd) break;
    unsigned at = cur[0];  // the particle's slot in bucket order
#pragma unroll
    for (int q = 1; q < 8; q++)
      if (q == bq) at = cur[q];
    const CornerW c = corner_weights(d, __ldg(sp.x + at), __ldg(sp.y + at), __ldg(sp.z + at), comp);
    const int dx = bq & 1, dy = (bq >> 1) & 1, dz = bq >> 2;
    const float a0 = __ldg(sp.v[0] + at);
    const float a1 = kComps == 3 ? __ldg(sp.v[1] + at) : 0.f;
    const float a2 = kComps == 3 ? __ldg(sp.v[2] + at) : 0.f;
    if (d.is3d) {
      const float w = c.T[dy] * (c.S[dx] * c.F[dz]);
      sum += w;
      r0 += w * a0;
      if (kComps == 3) {
        r1 += w * a1;
        r2 += w * a2;
      }
    } else {
#pragma unroll
      for (int layer = 0; layer < 2; layer++) {
        const int lz = zFirst0 ? layer : 1 - layer;
        const float w = c.T[dy] * (c.S[dx] * c.F[lz]);
        sum += w;
        r0 += w * a0;
        if (kComps == 3) {
          r1 += w * a1;
          r2 += w * a2;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (q == bq) {
        cur[q]++;
        head[q] = cur[q] < end[q] ? sorted[cur[q]] : kEnd;
      }
  }
  const long long o = ix(d, i, j, k);
  if (comp >= 0) {
    const float ws = sum < kVecEps ? 0.f : sum;
    const float v = ws != 0.f ? r0 / ws : r0;
    o0[o] = v;
    old[o] = v;
    if (wout) wout[o] = ws;
  } else if (sum < kVecEps) {
    o0[o] = 0.f;
    if (kComps == 3) {
      o1[o] = 0.f;
      o2[o] = 0.f;
    }
  } else {
    o0[o] = r0 / sum;
    if (kComps == 3) {
      o1[o] = r1 / sum;
      o2[o] = r2 / sum;
    }
  }
}

// ---------------------------------------------- particles -> MAC faces
// The serial sums of the faces of a tile of cells depend on nothing but the
// particles that reach the tile, in particle order.  So: list those (a
// particle near a tile's border is in up to eight lists: 1.9 on average with
// 8 x 8 x 4 cells, 2.6 with 4^3), put every list into particle order, and let
// one warp per tile walk its list.  Lane 8 c + k of it owns the faces of
// component c and parity k: it reads the particle's three weights and value of
// that component, forms its face's weight as the reference does, and adds in
// shared memory, about 20 instructions for a particle's 24 faces.  The weights
// come from a batch of 32 particles whose lanes prepared one each.
//
// At 128^3 with 16.0 M particles mapPartsToMAC takes 1.45 ms, lists 0.11 + 0.16,
// sort 0.38, splat 0.9, where a radix sort and eight-way merges per component took
// 5.5 (3.2 of it in the merges, about 100 instructions per contribution).  The
// splat is bound by shared memory, ten wavefronts per particle of a tile (96 % of
// the rate), the sort by its instructions.  With particles in random order the
// lists' atomics and the loads by index weigh more: 10.8 M in 108 x 125 x 100 take
// 3.3 ms, in seeding order 0.95 (sorted and merged: 5.8 and 3.8).
template <int X, int Y, int Z>
struct TileShape {
  static constexpr int x = X, y = Y, z = Z;
};
using TileLarge = TileShape<8, 8, 4>;
using TileSmall = TileShape<4, 4, 4>;
constexpr int kLine = 32;  // words of 128 bytes
// the two sorts in shared memory: most list entries, warps, most bits of a pass
constexpr int kSortShort = 4608, kShortWarps = 8, kShortBits = 10;
constexpr int kSortLong = 24576, kLongWarps = 32, kLongBits = 9;
constexpr int kPieceBits = 14;  // longer lists are sorted in pieces
struct Tiles {
  Dims d;
  long long n;
  int tx, ty, tz;
  bool large;         // TileLarge, not TileSmall
  unsigned* starts;   // [tiles + 1]: the lists' first entries
  unsigned* cursor;   // [tiles][kLine], word 0: counts, then next entries
  unsigned* list;     // particles by tile
  const float* v[3];  // velocity components
  __host__ __device__ int count() const { return tx * ty * tz; }
  __device__ unsigned* counter(int t) const { return cursor + (size_t)t * kLine; }
  // the lists too long for the first sort, in any order, in word 1; how many,
  // and how many of them are taken
  __device__ unsigned* job(unsigned q) const { return cursor + (size_t)q * kLine + 1; }
  __device__ unsigned* jobs() const { return cursor + 2; }
  __device__ unsigned* ticket() const { return cursor + 3; }
};

// one axis of BUILD_INDEX / BUILD_INDEX_SHIFT: first sample and upper weight
// (the lower one is 1 minus it, in the border clamps too)
__device__ __forceinline__ int axis_sample(float q, int n, float& w1) {
  int i = (int)q;
  w1 = q - (float)i;
  if (q < 0.f) {
    i = 0;
    w1 = 0.f;
  }
  if (i >= n - 1) {
    i = n - 2;
    w1 = 1.f;
  }
  return i;
}
__device__ __forceinline__ int axis_sample(float q, int n) {
  float w;
  return axis_sample(q, n, w);
}

// Counts of a tile's particles, or their entries (kFill).  A particle's faces
// of all three components lie in at most 2 x 2 x 2 tiles.  The lanes of a warp
// with the same tile take it with one atomic; particles in flight are mostly
// neighbours, so each tile's counter has a line of its own (side by side, the
// atomics queue at a few L2 slices: 295 and 361 us at 128^3, now 110
// and 156).
template <class T, bool kFill>
__global__ void __launch_bounds__(256) k_tile_lists(Tiles s, PartView p) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  float x = 0.f, y = 0.f, z = 0.f;
  bool live = i < s.n;
  if (live) {  // before the flag is known
    x = p.x[i];
    y = p.y[i];
    z = p.z[i];
    live = !part_skip(p, i);
  }
  const int a0 = axis_sample(x - 0.5f, s.d.nx) / T::x, a1 = (axis_sample(x, s.d.nx) + 1) / T::x;
  const int b0 = axis_sample(y - 0.5f, s.d.ny) / T::y, b1 = (axis_sample(y, s.d.ny) + 1) / T::y;
  const int c0 = axis_sample(z - 0.5f, s.d.nz) / T::z, c1 = (axis_sample(z, s.d.nz) + 1) / T::z;
  const int t0 = a0 + s.tx * (b0 + s.ty * c0);
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const bool in = live && (!(q & 1) || a1 > a0) && (!(q & 2) || b1 > b0) && (!(q & 4) || c1 > c0);
    if (!__any_sync(0xffffffffu, in)) continue;
    const int t = in ? t0 + (q & 1) + s.tx * ((q >> 1 & 1) + s.ty * (q >> 2)) : -1;
    const unsigned act = __ballot_sync(0xffffffffu, in);
    if (!in) continue;
    const unsigned peers = __match_any_sync(act, t);
    const int first = __ffs(peers) - 1;
    if (!kFill) {
      if (lane == first) atomicAdd(s.counter(t), (unsigned)__popc(peers));
    } else {
      unsigned at = 0;
      if (lane == first) at = atomicAdd(s.counter(t), (unsigned)__popc(peers));
      at = __shfl_sync(peers, at, first) + __popc(peers & ((1u << lane) - 1u));
      s.list[at] = (unsigned)i;
    }
  }
}

// counts to first entries, and the list of the long lists; one CTA, eight tiles
// per thread at a time
__global__ void __launch_bounds__(1024) k_tile_starts(Tiles s) {
  __shared__ unsigned sh[32];
  const int tiles = s.count();
  unsigned carry = 0;
  for (int t0 = threadIdx.x * 8; t0 - (int)threadIdx.x * 8 < tiles; t0 += 8192) {
    unsigned c[8], sum = 0, total;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      c[q] = t0 + q < tiles ? *s.counter(t0 + q) : 0u;
      sum += c[q];
    }
    unsigned at = carry + block_excl_scan(sum, sh, &total);
    carry += total;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      if (t0 + q < tiles) s.starts[t0 + q] = *s.counter(t0 + q) = at;
      if (c[q] > kSortShort) *s.job(atomicAdd(s.jobs(), 1u)) = t0 + q;
      at += c[q];
    }
  }
  if (threadIdx.x == 0) s.starts[tiles] = carry;
}

// A tile's list into particle order.  Up to kCap entries: an LSD radix sort in
// shared memory over the bits in which the list's entries can differ, kWarps
// warps on consecutive pieces of the list (digit counts per warp, scanned
// digit by digit, keep it stable), at most kBits bits to a pass.  A first
// kernel takes a CTA for every list and sorts the short ones, four CTAs of 8
// warps per SM; the longer ones, which k_tile_starts has listed, go to a second
// one, a CTA of 32 warps per SM that takes them one after another.  At 128^3
// lists are short up to nine particles per cell, and fit the shared memory up
// to 49; mapPartsToMAC with 8, 16, 27, 48 and 64 per cell in seeding order takes
// 1.6, 3.6, 5.9, 9.9 and 18 ms (sorted by cell and merged: 5.6, 11, 22, 48 and 79).
template <int kCap, int kWarps, int kBits>
__device__ __forceinline__ void sort_list(unsigned* list, unsigned n, unsigned* sm) {
  constexpr int kThreads = 32 * kWarps;
  __shared__ unsigned sh[32], range[2];
  unsigned *in = sm, *out = sm + kCap;
  unsigned short* const cnt = (unsigned short*)(sm + 2 * kCap);  // [warps][1 << width]
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) {
    range[0] = 0xffffffffu;
    range[1] = 0u;
  }
  unsigned least = 0xffffffffu, most = 0u;
  for (unsigned e = t; e < n; e += kThreads) {
    const unsigned v = list[e];
    in[e] = v;
    least = min(least, v);
    most = max(most, v);
  }
  least = __reduce_min_sync(0xffffffffu, least);
  most = __reduce_max_sync(0xffffffffu, most);
  __syncthreads();
  if (lane == 0) {
    atomicMin(range, least);
    atomicMax(range + 1, most);
  }
  __syncthreads();
  least = range[0];
  const int bits = 32 - __clz(range[1] - least), passes = (bits + kBits - 1) / kBits;
  const int width = max(8, (bits + passes - 1) / max(passes, 1)), digits = 1 << width;
  const int each = max(1, digits / kThreads);
  const unsigned mask = digits - 1;
  const unsigned per = ((n + kWarps - 1) / kWarps + 31) & ~31u;
  const unsigned from = min(n, w * per), to = min(n, from + per);
  unsigned short* const mine = cnt + w * digits;
  for (int pass = 0, shift = 0; pass < passes; pass++, shift += width) {
    for (int q = lane; q < digits / 2; q += 32) ((unsigned*)mine)[q] = 0u;
    __syncwarp();
    for (unsigned e = from + lane; e < to; e += 32) {
      const unsigned dig = (in[e] - least) >> shift & mask;
      atomicAdd((unsigned*)mine + (dig >> 1), 1u << (dig & 1) * 16);
    }
    __syncthreads();
    unsigned sum = 0, total;
    for (int g = t * each; g < min((t + 1) * each, digits); g++)
#pragma unroll
      for (int q = 0; q < kWarps; q++) sum += cnt[q * digits + g];
    unsigned at = block_excl_scan(sum, sh, &total);
    for (int g = t * each; g < min((t + 1) * each, digits); g++)
#pragma unroll
      for (int q = 0; q < kWarps; q++) {
        const unsigned c = cnt[q * digits + g];
        cnt[q * digits + g] = (unsigned short)at;
        at += c;
      }
    __syncthreads();
    for (unsigned e0 = from; e0 < to; e0 += 32) {
      const bool ok = e0 + lane < to;
      const unsigned v = ok ? in[e0 + lane] : 0u, dig = (v - least) >> shift & mask;
      // lanes with the same digit, by one vote per bit: __match_any_sync takes
      // far longer when all digits differ
      unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
      for (int q = 0; q < kBits; q++)
        if (q < width) {
          const unsigned ones = __ballot_sync(0xffffffffu, dig >> q & 1u);
          peers &= dig >> q & 1u ? ones : ~ones;
        }
      const unsigned rank = __popc(peers & ((1u << lane) - 1u)), at = mine[dig];
      __syncwarp();
      if (ok) {
        out[at + rank] = v;
        if (rank == 0) mine[dig] = (unsigned short)(at + __popc(peers));
      }
      __syncwarp();
    }
    __syncthreads();
    unsigned* const x = in;
    in = out;
    out = x;
  }
  for (unsigned e = t; e < n; e += kThreads) list[e] = in[e];
  __syncthreads();
}
constexpr size_t sort_smem(int cap, int warps, int bits) { return 2 * (size_t)cap * 4 + ((size_t)warps << bits) * 2; }
constexpr size_t kShortSmem = sort_smem(kSortShort, kShortWarps, kShortBits);
constexpr size_t kLongSmem = sort_smem(kSortLong, kLongWarps, kLongBits);

__global__ void __launch_bounds__(32 * kShortWarps) k_tile_sort(Tiles s) {
  extern __shared__ __align__(16) unsigned sm[];
  const unsigned lo = s.starts[blockIdx.x], n = s.starts[blockIdx.x + 1] - lo;
  if (n > 1 && n <= kSortShort) sort_list<kSortShort, kShortWarps, kShortBits>(s.list + lo, n, sm);
}

// Lists longer than the shared memory: pieces of kPiece entries are sorted,
// then merged two, four, ... at a time by a bitonic network, whose steps
// across pieces run in place in the list; what is left of a merge inside a
// piece is the piece's sort.  Every comparison is upward (the first step of a
// merge pairs an entry with its mirror image), so that places past the end
// count as larger and never move.
constexpr unsigned kPiece = 1u << kPieceBits;
static_assert(kPiece <= kSortLong, "a piece is sorted in shared memory");
__device__ void sort_list_pieces(unsigned* list, unsigned n, unsigned* sm) {
  auto pieces = [&]() {
    for (unsigned b = 0; b < n; b += kPiece) sort_list<kSortLong, kLongWarps, kLongBits>(list + b, min(kPiece, n - b), sm);
  };
  pieces();
  for (int top = kPieceBits; top < 31 && 1u << top < n; top++) {
    for (int lg = top; lg >= kPieceBits; lg--) {
      const unsigned h = 1u << lg, pairs = (((n - 1) >> (lg + 1)) + 1) << lg;
      for (unsigned e = threadIdx.x; e < pairs; e += 32 * kLongWarps) {
        const unsigned r = e & (h - 1), x = ((e >> lg) << (lg + 1)) + r, y = lg == top ? x + 2 * h - 1 - 2 * r : x + h;
        if (y >= n) continue;
        const unsigned vx = list[x], vy = list[y];
        if (vy < vx) {
          list[x] = vy;
          list[y] = vx;
        }
      }
      __syncthreads();
    }
    pieces();
  }
}
__global__ void __launch_bounds__(32 * kLongWarps) k_tile_sort_long(Tiles s) {
  extern __shared__ __align__(16) unsigned sm[];
  __shared__ unsigned taken;
  const unsigned jobs = *s.jobs();
  while (jobs > 0) {
    if (threadIdx.x == 0) taken = atomicAdd(s.ticket(), 1u);
    __syncthreads();
    const unsigned q = taken;
    __syncthreads();
    if (q >= jobs) break;
    const unsigned t = *s.job(q), lo = s.starts[t], n = s.starts[t + 1] - lo;
    if (n <= kSortLong) sort_list<kSortLong, kLongWarps, kLongBits>(s.list + lo, n, sm);
    else sort_list_pieces(s.list + lo, n, sm);
  }
}

// A tile's accumulators in shared memory, {weight, weighted value} per face.
// A lane owns the faces of one component and one parity along x, y and z: a
// particle has one face of each, and no two lanes ever add to the same one.
template <class T>
struct TileAcc {
  static constexpr int kRow = 32;  // lanes: no bank conflicts (with 24, the lanes that add: 20 % fewer tiles' worth of memory, 9 % slower)
  static constexpr int kY = T::x / 2, kZ = kY * (T::y / 2), kAll = kZ * (T::z / 2);
  float2 acc[kAll][kRow];
  // A batch of 32 particles.  Weights of the odd faces and value of particles
  // 2 i and 2 i + 1 by component, {x, x, y, y}, {z, z, value, value}:
  float4 w[16][7];
  uint4 in[3][8];  // 5-bit fields: first sample - tile's first cell + 8 per axis
  uint4 at[3][8];  // from bit 16: byte offset of the first sample's row of acc; below, the rows' steps along axes with an odd sample
};

// two floats in shared memory, without a branch
__device__ __forceinline__ void add_if(unsigned at, bool in, float x, float y) {
  asm volatile(
      "{.reg .pred p;\n .reg .f32 a, b;\n mov.f32 a, 0f00000000;\n mov.f32 b, a;\n setp.ne.b32 p, %1, 0;\n"
      " @p ld.shared.v2.f32 {a, b}, [%0];\n add.f32 a, a, %2;\n add.f32 b, b, %3;\n @p st.shared.v2.f32 [%0], {a, b};}" ::"r"(at),
      "r"((int)in), "f"(x), "f"(y)
      : "memory");
}

template <class T>
__global__ void __launch_bounds__(32) k_tile_splat(Tiles s, PartView p, float* vel, float* old, float* wout) {
  __shared__ TileAcc<T> sm;
  typedef TileAcc<T> A;
  const Dims& d = s.d;
  const int lane = threadIdx.x;
  const int x0 = blockIdx.x * T::x, y0 = blockIdx.y * T::y, z0 = blockIdx.z * T::z;
  const int t = blockIdx.x + s.tx * (blockIdx.y + s.ty * blockIdx.z);
  const unsigned lo = s.starts[t], n = s.starts[t + 1] - lo;
  const unsigned* const list = s.list + lo;
  for (int q = lane; q < A::kAll * A::kRow; q += 32) (&sm.acc[0][0])[q] = make_float2(0.f, 0.f);
  // This lane's component and parity.  Its weight along an axis is that of the
  // odd face, or 1 minus it.  (Exact: with an odd first sample the odd face has
  // the lower weight, 1 minus the upper one, which is a multiple of 2^-23.)
  const int c = min(lane >> 3, 2), ox = lane & 1, oy = lane >> 1 & 1, oz = lane >> 2 & 1;
  const float2 ax = both(ox ? 0.f : 1.f), bx = both(ox ? 1.f : -1.f);
  const float2 ay = both(oy ? 0.f : 1.f), by = both(oy ? 1.f : -1.f);
  const float2 az = both(oz ? 0.f : 1.f), bz = both(oz ? 1.f : -1.f);
  // The face's row is (first sample + 1 - parity) / 2 per axis, in the tile if
  // the fields' upper bits are 8; bit 15 keeps the last lanes out.
  const unsigned up = (unsigned)((1 - ox) | (1 - oy) << 5 | (1 - oz) << 10) | (lane < 24 ? 0u : 0x8000u);
  constexpr unsigned kMask = (0x1fu & ~(T::x - 1u)) | (0x1fu & ~(T::y - 1u)) << 5 | (0x3fu & ~(T::z - 1u)) << 10;
  constexpr unsigned kIn = 8u | 8u << 5 | 8u << 10;
  constexpr int kStep = 8 * A::kRow;
  static_assert((kStep & kStep * A::kY) == 0 && (kStep * A::kY & kStep * A::kZ) == 0 && (kStep & kStep * A::kZ) == 0, "steps share bits");
  const unsigned steps = (ox ? 0 : kStep) | (oy ? 0 : kStep * A::kY) | (oz ? 0 : kStep * A::kZ);
  const unsigned own = (unsigned)__cvta_generic_to_shared(&sm.acc[0][min(lane, A::kRow - 1)]);
  // a particle's index is fetched two batches ahead, the particle one
  unsigned next = 0;
  float px = 0.f, py = 0.f, pz = 0.f, v0 = 0.f, v1 = 0.f, v2 = 0.f;
  auto fetch = [&](unsigned e) {
    if (e >= n) return;
    px = __ldg(p.x + next);
    py = __ldg(p.y + next);
    pz = __ldg(p.z + next);
    v0 = __ldg(s.v[0] + next);
    v1 = __ldg(s.v[1] + next);
    v2 = __ldg(s.v[2] + next);
    if (e + 32 < n) next = list[e + 32];
  };
  if (lane < n) next = list[lane];
  fetch(lane);
  for (unsigned b = 0; b < n; b += 32) {
    {
      float sx, sy, sz, cx, cy, cz;
      const int isx = axis_sample(px, d.nx, sx) - x0, icx = axis_sample(px - 0.5f, d.nx, cx) - x0;
      const int isy = axis_sample(py, d.ny, sy) - y0, icy = axis_sample(py - 0.5f, d.ny, cy) - y0;
      const int isz = axis_sample(pz, d.nz, sz) - z0, icz = axis_sample(pz - 0.5f, d.nz, cz) - z0;
      auto odd = [](int i, float w) { return i & 1 ? 1.f - w : w; };
      auto pack = [&](int comp, int x, int y, int z, float wx, float wy, float wz, float v) {
        float* const w = (float*)&sm.w[lane >> 1][2 * comp] + (lane & 1);
        w[0] = wx;
        w[2] = wy;
        w[4] = wz;
        w[6] = v;
        const unsigned in = (unsigned)(x + 8) | (unsigned)(y + 8) << 5 | (unsigned)(z + 8) << 10;
        ((unsigned*)sm.in[comp])[lane] = b + lane < n ? in : 0u;
        ((unsigned*)sm.at[comp])[lane] = (unsigned)(kStep * ((x >> 1) + A::kY * (y >> 1) + A::kZ * (z >> 1))) << 16 |
                                         kStep * ((x & 1) + A::kY * (y & 1) + A::kZ * (z & 1));
      };
      sx = odd(isx, sx);
      sy = odd(isy, sy);
      sz = odd(isz, sz);
      cx = odd(icx, cx);
      cy = odd(icy, cy);
      cz = odd(icz, cz);
      pack(0, isx, icy, icz, sx, cy, cz, v0);
      pack(1, icx, isy, icz, cx, sy, cz, v1);
      pack(2, icx, icy, isz, cx, cy, sz, v2);
    }
    __syncwarp();
    fetch(b + 32 + lane);
    const int m = (int)min(32u, n - b);
    for (int k0 = 0; k0 < m; k0 += 4) {
      const uint4 i4 = sm.in[c][k0 >> 2], a4 = sm.at[c][k0 >> 2];
      const unsigned in[4] = {i4.x, i4.y, i4.z, i4.w}, at[4] = {a4.x, a4.y, a4.z, a4.w};
      float2 wk[2], wv[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const float4 xy = sm.w[(k0 >> 1) + k][2 * c], zv = sm.w[(k0 >> 1) + k][2 * c + 1];
        // fma with factors 1 and -1: the odd face's weight itself, or 1 minus it
        const float2 S = fma2(bx, make_float2(xy.x, xy.y), ax), Ty = fma2(by, make_float2(xy.z, xy.w), ay);
        const float2 F = fma2(bz, make_float2(zv.x, zv.y), az);
        wk[k] = mul2(Ty, mul2(S, F));
        wv[k] = mul2(wk[k], make_float2(zv.z, zv.w));
      }
#pragma unroll
      for (int k = 0; k < 4; k++)
        add_if(own + ((int)at[k] >> 16) + (at[k] & steps), ((in[k] + up) & kMask) == kIn, k & 1 ? wk[k >> 1].y : wk[k >> 1].x,
               k & 1 ? wv[k >> 1].y : wv[k >> 1].x);
    }
    __syncwarp();
  }
  __syncwarp();
  for (int q = lane; q < 3 * T::x * T::y * T::z; q += 32) {
    const int comp = q / (T::x * T::y * T::z), e = q % (T::x * T::y * T::z);
    const int x = e % T::x, y = e / T::x % T::y, z = e / (T::x * T::y);
    const int i = x0 + x, j = y0 + y, k = z0 + z;
    if (i >= d.nx || j >= d.ny || k >= d.nz) continue;
    // stomp and safeDivide, as k_p2g_gather for MAC components
    const float2 o = sm.acc[(x >> 1) + A::kY * (y >> 1) + A::kZ * (z >> 1)][8 * comp + (x & 1) + 2 * (y & 1) + 4 * (z & 1)];
    const long long g = comp * d.n + ix(d, i, j, k);
    const float ws = o.x < kVecEps ? 0.f : o.x;
    const float v = ws != 0.f ? o.y / ws : o.y;
    vel[g] = v;
    old[g] = v;
    if (wout) wout[g] = ws;
  }
}

// ----------------------------------------------------- grid -> particle
// mapMACToParts (knMapLinearMACGridToVec3_PIC, flip.cpp:643-650) and, with
// old, flipVelocityUpdate (knMapLinearMACGridToVec3_FLIP, :659-668):
//   pvel = flipRatio * (pvel + (v - vOld)) + (1.0 - flipRatio) * v
// where the second product is formed in double and rounded to float.
// The branch-free index (kClamp): 16 M particles at 128^3 that the flow has mixed
// take 842 us with it and 960 with selections (FLIP 1678 and 1818), particles in
// the grid's order 199 and 182 (359 and 342).  A few thousand particles take the
// selections (4000 at 16^3 5.2 us and 6.2, 20 000 at 32^3 4.3 and 4.7).
constexpr long long kFewParticles = 1 << 16;
template <bool kClamp>
__global__ void k_mac_to_parts(Dims d, PartView p, long long n, CMac vel, CMac old, float flipRatio, float* pu,
                               float* pv, float* pw) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n || part_skip(p, i)) return;
  const float x = p.x[i], y = p.y[i], z = p.z[i];
  const V3 v = interp_mac<true, kClamp>(d, vel, x, y, z);
  if (!old.u) {
    pu[i] = v.x;
    pv[i] = v.y;
    pw[i] = v.z;
    return;
  }
  const V3 o = interp_mac<true, kClamp>(d, old, x, y, z);
  const float dlx = v.x - o.x, dly = v.y - o.y, dlz = v.z - o.z;
  const double keep = 1.0 - (double)flipRatio;
  pu[i] = flipRatio * (pu[i] + dlx) + (float)(keep * (double)v.x);
  pv[i] = flipRatio * (pv[i] + dly) + (float)(keep * (double)v.y);
  pw[i] = flipRatio * (pw[i] + dlz) + (float)(keep * (double)v.z);
}

// mapGridToParts(Vec3) (knMapFromGrid, flip.cpp:625-631): every active
// particle, interpol<T> per component; by the branch-free index at every count (a
// Real, 2 M particles at 64^3 in the grid's order: 12.5 us and 13.4 by selections;
// 200 000 there 4.8 and 4.4; mixed, and below 65 536, alike)
__global__ void k_grid_to_parts(Dims d, PartView p, long long n, const float* __restrict__ g0,
                                const float* __restrict__ g1, const float* __restrict__ g2, float* t0, float* t1,
                                float* t2) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n || (p.flag[i] & kPDelete) != 0) return;
  const float x = p.x[i], y = p.y[i], z = p.z[i];
  t0[i] = interp<true>(d, g0, x, y, z);
  if (g1) {
    t1[i] = interp<true>(d, g1, x, y, z);
    t2[i] = interp<true>(d, g2, x, y, z);
  }
}

}  // namespace

// ================================================================ host side
struct mg_particles_s {
  mg_solver s;
  Dims d;
  cudaStream_t st;
  long long cap = 0, n = 0;
  float *x = nullptr, *y = nullptr, *z = nullptr;
  int* flag = nullptr;
  // Scratch of the transfers, ten words per particle: the tile lists of
  // mapPartsToMAC, or the sort's keys and particle indices (ping-pong) and the
  // particles in bucket order.  Beside it the sort's per-tile digit counts,
  // their scan's block totals and the bucket starts (ncells + 1).
  unsigned* scratch = nullptr;
  unsigned *keys[2] = {nullptr, nullptr}, *vals[2] = {nullptr, nullptr};
  unsigned *hist = nullptr, *sums = nullptr, *starts = nullptr;
  float* sorted[6] = {};  // positions and up to 3 values in bucket order
  void* stage = nullptr;  // 16 bytes per particle for record transfers
  void* tileMem = nullptr;  // the tile lists' starts and counters, from the first mapPartsToMAC on
  Tiles tiles{};
};

struct mg_pdata_s {
  mg_particles p;
  int kind;  // MG_REAL, MG_VEC3, MG_INT
  float* c[3] = {nullptr, nullptr, nullptr};
};

namespace {

std::mutex g_partMu;
std::set<mg_particles> g_parts;
std::set<mg_pdata> g_pdata;

bool valid_parts(mg_particles p) {
  std::lock_guard<std::mutex> lk(g_partMu);
  return p && g_parts.count(p);
}
bool valid_pdata(mg_pdata d) {
  std::lock_guard<std::mutex> lk(g_partMu);
  return d && g_pdata.count(d) && g_parts.count(d->p);
}

void free_parts(mg_particles p) {
  cudaStreamSynchronize(p->st);
  void* bufs[] = {p->x, p->y, p->z, p->flag, p->scratch, p->hist, p->sums, p->starts, p->stage, p->tileMem};
  for (void* b : bufs)
    if (b) cudaFree(b);
}

int tiles_of(long long n) { return (int)((n + kRsTile - 1) / kRsTile); }

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

int blocks_of(long long n, int b = 256) { return (int)std::max<long long>(1, (n + b - 1) / b); }

int launch_status(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(MG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return MG_OK;
}

// exclusive scan of m counts in place
void scan_counts(mg_particles p, unsigned* a, long long m) {
  const int blocks = (int)((m + kRsTile - 1) / kRsTile);
  count_launch();
  k_scan_tiles<<<blocks, kRsThreads, 0, p->st>>>(a, m, p->sums);
  count_launch();
  k_scan_sums<<<1, kRsThreads, 0, p->st>>>(p->sums, blocks);
  count_launch();
  k_scan_add<<<blocks_of(m), 256, 0, p->st>>>(a, m, p->sums);
}

// sort the live particles by the first cell of their stencil (comp -1: cell
// centred, 0..2: MAC component); returns the particle indices in bucket order
// and fills p->starts
const unsigned* sort_stencil(mg_particles p, int comp, const PartView& v) {
  const long long n = p->n, ncells = p->d.n;
  if (n == 0) {
    cudaMemsetAsync(p->starts, 0, (size_t)(ncells + 1) * sizeof(unsigned), p->st);
    return p->vals[0];
  }
  count_launch();
  k_stencil_keys<<<blocks_of(n), 256, 0, p->st>>>(p->d, v, n, comp, p->keys[0], p->vals[0]);
  int bits = 0;
  while (bits < 32 && (ncells >> bits) != 0) bits++;
  const int passes = (bits + 7) / 8;
  const int tiles = tiles_of(n);
  int a = 0;
  for (int pass = 0; pass < passes; pass++) {
    const int shift = 8 * pass;
    count_launch();
    k_rs_hist<<<tiles, kRsThreads, 0, p->st>>>(p->keys[a], n, shift, p->hist, tiles);
    scan_counts(p, p->hist, 256LL * tiles);
    count_launch();
    k_rs_scatter<<<tiles, kRsThreads, 0, p->st>>>(p->keys[a], p->vals[a], p->keys[1 - a], p->vals[1 - a], n, shift,
                                                   p->hist, tiles);
    a = 1 - a;
  }
  count_launch();
  k_bucket_starts<<<blocks_of(ncells + 1), 256, 0, p->st>>>(p->keys[a], n, ncells, p->starts);
  return p->vals[a];
}

// the live particles' positions and values (1 or 3 planes) in bucket order
SortedParts sorted_copy(mg_particles p, const unsigned* sorted, const PartView& v, const float* v0, const float* v1,
                        const float* v2) {
  const long long n = p->n;
  if (n > 0) {
    count_launch();
    k_sorted_copy<<<blocks_of(n), 256, 0, p->st>>>(n, sorted, v, v0, v1, v2, p->sorted[0], p->sorted[1],
                                                    p->sorted[2], p->sorted[3], p->sorted[4], p->sorted[5]);
  }
  SortedParts sp{p->sorted[0], p->sorted[1], p->sorted[2], {p->sorted[3], p->sorted[4], p->sorted[5]}};
  return sp;
}

// Whether mapPartsToMAC takes the tile lists: in 3D, with room for every
// particle in the eight tiles that it can reach (eight of the scratch's ten
// words), and memory for the tiles' tables.  The larger tiles from a million
// cells on: with the small ones a call by itself at 128^3 takes 2.31 instead of
// 1.58 ms.  Below, a large tile's list is too long a serial walk for the few tiles
// there are (75 x 62 x 90: 0.52 instead of 0.45 ms with the transfer back).
bool tile_lists(mg_particles p) {
  if (p->tileMem) return true;
  Tiles& s = p->tiles;
  s.d = p->d;
  s.large = s.d.n >= 1000000;
  auto across = [&](int n, int large, int small) { return s.large ? (n + large - 1) / large : (n + small - 1) / small; };
  s.tx = across(s.d.nx, TileLarge::x, TileSmall::x);
  s.ty = across(s.d.ny, TileLarge::y, TileSmall::y);
  s.tz = across(s.d.nz, TileLarge::z, TileSmall::z);
  const size_t cap = (size_t)std::max<long long>(p->cap, 1), tiles = (size_t)s.tx * s.ty * s.tz;
  if (!s.d.is3d || s.d.nx < 3 || s.d.ny < 3 || s.d.nz < 3 || 8 * cap > 0xffffffffu || s.ty > 65535 || s.tz > 65535) return false;
  const size_t starts = align256((tiles + 1) * 4);
  if (cudaFuncSetAttribute(k_tile_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShortSmem) != cudaSuccess ||
      cudaFuncSetAttribute(k_tile_sort_long, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLongSmem) != cudaSuccess ||
      cudaMalloc(&p->tileMem, starts + tiles * kLine * 4) != cudaSuccess) {
    cudaGetLastError();
    p->tileMem = nullptr;
    return false;
  }
  s.starts = (unsigned*)p->tileMem;
  s.cursor = (unsigned*)((char*)p->tileMem + starts);
  s.list = p->scratch;
  return true;
}

// mapPartsToMAC in 3D
template <class T>
void tile_mac(mg_particles p, const Tiles& s, const PartView& v, float* vel, float* old, float* w) {
  cudaStream_t st = p->st;
  if (s.n == 0) cudaMemsetAsync(s.starts, 0, (s.count() + 1) * sizeof(unsigned), st);
  else {
    cudaMemsetAsync(s.cursor, 0, (size_t)s.count() * kLine * sizeof(unsigned), st);
    const int blocks = blocks_of(s.n);
    count_launch();
    k_tile_lists<T, false><<<blocks, 256, 0, st>>>(s, v);
    count_launch();
    k_tile_starts<<<1, 1024, 0, st>>>(s);
    count_launch();
    k_tile_lists<T, true><<<blocks, 256, 0, st>>>(s, v);
    count_launch();
    k_tile_sort<<<s.count(), 32 * kShortWarps, kShortSmem, st>>>(s);
    count_launch();
    k_tile_sort_long<<<std::min(sm_count(), s.count()), 32 * kLongWarps, kLongSmem, st>>>(s);
  }
  count_launch();
  k_tile_splat<T><<<dim3(s.tx, s.ty, s.tz), 32, 0, st>>>(s, v, vel, old, w);
}

PartView view_of(mg_particles p, mg_pdata ptype, int exclude) {
  PartView v{p->x, p->y, p->z, p->flag, ptype ? (const int*)ptype->c[0] : nullptr, exclude};
  return v;
}

// a grid of the particle system's solver, of one of the given kinds
int grid_of(mg_particles p, mg_grid g, unsigned kindMask, const char* what, float** data, int* kind) {
  int nx, ny, nz, k;
  if (mg_grid_get_info(g, &nx, &ny, &nz, &k)) return set_error(MG_ERR_ARG, std::string(what) + ": invalid grid");
  if (!((kindMask >> k) & 1u)) return set_error(MG_ERR_ARG, std::string(what) + ": wrong grid type");
  void* dp = nullptr;
  void* sp = nullptr;
  mg_grid_device(g, &dp, &sp);
  if ((cudaStream_t)sp != p->st || nx != p->d.nx || ny != p->d.ny || nz != p->d.nz)
    return set_error(MG_ERR_ARG, std::string(what) + ": grid and particles belong to different solvers");
  *data = (float*)dp;
  if (kind) *kind = k;
  return MG_OK;
}

int pdata_of(mg_particles p, mg_pdata d, int kind, const char* what) {
  if (!valid_pdata(d)) return set_error(MG_ERR_ARG, std::string(what) + ": invalid particle data");
  if (d->p != p) return set_error(MG_ERR_ARG, std::string(what) + ": particle data of another particle system");
  if (d->kind != kind) return set_error(MG_ERR_ARG, std::string(what) + ": wrong particle data type");
  return MG_OK;
}

}  // namespace

extern "C" int mg_grid_get_info(mg_grid g, int* nx, int* ny, int* nz, int* kind);
extern "C" int mg_grid_device(mg_grid g, void** data, void** stream);

extern "C" int mg_particles_create(mg_solver s, long long capacity, mg_particles* out) {
  if (!out) return set_error(MG_ERR_ARG, "mg_particles_create: null out");
  if (capacity < 0 || capacity > (1LL << 30))
    return set_error(MG_ERR_ARG, "mg_particles_create: capacity must be in [0, 2^30]");
  auto p = new mg_particles_s();
  if (solver_info(s, &p->d, &p->st)) {
    delete p;
    return MG_ERR_ARG;
  }
  p->s = s;
  p->cap = capacity;
  const long long c = std::max<long long>(capacity, 1);
  const long long tiles = tiles_of(c);
  const long long histN = 256 * tiles;
  bool ok = cudaMalloc(&p->x, c * 4) == cudaSuccess && cudaMalloc(&p->y, c * 4) == cudaSuccess &&
            cudaMalloc(&p->z, c * 4) == cudaSuccess && cudaMalloc(&p->flag, c * 4) == cudaSuccess &&
            cudaMalloc(&p->scratch, 10 * align256(c * 4)) == cudaSuccess && cudaMalloc(&p->hist, histN * 4) == cudaSuccess &&
            cudaMalloc(&p->sums, ((histN + kRsTile - 1) / kRsTile) * 4) == cudaSuccess &&
            cudaMalloc(&p->starts, (p->d.n + 1) * 4) == cudaSuccess && cudaMalloc(&p->stage, c * 16) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    free_parts(p);
    delete p;
    return set_error(MG_ERR_NOMEM, "BasicParticleSystem: out of device memory");
  }
  auto part = [&](int q) { return p->scratch + q * (align256(c * 4) / 4); };
  for (int q = 0; q < 2; q++) {
    p->keys[q] = part(q);
    p->vals[q] = part(2 + q);
  }
  for (int q = 0; q < 6; q++) p->sorted[q] = (float*)part(4 + q);
  {
    std::lock_guard<std::mutex> lk(g_partMu);
    g_parts.insert(p);
  }
  *out = p;
  return MG_OK;
}

extern "C" int mg_particles_destroy(mg_particles p) {
  if (!p) return MG_OK;
  {
    std::lock_guard<std::mutex> lk(g_partMu);
    if (!g_parts.count(p)) return set_error(MG_ERR_ARG, "mg_particles_destroy: invalid particle system");
    g_parts.erase(p);
    cudaStreamSynchronize(p->st);
    // its particle data goes with it
    for (auto it = g_pdata.begin(); it != g_pdata.end();) {
      if ((*it)->p != p) {
        ++it;
        continue;
      }
      for (float* b : (*it)->c)
        if (b) cudaFree(b);
      delete *it;
      it = g_pdata.erase(it);
    }
  }
  free_parts(p);
  delete p;
  return MG_OK;
}

extern "C" int mg_particles_upload(mg_particles p, const void* host, long long count) {
  if (!valid_parts(p)) return set_error(MG_ERR_ARG, "mg_particles_upload: invalid particle system");
  if (count < 0 || count > p->cap) return set_error(MG_ERR_ARG, "mg_particles_upload: count exceeds the capacity");
  if (count > 0 && !host) return set_error(MG_ERR_ARG, "mg_particles_upload: null host buffer");
  if (count > 0) {
    if (cudaMemcpyAsync(p->stage, host, (size_t)count * 16, cudaMemcpyHostToDevice, p->st) != cudaSuccess)
      return launch_status("mg_particles_upload");
    count_launch();
    k_parts_unpack<<<blocks_of(count), 256, 0, p->st>>>(count, (const float4*)p->stage, p->x, p->y, p->z, p->flag);
  }
  p->n = count;
  return launch_status("mg_particles_upload");
}

extern "C" int mg_particles_download(mg_particles p, void* host, long long count) {
  if (!valid_parts(p)) return set_error(MG_ERR_ARG, "mg_particles_download: invalid particle system");
  if (count != p->n) return set_error(MG_ERR_ARG, "mg_particles_download: count must equal the particle count");
  if (count == 0) return MG_OK;
  if (!host) return set_error(MG_ERR_ARG, "mg_particles_download: null host buffer");
  count_launch();
  k_parts_pack<<<blocks_of(count), 256, 0, p->st>>>(count, (float4*)p->stage, p->x, p->y, p->z, p->flag);
  if (cudaMemcpyAsync(host, p->stage, (size_t)count * 16, cudaMemcpyDeviceToHost, p->st) != cudaSuccess ||
      cudaStreamSynchronize(p->st) != cudaSuccess)
    return launch_status("mg_particles_download");
  return launch_status("mg_particles_download");
}

extern "C" int mg_particles_size(mg_particles p, long long* count) {
  if (!valid_parts(p) || !count) return set_error(MG_ERR_ARG, "mg_particles_size: invalid argument");
  *count = p->n;
  return MG_OK;
}

extern "C" int mg_pdata_create(mg_particles p, int kind, mg_pdata* out) {
  if (!out) return set_error(MG_ERR_ARG, "mg_pdata_create: null out");
  if (!valid_parts(p)) return set_error(MG_ERR_ARG, "mg_pdata_create: invalid particle system");
  if (kind != MG_REAL && kind != MG_VEC3 && kind != MG_INT)
    return set_error(MG_ERR_ARG, "mg_pdata_create: kind must be MG_REAL, MG_VEC3 or MG_INT");
  auto d = new mg_pdata_s();
  d->p = p;
  d->kind = kind;
  const long long c = std::max<long long>(p->cap, 1);
  const int comps = kind == MG_VEC3 ? 3 : 1;
  bool ok = true;
  for (int q = 0; q < comps && ok; q++) ok = cudaMalloc(&d->c[q], c * 4) == cudaSuccess;
  for (int q = 0; q < comps && ok; q++) ok = cudaMemsetAsync(d->c[q], 0, c * 4, p->st) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    for (float* b : d->c)
      if (b) cudaFree(b);
    delete d;
    return set_error(MG_ERR_NOMEM, "ParticleDataImpl: out of device memory");
  }
  {
    std::lock_guard<std::mutex> lk(g_partMu);
    g_pdata.insert(d);
  }
  *out = d;
  return MG_OK;
}

extern "C" int mg_pdata_destroy(mg_pdata d) {
  if (!d) return MG_OK;
  mg_particles p;
  {
    std::lock_guard<std::mutex> lk(g_partMu);
    if (!g_pdata.count(d)) return set_error(MG_ERR_ARG, "mg_pdata_destroy: invalid particle data");
    g_pdata.erase(d);
    p = g_parts.count(d->p) ? d->p : nullptr;
  }
  if (p) cudaStreamSynchronize(p->st);
  for (float* b : d->c)
    if (b) cudaFree(b);
  delete d;
  return MG_OK;
}

static int pdata_transfer(mg_pdata d, void* host, long long count, bool up) {
  const char* what = up ? "mg_pdata_upload" : "mg_pdata_download";
  if (!valid_pdata(d)) return set_error(MG_ERR_ARG, std::string(what) + ": invalid particle data");
  mg_particles p = d->p;
  if (count != p->n) return set_error(MG_ERR_ARG, std::string(what) + ": count must equal the particle count");
  if (count == 0) return MG_OK;
  if (!host) return set_error(MG_ERR_ARG, std::string(what) + ": null host buffer");
  if (d->kind != MG_VEC3) {
    const cudaError_t e = up ? cudaMemcpyAsync(d->c[0], host, (size_t)count * 4, cudaMemcpyHostToDevice, p->st)
                             : cudaMemcpyAsync(host, d->c[0], (size_t)count * 4, cudaMemcpyDeviceToHost, p->st);
    if (e != cudaSuccess) return launch_status(what);
  } else if (up) {
    if (cudaMemcpyAsync(p->stage, host, (size_t)count * 12, cudaMemcpyHostToDevice, p->st) != cudaSuccess)
      return launch_status(what);
    count_launch();
    k_vec_transpose<<<blocks_of(count), 256, 0, p->st>>>(count, (float*)p->stage, d->c[0], d->c[1], d->c[2], 0);
  } else {
    count_launch();
    k_vec_transpose<<<blocks_of(count), 256, 0, p->st>>>(count, (float*)p->stage, d->c[0], d->c[1], d->c[2], 1);
    if (cudaMemcpyAsync(host, p->stage, (size_t)count * 12, cudaMemcpyDeviceToHost, p->st) != cudaSuccess)
      return launch_status(what);
  }
  if (!up && cudaStreamSynchronize(p->st) != cudaSuccess) return launch_status(what);
  return launch_status(what);
}

extern "C" int mg_pdata_upload(mg_pdata d, const void* host, long long count) {
  return pdata_transfer(d, const_cast<void*>(host), count, true);
}
extern "C" int mg_pdata_download(mg_pdata d, void* host, long long count) {
  return pdata_transfer(d, host, count, false);
}

// ----------------------------------------------------------- the transfers
extern "C" int mg_map_parts_to_mac(mg_grid flags, mg_grid vel, mg_grid velOld, mg_particles parts, mg_pdata partVel,
                                   mg_grid weight, mg_pdata ptype, int exclude) {
  const char* what = "mapPartsToMAC";
  if (!valid_parts(parts)) return set_error(MG_ERR_ARG, "mapPartsToMAC: invalid particle system");
  float *f, *v, *vo, *w = nullptr;
  if (grid_of(parts, flags, 1u << MG_FLAGS, what, &f, nullptr) || grid_of(parts, vel, 1u << MG_MAC, what, &v, nullptr) ||
      grid_of(parts, velOld, 1u << MG_MAC, what, &vo, nullptr))
    return MG_ERR_ARG;
  if (weight && grid_of(parts, weight, (1u << MG_VEC3) | (1u << MG_MAC), what, &w, nullptr)) return MG_ERR_ARG;
  if (pdata_of(parts, partVel, MG_VEC3, what)) return MG_ERR_ARG;
  if (ptype && pdata_of(parts, ptype, MG_INT, what)) return MG_ERR_ARG;
  const Dims& d = parts->d;
  const PartView pv = view_of(parts, ptype, exclude);
  if (tile_lists(parts)) {
    Tiles s = parts->tiles;
    s.n = parts->n;
    for (int c = 0; c < 3; c++) s.v[c] = partVel->c[c];
    if (s.large) tile_mac<TileLarge>(parts, s, pv, v, vo, w);
    else tile_mac<TileSmall>(parts, s, pv, v, vo, w);
    return launch_status(what);
  }
  const dim3 b(32, 8, 1);
  for (int c = 0; c < 3; c++) {
    const unsigned* sorted = sort_stencil(parts, c, pv);
    const SortedParts sp = sorted_copy(parts, sorted, pv, partVel->c[c], nullptr, nullptr);
    count_launch();
    k_p2g_gather<1><<<grid3(d, b), b, 0, parts->st>>>(d, c, sp, sorted, parts->starts, v + c * d.n, nullptr, nullptr,
                                                      vo + c * d.n, w ? w + c * d.n : nullptr);
  }
  return launch_status(what);
}

extern "C" int mg_map_parts_to_grid(mg_grid flags, mg_grid target, mg_particles parts, mg_pdata source) {
  const char* what = "mapPartsToGrid";
  if (!valid_parts(parts)) return set_error(MG_ERR_ARG, "mapPartsToGrid: invalid particle system");
  float *f, *t;
  int kind = 0;
  if (grid_of(parts, flags, 1u << MG_FLAGS, what, &f, nullptr) ||
      grid_of(parts, target, (1u << MG_REAL) | (1u << MG_LEVELSET) | (1u << MG_VEC3) | (1u << MG_MAC), what, &t,
              &kind))
    return MG_ERR_ARG;
  const bool vec = kind == MG_VEC3 || kind == MG_MAC;
  if (pdata_of(parts, source, vec ? MG_VEC3 : MG_REAL, what)) return MG_ERR_ARG;
  const Dims& d = parts->d;
  const PartView pv = view_of(parts, nullptr, 0);
  const unsigned* sorted = sort_stencil(parts, -1, pv);
  const SortedParts sp = sorted_copy(parts, sorted, pv, source->c[0], vec ? source->c[1] : nullptr,
                                     vec ? source->c[2] : nullptr);
  const dim3 b(32, 8, 1);
  count_launch();
  if (vec)
    k_p2g_gather<3><<<grid3(d, b), b, 0, parts->st>>>(d, -1, sp, sorted, parts->starts, t, t + d.n, t + 2 * d.n,
                                                      nullptr, nullptr);
  else
    k_p2g_gather<1><<<grid3(d, b), b, 0, parts->st>>>(d, -1, sp, sorted, parts->starts, t, nullptr, nullptr, nullptr,
                                                      nullptr);
  return launch_status(what);
}

static int mac_to_parts(const char* what, mg_grid flags, mg_grid vel, mg_grid velOld, mg_particles parts,
                        mg_pdata partVel, float flipRatio, mg_pdata ptype, int exclude) {
  if (!valid_parts(parts)) return set_error(MG_ERR_ARG, std::string(what) + ": invalid particle system");
  float *f, *v, *vo = nullptr;
  if (grid_of(parts, flags, 1u << MG_FLAGS, what, &f, nullptr) || grid_of(parts, vel, 1u << MG_MAC, what, &v, nullptr))
    return MG_ERR_ARG;
  if (velOld && grid_of(parts, velOld, 1u << MG_MAC, what, &vo, nullptr)) return MG_ERR_ARG;
  if (pdata_of(parts, partVel, MG_VEC3, what)) return MG_ERR_ARG;
  if (ptype && pdata_of(parts, ptype, MG_INT, what)) return MG_ERR_ARG;
  const Dims& d = parts->d;
  if (parts->n == 0) return MG_OK;
  const CMac cv{v, v + d.n, v + 2 * d.n};
  const CMac co = vo ? CMac{vo, vo + d.n, vo + 2 * d.n} : CMac{nullptr, nullptr, nullptr};
  count_launch();
  const auto k = parts->n < kFewParticles ? k_mac_to_parts<false> : k_mac_to_parts<true>;
  k<<<blocks_of(parts->n), 256, 0, parts->st>>>(d, view_of(parts, ptype, exclude), parts->n, cv, co, flipRatio,
                                                partVel->c[0], partVel->c[1], partVel->c[2]);
  return launch_status(what);
}

extern "C" int mg_map_mac_to_parts(mg_grid flags, mg_grid vel, mg_particles parts, mg_pdata partVel, mg_pdata ptype,
                                   int exclude) {
  return mac_to_parts("mapMACToParts", flags, vel, nullptr, parts, partVel, 0.f, ptype, exclude);
}

extern "C" int mg_flip_velocity_update(mg_grid flags, mg_grid vel, mg_grid velOld, mg_particles parts,
                                       mg_pdata partVel, float flipRatio, mg_pdata ptype, int exclude) {
  if (!velOld) return set_error(MG_ERR_ARG, "flipVelocityUpdate: null velOld");
  return mac_to_parts("flipVelocityUpdate", flags, vel, velOld, parts, partVel, flipRatio, ptype, exclude);
}

extern "C" int mg_map_grid_to_parts(mg_grid source, mg_particles parts, mg_pdata target) {
  const char* what = "mapGridToParts";
  if (!valid_parts(parts)) return set_error(MG_ERR_ARG, "mapGridToParts: invalid particle system");
  float* g;
  int kind = 0;
  if (grid_of(parts, source, (1u << MG_REAL) | (1u << MG_LEVELSET) | (1u << MG_VEC3) | (1u << MG_MAC), what, &g,
              &kind))
    return MG_ERR_ARG;
  const bool vec = kind == MG_VEC3 || kind == MG_MAC;
  if (pdata_of(parts, target, vec ? MG_VEC3 : MG_REAL, what)) return MG_ERR_ARG;
  if (parts->n == 0) return MG_OK;
  const Dims& d = parts->d;
  count_launch();
  k_grid_to_parts<<<blocks_of(parts->n), 256, 0, parts->st>>>(
      d, view_of(parts, nullptr, 0), parts->n, g, vec ? g + d.n : nullptr, vec ? g + 2 * d.n : nullptr, target->c[0],
      target->c[1], target->c[2]);
  return launch_status(what);
}

// mg_solver_destroy: the solver's particle systems and their data go with it
void mgpu::particles_release(mg_solver s) {
  std::lock_guard<std::mutex> lk(g_partMu);
  for (auto it = g_pdata.begin(); it != g_pdata.end();) {
    mg_pdata d = *it;
    if (s && d->p->s != s) {
      ++it;
      continue;
    }
    for (float* b : d->c)
      if (b) cudaFree(b);
    delete d;
    it = g_pdata.erase(it);
  }
  for (auto it = g_parts.begin(); it != g_parts.end();) {
    mg_particles p = *it;
    if (s && p->s != s) {
      ++it;
      continue;
    }
    free_parts(p);
    delete p;
    it = g_parts.erase(it);
  }
}
