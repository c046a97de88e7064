// MIC(0) preconditioner sweeps as warp wavefronts inside thread-block clusters.
//
// The reference factors and applies the modified incomplete Cholesky
// preconditioner with lexicographic loops (conjugategrad.cpp:66-97,
// 135-160): cell (x,y,z) needs the finished values of (x-1,y,z), (x,y-1,z)
// and (x,y,z-1).  Any order that respects those dependencies reproduces the
// serial result bit for bit.  What bounds a sweep is its critical path of
// nx + ny + nz dependent cells, so everything here shortens one step of it:
//
//  * A warp owns a bundle of 8 x 8 lines (y, z) over the whole x range; lane
//    (j, q) holds the lines z = 2q and 2q + 1 of row y = j, and at level L
//    works on x = L - j - z in both.  The x-neighbours are the lane's own last
//    values, the z-neighbour of the odd line its own even line, the other
//    neighbours three shuffles: no barrier and no memory between the levels.
//  * Values cross from warp to warp as single 32-bit words in the consumer's
//    shared memory, one slot for every level, empty (a NaN pattern that no
//    arithmetic produces) until the producer stores the value: the word is
//    its own flag.  The consumer looks one level ahead and waits only when
//    the word is not there.  Slots are never reused within a sweep, so there
//    is no flow control.
//  * A CTA holds 2 x 2 such warps (16 x 16 lines, one warp per scheduler) and
//    a cluster all CTAs of one or more z-blocks (up to 16 CTAs), so a word
//    travels through distributed shared memory where it leaves its CTA.
//    Between clusters, only in z, it goes through global memory: the last
//    warp polls the words for the warps of its CTA and empties them again for
//    the next sweep.
//  * The diagonal, the stencil bits, the residual and z are kept in level
//    order, bundle by bundle, so eight levels of a bundle are one contiguous
//    piece that a single bulk copy brings in or takes out.  A copying warp per
//    bundle keeps three pieces on their way and forms the dot product; the
//    computing warp touches global memory only through its words.  The other
//    kernels of an iteration turn between grid and level order (k_lvl_*).
//
// Clusters take their work from a ticket in dependency order, so a cluster
// waits only for clusters that run or have finished.  The backward sweep runs
// the same levels downward.
//
// Eight levels take 1000 cycles forward and 1070 back where their words are
// there, 1200 and 1300 where a pair of levels waits for one (four chunks in
// five); between chunks pass 280 and 410, most of it the wait for the copy's
// barrier.  A bundle runs 1900 to 2100 cycles behind the one that feeds it (seven
// levels of skew and the words' way), 5600 to 6900 where that is in another
// cluster.  At 128^3: 18 chunks 12 us, 27 hops 26 us and 3 between clusters 8.5 us
// make the 46 us of a forward sweep; a backward one takes 52, at 64^3 they take 21
// and 22.  Whole solves against the tile sweeps of micflow.cu: 64^3 smoke (50
// iterations) 9.3 -> 3.5 ms, 128^3 dam break (53) 21.3 -> 7.7 ms.  Grids with more
// than 256 rows or more than about 400 cells along x do not fit and keep the tiles.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cstring>

#include "mg_common.cuh"
#include "mg_kernels.h"
#include "mg_reduce.cuh"
#include "mg_tma.cuh"

namespace cg = cooperative_groups;

namespace mgpu {

namespace {

constexpr int kUY = 8, kUZ = 8;            // lines of a bundle
constexpr int kBlk = 16;                   // lines of a CTA per axis
constexpr int kMcWarps = 4;                // bundles of a CTA: 2 x 2
constexpr int kMcThreads = 32 * (2 * kMcWarps + 1);  // a computing and a copying warp each; one between clusters
constexpr int kCH = 8;                     // levels per chunk
constexpr int kStages = 4;                 // chunks in shared memory
constexpr int kSkew = kUY + kUZ - 2;       // levels a warp needs beyond nx
constexpr int kVecWords = 64 * kCH, kBitWords = 32 * kCH;  // a chunk of a vector or P, and of the stencil bits
constexpr int kPad = 8;                    // levels of slack before and after a warp's slots
constexpr unsigned kVoid = 0xffffffffu;   // a NaN that arithmetic never yields
constexpr int kMcMaxSmem = 220 * 1024;

// bits of a cell in level order
constexpr unsigned kLX = 1, kLY = 2, kLZ = 4, kFl = 8, kHX = 16, kHY = 32, kHZ = 64;

struct McArgs {
  MicClusterScene one;             // the scene of a single-scene launch
  const MicClusterScene* scenes;   // batched launch: the scene table
  const int2* jobs;                // batched: (scene, first z-block) in dependency order
  int njobs;
  unsigned* counter;               // ticket, back at 0 after every launch
  int* error;
  int* ndone;                      // batched: finished scenes
  long long waitNs;
  int nlpMax;                      // levels the shared memory is laid out for
  int init;                        // backward for doInit: sigma instead of beta
  int stall;                       // failure-path tests: 1 publish nothing, 2 fetch nothing
};

// words of this CTA's shared memory
__device__ __forceinline__ unsigned ld_face(unsigned addr) {
  unsigned v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 ld_face2(unsigned addr) {
  uint2 v;
  asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
// words into the cluster's shared memory or into global memory; predicated
// rather than branched around
__device__ __forceinline__ void st_face(unsigned* p, unsigned v, unsigned on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.volatile.u32 [%0], %1;\n\t}" ::"l"(p), "r"(v), "r"(on));
}
__device__ __forceinline__ void st_face2(unsigned* p, unsigned v0, unsigned v1, unsigned on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.volatile.v2.u32 [%0], {%1, %2};\n\t}" ::"l"(p), "r"(v0),
               "r"(v1), "r"(on));
}
__device__ __forceinline__ unsigned ld_glob(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_glob(unsigned* p, unsigned v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A wait has lasted too long: the sweep is lost.  That ends the CG (done), so that
// the solve's later launches return at once and the host reports the timeout.
__device__ __noinline__ void give_up(int* error, CgScalars* sc) {
  if (atomicExch(error, 7) == 0) {
    sc->status = 3;
    sc->done = 1;
  }
}

// wait for a phase of an mbarrier, with pauses of `pause` ns and the timer
// read only now and then: the warps that compute share the SM's pipes.  When
// the limit is over it is reported, and once more waited for as long (a copy
// must not arrive in shared memory that is no longer this CTA's); after that a
// thread's other waits are short.
__device__ __forceinline__ void wait_bar(uint64_t* bar, uint32_t parity, long long& limitNs, unsigned pause, int* error,
                                         CgScalars* sc) {
  unsigned long long t0 = 0ull;
  bool told = false;
  for (unsigned n = 0; !mbar_try(bar, parity); n++) {
    if (pause) __nanosleep(pause);
    if ((n & 1023u) == 0u) {
      if (n == 0u) t0 = gtimer();
      else if (gtimer() - t0 > (unsigned long long)limitNs) {
        if (told) {
          limitNs = 1000000LL;
          return;
        }
        give_up(error, sc);
        told = true;
        t0 = gtimer();
      }
    }
  }
}

// a piece of shared memory to global memory, in the thread's bulk group
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// true when a wait that began at t0 is to be given up: its time is over, or
// another wait has given up
__device__ __noinline__ bool expired(unsigned long long t0, long long limit, int* error, CgScalars* sc) {
  if (*((volatile int*)error) != 0) return true;
  if (gtimer() - t0 <= (unsigned long long)limit) return false;
  give_up(error, sc);
  return true;
}

}  // namespace

// One cell: its vector value (or diagonal) tv, P, stencil bits cw and the
// three upwind values -> the value it passes on, and the result in out.
// REG: every fluid cell of the chunk is linked exactly to its fluid
// neighbours, so the others pass on a zero and adding it stands for the test
// of the link; P is zero outside the fluid only.
template <int MODE, bool REG>
__device__ __forceinline__ float mic_cell(float tv, float p, unsigned cw, float vx, float vy, float vz, float& out) {
  if (MODE == 0) {
    // InitPreconditionModifiedIncompCholesky2 (conjugategrad.cpp:66-97)
    float pv = 0.f;
    if (cw & kFl) {
      float ev = tv;
      if (cw & kLX) ev = ev - vx * vx;
      if (cw & kLY) ev = ev - vy * vy;
      if (cw & kLZ) ev = ev - vz * vz;
      const float k1 = (float)((cw >> 7) & 3u), k2 = (float)((cw >> 9) & 3u), k3 = (float)((cw >> 11) & 3u);
      const float S3 = (k1 * (vx * vx) + k2 * (vy * vy)) + k3 * (vz * vz);
      ev = fmaf(-0.97f, S3, ev);  // e -= tau*(...): double in the reference, one rounding
      if (ev < 0.25f * tv) ev = tv;
      pv = 1.f / sqrtf(ev);
    }
    out = pv;
    return pv;
  }
  const bool fluid = REG ? p != 0.f : (cw & kFl) != 0u;
  if (MODE == 1) {
    // forward substitution (conjugategrad.cpp:141-148); neighbours pass on
    // z*P, the product the reference forms
    float t = tv + vx;
    if (!REG) t = (cw & kLX) ? t : tv;
    const float ty = t + vy;
    t = REG || (cw & kLY) ? ty : t;
    const float tz = t + vz;
    t = REG || (cw & kLZ) ? tz : t;
    out = fluid ? p * t : 0.f;
    return out * p;
  }
  // backward substitution (conjugategrad.cpp:150-159)
  float t = tv + vx * p;
  if (!REG) t = (cw & kHX) ? t : tv;
  const float ty = t + vy * p;
  t = REG || (cw & kHY) ? ty : t;
  const float tz = t + vz * p;
  t = REG || (cw & kHZ) ? tz : t;
  out = fluid ? p * t : 0.f;
  return out;
}

// What a computing warp carries from level to level: its last values in the
// even and odd line, and the face words of the coming two levels (missing: one
// of them has not arrived).
struct McState {
  float pa, pb;
  uint2 y0, y1;
  unsigned z0, z1;
  bool missing;
};
__device__ __forceinline__ bool is_void(const McState& s) {
  return s.y0.x == kVoid || s.y0.y == kVoid || s.z0 == kVoid || s.y1.x == kVoid || s.y1.y == kVoid || s.z1 == kVoid;
}
// the words of the levels i and i + step into s
__device__ __forceinline__ void ld_words(McState& s, unsigned adY, unsigned adZ, int i, int step) {
  s.y0 = ld_face2(adY + 32 * i);
  s.z0 = ld_face(adZ + 32 * i);
  s.y1 = ld_face2(adY + 32 * (i + step));
  s.z1 = ld_face(adZ + 32 * (i + step));
}

constexpr int kUnroll = 4;
// The eight levels of a chunk in one warp: vec the chunk's vector (in: r or z,
// out: z or P), pc its P or diagonal, cc its stencil bits, all at this lane.
// Whether the words have come is asked for two levels at a time: the branch
// on it costs 37 cycles, the arithmetic of a level 63.
template <int MODE, bool REG, class Overdue>
__device__ __forceinline__ void mic_levels(McState& s, bool inY, bool inZ, unsigned adY, unsigned adZ, unsigned outY,
                                           unsigned outZ, unsigned* puY, unsigned* puZ, int strideZ, float2* vec,
                                           const float2* pc, const unsigned* cc, bool readP, Overdue& overdue) {
  constexpr bool kBack = MODE == 2;
  constexpr int kSgn = kBack ? -1 : 1;
  constexpr unsigned kAll = 0xffffffffu;
  // upwind values from other lanes: y in both lines, z of the line whose
  // upwind z-neighbour is in another lane; asked for before the results of
  // the level are stored
  float ya, yb, zo;
  auto across = [&]() {
    ya = kBack ? __shfl_down_sync(kAll, s.pa, 1) : __shfl_up_sync(kAll, s.pa, 1);
    yb = kBack ? __shfl_down_sync(kAll, s.pb, 1) : __shfl_up_sync(kAll, s.pb, 1);
    zo = kBack ? __shfl_down_sync(kAll, s.pa, 8) : __shfl_up_sync(kAll, s.pb, 8);
  };
  if (kBack) {  // from the chunk's last level down
    adY += 32 * (kCH - 1);
    adZ += 32 * (kCH - 1);
    puY += 8 * (kCH - 1);
    puZ += (long long)strideZ * (kCH - 1);
    vec += 32 * (kCH - 1);
    pc += 32 * (kCH - 1);
    cc += 32 * (kCH - 1);
  }
  const long long stepZ = kSgn * (long long)strideZ;
  // (the value read ahead at the chunk's end is not used)
  float2 tn = MODE ? *vec : make_float2(0.f, 0.f), pn = readP ? *pc : make_float2(0.f, 0.f);
  across();
#pragma unroll kUnroll
  for (int pr = 0; pr < kCH / 2; pr++) {
    if (s.missing) {
      unsigned n = 0, some;
      unsigned long long t0 = 0ull;
      do {
        ld_words(s, adY, adZ, 0, kSgn);
        some = is_void(s);
        if (overdue(n, t0)) {
          s.y0 = s.y1 = make_uint2(0u, 0u);
          s.z0 = s.z1 = some = 0u;
        }
      } while (__any_sync(kAll, some));
    }
#pragma unroll
    for (int second = 0; second < 2; second++) {
      const int i = second ? kSgn : 0;
      const unsigned cw = REG ? 0u : cc[32 * i];
      const float2 tv = tn, p = pn;
      ya = inY ? __uint_as_float(second ? s.y1.x : s.y0.x) : ya;
      yb = inY ? __uint_as_float(second ? s.y1.y : s.y0.y) : yb;
      zo = inZ ? __uint_as_float(second ? s.z1 : s.z0) : zo;
      if (second) ld_words(s, adY, adZ, 2 * kSgn, kSgn);
      if (MODE) tn = vec[32 * (i + kSgn)];
      if (readP) pn = pc[32 * (i + kSgn)];
      const unsigned ca = cw & 0xffffu, cb = cw >> 16;
      const float da = MODE ? tv.x : readP ? p.x : (float)(ca >> 13), db = MODE ? tv.y : readP ? p.y : (float)(cb >> 13);
      float2 o;
      const float na = mic_cell<MODE, REG>(da, p.x, ca, s.pa, ya, kBack ? s.pb : zo, o.x);
      s.pb = mic_cell<MODE, REG>(db, p.y, cb, s.pb, yb, kBack ? zo : s.pa, o.y);
      s.pa = na;
      if (second) s.missing = __any_sync(kAll, is_void(s));
      across();
      // arithmetic's only NaN is 0x7fffffff, never kVoid
      st_face2(puY + 8 * i, __float_as_uint(s.pa), __float_as_uint(s.pb), outY);
      st_face(second ? puZ + stepZ : puZ, __float_as_uint(kBack ? s.pa : s.pb), outZ);
      vec[32 * i] = o;
    }
    adY += 64 * kSgn;
    adZ += 64 * kSgn;
    puY += 16 * kSgn;
    puZ += 2 * stepZ;
    vec += 64 * kSgn;
    pc += 64 * kSgn;
    cc += 64 * kSgn;
  }
}

// MODE 0: factor (P).  MODE 1: forward substitution r -> z.  MODE 2: backward
// substitution z -> z, dot(z, r), and from it beta (or sigma for doInit).
template <int MODE>
__global__ void __launch_bounds__(kMcThreads, 1) k_mic_cluster(McArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned* const s_face = reinterpret_cast<unsigned*>(smem);
  __shared__ int2 s_job;
  __shared__ double s_red[kMcWarps];
  __shared__ __align__(8) uint64_t s_full[kMcWarps][kStages];  // the stage's chunk has arrived
  __shared__ __align__(8) uint64_t s_done[kMcWarps][kStages];  // ... has been computed
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  constexpr bool kBack = MODE == 2;

  __shared__ __align__(16) unsigned s_zero[8 * (kCH + 4)];  // what lanes that take nothing from a neighbour look at
  for (int q = tid; q < 4 * kMcWarps * (a.nlpMax + 2 * kPad); q += kMcThreads)
    reinterpret_cast<uint4*>(s_face)[q] = make_uint4(kVoid, kVoid, kVoid, kVoid);
  for (int q = tid; q < 8 * (kCH + 4); q += kMcThreads) s_zero[q] = 0u;
  if (tid < kMcWarps * kStages) {
    mbar_init(&s_full[0][0] + tid, 1);
    mbar_init(&s_done[0][0] + tid, 32);
    mbar_fence_init();
  }
  pass_started();
  pass_wait();
  if (rank == 0 && tid == 0) {
    const int first = a.scenes ? 0 : *((volatile const int*)&a.one.sc->done);  // (beside the ticket's round trip)
    const int t = (int)atomicInc(a.counter, (unsigned)a.njobs - 1u);           // wraps to 0 with the last ticket
    const int q = kBack ? a.njobs - 1 - t : t;
    const int2 job = a.jobs ? a.jobs[q] : make_int2(0, q * a.one.zper);
    const int done = a.scenes ? *((volatile const int*)&a.scenes[job.x].sc->done) : first;
    s_job = make_int2(done ? -1 : job.x, job.y);  // done is read once: the same for the whole cluster
  }
  cl.sync();  // every CTA's slots are empty before a neighbour stores into them
  const int2 job = *cl.map_shared_rank(&s_job, 0);
  const int scene = job.x, zb0 = job.y;
  if (scene < 0) {
    cl.sync();  // rank 0 stays until everyone has read its job
    return;
  }
  const MicClusterScene& S = a.scenes ? a.scenes[scene] : a.one;
  const int nx = S.d.nx, ny = S.d.ny, nz = S.d.nz;
  const int nby = S.nby, zbn = min(S.zper, S.nbz - zb0), nl = nx + kSkew, nlp = S.nlp;
  const bool active = rank < nby * zbn;
  const int by = rank % nby, cz = rank / nby, bz = zb0 + cz;
  const int nyp = nby * kBlk;
  CgScalars* const sc = S.sc;
  TSum acc;

  constexpr int kSgn = kBack ? -1 : 1;
  const int u = w & (kMcWarps - 1), uy = u & 1, uz = u >> 1;  // the line bundle of this warp
  const int y0 = by * kBlk + uy * kUY, z0 = bz * kBlk + uz * kUZ;
  const bool bundle = active && w < 2 * kMcWarps && y0 < ny && z0 < nz;
  const long long unit = ((long long)bz * nby + by) * kMcWarps + u;
  const int nch = nlp / kCH;
  const bool readP = MODE != 0 || S.A0f != nullptr;
  // stages of this bundle: the vector (in, and the result in its place), P,
  // the residual for the dot product (backward), the stencil bits
  constexpr int kStageWords = (kBack ? 3 : 2) * kVecWords + kBitWords;
  float* const stages = reinterpret_cast<float*>(s_face + 16 * kMcWarps * (a.nlpMax + 2 * kPad)) + u * kStages * kStageWords;
  auto s_vec = [&](int st) { return stages + st * kStageWords; };
  auto s_p = [&](int st) { return stages + st * kStageWords + kVecWords; };
  auto s_bits = [&](int st) { return reinterpret_cast<unsigned*>(stages + st * kStageWords + 2 * kVecWords); };
  auto s_r = [&](int st) { return stages + st * kStageWords + 2 * kVecWords + kBitWords; };
  long long limit = 2 * a.waitNs + 1000000000LL;  // beyond what a computing warp's own waits can add up to
  // levels that a neighbour's word exists for: those with a cell inside the grid
  const int fLo = kBack ? 7 : 0, fHi = kBack ? nl : nx + 7;
  // gives up on behalf of the whole sweep once a wait has lasted too long
  auto overdue = [&](unsigned& n, unsigned long long& t0) {
    if ((++n & 255u) != 0u) return false;
    if (n == 256u) t0 = gtimer();
    return expired(t0, a.waitNs, a.error, sc);
  };

  if (bundle && w < kMcWarps) {
    // ---- the computing warp
    {
      const int ly = lane & (kUY - 1), lq = lane >> 3;
      const int gy = by * 2 + uy, gz = bz * 2 + uz;
      const int ngy = (ny + kUY - 1) / kUY, ngz = (nz + kUZ - 1) / kUZ;
      // slots of a warp: level-major, 8 words for the y face, then 8 for the z face
      const int wslots = 8 * (nlp + 2 * kPad);
      auto slotsY = [&](int wt) { return s_face + wt * 2 * wslots + 8 * kPad; };
      auto slotsZ = [&](int wt) { return s_face + (wt * 2 + 1) * wslots + 8 * kPad; };
      unsigned* const faceY = slotsY(w);
      unsigned* const faceZ = slotsZ(w);
      const bool upY = kBack ? gy + 1 < ngy : gy > 0, upZ = kBack ? gz + 1 < ngz : gz > 0;
      const bool dnY = kBack ? gy > 0 : gy + 1 < ngy, dnZ = kBack ? gz > 0 : gz + 1 < ngz;
      const unsigned char* const rp = S.regular + unit * nch;
      const int rLo = lane < nch && rp[lane], rHi = lane + 32 < nch && rp[lane + 32];
      // only levels with a cell inside the grid wait for a word
      for (int q = lane; q < 8 * (fLo + kPad); q += 32) faceY[q - 8 * kPad] = faceZ[q - 8 * kPad] = 0u;
      for (int q = 8 * fHi + lane; q < 8 * (nlp + kPad); q += 32) faceY[q] = faceZ[q] = 0u;
      // lanes whose neighbour is another warp's, or the outside (which counts as 0)
      const bool inY = ly == (kBack ? kUY - 1 : 0), inZ = lq == (kBack ? 3 : 0);
      const unsigned outY = dnY && a.stall != 1 && ly == (kBack ? 0 : kUY - 1);
      const unsigned outZ = dnZ && a.stall != 1 && lq == (kBack ? 0 : 3);
      // the next warps keep the word of this warp's level L at pub + stride * L
      // (it is their level L -+ 7; levels without a cell end up in the slack
      // or among words nobody reads)
      auto at_rank = [&](unsigned* p, int r) { return r == rank ? p : cl.map_shared_rank(p, r); };
      unsigned *pubY = s_face, *pubZ = s_face;
      int strideZ = 8;
      if (dnY) {
        const int g = gy + kSgn;
        pubY = at_rank(slotsY((g & 1) + 2 * uz), cz * nby + (g >> 1)) + 2 * lq - 8 * kSgn * 7;
      }
      if (dnZ) {
        const int g = gz + kSgn, cz2 = (g >> 1) - zb0;
        if (cz2 >= 0 && cz2 < zbn) {
          pubZ = at_rank(slotsZ(uy + 2 * (g & 1)), cz2 * nby + by) + ly - 8 * kSgn * 7;
        } else {
          const int b = zb0 / S.zper - (kBack ? 1 : 0);  // the boundary below or above this cluster
          strideZ = nyp;
          pubZ = S.gface + ((long long)(2 * b + (kBack ? 1 : 0)) * (nlp + 2 * kPad) + kPad - kSgn * 7) * nyp + y0 + ly;
        }
      }
      const unsigned long long regular = (unsigned long long)__ballot_sync(0xffffffffu, rLo) |
                                         (unsigned long long)__ballot_sync(0xffffffffu, rHi) << 32;
      __syncwarp();  // the zeros above, for every lane
      McState ms;
      ms.pa = ms.pb = 0.f;
      const int first = kBack ? nlp - 1 : 0;
      const bool fromY = inY && upY, fromZ = inZ && upZ;
      const unsigned baseY = smem_addr(fromY ? faceY + 2 * lq : s_zero + 16), baseZ = smem_addr(fromZ ? faceZ + ly : s_zero + 16);
      ld_words(ms, fromY ? baseY + 32 * first : baseY, fromZ ? baseZ + 32 * first : baseZ, 0, kSgn);
      ms.missing = __any_sync(0xffffffffu, is_void(ms));
      for (int c = 0; c < nch; c++) {
        const int ch = kBack ? nch - 1 - c : c, L0 = ch * kCH, st = c % kStages;
        // slots of level L0 (lanes that take nothing: zeros), and of the next warps
        const unsigned adY = fromY ? baseY + 32 * L0 : baseY, adZ = fromZ ? baseZ + 32 * L0 : baseZ;
        unsigned* const puY = pubY + 8 * L0;
        unsigned* const puZ = pubZ + (long long)strideZ * L0;
        float2* const vec = reinterpret_cast<float2*>(s_vec(st)) + lane;
        const float2* const pc = reinterpret_cast<const float2*>(s_p(st)) + lane;
        const unsigned* const cc = s_bits(st) + lane;
        wait_bar(&s_full[u][st], (c / kStages) & 1, limit, 0, a.error, sc);
        if (MODE != 0 && (regular >> ch & 1ull))
          mic_levels<MODE, true>(ms, inY, inZ, adY, adZ, outY, outZ, puY, puZ, strideZ, vec, pc, cc, readP, overdue);
        else
          mic_levels<MODE, false>(ms, inY, inZ, adY, adZ, outY, outZ, puY, puZ, strideZ, vec, pc, cc, readP, overdue);
        mbar_arrive(&s_done[u][st]);
      }
    }
  } else if (bundle) {
    // ---- the copying warp: chunks in, kStages ahead, and their results out
    float* const out = (MODE == 0 ? S.P : S.z) + unit * nlp * 64;
    auto fetch = [&](int c) {
      if (a.stall == 2) return;
      const int st = c % kStages;
      const long long at = (unit * nlp + (long long)(kBack ? nch - 1 - c : c) * kCH) * 32;
      const uint32_t vb = kVecWords * 4, bb = kBitWords * 4;
      mbar_arrive_expect(&s_full[u][st], (MODE ? vb : 0) + (readP ? vb : 0) + (kBack ? vb : 0) + bb);
      if (MODE) bulk_g2s(s_vec(st), (kBack ? S.z : S.r) + 2 * at, vb, &s_full[u][st]);
      if (readP) bulk_g2s(s_p(st), S.P + 2 * at, vb, &s_full[u][st]);
      if (kBack) bulk_g2s(s_r(st), S.r + 2 * at, vb, &s_full[u][st]);
      bulk_g2s(s_bits(st), S.cw + at, bb, &s_full[u][st]);
    };
    if (lane == 0)
      for (int c = 0; c < min(kStages, nch); c++) fetch(c);
    for (int c = 0; c < nch; c++) {
      const int st = c % kStages;
      wait_bar(&s_done[u][st], (c / kStages) & 1, limit, 100, a.error, sc);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the results, for the copy engine
      if (lane == 0) bulk_s2g(out + (long long)(kBack ? nch - 1 - c : c) * kVecWords, s_vec(st), kVecWords * 4);
      if (kBack) {
        const float2* z = reinterpret_cast<const float2*>(s_vec(st)) + lane;
        const float2* r = reinterpret_cast<const float2*>(s_r(st)) + lane;
#pragma unroll
        for (int i = 0; i < kCH; i++) {
          const float2 zv = z[32 * i], rv = r[32 * i];
          acc.add(zv.x * rv.x);
          acc.add(zv.y * rv.y);
        }
        __syncwarp();  // before the stage is filled again
      }
      if (lane == 0 && c + kStages < nch) {
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        fetch(c + kStages);
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else if (active && w == 2 * kMcWarps && (kBack ? cz == zbn - 1 && bz + 1 < S.nbz : cz == 0 && bz > 0)) {
    // ---- the last warp of a CTA at the cluster's upstream boundary: words from
    // global memory into the slots of the CTA's two boundary warps, sixteen
    // levels at a time (lane: line y, every other level)
    const int y = lane & (kBlk - 1), hl = lane >> 4;
    const int wt = (y >> 3) + 2 * (kBack ? 1 : 0);
    unsigned* const dst = s_face + (wt * 2 + 1) * 8 * (nlp + 2 * kPad) + 8 * kPad + (y & (kUY - 1));
    unsigned* const src = S.gface + ((long long)(2 * (zb0 / S.zper - (kBack ? 0 : 1)) + (kBack ? 1 : 0)) * (nlp + 2 * kPad) + kPad) * nyp +
                          by * kBlk + y;
    const bool mine = by * kBlk + (y & ~(kUY - 1)) < ny;                // the boundary warp exists
    for (int b = 0; b < nlp; b += 16) {
      const int B = kBack ? nlp - 16 - b : b;
      unsigned pend = 0u;
      unsigned v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int L = B + 2 * q + hl;
        if (mine && L >= fLo && L < fHi) pend |= 1u << q;
      }
      unsigned long long t0 = 0ull;
      unsigned n = 0;
      while (__any_sync(0xffffffffu, pend != 0u)) {
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (pend & (1u << q)) v[q] = ld_glob(src + (long long)(B + 2 * q + hl) * nyp);
#pragma unroll
        for (int q = 0; q < 8; q++)
          if ((pend & (1u << q)) && v[q] != kVoid) {
            const int L = B + 2 * q + hl;
            st_face(dst + 8 * L, v[q], 1u);
            st_glob(src + (long long)L * nyp, kVoid);
            pend &= ~(1u << q);
          }
        if ((++n & 63u) == 0u) {
          if (n == 64u) t0 = gtimer();
          if (expired(t0, a.waitNs, a.error, sc)) pend = 0u;
        }
      }
    }
  }
  if (kBack && active) {
    // dot(z, r): the CTA's share, then the scene's last CTA adds the shares
    // in block order and forms beta (GridCg::iterate) or sigma (doInit)
    double t = acc.value();
    t = warp_sum(t);
    if (w >= kMcWarps && w < 2 * kMcWarps && lane == 0) s_red[u] = t;
    __syncthreads();
    if (tid == 0) {
      double s = 0.;
      for (int q = 0; q < kMcWarps; q++) s += s_red[q];
      S.part[by + nby * bz] = s;
    }
    if (last_block(&sc->counters[6], (unsigned)(nby * S.nbz))) {
      const double s = sum_partials(S.part, nby * S.nbz);
      if (tid == 0) {
        const float sigmaNew = (float)s;
        if (!a.init) {
          sc->beta = sigmaNew / sc->sigma;
          if (!(sc->resNorm < 1e35f)) {
            sc->status = 2;
            sc->done = 1;
            if (a.ndone) atomicAdd(a.ndone, 1);
          }
        }
        sc->sigma = sigmaNew;
      }
    }
  }
  cl.sync();  // nobody leaves while a neighbour may still store into its slots
}

// Stencil bits in level order (and, with a ghost-fluid diagonal, its values
// in P's place for the factorisation): 32 levels of a block's four bundles,
// two warps each.
__global__ void __launch_bounds__(64 * kMcWarps) k_mic_order(McArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  typedef unsigned short CodeRow[34];
  typedef float DiagRow[33];
  CodeRow* const s_c = reinterpret_cast<CodeRow*>(smem);                              // [bundle * 64 + line]
  DiagRow* const s_a = reinterpret_cast<DiagRow*>(smem + sizeof(CodeRow) * 64 * kMcWarps);
  __shared__ unsigned s_reg[2 * kMcWarps];
  const MicClusterScene& S = a.scenes ? a.scenes[blockIdx.z] : a.one;
  const int nx = S.d.nx, ny = S.d.ny, nz = S.d.nz;
  const int b = blockIdx.x, L0 = blockIdx.y * 32;
  if (b >= S.nby * S.nbz || L0 >= S.nlp) return;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, u = w >> 1, hz = w & 1;
  const int y0 = (b % S.nby) * kBlk + (u & 1) * kUY, z0 = (b / S.nby) * kBlk + (u >> 1) * kUZ;
  bool reg = true;
  for (int q = 0; q < 32; q++) {
    const int yl = q & (kUY - 1), zl = 4 * hz + (q >> 3), y = y0 + yl, z = z0 + zl, x = L0 + lane - yl - zl;
    unsigned o = 0u;
    float av = 0.f;
    if (x >= 0 && x < nx && y < ny && z < nz) {
      const long long g = ix(S.d, x, y, z);
      const int c = S.code[g];
      if (c & kCodeFluid) {
        o = kFl | ((c >> 4) & 7) | (((c >> 7) & 7) << 4) | ((unsigned)(c & 7) << 13);
        const int cxl = x > 0 ? S.code[g - 1] : 0, cxh = x < nx - 1 ? S.code[g + 1] : 0;
        const int cyl = y > 0 ? S.code[g - S.d.sy] : 0, cyh = y < ny - 1 ? S.code[g + S.d.sy] : 0;
        const int czl = z > 0 ? S.code[g - S.d.sz] : 0, czh = z < nz - 1 ? S.code[g + S.d.sz] : 0;
        if (c & kLowX) o |= (unsigned)(((cxl & kHighY) ? 1 : 0) + ((cxl & kHighZ) ? 1 : 0)) << 7;
        if (c & kLowY) o |= (unsigned)(((cyl & kHighX) ? 1 : 0) + ((cyl & kHighZ) ? 1 : 0)) << 9;
        if (c & kLowZ) o |= (unsigned)(((czl & kHighX) ? 1 : 0) + ((czl & kHighY) ? 1 : 0)) << 11;
        // regular: linked to the fluid neighbours and no others, and a
        // diagonal from which P comes out finite and not zero
        const int fl = ((cxl & kCodeFluid) ? kLowX : 0) | ((cyl & kCodeFluid) ? kLowY : 0) | ((czl & kCodeFluid) ? kLowZ : 0) |
                       ((cxh & kCodeFluid) ? kHighX : 0) | ((cyh & kCodeFluid) ? kHighY : 0) | ((czh & kCodeFluid) ? kHighZ : 0);
        av = S.A0f ? S.A0f[g] : (float)(c & 7);
        reg = reg && (c & (kLowX | kLowY | kLowZ | kHighX | kHighY | kHighZ)) == fl && av > 1e-6f && av < 1e6f;
      }
    }
    s_c[u * 64 + zl * 8 + yl][lane] = (unsigned short)o;
    s_a[u * 64 + zl * 8 + yl][lane] = av;
  }
  const unsigned all = __ballot_sync(0xffffffffu, reg);
  if (lane == 0) s_reg[w] = all;
  __syncthreads();
  const long long unit = (long long)b * kMcWarps + u;
  const unsigned both = s_reg[2 * u] & s_reg[2 * u + 1];
  const int ch = L0 / kCH + lane;
  if (hz == 0 && lane < 32 / kCH && ch < S.nlp / kCH)
    S.regular[unit * (S.nlp / kCH) + ch] = ((both >> (kCH * lane)) & 0xffu) == 0xffu ? 1 : 0;
  // lane (j, q): lines z = 2q and 2q + 1 of row j; this warp writes 16 levels
  const int la = u * 64 + (lane & 7) + 16 * (lane >> 3);
  for (int i = 16 * hz; i < 16 * hz + 16 && L0 + i < S.nlp; i++) {
    S.cw[(unit * S.nlp + L0 + i) * 32 + lane] = (unsigned)s_c[la][i] | ((unsigned)s_c[la + 8][i] << 16);
    if (S.A0f) reinterpret_cast<float2*>(S.P)[(unit * S.nlp + L0 + i) * 32 + lane] = make_float2(s_a[la][i], s_a[la + 8][i]);
  }
}
constexpr size_t kOrderSmem = 64 * kMcWarps * (34 * sizeof(unsigned short) + 33 * sizeof(float));

// Between grid and level order, with the element-wise work of the iteration
// on the way: a CTA takes one bundle over 32 levels, rows of 32 cells on the
// grid side, turned in shared memory.  All of it is memory traffic; the skewed
// rows cost a fifth more sectors than aligned ones.  A CTA per block (48 at
// 64^3) with its rows in four batches took 11.3 us for axpy and 6.4 for the
// update there, a CTA per bundle with one batch 8.3 and 6.4 (cold caches); with
// the chain's launches overlapped (pass_started) an iteration of the solver
// takes 73 instead of 82 us at 64^3, 142 instead of 154 on the dam at 128^3.
enum { kLvlInit = 0, kLvlAxpy = 1, kLvlUpdate = 2, kLvlSearch = 3 };
constexpr int kLvlThreads = 256;
template <int OP, bool L2 = false>
__global__ void __launch_bounds__(kLvlThreads, 3) k_lvl(McArgs a) {
  __shared__ float tile[64][33];
  pass_started();
  pass_wait();
  const MicClusterScene& S = a.scenes ? a.scenes[blockIdx.y] : a.one;
  CgScalars* const sc = S.sc;
  const int nx = S.d.nx, ny = S.d.ny, nz = S.d.nz, nlp = S.nlp;
  // part has a slot for every block's 32 levels, in a single solve for more
  const int tiles = (nlp + 31) / 32, total = S.nby * S.nbz * tiles * kMcWarps;
  const int ctas = min((int)gridDim.x, a.scenes ? total / kMcWarps : total);
  if ((int)blockIdx.x >= ctas) return;
  if ((OP == kLvlAxpy || OP == kLvlUpdate) && sc->done) return;
  const float alpha = OP == kLvlAxpy ? sc->alpha : 0.f, na = -alpha;
  const float beta = OP == kLvlUpdate ? sc->beta : 0.f;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float mn = FLT_MAX, mx = -FLT_MAX;
  double ss = 0.;
  for (int t = blockIdx.x; t < total; t += ctas) {
    const int ub = t / tiles, L0 = (t - ub * tiles) * 32, u = ub & (kMcWarps - 1), b = ub / kMcWarps;
    const int y0 = (b % S.nby) * kBlk + (u & 1) * kUY, z0 = (b / S.nby) * kBlk + (u >> 1) * kUZ;
    // grid side: this warp's line z = w of the bundle, eight rows y.  All loads
    // are issued before the first store.
    const long long g0 = ((long long)(z0 + w) * ny + y0) * nx + L0 + lane - w;
    const int line = (w & 1) * 32 + (w >> 1) * 8;
    auto cell = [&](int q) { return g0 + (long long)q * (nx - 1); };
    unsigned in = 0u;
#pragma unroll
    for (int q = 0; q < kUY; q++)
      in |= ((unsigned)(L0 + lane - q - w) < (unsigned)nx && y0 + q < ny && z0 + w < nz) ? 1u << q : 0u;
    // level side: levels 4w .. 4w + 3; a lane's even line in tile row lane, its odd one in row 32 + lane
    const long long base = (((long long)b * kMcWarps + u) * nlp + L0 + 4 * w) * 32 + lane;
    const float *ta = &tile[lane][4 * w], *tb = &tile[32 + lane][4 * w];
    const int levels = min(4, nlp - L0 - 4 * w);
    const int y = y0 + (lane & 7), z = z0 + 2 * (lane >> 3), xs = L0 + 4 * w - (lane & 7) - 2 * (lane >> 3);
    float2* const r2 = reinterpret_cast<float2*>(S.r) + base;
    if (OP == kLvlInit || OP == kLvlAxpy) {
      float t8[kUY], s8[kUY], p8[kUY];
#pragma unroll
      for (int q = 0; q < kUY; q++) {
        const bool ok = in >> q & 1u;
        const long long g = cell(q);
        t8[q] = ok ? (OP == kLvlInit ? S.rhs[g] : S.t[g]) : 0.f;
        if (OP == kLvlAxpy) {
          s8[q] = ok ? S.s[g] : 0.f;
          p8[q] = ok ? S.p[g] : 0.f;
        }
      }
      float2 o[4];
      if (OP == kLvlAxpy)
#pragma unroll
        for (int i = 0; i < 4; i++) o[i] = i < levels ? r2[32 * i] : make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < kUY; q++) {
        tile[line + q][lane] = t8[q];
        if (in >> q & 1u) S.p[cell(q)] = OP == kLvlInit ? 0.f : p8[q] + alpha * s8[q];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float2 r = make_float2(ta[i], tb[i]);
        if (OP == kLvlAxpy) {
          const bool oka = y < ny && z < nz && (unsigned)(xs + i) < (unsigned)nx;
          const bool okb = y < ny && z + 1 < nz && (unsigned)(xs + i - 1) < (unsigned)nx;
          r.x = oka ? o[i].x + na * r.x : 0.f;
          r.y = okb ? o[i].y + na * r.y : 0.f;
          if (oka) {
            mn = fminf(mn, r.x);
            mx = fmaxf(mx, r.x);
          }
          if (okb) {
            mn = fminf(mn, r.y);
            mx = fmaxf(mx, r.y);
          }
          if (L2) ss += (double)r.x * (double)r.x + (double)r.y * (double)r.y;
        }
        if (i < levels) r2[32 * i] = r;
      }
    } else {
      const float2* const z2 = reinterpret_cast<const float2*>(S.z) + base;
      float s8[kUY];
      if (OP == kLvlUpdate)
#pragma unroll
        for (int q = 0; q < kUY; q++) s8[q] = (in >> q & 1u) ? S.s[cell(q)] : 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float2 v = i < levels ? z2[32 * i] : make_float2(0.f, 0.f);
        tile[lane][4 * w + i] = v.x;
        tile[32 + lane][4 * w + i] = v.y;
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kUY; q++)
        if (in >> q & 1u) S.s[cell(q)] = OP == kLvlSearch ? tile[line + q][lane] : tile[line + q][lane] + beta * s8[q];
    }
    __syncthreads();
  }
  if (OP != kLvlAxpy) return;
  // residual norm and convergence test (conjugategrad.cpp:262-276)
  block_minmax(mn, mx);
  const double bs = L2 ? block_sum(ss) : 0.;
  float* const pf = reinterpret_cast<float*>(S.part);
  if (threadIdx.x == 0) {
    if (L2) {
      S.part[blockIdx.x] = bs;
    } else {
      pf[2 * blockIdx.x] = mn;
      pf[2 * blockIdx.x + 1] = mx;
    }
  }
  if (last_block(&sc->counters[2], ctas)) {
    float res;
    if (L2) {
      res = (float)sum_partials(S.part, (int)ctas);
    } else {
      float lo, hi;
      minmax_partials(pf, (int)ctas, lo, hi);
      const float p = fabsf(lo), q = fabsf(hi);
      res = hi < lo ? S.nanNorm : p < q ? q : p;
    }
    if (threadIdx.x != 0) return;
    sc->iterations += 1;
    sc->resNorm = res;
    if (res < sc->accuracy) {
      sc->sigma = res;
      sc->done = 1;
      if (a.ndone) atomicAdd(a.ndone, 1);
    } else if (a.ndone && sc->iterations >= sc->maxIter) {
      sc->done = 1;
      atomicAdd(a.ndone, 1);
    }
  }
}

// ---------------------------------------------------------------- host side
static int g_mcCluster = 0;  // CTAs of a cluster (0: no clusters of 8 or 16)

static_assert(kCH == 8, "a chunk's bits in a byte");
static size_t mc_smem(int nlp) {
  return (size_t)16 * kMcWarps * (nlp + 2 * kPad) * sizeof(unsigned) + (size_t)kMcWarps * kStages * (3 * kVecWords + kBitWords) * sizeof(float);
}
static int mc_levels(int nx) { return (nx + kSkew + kCH - 1) / kCH * kCH; }

typedef void (*McKernel)(McArgs);
static McKernel mc_kernel(int mode) {
  return mode == 0 ? k_mic_cluster<0> : mode == 1 ? k_mic_cluster<1> : k_mic_cluster<2>;
}
static cudaLaunchConfig_t mc_config(int clusters, size_t smem, cudaLaunchAttribute* at, cudaStream_t s) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = g_mcCluster;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * g_mcCluster));
  cfg.blockDim = dim3(kMcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

int mic_cluster_prepare() {
  g_mcCluster = 0;
  for (int mode = 0; mode < 3; mode++)
    if (cudaFuncSetAttribute(mc_kernel(mode), cudaFuncAttributeMaxDynamicSharedMemorySize, kMcMaxSmem) != cudaSuccess ||
        cudaFuncSetAttribute(mc_kernel(mode), cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      return 1;
  if (cudaFuncSetAttribute(k_mic_order, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOrderSmem) != cudaSuccess) return 1;
  for (int c = 16; c >= 8 && !g_mcCluster; c /= 2) {
    cudaLaunchAttribute at[1];
    g_mcCluster = c;
    const cudaLaunchConfig_t cfg = mc_config(1, kMcMaxSmem, at, nullptr);
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, k_mic_cluster<2>, &cfg) != cudaSuccess || nc < 1) g_mcCluster = 0;
  }
  cudaGetLastError();  // without clusters the tile sweeps run
  return 0;
}

// A cluster spans the y range (16 lines per CTA) and as many z-blocks as
// then fit; the slots of every level fit the shared memory.
bool mic_cluster_plan_for(const Dims& d, int ctas, MicClusterScene* s) {
  if (!d.is3d || !ctas) return false;
  s->d = d;
  s->nby = (d.ny + kBlk - 1) / kBlk;
  s->nbz = (d.nz + kBlk - 1) / kBlk;
  s->nlp = mc_levels(d.nx);
  if (s->nby > ctas || s->nlp > 64 * kCH || mc_smem(s->nlp) > (size_t)kMcMaxSmem) return false;
  s->zper = std::min(s->nbz, ctas / s->nby);
  return true;
}
bool mic_cluster_plan(const Dims& d, MicClusterScene* s) { return mic_cluster_plan_for(d, g_mcCluster, s); }
static size_t mc_units(const MicClusterScene& s) { return (size_t)s.nby * s.nbz * kMcWarps; }
size_t mic_cluster_floats(const MicClusterScene& s) { return mc_units(s) * s.nlp * 64; }
size_t mic_cluster_flag_bytes(const MicClusterScene& s) { return mc_units(s) * (s.nlp / kCH); }
size_t mic_cluster_face_words(const MicClusterScene& s) {
  return (size_t)2 * ((s.nbz + s.zper - 1) / s.zper) * (s.nlp + 2 * kPad) * s.nby * kBlk;
}
int mic_cluster_jobs(const MicClusterScene& s) { return (s.nbz + s.zper - 1) / s.zper; }

static McArgs mc_args(const MicClusterLaunch& m) {
  McArgs a;
  memset(&a, 0, sizeof(a));
  a.one = m.one;
  a.scenes = m.scenes;
  a.jobs = m.jobs;
  a.njobs = m.njobs;
  a.counter = m.counter;
  a.error = m.error;
  a.ndone = m.ndone;
  a.waitNs = m.waitNs;
  a.nlpMax = m.nlpMax;
  a.stall = m.stall;
  return a;
}

cudaError_t launch_mic_cluster_order(const MicClusterLaunch& m, cudaStream_t s) {
  const McArgs a = mc_args(m);
  count_launch();
  k_mic_order<<<dim3((unsigned)m.maxBlocks, (unsigned)((m.nlpMax + 31) / 32), (unsigned)m.nscenes), 64 * kMcWarps,
                kOrderSmem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mic_level(const MicClusterLaunch& m, int op, cudaStream_t s) {
  const McArgs a = mc_args(m);
  const int tiles = m.maxBlocks * ((m.nlpMax + 31) / 32) * (m.scenes ? 1 : kMcWarps);
  const dim3 g((unsigned)std::min(tiles, m.maxParts), (unsigned)m.nscenes);
  const auto k = op == kMicInit ? k_lvl<kLvlInit> : op == kMicAxpy ? (m.l2 ? k_lvl<kLvlAxpy, true> : k_lvl<kLvlAxpy>)
                 : op == kMicUpdate ? k_lvl<kLvlUpdate> : k_lvl<kLvlSearch>;
  count_launch();
  return launch_pass(k, g, dim3(kLvlThreads), 0, s, !m.scenes, a);
}

// mode: 0 factor, 1 forward, 2 backward (beta), 3 backward for doInit (sigma)
cudaError_t launch_mic_cluster(const MicClusterLaunch& m, int mode, cudaStream_t s) {
  McArgs a = mc_args(m);
  a.init = mode == 3 ? 1 : 0;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = mc_config(m.njobs, mc_smem(m.nlpMax), at, s);
  if (!m.scenes) {
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  count_launch();
  return cudaLaunchKernelEx(&cfg, mc_kernel(mode), a);
}

}  // namespace mgpu
