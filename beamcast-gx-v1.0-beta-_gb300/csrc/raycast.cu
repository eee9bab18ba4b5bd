// Ray-cast kernels: exact closest hit and any hit over the BVH8, one thread
// per ray. Rays are 32-byte records (ox, oy, oz, tmin, dx, dy, dz, tmax) read
// with two 128-bit loads; results are written as coalesced 4-byte streams.
#include <algorithm>

#include "kernels.h"
#include "trace_core.cuh"

namespace bcgx {

int stack_variant(int need) {
  if (need <= 64) return 64;
  if (need <= 128) return 128;
  if (need <= 256) return 256;
  return 0;
}

namespace {

template <int STACK, bool SPHERES, int MINB>
__global__ void __launch_bounds__(128, MINB) k_closest_exact(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                       float* __restrict__ t_out, int32_t* __restrict__ prim_out,
                                                       unsigned* status) {
  // No early return: every lane reaches the warp-converged fp64 settlement.
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n;
  float4 a = make_float4(0, 0, 0, 0), b = a;
  if (active) {
    a = __ldg(rays + 2 * i);
    b = __ldg(rays + 2 * i + 1);
  }
  const Ray32 r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
  const HitResult h = closest_hit_exact<STACK, SPHERES>(sv, r, b.w, status, active);
  if (!active) return;
  if (h.slot >= 0) {
    t_out[i] = __double2float_rn(h.t64);
    prim_out[i] = h.tie ? kTieMark : __ldg(sv.slot_prim + h.slot);
  } else {
    t_out[i] = -1.0f;
    prim_out[i] = -1;
  }
}

template <int STACK, bool SPHERES, int MINB>
__global__ void __launch_bounds__(128, MINB) k_any_exact(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                   uint8_t* __restrict__ out, unsigned* status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = __ldg(rays + 2 * i);
  const float4 b = __ldg(rays + 2 * i + 1);
  const Ray32 r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
  out[i] = any_hit_exact<STACK, SPHERES>(sv, r, b.w, status) ? 1 : 0;
}

// Fast variant: the same walk with plain fp32 tests (no exactness contract:
// near ties and edge grazes may differ from the fp64 path).
template <int STACK, bool SPHERES>
__global__ void __launch_bounds__(128) k_closest_fast(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                      float* __restrict__ t_out, int32_t* __restrict__ prim_out,
                                                      unsigned* status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = __ldg(rays + 2 * i);
  const float4 b = __ldg(rays + 2 * i + 1);
  const Ray32 r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
  const HitResult h = closest_hit_fast<STACK, SPHERES>(sv, r, b.w, status);
  t_out[i] = h.slot >= 0 ? h.t32 : -1.0f;
  prim_out[i] = h.slot >= 0 ? __ldg(sv.slot_prim + h.slot) : -1;
}

__device__ __forceinline__ const int32_t* walk_order(const int32_t* perm);

// ---- persistent kernels with per-lane refill -------------------------------
// Lanes whose rays are done fetch the next ray indices once kRefillLanes of the
// warp's lanes are idle (one atomic per warp for all of them), so the warp does
// not idle until its slowest ray ends. The exact kernel parks each finished ray's contenders in a
// per-warp queue in shared memory; when 32 are parked, the warp settles them
// in fp64 with every lane active. Triangle-only scenes: the settlement here runs the
// triangles' test alone (spheres use the kernels above).
constexpr int kParkTie = 0x100;  // npend flag: the walk already compared two equal fp64 distances

struct ParkQueue {
  long long idx[32];
  int bslot[32];
  float bhi[32];
  int npend[32];
  int pslot[kPending][32];
  float plo[kPending][32];
};

__device__ __forceinline__ void settle_parked(const SceneView& sv, const float4* __restrict__ rays,
                                              const ParkQueue& q, int k, float* __restrict__ t_out,
                                              int32_t* __restrict__ prim_out, unsigned* status) {
  const long long i = q.idx[k];
  const float4 a = __ldg(rays + 2 * i), b = __ldg(rays + 2 * i + 1);
  const D3 o{(double)a.x, (double)a.y, (double)a.z}, d{(double)b.x, (double)b.y, (double)b.z};
  const double tmin = (double)a.w, tmax = (double)b.w;
  const int bslot = q.bslot[k];
  const float bhi = q.bhi[k];
  int win = -1;
  double wt = 0.0;
  if (bslot >= 0) {
    double t;
    if (tri_hit64(sv.slot64 + 9 * (size_t)bslot, o, d, tmin, tmax, &t)) {
      win = bslot;
      wt = t;
    } else {
      atomicOr(status, kStatusBound);  // a certain hit must pass its fp64 test
    }
  }
  const int np = q.npend[k] & 0xff;
  bool tie = (q.npend[k] & kParkTie) != 0;
#pragma unroll
  for (int j = 0; j < kPending; j++) {
    if (j < np && !(bslot >= 0 && q.plo[j][k] > bhi)) {
      const int sj = q.pslot[j][k];
      double t;
      if (tri_hit64(sv.slot64 + 9 * (size_t)sj, o, d, tmin, tmax, &t)) {
        tie = tie || (win >= 0 && t == wt);
        if (win < 0 || t < wt || (t == wt && sj > win)) {
          win = sj;
          wt = t;
        }
      }
    }
  }
  if (win >= 0) {
    t_out[i] = __double2float_rn(wt);
    prim_out[i] = tie ? kTieMark : __ldg(sv.slot_prim + win);
  } else {
    t_out[i] = -1.0f;
    prim_out[i] = -1;
  }
}

template <int STACK, int MINB>
__global__ void __launch_bounds__(128, MINB) k_closest_exact_persistent(SceneView sv, const float4* __restrict__ rays,
                                                                        int64_t n, float* __restrict__ t_out,
                                                                        int32_t* __restrict__ prim_out,
                                                                        unsigned* status, unsigned long long* work,
                                                                        const int32_t* __restrict__ order) {
  const int32_t* __restrict__ perm = walk_order(order);
  __shared__ ParkQueue park[4];
  ParkQueue& q = park[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  long long idx = -1;
  bool exhausted = false;
  Ray32 r = make_ray(0, 0, 0, 0, 0, 0, 0);
  ExactClosestLeaf<false> leaf(sv, r, 0.0f, status);
  Walker<STACK, kExactLeafVote> w;
  w.reset(r);
  int parked = 0;  // warp-uniform
  for (;;) {
    const bool need = idx < 0 && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m && (__popc(m) >= kRefillLanes || !__any_sync(0xffffffffu, idx >= 0))) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if ((int)lane == leader) base = atomicAdd(work, (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const unsigned long long my = base + (unsigned long long)__popc(m & below);
        if (my < (unsigned long long)n) {
          idx = perm ? (long long)perm[my] : (long long)my;
          const float4 a = __ldg(rays + 2 * idx), b = __ldg(rays + 2 * idx + 1);
          r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
          leaf.reset(b.w);
          w.reset(r);
        } else {
          exhausted = true;
        }
      }
    }
    const bool active = idx >= 0;
    if (!__any_sync(0xffffffffu, active)) break;
    bool finished = false;
    if (active) finished = w.step(sv, r, leaf, status);
    const unsigned pm = __ballot_sync(0xffffffffu, finished);
    if (pm) {
      if (parked + __popc(pm) > 32) {
        __syncwarp();
        if ((int)lane < parked) settle_parked(sv, rays, q, (int)lane, t_out, prim_out, status);
        __syncwarp();
        parked = 0;
      }
      if (finished) {
        const int k = parked + __popc(pm & below);
        q.idx[k] = idx;
        q.bslot[k] = leaf.best.slot;
        q.bhi[k] = leaf.best.hi;
        q.npend[k] = leaf.npend | (leaf.tie ? kParkTie : 0);
#pragma unroll
        for (int j = 0; j < kPending; j++) {
          q.pslot[j][k] = leaf.pend[j].slot;
          q.plo[j][k] = leaf.pend[j].lo;
        }
        idx = -1;
      }
      parked += __popc(pm);
    }
  }
  __syncwarp();
  if ((int)lane < parked) settle_parked(sv, rays, q, (int)lane, t_out, prim_out, status);
}

// ---- exact closest hit in passes: walk, then settle ----------------------------
// The one-kernel form above keeps the fp64 settlement (and the in-walk fp64
// re-test of a full contender list) in the walking kernel, whose register
// allocation then covers the fp64 code: 80 registers with spills at six
// 128-thread blocks per SM. Split, the walk holds no fp64 code and fits 40
// registers without spills (twelve blocks per SM; 9.74 ms -> 7.71 ms on the
// 1M-triangle / 4M-ray cast, settlement and ray order included):
//   pass 1, k_exact_walk: the persistent walk with the fp32 classifier; a
//     finished ray leaves a record (best certain hit: slot and upper bound of
//     its distance; the pending contenders: slot and lower bound). A ray with
//     more contenders than the list holds stops walking and is marked.
//   pass 2, k_exact_settle: one thread per ray settles its record in fp64 with
//     triHit's operation order (the same decisions as settle_parked) and writes
//     the result; marked rays go to a list.
//   pass 3, k_closest_exact_list: the marked rays, traced again by the
//     one-kernel exact walk, whose full list falls back to fp64 in the walk.
// Triangle-only scenes (as the persistent one-kernel form). The rays and the
// records pass through L2 once each way, so the walk and the settlement read
// and write them evict-first (ld/st.global.cs): L2 stays with the scene.
struct ExactRecords {
  int32_t* bslot;   // [n]: best certain hit, -1 none
  float* bhi;       // [n]: upper bound of its distance
  int32_t* npend;   // [n]: pending contenders; kPending + 1: list overflowed
  int32_t* pslot;   // [kPending * n]
  float* plo;       // [kPending * n]
  long long* redo;  // [n]: rays of pass 3
  unsigned long long* n_redo;
  unsigned* n_tie;  // nonzero: some ray is marked kTieMark
};


size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// Layout of the records in the caller's scratch (exact_record_bytes(n) bytes).
ExactRecords exact_records(void* p, int64_t n) {
  auto up = up256;
  char* q = (char*)p;
  ExactRecords r;
  r.n_redo = (unsigned long long*)q;
  r.n_tie = (unsigned*)(q + 8);
  q += 256;
  r.bslot = (int32_t*)q;
  q += up((size_t)n * 4);
  r.bhi = (float*)q;
  q += up((size_t)n * 4);
  r.npend = (int32_t*)q;
  q += up((size_t)n * 4);
  r.pslot = (int32_t*)q;
  q += up((size_t)n * 4 * kPending);
  r.plo = (float*)q;
  q += up((size_t)n * 4 * kPending);
  r.redo = (long long*)q;
  return r;
}

// ExactClosestLeaf's decisions without its fp64 fallback: where that leaf
// resolves a contender in fp64 because its list is full, this one marks the
// ray (npend = kPending + 1) and ends the walk (done).
struct FilterLeaf {
  const SceneView& sv;
  const Ray32& r;
  float tmax_ray;
  float tlim;
  bool done;
  int32_t bslot;
  float blo, bhi;
  int npend;
  PendEntry pend[kPending];

  __device__ FilterLeaf(const SceneView& s, const Ray32& ray) : sv(s), r(ray) { reset(0.0f); }
  __device__ __forceinline__ void reset(float tmax) {
    tmax_ray = tmax;
    tlim = widen(tmax);
    done = false;
    npend = 0;
    bslot = -1;
    blo = tmax;
    bhi = tmax;
  }
  __device__ __forceinline__ void overflow() {
    npend = kPending + 1;
    done = true;
  }
  __device__ __forceinline__ void take_certain(int slot, float lo, float hi) {
    if (bslot < 0 || hi < blo) {
      bslot = slot;
      blo = lo;
      bhi = hi;
    } else if (lo > bhi) {
      return;
    } else if (npend < kPending) {
      if (hi < bhi) {
        pend[npend++] = PendEntry{bslot, blo};
        bslot = slot;
        blo = lo;
        bhi = hi;
      } else {
        pend[npend++] = PendEntry{slot, lo};
      }
    } else {
      overflow();
      return;
    }
    tlim = widen(bhi);
  }
  __device__ __forceinline__ void operator()(uint32_t ref) {
    const int cnt = (int)((ref >> 27) & 15u) + 1;
    const int s0 = (int)(ref & kSlotMask);
    for (int k = 0; k < cnt && !done; k++) {
      const int s = s0 + k;
      const float4 A = __ldg(sv.tri + 3 * s);
      const float4 E1 = __ldg(sv.tri + 3 * s + 1);
      const float4 E2 = __ldg(sv.tri + 3 * s + 2);
      const TriClass tc = tri_classify(A, E1, E2, r, tmax_ray, tlim);
      if (tc.state == kMiss) continue;
      const float lo = __fsub_rd(tc.t, tc.et), hi = __fadd_ru(tc.t, tc.et);
      if (bslot >= 0 && lo > bhi) continue;
      if (tc.state == kHit) take_certain(s, lo, hi);
      else if (npend < kPending) pend[npend++] = PendEntry{s, lo};
      else overflow();
    }
  }
};

template <int STACK>
__global__ void __launch_bounds__(128, 12) k_exact_walk(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                       ExactRecords rec, unsigned* status, unsigned long long* work,
                                                       const int32_t* __restrict__ order) {
  const int32_t* __restrict__ perm = walk_order(order);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  long long idx = -1;
  bool exhausted = false;
  Ray32 r = make_ray(0, 0, 0, 0, 0, 0, 0);
  FilterLeaf leaf(sv, r);
  Walker<STACK, kExactLeafVote> w;
  w.reset(r);
  for (;;) {
    const bool need = idx < 0 && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m && (__popc(m) >= kRefillLanes || !__any_sync(0xffffffffu, idx >= 0))) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if ((int)lane == leader) base = atomicAdd(work, (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const unsigned long long my = base + (unsigned long long)__popc(m & below);
        if (my < (unsigned long long)n) {
          idx = perm ? (long long)perm[my] : (long long)my;
          const float4 a = __ldcs(rays + 2 * idx), b = __ldcs(rays + 2 * idx + 1);
          r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
          leaf.reset(b.w);
          w.reset(r);
        } else {
          exhausted = true;
        }
      }
    }
    if (!__any_sync(0xffffffffu, idx >= 0)) break;
    if (idx >= 0 && w.step(sv, r, leaf, status)) {
      __stcs(rec.bslot + idx, leaf.bslot);
      __stcs(rec.bhi + idx, leaf.bhi);
      __stcs(rec.npend + idx, leaf.npend);
      const int np = min(leaf.npend, kPending);
      for (int j = 0; j < np; j++) {
        __stcs(rec.pslot + (size_t)j * n + idx, leaf.pend[j].slot);
        __stcs(rec.plo + (size_t)j * n + idx, leaf.pend[j].lo);
      }
      idx = -1;
    }
  }
}

// The distance of a triangle that is certainly hit: triHit's operations
// (tri_hit64) without the barycentric tests that decide the hit.
__device__ __forceinline__ double tri_t64(const double* __restrict__ q, D3 o, D3 d) {
  const D3 a{__ldg(q + 0), __ldg(q + 1), __ldg(q + 2)};
  const D3 e1{__ldg(q + 3), __ldg(q + 4), __ldg(q + 5)};
  const D3 e2{__ldg(q + 6), __ldg(q + 7), __ldg(q + 8)};
  const double f = __ddiv_rn(1.0, ddot(e1, dcross(d, e2)));
  return dm(f, ddot(e2, dcross(dsub3(o, a), e1)));
}

// Settles the records. The kernel is bound by the fp64 pipe (1/64 of the fp32
// rate), which a warp pays for whole whatever lanes take part, so a warp sorts
// its rays first: misses are written at once, rays with one certain hit and no
// contender need only its distance, the others the full tests (4,194,304 rays
// against 1,000,000 triangles: 0.74 -> 0.45 ms);
// each kind is settled 32 at a time. That a certain hit passes its fp64 test is checked
// on one group of 32 in sixteen (in each warp from another one on); on all of them it
// costs the ray cast 2% (5.95 -> 6.07 ms).
__global__ void __launch_bounds__(128) k_exact_settle(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                      ExactRecords rec, float* __restrict__ t_out,
                                                      int32_t* __restrict__ prim_out, unsigned* status) {
  __shared__ unsigned queue[4][2][64];  // rays to settle, relative to the warp's first: [0] distance only, [1] full
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  // a contiguous stretch of rays per warp
  const int64_t warps = (int64_t)gridDim.x * 4, per = ((n + warps - 1) / warps + 31) / 32 * 32;
  const int64_t first = ((int64_t)blockIdx.x * 4 + w) * per, last = min((int64_t)n, first + per);
  int len[2] = {0, 0};  // warp-uniform
  unsigned distances = blockIdx.x * 4 + w;  // groups of 32 settled by their distance, from a start of the warp's own
  for (int64_t base = first; base < last || len[0] > 0 || len[1] > 0; base += 32) {
    if (base < last) {
      const int64_t i = base + lane;
      int kind = -1;
      if (i < last) {
        const int np = __ldcs(rec.npend + i);
        if (np > kPending) {
          rec.redo[atomicAdd(rec.n_redo, 1ull)] = i;
        } else if (np > 0) {
          kind = 1;
        } else if (__ldcs(rec.bslot + i) >= 0) {
          kind = 0;
        } else {
          t_out[i] = -1.0f;
          prim_out[i] = -1;
        }
      }
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const unsigned m = __ballot_sync(0xffffffffu, kind == k);
        if (kind == k) queue[w][k][len[k] + __popc(m & below)] = (unsigned)(i - first);
        len[k] += __popc(m);
      }
      __syncwarp();
    }
    const bool drain = base + 32 >= last;
    if (len[0] >= 32 || (drain && len[0] > 0)) {
      const int take = min(len[0], 32), at = len[0] - take;
      if (lane < take) {
        const int64_t i = first + queue[w][0][at + lane];
        const float4 a = __ldcs(rays + 2 * i), b = __ldcs(rays + 2 * i + 1);
        const int slot = __ldcs(rec.bslot + i);
        const double* q = sv.slot64 + 9 * (size_t)slot;
        const D3 o{(double)a.x, (double)a.y, (double)a.z}, d{(double)b.x, (double)b.y, (double)b.z};
        const double tmin = (double)a.w, tmax = (double)b.w;
        double t;
        bool hit = true;
        if (distances % 16 == 0) hit = tri_hit64(q, o, d, tmin, tmax, &t);
        if (distances % 16 != 0 || !hit) t = tri_t64(q, o, d);
        if (!(hit && t >= tmin && t <= tmax)) atomicOr(status, kStatusBound);
        t_out[i] = __double2float_rn(t);
        prim_out[i] = __ldg(sv.slot_prim + slot);
      }
      len[0] = at;
      distances++;
      __syncwarp();
    }
    if (len[1] >= 32 || (drain && len[1] > 0)) {
      const int take = min(len[1], 32), at = len[1] - take;
      if (lane < take) {
        const int64_t i = first + queue[w][1][at + lane];
        const int np = __ldcs(rec.npend + i);
        const float4 a = __ldcs(rays + 2 * i), b = __ldcs(rays + 2 * i + 1);
        const D3 o{(double)a.x, (double)a.y, (double)a.z}, d{(double)b.x, (double)b.y, (double)b.z};
        const double tmin = (double)a.w, tmax = (double)b.w;
        const int bslot = __ldcs(rec.bslot + i);
        const float bhi = __ldcs(rec.bhi + i);
        int win = -1;
        double wt = 0.0;
        bool tie = false;
        if (bslot >= 0) {
          double t;
          if (tri_hit64(sv.slot64 + 9 * (size_t)bslot, o, d, tmin, tmax, &t)) {
            win = bslot;
            wt = t;
          } else {
            atomicOr(status, kStatusBound);  // a certain hit must pass its fp64 test
          }
        }
        for (int j = 0; j < np; j++) {
          const float lo = __ldcs(rec.plo + (size_t)j * n + i);
          if (bslot >= 0 && lo > bhi) continue;
          const int sj = __ldcs(rec.pslot + (size_t)j * n + i);
          double t;
          if (tri_hit64(sv.slot64 + 9 * (size_t)sj, o, d, tmin, tmax, &t)) {
            tie = tie || (win >= 0 && t == wt);
            if (win < 0 || t < wt || (t == wt && sj > win)) {
              win = sj;
              wt = t;
            }
          }
        }
        t_out[i] = win >= 0 ? __double2float_rn(wt) : -1.0f;
        prim_out[i] = win >= 0 ? (tie ? kTieMark : __ldg(sv.slot_prim + win)) : -1;
        if (win >= 0 && tie) *rec.n_tie = 1u;  // any number of rays store the same value
      }
      len[1] = at;
      __syncwarp();
    }
  }
}

// Pass 3: the listed rays with the one-kernel exact walk. Every lane of a warp
// runs the same number of iterations (the warp-converged settlement inside
// closest_hit_exact needs all 32 lanes).
template <int STACK>
__global__ void __launch_bounds__(128) k_closest_exact_list(SceneView sv, const float4* __restrict__ rays,
                                                            ExactRecords rec, float* __restrict__ t_out,
                                                            int32_t* __restrict__ prim_out, unsigned* status) {
  const long long cnt = (long long)*((volatile unsigned long long*)rec.n_redo);
  for (long long base = (long long)blockIdx.x * blockDim.x; base < cnt; base += (long long)gridDim.x * blockDim.x) {
    const long long k = base + threadIdx.x;
    const bool active = k < cnt;
    const long long i = active ? rec.redo[k] : 0;
    float4 a = make_float4(0, 0, 0, 0), b = a;
    if (active) {
      a = __ldg(rays + 2 * i);
      b = __ldg(rays + 2 * i + 1);
    }
    const Ray32 r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
    const HitResult h = closest_hit_exact<STACK, false>(sv, r, b.w, status, active);
    if (active) {
      t_out[i] = h.slot >= 0 ? __double2float_rn(h.t64) : -1.0f;
      prim_out[i] = h.slot >= 0 ? (h.tie ? kTieMark : __ldg(sv.slot_prim + h.slot)) : -1;
      if (h.slot >= 0 && h.tie) *rec.n_tie = 1u;
    }
  }
}

// ---- exact any hit in passes -----------------------------------------------------
// The same split for Scene.Occluded: the walk (no fp64 code) decides a ray when
// a triangle certainly blocks it or when no triangle might; a ray with
// undecided ("maybe") triangles is appended to a list with up to kPending of
// them, which the second pass tests in fp64 (triAnyHit's operation order); a
// ray with more is re-traced there by the one-kernel exact any-hit walk.
struct AnyRecords {
  long long* idx;   // [n] listed rays
  int32_t* npend;   // [n] maybe-triangles listed; kPending + 1: list overflowed
  int32_t* pslot;   // [kPending * n]
  unsigned long long* count;
};

AnyRecords any_records(void* p, int64_t n) {
  char* q = (char*)p;
  AnyRecords r;
  r.count = (unsigned long long*)q;
  q += 256;
  r.idx = (long long*)q;
  q += up256((size_t)n * 8);
  r.npend = (int32_t*)q;
  q += up256((size_t)n * 4);
  r.pslot = (int32_t*)q;
  return r;
}

// ExactAnyLeaf's decisions without its fp64 test: a maybe-triangle is listed.
struct FilterAnyLeaf {
  const SceneView& sv;
  const Ray32& r;
  float tmax_ray;
  float tlim;
  bool done, hit;
  int npend;
  int32_t pend[kPending];

  __device__ FilterAnyLeaf(const SceneView& s, const Ray32& ray) : sv(s), r(ray) { reset(0.0f); }
  __device__ __forceinline__ void reset(float tmax) {
    tmax_ray = tmax;
    tlim = widen(tmax);
    done = false;
    hit = false;
    npend = 0;
  }
  __device__ __forceinline__ void operator()(uint32_t ref) {
    const int cnt = (int)((ref >> 27) & 15u) + 1;
    const int s0 = (int)(ref & kSlotMask);
    for (int k = 0; k < cnt && !done; k++) {
      const int s = s0 + k;
      const float4 A = __ldg(sv.tri + 3 * s);
      const float4 E1 = __ldg(sv.tri + 3 * s + 1);
      const float4 E2 = __ldg(sv.tri + 3 * s + 2);
      const TriClass tc = tri_classify(A, E1, E2, r, tmax_ray, tlim);
      if (tc.state == kHit) {
        hit = true;
        done = true;
      } else if (tc.state == kMaybe) {
        if (npend < kPending) {
          pend[npend++] = s;
        } else {
          npend = kPending + 1;
          done = true;
        }
      }
    }
  }
};

template <int STACK>
__global__ void __launch_bounds__(128, 12) k_any_walk(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                      uint8_t* __restrict__ out, AnyRecords rec, unsigned* status,
                                                      unsigned long long* work,
                                                      const int32_t* __restrict__ order) {
  const int32_t* __restrict__ perm = walk_order(order);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  long long idx = -1;
  bool exhausted = false;
  Ray32 r = make_ray(0, 0, 0, 0, 0, 0, 0);
  FilterAnyLeaf leaf(sv, r);
  Walker<STACK, kAnyLeafVote> w;
  w.reset(r);
  for (;;) {
    const bool need = idx < 0 && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m && (__popc(m) >= kRefillLanes || !__any_sync(0xffffffffu, idx >= 0))) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if ((int)lane == leader) base = atomicAdd(work, (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const unsigned long long my = base + (unsigned long long)__popc(m & below);
        if (my < (unsigned long long)n) {
          idx = perm ? (long long)perm[my] : (long long)my;
          const float4 a = __ldcs(rays + 2 * idx), b = __ldcs(rays + 2 * idx + 1);
          r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
          leaf.reset(b.w);
          w.reset(r);
        } else {
          exhausted = true;
        }
      }
    }
    if (!__any_sync(0xffffffffu, idx >= 0)) break;
    if (idx >= 0 && w.step(sv, r, leaf, status)) {
      if (leaf.hit || leaf.npend == 0) {
        out[idx] = leaf.hit ? 1 : 0;
      } else {
        const unsigned long long k = atomicAdd(rec.count, 1ull);
        rec.idx[k] = idx;
        rec.npend[k] = leaf.npend;
        const int np = min(leaf.npend, kPending);
        for (int j = 0; j < np; j++) rec.pslot[(size_t)j * n + k] = leaf.pend[j];
      }
      idx = -1;
    }
  }
}

template <int STACK>
__global__ void __launch_bounds__(128) k_any_settle(SceneView sv, const float4* __restrict__ rays, int64_t n,
                                                    uint8_t* __restrict__ out, AnyRecords rec, unsigned* status) {
  const long long cnt = (long long)*((volatile unsigned long long*)rec.count);
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += (long long)gridDim.x * blockDim.x) {
    const long long i = rec.idx[k];
    const float4 a = __ldcs(rays + 2 * i), b = __ldcs(rays + 2 * i + 1);
    const int np = rec.npend[k];
    if (np > kPending) {
      const Ray32 r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
      out[i] = any_hit_exact<STACK, false>(sv, r, b.w, status) ? 1 : 0;
      continue;
    }
    const D3 o{(double)a.x, (double)a.y, (double)a.z}, d{(double)b.x, (double)b.y, (double)b.z};
    bool hit = false;
    for (int j = 0; j < np && !hit; j++) {
      double t;
      hit = tri_hit64(sv.slot64 + 9 * (size_t)rec.pslot[(size_t)j * n + k], o, d, (double)a.w, (double)b.w, &t);
    }
    out[i] = hit ? 1 : 0;
  }
}

template <int STACK>
__global__ void __launch_bounds__(128) k_closest_fast_persistent(SceneView sv, const float4* __restrict__ rays,
                                                                 int64_t n, float* __restrict__ t_out,
                                                                 int32_t* __restrict__ prim_out, unsigned* status,
                                                                 unsigned long long* work,
                                                                 const int32_t* __restrict__ order) {
  const int32_t* __restrict__ perm = walk_order(order);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  long long idx = -1;
  bool exhausted = false;
  Ray32 r = make_ray(0, 0, 0, 0, 0, 0, 0);
  FastClosestLeaf<false> leaf(sv, r, 0.0f);
  FastWalker<STACK, kLeafVote> w;
  w.reset(r);
  for (;;) {
    const bool need = idx < 0 && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m && (__popc(m) >= kRefillLanes || !__any_sync(0xffffffffu, idx >= 0))) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if ((int)lane == leader) base = atomicAdd(work, (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const unsigned long long my = base + (unsigned long long)__popc(m & below);
        if (my < (unsigned long long)n) {
          idx = perm ? (long long)perm[my] : (long long)my;
          const float4 a = __ldg(rays + 2 * idx), b = __ldg(rays + 2 * idx + 1);
          r = make_ray(a.x, a.y, a.z, b.x, b.y, b.z, a.w);
          leaf.reset(b.w);
          w.reset(r);
        } else {
          exhausted = true;
        }
      }
    }
    const bool active = idx >= 0;
    if (!__any_sync(0xffffffffu, active)) break;
    if (active && w.step(sv, r, leaf, status)) {
      t_out[idx] = leaf.best_slot >= 0 ? leaf.best_t : -1.0f;
      prim_out[idx] = leaf.best_slot >= 0 ? __ldg(sv.slot_prim + leaf.best_slot) : -1;
      idx = -1;
    }
  }
}

// ---- ray order -------------------------------------------------------------------
// Batches of at least min_ordered_rays rays that come in no order of their own
// (k_ray_probe) are traced in the order of a 21-bit key: the Morton code of the origin
// on a 64^3 grid over the scene bounds, then the direction octant, so a warp's
// rays start near each other and head the same way (fewer divergent node
// visits, better L1 reuse). A counting sort over the 2^21 keys gives the
// permutation; rays and results stay in the caller's order.
constexpr int kKeyBits = 21, kKeyBins = 1 << kKeyBits, kScanBlock = 1024;

__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // 6 bits -> every third bit
  v &= 63u;
  v = (v | (v << 8)) & 0x0000f00fu;
  v = (v | (v << 4)) & 0x000c30c3u;
  v = (v | (v << 2)) & 0x00249249u;
  return v;
}

__device__ __forceinline__ uint3 ray_cell(float4 a, float3 lo, float3 scale) {  // NaN origins -> 0
  return make_uint3((uint32_t)min(max((a.x - lo.x) * scale.x, 0.0f), 63.0f),
                    (uint32_t)min(max((a.y - lo.y) * scale.y, 0.0f), 63.0f),
                    (uint32_t)min(max((a.z - lo.z) * scale.z, 0.0f), 63.0f));
}

// Clears the bins and decides whether the batch is ordered at all: only when at
// least half of 1,024 sampled neighbours (rays i and i + 1) start more than a
// cell apart. Rays that come in an order of their own (pixels of a camera,
// texels of a surface) are walked faster as they come: 1,048,576 any-hit rays off
// a 200,000-triangle surface 493 us ordered against 425 us, camera rays 293
// against 209; rays with random origins gain (4,194,304 against 1,000,000 triangles
// 7.09 -> 6.53 ms), from a million rays on.
__global__ void __launch_bounds__(kScanBlock) k_ray_probe(const float4* __restrict__ rays, int64_t n, float3 lo,
                                                          float3 scale, int32_t* __restrict__ bins,
                                                          int32_t* __restrict__ flag) {
  reinterpret_cast<int4*>(bins)[blockIdx.x * kScanBlock + threadIdx.x] = make_int4(0, 0, 0, 0);
  if (blockIdx.x != 0) return;
  const int64_t i = (n - 1) / kScanBlock * threadIdx.x;  // n >= 2 kScanBlock: i + 1 < n
  const uint3 p = ray_cell(__ldg(rays + 2 * i), lo, scale), q = ray_cell(__ldg(rays + 2 * i + 2), lo, scale);
  const bool apart = abs((int)p.x - (int)q.x) > 1 || abs((int)p.y - (int)q.y) > 1 || abs((int)p.z - (int)q.z) > 1;
  const int count = __syncthreads_count(apart);
  if (threadIdx.x == 0) *flag = count >= kScanBlock / 2 ? 1 : 0;
}

// The order to walk the rays in: perm where the batch was ordered (the flag lies
// before it), else as they come.
__device__ __forceinline__ const int32_t* walk_order(const int32_t* perm) {
  return perm && perm[-1] ? perm : nullptr;
}

// The lanes of the warp with this lane's key. Rays from one point (a camera's) share a key,
// and with one atomic per ray 262,144 of them took 0.4 ms to order, so equal keys take one
// atomic. Where no two neighbours' keys are equal the match is left out (a lane is its only
// peer): on random keys it costs more than it saves, 4,194,304 any-hit rays over 12 triangles
// 299 -> 345 us.
__device__ __forceinline__ unsigned key_peers(unsigned am, uint32_t key) {
  const int lane = threadIdx.x & 31;
  const uint32_t before = __shfl_up_sync(am, key, 1);
  if (!__any_sync(am, lane > 0 && before == key)) return 1u << lane;
  return __match_any_sync(am, key);
}

__global__ void k_ray_keys(const float4* __restrict__ rays, int64_t n, float3 lo, float3 scale,
                           uint32_t* __restrict__ keys, int32_t* __restrict__ bins,
                           const int32_t* __restrict__ flag) {
  if (!*flag) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned am = __ballot_sync(0xffffffffu, i < n);
  if (i >= n) return;
  const float4 a = __ldg(rays + 2 * i), b = __ldg(rays + 2 * i + 1);
  const uint3 q = ray_cell(a, lo, scale);
  const uint32_t oct = (b.x < 0.0f ? 1u : 0u) | (b.y < 0.0f ? 2u : 0u) | (b.z < 0.0f ? 4u : 0u);
  const uint32_t key = ((spread3(q.x) | (spread3(q.y) << 1) | (spread3(q.z) << 2)) << 3) | oct;
  keys[i] = key;
  const unsigned peers = key_peers(am, key);
  if ((int)(threadIdx.x & 31u) == __ffs(peers) - 1) atomicAdd(&bins[key], __popc(peers));
}

// exclusive scan of each 1024-bin block in place; block totals out
__global__ void __launch_bounds__(kScanBlock) k_scan_bins(int32_t* __restrict__ bins, int32_t* __restrict__ totals,
                                                          const int32_t* __restrict__ flag) {
  if (!*flag) return;
  __shared__ int32_t sh[kScanBlock];
  const int i = blockIdx.x * kScanBlock + threadIdx.x;
  const int v = bins[i];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < kScanBlock; o <<= 1) {
    const int add = (int)threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
    __syncthreads();
    sh[threadIdx.x] += add;
    __syncthreads();
  }
  bins[i] = sh[threadIdx.x] - v;
  if (threadIdx.x == kScanBlock - 1) totals[blockIdx.x] = sh[threadIdx.x];
}

// exclusive scan of the block totals (kKeyBins / kScanBlock = 2048 of them), one block
__global__ void __launch_bounds__(kScanBlock) k_scan_totals(int32_t* __restrict__ totals) {
  __shared__ int32_t sh[kScanBlock];
  const int a = totals[2 * threadIdx.x], b = totals[2 * threadIdx.x + 1];
  sh[threadIdx.x] = a + b;
  __syncthreads();
  for (int o = 1; o < kScanBlock; o <<= 1) {
    const int add = (int)threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
    __syncthreads();
    sh[threadIdx.x] += add;
    __syncthreads();
  }
  const int ex = sh[threadIdx.x] - (a + b);
  totals[2 * threadIdx.x] = ex;
  totals[2 * threadIdx.x + 1] = ex + a;
}

__global__ void k_ray_scatter(int64_t n, const uint32_t* __restrict__ keys, int32_t* __restrict__ bins,
                              const int32_t* __restrict__ totals, int32_t* __restrict__ perm,
                              const int32_t* __restrict__ flag) {
  if (!*flag) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned am = __ballot_sync(0xffffffffu, i < n);
  if (i >= n) return;
  const uint32_t k = keys[i];
  const unsigned peers = key_peers(am, k);
  const int leader = __ffs(peers) - 1;
  int at = 0;
  if ((int)(threadIdx.x & 31u) == leader) at = atomicAdd(&bins[k], __popc(peers));
  at = __shfl_sync(peers, at, leader) + __popc(peers & ((1u << (threadIdx.x & 31u)) - 1u));
  perm[totals[k / kScanBlock] + at] = (int32_t)i;
}

// ---- exact ties: the reference's own walk ------------------------------------
// A ray marked kTieMark has its closest fp64 distance shared by two or more
// primitives. Which of them the reference returns depends on its traversal
// order: triHit accepts t == closest (renderer.go:702), so the last one tested
// at that distance wins. Such a ray is walked again here exactly as Scene.Hit
// walks the caller's binary BVH (renderer.go:777-849): a 16-entry stack of
// (node, entry distance); a popped entry at or beyond the closest hit is
// skipped (796); a leaf tests its primitives in Order (800-808); both children
// are box-tested against the closest hit and pushed far first, the left one
// nearer on equal entry distances (828-839); with the stack full, the
// recursive descent of hitRecursive (815-826, 914-939) takes the left subtree,
// then the right one, each node box-tested when it is reached. Arithmetic is
// fp64 in the reference's operation order: prepareRay and HitAccel
// (renderer.go:59-81, 147-210), triHit and sphereHitAccel.
constexpr int kReplayDepth = 256;  // pending subtrees of the recursive descent

struct Accel64 {
  D3 o, inv;
  bool zx, zy, zz;
};

// One slab of HitAccel: an axis with |d| < 1e-15 only checks the origin.
__device__ __forceinline__ bool slab64(bool zero, double o, double inv, double mn, double mx, double* near,
                                       double* far) {
  if (zero) return !(o < mn || o > mx);
  double t0 = __dmul_rn(__dsub_rn(mn, o), inv);
  double t1 = __dmul_rn(__dsub_rn(mx, o), inv);
  if (inv < 0) {
    const double x = t0;
    t0 = t1;
    t1 = x;
  }
  if (t0 > *near) *near = t0;
  if (t1 < *far) *far = t1;
  return !(*far <= *near);
}

__device__ __forceinline__ bool box64(const BinNode* __restrict__ b, const Accel64& a, double tmin, double tmax,
                                      double* near_out) {
  double near = tmin, far = tmax;
  if (!slab64(a.zx, a.o.x, a.inv.x, __ldg(&b->lo[0]), __ldg(&b->hi[0]), &near, &far)) return false;
  if (!slab64(a.zy, a.o.y, a.inv.y, __ldg(&b->lo[1]), __ldg(&b->hi[1]), &near, &far)) return false;
  if (!slab64(a.zz, a.o.z, a.inv.z, __ldg(&b->lo[2]), __ldg(&b->hi[2]), &near, &far)) return false;
  *near_out = near;
  return true;
}

// A leaf's primitives in Order; each accepted hit becomes the closest.
__device__ __forceinline__ void leaf64(const SceneView& sv, const BinNode* __restrict__ b, D3 o, D3 d, double tmin,
                                       double* closest, int* best) {
  const int s0 = __ldg(&b->start), cnt = __ldg(&b->count);
  for (int k = 0; k < cnt; k++) {
    const int s = s0 + k;
    const bool sphere = __ldg(reinterpret_cast<const float*>(sv.tri + 3 * (size_t)s + 2) + 3) < 0.0f;
    double t;
    const bool hit = sphere ? sphere_hit64(sv.slot64 + 9 * (size_t)s, o, d, tmin, *closest, &t)
                            : tri_hit64(sv.slot64 + 9 * (size_t)s, o, d, tmin, *closest, &t);
    if (hit) {
      *closest = t;
      *best = s;
    }
  }
}

// Returns the winning slot (-1: miss) and its distance.
__device__ int replay_closest(const SceneView& sv, const BinNode* __restrict__ bin, D3 o, D3 d, double tmin,
                              double tmax, double* t_out, unsigned* status) {
  Accel64 a;
  a.o = o;
  a.zx = fabs(d.x) < 1e-15;
  a.zy = fabs(d.y) < 1e-15;
  a.zz = fabs(d.z) < 1e-15;
  a.inv.x = a.zx ? 0.0 : __ddiv_rn(1.0, d.x);
  a.inv.y = a.zy ? 0.0 : __ddiv_rn(1.0, d.y);
  a.inv.z = a.zz ? 0.0 : __ddiv_rn(1.0, d.z);
  double closest = tmax;
  int best = -1;
  double root_near;
  if (!box64(bin, a, tmin, tmax, &root_near)) return -1;
  int sn[16];
  double sd[16];
  int dfs[kReplayDepth];
  int sp = 1;
  sn[0] = 0;
  sd[0] = root_near;
  while (sp > 0) {
    sp--;
    if (sd[sp] >= closest) continue;
    const BinNode* n = bin + sn[sp];
    if (__ldg(&n->count) > 0) {
      leaf64(sv, n, o, d, tmin, &closest, &best);
      continue;
    }
    const int l = __ldg(&n->left), r = __ldg(&n->right);
    double ln = 0.0, rn = 0.0;
    const bool lok = box64(bin + l, a, tmin, closest, &ln);
    const bool rok = box64(bin + r, a, tmin, closest, &rn);
    if (!lok && !rok) continue;
    if (sp + 2 > 16) {  // hitRecursive on the left child, then on the right one
      int dp = 0;
      if (rok) dfs[dp++] = r;
      if (lok) dfs[dp++] = l;
      while (dp > 0) {
        const BinNode* m = bin + dfs[--dp];
        double mn;
        if (!box64(m, a, tmin, closest, &mn)) continue;
        if (__ldg(&m->count) > 0) {
          leaf64(sv, m, o, d, tmin, &closest, &best);
          continue;
        }
        if (dp + 2 > kReplayDepth) {  // a tree deeper than the replay holds: report, never guess
          atomicOr(status, kStatusStackOverflow);
          return -1;
        }
        dfs[dp++] = __ldg(&m->right);
        dfs[dp++] = __ldg(&m->left);
      }
      continue;
    }
    if (lok && rok) {
      if (ln <= rn) {
        sn[sp] = r; sd[sp++] = rn;
        sn[sp] = l; sd[sp++] = ln;
      } else {
        sn[sp] = l; sd[sp++] = ln;
        sn[sp] = r; sd[sp++] = rn;
      }
    } else if (lok) {
      sn[sp] = l; sd[sp++] = ln;
    } else {
      sn[sp] = r; sd[sp++] = rn;
    }
  }
  *t_out = closest;
  return best;
}

__global__ void __launch_bounds__(128) k_tie_replay(SceneView sv, const BinNode* __restrict__ bin,
                                                    const float4* __restrict__ rays, int64_t n,
                                                    float* __restrict__ t_out, int32_t* __restrict__ prim_out,
                                                    unsigned* status, const unsigned* any_tie) {
  if (any_tie && !*any_tie) return;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (prim_out[i] != kTieMark) continue;
    const float4 a = __ldg(rays + 2 * i), b = __ldg(rays + 2 * i + 1);
    const D3 o{(double)a.x, (double)a.y, (double)a.z}, d{(double)b.x, (double)b.y, (double)b.z};
    double t = 0.0;
    const int s = replay_closest(sv, bin, o, d, (double)a.w, (double)b.w, &t, status);
    t_out[i] = s >= 0 ? __double2float_rn(t) : -1.0f;
    prim_out[i] = s >= 0 ? __ldg(sv.slot_prim + s) : -1;
  }
}

// ---- small batches: eight lanes per ray ------------------------------------------
// A batch that does not fill the chip with a ray per lane is bound by one ray's
// chain of node visits: eight box tests, the ordering of the hit children and
// the leaf's triangles one after another in one lane, and around the walk the
// separate passes' launches. Here eight lanes take a ray, a lane per child of
// the visited node and a lane per triangle of a leaf; the stack lies in shared
// memory, contenders in the lanes' registers, and the same kernel settles them in
// fp64 (and replays exact ties), so a call is one launch. 1,000 rays against
// 20,000 triangles, among other calls: 118 -> 31 us. Bound by latency: 18% of the issue
// slots, 6% of the warps resident, three waiting cycles on a load per instruction.
// A lane holds at most one contender: a primitive that may be the closest hit,
// with the lower end of its distance interval. `hi` is the least upper end of
// the certain ones; contenders beyond it are dropped. When more than eight
// remain, they are settled at once and the winner stays.
struct GroupBest {
  int slot;      // this lane's contender, -1: none
  float lo;      // lower end of its distance interval
  bool certain;  // it must pass its fp64 test
};

// Settles the group's contenders: every lane gets the winning slot (-1: none),
// its distance, and whether another contender shares it.
__device__ __forceinline__ int group_settle(const SceneView& sv, unsigned gm, const GroupBest& c, float hi, D3 o, D3 d,
                                            double tmin, double tmax, double* t_out, bool* tie, unsigned* status) {
  double t = INFINITY;
  int s = -1;
  if (c.slot >= 0 && !(c.lo > hi)) {
    double x;
    if (tri_hit64(sv.slot64 + 9 * (size_t)c.slot, o, d, tmin, tmax, &x)) {
      t = x;
      s = c.slot;
    } else if (c.certain) {
      atomicOr(status, kStatusBound);  // a certain hit must pass its fp64 test
    }
  }
  double best = t;
  int win = s;
#pragma unroll
  for (int o2 = 4; o2 > 0; o2 >>= 1) {
    const double y = __shfl_xor_sync(gm, best, o2);
    const int ys = __shfl_xor_sync(gm, win, o2);
    if (ys >= 0 && (win < 0 || y < best || (y == best && ys > win))) {
      best = y;
      win = ys;
    }
  }
  *tie = __popc(__ballot_sync(gm, s >= 0 && t == best)) > 1;
  *t_out = best;
  return win;
}

template <bool ANY, int MINB>
__global__ void __launch_bounds__(128, MINB) k_cast_group(SceneView sv, const BinNode* __restrict__ bin,
                                                    const float4* __restrict__ rays, int64_t n, int per_warp,
                                                    int stack, float* __restrict__ t_out, int32_t* __restrict__ prim_out,
                                                    uint8_t* __restrict__ occ_out, unsigned* status) {
  extern __shared__ uint2 group_stack[];
  const int lane = threadIdx.x & 31, g = lane >> 3, sub = lane & 7;
  if (g >= per_warp) return;  // few rays: fewer groups share a warp's issue slots
  const int64_t i = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp + g;
  if (i >= n) return;
  const unsigned gm = 0xffu << (8 * g);
  uint2* st = group_stack + ((threadIdx.x >> 5) * per_warp + g) * stack;
  const float4 ra = __ldg(rays + 2 * i), rb = __ldg(rays + 2 * i + 1);
  const Ray32 r = make_ray(ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w);
  const RayPre rp = ray_pre(r);
  const float tmax = rb.w;
  const D3 o{(double)r.ox, (double)r.oy, (double)r.oz}, d{(double)r.dx, (double)r.dy, (double)r.dz};
  const double tmin64 = (double)r.tmin, tmax64 = (double)tmax;
  // near and far bound arrays of a node by the direction's signs (node_children_fused)
  const int nxo = rp.ivx < 0.0f ? 56 : 48, nyo = rp.ivy < 0.0f ? 72 : 64, nzo = rp.ivz < 0.0f ? 88 : 80;
  const int fxo = 104 - nxo, fyo = 136 - nyo, fzo = 168 - nzo;
  float hi = tmax, tlim = widen(tmax);
  GroupBest c{-1, 0.0f, false};
  bool tie = false, occluded = false;
  int sp = 0;
  uint32_t ref = 0;
  while (ref != kEnd) {
    if (!(ref & kLeafBit)) {
      const char* nd = reinterpret_cast<const char*>(sv.nodes + ref);
      const float4 w0 = __ldg(reinterpret_cast<const float4*>(nd));
      const uint32_t child = __ldg(reinterpret_cast<const uint32_t*>(nd + 16) + sub);
      const uint8_t* q = reinterpret_cast<const uint8_t*>(nd) + sub;
      const uint32_t qnx = __ldg(q + nxo), qny = __ldg(q + nyo), qnz = __ldg(q + nzo);
      const uint32_t qfx = __ldg(q + fxo), qfy = __ldg(q + fyo), qfz = __ldg(q + fzo);
      // the conservative test of node_children_fused for this lane's child
      const uint32_t meta = __float_as_uint(w0.w);
      const float bx = __uint_as_float((meta & 0xffu) << 23) * rp.ivx * 32768.0f;
      const float by = __uint_as_float(((meta >> 8) & 0xffu) << 23) * rp.ivy * 32768.0f;
      const float bz = __uint_as_float(((meta >> 16) & 0xffu) << 23) * rp.ivz * 32768.0f;
      const float a1x = fmaf(w0.x, rp.ivx, rp.nox), a1y = fmaf(w0.y, rp.ivy, rp.noy), a1z = fmaf(w0.z, rp.ivz, rp.noz);
      const float ex = fmaf(fabsf(a1x) + fabsf(bx) + rp.mx, 5.0f * kU, 1e-30f);
      const float ey = fmaf(fabsf(a1y) + fabsf(by) + rp.my, 5.0f * kU, 1e-30f);
      const float ez = fmaf(fabsf(a1z) + fabsf(bz) + rp.mz, 5.0f * kU, 1e-30f);
      const float tnx = fmaf(__uint_as_float(0x3f800000u | qnx << 8), bx, a1x - bx - ex);
      const float tny = fmaf(__uint_as_float(0x3f800000u | qny << 8), by, a1y - by - ey);
      const float tnz = fmaf(__uint_as_float(0x3f800000u | qnz << 8), bz, a1z - bz - ez);
      const float tfx = fmaf(__uint_as_float(0x3f800000u | qfx << 8), bx, a1x - bx + ex);
      const float tfy = fmaf(__uint_as_float(0x3f800000u | qfy << 8), by, a1y - by + ey);
      const float tfz = fmaf(__uint_as_float(0x3f800000u | qfz << 8), bz, a1z - bz + ez);
      const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, r.tmin));
      const float tf = fminf(widen(fminf(fminf(tfx, tfy), tfz)), tlim);
      const bool hit = sub < (int)(meta >> 24) && tn <= tf;
      const unsigned m = __ballot_sync(gm, hit);
      const int hits = __popc(m);
      if (hits == 1) {
        ref = __shfl_sync(gm, child, __ffs(m) - 1);
        continue;
      }
      if (hits > 1) {
        if (sp + 7 > stack) {  // cannot happen: the host sizes the stack for the tree
          if (sub == 0) atomicOr(status, kStatusStackOverflow);
          break;
        }
        const float key = hit ? tn : __int_as_float(0x7f800000);
        int rank = 0;  // hit children nearer than this lane's
#pragma unroll
        for (int k = 1; k < 8; k++) {
          const float y = __shfl_xor_sync(gm, key, k);
          rank += (y < key || (y == key && (sub ^ k) < sub)) ? 1 : 0;
        }
        if (hit && rank > 0) st[sp + hits - 1 - rank] = make_uint2(child, __float_as_uint(tn));
        __syncwarp(gm);
        sp += hits - 1;
        ref = __shfl_sync(gm, child, __ffs(__ballot_sync(gm, hit && rank == 0)) - 1);
        continue;
      }
    } else {
      const int cnt = (int)((ref >> 27) & 15u) + 1, s0 = (int)(ref & kSlotMask);
      for (int k0 = 0; k0 < cnt; k0 += 8) {
        const int s = s0 + k0 + sub;
        int state = kMiss;
        float lo = 0.0f, up = 0.0f;
        if (k0 + sub < cnt) {
          const float4 A = __ldg(sv.tri + 3 * (size_t)s), E1 = __ldg(sv.tri + 3 * (size_t)s + 1),
                       E2 = __ldg(sv.tri + 3 * (size_t)s + 2);
          const TriClass tc = tri_classify(A, E1, E2, r, tmax, tlim);
          state = tc.state;
          lo = __fsub_rd(tc.t, tc.et);
          up = __fadd_ru(tc.t, tc.et);
          if (ANY && state == kMaybe) {
            double t;
            state = tri_hit64(sv.slot64 + 9 * (size_t)s, o, d, tmin64, tmax64, &t) ? kHit : kMiss;
          }
        }
        if (ANY) {
          if (__ballot_sync(gm, state == kHit)) occluded = true;
          if (occluded) break;
          continue;
        }
        unsigned fresh = __ballot_sync(gm, state != kMiss && !(lo > hi));
        if (!fresh) continue;
        float least = state == kHit ? up : hi;
#pragma unroll
        for (int k = 4; k > 0; k >>= 1) least = fminf(least, __shfl_xor_sync(gm, least, k));
        hi = fminf(hi, least);
        const bool take = state != kMiss && !(lo > hi);
        fresh = __ballot_sync(gm, take);
        const unsigned freel = __ballot_sync(gm, c.slot < 0 || c.lo > hi);
        if (__popc(fresh) > __popc(freel)) {  // no room: settle all of them now, the winner stays
          double wt, wf;
          bool t2, t3;
          int win = group_settle(sv, gm, c, hi, o, d, tmin64, tmax64, &wt, &t2, status);
          const int wfs = group_settle(sv, gm, GroupBest{take ? s : -1, lo, state == kHit}, hi, o, d, tmin64,
                                                tmax64, &wf, &t3, status);
          tie = tie || t2 || t3 || (win >= 0 && wfs >= 0 && wt == wf);
          if (wfs >= 0 && (win < 0 || wf < wt || (wf == wt && wfs > win))) {
            win = wfs;
            wt = wf;
          }
          c.slot = sub == 0 ? win : -1;
          c.lo = win >= 0 ? __double2float_rd(wt) : 0.0f;
          c.certain = true;
          if (win >= 0) hi = fminf(hi, __double2float_ru(wt));
          tlim = widen(hi);
          continue;
        }
        // the k-th fresh primitive goes to the k-th free lane
        const bool mine = (freel >> lane & 1u) != 0;
        const int k = __popc(freel & ((1u << lane) - 1u));
        const int src = mine && k < __popc(fresh) ? (int)__fns(fresh, 0, k + 1) : lane;
        const int ns = __shfl_sync(gm, s, src);
        const float nlo = __shfl_sync(gm, lo, src);
        const int nst = __shfl_sync(gm, state, src);
        if (mine) {
          const bool got = k < __popc(fresh);
          c.slot = got ? ns : -1;
          c.lo = nlo;
          c.certain = got && nst == kHit;
        }
        tlim = widen(hi);
      }
      if (ANY && occluded) break;
    }
    // pop: the nearest pending node still within the bound, eight entries a look
    ref = kEnd;
    while (sp > 0) {
      const int at = sp - 1 - sub;
      const uint2 e = at >= 0 ? st[at] : make_uint2(kEnd, 0x7f800000u);
      const unsigned ok = __ballot_sync(gm, at >= 0 && __uint_as_float(e.y) <= tlim);
      if (ok) {
        const int src = __ffs(ok) - 1;
        ref = __shfl_sync(gm, e.x, src);
        sp -= src - 8 * g + 1;
        break;
      }
      sp -= 8;
    }
    if (sp < 0) sp = 0;
    __syncwarp(gm);  // the entries are read before the next visit overwrites them
  }
  if (ANY) {
    if (sub == 0) occ_out[i] = occluded ? 1 : 0;
    return;
  }
  double wt;
  bool t2;
  int win = group_settle(sv, gm, c, hi, o, d, tmin64, tmax64, &wt, &t2, status);
  if (sub != 0) return;
  if (win >= 0 && (tie || t2)) win = replay_closest(sv, bin, o, d, tmin64, tmax64, &wt, status);
  t_out[i] = win >= 0 ? __double2float_rn(wt) : -1.0f;
  prim_out[i] = win >= 0 ? __ldg(sv.slot_prim + win) : -1;
}

template <class K>
int persistent_blocks(K kernel) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 128, 0);
  return sms * (per > 0 ? per : 1);
}

SceneView view_of(const DeviceScene& s) {
  SceneView v;
  v.nodes = s.nodes;
  v.tri = s.tri;
  v.slot64 = s.slot64;
  v.snorm = s.snorm;
  v.slot_prim = s.slot_prim;
  return v;
}

// Occupancy variants: MINB = minimum resident 128-thread blocks per SM the
// register allocation must allow (1: unconstrained, 6: <= 80 registers,
// 8: <= 64 registers). Selected per context (bc_set_option "raycast_minblocks").
template <int STACK, int MINB>
cudaError_t closest_stack(const DeviceScene& s, const float4* rays, int64_t n, float* t, int32_t* p, unsigned* status,
                          unsigned long long* work, const int32_t* perm, cudaStream_t st) {
  const int64_t grid = (n + 127) / 128;
  if (s.has_spheres) {
    k_closest_exact<STACK, true, MINB><<<(unsigned)grid, 128, 0, st>>>(view_of(s), rays, n, t, p, status);
  } else {
    static int blocks = 0;
    if (!blocks) blocks = persistent_blocks(k_closest_exact_persistent<STACK, MINB>);
    cudaError_t e = cudaMemsetAsync(work, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    const int g = (int)std::min<int64_t>(blocks, (n + 127) / 128);
    k_closest_exact_persistent<STACK, MINB><<<g, 128, 0, st>>>(view_of(s), rays, n, t, p, status, work, perm);
  }
  return cudaGetLastError();
}

template <int STACK>
cudaError_t closest_split(const DeviceScene& s, const float4* rays, int64_t n, float* t, int32_t* p, unsigned* status,
                          unsigned long long* work, const int32_t* perm, void* rec_scratch, cudaStream_t st) {
  static int blocks = 0;
  if (!blocks) blocks = persistent_blocks(k_exact_walk<STACK>);
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms < 1) sms = 1;
  }
  const ExactRecords rec = exact_records(rec_scratch, n);
  cudaError_t e = cudaMemsetAsync(work, 0, sizeof(unsigned long long), st);
  if (!e) e = cudaMemsetAsync(rec.n_redo, 0, 2 * sizeof(unsigned long long), st);  // n_redo and n_tie
  if (e) return e;
  const int64_t grid = (n + 127) / 128;
  k_exact_walk<STACK><<<(int)std::min<int64_t>(blocks, grid), 128, 0, st>>>(view_of(s), rays, n, rec, status, work,
                                                                           perm);
  k_exact_settle<<<(int)std::min<int64_t>((int64_t)sms * 16, grid), 128, 0, st>>>(view_of(s), rays, n, rec, t, p,
                                                                                 status);
  k_closest_exact_list<STACK><<<sms * 4, 128, 0, st>>>(view_of(s), rays, rec, t, p, status);
  return cudaGetLastError();
}

template <int STACK>
cudaError_t any_split(const DeviceScene& s, const float4* rays, int64_t n, uint8_t* out, unsigned* status,
                      unsigned long long* work, void* rec_scratch, const int32_t* perm, cudaStream_t st) {
  static int blocks = 0;
  if (!blocks) blocks = persistent_blocks(k_any_walk<STACK>);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const AnyRecords rec = any_records(rec_scratch, n);
  cudaError_t e = cudaMemsetAsync(work, 0, sizeof(unsigned long long), st);
  if (!e) e = cudaMemsetAsync(rec.count, 0, sizeof(unsigned long long), st);
  if (e) return e;
  const int64_t grid = (n + 127) / 128;
  k_any_walk<STACK><<<(int)std::min<int64_t>(blocks, grid), 128, 0, st>>>(view_of(s), rays, n, out, rec, status, work, perm);
  k_any_settle<STACK><<<std::max(sms, 1) * 4, 128, 0, st>>>(view_of(s), rays, n, out, rec, status);
  return cudaGetLastError();
}

template <int STACK, int MINB>
cudaError_t any_stack(const DeviceScene& s, const float4* rays, int64_t n, uint8_t* out, unsigned* status,
                      cudaStream_t st) {
  const int64_t grid = (n + 127) / 128;
  if (s.has_spheres)
    k_any_exact<STACK, true, MINB><<<(unsigned)grid, 128, 0, st>>>(view_of(s), rays, n, out, status);
  else
    k_any_exact<STACK, false, MINB><<<(unsigned)grid, 128, 0, st>>>(view_of(s), rays, n, out, status);
  return cudaGetLastError();
}

template <int STACK>
cudaError_t closest_var(const DeviceScene& s, const float4* rays, int64_t n, float* t, int32_t* p, unsigned* status,
                        unsigned long long* work, int variant, const int32_t* perm, void* rec_scratch,
                        cudaStream_t st) {
  if (variant != 0 && rec_scratch && !s.has_spheres)
    return closest_split<STACK>(s, rays, n, t, p, status, work, perm, rec_scratch, st);
  if (variant == 0) {  // fast, not exact
    const int64_t grid = (n + 127) / 128;
    if (s.has_spheres) {
      k_closest_fast<STACK, true><<<(unsigned)grid, 128, 0, st>>>(view_of(s), rays, n, t, p, status);
    } else {
      static int blocks = 0;
      if (!blocks) blocks = persistent_blocks(k_closest_fast_persistent<STACK>);
      cudaError_t e = cudaMemsetAsync(work, 0, sizeof(unsigned long long), st);
      if (e != cudaSuccess) return e;
      const int g = (int)std::min<int64_t>(blocks, grid);
      k_closest_fast_persistent<STACK><<<g, 128, 0, st>>>(view_of(s), rays, n, t, p, status, work, perm);
    }
    return cudaGetLastError();
  }
  switch (variant) {
    case 6: return closest_stack<STACK, 6>(s, rays, n, t, p, status, work, perm, st);
    case 8: return closest_stack<STACK, 8>(s, rays, n, t, p, status, work, perm, st);
    default: return closest_stack<STACK, 1>(s, rays, n, t, p, status, work, perm, st);
  }
}

template <int STACK>
cudaError_t any_var(const DeviceScene& s, const float4* rays, int64_t n, uint8_t* out, unsigned* status, int variant,
                    unsigned long long* work, void* rec_scratch, const int32_t* perm, cudaStream_t st) {
  if (rec_scratch && work && !s.has_spheres)
    return any_split<STACK>(s, rays, n, out, status, work, rec_scratch, perm, st);
  switch (variant) {
    case 6: return any_stack<STACK, 6>(s, rays, n, out, status, st);
    case 8: return any_stack<STACK, 8>(s, rays, n, out, status, st);
    default: return any_stack<STACK, 1>(s, rays, n, out, status, st);
  }
}

}  // namespace

size_t any_record_bytes(int64_t n) {
  return 256 + up256((size_t)n * 8) + up256((size_t)n * 4) + up256((size_t)n * 4 * kPending);
}

size_t exact_record_bytes(int64_t n) {
  return 256 + 3 * up256((size_t)n * 4) + 2 * up256((size_t)n * 4 * kPending) + up256((size_t)n * 8);
}

size_t ray_order_bytes(int64_t n) {
  return (size_t)kKeyBins * 4 + (size_t)(kKeyBins / kScanBlock) * 4 + (size_t)n * 8 + 5 * 256;
}

// The least batch that is ordered. Ordering is worth more in a scene that caches hold
// less of: rays with random origins, us per closest-hit call as they come / ordered, at
// 262,144 / 524,288 / 786,432 / 1,048,575 rays: 200,000 triangles 702 / 724, 1041 / 1071,
// 1367 / 1398, 1712 / 1743; 500,000: 787 / 824, 1180 / 1190, 1549 / 1556, 1926 / 1913;
// 1,000,000: 814 / 826, 1220 / 1232, 1663 / 1606, 2016 / 1970; 2,000,000: 866 / 966,
// 1287 / 1279, 1768 / 1691, 2171 / 2074. A batch that the probe finds in an order of its own
// pays 30 us for the five launches (786,432 camera rays, 1,000,000 triangles: 740 -> 770;
// ordered they would take 1,860).
int64_t min_ordered_rays(const DeviceScene& s) { return s.n_prims >= 3 << 18 ? 5 << 17 : 1 << 20; }

// Spatially coherent ray order (see k_ray_keys) into order_scratch; *perm is
// left NULL when the batch is not ordered (no scratch, fewer than
// min_ordered_rays rays, 2^31 rays or more: the order holds 32-bit indices, or a
// scene with spheres, whose kernels read rays in order).
static cudaError_t order_rays(const DeviceScene& s, const float4* rays, int64_t n, void* order_scratch,
                              const int32_t** perm, cudaStream_t st) {
  *perm = nullptr;
  if (!order_scratch || n < min_ordered_rays(s) || n >= (int64_t(1) << 31) || s.has_spheres) return cudaSuccess;
  char* q = (char*)order_scratch;
  int32_t* bins = (int32_t*)q;
  int32_t* totals = (int32_t*)(q + (size_t)kKeyBins * 4);
  uint32_t* keys = (uint32_t*)(q + (size_t)kKeyBins * 4 + ((kKeyBins / kScanBlock) * 4 + 255) / 256 * 256);
  int32_t* pm = (int32_t*)((char*)keys + ((size_t)n * 4 + 255) / 256 * 256 + 256);  // the flag lies before it
  const float3 lo = make_float3(s.lo[0], s.lo[1], s.lo[2]);
  auto sc = [](float a, float b) { return b > a ? 64.0f / (b - a) : 0.0f; };
  const float3 scale = make_float3(sc(s.lo[0], s.hi[0]), sc(s.lo[1], s.hi[1]), sc(s.lo[2], s.hi[2]));
  const unsigned g = (unsigned)((n + 255) / 256);
  k_ray_probe<<<kKeyBins / (4 * kScanBlock), kScanBlock, 0, st>>>(rays, n, lo, scale, bins, pm - 1);
  k_ray_keys<<<g, 256, 0, st>>>(rays, n, lo, scale, keys, bins, pm - 1);
  k_scan_bins<<<kKeyBins / kScanBlock, kScanBlock, 0, st>>>(bins, totals, pm - 1);
  k_scan_totals<<<1, kScanBlock, 0, st>>>(totals);
  k_ray_scatter<<<g, 256, 0, st>>>(n, keys, bins, totals, pm, pm - 1);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  *perm = pm;
  return cudaSuccess;
}

// Which batches go to the groups: up to 32,768 rays for the closest hit and
// 65,536 for any hit. Measured
// against the walk and its passes, us per call at 1,000 / 16,000 / 32,000 /
// 64,000 rays: closest hit, 20,000 triangles 118 -> 31, 136 -> 85, 150 -> 139, 180 <
// 222; 1,000,000 triangles 286 -> 80, 312 -> 191, 438 -> 351, 493 < 520; any hit,
// 20,000 triangles 125 -> 29, 131 -> 63, 150 -> 102, 177 -> 167. Scenes with spheres
// keep the one-thread kernels (822 spheres, camera rays: faster from 1,000 rays on).
bool cast_in_groups(const DeviceScene& s, int64_t n, bool any) {
  return !s.has_spheres && n <= (any ? kGroupRaysAny : kGroupRaysClosest);
}

// Groups per warp: one while the warps fit the chip a few times, then two, then
// four; and past 8,192 rays 64 registers (spilling a little) for eight blocks per SM
// instead of four without spills. us per call, closest hit, 20,000 triangles, at 1,000 /
// 4,000 / 6,000 / 8,000 / 16,000 / 32,000 rays: one group a warp at four blocks 33 / 48 /
// 54 / 63 / 105 / 192, two 45 / 47 / 56 / 63 / 96 / 163, four 49 / 54 / 60 / 58 / 87 / 145;
// at eight blocks one 43 / 49 / 55 / 63 / 95 / 163, two 62 / 64 / 61 / 63 / 92 / 144, four
// 66 / 72 / 78 / 77 / 88 / 136. The lines lie by these; over 1,000,000 triangles one group
// at four blocks leads longer: 96 / 104 / 123 / 147 / 233 / 403, four 118 / 141 / 123 / 166 /
// 189 / 309, four at eight blocks 159 / 192 / 164 / 227 / 197 / 304.
template <bool ANY>
static cudaError_t cast_groups(const DeviceScene& s, const float4* rays, int64_t n, float* t, int32_t* p, uint8_t* occ,
                               unsigned* status, cudaStream_t st) {
  if (!s.bin || !stack_variant(s.stack_need)) return cudaErrorInvalidValue;
  const int per = n <= 4096 ? 1 : n <= 6144 ? 2 : 4, stack = s.stack_need + 8;
  const unsigned grid = (unsigned)((n + 4 * per - 1) / (4 * per));
  const size_t smem = (size_t)4 * per * stack * sizeof(uint2);
  if (n <= 8192)
    k_cast_group<ANY, 4><<<grid, 128, smem, st>>>(view_of(s), s.bin, rays, n, per, stack, t, p, occ, status);
  else
    k_cast_group<ANY, 8><<<grid, 128, smem, st>>>(view_of(s), s.bin, rays, n, per, stack, t, p, occ, status);
  return cudaGetLastError();
}

cudaError_t launch_raycast_closest(const DeviceScene& s, const float4* rays, int64_t n, float* t_out,
                                   int32_t* prim_out, unsigned* status, unsigned long long* work, int variant,
                                   bool split, void* order_scratch, void* rec_scratch, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (split && variant != 0 && cast_in_groups(s, n, false))
    return cast_groups<false>(s, rays, n, t_out, prim_out, nullptr, status, st);
  const int32_t* perm = nullptr;
  cudaError_t e = order_rays(s, rays, n, order_scratch, &perm, st);
  if (e) return e;
  switch (stack_variant(s.stack_need)) {
    case 64: e = closest_var<64>(s, rays, n, t_out, prim_out, status, work, variant, perm, rec_scratch, st); break;
    case 128: e = closest_var<128>(s, rays, n, t_out, prim_out, status, work, variant, perm, rec_scratch, st); break;
    case 256: e = closest_var<256>(s, rays, n, t_out, prim_out, status, work, variant, perm, rec_scratch, st); break;
    default: return cudaErrorInvalidValue;
  }
  if (e || variant == 0) return e;  // the plain fp32 form makes no tie promise
  if (!s.bin) return cudaErrorInvalidValue;  // every uploaded scene carries its binary tree
  // exact ties: rays the passes above marked are walked again as the reference walks them
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms < 1) sms = 1;
  }
  // (the split passes say whether there is any)
  const unsigned* any_tie =
      split && variant != 0 && rec_scratch && !s.has_spheres ? exact_records(rec_scratch, n).n_tie : nullptr;
  k_tie_replay<<<(int)std::min<int64_t>((int64_t)sms * 4, (n + 127) / 128), 128, 0, st>>>(view_of(s), s.bin, rays, n,
                                                                                        t_out, prim_out, status, any_tie);
  return cudaGetLastError();
}

cudaError_t launch_raycast_any(const DeviceScene& s, const float4* rays, int64_t n, uint8_t* out, unsigned* status,
                               int variant, bool split, unsigned long long* work, void* rec_scratch, void* order_scratch,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (split && cast_in_groups(s, n, true)) return cast_groups<true>(s, rays, n, nullptr, nullptr, out, status, st);
  const int32_t* perm = nullptr;
  if (rec_scratch) {  // only the split walk reads rays through the order
    cudaError_t e = order_rays(s, rays, n, order_scratch, &perm, st);
    if (e) return e;
  }
  switch (stack_variant(s.stack_need)) {
    case 64: return any_var<64>(s, rays, n, out, status, variant, work, rec_scratch, perm, st);
    case 128: return any_var<128>(s, rays, n, out, status, variant, work, rec_scratch, perm, st);
    case 256: return any_var<256>(s, rays, n, out, status, variant, work, rec_scratch, perm, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace bcgx
