// Photon map of the photon-mapping integrator on the device (PhotonMap,
// renderer.go:1623-1761) and the hit-surface helper shared by the photon
// tracer and the shading kernels.
//
// The reference keeps map[uint64][]int from photonCellKey to the indices of
// the photons in that cell, in append order. Here the photons are sorted by
// (cell key, append index), so every key's photons are one contiguous run in
// the reference's order; an open-addressing table maps a key to its run.
#pragma once
#include <stdint.h>

#include "sampling.cuh"
#include "trace_core.cuh"

namespace bcgx {

constexpr uint64_t kPhotonStream = 0xFFFFFFFFull;  // sample index of the photon emission streams
constexpr int kGatherMax = 64;                      // tracePhotonMapped gathers at most 64 photons

// Box of a photon map's cell runs and neighbour lists, written on the device with the map:
// the photons' cells and two more on each side, [g0, g0 + dim), so the 27
// neighbours of every cell within one cell of a photon's are in it;
// dim[0] == 0: neither (the hash lookup serves).
struct PhotonGrid {
  long long g0[3];
  int dim[3];
  int used;  // list entries taken
};

struct PhotonView {
  const float4* pos;                // photons in (cell key, append index) order: position
  const float4* nrm;                // facing normal at the deposit
  const float4* flux;               // flux
  const unsigned long long* ukey;   // distinct cell keys
  const int2* span;                 // (first photon, count) of each distinct key
  const int* table;                 // 0: empty slot, else distinct-key index + 1; null: empty map
  int mask;                         // table size - 1
  float cell, r2, pir2;             // cell size (= radius), radius^2, pi radius^2
  const PhotonGrid* grid;           // null: no runs and no neighbour lists
  const int* runs;                  // per cell of the box: the run its key's lookup gives, -1: none
  const int2* list;                 // per cell of the box: (first entry, entries); first < 0: none, use the hash
  const float4* lent;               // list entries, three float4 each: (position, normal x) (normal y z, flux x y) (flux z)
};

// photonCellKey (renderer.go:1636-1639): the int64 products wrap, as unsigned products do.
__host__ __device__ __forceinline__ unsigned long long photon_cell_key(long long x, long long y, long long z) {
  return ((unsigned long long)x * 73856093ull) ^ ((unsigned long long)y * 19349663ull) ^
         ((unsigned long long)z * 83492791ull);
}

__host__ __device__ __forceinline__ uint32_t photon_slot_hash(unsigned long long k) {
  return (uint32_t)((k * 0x9E3779B97F4A7C15ull) >> 32);
}

// Index of the distinct key `key`, or -1.
__device__ __forceinline__ int photon_cell_lookup(const PhotonView& pm, unsigned long long key) {
  uint32_t h = photon_slot_hash(key) & (uint32_t)pm.mask;
  for (int probe = 0; probe <= pm.mask; probe++) {
    const int t = __ldg(pm.table + h);
    if (t == 0) return -1;
    if (__ldg(pm.ukey + t - 1) == key) return t - 1;
    h = (h + 1) & (uint32_t)pm.mask;
  }
  return -1;
}

// One candidate of a gather (renderer.go:1745-1752): counted when it is within
// the radius of p and faces n (then *nd is its cosine).
__device__ __forceinline__ bool photon_counts(float r2, float3 P, float3 N, float3 p, float3 n, float* nd) {
  const float3 d = P - p;
  if (dot3(d, d) > r2) return false;
  *nd = dot3(N, n);
  return !(*nd <= 0.05f);
}
// The same with its flux; true once kGatherMax photons are counted.
__device__ __forceinline__ bool gather_photon(float r2, float3 P, float3 N, float3 F, float3 p, float3 n, float3& sum,
                                              int& count) {
  float nd;
  if (!photon_counts(r2, P, N, p, n, &nd)) return false;
  sum = fma3(F, nd, sum);
  return ++count >= kGatherMax;
}

// PhotonMap.gather(p, n, 64) (renderer.go:1730-1761): the 27 cells around p in
// (dz, dy, dx) order, each cell's photons in append order; a key shared by two
// of the cells is visited twice, as the reference's map lookups do.
// A cell's neighbour list holds exactly those photons in exactly that order, so
// a gather is one lookup (gather_run) and one contiguous run (gather_sum) whose
// loads do not depend on what the candidates before them gave. A cell without a list is
// gathered from the 27 runs, found with 27 loads in the lists' box and in the hash outside
// of it: in a map without lists, or with more than kLongRun candidates around it. Thousands
// lie around a few cells where a scene is much larger than its lit part; most of them are
// turned down for their normals, and the copies would not fit. Analytic spheres on a ground
// sphere of radius 1,000 (the gathers of 155 x 495, 3 samples, 14 bounces; 8,192 photons): 25.0
// ms from lists, where they found room, 12.7 ms from runs; 2,048 photons: 3.7 ms and 4.5.
constexpr int kLongRun = 2048;

// The run of p's cell: (first entry, entries), entries 0 where the gather is
// zero; first < 0: no list, the cells' runs serve. A point more than one cell outside
// the photons' cells has no photon within the radius (cells are one radius
// wide), so its gather is zero, as the loop would find.
__device__ __forceinline__ int2 gather_run(const PhotonView& pm, float3 p) {
  if (!pm.table) return make_int2(0, 0);
  const PhotonGrid* G = pm.grid;
  const int gx = G ? __ldg(&G->dim[0]) : 0;
  if (gx == 0) return make_int2(-1, 0);
  const int gy = __ldg(&G->dim[1]), gz = __ldg(&G->dim[2]);
  const long long lx = (long long)floorf(p.x / pm.cell) - __ldg(&G->g0[0]);
  const long long ly = (long long)floorf(p.y / pm.cell) - __ldg(&G->g0[1]);
  const long long lz = (long long)floorf(p.z / pm.cell) - __ldg(&G->g0[2]);
  if (lx < 1 || ly < 1 || lz < 1 || lx > gx - 2 || ly > gy - 2 || lz > gz - 2) return make_int2(0, 0);
  return pm.list ? __ldg(pm.list + (lz * gy + ly) * (long long)gx + lx) : make_int2(-1, 0);
}

// The candidates of p's 27 cells from their runs, or from hash lookups outside of the
// runs' box: AHEAD candidates' positions and normals in flight, flux for those that count.
// Bound by the latency of these loads: the scene above 23.1 ms with one, 16.7 with two, 12.7
// with four.
template <int AHEAD>
__device__ __forceinline__ float3 cells_sum(const PhotonView& pm, float3 p, float3 n, int& count) {
  const long long cx = (long long)floorf(p.x / pm.cell);
  const long long cy = (long long)floorf(p.y / pm.cell);
  const long long cz = (long long)floorf(p.z / pm.cell);
  // gather_run has found the cell at least one inside the box
  const PhotonGrid* G = pm.grid;
  const int gx = G ? __ldg(&G->dim[0]) : 0, gy = gx ? __ldg(&G->dim[1]) : 0;
  const int* runs = nullptr;
  if (gx) runs = pm.runs + ((cz - __ldg(&G->g0[2])) * gy + cy - __ldg(&G->g0[1])) * (long long)gx + cx - __ldg(&G->g0[0]);
  const float r2 = pm.r2;
  float3 sum = f3(0.0f, 0.0f, 0.0f);
#pragma unroll 1  // 27 copies of the body would not stay in the instruction cache
  for (int dz = -1; dz <= 1; dz++)
#pragma unroll 1
    for (int dy = -1; dy <= 1; dy++)
#pragma unroll 1
      for (int dx = -1; dx <= 1; dx++) {
        const int u = runs ? __ldg(runs + (dz * gy + dy) * (long long)gx + dx)
                           : photon_cell_lookup(pm, photon_cell_key(cx + dx, cy + dy, cz + dz));
        if (u < 0) continue;
        const int2 sp = __ldg(pm.span + u);
        const int end = sp.x + sp.y;
        for (int i = sp.x; i < end; i += AHEAD) {
          float4 P[AHEAD], N[AHEAD];
#pragma unroll
          for (int k = 0; k < AHEAD; k++) {
            P[k] = __ldg(pm.pos + min(i + k, end - 1));
            N[k] = __ldg(pm.nrm + min(i + k, end - 1));
          }
#pragma unroll
          for (int k = 0; k < AHEAD; k++) {
            float nd;
            if (i + k >= end || !photon_counts(r2, f3(P[k].x, P[k].y, P[k].z), f3(N[k].x, N[k].y, N[k].z), p, n, &nd)) continue;
            const float4 F = __ldg(pm.flux + i + k);
            sum = fma3(f3(F.x, F.y, F.z), nd, sum);
            if (++count >= kGatherMax) return sum;
          }
        }
      }
  return sum;
}

// Out of line: its registers stay out of gather_sum's loop.
static __device__ __noinline__ float3 gather_cells(const PhotonView& pm, float3 p, float3 n, int& count) {
  return cells_sum<4>(pm, p, n, count);
}

// INLINE: without a call (the one-kernel form, which would keep its whole state across it).
template <bool INLINE>
__device__ __forceinline__ float3 gather_sum(const PhotonView& pm, int2 run, float3 p, float3 n) {
  float3 sum = f3(0.0f, 0.0f, 0.0f);
  int count = 0;
  if (run.x < 0) {
    sum = INLINE ? cells_sum<2>(pm, p, n, count) : gather_cells(pm, p, n, count);
  } else {
    const float4* e = pm.lent + 3 * (size_t)run.x;
    for (int i = 0; i < run.y; i += 2) {  // two candidates in flight; the last pair may read the last entry twice
      const float4* e1 = e + 3 * (size_t)min(i + 1, run.y - 1);
      const float4 a0 = __ldg(e + 3 * (size_t)i), a1 = __ldg(e + 3 * (size_t)i + 1), a2 = __ldg(e + 3 * (size_t)i + 2);
      const float4 b0 = __ldg(e1), b1 = __ldg(e1 + 1), b2 = __ldg(e1 + 2);
      if (gather_photon(pm.r2, f3(a0.x, a0.y, a0.z), f3(a0.w, a1.x, a1.y), f3(a1.z, a1.w, a2.x), p, n, sum, count)) break;
      if (i + 1 < run.y &&
          gather_photon(pm.r2, f3(b0.x, b0.y, b0.z), f3(b0.w, b1.x, b1.y), f3(b1.z, b1.w, b2.x), p, n, sum, count))
        break;
    }
  }
  if (count == 0) return f3(0.0f, 0.0f, 0.0f);
  return sum * (1.0f / (pm.pir2 * (float)count));
}

__device__ __forceinline__ float3 photon_gather(const PhotonView& pm, float3 p, float3 n) {
  const int2 run = gather_run(pm, p);
  if (run.x >= 0 && run.y == 0) return f3(0.0f, 0.0f, 0.0f);
  return gather_sum<true>(pm, run, p, n);
}

// Hit point and facing normal of a closest hit at fp32 distance t: the
// sphereHitAccel normal (renderer.go:670-677) or the triangle's unit normal,
// flipped to face the ray (triHit, renderer.go:704-710). `nrm` is the slot's snorm word.
struct Surface {
  float3 p, N;
  float radius;  // sphere radius, 0 for triangles
  bool front, sphere;
};
__device__ __forceinline__ Surface hit_surface(const SceneView& sv, int slot, float4 nrm, float3 o, float3 d, float t) {
  Surface S;
  S.p = fma3(d, t, o);
  const float4 r2 = __ldg(sv.tri + 3 * slot + 2);
  S.sphere = r2.w < 0.0f;
  S.radius = 0.0f;
  if (S.sphere) {
    const float4 c = __ldg(sv.tri + 3 * slot);
    S.radius = c.w;
    const float3 outward = (S.p - f3(c.x, c.y, c.z)) * (1.0f / c.w);
    S.front = dot3(d, outward) < 0.0f;
    S.N = S.front ? outward : outward * -1.0f;
  } else {
    S.N = f3(nrm.x, nrm.y, nrm.z);
    S.front = dot3(d, S.N) < 0.0f;
    if (!S.front) S.N = S.N * -1.0f;
  }
  return S;
}

}  // namespace bcgx
