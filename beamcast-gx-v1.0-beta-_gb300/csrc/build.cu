// Binned SAH build on the device, reproducing buildNodeSAH
// (renderer.go:526-633) node for node: the same bounds, axis, bins, split
// costs and leaf rule in fp64 with the reference's operation order, the same
// in-place partition of Scene.Order, and the reference's pre-order node
// numbering (left subtree first).
//
// Two phases. Tasks (node ranges of the Order array) of more than kSmall
// elements are split a level at a time, all tasks of a level together (k_bins,
// k_split, k_rank, k_permute); a task of at most kSmall elements is finished by
// one warp, its whole subtree at once (k_small). Bounds use an order-preserving
// 64-bit key of each double so min/max run on integers; the key orders -0
// before +0, which is what Go's math.Min/Max do with signed zeros, and a
// min/max reduction is order-independent, so the boxes equal the sequential
// ones bit for bit.
//
// The partition loop of the reference (i from the left, j from the right;
// a right-side element at i is swapped with the element at j, j moves down)
// has a closed form, computed here with per-task prefix counts. With L the
// number of left-side elements of the range [s, e):
//   * a left element in [s, s+L) stays;
//   * the m-th right element in [s, s+L) (m = 1, 2, ...) goes to l_{m-1} - 1,
//     where l_k is the position of the k-th left element of [s+L, e) counted
//     from the end (l_0 = e), and that k-th left element goes to the position
//     of the k-th right element of [s, s+L);
//   * a right element at p in (s+L, e) goes to p - 1, and the one at s+L (if it
//     is a right element) to l_M - 1 (e - 1 if M = 0), M being the number of
//     right elements in [s, s+L).
// The median fallback of the reference is unreachable: the chosen split has
// both sides non-empty.
#include <algorithm>

#include "../../include/bc_host_scene.h"
#include "context.h"

namespace bcgx {
namespace {

constexpr int kBins = 32;
constexpr int kFields = 7;  // of a bin: count, box keys (min xyz, max xyz)
// Elements per chunk of the level kernels, one warp each: a task of 33 to 256
// elements is one chunk (its bins are stored without atomics).
constexpr int kChunk = 256;
// Largest task that k_small finishes: one lane per element.
constexpr int kSmall = 32;
constexpr int kThreads = 128;  // four chunk warps per block

__device__ __forceinline__ unsigned long long dkey(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double kdbl(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}
constexpr unsigned long long kKeyPosInf = 0xfff0000000000000ull;  // dkey(+inf): identity of min
constexpr unsigned long long kKeyNegInf = 0x000fffffffffffffull;  // dkey(-inf): identity of max, ~kKeyPosInf

// AABB.SurfaceArea (renderer.go:133-139), unfused.
__device__ __forceinline__ double box_area(const double* mn, const double* mx) {
  const double ex = __dsub_rn(mx[0], mn[0]), ey = __dsub_rn(mx[1], mn[1]), ez = __dsub_rn(mx[2], mn[2]);
  if (ex < 0 || ey < 0 || ez < 0) return 0;
  return __dmul_rn(2.0, __dadd_rn(__dadd_rn(__dmul_rn(ex, ey), __dmul_rn(ey, ez)), __dmul_rn(ez, ex)));
}
// The same of six keys (minima, maxima).
__device__ __forceinline__ double key_area(const unsigned long long* k) {
  const double mn[3] = {kdbl(k[0]), kdbl(k[1]), kdbl(k[2])}, mx[3] = {kdbl(k[3]), kdbl(k[4]), kdbl(k[5])};
  return box_area(mn, mx);
}

// The tasks of one level, and the chunks they are cut into.
struct Level {
  int32_t *s, *e, *node;        // range of Order, upper node
  int32_t* chunk0;              // first chunk
  unsigned long long* cb;       // 6 per task: centroid bounds as keys
  unsigned long long* bins;     // [field][bin] per task
  int32_t *ctask, *cidx;        // per chunk: task, index within the task
  int* T;                       // tasks
  int* C;                       // chunks
};

// Ends of the level-wise phase: a range that k_small finishes (kind 0 or 1: the
// Order buffer it lies in), or a leaf of any size (kLeafTerm).
constexpr int kLeafTerm = 2;

struct BuildArgs {
  const double* pbox;  // 6 per primitive (padded box)
  const double* cent;  // 3 per primitive
  int n, nb, leaf;
  int32_t* order[2];   // Order of a level and of the next
  int32_t* order_out;
  int32_t *rpos, *lpos;
  uint8_t* bin;
  Level lv[2];
  // per task of the level: decided by k_split
  int32_t *tbest, *tL, *tM;
  int32_t* tchild;         // 2 per task: the children's tasks of the next level, -1 for a terminal
  uint16_t* cbins;         // 32 per chunk: elements per bin
  int32_t* cleft;          // per chunk: left-side elements of the task before it
  // upper nodes (those of the level-wise phase), in order of creation
  double* nbox;            // 6 per node
  int32_t *nleft, *nparent, *nsize, *narrive;
  int* n_nodes;
  // terminals: range, upper node, kind, nodes of the finished subtree
  int32_t *zs, *ze, *znode, *zkind, *zsize;
  int* n_term;
  // nodes of the finished subtrees: those of the terminal [s, e) at 2s + k, in
  // order of creation; lidx is the node's pre-order index in its subtree,
  // lright that of its right child (the left one follows its parent)
  double* lbox;
  int32_t *lstart, *lcount, *lidx, *lright;
};

// Split axis and bin scale of a range from its centroid bounds; false when the
// extent is too small to split (renderer.go:485-493, 536-545).
__device__ __forceinline__ bool split_axis(const double cmn[3], const double cmx[3], int* axis_out, double* minc,
                                           double* inv) {
  double ext[3];
  for (int j = 0; j < 3; j++) ext[j] = __dsub_rn(cmx[j], cmn[j]);
  int axis = 0;  // largestAxis
  if (ext[1] > ext[0] && ext[1] >= ext[2]) axis = 1;
  else if (ext[2] > ext[0] && ext[2] > ext[1]) axis = 2;
  const double axis_extent = axis == 0 ? ext[0] : (axis == 1 ? ext[1] : ext[2]);
  *axis_out = axis;
  *minc = axis == 0 ? cmn[0] : (axis == 1 ? cmn[1] : cmn[2]);
  if (axis_extent < 1e-12) return false;
  *inv = __ddiv_rn(1.0, axis_extent);
  return true;
}
__device__ __forceinline__ bool task_axis(const unsigned long long* cb, int* axis, double* minc, double* inv) {
  double mn[3], mx[3];
  for (int j = 0; j < 3; j++) {
    mn[j] = kdbl(cb[j]);
    mx[j] = kdbl(cb[3 + j]);
  }
  return split_axis(mn, mx, axis, minc, inv);
}

__device__ __forceinline__ int bin_of(double c, double minc, double inv, int nb) {
  const double x = __dmul_rn(__dmul_rn(__dsub_rn(c, minc), inv), (double)nb);
  int b = (int)x;  // truncation toward zero, as Go's int()
  return b < 0 ? 0 : (b >= nb ? nb - 1 : b);
}

__device__ __forceinline__ unsigned long long warp_min64(unsigned long long v) {
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Order before the first split, and the identities of the root's bounds.
__global__ void k_start(int n, int32_t* __restrict__ order, unsigned long long* __restrict__ keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) order[i] = i;
  if (i < 12) keys[i] = (i % 6) < 3 ? kKeyPosInf : kKeyNegInf;
}

// The root's box and centroid bounds into keys[12] (box min, box max, centroid min,
// centroid max).
__global__ void __launch_bounds__(256) k_root_bounds(const double* __restrict__ pbox, const double* __restrict__ cent,
                                                     int n, unsigned long long* keys) {
  unsigned long long m[12];  // maxima as complements, so every field is a minimum
#pragma unroll
  for (int j = 0; j < 12; j++) m[j] = kKeyPosInf;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
      m[j] = min(m[j], dkey(pbox[6 * (size_t)q + j]));
      m[3 + j] = min(m[3 + j], ~dkey(pbox[6 * (size_t)q + 3 + j]));
      const unsigned long long ck = dkey(cent[3 * (size_t)q + j]);
      m[6 + j] = min(m[6 + j], ck);
      m[9 + j] = min(m[9 + j], ~ck);
    }
  }
#pragma unroll
  for (int j = 0; j < 12; j++) {
    const unsigned long long v = warp_min64(m[j]);
    if ((threadIdx.x & 31) == 0) {
      if ((j % 6) < 3) atomicMin(&keys[j], v);
      else atomicMax(&keys[j], ~v);
    }
  }
}

// The root as the only task of level 0 (more than kSmall elements), or as the only terminal.
__global__ void k_root_task(BuildArgs a, const unsigned long long* keys) {
  const int chunks = (a.n + kChunk - 1) / kChunk;
  const bool small = a.n <= kSmall;
  const Level& lv = a.lv[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (int j = 0; j < 6; j++) a.nbox[j] = kdbl(keys[j]);
    a.nleft[0] = -1;
    a.nparent[0] = -1;
    a.narrive[0] = 0;
    if (small) {
      a.zs[0] = 0;
      a.ze[0] = a.n;
      a.znode[0] = 0;
      a.zkind[0] = 0;
    } else {
      lv.s[0] = 0;
      lv.e[0] = a.n;
      lv.node[0] = 0;
      lv.chunk0[0] = 0;
      for (int j = 0; j < 6; j++) lv.cb[j] = keys[6 + j];
    }
    *lv.T = small ? 0 : 1;
    *lv.C = small ? 0 : chunks;
    *a.n_nodes = 1;
    *a.n_term = small ? 1 : 0;
  }
  if (small) return;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < chunks; c += gridDim.x * blockDim.x) {
    lv.ctask[c] = 0;
    lv.cidx[c] = c;
  }
  if (blockIdx.x == 0)
    for (int j = threadIdx.x; j < kFields * kBins; j += blockDim.x)
      lv.bins[j] = j < kBins ? 0ull : (j < 4 * kBins ? kKeyPosInf : kKeyNegInf);
}

// Bins of every chunk (one warp each): element counts and boxes in shared
// memory, merged into the task's bins. The level reads each element's Order
// entry, box and centroid once: 76 B per element, gathered.
__global__ void __launch_bounds__(kThreads) k_bins(BuildArgs a, int cur) {
  __shared__ unsigned long long sb[kThreads / 32][6][kBins + 1];
  __shared__ int sc[kThreads / 32][kBins];
  const Level& lv = a.lv[cur];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // k_split of this level fills the next one
    *a.lv[cur ^ 1].T = 0;
    *a.lv[cur ^ 1].C = 0;
  }
  const int total = *lv.C;
  const int32_t* __restrict__ order = a.order[cur];
  for (int c = blockIdx.x * (kThreads / 32) + w; c < total; c += gridDim.x * (kThreads / 32)) {
    const int k = lv.ctask[c];
    const int s = lv.s[k], e = lv.e[k];
    int axis;
    double minc, inv;
    if (!task_axis(lv.cb + 6 * (size_t)k, &axis, &minc, &inv)) continue;  // a leaf
#pragma unroll
    for (int f = 0; f < 6; f++) sb[w][f][lane] = f < 3 ? kKeyPosInf : kKeyNegInf;
    sc[w][lane] = 0;
    __syncwarp();
    const int p0 = s + lv.cidx[c] * kChunk, p1 = min(e, p0 + kChunk);
    for (int p = p0 + lane; p < p1; p += 32) {
      const int q = order[p];
      const int b = bin_of(a.cent[3 * (size_t)q + axis], minc, inv, a.nb);
      a.bin[p] = (uint8_t)b;
      atomicAdd(&sc[w][b], 1);
#pragma unroll
      for (int j = 0; j < 3; j++) {
        atomicMin(&sb[w][j][b], dkey(a.pbox[6 * (size_t)q + j]));
        atomicMax(&sb[w][3 + j][b], dkey(a.pbox[6 * (size_t)q + 3 + j]));
      }
    }
    __syncwarp();
    const int cnt = sc[w][lane];
    a.cbins[kBins * (size_t)c + lane] = (uint16_t)cnt;
    unsigned long long* tb = lv.bins + (size_t)k * kFields * kBins + lane;
    if (e - s <= kChunk) {  // the task's only chunk
      tb[0] = (unsigned long long)cnt;
#pragma unroll
      for (int f = 0; f < 6; f++) tb[(f + 1) * kBins] = sb[w][f][lane];
    } else if (cnt > 0) {
      atomicAdd(&tb[0], (unsigned long long)cnt);
#pragma unroll
      for (int f = 0; f < 6; f++) {
        if (f < 3) atomicMin(&tb[(f + 1) * kBins], sb[w][f][lane]);
        else atomicMax(&tb[(f + 1) * kBins], sb[w][f][lane]);
      }
    }
    __syncwarp();
  }
}

// One block per task. Its first warp (lane = bin) finds the split of least SAH
// cost (renderer.go:566-604) from prefix and suffix scans of the bins, or makes
// the task a leaf, and creates the children: their boxes are the two sides'
// unions. The block then turns the chunks' bin counts into left counts before
// each chunk, and lists the chunks of the children.
__global__ void k_split(BuildArgs a, int cur) {
  __shared__ int sh_best, sh_base, warp_sum[8];
  __shared__ int sh_child[2], sh_lo[2], sh_hi[2], sh_chunk[2];
  const Level& lv = a.lv[cur];
  const Level& nx = a.lv[cur ^ 1];
  const int T = *lv.T;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = blockIdx.x; k < T; k += gridDim.x) {
    const int s = lv.s[k], e = lv.e[k], cnt = e - s;
    if (w == 0) {
      const int node = lv.node[k];
      int axis, best = -1, L = 0;
      double minc, inv;
      if (task_axis(lv.cb + 6 * (size_t)k, &axis, &minc, &inv)) {
        const unsigned long long* tb = lv.bins + (size_t)k * kFields * kBins + lane;
        int lc = (int)tb[0];
        unsigned long long lk[6], rk[6];
#pragma unroll
        for (int f = 0; f < 6; f++) lk[f] = rk[f] = lane < a.nb ? tb[(f + 1) * kBins] : (f < 3 ? kKeyPosInf : kKeyNegInf);
        if (lane >= a.nb) lc = 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int yc = __shfl_up_sync(0xffffffffu, lc, o);
          if (lane >= o) lc += yc;
#pragma unroll
          for (int f = 0; f < 6; f++) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, lk[f], o), z = __shfl_down_sync(0xffffffffu, rk[f], o);
            if (lane >= o) lk[f] = f < 3 ? min(lk[f], y) : max(lk[f], y);
            if (lane + o < 32) rk[f] = f < 3 ? min(rk[f], z) : max(rk[f], z);
          }
        }
#pragma unroll
        for (int f = 0; f < 6; f++) rk[f] = __shfl_down_sync(0xffffffffu, rk[f], 1);  // the bins above this lane's
        double cost = INFINITY;
        if (lane < a.nb - 1 && lc > 0 && lc < cnt)
          cost = __dadd_rn(__dmul_rn(key_area(lk), (double)lc), __dmul_rn(key_area(rk), (double)(cnt - lc)));
        // costs are not negative: their bit patterns order as they do
        const bool valid = cost < INFINITY;
        const unsigned long long ck = valid ? (unsigned long long)__double_as_longlong(cost) : ~0ull;
        const unsigned long long cmin = warp_min64(ck);
        const unsigned m = __ballot_sync(0xffffffffu, valid && ck == cmin);
        if (m) {
          best = __ffs(m) - 1;  // the first bin of least cost
          L = __shfl_sync(0xffffffffu, lc, best);
          const double* nb6 = a.nbox + 6 * (size_t)node;
          const double leaf_cost = __dmul_rn(box_area(nb6, nb6 + 3), (double)cnt);
          if (cnt <= a.leaf * 2 && __longlong_as_double((long long)cmin) >= __dmul_rn(leaf_cost, 0.98)) best = -1;
        }
        if (best >= 0) {
          int id = 0;
          if (lane == 0) id = atomicAdd(a.n_nodes, 2);
          id = __shfl_sync(0xffffffffu, id, 0);
          if (lane == best)
            for (int f = 0; f < 6; f++) {
              a.nbox[6 * (size_t)id + f] = kdbl(lk[f]);
              a.nbox[6 * (size_t)id + 6 + f] = kdbl(rk[f]);
            }
          if (lane == 0) a.nleft[node] = id;
          if (lane < 2) {  // the children: lane 0 the left one
            const int cs = lane == 0 ? s : s + L, ce = lane == 0 ? s + L : e, cn = ce - cs;
            a.nleft[id + lane] = -1;
            a.nparent[id + lane] = node;
            a.narrive[id + lane] = 0;
            int child = -1, ch0 = 0;
            if (cn <= kSmall) {
              const int z = atomicAdd(a.n_term, 1);
              a.zs[z] = cs;
              a.ze[z] = ce;
              a.znode[z] = id + lane;
              a.zkind[z] = cur ^ 1;
            } else {
              child = atomicAdd(nx.T, 1);
              ch0 = atomicAdd(nx.C, (cn + kChunk - 1) / kChunk);
              nx.s[child] = cs;
              nx.e[child] = ce;
              nx.node[child] = id + lane;
              nx.chunk0[child] = ch0;
              for (int j = 0; j < 6; j++) nx.cb[6 * (size_t)child + j] = j < 3 ? kKeyPosInf : kKeyNegInf;
            }
            a.tchild[2 * k + lane] = child;
            sh_child[lane] = child;
            sh_lo[lane] = cs;
            sh_hi[lane] = ce;
            sh_chunk[lane] = ch0;
          }
        }
      }
      if (best < 0 && lane == 0) {  // a leaf; k_permute copies its elements out
        const int z = atomicAdd(a.n_term, 1);
        a.zs[z] = s;
        a.ze[z] = e;
        a.znode[z] = node;
        a.zkind[z] = kLeafTerm;
      }
      if (lane == 0) {
        a.tbest[k] = best;
        a.tL[k] = L;
        a.tM[k] = 0;
        sh_best = best;
        sh_base = 0;
      }
    }
    __syncthreads();
    const int best = sh_best;
    if (best >= 0) {
      const int chunks = (cnt + kChunk - 1) / kChunk, c0 = lv.chunk0[k];
      if (chunks == 1) {
        if (threadIdx.x == 0) a.cleft[c0] = 0;
      } else {
        for (int base = 0; base < chunks; base += blockDim.x) {  // left counts before each chunk
          const int j = base + threadIdx.x;
          int v = 0;
          if (j < chunks) {
            const uint4* cb = reinterpret_cast<const uint4*>(a.cbins + kBins * (size_t)(c0 + j));
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const uint4 x = cb[q];
              const unsigned u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
              for (int t = 0; t < 4; t++) {
                const int b = 8 * q + 2 * t;
                if (b <= best) v += (int)(u[t] & 0xffffu);
                if (b + 1 <= best) v += (int)(u[t] >> 16);
              }
            }
          }
          int x = v;
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
          }
          if (lane == 31) warp_sum[w] = x;
          __syncthreads();
          int below = sh_base, all = 0;
          for (int q = 0; q < (int)(blockDim.x >> 5); q++) {
            if (q < w) below += warp_sum[q];
            all += warp_sum[q];
          }
          if (j < chunks) a.cleft[c0 + j] = below + x - v;
          __syncthreads();
          if (threadIdx.x == 0) sh_base += all;
          __syncthreads();
        }
      }
      for (int side = 0; side < 2; side++) {
        const int child = sh_child[side];
        if (child < 0) continue;
        const int cc = (sh_hi[side] - sh_lo[side] + kChunk - 1) / kChunk;
        for (int j = threadIdx.x; j < cc; j += blockDim.x) {
          nx.ctask[sh_chunk[side] + j] = child;
          nx.cidx[sh_chunk[side] + j] = j;
        }
        if (cc > 1)  // the chunks' bins are merged into these; an only chunk stores its own
          for (int j = threadIdx.x; j < kFields * kBins; j += blockDim.x)
            nx.bins[(size_t)child * kFields * kBins + j] = j < kBins ? 0ull : (j < 4 * kBins ? kKeyPosInf : kKeyNegInf);
      }
    }
    __syncthreads();
  }
}

// The tables of misplaced elements, and M (one warp per chunk).
__global__ void __launch_bounds__(kThreads) k_rank(BuildArgs a, int cur) {
  const Level& lv = a.lv[cur];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int total = *lv.C;
  for (int c = blockIdx.x * (kThreads / 32) + w; c < total; c += gridDim.x * (kThreads / 32)) {
    const int k = lv.ctask[c], best = a.tbest[k];
    if (best < 0) continue;
    const int s = lv.s[k], e = lv.e[k], L = a.tL[k];
    const int p0 = s + lv.cidx[c] * kChunk, p1 = min(e, p0 + kChunk);
    int base = a.cleft[c];
    for (int p = p0; p < p1; p += 32) {
      const int pp = p + lane;
      const bool in = pp < p1;
      const bool left = in && a.bin[pp] <= best;
      const unsigned m = __ballot_sync(0xffffffffu, left);
      const int lb = base + __popc(m & ((1u << lane) - 1u));
      if (in) {
        if (pp == s + L) a.tM[k] = L - lb;
        if (pp < s + L && !left) a.rpos[s + ((pp - s) - lb)] = pp;  // misplaced right, rank (pp - s) - lb
        if (pp >= s + L && left) a.lpos[s + (L - lb) - 1] = pp;     // left beyond L, rank L - lb from the end
      }
      base += __popc(m);
    }
  }
}

// The reference's partition as a permutation into the next level's Order, and
// the centroid bounds of the children that are tasks of the next level (one
// warp per chunk).
__global__ void __launch_bounds__(kThreads) k_permute(BuildArgs a, int cur) {
  const Level& lv = a.lv[cur];
  const Level& nx = a.lv[cur ^ 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int total = *lv.C;
  const int32_t* __restrict__ order = a.order[cur];
  int32_t* __restrict__ next = a.order[cur ^ 1];
  for (int c = blockIdx.x * (kThreads / 32) + w; c < total; c += gridDim.x * (kThreads / 32)) {
    const int k = lv.ctask[c], best = a.tbest[k];
    const int s = lv.s[k], e = lv.e[k];
    const int p0 = s + lv.cidx[c] * kChunk, p1 = min(e, p0 + kChunk);
    if (best < 0) {
      for (int p = p0 + lane; p < p1; p += 32) a.order_out[p] = order[p];
      continue;
    }
    const int L = a.tL[k], M = a.tM[k];
    const int cl = a.tchild[2 * k], cr = a.tchild[2 * k + 1];
    unsigned long long m[12];  // left and right centroid bounds, maxima as complements
#pragma unroll
    for (int j = 0; j < 12; j++) m[j] = kKeyPosInf;
    int base = a.cleft[c];
    for (int p = p0; p < p1; p += 32) {
      const int pp = p + lane;
      const bool in = pp < p1;
      const bool left = in && a.bin[pp] <= best;
      const unsigned bal = __ballot_sync(0xffffffffu, left);
      const int lb = base + __popc(bal & ((1u << lane) - 1u));
      base += __popc(bal);
      if (!in) continue;
      int dest;
      if (left) {
        dest = pp < s + L ? pp : a.rpos[s + (L - lb) - 1];
      } else if (pp < s + L) {
        const int m0 = (pp - s) - lb;  // right elements of [s, pp)
        dest = (m0 == 0 ? e : a.lpos[s + m0 - 1]) - 1;
      } else if (pp == s + L) {
        dest = (M > 0 ? a.lpos[s + M - 1] : e) - 1;
      } else {
        dest = pp - 1;
      }
      const int q = order[pp];
      next[dest] = q;
      if (left ? cl >= 0 : cr >= 0) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const unsigned long long key = dkey(a.cent[3 * (size_t)q + j]);
          m[j] = min(m[j], left ? key : kKeyPosInf);
          m[3 + j] = min(m[3 + j], left ? ~key : kKeyPosInf);
          m[6 + j] = min(m[6 + j], left ? kKeyPosInf : key);
          m[9 + j] = min(m[9 + j], left ? kKeyPosInf : ~key);
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 12; j++) {
      const int child = j < 6 ? cl : cr;
      if (child < 0) continue;  // uniform over the warp
      const unsigned long long v = warp_min64(m[j]);
      if (lane == 0) {
        unsigned long long* dst = nx.cb + 6 * (size_t)child + j % 6;
        if (j % 6 < 3) atomicMin(dst, v);
        else atomicMax(dst, ~v);
      }
    }
  }
}

// One warp finishes a terminal of at most kSmall elements, one lane per
// position of the range, the nodes of a depth all at once: a lane's node is the
// segment [s, e) it lies in. Every lane loops over its segment for the centroid
// bounds and takes its own bin as a split candidate: only occupied bins can be
// the first split of least cost (an empty one costs what the occupied one below
// it costs), so the candidates of a segment are its elements' bins, and a
// second loop gives each candidate's two boxes. Quadratic in the segment, but
// without bins, scans or launches: over the million-triangle build the
// level-wise kernels spent 18 of 25 ms on tasks of at most 32 elements, a
// 256-thread block each.
// A node's pre-order index is the number of nodes that start before it plus
// its rank among those that start with it (its ancestors); lane i counts the
// nodes that start at position i.
__global__ void __launch_bounds__(kThreads) k_small(BuildArgs a) {
  constexpr int kW = kThreads / 32;
  __shared__ unsigned long long sk[kW][6][kSmall + 1];  // box keys, maxima as complements
  __shared__ double sc[kW][3][kSmall + 1];
  __shared__ int sid[kW][kSmall];                       // primitive of each loaded element
  __shared__ uint8_t sord[kW][kSmall], srp[kW][kSmall], slp[kW][kSmall], sbin[kW][kSmall];
  __shared__ uint8_t ns[kW][2 * kSmall], nrank[kW][2 * kSmall], nrs[kW][2 * kSmall];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int terms = *a.n_term;
  for (int z = blockIdx.x * kW + w; z < terms; z += gridDim.x * kW) {
    const int g0 = a.zs[z], kind = a.zkind[z], n = a.ze[z] - g0;
    const size_t out = 2 * (size_t)g0;
    if (kind == kLeafTerm) {
      if (lane < 6) a.lbox[6 * out + lane] = a.nbox[6 * (size_t)a.znode[z] + lane];
      if (lane == 0) {
        a.lstart[out] = g0;
        a.lcount[out] = n;
        a.lidx[out] = 0;
        a.lright[out] = -1;
        a.zsize[z] = 1;
      }
      continue;
    }
    __syncwarp();
    if (lane < n) {
      const int q = a.order[kind][g0 + lane];
      sid[w][lane] = q;
      sord[w][lane] = (uint8_t)lane;
#pragma unroll
      for (int j = 0; j < 3; j++) {
        sk[w][j][lane] = dkey(a.pbox[6 * (size_t)q + j]);
        sk[w][3 + j][lane] = ~dkey(a.pbox[6 * (size_t)q + 3 + j]);
        sc[w][j][lane] = a.cent[3 * (size_t)q + j];
      }
    }
    __syncwarp();
    int s = 0, e = n;           // this lane's segment
    bool open = lane < n;       // its node is still to be made
    int started = 0, n_nodes = 0;
    while (__any_sync(0xffffffffu, open)) {
      const int cnt = e - s;
      bool split = open && cnt > a.leaf;
      int axis = 0;
      double minc = 0.0, inv = 0.0;
      if (split) {
        unsigned long long lo[3] = {kKeyPosInf, kKeyPosInf, kKeyPosInf}, hi[3] = {kKeyPosInf, kKeyPosInf, kKeyPosInf};
        for (int k = s; k < e; k++) {
          const int el = sord[w][k];
#pragma unroll
          for (int j = 0; j < 3; j++) {
            const unsigned long long ck = dkey(sc[w][j][el]);
            lo[j] = min(lo[j], ck);
            hi[j] = min(hi[j], ~ck);
          }
        }
        double mn[3], mx[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
          mn[j] = kdbl(lo[j]);
          mx[j] = kdbl(~hi[j]);
        }
        split = split_axis(mn, mx, &axis, &minc, &inv);
      }
      int b = 0;
      if (split) b = bin_of(sc[w][axis][sord[w][lane]], minc, inv, a.nb);
      sbin[w][lane] = (uint8_t)b;
      __syncwarp();
      unsigned long long lk[6], rk[6];
#pragma unroll
      for (int f = 0; f < 6; f++) lk[f] = rk[f] = kKeyPosInf;
      int lc = 0;
      if (open)
        for (int k = s; k < e; k++) {
          const int el = sord[w][k];
          const bool left = sbin[w][k] <= b;
          lc += left ? 1 : 0;
#pragma unroll
          for (int f = 0; f < 6; f++) {
            const unsigned long long v = sk[w][f][el];
            if (left) lk[f] = min(lk[f], v);
            else rk[f] = min(rk[f], v);
          }
        }
      double cost = INFINITY;
      if (split && lc < cnt) {
        unsigned long long l6[6], r6[6];
#pragma unroll
        for (int f = 0; f < 6; f++) {
          l6[f] = f < 3 ? lk[f] : ~lk[f];
          r6[f] = f < 3 ? rk[f] : ~rk[f];
        }
        cost = __dadd_rn(__dmul_rn(key_area(l6), (double)lc), __dmul_rn(key_area(r6), (double)(cnt - lc)));
      }
      // the segment's least cost and, among its candidates, the lowest bin
      const bool valid = cost < INFINITY;
      unsigned long long ck = valid ? (unsigned long long)__double_as_longlong(cost) : ~0ull;
      int cb = valid ? b : kBins, cl = lc;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {  // segmented inclusive scan: the segment's last lane gets its minimum
        const unsigned long long yk = __shfl_up_sync(0xffffffffu, ck, o);
        const int yb = __shfl_up_sync(0xffffffffu, cb, o), yl = __shfl_up_sync(0xffffffffu, cl, o);
        if (lane - o >= s && (yk < ck || (yk == ck && yb < cb))) {
          ck = yk;
          cb = yb;
          cl = yl;
        }
      }
      const int last = open ? e - 1 : lane;
      ck = __shfl_sync(0xffffffffu, ck, last);
      cb = __shfl_sync(0xffffffffu, cb, last);
      const int L = __shfl_sync(0xffffffffu, cl, last);
      split = split && cb < kBins;
      // every lane holds its node's box: the union of its candidate's sides
#pragma unroll
      for (int f = 0; f < 6; f++) lk[f] = min(lk[f], rk[f]);
      if (split && cnt <= a.leaf * 2) {
        unsigned long long n6[6];
#pragma unroll
        for (int f = 0; f < 6; f++) n6[f] = f < 3 ? lk[f] : ~lk[f];
        const double leaf_cost = __dmul_rn(key_area(n6), (double)cnt);
        if (__longlong_as_double((long long)ck) >= __dmul_rn(leaf_cost, 0.98)) split = false;
      }
      // the nodes of this depth, one per open segment
      const bool head = open && lane == s;
      const unsigned heads = __ballot_sync(0xffffffffu, head);
      if (head) {
        const int j = n_nodes + __popc(heads & ((1u << lane) - 1u));
        ns[w][j] = (uint8_t)s;
        nrank[w][j] = (uint8_t)started;
        nrs[w][j] = (uint8_t)(split ? s + L : 255);
        started++;
#pragma unroll
        for (int f = 0; f < 6; f++) a.lbox[6 * (out + j) + f] = kdbl(f < 3 ? lk[f] : ~lk[f]);
        a.lstart[out + j] = split ? 0 : g0 + s;
        a.lcount[out + j] = split ? 0 : cnt;
      }
      n_nodes += __popc(heads);
      // partition of the split segments
      const bool left = split && b <= cb;
      const unsigned m = __ballot_sync(0xffffffffu, left);
      const unsigned seg = (e >= 32 ? 0xffffffffu : ((1u << e) - 1u)) & ~((1u << s) - 1u);
      const int lb = __popc(m & seg & ((1u << lane) - 1u));
      const int lefts_in = __popc(m & seg & ((s + L >= 32 ? 0xffffffffu : ((1u << (s + L)) - 1u))));
      const int M = L - lefts_in;
      if (split && lane < s + L && !left) srp[w][s + (lane - s) - lb] = (uint8_t)lane;
      if (split && lane >= s + L && left) slp[w][s + (L - lb) - 1] = (uint8_t)lane;
      const int el = lane < n ? sord[w][lane] : 0;
      __syncwarp();
      if (split) {
        int dest;
        if (left) {
          dest = lane < s + L ? lane : srp[w][s + (L - lb) - 1];
        } else if (lane < s + L) {
          const int m0 = (lane - s) - lb;
          dest = (m0 == 0 ? e : slp[w][s + m0 - 1]) - 1;
        } else if (lane == s + L) {
          dest = (M > 0 ? slp[w][s + M - 1] : e) - 1;
        } else {
          dest = lane - 1;
        }
        sord[w][dest] = (uint8_t)el;
        if (lane < s + L) e = s + L;
        else s = s + L;
      } else {
        open = false;
      }
      __syncwarp();
    }
    if (lane < n) a.order_out[g0 + lane] = sid[w][sord[w][lane]];
    int x = started;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int first = x - started;  // nodes that start before this position
    for (int j0 = 0; j0 < n_nodes; j0 += 32) {
      const int j = j0 + lane;
      const bool in = j < n_nodes;
      const int st = in ? ns[w][j] : 0, rs = in ? nrs[w][j] : 255;
      const int fs = __shfl_sync(0xffffffffu, first, st), fr = __shfl_sync(0xffffffffu, first, rs & 31);
      if (in) {
        a.lidx[out + j] = fs + nrank[w][j];
        a.lright[out + j] = rs == 255 ? -1 : fr;
      }
    }
    if (lane == 0) a.zsize[z] = n_nodes;
  }
}

// Subtree sizes of the upper nodes: each terminal climbs, the second child to
// arrive at a node sums and goes on.
__global__ void k_sizes(BuildArgs a) {
  const int terms = *a.n_term;
  for (int z = blockIdx.x * blockDim.x + threadIdx.x; z < terms; z += gridDim.x * blockDim.x) {
    int u = a.znode[z];
    a.nsize[u] = a.zsize[z];
    for (;;) {
      const int p = a.nparent[u];
      if (p < 0) break;
      __threadfence();
      if (atomicAdd(&a.narrive[p], 1) == 0) break;
      __threadfence();
      const int l = a.nleft[p];
      a.nsize[p] = 1 + __ldcg(a.nsize + l) + __ldcg(a.nsize + l + 1);
      u = p;
    }
  }
}

// Pre-order index of upper node u: on the way to the root, a left child adds
// one, a right child one and its sibling's subtree.
__device__ __forceinline__ int preorder(const BuildArgs& a, int u) {
  int d = 0;
  for (int p = a.nparent[u]; p >= 0; p = a.nparent[u]) {
    const int l = a.nleft[p];
    d += u == l ? 1 : 1 + a.nsize[l];
    u = p;
  }
  return d;
}

// The tree in the reference's numbering: a thread per upper inner node, a warp
// per terminal's subtree.
__global__ void __launch_bounds__(kThreads) k_emit(BuildArgs a, double* __restrict__ obox, int32_t* __restrict__ ol,
                                                   int32_t* __restrict__ orr, int32_t* __restrict__ os,
                                                   int32_t* __restrict__ oc) {
  const int upper = *a.n_nodes, terms = *a.n_term;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int u = tid; u < upper; u += step) {
    const int l = a.nleft[u];
    if (l < 0) continue;
    const int d = preorder(a, u);
    for (int j = 0; j < 6; j++) obox[6 * (size_t)d + j] = a.nbox[6 * (size_t)u + j];
    ol[d] = d + 1;
    orr[d] = d + 1 + a.nsize[l];
    os[d] = 0;
    oc[d] = 0;
  }
  const int lane = threadIdx.x & 31;
  for (int z = tid >> 5; z < terms; z += step >> 5) {
    const int d0 = preorder(a, a.znode[z]);
    const size_t src = 2 * (size_t)a.zs[z];
    const int n = a.zsize[z];
    for (int j = lane; j < n; j += 32) {
      const int li = a.lidx[src + j], rt = a.lright[src + j], d = d0 + li;
      ol[d] = rt < 0 ? -1 : d + 1;
      orr[d] = rt < 0 ? -1 : d0 + rt;
      os[d] = a.lstart[src + j];
      oc[d] = a.lcount[src + j];
    }
    for (int i = lane; i < 6 * n; i += 32) {
      const int j = i / 6;
      obox[6 * (size_t)(d0 + a.lidx[src + j]) + (i - 6 * j)] = a.lbox[6 * src + i];
    }
  }
}

}  // namespace

// Carves 256-byte aligned sub-buffers out of one device allocation; with a null
// base it only measures.
struct Carver {
  char* base;
  size_t used = 0;
  template <class T>
  T* take(size_t n) {
    T* r = reinterpret_cast<T*>(base + used);
    used += ((n * sizeof(T) + 255) / 256) * 256;
    return r;
  }
};

struct BuildBuffers {
  BuildArgs a;
  double *pbox, *cent;
  unsigned long long* keys;
  int* counters;  // tasks and chunks of the two levels, upper nodes, terminals
  double* obox;
  int32_t *ol, *orr, *os, *oc;
};

static size_t carve_build(char* base, int32_t n, BuildBuffers* b) {
  Carver cv{base};
  BuildArgs& a = b->a;
  const size_t N = (size_t)n, NN = 2 * N;
  const size_t T = N / (kSmall + 1) + 1;      // tasks of a level: more than kSmall elements each
  const size_t C = N / kChunk + T + 1;        // their chunks
  b->pbox = cv.take<double>(N * 6);
  b->cent = cv.take<double>(N * 3);
  b->keys = cv.take<unsigned long long>(12);
  b->counters = cv.take<int>(16);
  a.order[0] = cv.take<int32_t>(N);
  a.order[1] = cv.take<int32_t>(N);
  a.order_out = cv.take<int32_t>(N);
  a.rpos = cv.take<int32_t>(N);
  a.lpos = cv.take<int32_t>(N);
  a.bin = cv.take<uint8_t>(N);
  for (int k = 0; k < 2; k++) {
    Level& l = a.lv[k];
    l.s = cv.take<int32_t>(T);
    l.e = cv.take<int32_t>(T);
    l.node = cv.take<int32_t>(T);
    l.chunk0 = cv.take<int32_t>(T);
    l.cb = cv.take<unsigned long long>(6 * T);
    l.bins = cv.take<unsigned long long>(T * kFields * kBins);
    l.ctask = cv.take<int32_t>(C);
    l.cidx = cv.take<int32_t>(C);
    l.T = b->counters + 2 * k;
    l.C = b->counters + 2 * k + 1;
  }
  a.n_nodes = b->counters + 4;
  a.n_term = b->counters + 5;
  a.tbest = cv.take<int32_t>(T);
  a.tL = cv.take<int32_t>(T);
  a.tM = cv.take<int32_t>(T);
  a.tchild = cv.take<int32_t>(2 * T);
  a.cbins = cv.take<uint16_t>(C * kBins);
  a.cleft = cv.take<int32_t>(C);
  a.nbox = cv.take<double>(NN * 6);
  a.nleft = cv.take<int32_t>(NN);
  a.nparent = cv.take<int32_t>(NN);
  a.nsize = cv.take<int32_t>(NN);
  a.narrive = cv.take<int32_t>(NN);
  a.zs = cv.take<int32_t>(N);
  a.ze = cv.take<int32_t>(N);
  a.znode = cv.take<int32_t>(N);
  a.zkind = cv.take<int32_t>(N);
  a.zsize = cv.take<int32_t>(N);
  a.lbox = cv.take<double>(NN * 6);
  a.lstart = cv.take<int32_t>(NN);
  a.lcount = cv.take<int32_t>(NN);
  a.lidx = cv.take<int32_t>(NN);
  a.lright = cv.take<int32_t>(NN);
  b->obox = cv.take<double>(NN * 6);
  b->ol = cv.take<int32_t>(NN);
  b->orr = cv.take<int32_t>(NN);
  b->os = cv.take<int32_t>(NN);
  b->oc = cv.take<int32_t>(NN);
  return cv.used;
}

// Device build: fills the caller's host arrays (node arrays sized 2n - 1).
bc_status build_sah_device(bc_context* ctx, int32_t n, const double* prim_box, const double* centroid, int32_t bins,
                           int32_t leaf, int32_t* n_nodes_out, double* node_box, int32_t* node_left,
                           int32_t* node_right, int32_t* node_start, int32_t* node_count, int32_t* order_out) {
  cudaStream_t st = ctx->stream;
  const size_t N = (size_t)n;
  BuildBuffers bb;
  cudaError_t e = ctx->d_build.ensure(carve_build(nullptr, n, &bb));
  if (e) return cuda_status(ctx, e, "BVH build buffers");
  carve_build((char*)ctx->d_build.p, n, &bb);
  BuildArgs& a = bb.a;
  a.pbox = bb.pbox;
  a.cent = bb.cent;
  a.n = n;
  a.nb = bins;
  a.leaf = leaf;
  e = cudaMemcpyAsync(bb.pbox, prim_box, N * 6 * 8, cudaMemcpyHostToDevice, st);
  if (!e) e = cudaMemcpyAsync(bb.cent, centroid, N * 3 * 8, cudaMemcpyHostToDevice, st);
  if (e) return cuda_status(ctx, e, "BVH build upload");

  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms < 1) sms = 1;
  k_start<<<(n + 255) / 256, 256, 0, st>>>(n, a.order[0], bb.keys);
  k_root_bounds<<<std::min(sms * 4, (n + 255) / 256), 256, 0, st>>>(bb.pbox, bb.cent, n, bb.keys);
  k_root_task<<<std::min(sms, (n + 255) / 256), 256, 0, st>>>(a, bb.keys);
  // Levels are launched without waiting while a balanced tree would still have
  // tasks, then two at a time: a level without tasks costs four empty launches,
  // a look at the counters a round trip to the host.
  // Where the first centroids are all one point the tree may be a leaf: looked at at once
  // (100,000 equal centroids: 12 empty levels took 85 of 415 us).
  int cur = 0, levels = 0, balanced = 1;
  while ((N >> balanced) > (size_t)kSmall) balanced++;
  bool one_point = true;
  for (size_t i = 3; i < 3 * std::min<size_t>(N, 64) && one_point; i++) one_point = centroid[i] == centroid[i % 3];
  int look = one_point ? 1 : balanced;
  for (;;) {
    for (; levels < look; levels++) {
      // chunks of this level: known only on the device; the kernels stride
      const int64_t most = std::min<int64_t>((int64_t)sms * 16, (int64_t)(N / kChunk + (N / kSmall) + kThreads) / (kThreads / 32));
      const int cgrid = (int)std::max<int64_t>(1, most);
      // few tasks, many chunks each: wide blocks; many tasks: narrow ones
      const bool wide = levels < 10;
      k_bins<<<cgrid, kThreads, 0, st>>>(a, cur);
      k_split<<<wide ? std::min(sms * 8, 1 << levels) : sms * 16, wide ? 256 : 64, 0, st>>>(a, cur);
      k_rank<<<cgrid, kThreads, 0, st>>>(a, cur);
      k_permute<<<cgrid, kThreads, 0, st>>>(a, cur);
      cur ^= 1;
    }
    if ((e = cudaGetLastError())) return cuda_status(ctx, e, "BVH build launch");
    int hdr[6];
    e = cudaMemcpyAsync(hdr, bb.counters, sizeof(hdr), cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (e) return cuda_status(ctx, e, "BVH build");
    if (hdr[2 * cur] == 0) break;
    if (levels >= 4096) return set_error(ctx, BC_ERR_CAPACITY, "BVH deeper than 4096 levels: build on the host");
    look = std::max(levels + 2, balanced);
  }
  k_small<<<sms * 8, kThreads, 0, st>>>(a);
  k_sizes<<<sms * 4, 256, 0, st>>>(a);
  k_emit<<<sms * 8, kThreads, 0, st>>>(a, bb.obox, bb.ol, bb.orr, bb.os, bb.oc);
  e = cudaGetLastError();
  int n_nodes = 0;
  if (!e) e = cudaMemcpyAsync(&n_nodes, a.nsize, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaMemcpyAsync(order_out, a.order_out, N * 4, cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaStreamSynchronize(st);
  if (e) return cuda_status(ctx, e, "BVH build");
  if (n_nodes < 1 || (size_t)n_nodes > 2 * N - 1) return set_error(ctx, BC_ERR_CAPACITY, "BVH build node count");
  e = cudaMemcpyAsync(node_box, bb.obox, (size_t)n_nodes * 48, cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaMemcpyAsync(node_left, bb.ol, (size_t)n_nodes * 4, cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaMemcpyAsync(node_right, bb.orr, (size_t)n_nodes * 4, cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaMemcpyAsync(node_start, bb.os, (size_t)n_nodes * 4, cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaMemcpyAsync(node_count, bb.oc, (size_t)n_nodes * 4, cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaStreamSynchronize(st);
  if (e) return cuda_status(ctx, e, "BVH build readback");
  *n_nodes_out = n_nodes;
  return BC_OK;
}

using TreeBuildFn = bc_status (*)(void* user, int32_t n, const double* pbox, const double* cent, int32_t bins,
                                  int32_t leaf, int32_t* n_nodes, double* box, int32_t* left, int32_t* right,
                                  int32_t* start, int32_t* count, int32_t* order);
bc_status hscene_build_external(bc_hscene* s, TreeBuildFn fn, void* user);  // host_scene.cpp

}  // namespace bcgx

using namespace bcgx;

extern "C" bc_status bc_build_sah(bc_context* ctx, int32_t n_prims, const double* prim_box, const double* centroid,
                                  int32_t bins, int32_t leaf_size, int32_t* n_nodes_out, double* node_box,
                                  int32_t* node_left, int32_t* node_right, int32_t* node_start, int32_t* node_count,
                                  int32_t* order_out) {
  if (!ctx || n_prims < 1 || !prim_box || !centroid || !n_nodes_out || !node_box || !node_left || !node_right ||
      !node_start || !node_count || !order_out)
    return set_error(ctx, BC_ERR_INVALID_ARG, "NULL argument or no primitives");
  if (n_prims >= (1 << 27)) return set_error(ctx, BC_ERR_INVALID_ARG, "at most 2^27 primitives");
  if (bins < 4) bins = 16;  // Scene.Build's clamps (renderer.go:413-427)
  if (bins > 32) bins = 32;
  if (leaf_size < 1) leaf_size = 4;
  if (leaf_size > 16) leaf_size = 16;
  use_context(ctx);
  return build_sah_device(ctx, n_prims, prim_box, centroid, bins, leaf_size, n_nodes_out, node_box, node_left,
                          node_right, node_start, node_count, order_out);
}

static bc_status device_tree(void* user, int32_t n, const double* pbox, const double* cent, int32_t bins,
                             int32_t leaf, int32_t* n_nodes, double* box, int32_t* left, int32_t* right,
                             int32_t* start, int32_t* count, int32_t* order) {
  return bc_build_sah(static_cast<bc_context*>(user), n, pbox, cent, bins, leaf, n_nodes, box, left, right, start,
                      count, order);
}

extern "C" bc_status bc_hscene_build_device(bc_hscene* s, bc_context* ctx) {
  if (!s || !ctx) return BC_ERR_INVALID_ARG;
  return hscene_build_external(s, device_tree, ctx);
}
