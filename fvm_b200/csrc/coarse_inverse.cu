// Dense inverse of a sparse symmetric diagonally dominant level (the
// coarsest level of a diffusion hierarchy, up to 4096 rows).
//
// The sweep operator (Beaton; Goodnight, Am. Stat. 33, 1979) over a block K
// of pivots, D = A[K][K], keeps the matrix symmetric:
//   A[K][K] <- -D^-1   A[K][j] <- D^-1 A[K][j]   A[i][j] <- A[i][j] - A[i][K] D^-1 A[K][j]
// and after all blocks the matrix is -A^-1. In the level's own order that is
// n / 32 dependent panels, each an update of the whole matrix: 59 panels of
// 32 us on 1862 rows, 104 of 48 us on 3300, bounded by the chain of panels
// and by sweeping tiles that are still zero.
//
// Here the rows are put in nested-dissection order first (George, SIAM J.
// Numer. Anal. 10, 1973): a part is halved across the axis in which it is
// longest and the rows of one half that touch the other become a separator;
// independent components split for free. Then
//  * blocks of pivots in different parts do not couple and are swept in the
//    same step: the chain is the height of the tree;
//  * a tile not yet reached by fill is skipped (a flag per 32 x 32 block).
// A step is two kernels: k_inv_panel forms the new pivot rows R = D^-1 A[K][:]
// of every pivot block of the step, k_inv_update applies them to the 64 x 64
// tiles on and above the diagonal and inverts the next step's pivot blocks.
// Measured, order and unpermuting included: 3313 rows (41k tets) 5.4 -> 0.93
// ms in 23 steps instead of 104 (1.1 before the FP64 matrix instructions and
// the chained launches), 3385 rows (100^3 hexes, two phases) 5.6 -> 1.22 ms
// in 29 instead of 106, 2151 rows (1.5M tets) 2.4 -> 0.73 ms in 22 instead of
// 68, 24 independent meshes of 3930 rows 7.7 -> 0.44 ms in 11 instead of 123.
// The order alone is 0.13, 0.26, 0.16 and 0.12 ms of them.
//
// The result depends on nothing but the matrix (ties by row index, sums in
// a fixed order). Built with contraction: no reference arithmetic here.
#include "coarse_inverse.cuh"

#include <algorithm>
#include <vector>

#include "common.hpp"
#include "pdl.cuh"

namespace fvm {
namespace dev {
namespace {

constexpr int kMaxN = 4096;
constexpr int kLeaf = 256;     // parts of at most this many rows are not split
constexpr int kDepth = 5;      // levels of separators: at most 32 leaves
constexpr int kParts = 32;
constexpr int kNodes = 64;
constexpr int kBins = 256;     // places along an axis (or root indices) told apart
constexpr int kBlk = 32;
// padding: every node is rounded up to whole blocks, the total to whole tiles
constexpr int kMaxBlocks = (kMaxN + (kNodes - 1) * (kBlk - 1)) / kBlk + 2;
constexpr int kOrderThreads = 1024;
constexpr int kPer = kMaxN / kOrderThreads;

struct InvPlan {
  int blocks;  // of 32 rows, even
  int steps;
  int start[kMaxBlocks + 1];  // first pivot block of each step
  int pivot[kMaxBlocks];
};

__device__ __forceinline__ int4 slice_of_row(const SellView<double>& a, const int* rowSlice, int i, int& lane) {
  const int4 m = a.meta[rowSlice[i]];
  lane = i - m.x;
  return m;
}

// one warp per row, one lane per entry
__global__ void __launch_bounds__(256) k_inv_check(SellView<double> a, const int* __restrict__ rowSlice, int* flags) {
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= a.n) return;
  int li;
  const int4 m = slice_of_row(a, rowSlice, i, li);
  double sum = 0.0;
  bool symmetric = true;
  for (int k = lane; k < m.w; k += 32) {
    const int j = a.cols[m.z + 32 * k + li];
    const double v = a.vals[m.z + 32 * k + li];
    if (j == i) continue;
    sum += fabs(v);
    int lj;
    const int4 mj = slice_of_row(a, rowSlice, j, lj);
    int at = -1;
    for (int q = 0; q < mj.w; q++)
      if (a.cols[mj.z + 32 * q + lj] == i) at = mj.z + 32 * q + lj;
    const double w = at >= 0 ? a.vals[at] : 0.0;
    symmetric = symmetric && fabs(v - w) <= 1e-12 * fmax(fabs(v), fabs(w));
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const bool all = __all_sync(0xffffffffu, symmetric);
  if (lane) return;
  const double d = a.diag[i];
  const int bad = (d != 0.0 && sum <= fabs(d) * (1.0 + 1e-8) ? 0 : 1) | (all ? 0 : 2);
  if (bad) atomicOr(flags, bad);
}

// Nested-dissection order of the level's graph by one CTA: pos[i] is row
// i's place in the padded order. Points: x, y, z of every row (n each), or
// null; without them the distances from three far-apart rows of the largest
// component stand in (breadth-first, 16 lanes per row of the queue).
struct OrderShared {
  float at[3][kMaxN];
  int dist[kMaxN], label[kMaxN];  // (label: first the union-find parent)
  unsigned short part[kMaxN], node[kMaxN], queue[2][kMaxN], component[kMaxN];
  unsigned char side[kMaxN];  // 0, 1; +2 when the row touches the other side
  int queued[2], key;
  int hist[kParts][kBins];
  int size[kParts], seed[kParts], mode[kParts], cut[kParts], sep[kParts], child[kParts][2], touch[kParts][2];
  int lo[kParts][3], hi[kParts][3];  // extents, as ordered integers
  int axis[kParts];
  int nodeDepth[kNodes], nodeCount[kNodes], nodeBlock[kNodes];
  int warpCount[kOrderThreads / 32][kNodes];
  int parts, nodes;
  unsigned short place[kMaxN];
};

// floats as integers of the same order, and back
__device__ __forceinline__ int ordered(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void __launch_bounds__(kOrderThreads) k_inv_order(SellView<double> a, const int* __restrict__ rowSlice,
                                                             const float* __restrict__ points, int* pos,
                                                             InvPlan* plan) {
  extern __shared__ __align__(16) unsigned char raw[];
  OrderShared& s = *reinterpret_cast<OrderShared*>(raw);
  const int n = a.n, t = threadIdx.x;
  constexpr unsigned short kNone = 0xffff;
  constexpr int kFar = 0x7fffffff;
  const int lane = t & 31;
  auto range = [&](int i, int& base, int& width) {
    int l;
    const int4 m = slice_of_row(a, rowSlice, i, l);
    base = m.z + l;
    width = m.w;
  };
  // a thread's rows: t + 1024 q, their entries from base, width of them
  int base[kPer], width[kPer];
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads;
    base[q] = width[q] = 0;
    if (i >= n) continue;
    range(i, base[q], width[q]);
    s.part[i] = 0;
    s.node[i] = kNone;
    for (int d = 0; d < 3; d++) s.at[d][i] = points ? points[(size_t)d * n + i] : 0.0f;
  }
  // fn(j) for every column j of the thread's q-th row, eight loads in flight
  auto columns = [&](int q, auto&& fn) {
    for (int k = 0; k < width[q]; k += 8) {
      int j[8];
#pragma unroll
      for (int u = 0; u < 8; u++) j[u] = __ldg(a.cols + base[q] + 32 * min(k + u, width[q] - 1));
#pragma unroll
      for (int u = 0; u < 8; u++) fn(j[u]);
    }
  };
  // count[key] += 1 for every lane with a key >= 0: one atomic per warp and
  // key (most rows share a component and a node; 3313 atomics on one address
  // took 43k cycles)
  auto tally = [&](int* count, int key) {
    const unsigned same = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && lane == __ffs(same) - 1) atomicAdd(&count[key], __popc(same));
  };
  if (t == 0) {
    s.parts = 1;
    s.nodes = 0;
    s.key = 0;
  }
  __syncthreads();
  // components by union-find (the larger root goes under the smaller, so a
  // component's root is its smallest row): every row under its smallest
  // neighbour, pointers halved, then the entries that still join two trees
  volatile int* parent = s.label;
  auto find = [&](int i) {
    int p = parent[i];
    while (p != i) {
      i = p;
      p = parent[i];
    }
    return i;
  };
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads;
    if (i >= n) continue;
    int low = i;
    columns(q, [&](int j) { low = min(low, j); });
    s.label[i] = low;
  }
  __syncthreads();
  for (int k = 1; k < kMaxN; k *= 2) {
    int up[kPer];
    bool moved = false;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int i = t + q * kOrderThreads;
      const int l = i < n ? s.label[i] : 0;
      up[q] = i < n ? s.label[l] : 0;
      moved = moved || up[q] != l;
    }
    if (!__syncthreads_or(moved)) break;
#pragma unroll
    for (int q = 0; q < kPer; q++)
      if (t + q * kOrderThreads < n) s.label[t + q * kOrderThreads] = up[q];
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads;
    if (i >= n) continue;
    columns(q, [&](int j) {
      if (j >= i || parent[j] == parent[i]) return;  // mostly one tree already
      int x = i, y = j;
      while (true) {
        x = find(x);
        y = find(y);
        if (x == y) break;
        const int hi = max(x, y), lo = min(x, y);
        if (atomicCAS(&s.label[hi], hi, lo) == hi) break;
      }
    });
  }
  __syncthreads();
  int root[kPer];
#pragma unroll
  for (int q = 0; q < kPer; q++) root[q] = t + q * kOrderThreads < n ? find(t + q * kOrderThreads) : 0;
  for (int e = t; e < n; e += kOrderThreads) s.dist[e] = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads;
    if (i < n) s.label[i] = root[q];
    tally(s.dist, i < n ? root[q] : -1);
  }
  __syncthreads();
  // rows of each row's component; the largest component's first row
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads;
    if (i >= n) continue;
    s.component[i] = (unsigned short)s.dist[root[q]];
    if (!points) atomicMax(&s.key, s.dist[root[q]] << 12 | (kMaxN - 1 - i));
  }
  __syncthreads();
  if (!points) {
    // from the row farthest from the first row, from the row farthest from
    // that one, and from the row farthest from both
    for (int pass = 0; pass < 4; pass++) {
      const int seed = kMaxN - 1 - (s.key & (kMaxN - 1));
      for (int i = t; i < n; i += kOrderThreads) s.dist[i] = kFar;
      __syncthreads();
      if (t == 0) {
        s.dist[seed] = 0;
        s.queue[0][0] = (unsigned short)seed;
        s.queued[0] = 1;
        s.queued[1] = 0;
        s.key = 0;
      }
      __syncthreads();
      for (int cur = 0; cur < n; cur++) {
        const int len = s.queued[cur & 1];
        if (len == 0) break;
        const unsigned short* from = s.queue[cur & 1];
        unsigned short* to = s.queue[(cur & 1) ^ 1];
        int* count = &s.queued[(cur & 1) ^ 1];
        for (int f = t >> 4; f < len; f += kOrderThreads / 16) {
          int fb, fw;
          range(from[f], fb, fw);
          for (int k = t & 15; k < fw; k += 16) {
            const int j = __ldg(a.cols + fb + 32 * k);
            if (s.dist[j] == kFar && atomicCAS(&s.dist[j], kFar, cur + 1) == kFar)
              to[atomicAdd(count, 1)] = (unsigned short)j;
          }
        }
        __syncthreads();
        if (t == 0) s.queued[cur & 1] = 0;
        __syncthreads();
      }
      for (int i = t; i < n; i += kOrderThreads) {
        if (s.dist[i] == kFar) continue;
        if (pass > 0) s.at[pass - 1][i] = (float)s.dist[i];
        const int far = pass == 2 ? min((int)s.at[0][i], s.dist[i]) : s.dist[i];
        atomicMax(&s.key, far << 12 | (kMaxN - 1 - i));
      }
      __syncthreads();
    }
  }
  for (int depth = 0; depth < kDepth; depth++) {
    const int P = s.parts;
    if (t < kParts) {
      s.size[t] = s.seed[t] = s.mode[t] = s.touch[t][0] = s.touch[t][1] = 0;
      s.sep[t] = s.child[t][0] = s.child[t][1] = -1;
      for (int d = 0; d < 3; d++) {
        s.lo[t][d] = kFar;
        s.hi[t][d] = -kFar;
      }
    }
    for (int e = t; e < kParts * kBins; e += kOrderThreads) (&s.hist[0][0])[e] = 0;
    __syncthreads();
    // (one atomic per warp and part)
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int i = t + q * kOrderThreads;
      const int p = i < n && s.node[i] == kNone ? (int)s.part[i] : kParts;
      const unsigned same = __match_any_sync(0xffffffffu, p);
      if (p == kParts) continue;
      const bool leader = lane == __ffs(same) - 1;
      const int big = __reduce_max_sync(same, (int)s.component[i]);  // its largest component
      if (leader) {
        atomicAdd(&s.size[p], __popc(same));
        atomicMax(&s.seed[p], big);
      }
      for (int d = 0; d < 3; d++) {
        const int v = ordered(s.at[d][i]);
        const int lo = __reduce_min_sync(same, v), hi = __reduce_max_sync(same, v);
        if (leader) {
          atomicMin(&s.lo[p][d], lo);
          atomicMax(&s.hi[p][d], hi);
        }
      }
    }
    __syncthreads();
    // mode 1: split by component, 2: across the longest axis
    if (t < P && s.size[t] > kLeaf) {
      s.mode[t] = 5 * s.seed[t] <= 3 * s.size[t] ? 1 : 2;
      float best = -1.0f;
      for (int d = 0; d < 3; d++) {
        const float e = from_ordered(s.hi[t][d]) - from_ordered(s.lo[t][d]);
        if (e > best) {
          best = e;
          s.axis[t] = d;
        }
      }
    }
    if (!__syncthreads_or(t < P && s.mode[t] != 0)) break;
    // a row's bin: by its place on the axis, or by its component's root
    auto bin = [&](int i, int p) {
      if (s.mode[p] == 1) return s.label[i] / (kMaxN / kBins);
      const int d = s.axis[p];
      const float lo = from_ordered(s.lo[p][d]), hi = from_ordered(s.hi[p][d]);
      const float f = hi > lo ? (s.at[d][i] - lo) / (hi - lo) * kBins : 0.0f;
      return min(max((int)f, 0), kBins - 1);
    };
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int i = t + q * kOrderThreads;
      int key = -1;
      if (i < n && s.node[i] == kNone && s.mode[s.part[i]]) key = s.part[i] * kBins + bin(i, s.part[i]);
      const unsigned same = __match_any_sync(0xffffffffu, key);
      if (key >= 0 && lane == __ffs(same) - 1) atomicAdd(&s.hist[0][0] + key, __popc(same));
    }
    __syncthreads();
    // the most even cut of part w, by warp w
    {
      const int p = t >> 5;
      if (p < P && s.mode[p]) {
        int h[kBins / 32], sum = 0;
#pragma unroll
        for (int k = 0; k < kBins / 32; k++) {
          h[k] = s.hist[p][lane * (kBins / 32) + k];
          sum += h[k];
        }
        int before = sum;
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, before, o);
          if (lane >= o) before += v;
        }
        before -= sum;
        const int size = s.size[p];
        int best = kFar;
#pragma unroll
        for (int k = 0; k < kBins / 32; k++) {
          before += h[k];
          if (before > 0 && before < size)
            best = min(best, max(before, size - before) << 8 | (lane * (kBins / 32) + k));
        }
        for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (lane == 0) {
          s.cut[p] = best & (kBins - 1);
          // all in one bin, or a sliver: a leaf
          if (best == kFar || 8 * (best >> 8) > 7 * size) s.mode[p] = 0;
        }
      }
    }
    __syncthreads();
    // (place: a row's part and side in one word, none for rows not being split)
    for (int i = t; i < n; i += kOrderThreads) {
      int place = 0xffff;
      if (s.node[i] == kNone && s.mode[s.part[i]]) {
        const int side = bin(i, s.part[i]) > s.cut[s.part[i]] ? 1 : 0;
        s.side[i] = (unsigned char)side;
        place = 2 * s.part[i] + side;
      }
      s.place[i] = (unsigned short)place;
    }
    __syncthreads();
    // the rows of either side that touch the other
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int i = t + q * kOrderThreads;
      int key = -1;
      if (i < n && s.node[i] == kNone && s.mode[s.part[i]] == 2) {
        const int p = s.part[i], mine = s.side[i] & 1, across = 2 * p + 1 - mine;
        bool hit = false;
        columns(q, [&](int j) { hit = hit || s.place[j] == across; });
        if (hit) {
          s.side[i] = (unsigned char)(mine | 2);
          key = 2 * p + mine;
        }
      }
      const unsigned same = __match_any_sync(0xffffffffu, key);
      if (key >= 0 && lane == __ffs(same) - 1) atomicAdd(&s.touch[0][0] + key, __popc(same));
    }
    __syncthreads();
    if (t == 0) {
      // children keep the part's id and take a new one
      int parts = P, nodes = s.nodes;
      for (int p = 0; p < P; p++) {
        if (!s.mode[p]) continue;
        const int fewer = min(s.touch[p][0], s.touch[p][1]);
        // a separator of more than half the part does not help
        if (parts >= kParts || 2 * fewer > s.size[p]) {
          s.mode[p] = 0;
          continue;
        }
        s.child[p][0] = p;
        s.child[p][1] = parts++;
        if (fewer > 0) {
          s.nodeDepth[nodes] = depth;
          s.sep[p] = nodes++;
        }
      }
      s.parts = parts;
      s.nodes = nodes;
    }
    __syncthreads();
    for (int i = t; i < n; i += kOrderThreads) {
      if (s.node[i] != kNone) continue;
      const int p = s.part[i];
      if (!s.mode[p]) continue;
      const int mine = s.side[i] & 1;
      const int from = s.touch[p][0] < s.touch[p][1] ? 0 : 1;  // the side that gives the separator
      if ((s.side[i] & 2) && mine == from)
        s.node[i] = (unsigned short)s.sep[p];
      else
        s.part[i] = (unsigned short)s.child[p][mine];
    }
    __syncthreads();
  }
  // what is left of the parts are the leaves
  const int separators = s.nodes;
  if (t < kNodes) s.nodeCount[t] = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads;
    if (i < n && s.node[i] == kNone) s.node[i] = (unsigned short)(separators + s.part[i]);
    tally(s.nodeCount, i < n ? (int)s.node[i] : -1);
  }
  __syncthreads();
  // leaves first, then the separators from the deepest up; in each group
  // step q sweeps the q-th block of every node (one warp, two nodes a lane)
  if (t < 32) {
    const int nodes = separators + s.parts;
    int depthOf[2], blocks[2], first[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int k = lane + 32 * u;
      depthOf[u] = k >= nodes ? -1 : k >= separators ? kDepth : s.nodeDepth[k];
      blocks[u] = k < nodes ? (s.nodeCount[k] + kBlk - 1) / kBlk : 0;
    }
    int block = 0, steps = 0, np = 0;
    for (int d = kDepth; d >= 0; d--) {
      int most = 0;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int nb = depthOf[u] == d ? blocks[u] : 0;
        int before = nb;
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, before, o);
          if (lane >= o) before += v;
        }
        if (depthOf[u] == d) first[u] = block + before - nb;
        block += __shfl_sync(0xffffffffu, before, 31);
        most = max(most, __reduce_max_sync(0xffffffffu, nb));
      }
      for (int q = 0; q < most; q++) {
        if (lane == 0) plan->start[steps] = np;
        steps++;
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const bool on = depthOf[u] == d && q < blocks[u];
          const unsigned m = __ballot_sync(0xffffffffu, on);
          if (on) plan->pivot[np + __popc(m & ((1u << lane) - 1u))] = first[u] + q;
          np += __popc(m);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (depthOf[u] >= 0) s.nodeBlock[lane + 32 * u] = first[u];
    if (lane == 0) {
      plan->start[steps] = np;
      plan->steps = steps;
      plan->blocks = (block + 1) / 2 * 2;
    }
  }
  __syncthreads();
  if (t < kNodes) s.nodeCount[t] = 0;
  __syncthreads();
  // rows of a node in ascending order: chunks of 1024 rows, the warps'
  // counts per node prefixed in warp order
  for (int q = 0; q < kPer; q++) {
    const int i = t + q * kOrderThreads, w = t >> 5;
    for (int e = t; e < (kOrderThreads / 32) * kNodes; e += kOrderThreads) (&s.warpCount[0][0])[e] = 0;
    __syncthreads();
    const int node = i < n ? (int)s.node[i] : kNodes;
    const unsigned same = __match_any_sync(0xffffffffu, node);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (node < kNodes && rank == 0) s.warpCount[w][node] = __popc(same);
    __syncthreads();
    if (t < kNodes) {
      int run = s.nodeCount[t];
      for (int v = 0; v < kOrderThreads / 32; v++) {
        const int c = s.warpCount[v][t];
        s.warpCount[v][t] = run;
        run += c;
      }
      s.nodeCount[t] = run;
    }
    __syncthreads();
    if (i < n) pos[i] = s.nodeBlock[node] * kBlk + s.warpCount[w][node] + rank;
    __syncthreads();
  }
}

// blocks (I <= J) on and above the diagonal, row by row
__device__ __forceinline__ size_t block_at(int NB, int I, int J) {
  return ((size_t)I * NB - (size_t)I * (I - 1) / 2 + (J - I)) * (kBlk * kBlk);
}

// which blocks hold entries (one byte per block pair)
__global__ void __launch_bounds__(128) k_inv_flag(SellView<double> a, const int* __restrict__ rowSlice,
                                                  const int* pos, int NB, unsigned char* nz, int* rowAt) {
  FVM_PDL();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NB) nz[(size_t)i * NB + i] = 1;
  if (i >= a.n) return;
  int lane;
  const int4 m = slice_of_row(a, rowSlice, i, lane);
  const int bi = pos[i] / kBlk;
  rowAt[pos[i]] = i;
  for (int k = 0; k < m.w; k++) {
    const int bj = pos[a.cols[m.z + 32 * k + lane]] / kBlk;
    if (bi <= bj) nz[(size_t)bi * NB + bj] = 1;
  }
}
// flagged blocks to zero, the diagonal to one (the padding rows keep it)
__global__ void __launch_bounds__(256) k_inv_clear(int NB, const unsigned char* nz, double* A) {
  FVM_PDL();
  const int I = blockIdx.y, J = blockIdx.x;
  if (J < I || !nz[(size_t)I * NB + J]) return;
  double* b = A + block_at(NB, I, J);
  for (int e = threadIdx.x; e < kBlk * kBlk; e += 256) b[e] = I == J && e / kBlk == e % kBlk ? 1.0 : 0.0;
}
__global__ void __launch_bounds__(128) k_inv_scatter(SellView<double> a, const int* __restrict__ rowSlice,
                                                     const int* pos, int NB, double* A) {
  FVM_PDL();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  int lane;
  const int4 m = slice_of_row(a, rowSlice, i, lane);
  const int p = pos[i], bi = p / kBlk;
  double* d = A + block_at(NB, bi, bi) + (p % kBlk) * kBlk + p % kBlk;
  *d = a.diag[i];
  for (int k = 0; k < m.w; k++) {
    const int q = pos[a.cols[m.z + 32 * k + lane]], bj = q / kBlk;
    const double v = a.vals[m.z + 32 * k + lane];
    // an entry below the diagonal is stored by the other row
    if (v != 0.0 && bi <= bj) A[block_at(NB, bi, bj) + (p % kBlk) * kBlk + q % kBlk] += v;
  }
}

// The inverse of a symmetric 32 x 32 block by the sweep operator, one pivot
// at a time without pivoting: thread (w, c) of 256 holds rows 4 w .. 4 w + 3
// of column c. By symmetry the pivot's row is all a step needs; its owners
// leave it in shared memory (two buffers, one barrier per step).
struct BlockInverse {
  double row[2][kBlk];
};
__device__ void invert_block(double (&d)[4], BlockInverse& s, double* out, int* status) {
  const int w = threadIdx.x >> 5, c = threadIdx.x & 31;
  if (w == 0) s.row[0][c] = d[0];
#pragma unroll
  for (int t = 0; t < kBlk; t++) {
    __syncthreads();
    const double* row = s.row[t & 1];
    const double pv = row[t], ip = 1.0 / pv, scaled = row[c] * ip;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double v = row[4 * w + k];  // = D[4 w + k][t]
      if (w == t / 4 && k == t % 4)
        d[k] = c == t ? -ip : scaled;
      else
        d[k] = c == t ? v * ip : d[k] - v * scaled;
      if (t + 1 < kBlk && k == (t + 1) % 4 && w == (t + 1) / 4) s.row[(t + 1) & 1][c] = d[k];
    }
    if (pv == 0.0 && threadIdx.x == 0) atomicExch(status, 1);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) out[(4 * w + k) * kBlk + c] = -d[k];
}

// the first step's pivot blocks inverted
__global__ void __launch_bounds__(256) k_inv_first(int NB, const int* pivots, const double* A, double* Dinv,
                                                   int* status) {
  __shared__ BlockInverse ws;
  FVM_PDL();
  const int K = pivots[blockIdx.x];
  const double* b = A + block_at(NB, K, K);
  double d[4];
#pragma unroll
  for (int k = 0; k < 4; k++) d[k] = b[(4 * (threadIdx.x >> 5) + k) * kBlk + (threadIdx.x & 31)];
  invert_block(d, ws, Dinv + (size_t)K * kBlk * kBlk, status);
}

// For block row i and the step's q-th pivot block K: C = A[i][K] (old) and
// R = D^-1 A[K][i], both 32 x 32 at slot (q, i); act[q][i] says whether
// they couple at all.
// (pivots: complete before the first step, read ahead of the wait)
__global__ void __launch_bounds__(256) k_inv_panel(int NB, const int* __restrict__ pivots, const double* A,
                                                   const double* Dinv, const unsigned char* nz, double* C, double* R,
                                                   unsigned char* act) {
  __shared__ double S[kBlk][kBlk + 1], D[kBlk][kBlk + 1];
  FVM_PDL_TRIGGER();
  const int i = blockIdx.x, q = blockIdx.y, K = pivots[q];
  FVM_PDL_WAIT();
  const bool on = i != K && nz[(size_t)min(i, K) * NB + max(i, K)];
  if (threadIdx.x == 0) act[(size_t)q * NB + i] = on;
  if (!on) return;
  const double* b = A + block_at(NB, min(i, K), max(i, K));
  const double* dk = Dinv + (size_t)K * kBlk * kBlk;
  const int r0 = threadIdx.x >> 5, c = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int r = r0 + 8 * u;
    // S[row of i][row of K]
    if (i < K)
      S[r][c] = b[r * kBlk + c];
    else
      S[c][r] = b[r * kBlk + c];
    D[r][c] = dk[r * kBlk + c];
  }
  __syncthreads();
  const size_t o = ((size_t)q * NB + i) * kBlk * kBlk;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int k = 0; k < kBlk; k++) {
    const double s = S[c][k];
#pragma unroll
    for (int u = 0; u < 4; u++) acc[u] += D[r0 + 8 * u][k] * s;
  }
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int r = r0 + 8 * u;
    R[o + r * kBlk + c] = acc[u];
    C[o + r * kBlk + c] = S[r][c];
  }
}

__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

struct UpdateStage {
  double C[64][kBlk + 4], R[kBlk][64 + 4];  // (rows 4 banks of 8 bytes on: fragment loads without conflicts)
};

// D (8 x 8) += A (8 x 4) B (4 x 8): lane l holds A[l / 4][l % 4], B[l % 4][l / 4]
// and D[l / 4][2 (l % 4) .. + 1]
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// One step over the 64 x 64 tiles on and above the diagonal (four blocks
// each, one CTA per tile, two warps per block). A tile that no pivot of the
// step reaches returns at once. With a 4 x 4 register tile of FP64 FMAs a
// thread a step over a full matrix of 3840 padded rows took 41 us: 11 us of
// FP64 at the chip's rate, as long again in shared-memory reads, and three
// CTAs of 80 registers per SM to hide those and the tile's loads behind each
// other. The FP64 matrix instruction reads 6 operands for 8 products of 8 x 8
// x 4 where that read 8 for 16 FMAs; one stage suffices where the step has
// one pivot; the pivots are read ahead of the wait. Over the 23 steps of 3313
// rows 31 -> 21.5 us a step (64 registers and four CTAs, with spills: 22.8).
__global__ void __launch_bounds__(256, 3) k_inv_update(int NB, int np, const int* __restrict__ pivots, int nNext,
                                                       const int* __restrict__ next, double* A, const double* C,
                                                       const double* R, const unsigned char* act, double* Dinv,
                                                       unsigned char* nz, int* status) {
  // two stages (one when np = 1): the next pivot's operands arrive while one
  // is multiplied
  FVM_PDL_TRIGGER();
  extern __shared__ __align__(16) unsigned char raw[];
  UpdateStage* stage = reinterpret_cast<UpdateStage*>(raw);
  // the diagonal tiles first (they may go on to invert a pivot block), then
  // the tiles above the diagonal, row by row
  const int T = NB / 2;
  int I = blockIdx.x, J = I;
  if (I >= T) {
    const int p = I - T;
    const float f = 2.0f * T - 1.0f;
    I = (int)((f - sqrtf(f * f - 8.0f * p)) * 0.5f);
    while (I > 0 && I * (T - 1) - I * (I - 1) / 2 > p) I--;
    while ((I + 1) * (T - 1) - (I + 1) * I / 2 <= p) I++;
    J = I + 1 + p - (I * (T - 1) - I * (I - 1) / 2);
  }
  const int tid = threadIdx.x, lane = tid & 31;
  // lane q: how pivot q meets the tile's block rows and columns
  bool r0 = false, r1 = false, c0 = false, c1 = false;
  int K = -1;
  // the blocks of the tile: (I, J), (I, J+), (I+, J), (I+, J+); on the
  // diagonal (I+, J) lies below it and is not stored
  // (warp w: block (x, y), its rows 16 (w / 2 % 2) .. + 15)
  const int warp = tid >> 5, x = warp >> 2, y = warp & 1, h = (warp >> 1) & 1;
  if (lane < np) K = pivots[lane];
  int nextHere = 0;  // pivots of the next step on this tile's diagonal
  if (I == J) {
    int v = 0;
    for (int k = lane; k < nNext; k += 32) {
      const int b = next[k];
      v |= b == 2 * I ? 1 : b == 2 * I + 1 ? 2 : 0;
    }
    nextHere = __reduce_or_sync(0xffffffffu, v);
  }
  FVM_PDL_WAIT();
  const int bi = 2 * I + x, bj = 2 * J + y;
  const bool stored = bi <= bj, filled = stored && nz[(size_t)bi * NB + bj];
  if (lane < np) {
    const unsigned char* f = act + (size_t)lane * NB;
    r0 = f[2 * I];
    r1 = f[2 * I + 1];
    c0 = f[2 * J];
    c1 = f[2 * J + 1];
  }
  constexpr unsigned kAll = 0xffffffffu;
  const unsigned mr0 = __ballot_sync(kAll, r0), mr1 = __ballot_sync(kAll, r1), mc0 = __ballot_sync(kAll, c0),
                 mc1 = __ballot_sync(kAll, c1);
  // the pivot (its index in the step, -1: none) that is a block row / column
  auto pivotAt = [&](int b) {
    const unsigned m = __ballot_sync(kAll, K == b);
    return m ? __ffs(m) - 1 : -1;
  };
  const int pr0 = pivotAt(2 * I), pr1 = pivotAt(2 * I + 1), pc0 = pivotAt(2 * J), pc1 = pivotAt(2 * J + 1);
  const unsigned work = (mr0 | mr1) & (mc0 | mc1);
  const bool meets = pr0 >= 0 || pr1 >= 0 || pc0 >= 0 || pc1 >= 0;
  if (!work && !meets && !nextHere) return;
  // the warp's 16 x 32 as two rows of four 8 x 8 fragments
  const int fr = 16 * h + (lane >> 2), fc = 2 * (lane & 3);  // the lane's first element in the block
  double acc[2][4][2];
  {
    const double* b = A + block_at(NB, min(bi, bj), max(bi, bj)) + fr * kBlk + fc;
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const double2 d = filled ? *reinterpret_cast<const double2*>(b + 8 * u * kBlk + 8 * v) : make_double2(0.0, 0.0);
        acc[u][v][0] = d.x;
        acc[u][v][1] = d.y;
      }
  }
  // thread t copies C row t / 16 (+ 16 u), columns 2 (t mod 16), and R row
  // t / 32 (+ 8 u), columns 2 (t mod 32)
  const unsigned mcT = (lane >> 4) ? mc1 : mc0;
  const double* const cFrom = C + ((size_t)(2 * I) * kBlk + (tid >> 4)) * kBlk + (tid & 15) * 2;
  const double* const rFrom = R + ((size_t)(2 * J + (lane >> 4)) * kBlk + (tid >> 5)) * kBlk + ((lane * 2) & 31);
  auto fetch = [&](int q, UpdateStage& g) {
    const size_t slot = (size_t)q * NB * kBlk * kBlk;
    const bool on0 = mr0 >> q & 1, on1 = mr1 >> q & 1, onC = mcT >> q & 1;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      double* c = &g.C[(tid >> 4) + 16 * u][(tid & 15) * 2];
      if (u < 2 ? on0 : on1)
        copy16(c, cFrom + slot + 16 * u * kBlk);
      else
        c[0] = c[1] = 0.0;
      double* r = &g.R[(tid >> 5) + 8 * u][lane * 2];
      if (onC)
        copy16(r, rFrom + slot + 8 * u * kBlk);
      else
        r[0] = r[1] = 0.0;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  if (work) fetch(__ffs(work) - 1, stage[0]);
  int cur = 0;
  for (unsigned m = work; m; m &= m - 1, cur ^= 1) {
    const unsigned left = m & (m - 1);
    if (left) {
      fetch(__ffs(left) - 1, stage[cur ^ 1]);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const UpdateStage& g = stage[cur];
    const double* ca = &g.C[32 * x + fr][lane & 3];
    const double* rb = &g.R[lane & 3][32 * y + (lane >> 2)];
#pragma unroll
    for (int k = 0; k < kBlk; k += 4) {
      double c[2], r[4];
#pragma unroll
      for (int u = 0; u < 2; u++) c[u] = -ca[8 * u * (kBlk + 4) + k];
#pragma unroll
      for (int v = 0; v < 4; v++) r[v] = rb[k * (64 + 4) + 8 * v];
#pragma unroll
      for (int u = 0; u < 2; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) mma_f64(acc[u][v], c[u], r[v]);
    }
    __syncthreads();  // the stage is free for the pivot after the next
  }
  // write the block: pivot rows and columns take R, the pivot block -D^-1
  const unsigned mrx = x ? mr1 : mr0, mcy = y ? mc1 : mc0;
  const int kr = x ? pr1 : pr0, kc = y ? pc1 : pc0;
  if (stored) {
    double* b = A + block_at(NB, bi, bj) + fr * kBlk + fc;
    if (kr < 0 && kc < 0) {
      if (mrx & mcy) {
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
          for (int v = 0; v < 4; v++)
            *reinterpret_cast<double2*>(b + 8 * u * kBlk + 8 * v) = make_double2(acc[u][v][0], acc[u][v][1]);
        if (!filled && h == 0 && lane == 0) nz[(size_t)bi * NB + bj] = 1;
      }
    } else {
      // R of column bj, R^T of row bi, or -D^-1; a block that the pivot does
      // not couple to stays as it is
      const double* from = nullptr;
      int rs = kBlk, cs = 1;
      double sign = 1.0;
      if (bi == bj) {
        from = Dinv + (size_t)bi * kBlk * kBlk;
        sign = -1.0;
      } else if (kr >= 0) {
        if (mcy >> kr & 1) from = R + ((size_t)kr * NB + bj) * kBlk * kBlk;
      } else if (mrx >> kc & 1) {
        from = R + ((size_t)kc * NB + bi) * kBlk * kBlk;
        rs = 1;
        cs = kBlk;
      }
      if (from)
        for (int u = 0; u < 2; u++)
          for (int v = 0; v < 4; v++)
            for (int e = 0; e < 2; e++)
              b[8 * u * kBlk + 8 * v + e] = sign * from[(fr + 8 * u) * rs + (fc + 8 * v + e) * cs];
    }
  }
  for (int z = 0; z < 2; z++) {
    if (!(nextHere >> z & 1)) continue;
    // the block's values from the registers (a pivot of the next step is no
    // pivot of this one)
    __syncthreads();
    if (x == z && y == z)
#pragma unroll
      for (int u = 0; u < 2; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          stage[0].C[fr + 8 * u][fc + 8 * v] = acc[u][v][0];
          stage[0].C[fr + 8 * u][fc + 8 * v + 1] = acc[u][v][1];
        }
    __syncthreads();
    double d[4];
#pragma unroll
    for (int k = 0; k < 4; k++) d[k] = stage[0].C[4 * (tid >> 5) + k][lane];
    invert_block(d, *reinterpret_cast<BlockInverse*>(&stage[0].R[0][0]), Dinv + (size_t)(2 * I + z) * kBlk * kBlk, status);
  }
}

// out = the negated, unpermuted matrix: a CTA takes W consecutive rows of
// the padded order, mirrors them from the stored triangle into shared
// memory and writes each to its own row (ld apart, zero past column n),
// columns gathered there
template <class T, int W>
__global__ void __launch_bounds__(512) k_inv_finish(int n, int NB, const int* pos, const int* rowAt, const double* A,
                                                    const unsigned char* nz, T* out, int ld) {
  extern __shared__ __align__(16) unsigned char raw[];
  FVM_PDL();
  T* strip = reinterpret_cast<T*>(raw);  // [W][NB * 32]
  const int N = NB * kBlk, p0 = blockIdx.x * W, I = p0 / kBlk, r0 = p0 % kBlk;
  const int lane = threadIdx.x & 31;
  for (int J = threadIdx.x >> 5; J < NB; J += 16) {
    const bool on = nz[(size_t)min(I, J) * NB + max(I, J)];
    const double* b = A + block_at(NB, min(I, J), max(I, J));
    const int rs = I <= J ? kBlk : 1, cs = I <= J ? 1 : kBlk;
    double v[W];
#pragma unroll
    for (int r = 0; r < W; r++) v[r] = on ? -b[(r0 + r) * rs + lane * cs] : 0.0;
#pragma unroll
    for (int r = 0; r < W; r++) strip[(size_t)r * N + J * kBlk + lane] = (T)v[r];
  }
  int row[W];
#pragma unroll
  for (int r = 0; r < W; r++) row[r] = rowAt[p0 + r];
  __syncthreads();
  for (int j = threadIdx.x; j < ld; j += 512) {
    const int at = j < n ? pos[j] : -1;
#pragma unroll
    for (int r = 0; r < W; r++)
      if (row[r] >= 0) out[(size_t)row[r] * ld + j] = at >= 0 ? strip[(size_t)r * N + at] : T(0);
  }
}

// a coarse row's point: the mean of its fine rows'
__global__ void __launch_bounds__(128) k_coarse_points(int nc, const int* __restrict__ c2fRow,
                                                       const int* __restrict__ c2fCol, const int* __restrict__ fineCell,
                                                       const double* __restrict__ fineXyz, int nFine,
                                                       const float* __restrict__ finePoints, float* points) {
  const int I = blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= nc) return;
  float sum[3] = {0.0f, 0.0f, 0.0f};
  const int e0 = c2fRow[I], e1 = c2fRow[I + 1];
  for (int e = e0; e < e1; e++) {
    const int f = c2fCol[e];
    for (int d = 0; d < 3; d++)
      sum[d] += fineXyz ? (float)fineXyz[3 * (size_t)(fineCell ? fineCell[f] : f) + d] : finePoints[(size_t)d * nFine + f];
  }
  for (int d = 0; d < 3; d++) points[(size_t)d * nc + I] = e1 > e0 ? sum[d] / (float)(e1 - e0) : 0.0f;
}

void ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw Error(kDeviceError, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace

void dominant_symmetric_check(const SellView<double>& a, const int* rowSlice, int* flags, cudaStream_t st) {
  k_inv_check<<<(a.n + 7) / 8, 256, 0, st>>>(a, rowSlice, flags);
}

void coarse_points(int nc, const int* c2fRow, const int* c2fCol, const int* fineCell, const double* fineXyz, int nFine,
                   const float* finePoints, float* points, cudaStream_t st) {
  k_coarse_points<<<(nc + 127) / 128, 128, 0, st>>>(nc, c2fRow, c2fCol, fineCell, fineXyz, nFine, finePoints, points);
}

void inverse_symmetric(const SellView<double>& a, const int* rowSlice, const float* points, double* out64, float* outF,
                       int* status, const std::function<void*(size_t)>& alloc, cudaStream_t st) {
  const int n = a.n;
  FVM_REQUIRE(n >= 1 && n <= kMaxN, kTooLarge, "coarsest level too large for the dense direct solve");
  int* pos = (int*)alloc(sizeof(int) * (size_t)kMaxN);
  InvPlan* dPlan = (InvPlan*)alloc(sizeof(InvPlan));
  ok(cudaFuncSetAttribute(k_inv_order, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OrderShared)),
     "cudaFuncSetAttribute");
  k_inv_order<<<1, kOrderThreads, sizeof(OrderShared), st>>>(a, rowSlice, points, pos, dPlan);
  InvPlan plan;
  ok(cudaMemcpyAsync(&plan, dPlan, sizeof(plan), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  ok(cudaStreamSynchronize(st), "elimination order");
  const int NB = plan.blocks;
  FVM_REQUIRE(NB >= 1 && NB <= kMaxBlocks && plan.steps >= 1 && plan.steps <= kMaxBlocks, kDeviceError,
              "elimination order out of range");
  int widest = 1;
  for (int s = 0; s < plan.steps; s++) widest = std::max(widest, plan.start[s + 1] - plan.start[s]);
  constexpr size_t blk = sizeof(double) * kBlk * kBlk;
  double* A = (double*)alloc(blk * (size_t)NB * (NB + 1) / 2);
  double* C = (double*)alloc(blk * (size_t)NB * widest);
  double* R = (double*)alloc(blk * (size_t)NB * widest);
  double* Dinv = (double*)alloc(blk * (size_t)NB);
  unsigned char* nz = (unsigned char*)alloc((size_t)NB * NB);
  unsigned char* act = (unsigned char*)alloc((size_t)widest * NB);
  int* rowAt = (int*)alloc(sizeof(int) * (size_t)NB * kBlk);
  ok(cudaMemsetAsync(nz, 0, (size_t)NB * NB, st), "cudaMemsetAsync");
  ok(cudaMemsetAsync(rowAt, 0xff, sizeof(int) * (size_t)NB * kBlk, st), "cudaMemsetAsync");
  const int rows = (std::max(n, NB) + 127) / 128;
  pdl_launch(k_inv_flag, rows, 128, st, a, rowSlice, pos, NB, nz, rowAt);
  pdl_launch(k_inv_clear, dim3(NB, NB), 256, st, NB, nz, A);
  pdl_launch(k_inv_scatter, rows, 128, st, a, rowSlice, pos, NB, A);
  const int* pivots = dPlan->pivot;  // (device address arithmetic only)
  pdl_launch(k_inv_first, plan.start[1], 256, st, NB, pivots, A, Dinv, status);
  const int tiles = (NB / 2) * (NB / 2 + 1) / 2;
  ok(cudaFuncSetAttribute(k_inv_update, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (int)sizeof(UpdateStage)),
     "cudaFuncSetAttribute");
  for (int s = 0; s < plan.steps; s++) {
    const int np = plan.start[s + 1] - plan.start[s];
    const int nNext = s + 1 < plan.steps ? plan.start[s + 2] - plan.start[s + 1] : 0;
    const int* at = pivots + plan.start[s];
    pdl_launch(k_inv_panel, dim3(NB, np), 256, st, NB, at, A, Dinv, nz, C, R, act);
    pdl_launch_smem(k_inv_update, tiles, 256, (np > 1 ? 2 : 1) * sizeof(UpdateStage), st, NB, np, at, nNext,
                    pivots + plan.start[s + 1], A, C, R, act, Dinv, nz, status);
  }
  const int N = NB * kBlk;
  if (out64) {
    const size_t smem = sizeof(double) * 4 * (size_t)N;
    ok(cudaFuncSetAttribute(k_inv_finish<double, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
       "cudaFuncSetAttribute");
    pdl_launch_smem(k_inv_finish<double, 4>, N / 4, 512, smem, st, n, NB, pos, rowAt, A, nz, out64, n);
  } else {
    const size_t smem = sizeof(float) * 8 * (size_t)N;
    ok(cudaFuncSetAttribute(k_inv_finish<float, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
       "cudaFuncSetAttribute");
    pdl_launch_smem(k_inv_finish<float, 8>, N / 8, 512, smem, st, n, NB, pos, rowAt, A, nz, outF, inverse_f32_stride(n));
  }
  ok(cudaGetLastError(), "coarsest inverse");
}

}  // namespace dev
}  // namespace fvm
