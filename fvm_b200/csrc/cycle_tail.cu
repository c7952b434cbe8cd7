// The coarse levels of an AMG cycle as one thread-block-cluster kernel.
//
// What bounds a cycle on small levels is not bytes but the chain of passes:
// a V(1,1) cycle with multicolour Gauss-Seidel makes about twenty dependent
// passes per level, each over a few thousand rows at most, and as launches
// of their own (programmatic dependent launches in a CUDA graph) every one
// costs about 2.2 us whatever its size. Here one cluster of CTAs runs them
// all: the levels' x, b and r live in the CTAs' shared memory, a pass
// gathers x by distributed-shared-memory loads, and passes are separated by
// a cluster barrier (0.26 us for 16 CTAs of 512 threads) instead of a
// launch. Levels small enough for one CTA run in the first CTA alone, with
// CTA barriers (0.03 us).
//
// With the barrier this cheap, a pass is bounded by the instructions a warp
// issues between two barriers. So a thread keeps its row of the level --
// the shared-memory addresses of its columns, its values, its diagonal and
// the diagonal's reciprocal -- in registers over all passes of a visit, in
// which a pass is one round of gathers, the sum in stored order and a
// division of five operations on the precomputed reciprocal. Measured per
// Gauss-Seidel pass at 4 / 8 / 16 / 24 entries a row: 0.11 / 0.14 / 0.20 /
// 0.27 us in one CTA (384 rows), 0.53 / 0.66 / 0.95 / 1.24 us over 16 (7104
// rows); reading the row anew in every pass cost 1.0-4 us. Slices that
// couple sit in the same CTA: with slices dealt out round-robin the 7104-row
// pass at 16 entries took 1.87 us.
//
// The passes are a list of steps made on the host (AmgHierarchy::buildTail),
// so V, W and F cycles and all smoothers go through the same kernel. The
// file is built without contraction: bitwise the values of the separate
// kernels, over the whole range of the formats (divide).
#include "cycle_tail.cuh"

#include <cmath>
#include <cstdint>

#include "pdl.cuh"

namespace fvm {
namespace dev {
namespace {

// (.aligned: the warp's threads arrive together)
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// address of the element at a place of the vector at shared address `base`
// in the cluster's window (Solo: in this CTA's own)
template <class T, bool Solo>
__device__ __forceinline__ unsigned element(unsigned base, int place) {
  unsigned a = base + ((unsigned)place >> 4) * (unsigned)sizeof(T);
  if constexpr (!Solo) asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"((unsigned)place & 15u));
  return a;
}
template <bool Solo>
__device__ __forceinline__ void load(unsigned a, double& v) {
  if constexpr (Solo)
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  else
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
template <bool Solo>
__device__ __forceinline__ void load(unsigned a, float& v) {
  if constexpr (Solo)
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  else
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
template <bool Solo>
__device__ __forceinline__ void pass_barrier() {
  if constexpr (Solo) {
    __syncthreads();
  } else {
    cluster_arrive();
    cluster_wait();
  }
}

// a / d rounded as the IEEE division rounds it, from rd = 1 / d rounded to
// nearest: Newton steps on the quotient whose remainder the fused
// multiply-add gives exactly. a * rd is within two units in the last place,
// the first step brings it within one, and from there the step with the
// correctly rounded reciprocal rounds correctly (Markstein, IBM J. Res.
// Dev. 34, 1990). That holds while rd and the quotient are normal numbers and
// the remainder, a multiple of the product of both last places, is
// representable: for d and a * rd within the bounds below (|a| is then within
// 2^-811 and 2^813, the remainder a multiple of 2^-915; FP32 2^-93, 2^125
// and 2^-139). Outside them, and for infinities and NaN, the division itself;
// reciprocal() marks a d out of bounds with NaN, so that one test of a * rd
// sees all of it. (Values of a heat problem's rows lie inside; zeros, which
// a * rd has right with their sign, do not take the division either.)
//
// word: the part of a number that has its sign and exponent; the exponent's
// upper two bits differ (01, 10) in the middle half of its range, which is
// where a * rd has to lie: 2^-511 to 2^513, FP32 2^-63 to 2^65.
__device__ __forceinline__ unsigned word(double v) { return (unsigned)__double2hiint(v); }
__device__ __forceinline__ unsigned word(float v) { return __float_as_uint(v); }
template <class T>
__device__ __forceinline__ bool middle(T v) {
  const unsigned w = word(v);
  return ((w ^ (w << 1)) & 0x40000000u) != 0u;
}
__device__ __forceinline__ double reciprocal(double d) {
  return fabs(d) >= 0x1p-300 && fabs(d) <= 0x1p300 ? 1.0 / d : double(NAN);
}
__device__ __forceinline__ float reciprocal(float d) {
  return fabsf(d) >= 0x1p-30f && fabsf(d) <= 0x1p60f ? 1.0f / d : float(NAN);
}
__device__ __forceinline__ double fused(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fused(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// (The test runs beside the Newton steps: a cycle of 576 rows, all on one CTA,
// 28.3 us without a test, 29.0 so, 29.6 with the steps behind the test; of
// 65536 rows 117.0, 118.0 and 119.8.)
__device__ __forceinline__ void hold(double& v) { asm volatile("" : "+d"(v)); }
__device__ __forceinline__ void hold(float& v) { asm volatile("" : "+f"(v)); }
template <class T>
__device__ __noinline__ T divide_any(T a, T d) {
  return a / d;
}
template <class T>
__device__ __forceinline__ T divide(T a, T d, T rd) {
  const T q0 = a * rd;
  T q = fused(fused(-q0, d, a), rd, q0);
  q = fused(fused(-q, d, a), rd, q);
  hold(q);
  if (!middle(q0)) q = a == T(0) && rd == rd ? q0 : divide_any(a, d);
  return q;
}

// the barrier a step begins with (arrived at when the last one ended)
__device__ __forceinline__ void step_barrier(int flags, bool mine) {
  if (flags & kTailBarCluster)
    cluster_wait();
  else if ((flags & kTailBarCta) && mine)
    __syncthreads();
}

// the j-th slice of this thread's warp in the CTA of the given rank (-1: none)
template <class T>
__device__ __forceinline__ int slice_at(const TailLevel<T>& L, int rank, int j) {
  const int w = (threadIdx.x >> 5) + j * kTailWarps;
  const int s = (L.lc ? rank : 0) * L.per + w;
  return w < L.per && s < L.slices ? s : -1;
}

// A visit of level L: all passes of a smoothing step, and the residual. K
// entries of each of the thread's R rows are in registers; further ones
// (only K = kTailRow) are read in every pass.
template <class T, int K, int R, bool Solo>
__device__ __forceinline__ void smooth(const TailLevel<T>& L, unsigned smem, int rank, int op, int flags, int sweeps,
                                       T weight) {
  const int lane = threadIdx.x & 31, w = L.width;
  const unsigned xa = smem + L.x, toR = L.r - L.x;
  unsigned c[R][K], own[R];
  T v[R][K], d[R], rd[R], b[R];
  int colour[R], e0[R];  // colour -1: no row
#pragma unroll
  for (int j = 0; j < R; j++) {
    const int s = slice_at(L, rank, j);
    const int at = s * 32 + lane;
    int slot = -1;
    if (s >= 0) slot = __ldg(L.slot + at);
    colour[j] = slot >= 0 ? slot >> 20 : -1;
    own[j] = (threadIdx.x + j * kTailThreads) * (unsigned)sizeof(T);
    d[j] = rd[j] = T(1);
    e0[j] = s * w * 32 + lane;
#pragma unroll
    for (int k = 0; k < K; k++) {
      c[j][k] = xa + own[j];
      v[j][k] = T(0);
    }
    if (slot >= 0) {
#pragma unroll
      for (int k = 0; k < K; k++)
        if (k < w) {
          c[j][k] = (unsigned)__ldg(L.idx + e0[j] + k * 32);
          v[j][k] = __ldg(L.val + e0[j] + k * 32);
        }
      d[j] = __ldg(L.diag + at);
      rd[j] = __ldg(L.rdiag + at);
    }
  }
#pragma unroll
  for (int j = 0; j < R; j++)
    if (colour[j] >= 0) {
#pragma unroll
      for (int k = 0; k < K; k++)
        if (k < w) c[j][k] = element<T, Solo>(xa, (int)c[j][k]);
    }
  step_barrier(flags, true);
#pragma unroll
  for (int j = 0; j < R; j++) {
    b[j] = T(0);
    if (colour[j] >= 0) load<true>(smem + L.b + own[j], b[j]);
  }
  auto row = [&](int j, unsigned from, T sum) -> T {
    // eight gathers in flight at a time
    constexpr int G = K < 8 ? K : 8;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += G) {
      T x[G];
#pragma unroll
      for (int k = 0; k < G; k++)
        if (k0 + k < K) load<Solo>(c[j][k0 + k] + from, x[k]);
#pragma unroll
      for (int k = 0; k < G; k++)
        if (k0 + k < K) sum = sum + v[j][k0 + k] * x[k];
    }
    // (a plain if: nvcc 12.9 drops the return after an if constexpr here)
    if (K == kTailRow)
      for (int k = K; k < w; k++) {
        T y;
        load<Solo>(element<T, Solo>(xa + from, __ldg(L.idx + e0[j] + k * 32)), y);
        sum = sum + __ldg(L.val + e0[j] + k * 32) * y;
      }
    return sum;
  };
  auto put = [&](int j, unsigned to, T o) {
    if constexpr (sizeof(T) == 8)
      asm volatile("st.shared.f64 [%0], %1;" ::"r"(xa + to + own[j]), "d"((double)o) : "memory");
    else
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(xa + to + own[j]), "f"((float)o) : "memory");
  };
  bool first = true;
  if (flags & kTailZero) {
#pragma unroll
    for (int j = 0; j < R; j++)
      if (colour[j] >= 0) put(j, 0u, T(0));
    first = false;
  }
  if (op == kTailGs) {
    const int C = L.colors;
    const bool forward = (flags & kTailForward) != 0;
    for (int q = 0; q < sweeps; q++) {
      // forward over the colours, then back; a sweep after a reverse one
      // would repeat its last pass (see AmgHierarchy::sweeps)
      const int last = forward ? C - 1 : 2 * C - 2;
      for (int p = (q > 0 && !forward) ? 1 : 0; p <= last; p++) {
        const int now = p < C ? p : 2 * C - 2 - p;
        if (!first) pass_barrier<Solo>();
        first = false;
#pragma unroll
        for (int j = 0; j < R; j++)
          if (colour[j] == now) put(j, 0u, divide(-row(j, 0u, b[j]), d[j], rd[j]));
      }
    }
  } else {
    for (int q = 0; q < 2 * sweeps; q++) {
      const unsigned from = (q & 1) ? toR : 0u, to = (q & 1) ? 0u : toR;
      if (!first) pass_barrier<Solo>();
      first = false;
#pragma unroll
      for (int j = 0; j < R; j++)
        if (colour[j] >= 0) {
          T o = divide(-row(j, from, b[j]), d[j], rd[j]);
          if (op == kTailDamped) {
            T xo;
            load<true>(xa + from + own[j], xo);
            o = xo + weight * (o - xo);
          }
          put(j, to, o);
        }
    }
  }
  if (flags & kTailResidual) {
    if (!first) pass_barrier<Solo>();
#pragma unroll
    for (int j = 0; j < R; j++)
      if (colour[j] >= 0) {
        // reference order: r = b + d x, then r += a_ij x_j
        T xo;
        load<true>(xa + own[j], xo);
        put(j, toR, row(j, 0u, b[j] + d[j] * xo));
      }
  }
}

template <class T>
__global__ void __launch_bounds__(kTailThreads, 1) k_cycle_tail(const __grid_constant__ TailArgs<T> a) {
  extern __shared__ __align__(16) unsigned char shared[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const unsigned smem = (unsigned)__cvta_generic_to_shared(shared);
  const int rank = (int)cluster_rank();
  const int lane = threadIdx.x & 31, t = threadIdx.x;
  auto fetch = [&](int k) {
    const int4 q = __ldg(reinterpret_cast<const int4*>(a.steps) + k);
    return TailStep{q.x, q.y, q.z, q.w};
  };
  TailStep cur = fetch(0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int k = 0; k < a.nSteps; k++) {
    const int op = cur.op & 255, flags = cur.op >> 8;
    const TailLevel<T>& L = a.lv[cur.level];
    const bool mine = !(flags & kTailSolo) || rank == 0;
    TailStep nxt = cur;
    if (k + 1 < a.nSteps) nxt = fetch(k + 1);
    if (op >= kTailGs && op <= kTailDamped) {
      // the registers hold the thread's rows (one, or two of up to
      // kTailTwo entries) at the level's width, rounded up
#define FVM_TAIL_ROWS(K, R, SOLO) smooth<T, K, R, SOLO>(L, smem, rank, op, flags, cur.n, a.w)
#define FVM_TAIL_WIDTHS(SOLO)            \
  if (L.width <= 4)                      \
    FVM_TAIL_ROWS(4, 1, SOLO);           \
  else if (L.width <= 8)                 \
    FVM_TAIL_ROWS(8, 1, SOLO);           \
  else if (L.width <= 12)                \
    FVM_TAIL_ROWS(12, 1, SOLO);          \
  else if (L.width <= 16)                \
    FVM_TAIL_ROWS(16, 1, SOLO);          \
  else                                   \
    FVM_TAIL_ROWS(kTailRow, 1, SOLO);
      if (L.lc == 0) {
        if (mine) {
          FVM_TAIL_WIDTHS(true)
        } else if (flags & kTailBarCluster) {
          cluster_wait();
        }
      } else if (L.per <= kTailWarps) {
        FVM_TAIL_WIDTHS(false)
      } else if (L.width <= 4) {
        FVM_TAIL_ROWS(4, 2, false);
      } else if (L.width <= 8) {
        FVM_TAIL_ROWS(8, 2, false);
      } else {
        FVM_TAIL_ROWS(kTailTwo, 2, false);
      }
#undef FVM_TAIL_WIDTHS
#undef FVM_TAIL_ROWS
    } else if (op == kTailRestrict || op == kTailRestrictRhs) {
      // one thread per row of the next level, in the CTA that holds it
      const TailLevel<T>& C = a.lv[cur.level + 1];
      const unsigned src = smem + (op == kTailRestrict ? L.r : L.b);
      bool waited = false;
      for (int j = 0; j < kTailRowsMax; j++) {
        const int s = mine ? slice_at(C, rank, j) : -1;
        int e0 = 0, e1 = 0, c0 = 0, c1 = 0;
        bool live = false;
        if (s >= 0) {
          const int I = __ldg(C.slot + s * 32 + lane);
          live = I >= 0;
          if (live) {
            e0 = __ldg(L.c2fRow + (I & 0xfffff));
            e1 = __ldg(L.c2fRow + (I & 0xfffff) + 1);
            if (e0 < e1) c0 = __ldg(L.c2fIdx + e0);
            if (e0 + 1 < e1) c1 = __ldg(L.c2fIdx + e0 + 1);
          }
        }
        if (!waited) step_barrier(flags, mine);
        waited = true;
        if (live) {
          T sum = T(0), v0 = T(0), v1 = T(0);
          if (e0 < e1) load<false>(element<T, false>(src, c0), v0);
          if (e0 + 1 < e1) load<false>(element<T, false>(src, c1), v1);
          if (e0 < e1) sum = sum + v0;
          if (e0 + 1 < e1) sum = sum + v1;
          for (int e = e0 + 2; e < e1; e++) {
            load<false>(element<T, false>(src, __ldg(L.c2fIdx + e)), v0);
            sum = sum + v0;
          }
          reinterpret_cast<T*>(shared + C.b)[t + j * kTailThreads] = sum;
          reinterpret_cast<T*>(shared + C.x)[t + j * kTailThreads] = T(0);
        }
      }
    } else {
      const bool up = op == kTailProlong || op == kTailAssign;
      bool waited = false;
      for (int j = 0; j < kTailRowsMax; j++) {
        const int s = mine ? slice_at(L, rank, j) : -1;
        int i = -1, c = -1;
        if (s >= 0) {
          i = __ldg(L.slot + s * 32 + lane);
          if (i >= 0) i &= 0xfffff;
          if (up) c = __ldg(L.ci + s * 32 + lane);
        }
        if (!waited) step_barrier(flags, mine);
        waited = true;
        if (i >= 0) {
          T* x = reinterpret_cast<T*>(shared + L.x) + t + j * kTailThreads;
          if (up) {
            T v = T(0);
            if (c >= 0) load<false>(element<T, false>(smem + a.lv[cur.level + 1].x, c), v);
            if (op == kTailAssign)
              *x = v;
            else if (c >= 0)
              *x = *x + v;
          } else if (op == kTailLoad) {
            reinterpret_cast<T*>(shared + L.b)[t + j * kTailThreads] = a.bIn[i];
            *x = (flags & kTailZero) ? T(0) : a.xIo[i];
          } else {
            a.xIo[i] = *x;
          }
        }
      }
    }
    if (k + 1 < a.nSteps && ((nxt.op >> 8) & kTailBarCluster)) cluster_arrive();
    cur = nxt;
  }
  // no CTA leaves while another may still read its shared memory
  cluster_arrive();
  cluster_wait();
}

// the place of row i of a level: thread index * 16 + CTA
template <class T>
__device__ __forceinline__ int place(const TailLevel<T>& L, const TailPack<T>& P, int i) {
  int s = i >> 5, lane = i & 31;
  if (!P.a.ellWidth) {
    s = P.rowSlice[i];
    lane = i - P.a.meta[s].x;
  }
  const int h = P.home[s];
  return (((h % L.per) * 32 + lane) << 4) | (h / L.per);
}

// The levels' matrices and maps in the kernel's own form: blockIdx.y is a
// level, the threads stride over its slots
template <class T>
__global__ void __launch_bounds__(128) k_tail_pack(const __grid_constant__ TailArgs<T> a,
                                                   const __grid_constant__ TailPackArgs<T> p) {
  const int l = blockIdx.y;
  const TailLevel<T>& L = a.lv[l];
  const TailPack<T>& P = p.lv[l];
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (int q = t0; q < L.slices * 32; q += nt) {
    const int h = q >> 5, lane = q & 31, s = P.order[h];
    int4 m;
    if (P.a.ellWidth)
      m = make_int4(s * 32, min(32, L.n - s * 32), s * 32 * P.a.ellWidth, P.a.ellWidth);
    else
      m = P.a.meta[s];
    const bool live = lane < m.y;
    const int i = m.x + lane;
    int colour = 0;
    if (live && P.colorRow)
      while (i >= P.colorRow[colour + 1]) colour++;
    P.slot[q] = live ? i | colour << 20 : -1;
    const T d = live ? P.a.diag[i] : T(1);
    P.diag[q] = d;
    P.rdiag[q] = reciprocal(d);
    const int self = (((h % L.per) * 32 + lane) << 4) | (h / L.per);
    for (int k = 0; k < L.width; k++) {
      const int e = (h * L.width + k) * 32 + lane;
      const bool has = live && k < m.w;  // padding: the row itself, times zero
      P.idx[e] = has ? place(L, P, P.a.cols[m.z + (k << 5) + lane]) : self;
      P.val[e] = has ? P.a.vals[m.z + (k << 5) + lane] : T(0);
    }
    if (P.ciOut) {
      const int c = live ? P.ci[i] : -1;
      P.ciOut[q] = c >= 0 ? place(a.lv[l + 1], p.lv[l + 1], c) : -1;
    }
  }
  if (P.c2fOut)
    for (int e = t0, m = P.c2fRow[P.nCoarse]; e < m; e += nt) P.c2fOut[e] = place(L, P, P.c2fCol[e]);
}

template <class T>
cudaError_t prepare(size_t smemBytes) {
  cudaError_t e = cudaFuncSetAttribute(k_cycle_tail<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_cycle_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemBytes);
  return e;
}

template <class T>
cudaLaunchConfig_t config(int lc, size_t smemBytes, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1u << lc);
  cfg.blockDim = dim3(kTailThreads);
  cfg.dynamicSmemBytes = smemBytes;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1u << lc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

template <class T>
int cluster_for(size_t smemBytes) {
  if (prepare<T>(smemBytes) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  for (int lc = 4; lc >= 3; lc--) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = config<T>(lc, smemBytes, nullptr, attr);
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_cycle_tail<T>, &cfg) == cudaSuccess && n >= 1) return lc;
    cudaGetLastError();
  }
  return -1;
}

}  // namespace

int cycle_tail_cluster(bool f32, size_t smemBytes) {
  return f32 ? cluster_for<float>(smemBytes) : cluster_for<double>(smemBytes);
}

template <class T>
void cycle_tail_pack(const TailArgs<T>& a, const TailPackArgs<T>& p, cudaStream_t st) {
  k_tail_pack<T><<<dim3(64, p.levels), 128, 0, st>>>(a, p);
}
template void cycle_tail_pack<float>(const TailArgs<float>&, const TailPackArgs<float>&, cudaStream_t);
template void cycle_tail_pack<double>(const TailArgs<double>&, const TailPackArgs<double>&, cudaStream_t);

template <class T>
void cycle_tail(const TailArgs<T>& a, size_t smemBytes, cudaStream_t st) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = config<T>(a.lc, smemBytes, st, attr);
  launchesIssued++;
  cudaLaunchKernelEx(&cfg, k_cycle_tail<T>, a);
}
template void cycle_tail<float>(const TailArgs<float>&, size_t, cudaStream_t);
template void cycle_tail<double>(const TailArgs<double>&, size_t, cudaStream_t);

}  // namespace dev
}  // namespace fvm
