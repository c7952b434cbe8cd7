// The coarse levels of an AMG cycle as one thread-block-cluster kernel.
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace fvm {
namespace dev {

constexpr int kTailMaxLevels = 20;
constexpr int kTailThreads = 512;
constexpr int kTailWarps = kTailThreads / 32;
// A thread holds one row of a level in registers, kTailRow entries of it at
// most, or two rows of at most kTailTwo entries.
constexpr int kTailRow = 24;
constexpr int kTailTwo = 12;
constexpr int kTailRowsMax = 2;
constexpr int kTailMaxColors = 2047;  // a slot holds its row in 20 bits, its colour above

enum TailOp {
  kTailLoad = 0,     // b <- global; x <- global or (flag) 0
  kTailGs,           // n Gauss-Seidel sweeps over the colours
  kTailJacobi,       // n sweeps of two Jacobi passes
  kTailDamped,       // n sweeps of two damped Jacobi passes
  kTailRestrict,     // next level's b = sum of r over its rows, its x = 0
  kTailRestrictRhs,  // the same of b (zero guess, no pre-smoothing)
  kTailProlong,      // x += next level's x
  kTailAssign,       // x = next level's x
  kTailStore         // global <- x
};
// flags of a step
constexpr int kTailSolo = 1;        // executed by the cluster's first CTA alone
constexpr int kTailZero = 2;        // kTailLoad: x = 0; a smoothing step: x = 0 first
constexpr int kTailBarCta = 4;      // barrier before the step: the CTA's
constexpr int kTailBarCluster = 8;  //                          the cluster's
constexpr int kTailResidual = 16;   // a smoothing step (n may be 0) ends with r = b + A x
constexpr int kTailForward = 32;    // Gauss-Seidel sweeps without their reverse pass

struct TailStep {
  int op, level;  // op | flags << 8
  int n, pad;
};

// One level in slots of one row each, 32 slots per slice as the level's
// SELL-32 / ELL-32 slices have them. Slices are renumbered so that slices
// at like places of their colours, whose rows couple, follow each other;
// slice h then belongs to CTA h div per, there to warp (h mod per) mod 16.
// So a thread has one or two rows of a level, a row's x, b and r are at the
// thread's own index (+ 512 for the second) in its CTA's shared memory, and most of its columns are in the same
// CTA. A column is stored as the place of its row: that index * 16 + CTA.
template <class T>
struct TailLevel {
  int n, slices, lc, per;
  int width;  // entries per slot
  int colors;
  const int* slot;       // row | colour << 20, -1: none
  const int* idx;        // (slice * width + k) * 32 + lane: column's place
  const T* val;
  const T *diag, *rdiag;       // by slot: diagonal and its reciprocal (NaN: see divide)
  const int* ci;               // by slot: coarse row's place (-1: none)
  const int *c2fRow, *c2fIdx;  // by coarse row: places of its rows
  unsigned x, b, r;            // byte offsets in shared memory
};

template <class T>
struct TailArgs {
  TailLevel<T> lv[kTailMaxLevels];
  const TailStep* steps;
  int nSteps;
  int lc;  // log2 of the cluster size
  T w;     // damped-Jacobi weight
  const T* bIn;
  T* xIo;
};

// Input of tail_pack for one level: the matrix as the other kernels read it
// and the transfer maps, to be rewritten into the arrays above.
template <class T>
struct TailPack {
  SellView<T> a;
  const int* rowSlice;
  const int *order, *home;  // new slice -> slice and back
  const int* colorRow;  // colors + 1 first rows of the colours (null: one colour)
  const int *ci, *c2fRow, *c2fCol;
  int nCoarse;
  int *slot, *idx;
  T* val;
  T *diag, *rdiag;
  int *ciOut, *c2fOut;
};
template <class T>
struct TailPackArgs {
  TailPack<T> lv[kTailMaxLevels];
  int levels;
};

// log2 of the cluster size the device runs with smemBytes of dynamic shared
// memory per CTA, -1 when no cluster of eight or sixteen fits
int cycle_tail_cluster(bool f32, size_t smemBytes);
// fills every level's arrays (a: the levels as cycle_tail will get them)
template <class T>
void cycle_tail_pack(const TailArgs<T>& a, const TailPackArgs<T>& p, cudaStream_t st);
template <class T>
void cycle_tail(const TailArgs<T>& a, size_t smemBytes, cudaStream_t st);

}  // namespace dev
}  // namespace fvm
