// BiCGStab on the GPU: the recurrences of the reference solver
// (gpu/bicgstab.cu:387-513, optional point-Jacobi right preconditioning as in
// :201-238), restructured for GB300.
//
// One iteration is five phases over all rows on a fixed grid; the scalars
// rho, alpha, omega, beta live in device memory (DevState), so no host round
// trip separates the phases (the reference did four blocking copies and a
// print per iteration, gpu/bicgstab.cu:447-510):
//
//   phase 1  p = r + beta (p - omega v);   q = P p
//   phase 2  v = A q, partial (rh, v)       fused into the SpMV epilogue
//            -> alpha = rho / (rh, v)
//   phase 3  s = r - alpha v;  z = P s
//   phase 4  t = A z, partials (t, s), (t, t)
//            -> omega = (t, s) / (t, t)
//   phase 5  x' += alpha q + omega z;  r = s - omega t
//            partials (rh, r), (r, r), (x', x')
//            -> convergence, limit and breakdown tests, the replacement
//               decision, beta = (rho / rho_prev)(alpha / omega)
//
// Algorithmic traffic per iteration: 2 SpMV + 17 n vector elements (no
// preconditioner). Each CTA reduces its threads' terms to one partial per dot
// product; the CTA that finishes a phase last (an acq_rel arrival counter)
// sums the grid's partials in index order and derives the scalars (the
// arrows above), so a solve is deterministic for a given grid.
//
// The phases run in one of two ways, with the same bits on the same grid:
// a CUDA graph of five kernels per iteration (`chunk` iterations per graph),
// or one persistent cooperative kernel per `chunk` iterations whose phases
// are separated by grid barriers, the last CTA to reach a barrier doing the
// phase's scalar work (the auto choice from kPersistentRows rows). Below that
// the auto mode runs the same recurrences in one cooperative kernel whose CTAs
// keep their rows' vectors in shared memory (resident.cuh). The host only
// polls the done flag between launches; phases after convergence return at
// once.
//
// Residual replacement with group update (van der Vorst and Ye 2000, see
// DevState): the decision at the end of phase 5 tracks the deviation bound
// and, when it is time, the next iteration's phase 1 does the fold
// g += x', x' = 0 instead of the p update; phase 2 then computes r = c - A g
// instead of v = A q (and (rh, r), (r, r)), phases 3 and 4 return at once and
// phase 5 only takes the decision on those sums. No kernel is added to the
// graph for it.
//
// Differences from the reference, on purpose: the solution returned is the
// last iterate (the reference copied buffer half 0, bicgstab.cu:515), the
// recursive residual is replaced by the true one near convergence (above),
// and a solve finishes with a true-residual check b - A x (restarting from
// the true residual when the recursive one has drifted below the tolerance
// first).
#include "reduce.cuh"
#include "solver.h"
#include "spmv_core.cuh"

#include <cuda/atomic>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

namespace bmfp
{
using namespace reduce;

namespace
{
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

enum PartKind
{
  kRhR = 0,
  kRR = 1,
  kRhV = 2,
  kTS = 3,
  kTT = 4,
  kResRR = 5,
  kResBB = 6,
  kXX = 7, // (x', x') of phase 5
  kGG = 8, // (g, g) after a fold (phase 1) or 0 at a run's start
  kParts = 9
};
// The allocation-free entry point sizes its partial-sum slot by kRawParts.
static_assert (kParts == kRawParts, "solver.h kRawParts must equal the number of partial kinds");

template <typename T> struct Args
{
  int nbr, bs;
  const int *rp, *cols;
  const T *vals;
  int64_t n;
  T *x, *r, *rh, *p, *v, *q, *s, *z, *t;
  const T *P;
  T *g, *xp; // group base and updates accumulated since the last replacement
  double *part;
  int grid;
  DevState *st;
  // Sliced copy of a CSR or bs = 2 matrix (SellOp), or null.
  const int *soff, *scols;
  const T *svals;
  bool stream; // the sliced copy does not stay in L2
  int nslices;
};

// done and rep_now in one load. Both are written by earlier kernels (done
// also by block 0 of phases 1, 3 and 5, in cases where every block of that
// phase takes the same early return anyway), so a plain load suffices.
__device__ __forceinline__ int2 flags (const DevState *st)
{
  return *reinterpret_cast<const int2 *> (&st->done);
}

__device__ __forceinline__ bool is_done (const DevState *st) { return flags (st).x != 0; }

// Sum the grid partials of NK kinds in a fixed order, broadcast to the CTA.
// Every thread loads its share of the partials at once (the grid is a few
// CTAs per SM, so a handful of loads each), then the warps sum, and warp k
// sums the warps' totals of kind k.
template <int NK>
__device__ __forceinline__ void sum_parts (const double *part, int grid, const int (&ks)[NK],
                                           double (&out)[NK])
{
  __shared__ double sh_w[NK][kWarps];
  __shared__ double sh[NK];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double acc[NK];
#pragma unroll
  for (int k = 0; k < NK; k++)
    acc[k] = 0.0;
  // __ldcg: the partials were written by other CTAs of this kernel (L2 is
  // coherent, this SM's L1 need not be)
  for (int i = threadIdx.x; i < grid; i += kThreads)
#pragma unroll
    for (int k = 0; k < NK; k++)
      acc[k] += __ldcg (part + ks[k] * grid + i);
  double ws[NK];
  warp_sums<NK> (acc, ws);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NK; k++)
      sh_w[k][w] = ws[k];
  __syncthreads ();
  if (w < NK)
    {
      const double a = warp_sum (lane < kWarps ? sh_w[w][lane] : 0.0);
      if (lane == 0)
        sh[w] = a;
    }
  __syncthreads ();
#pragma unroll
  for (int k = 0; k < NK; k++)
    out[k] = sh[k];
}

// True in exactly one CTA of the kernel: the last to finish writing its
// partials (each CTA's thread 0 wrote them, fences, then counts itself in
// st->arrive). That CTA resets the counter for the next kernel. No thread
// waits on another: the last CTA just finds everyone else already done.
__device__ __forceinline__ bool arrive_last (DevState *st, int grid)
{
  __shared__ int sh_last;
  __syncthreads ();
  if (threadIdx.x == 0)
    {
      // acq_rel at device scope: releases this thread's partial writes to
      // the CTA that comes last, and acquires everyone's for that CTA.
      cuda::atomic_ref<unsigned, cuda::thread_scope_device> arrive (st->arrive);
      const unsigned t = arrive.fetch_add (1u, cuda::memory_order_acq_rel);
      sh_last = t == (unsigned) grid - 1;
      if (sh_last)
        arrive.store (0u, cuda::memory_order_relaxed);
    }
  __syncthreads ();
  return sh_last != 0;
}

// Reduce per-thread values over the CTA into part[k][blockIdx]: warps, then
// warp k over the warps' totals of kind k.
template <int NK>
__device__ __forceinline__ void store_parts (double (&v)[NK], double *part, int grid,
                                             const int (&ks)[NK])
{
  __shared__ double sh[NK][kWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double ws[NK];
  warp_sums<NK> (v, ws);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NK; k++)
      sh[k][w] = ws[k];
  __syncthreads ();
#pragma unroll
  for (int k = 0; k < NK; k++)
    if (w == k)
      {
        const double a = warp_sum (lane < kWarps ? sh[k][lane] : 0.0);
        if (lane == 0)
          part[ks[k] * grid + blockIdx.x] = a;
      }
}

#define GRID_STRIDE(i, n)                                                                          \
  for (int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < (n);                       \
       i += (int64_t) gridDim.x * blockDim.x)

// ------------------------------------------------------------ SpMV phases

template <typename T, int BS, int G, class XL = dev::XNc> struct FlatOp
{
  template <class Epi>
  __device__ static void run (const Args<T> &a, const T *x, T *y, Epi &e)
  {
    const int64_t group = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int64_t ng = (int64_t) gridDim.x * blockDim.x / G;
    for (int64_t row = group; row < a.nbr; row += ng)
      core::flat_row<T, BS, G, 4, XL> ((int) row, a.rp, a.cols, a.vals, x, y, e);
  }
};

// Scalar rows per slice of the sliced matrix: one warp, one row per lane.
constexpr int kSlice = 32;

// Block size B = 1 (CSR) or 2 on the sliced copy: step k of a slice holds line r
// of the k-th block of each of its 32 scalar rows side by side, so a warp reads
// 512 (FP64, B = 2) consecutive bytes per step where the row-by-row walk of the block rows
// touched 16 lines, and every lane runs the same number of steps. Three
// steps' x in flight and the next three steps' values and columns behind
// them: the walk is bound by latency otherwise. Rows are padded to the
// slice's longest with zero blocks on a column the row already reads.
// Steps that fill no group run together too: taken one by one, each waited for its
// column and then its x, and rows of 5 to 8 blocks were slower than the walk of
// the block rows (us per iteration, block rows / one by one / together: FP32,
// 1.2 M rows, persistent, 7 blocks 67 / 92 / 68; FP64, 400 000 rows, graphs with
// one CTA per SM, 5 blocks 64 / 73 / 55, 8 blocks 81 / 92 / 76).
// A copy larger than L2 is read evict-first, columns included (Stream).
// 2000x500 Q4 grid, FP64, phases 2 and 4 by block rows and by slices: 84.5 and
// 88.4 us -> 74.9 and 80.3 us (FP64 pipe 74 % -> 80 % busy, its work alone 61
// and 64 us).
template <typename T, int B, class XL = dev::XNc> struct SellOp
{
  static constexpr int U = sizeof (T) == 4 ? 9 : B == 1 ? 6 : 3;
  // Steps that fill no group: in the FP64 phase kernels first, with the first
  // group on its way behind them, else last (the persistent kernel's 80 registers
  // do not hold both).
  static constexpr bool kAhead = sizeof (T) == 8 && std::is_same_v<XL, dev::XNc>;
  struct Step
  {
    T v[B];
    int c;
  };
  template <bool Stream> __device__ static __forceinline__ Step load (const T *v, const int *c, int k)
  {
    Step s;
    if constexpr (B == 1)
      s.v[0] = __ldcs (v + (size_t) k * kSlice);
    else if constexpr (sizeof (T) == 8)
      {
        const double2 t = __ldcs (reinterpret_cast<const double2 *> (v) + (size_t) k * kSlice);
        s.v[0] = t.x;
        s.v[1] = t.y;
      }
    else
      {
        const float2 *q = reinterpret_cast<const float2 *> (v) + (size_t) k * kSlice;
        const float2 t = Stream ? __ldcs (q) : __ldg (q);
        s.v[0] = t.x;
        s.v[1] = t.y;
      }
    const int *q = c + (size_t) k * (kSlice / B);
    s.c = Stream ? __ldcs (q) : __ldg (q);
    return s;
  }
  __device__ static __forceinline__ void gather (const T *x, int c, T (&xv)[B])
  {
    if constexpr (B == 1)
      xv[0] = XL::ld (x + c);
    else
      XL::ld2 (x + (size_t) c * 2, xv[0], xv[1]);
  }
  __device__ static __forceinline__ T add (const Step &s, const T (&xv)[B], T acc)
  {
#pragma unroll
    for (int j = 0; j < B; j++)
      acc = fma (s.v[j], xv[j], acc);
    return acc;
  }
  template <class Epi>
  __device__ static __forceinline__ void run (const Args<T> &a, const T *x, T *y, Epi &e)
  {
    if constexpr (B == 1 || sizeof (T) == 4)
      if (a.stream)
        {
          walk<true> (a, x, y, e);
          return;
        }
    walk<false> (a, x, y, e);
  }
  template <bool Stream, class Epi>
  __device__ static __forceinline__ void walk (const Args<T> &a, const T *x, T *y, Epi &e)
  {
    const int lane = threadIdx.x & 31;
    const int nw = (int) (gridDim.x * blockDim.x / kSlice);
    int slice = (int) ((blockIdx.x * blockDim.x + threadIdx.x) / kSlice);
    if (slice >= a.nslices)
      return;
    int beg = __ldg (a.soff + slice), end = __ldg (a.soff + slice + 1);
    for (;;)
      {
        const int next = slice + nw;
        int nbeg = 0, nend = 0;
        if (next < a.nslices)
          {
            nbeg = __ldg (a.soff + next);
            nend = __ldg (a.soff + next + 1);
          }
        const int64_t i = (int64_t) slice * kSlice + lane;
        if (i < a.n)
          e.pre (i);
        const T *v = a.svals + ((size_t) beg * kSlice + lane) * B;
        const int *c = a.scols + (size_t) beg * (kSlice / B) + lane / B;
        const int n = end - beg;
        T acc = 0;
        // The odd steps, together: past their end the last again, not added.
        auto odd = [&] (int from, int left) {
          Step t[U - 1];
          T xv[U - 1][B];
#pragma unroll
          for (int u = 0; u < U - 1; u++)
            t[u] = load<Stream> (v, c, from + min (u, left - 1));
#pragma unroll
          for (int u = 0; u < U - 1; u++)
            gather (x, t[u].c, xv[u]);
#pragma unroll
          for (int u = 0; u < U - 1; u++)
            if (u < left)
              acc = add (t[u], xv[u], acc);
        };
        int k = kAhead ? n % U : 0;
        Step s[U];
        if (n >= U)
#pragma unroll
          for (int u = 0; u < U; u++)
            s[u] = load<Stream> (v, c, k + u);
        if (kAhead && k > 0)
          odd (0, k);
        if (n >= U)
          {
            for (; k + 2 * U <= n; k += U)
              {
                Step t[U];
                T xv[U][B];
#pragma unroll
                for (int u = 0; u < U; u++)
                  gather (x, s[u].c, xv[u]);
#pragma unroll
                for (int u = 0; u < U; u++)
                  t[u] = load<Stream> (v, c, k + U + u);
#pragma unroll
                for (int u = 0; u < U; u++)
                  acc = add (s[u], xv[u], acc);
#pragma unroll
                for (int u = 0; u < U; u++)
                  s[u] = t[u];
              }
            T xv[U][B];
#pragma unroll
            for (int u = 0; u < U; u++)
              gather (x, s[u].c, xv[u]);
#pragma unroll
            for (int u = 0; u < U; u++)
              acc = add (s[u], xv[u], acc);
            k += U;
          }
        if (!kAhead && k < n)
          odd (k, n - k);
        if (i < a.n)
          {
            y[i] = acc;
            e.now (i, acc);
          }
        if (next >= a.nslices)
          break;
        slice = next;
        beg = nbeg;
        end = nend;
      }
  }
};

// The sliced copy's layout: slice widths (its longest row, in blocks), their
// running sum by one CTA (off[nslices] the total), and the fill.
__global__ void sell_width_kernel (int nbr, int per, const int *rp, int nslices, int *width)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nslices)
    return;
  const int r1 = min (nbr, (s + 1) * per);
  int w = 0;
  for (int r = s * per; r < r1; r++)
    w = max (w, rp[r + 1] - rp[r]);
  width[s] = w;
}

__global__ void __launch_bounds__ (1024) sell_scan_kernel (int nslices, const int *width, int *off,
                                                           unsigned long long *total)
{
  __shared__ unsigned long long sh[1024];
  const int per = (nslices + 1023) / 1024;
  const int64_t s0 = min ((int64_t) nslices, (int64_t) threadIdx.x * per), s1 = min ((int64_t) nslices, s0 + per);
  unsigned long long sum = 0;
  for (int64_t s = s0; s < s1; s++)
    sum += (unsigned) width[s];
  sh[threadIdx.x] = sum;
  __syncthreads ();
  for (int h = 1; h < 1024; h <<= 1)
    {
      const unsigned long long v = (int) threadIdx.x >= h ? sh[threadIdx.x - h] : 0;
      __syncthreads ();
      sh[threadIdx.x] += v;
      __syncthreads ();
    }
  unsigned long long at = sh[threadIdx.x] - sum;
  for (int64_t s = s0; s < s1; s++)
    {
      off[s] = (int) at;
      at += (unsigned) width[s];
    }
  if (threadIdx.x == 1023)
    {
      off[nslices] = (int) sh[1023];
      *total = sh[1023];
    }
}

template <typename T, int B>
__global__ void sell_fill_kernel (int nbr, const int *rp, const int *cols, const T *vals, int nslices, const int *off,
                                  int *scols, T *svals)
{
  const int lane = threadIdx.x & 31;
  const int nw = (int) (gridDim.x * blockDim.x / 32);
  for (int s = (int) ((blockIdx.x * blockDim.x + threadIdx.x) / 32); s < nslices; s += nw)
    {
      const int row = s * (kSlice / B) + lane / B;
      const int beg = row < nbr ? rp[row] : 0, len = row < nbr ? rp[row + 1] - beg : 0;
      const int pad = len > 0 ? cols[beg] : min (row, nbr - 1);
      const int o = off[s], w = off[s + 1] - o;
      for (int k = 0; k < w; k++)
        {
          const size_t at = ((size_t) (o + k) * kSlice + lane) * B;
          const bool in = k < len;
          for (int j = 0; j < B; j++)
            svals[at + j] = in ? vals[(size_t) (beg + k) * B * B + (lane % B) * B + j] : (T) 0;
          if (lane % B == 0)
            scols[(size_t) (o + k) * (kSlice / B) + lane / B] = in ? cols[beg + k] : pad;
        }
    }
}

template <typename T, int BSC, class XL = dev::XNc> struct TprOp
{
  template <class Epi>
  __device__ static void run (const Args<T> &a, const T *x, T *y, Epi &e)
  {
    const int64_t warp = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = (int64_t) gridDim.x * blockDim.x >> 5;
    for (int64_t row = warp; row < a.nbr; row += nw)
      core::tpr_row<T, BSC, XL> ((int) row, a.bs, a.rp, a.cols, a.vals, x, y, e);
  }
};

template <typename T, int G, class XL = dev::XNc> struct CsrOp
{
  template <class Epi>
  __device__ static void run (const Args<T> &a, const T *x, T *y, Epi &e)
  {
    const int64_t group = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int64_t ng = (int64_t) gridDim.x * blockDim.x / G;
    for (int64_t row = group; row < a.nbr; row += ng)
      core::csr_row<T, G, XL> ((int) row, a.rp, a.cols, a.vals, x, y, e);
  }
};

// Dot-product accumulators of the SpMV epilogues and phase 5 run in T: each
// thread sums a handful of terms, then warps, CTAs and the grid combine the
// partials in FP64. For FP64 solves that is FP64 throughout; the FP32 engine
// (inner solves of mixed precision, asked for 1e-4) keeps GB300's narrow
// FP64 pipe out of its per-element work.
template <typename T> struct EpiDot
{
  const T *a;
  T acc = 0;
  T ai = 0; // a[i], where the product routine asks for it ahead (pre)
  __device__ void pre (int64_t i) { ai = a[i]; }
  __device__ void operator() (int64_t i, T y) { acc = fma (a[i], y, acc); }
  __device__ void now (int64_t, T y) { acc = fma (ai, y, acc); }
};

template <typename T> struct EpiTS
{
  const T *s;
  T ts = 0, tt = 0;
  T si = 0;
  __device__ void pre (int64_t i) { si = s[i]; }
  __device__ void operator() (int64_t i, T t)
  {
    ts = fma (s[i], t, ts);
    tt = fma (t, t, tt);
  }
  __device__ void now (int64_t, T t)
  {
    ts = fma (si, t, ts);
    tt = fma (t, t, tt);
  }
};

template <typename T> struct EpiResidual
{
  const T *b;
  T *r;
  double rr = 0.0, bb = 0.0;
  __device__ void operator() (int64_t i, T y)
  {
    const T bi = b[i];
    const T ri = bi - y;
    r[i] = ri;
    rr = fma ((double) ri, (double) ri, rr);
    bb = fma ((double) bi, (double) bi, bb);
  }
  __device__ void pre (int64_t) {}
  __device__ void now (int64_t i, T y) { (*this) (i, y); }
};

// Residual replacement: r = c - A g, with (rh, r) and (r, r).
template <typename T> struct EpiReplace
{
  const T *c;
  T *r;
  const T *rh;
  T rhr = 0, rr = 0;
  __device__ void operator() (int64_t i, T y)
  {
    const T ri = c[i] - y;
    r[i] = ri;
    rhr = fma (rh[i], ri, rhr);
    rr = fma (ri, ri, rr);
  }
  __device__ void pre (int64_t) {}
  __device__ void now (int64_t i, T y) { (*this) (i, y); }
};

// The scalars that open an iteration, from the sums of (rh, r), (r, r) and nn
// ((g, g) after a replacement or at a run's start, which resets the deviation
// bound; else (x', x')): the convergence, limit and breakdown tests, the
// replacement decision and beta. One thread runs it, given the divides and
// square roots: rho / rho_prev, alpha / omega, ||r|| and sqrt (nn).
__device__ __forceinline__ void decide_scalars (DevState *st, double rho, double rr, double rho_ratio, double step_ratio,
                                                double nr, double root_nn, bool after_rep)
{
  const double eps = st->eps;
  double nb = st->norm_b;
  if (nb < 0.0)
    st->norm_b = nb = nr; // ||r0|| of a fresh solve
  int status = kStateRunning;
  double beta = 0.0;
  if (is_zero (nb) || less_abs (nr, st->tol * nb)) // gpu/bicgstab.cu:512
    status = kStateConverged;
  else if (st->iter >= st->max_iter)
    status = kStateMaxIter;
  else if (is_zero (rho) || is_zero (st->omega) || !is_finite (rho))
    status = kStateBreakdown;
  else
    {
      beta = rho_ratio * step_ratio; // gpu/bicgstab.cu:451
      if (!is_finite (beta))
        status = kStateBreakdown;
    }
  int rep = 0;
  if (status == kStateRunning && eps > 0.0)
    {
      const double limit = kReplaceThreshold * nr;
      if (after_rep)
        {
          st->dev = eps * (st->cA * root_nn + nr);
          st->dev_min = 1.1 * st->dev;
        }
      else
        {
          const double dev = fma (eps, st->cA * root_nn + nr, st->dev);
          rep = !less_abs (st->limit_prev, st->dev) && less_abs (limit, dev) && less_abs (st->dev_min, dev);
          st->dev = dev;
        }
      st->limit_prev = limit;
    }
  st->rr = rr;
  if (status != kStateRunning)
    {
      st->status = status;
      *reinterpret_cast<volatile int *> (&st->done) = 1;
    }
  else if (rep)
    {
      st->rep_now = 1;
      st->replacements = st->replacements + 1;
    }
  else
    {
      st->rep_now = 0;
      st->rho = rho;
      st->beta = beta;
    }
}

// The last CTA of the kernel that completed the sums runs this, all threads. An
// FP64 divide or square root takes about 700 cycles on GB300's narrow FP64
// pipe, so the four of them run side by side, one to a warp.
__device__ __forceinline__ void decide (DevState *st, double rho, double rr, double nn, bool after_rep,
                                        double rho_prev)
{
  __shared__ double sh[4];
  static_assert (kWarps >= 4, "one warp per divide and square root");
  if (threadIdx.x == 0)
    sh[0] = rho / rho_prev;
  else if (threadIdx.x == 32)
    sh[1] = st->alpha / st->omega;
  else if (threadIdx.x == 64)
    sh[2] = sqrt (rr);
  else if (threadIdx.x == 96)
    sh[3] = st->eps > 0.0 ? sqrt (nn) : 0.0;
  __syncthreads ();
  if (threadIdx.x == 0)
    decide_scalars (st, rho, rr, sh[0], sh[1], sh[2], sh[3], after_rep);
}

// Each phase is a body, run by every CTA, and (for phases that end in a dot
// product) a tail that turns the grid's partial sums into the next scalars.
// The phase kernels of the iteration graph run the tail in the last CTA to
// finish (arrive_last) on the device state in global memory; the persistent
// iteration kernel runs it in every CTA, on a copy of the state in shared
// memory, after a grid barrier. Both sum the partials in the same order, so
// both give the same bits.

// phase 2: v = A q, partial (rh, v). In a replacement iteration r = c - A g
// with partials (rh, r), (r, r) instead (A g lands in t, free until phase 4).
template <typename T, class Op> __device__ __forceinline__ void body_v (const Args<T> &a, const DevState *sc, bool rep)
{
  if (rep)
    {
      EpiReplace<T> e{ static_cast<const T *> (sc->c), a.r, a.rh };
      Op::run (a, a.g, a.t, e);
      double vals[2] = { (double) e.rhr, (double) e.rr };
      const int ks[2] = { kRhR, kRR };
      store_parts<2> (vals, a.part, a.grid, ks);
      return;
    }
  EpiDot<T> e{ a.rh };
  Op::run (a, a.q, a.v, e);
  double vals[1] = { (double) e.acc };
  const int ks[1] = { kRhV };
  store_parts<1> (vals, a.part, a.grid, ks);
}

// alpha from (rh, v), or a breakdown.
__device__ __forceinline__ void tail_v (DevState *st, const double *part, int grid)
{
  double sv[1];
  const int ks[1] = { kRhV };
  sum_parts<1> (part, grid, ks, sv);
  if (threadIdx.x == 0)
    {
      const double alpha = st->rho / sv[0]; // gpu/bicgstab.cu:466
      if (!is_zero (sv[0]) && is_finite (alpha))
        st->alpha = alpha;
      else
        {
          st->status = kStateBreakdown;
          *reinterpret_cast<volatile int *> (&st->done) = 1;
        }
    }
}

// phase 4: t = A z, partials (t, s), (t, t).
template <typename T, class Op> __device__ __forceinline__ void body_t (const Args<T> &a)
{
  EpiTS<T> e{ a.s };
  Op::run (a, a.z, a.t, e);
  double vals[2] = { (double) e.ts, (double) e.tt };
  const int ks[2] = { kTS, kTT };
  store_parts<2> (vals, a.part, a.grid, ks);
}

// omega from (t, s) and (t, t), or a breakdown.
__device__ __forceinline__ void tail_t (DevState *st, const double *part, int grid)
{
  double sv[2];
  const int ks[2] = { kTS, kTT };
  sum_parts<2> (part, grid, ks, sv);
  if (threadIdx.x == 0)
    {
      const double omega = is_zero (sv[1]) ? 0.0 : sv[0] / sv[1]; // :488
      if (is_finite (omega))
        st->omega = omega;
      else
        {
          // Leave x' untouched so the run keeps the last finite iterate.
          st->status = kStateBreakdown;
          *reinterpret_cast<volatile int *> (&st->done) = 1;
        }
    }
}

// End of an iteration: the decision that opens the next one, from (rh, r),
// (r, r) and (x', x') of phase 5, or in a replacement iteration from r,
// (rh, r) and (r, r) of phase 2 and (g, g) of phase 1.
__device__ __forceinline__ void tail_end (DevState *st, const double *part, int grid, bool rep)
{
  double sv[3];
  const int ks[3] = { kRhR, kRR, rep ? kGG : kXX };
  sum_parts<3> (part, grid, ks, sv);
  const double rho_prev = rep ? st->rho_prev : st->rho;
  __syncthreads (); // rho_prev is read
  if (threadIdx.x == 0 && !rep)
    {
      st->rho_prev = rho_prev;
      st->iter = st->iter + 1;
    }
  decide (st, sv[0], sv[1], sv[2], rep, rho_prev);
}

template <typename T, class Op>
__global__ void __launch_bounds__ (kThreads) phase_v (Args<T> a)
{
  DevState *st = a.st;
  const int2 f = flags (st);
  if (f.x)
    return;
  body_v<T, Op> (a, st, f.y != 0);
  if (f.y || !arrive_last (st, a.grid))
    return;
  tail_v (st, a.part, a.grid);
}

template <typename T, class Op>
__global__ void __launch_bounds__ (kThreads) phase_t (Args<T> a)
{
  DevState *st = a.st;
  const int2 f = flags (st);
  if (f.x || f.y)
    return;
  body_t<T, Op> (a);
  if (!arrive_last (st, a.grid))
    return;
  tail_t (st, a.part, a.grid);
}

// r = b - A x (x given), partials ||r||^2, ||b||^2 — the true residual.
template <typename T, class Op>
__global__ void __launch_bounds__ (kThreads)
  residual_kernel (Args<T> a, const T *x, const T *b, T *r, T *y)
{
  EpiResidual<T> e{ b, r };
  Op::run (a, x, y, e);
  double vals[2] = { e.rr, e.bb };
  const int ks[2] = { kResRR, kResBB };
  store_parts<2> (vals, a.part, a.grid, ks);
}

// ------------------------------------------------------------ vector phases

// Start of a run solving A e = c from e = 0 (ZERO: a fresh solve; else a
// restart whose c is the true residual of the current x). x itself is not
// touched until the run ends. Its last CTA takes the first decision.
template <typename T, bool ZERO>
__global__ void __launch_bounds__ (kThreads)
  start_kernel (Args<T> a, const T *src, double tol, int max_iter, double norm_b, int iter0, double eps,
                double cA, int new_shadow)
{
  DevState *st = a.st;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    {
      st->rho_prev = 1.0; // gpu/bicgstab.cu:414-420
      st->alpha = 1.0;
      st->omega = 1.0;
      st->rho = 0.0;
      st->beta = 0.0;
      st->tol = tol;
      st->max_iter = max_iter;
      st->done = 0;
      st->status = kStateRunning;
      st->eps = eps;
      st->cA = cA;
      st->c = src;
      st->rep_now = 0;
      st->replacements = 0;
      st->dev = st->dev_min = st->limit_prev = 0.0;
      if (ZERO)
        {
          st->iter = 0;
          st->norm_b = -1.0; // set by the first decision
        }
      else
        {
          if (norm_b > 0.0)
            st->norm_b = norm_b;
          if (iter0 >= 0)
            st->iter = iter0;
        }
    }
  double rr = 0.0, rhr = 0.0;
  GRID_STRIDE (i, a.n)
  {
    const T ri = src[i];
    const T hi = new_shadow ? (T) (ri * shadow_factor (i)) : ri;
    a.r[i] = ri;
    a.rh[i] = hi;
    a.p[i] = 0;
    a.v[i] = 0;
    a.g[i] = 0;
    a.xp[i] = 0;
    rr = fma ((double) ri, (double) ri, rr);
    rhr = fma ((double) hi, (double) ri, rhr);
  }
  double vals[3] = { rhr, rr, 0.0 };
  const int ks[3] = { kRhR, kRR, kGG };
  store_parts<3> (vals, a.part, a.grid, ks);
  if (!arrive_last (st, a.grid))
    return;
  double sv[3];
  sum_parts<3> (a.part, a.grid, ks, sv);
  decide (st, sv[0], sv[1], sv[2], true, 1.0);
}

// Preconditioner of the vector phases (right preconditioning, q = M^-1 p,
// z = M^-1 s): none, point Jacobi (gpu/bicgstab.cu:201-238), or block
// Jacobi (M^-1 = the inverses of the bs x bs diagonal blocks), the latter
// for bs = 2 with the block in registers and for any bs <= 8 (a block and
// its inverse fit a thread's registers and a small local frame; the FEM
// operators this serves have bs 2 or 3).
enum PreKind
{
  kPreNone = 0,
  kPrePoint = 1,
  kPreBlock2 = 2,
  kPreBlockAny = 3
};

constexpr int kMaxBlockJacobi = 8;

// One block row of a phase with block Jacobi: out = new values of the block
// (computed by f(k) for k < bs, stored to dst), then prec = Minv * out.
template <typename T, int PK, class F>
__device__ __forceinline__ void block_row_apply (const Args<T> &a, int64_t br, T *dst, T *prec, F f)
{
  const int bs = PK == kPreBlock2 ? 2 : a.bs;
  const int64_t base = br * bs;
  const T *M = a.P + (size_t) br * bs * bs;
  T u[PK == kPreBlock2 ? 2 : kMaxBlockJacobi];
  for (int k = 0; k < bs; k++)
    {
      u[k] = f (base + k);
      dst[base + k] = u[k];
    }
  for (int r = 0; r < bs; r++)
    {
      T acc = 0;
      for (int c = 0; c < bs; c++)
        acc = fma (M[r * bs + c], u[c], acc);
      prec[base + r] = acc;
    }
}

// phase 1: p = r + beta (p - omega v) (q = M^-1 p), with beta from the
// decision that closed the previous kernel; in a replacement iteration the
// fold g += x', x' = 0 and the partial (g, g) instead.
template <typename T, int PK> __device__ __forceinline__ void body_p (const Args<T> &a, const DevState *sc, bool rep)
{
  const int64_t stride = (int64_t) gridDim.x * blockDim.x;
  if (rep)
    {
      // Group update: fold the accumulated updates into the base, which
      // phase 2 multiplies by A for the true residual.
      double gg = 0.0;
      GRID_STRIDE (i, a.n)
      {
        const T gi = a.g[i] + a.xp[i];
        a.g[i] = gi;
        a.xp[i] = 0;
        gg = fma ((double) gi, (double) gi, gg);
      }
      double vals[1] = { gg };
      const int kg[1] = { kGG };
      store_parts<1> (vals, a.part, a.grid, kg);
      return;
    }
  const T tb = (T) sc->beta, tw = (T) sc->omega;
  if constexpr (PK >= kPreBlock2)
    {
      // block Jacobi: one block row per thread, q = Minv p of the block
      for (int64_t br = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; br < a.nbr; br += stride)
        block_row_apply<T, PK> (a, br, a.p, a.q,
                                [&] (int64_t i) { return a.r[i] + tb * (a.p[i] - tw * a.v[i]); });
      return;
    }
  const bool PRE = PK == kPrePoint;
  // Four grid-stride elements per pass, loads first (the arrays may alias as
  // far as the compiler knows, so it would not hoist them itself).
  int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < a.n; i += 4 * stride)
    {
      T rv[4], pv[4], vv[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          rv[u] = a.r[i + u * stride];
          pv[u] = a.p[i + u * stride];
          vv[u] = a.v[i + u * stride];
        }
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          const T pn = rv[u] + tb * (pv[u] - tw * vv[u]); // :286-304
          a.p[i + u * stride] = pn;
          if (PRE)
            a.q[i + u * stride] = a.P[i + u * stride] * pn; // :227-238
        }
    }
  for (; i < a.n; i += stride)
    {
      const T pn = a.r[i] + tb * (a.p[i] - tw * a.v[i]);
      a.p[i] = pn;
      if (PRE)
        a.q[i] = a.P[i] * pn;
    }
}

// phase 3
template <typename T, int PK> __device__ __forceinline__ void body_s (const Args<T> &a, const DevState *sc)
{
  const T ta = (T) sc->alpha;
  const int64_t stride = (int64_t) gridDim.x * blockDim.x;
  if constexpr (PK >= kPreBlock2)
    {
      for (int64_t br = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; br < a.nbr; br += stride)
        block_row_apply<T, PK> (a, br, a.s, a.z, [&] (int64_t i) { return a.r[i] - ta * a.v[i]; });
      return;
    }
  const bool PRE = PK == kPrePoint;
  int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < a.n; i += 4 * stride)
    {
      T rv[4], vv[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          rv[u] = a.r[i + u * stride];
          vv[u] = a.v[i + u * stride];
        }
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          const T si = rv[u] - ta * vv[u]; // :306-327
          a.s[i + u * stride] = si;
          if (PRE)
            a.z[i + u * stride] = a.P[i + u * stride] * si;
        }
    }
  for (; i < a.n; i += stride)
    {
      const T si = a.r[i] - ta * a.v[i];
      a.s[i] = si;
      if (PRE)
        a.z[i] = a.P[i] * si;
    }
}

// phase 5: x' += alpha q + omega z, r = s - omega t, partials (rh, r),
// (r, r), (x', x'); its last CTA takes the decision that opens the next
// iteration.
template <typename T, int PK> __device__ __forceinline__ void body_x (const Args<T> &a, const DevState *sc)
{
  const T ta = (T) sc->alpha, tw = (T) sc->omega;
  // (x', x') feeds the replacement bound only: skipped (0) when it is off.
  const bool track = sc->eps > 0.0;
  T rhr = 0, rr = 0, xx = 0;
  const T *qa = PK != kPreNone ? a.q : a.p;
  const T *za = PK != kPreNone ? a.z : a.s;
  const int64_t stride = (int64_t) gridDim.x * blockDim.x;
  int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < a.n; i += 4 * stride)
    {
      T xv[4], qv[4], zv[4], sv[4], tv[4], hv[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          const int64_t k = i + u * stride;
          xv[u] = a.xp[k];
          qv[u] = qa[k];
          zv[u] = za[k];
          sv[u] = a.s[k];
          tv[u] = a.t[k];
          hv[u] = a.rh[k];
        }
      // Same per-thread accumulation order as one element at a time.
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          const int64_t k = i + u * stride;
          const T xn = xv[u] + ta * qv[u] + tw * zv[u]; // h = x + alpha q; x = h + omega z
          a.xp[k] = xn;
          const T ri = sv[u] - tw * tv[u];              // :340-357
          a.r[k] = ri;
          rhr = fma (hv[u], ri, rhr);
          rr = fma (ri, ri, rr);
          if (track)
            xx = fma (xn, xn, xx);
        }
    }
  for (; i < a.n; i += stride)
    {
      const T xn = a.xp[i] + ta * qa[i] + tw * za[i];
      a.xp[i] = xn;
      const T ri = a.s[i] - tw * a.t[i];
      a.r[i] = ri;
      rhr = fma (a.rh[i], ri, rhr);
      rr = fma (ri, ri, rr);
      if (track)
        xx = fma (xn, xn, xx);
    }
  double vals[3] = { (double) rhr, (double) rr, (double) xx };
  const int kk[3] = { kRhR, kRR, kXX };
  store_parts<3> (vals, a.part, a.grid, kk);
}

template <typename T, int PK>
__global__ void __launch_bounds__ (kThreads) phase_p (Args<T> a)
{
  const int2 f = flags (a.st);
  if (f.x)
    return;
  body_p<T, PK> (a, a.st, f.y != 0);
}

template <typename T, int PK>
__global__ void __launch_bounds__ (kThreads) phase_s (Args<T> a)
{
  const int2 f = flags (a.st);
  if (f.x || f.y)
    return;
  body_s<T, PK> (a, a.st);
}

// phase 5 ends the iteration: its last CTA takes the decision that opens the
// next one (in a replacement iteration on phase 1 and 2's partials).
template <typename T, int PK>
__global__ void __launch_bounds__ (kThreads) phase_x (Args<T> a)
{
  DevState *st = a.st;
  const int2 f = flags (st);
  if (f.x)
    return;
  if (!f.y)
    body_x<T, PK> (a, st);
  if (!arrive_last (st, a.grid))
    return;
  tail_end (st, a.part, a.grid, f.y != 0);
}

// ------------------------------------------------------------ persistent iteration

// A grid barrier waits at most this long (the longest phase of the largest
// system this engine runs takes milliseconds); past it the CTA records a
// fault and leaves, and so does every CTA behind a later barrier.
constexpr unsigned long long kBarrierLimitNs = 4000000000ull;

// Scalar rows from which the auto launch mode runs the persistent kernel,
// and its CTAs per SM at most (launch bounds: up to 80 registers a thread).
constexpr int64_t kPersistentRows = 1000000;
constexpr int kIterateCtasPerSm = 3;

__device__ __forceinline__ unsigned long long global_ns ()
{
  unsigned long long t;
  asm volatile ("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier over the whole cooperative grid, after which every CTA sees every
// CTA's writes from before it. Thread 0 of each CTA counts the CTA in with an
// acq_rel add; the last one in runs `tail` (the phase's scalar work, with the
// whole CTA, on the device state) before it resets the count and advances
// the generation with a release; the others wait for that with a bounded
// acquire poll. gen is thread 0's copy of the generation. False when the wait
// gave up (the fault is recorded): the caller must return. (Two-level
// arrival through counters of 4 or 16 CTAs, and polls backing off to 32 or
// 256 ns, measured slower on GB300: 33-34 against 29 us per iteration at
// 20 000 rows.)
template <class Tail>
__device__ __forceinline__ bool grid_sync (DevState *st, int grid, unsigned &gen, Tail tail,
                                          unsigned long long limit_ns = kBarrierLimitNs)
{
  __shared__ int s_last, s_ok;
  __syncthreads ();
  cuda::atomic_ref<unsigned, cuda::thread_scope_device> arrive (st->arrive);
  cuda::atomic_ref<unsigned, cuda::thread_scope_device> g (st->gen);
  if (threadIdx.x == 0)
    {
      int ok = 1;
      const int last = arrive.fetch_add (1u, cuda::memory_order_acq_rel) == (unsigned) grid - 1;
      if (!last)
        {
          const unsigned long long t0 = global_ns ();
          unsigned polls = 0;
          while (g.load (cuda::memory_order_acquire) == gen)
            {
              if ((++polls & 255u) == 0 && global_ns () - t0 > limit_ns)
                {
                  ok = 0;
                  cuda::atomic_ref<int, cuda::thread_scope_device> fault (st->fault);
                  fault.store (1, cuda::memory_order_relaxed);
                  break;
                }
              __nanosleep (20);
            }
        }
      gen++;
      s_last = last;
      s_ok = ok;
    }
  __syncthreads ();
  if (s_last)
    {
      tail ();
      __syncthreads ();
      if (threadIdx.x == 0)
        {
          arrive.store (0u, cuda::memory_order_relaxed);
          g.store (gen, cuda::memory_order_release);
        }
    }
  return s_ok != 0;
}

// Up to `iters` BiCGStab iterations in one cooperative launch: the five phase
// bodies separated by grid barriers instead of kernel boundaries, the scalar
// work of a phase done by the last CTA to reach its barrier, on the device
// state, as the last CTA of the phase kernels does it (the same sums in the
// same order: the same bits). The x vector of each product was written by
// other CTAs of this kernel, so the products load it coherently (XCoh).
template <typename T, class Op, int PK>
__global__ void __launch_bounds__ (kThreads, kIterateCtasPerSm) iterate_kernel (Args<T> a, int iters)
{
  DevState *st = a.st;
  unsigned gen = 0;
  if (threadIdx.x == 0)
    gen = cuda::atomic_ref<unsigned, cuda::thread_scope_device> (st->gen).load (cuda::memory_order_relaxed);
  const double *part = a.part;
  const int grid = a.grid;
  auto none = [] () {};
  for (int it = 0; it < iters; it++)
    {
      const int2 f = flags (st);
      if (f.x)
        break;
      const bool rep = f.y != 0;
      body_p<T, PK> (a, st, rep);
      if (!grid_sync (st, grid, gen, none))
        return;
      body_v<T, Op> (a, st, rep);
      if (rep)
        {
          if (!grid_sync (st, grid, gen, [&] () { tail_end (st, part, grid, true); }))
            return;
          continue;
        }
      if (!grid_sync (st, grid, gen, [&] () { tail_v (st, part, grid); }))
        return;
      if (flags (st).x)
        break;
      body_s<T, PK> (a, st);
      if (!grid_sync (st, grid, gen, none))
        return;
      body_t<T, Op> (a);
      if (!grid_sync (st, grid, gen, [&] () { tail_t (st, part, grid); }))
        return;
      if (flags (st).x)
        break;
      body_x<T, PK> (a, st);
      if (!grid_sync (st, grid, gen, [&] () { tail_end (st, part, grid, false); }))
        return;
    }
}

#include "resident.cuh"

// The grid barrier's bounded wait, exercised: every CTA waits for one CTA
// more than the grid holds, so no CTA is ever last; each gives up after
// limit_ns, records the fault and returns, and the context stays usable.
__global__ void barrier_selftest_kernel (DevState *st, unsigned long long limit_ns)
{
  unsigned gen = 0;
  if (threadIdx.x == 0)
    gen = cuda::atomic_ref<unsigned, cuda::thread_scope_device> (st->gen).load (cuda::memory_order_relaxed);
  grid_sync (st, (int) gridDim.x + 1, gen, [] () {}, limit_ns);
}

// End of a run: x = e (a fresh solve) or x += e (a restart), with e the run's
// result g + x' or, when a snapshot is restored, the snapshot.
template <typename T>
__global__ void finish_kernel (int64_t n, T *x, const T *g, const T *xp, const T *snap, int add)
{
  GRID_STRIDE (i, n)
  {
    const T e = snap ? snap[i] : g[i] + xp[i];
    x[i] = add ? x[i] + e : e;
  }
}

// The run's current iterate g + x' into snap (the best-point copy).
template <typename T> __global__ void snapshot_kernel (int64_t n, const T *g, const T *xp, T *snap)
{
  GRID_STRIDE (i, n)
  snap[i] = g[i] + xp[i];
}

// cA = (entries per scalar row) * ||A||_inf, maxima over rows by atomics on
// the bit patterns (non-negative doubles order like their bits).
template <typename T>
__global__ void row_norm_kernel (int nbr, int bs, const int *rp, const T *vals, unsigned long long *max_abs,
                                 int *max_count)
{
  const int b = bs > 0 ? bs : 1;
  // Each thread keeps its own maxima, then the warp combines them: one
  // atomic per warp, not one per row on two addresses.
  unsigned long long amax = 0;
  int cmax = 0;
  GRID_STRIDE (i, (int64_t) nbr * b)
  {
    const int br = (int) (i / b), r = (int) (i % b);
    double sum = 0.0;
    int count = 0;
    for (int k = rp[br]; k < rp[br + 1]; k++)
      {
        if (bs > 0)
          for (int c = 0; c < bs; c++)
            sum += fabs ((double) vals[(size_t) k * bs * bs + (size_t) r * bs + c]);
        else
          sum += fabs ((double) vals[k]);
        count += b;
      }
    amax = max (amax, (unsigned long long) __double_as_longlong (sum));
    cmax = max (cmax, count);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    {
      amax = max (amax, __shfl_xor_sync (0xffffffffu, amax, off));
      cmax = max (cmax, __shfl_xor_sync (0xffffffffu, cmax, off));
    }
  if ((threadIdx.x & 31) == 0)
    {
      atomicMax (max_abs, amax);
      atomicMax (max_count, cmax);
    }
}

// Point Jacobi from the diagonal blocks: P = 1/a_rr (1 when |a_rr| < 1e-20
// or when the row stores no diagonal), gpu/bicgstab.cu:201-225.
template <typename T>
__global__ void jacobi_kernel (int nbr, int bs, const int *rp, const int *cols, const T *vals, T *P)
{
  GRID_STRIDE (i, (int64_t) nbr * bs)
  {
    const int br = (int) (i / bs), r = (int) (i % bs);
    T d = 1;
    for (int b = rp[br]; b < rp[br + 1]; b++)
      if (cols[b] == br)
        {
          const T a = vals[(size_t) b * bs * bs + r * bs + r];
          d = fabs ((double) a) < 1e-20 ? (T) 1 : (T) 1 / a;
          break;
        }
    P[i] = d;
  }
}

// Block Jacobi: Minv[br] = inverse of the diagonal block of block row br
// (Gauss-Jordan with partial pivoting in FP64, one thread per block row),
// the identity when the row stores no diagonal block or a pivot falls below
// 1e-20 times the block's largest entry: the block form of the point rule
// above (1 where |a_ii| < 1e-20 or no diagonal is stored).
template <typename T>
__global__ void block_jacobi_kernel (int nbr, int bs, const int *rp, const int *cols, const T *vals, T *Minv)
{
  GRID_STRIDE (br, (int64_t) nbr)
  {
    const int e = bs * bs;
    T *out = Minv + (size_t) br * e;
    const T *blk = nullptr;
    for (int b = rp[br]; b < rp[br + 1]; b++)
      if (cols[b] == (int) br)
        {
          blk = vals + (size_t) b * e;
          break;
        }
    double a[kMaxBlockJacobi * kMaxBlockJacobi], inv[kMaxBlockJacobi * kMaxBlockJacobi];
    double amax = 0.0;
    for (int k = 0; k < e; k++)
      {
        a[k] = blk ? (double) blk[k] : 0.0;
        inv[k] = (k / bs == k % bs) ? 1.0 : 0.0;
        amax = fmax (amax, fabs (a[k]));
      }
    bool ok = blk != nullptr && amax > 0.0;
    for (int c = 0; c < bs && ok; c++)
      {
        int piv = c;
        for (int r = c + 1; r < bs; r++)
          if (fabs (a[r * bs + c]) > fabs (a[piv * bs + c]))
            piv = r;
        if (!(fabs (a[piv * bs + c]) >= 1e-20 * amax))
          {
            ok = false;
            break;
          }
        if (piv != c)
          for (int k = 0; k < bs; k++)
            {
              double t = a[c * bs + k];
              a[c * bs + k] = a[piv * bs + k];
              a[piv * bs + k] = t;
              t = inv[c * bs + k];
              inv[c * bs + k] = inv[piv * bs + k];
              inv[piv * bs + k] = t;
            }
        const double d = 1.0 / a[c * bs + c];
        for (int k = 0; k < bs; k++)
          {
            a[c * bs + k] *= d;
            inv[c * bs + k] *= d;
          }
        for (int r = 0; r < bs; r++)
          if (r != c)
            {
              const double f = a[r * bs + c];
              if (f != 0.0)
                for (int k = 0; k < bs; k++)
                  {
                    a[r * bs + k] -= f * a[c * bs + k];
                    inv[r * bs + k] -= f * inv[c * bs + k];
                  }
            }
      }
    for (int k = 0; k < e; k++)
      out[k] = ok ? (T) inv[k] : (T) ((k / bs == k % bs) ? 1 : 0);
  }
}

// ------------------------------------------------------------ dispatch

enum SpmvKind
{
  kCsr8,
  kFlat2,
  kFlat4,
  kFlat8,
  kFlat16,
  kFlat32,
  kTpr3,
  kTprAny,
  kSell1, // CSR and bs = 2 on the engine's sliced copy
  kSell2
};

template <typename T, int K, class XL = dev::XNc> struct OpOf;
template <typename T, class XL> struct OpOf<T, kCsr8, XL> { using type = CsrOp<T, 8, XL>; };
// Few lanes per block row: every lane then holds whole block lines, so the
// warp-level FP64 instructions are not spent on predicated-off lanes or on
// shuffle-reduction adds (each FP64 warp instruction costs the same issue
// time on GB300's narrow FP64 pipe however many lanes are active).
template <typename T, class XL> struct OpOf<T, kFlat2, XL> { using type = FlatOp<T, 2, 2, XL>; };
template <typename T, class XL> struct OpOf<T, kSell1, XL> { using type = SellOp<T, 1, XL>; };
template <typename T, class XL> struct OpOf<T, kSell2, XL> { using type = SellOp<T, 2, XL>; };
template <typename T, class XL> struct OpOf<T, kFlat4, XL> { using type = FlatOp<T, 4, 4, XL>; };
template <typename T, class XL> struct OpOf<T, kFlat8, XL> { using type = FlatOp<T, 8, 4, XL>; };
template <typename T, class XL> struct OpOf<T, kFlat16, XL> { using type = FlatOp<T, 16, 8, XL>; };
template <typename T, class XL> struct OpOf<T, kFlat32, XL> { using type = FlatOp<T, 32, 16, XL>; };
template <typename T, class XL> struct OpOf<T, kTpr3, XL> { using type = TprOp<T, 3, XL>; };
template <typename T, class XL> struct OpOf<T, kTprAny, XL> { using type = TprOp<T, 0, XL>; };

int spmv_kind_for (const bmfp_matrix_s *A)
{
  switch (A->bs)
    {
    case 0:
    case 1: return kCsr8;
    case 2: return kFlat2;
    case 4: return kFlat4;
    case 8: return kFlat8;
    case 16: return kFlat16;
    case 32: return kFlat32;
    case 3: return kTpr3;
    default: return kTprAny;
    }
}

template <typename T, int K>
void launch_spmv_phase (int phase, const Args<T> &a, cudaStream_t s)
{
  using Op = typename OpOf<T, K>::type;
  if (phase == 2)
    phase_v<T, Op><<<a.grid, kThreads, 0, s>>> (a);
  else
    phase_t<T, Op><<<a.grid, kThreads, 0, s>>> (a);
}

template <typename T>
void launch_spmv_dispatch (int kind, int phase, const Args<T> &a, cudaStream_t s)
{
  switch (kind)
    {
    case kCsr8: launch_spmv_phase<T, kCsr8> (phase, a, s); break;
    case kFlat2: launch_spmv_phase<T, kFlat2> (phase, a, s); break;
    case kSell1: launch_spmv_phase<T, kSell1> (phase, a, s); break;
    case kSell2: launch_spmv_phase<T, kSell2> (phase, a, s); break;
    case kFlat4: launch_spmv_phase<T, kFlat4> (phase, a, s); break;
    case kFlat8: launch_spmv_phase<T, kFlat8> (phase, a, s); break;
    case kFlat16: launch_spmv_phase<T, kFlat16> (phase, a, s); break;
    case kFlat32: launch_spmv_phase<T, kFlat32> (phase, a, s); break;
    case kTpr3: launch_spmv_phase<T, kTpr3> (phase, a, s); break;
    default: launch_spmv_phase<T, kTprAny> (phase, a, s); break;
    }
}

template <typename T>
void launch_residual (int kind, const Args<T> &a, const T *x, const T *b, T *r, T *y, cudaStream_t s)
{
  switch (kind)
    {
#define BMFP_RES(K) case K: residual_kernel<T, typename OpOf<T, K>::type><<<a.grid, kThreads, 0, s>>> (a, x, b, r, y); break;
      BMFP_RES (kCsr8) BMFP_RES (kFlat2) BMFP_RES (kFlat4) BMFP_RES (kFlat8) BMFP_RES (kFlat16)
      BMFP_RES (kFlat32) BMFP_RES (kTpr3) BMFP_RES (kSell1) BMFP_RES (kSell2)
#undef BMFP_RES
    default: residual_kernel<T, typename OpOf<T, kTprAny>::type><<<a.grid, kThreads, 0, s>>> (a, x, b, r, y); break;
    }
}

template <typename T>
Args<T> make_args (const bmfp_matrix_s *A, int64_t n, void *x, void *r, void *rh, void *p, void *v,
                   void *q, void *s, void *z, void *t, void *P, void *g, void *xp, double *part, int grid,
                   DevState *st)
{
  Args<T> a;
  a.nbr = A->n_rows;
  a.bs = A->bs ? A->bs : 1;
  a.rp = A->d_row_ptr;
  a.cols = A->d_cols;
  a.vals = (const T *) A->d_vals;
  a.n = n;
  a.x = (T *) x;
  a.r = (T *) r;
  a.rh = (T *) rh;
  a.p = (T *) p;
  a.v = (T *) v;
  a.q = (T *) q;
  a.s = (T *) s;
  a.z = (T *) z;
  a.t = (T *) t;
  a.P = (const T *) P;
  a.g = (T *) g;
  a.xp = (T *) xp;
  a.part = part;
  a.grid = grid;
  a.st = st;
  a.soff = a.scols = nullptr;
  a.svals = nullptr;
  a.stream = false;
  a.nslices = 0;
  return a;
}

template <typename T, int PK>
void launch_vector_phase_k (int phase, const Args<T> &a, cudaStream_t s)
{
  if (phase == 1)
    phase_p<T, PK><<<a.grid, kThreads, 0, s>>> (a);
  else if (phase == 3)
    phase_s<T, PK><<<a.grid, kThreads, 0, s>>> (a);
  else
    phase_x<T, PK><<<a.grid, kThreads, 0, s>>> (a);
}

template <typename T> void launch_vector_phase (int pk, int phase, const Args<T> &a, cudaStream_t s)
{
  switch (pk)
    {
    case kPrePoint: launch_vector_phase_k<T, kPrePoint> (phase, a, s); break;
    case kPreBlock2: launch_vector_phase_k<T, kPreBlock2> (phase, a, s); break;
    case kPreBlockAny: launch_vector_phase_k<T, kPreBlockAny> (phase, a, s); break;
    default: launch_vector_phase_k<T, kPreNone> (phase, a, s); break;
    }
}

template <typename T, int K> const void *iterate_for_pre (int pk)
{
  using Op = typename OpOf<T, K, dev::XCoh>::type;
  if (pk == kPreNone)
    return reinterpret_cast<const void *> (&iterate_kernel<T, Op, kPreNone>);
  if (pk == kPrePoint)
    return reinterpret_cast<const void *> (&iterate_kernel<T, Op, kPrePoint>);
  return nullptr; // block Jacobi runs as graphs
}

// The persistent iteration kernel for a product kind and preconditioner, or
// null. Its grid must fit the device at once (3 CTAs of 256 threads per SM,
// 80 registers a thread): the products of bs 8, 16 and 32 need more
// registers than that, and with their long rows the launch gaps the kernel
// saves matter least; they run as graphs.
template <typename T> const void *iterate_for (int kind, int pk)
{
  switch (kind)
    {
    case kCsr8: return iterate_for_pre<T, kCsr8> (pk);
    case kFlat2: return iterate_for_pre<T, kFlat2> (pk);
    case kSell1: return iterate_for_pre<T, kSell1> (pk);
    case kSell2: return iterate_for_pre<T, kSell2> (pk);
    case kFlat4: return iterate_for_pre<T, kFlat4> (pk);
    case kTpr3: return iterate_for_pre<T, kTpr3> (pk);
    case kTprAny: return iterate_for_pre<T, kTprAny> (pk);
    default: return nullptr;
    }
}

template <typename T, int B, int PK> const void *resident_for (bool matrix)
{
  return matrix ? reinterpret_cast<const void *> (&resident_kernel<T, B, PK, true>)
                : reinterpret_cast<const void *> (&resident_kernel<T, B, PK, false>);
}

template <typename T> const void *resident_for (int kind, int pk, bool matrix)
{
  if (kind == kSell2)
    return pk == kPrePoint ? resident_for<T, 2, kPrePoint> (matrix) : resident_for<T, 2, kPreNone> (matrix);
  return pk == kPrePoint ? resident_for<T, 1, kPrePoint> (matrix) : resident_for<T, 1, kPreNone> (matrix);
}

// Unit roundoff of the engine's precision (replacement bound).
double unit_roundoff (int dtype) { return dtype == BMFP_R64F ? 0x1p-53 : 0x1p-24; }

// cA = max entries per scalar row * max absolute row sum of A (synchronises).
int matrix_bound (const bmfp_matrix_s *A, int grid, double *cA, cudaStream_t s)
{
  struct Maxima
  {
    unsigned long long abs_bits;
    int count;
  };
  Maxima *d = nullptr;
  BMFP_CUDA (cudaMallocAsync (&d, sizeof (Maxima), s));
  BMFP_CUDA (cudaMemsetAsync (d, 0, sizeof (Maxima), s));
  if (A->dtype == BMFP_R64F)
    row_norm_kernel<double><<<grid, kThreads, 0, s>>> (A->n_rows, A->bs, A->d_row_ptr, (const double *) A->d_vals,
                                                        &d->abs_bits, &d->count);
  else
    row_norm_kernel<float><<<grid, kThreads, 0, s>>> (A->n_rows, A->bs, A->d_row_ptr, (const float *) A->d_vals,
                                                       &d->abs_bits, &d->count);
  cudaError_t e = cudaGetLastError ();
  Maxima h{};
  if (e == cudaSuccess)
    e = cudaMemcpyAsync (&h, d, sizeof (Maxima), cudaMemcpyDeviceToHost, s);
  cudaFreeAsync (d, s);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize (s);
  if (e != cudaSuccess)
    return cuda_fail (e, "matrix_bound", __FILE__, __LINE__);
  double amax;
  const long long bits = (long long) h.abs_bits;
  std::memcpy (&amax, &bits, sizeof amax);
  *cA = (double) h.count * amax;
  return BMFP_SUCCESS;
}
} // namespace

// ------------------------------------------------------------ WideEngine

WideEngine::~WideEngine ()
{
  if (graph_)
    cudaGraphExecDestroy (graph_);
  if (capture_stream_)
    cudaStreamDestroy (capture_stream_);
  for (cudaEvent_t e : ev_)
    if (e)
      cudaEventDestroy (e);
  for (void *ptr : { x_, r_, rh_, p_, v_, q_, s_, z_, t_, P_, g_, xp_ })
    cudaFree (ptr);
  cudaFree (part_);
  cudaFree (state_);
  cudaFree (svals_);
  cudaFree (resident_mem_);
  cudaFree (resident_pub_);
  if (h_state_)
    cudaFreeHost (h_state_);
}

int WideEngine::init (const bmfp_matrix_s *A, int precond, int chunk, cudaStream_t stream, int ctas_per_sm,
                      int launch_mode, bool plain)
{
  if (!A)
    return fail (BMFP_ERROR_INVALID_VALUE, "null matrix");
  const int bs = A->bs ? A->bs : 1;
  if (precond == BMFP_PRECOND_BLOCK_JACOBI && bs > kMaxBlockJacobi)
    return fail (BMFP_ERROR_NOT_SUPPORTED, "block Jacobi takes bs <= %d (bs %d)", kMaxBlockJacobi, bs);
  if (A->bs && A->n_rows != A->n_cols)
    return fail (BMFP_ERROR_INVALID_VALUE, "BiCGStab needs a square matrix");
  if (!A->bs && A->n_rows != A->n_cols)
    return fail (BMFP_ERROR_INVALID_VALUE, "BiCGStab needs a square matrix");
  A_ = A;
  dtype_ = A->dtype;
  jacobi_ = precond != BMFP_PRECOND_NONE;
  const bool block = precond == BMFP_PRECOND_BLOCK_JACOBI;
  // 1x1 blocks multiply elementwise (P holds the blocks' inverses).
  pre_kind_ = !jacobi_ ? kPreNone : !block || bs == 1 ? kPrePoint : bs == 2 ? kPreBlock2 : kPreBlockAny;
  replace_ = dtype_ == BMFP_R64F;
  chunk_ = std::max (1, std::min (chunk, 256));
  n_ = (int64_t) A->n_rows * bs;
  spmv_kind_ = spmv_kind_for (A);
  if (!plain && (spmv_kind_ == kFlat2 || spmv_kind_ == kCsr8))
    {
      const int rc = build_sliced (stream);
      if (rc != BMFP_SUCCESS)
        return rc;
    }
  // Flat phases need 16-byte aligned values; cudaMalloc'd handles always are.
  int dev = 0, sms = 0;
  BMFP_CUDA (cudaGetDevice (&dev));
  BMFP_CUDA (cudaDeviceGetAttribute (&sms, cudaDevAttrMultiProcessorCount, dev));
  // Persistent iterations need a cooperative launch whose CTAs all fit on
  // the device at once: at most kIterateCtasPerSm CTAs per SM (the kernel's
  // launch bounds). Auto takes them from kPersistentRows up (measured on the
  // Q4 elasticity operator, FP64, us per iteration, graph at 4 CTAs per SM /
  // persistent at 3: 500 000 rows 79.3 / 79.9, 1.1 M rows 147.7 / 134.3,
  // 2 M rows 251.3 / 234.0; at 4 CTAs per SM and 64 registers the
  // persistent kernel spilled and took 84.2 / 142.2 / 234.0).
  iterate_ = nullptr;
  auto_ = launch_mode == BMFP_LAUNCH_AUTO;
  int cps = std::max (1, std::min (ctas_per_sm, 8));
  if (launch_mode == BMFP_LAUNCH_PERSISTENT || (launch_mode == BMFP_LAUNCH_AUTO && n_ >= kPersistentRows))
    {
      const void *fn = block                 ? nullptr
                       : dtype_ == BMFP_R64F ? iterate_for<double> (spmv_kind_, pre_kind_)
                                             : iterate_for<float> (spmv_kind_, pre_kind_);
      int coop = 0, per_sm = 0;
      BMFP_CUDA (cudaDeviceGetAttribute (&coop, cudaDevAttrCooperativeLaunch, dev));
      if (fn && coop)
        BMFP_CUDA (cudaOccupancyMaxActiveBlocksPerMultiprocessor (&per_sm, fn, kThreads, 0));
      if (fn && coop && per_sm >= 1)
        {
          iterate_ = fn;
          cps = std::min (cps, per_sm);
        }
      else if (launch_mode == BMFP_LAUNCH_PERSISTENT)
        return fail (BMFP_ERROR_NOT_SUPPORTED,
                     "persistent iterations need no preconditioner or point Jacobi, bs other than 8, 16 "
                     "and 32, and a device with cooperative launch");
    }
  // A few CTAs per SM, never more than the rows need.
  const int64_t want = std::max<int64_t> (1, (n_ + kThreads - 1) / kThreads);
  grid_ = (int) std::min<int64_t> ((int64_t) sms * cps, want);
  const size_t S = dtype_size (dtype_);
  const size_t vb = S * (size_t) std::max<int64_t> (n_, 1);
  for (void **ptr : { &x_, &r_, &rh_, &p_, &v_, &s_, &t_, &g_, &xp_ })
    BMFP_CUDA (cudaMalloc (ptr, vb));
  BMFP_CUDA (cudaMemsetAsync (x_, 0, vb, stream));
  if (jacobi_)
    {
      BMFP_CUDA (cudaMalloc (&q_, vb));
      BMFP_CUDA (cudaMalloc (&z_, vb));
      BMFP_CUDA (cudaMalloc (&P_, block ? vb * (size_t) bs : vb)); // block: bs x bs per block row
      if (block && dtype_ == BMFP_R64F)
        block_jacobi_kernel<double><<<grid_, kThreads, 0, stream>>> (A->n_rows, bs, A->d_row_ptr, A->d_cols,
                                                                      (const double *) A->d_vals, (double *) P_);
      else if (block)
        block_jacobi_kernel<float><<<grid_, kThreads, 0, stream>>> (A->n_rows, bs, A->d_row_ptr, A->d_cols,
                                                                     (const float *) A->d_vals, (float *) P_);
      else if (dtype_ == BMFP_R64F)
        jacobi_kernel<double><<<grid_, kThreads, 0, stream>>> (A->n_rows, bs, A->d_row_ptr, A->d_cols,
                                                                (const double *) A->d_vals, (double *) P_);
      else
        jacobi_kernel<float><<<grid_, kThreads, 0, stream>>> (A->n_rows, bs, A->d_row_ptr, A->d_cols,
                                                               (const float *) A->d_vals, (float *) P_);
      BMFP_LAUNCH_CHECK ();
    }
  else
    {
      q_ = nullptr;
      z_ = nullptr;
    }
  part_bytes_ = sizeof (double) * (size_t) kParts * grid_;
  BMFP_CUDA (cudaMalloc (&part_, part_bytes_));
  BMFP_CUDA (cudaMemsetAsync (part_, 0, part_bytes_, stream));
  BMFP_CUDA (cudaMalloc (&state_, sizeof (DevState)));
  BMFP_CUDA (cudaMemsetAsync (state_, 0, sizeof (DevState), stream));
  BMFP_CUDA (cudaMallocHost (&h_state_, 2 * sizeof (DevState)));
  BMFP_CUDA (cudaEventCreateWithFlags (&ev_[0], cudaEventDisableTiming));
  BMFP_CUDA (cudaEventCreateWithFlags (&ev_[1], cudaEventDisableTiming));
  BMFP_CUDA (cudaStreamCreateWithFlags (&capture_stream_, cudaStreamNonBlocking));
  int rc = matrix_bound (A, grid_, &cA_, stream); // synchronises the stream
  if (rc == BMFP_SUCCESS && launch_mode == BMFP_LAUNCH_AUTO && !iterate_ && svals_ && n_ < kPersistentRows
      && pre_kind_ <= kPrePoint)
    rc = plan_resident (dev, sms, stream);
  if (rc != BMFP_SUCCESS)
    return rc;
  return iterate_ ? BMFP_SUCCESS : capture (capture_stream_);
}

// Whether the sliced copy's loads leave L2 (129 MB) to the vectors. FP32 blocks: once
// the copy and the eight vectors of an iteration no longer fit together, whatever
// the row length. us per iteration as graphs, usual -> evicted first, by blocks a
// row and MB of copy + vectors: 3 blocks 70 + 75 118 -> 104; 5 blocks 70 + 45
// 81 -> 79, 84 + 54 100 -> 87; 7 blocks 70 + 32 62 -> 67, 84 + 38 80 -> 74; 8 blocks
// 70 + 28 58 -> 65, 84 + 34 76 -> 73, 96 + 38 86 -> 77; 9 blocks 70 + 25 57 -> 64,
// 84 + 30 70 -> 71, 96 + 34 82 -> 76, 140 + 50 110 -> 95; 13 blocks 84 + 21 65 -> 71,
// 96 + 24 77 -> 76, 110 + 27 92 -> 83.
// CSR, by the copy alone, as graphs / persistent: FP32 137 MB 67 / 71 -> 71 / 73, 173 MB
// 93 / 101 -> 82 / 87; FP64 108 MB 67 / 69 -> 68 / 73, 205 MB 117 / 119 -> 108 / 113, 432 MB
// 213 / 222 -> 202 / 213.
// FP64 blocks, bound by the FP64 pipe, do not care: 216 MB 130 / 134 -> 132 / 135.
bool streams (int dtype, int b, size_t bytes, int64_t n)
{
  if (b == 2)
    return dtype == BMFP_R32F && bytes + 8 * sizeof (float) * (size_t) n > (size_t) 115 << 20;
  return bytes > (size_t) 160 << 20;
}

// The sliced copy of a CSR or bs = 2 matrix: one more pass over it at creation and as
// many bytes again, kept where rows of one slice differ so little that the
// padding stays below an eighth (a structured grid's below 1 %) and it takes at
// most a quarter of the free memory; the products walk the block rows
// otherwise.
// Blocks of the copy at most, padding included.
size_t sliced_blocks (int64_t nnz) { return (size_t) (nnz + nnz / 8 + 1024); }

size_t sliced_bytes (const bmfp_matrix_s *A, const bmfp_solver_options &o)
{
  const size_t B = A->bs == 2 ? 2 : 1;
  if (A->bs > 2 || o.check_true_residual == 0)
    return 0;
  const size_t rows = (size_t) A->n_rows * B, entries = sliced_blocks (A->nnz);
  auto copy = [&] (size_t S) { return entries * (B * B * S + sizeof (int)) + sizeof (int) * (rows / kSlice + 2); };
  return (o.precision != BMFP_SOLVE_FP32 ? copy (8) : 0) + (o.precision != BMFP_SOLVE_FP64 ? copy (4) : 0);
}

int WideEngine::build_sliced (cudaStream_t s)
{
  const int nbr = A_->n_rows;
  if (nbr == 0 || A_->nnz == 0)
    return BMFP_SUCCESS;
  const int B = spmv_kind_ == kFlat2 ? 2 : 1, per = kSlice / B;
  const int ns = (nbr + per - 1) / per;
  const size_t S = dtype_size (dtype_);
  // Temporaries from the stream-ordered pool: a cudaFree here would wait for
  // every other stream of the device (the server's lanes create solvers while
  // others run).
  unsigned long long *tmp = nullptr, total = 0;
  BMFP_CUDA (cudaMallocAsync (&tmp, 8 + sizeof (int) * (2 * (size_t) ns + 1), s));
  int *width = (int *) (tmp + 1), *off = width + ns;
  sell_width_kernel<<<(ns + 255) / 256, 256, 0, s>>> (nbr, per, A_->d_row_ptr, ns, width);
  sell_scan_kernel<<<1, 1024, 0, s>>> (ns, width, off, tmp);
  cudaError_t e = cudaGetLastError ();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync (&total, tmp, 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize (s);
  const size_t blocks = (size_t) total * per;
  const size_t o_off = (B * B * S + sizeof (int)) * blocks;
  size_t mem_free = 0, mem_total = 0;
  if (e == cudaSuccess)
    e = cudaMemGetInfo (&mem_free, &mem_total);
  if (e == cudaSuccess && o_off < mem_free / 4 && blocks <= sliced_blocks (A_->nnz) && total <= INT32_MAX
      && cudaMalloc (&svals_, o_off + sizeof (int) * ((size_t) ns + 1)) == cudaSuccess)
    {
      scols_ = (int *) ((char *) svals_ + B * B * S * blocks);
      soff_ = (int *) ((char *) svals_ + o_off);
      e = cudaMemcpyAsync (soff_, off, sizeof (int) * ((size_t) ns + 1), cudaMemcpyDeviceToDevice, s);
      const int grid = std::min ((ns + 7) / 8, 152 * 8);
      auto fill = [&] (auto zero, auto width_c) {
        using T = decltype (zero);
        sell_fill_kernel<T, decltype (width_c)::value><<<grid, 256, 0, s>>> (
          nbr, A_->d_row_ptr, A_->d_cols, (const T *) A_->d_vals, ns, off, scols_, (T *) svals_);
      };
      using One = std::integral_constant<int, 1>;
      using Two = std::integral_constant<int, 2>;
      if (dtype_ == BMFP_R64F)
        B == 2 ? fill (0.0, Two ()) : fill (0.0, One ());
      else
        B == 2 ? fill (0.0f, Two ()) : fill (0.0f, One ());
      if (e == cudaSuccess)
        e = cudaGetLastError ();
    }
  else
    cudaGetLastError (); // no room: walk the block rows
  cudaFreeAsync (tmp, s);
  if (e != cudaSuccess)
    return cuda_fail (e, "sliced copy of the matrix", __FILE__, __LINE__);
  if (!svals_)
    return BMFP_SUCCESS;
  nslices_ = ns;
  stream_ = streams (dtype_, B, o_off, n_);
  spmv_kind_ = B == 2 ? kSell2 : kSell1;
  return BMFP_SUCCESS;
}

// The resident iteration kernel's plan, for the auto launch mode: a sliced
// matrix, no preconditioner or point Jacobi, fewer rows than the persistent
// kernel's, and vectors that fit the SMs' shared memory beside each other. Where
// its own allocations find no room the graphs run.
constexpr int kStagedRows = 1408;

int WideEngine::plan_resident (int dev, int sms, cudaStream_t s)
{
  const int B = spmv_kind_ == kSell2 ? 2 : 1;
  const int64_t S = (int64_t) dtype_size (dtype_);
  int coop = 0, most = 0;
  BMFP_CUDA (cudaDeviceGetAttribute (&coop, cudaDevAttrCooperativeLaunch, dev));
  BMFP_CUDA (cudaDeviceGetAttribute (&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  most -= 2048; // the kernel's own
  ResidentPlan P{};
  // At least four warps of rows: one per FP64 pipe of an SM.
  P.rows = (int) std::max<int64_t> (128, ((n_ + sms - 1) / sms + kSlice - 1) / kSlice * kSlice);
  P.grid = (int) ((n_ + P.rows - 1) / P.rows);
  const int64_t vectors = 7 * S * P.rows;
  if (!coop || vectors > most)
    return BMFP_SUCCESS;
  const size_t o_flags = sizeof (unsigned long long) * 2 * kSlotKinds * 2 * kCopies * (size_t) P.grid;
  const size_t o_need = (o_flags + sizeof (unsigned) * kFlagStride * (size_t) P.grid + 15) / 16 * 16;
  auto give_up = [&] () {
    cudaGetLastError ();
    cudaFree (resident_mem_);
    cudaFree (resident_pub_);
    resident_mem_ = resident_pub_ = nullptr;
    return BMFP_SUCCESS;
  };
  if (cudaMalloc (&resident_mem_, o_need + sizeof (int2) * ((size_t) P.grid + 1)) != cudaSuccess)
    return give_up ();
  resident_zero_ = o_need;
  BMFP_CUDA (cudaMemsetAsync (resident_mem_, 0, o_need + sizeof (int2) * ((size_t) P.grid + 1), s));
  P.slots = (unsigned long long *) resident_mem_;
  P.flags = (unsigned *) ((char *) resident_mem_ + o_flags);
  int2 *need = (int2 *) ((char *) resident_mem_ + o_need), steps{};
  P.need = need;
  resident_need_kernel<<<P.grid, 256, 0, s>>> (n_, P.rows, B, soff_, scols_, need);
  BMFP_LAUNCH_CHECK ();
  BMFP_CUDA (cudaMemcpyAsync (&steps, need + P.grid, sizeof steps, cudaMemcpyDeviceToHost, s));
  BMFP_CUDA (cudaStreamSynchronize (s));
  const int64_t vals = (int64_t) steps.x * kSlice * B * S, cols = (int64_t) steps.x * (kSlice / B) * 4;
  P.o_vals = (int) ((vectors + 15) / 16 * 16);
  // Staged, and with tagged words, wherever it fits, up to the rows per CTA that
  // were measured (us per iteration on the Q4 operator, staged against not:
  // FP64 132 rows a CTA 14.9 / 16.2, 527 23.1 / 24.4, 697 24.0 / 25.6, 890
  // 25.7 / 28.2, 1032 30.6 / 31.1; FP32 527 16.3 / 18.0, 890 17-19 / 20, 1185
  // 19-21 / 21.9, 1382 20.9 / 22). From there on the tags' traffic grows.
  P.matrix = P.rows <= kStagedRows && P.o_vals + vals + cols <= most;
  P.threads = std::min (P.rows, resident_threads ((int) S, P.matrix));
  P.o_cols = P.matrix ? (int) (P.o_vals + vals) : 0;
  P.smem = (int) (P.matrix ? P.o_vals + vals + cols : vectors);
  if (P.matrix)
    {
      // p and s as tagged words: a tag beside every four bytes
      const size_t vec = (size_t) S * 2 * (size_t) n_;
      resident_pub_bytes_ = 2 * vec;
      if (cudaMalloc (&resident_pub_, resident_pub_bytes_) != cudaSuccess)
        return give_up ();
      BMFP_CUDA (cudaMemsetAsync (resident_pub_, 0, resident_pub_bytes_, s));
      BMFP_CUDA (cudaStreamSynchronize (s)); // a solve on another stream would meet it
      P.pub[0] = (unsigned long long *) resident_pub_;
      P.pub[1] = (unsigned long long *) ((char *) resident_pub_ + vec);
    }
  const void *fn = dtype_ == BMFP_R64F ? resident_for<double> (spmv_kind_, pre_kind_, P.matrix)
                                       : resident_for<float> (spmv_kind_, pre_kind_, P.matrix);
  int per_sm = 0;
  BMFP_CUDA (cudaFuncSetAttribute (fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  BMFP_CUDA (cudaOccupancyMaxActiveBlocksPerMultiprocessor (&per_sm, fn, P.threads, (size_t) P.smem));
  if ((int64_t) per_sm * sms < P.grid)
    return give_up ();
  resident_ = P;
  iterate_ = fn;
  return BMFP_SUCCESS;
}

// Every kernel argument, q and z being p and s where there is no
// preconditioner.
template <typename T> struct WideEngine::ArgsOf
{
  static Args<T> make (const WideEngine &e, void *q, void *z)
  {
    Args<T> a = make_args<T> (e.A_, e.n_, e.x_, e.r_, e.rh_, e.p_, e.v_, q, e.s_, z, e.t_, e.P_, e.g_, e.xp_, e.part_,
                              e.grid_, e.state_);
    a.soff = e.soff_;
    a.scols = e.scols_;
    a.svals = (const T *) e.svals_;
    a.stream = e.stream_;
    a.nslices = e.nslices_;
    return a;
  }
};

int WideEngine::launch_iterations (cudaStream_t s)
{
  void *q = jacobi_ ? q_ : p_;
  void *z = jacobi_ ? z_ : s_;
  int iters = chunk_;
  cudaLaunchConfig_t cfg = {};
  const bool res = resident_.grid > 0;
  cfg.gridDim = dim3 ((unsigned) (res ? resident_.grid : grid_));
  cfg.blockDim = dim3 ((unsigned) (res ? resident_.threads : kThreads));
  cfg.dynamicSmemBytes = (size_t) resident_.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e;
  auto launch = [&] (auto a) {
    void *plain[] = { &a, &iters }, *planned[] = { &a, &resident_, &iters };
    return cudaLaunchKernelExC (&cfg, iterate_, res ? planned : plain);
  };
  if (dtype_ == BMFP_R64F)
    e = launch (ArgsOf<double>::make (*this, q, z));
  else
    e = launch (ArgsOf<float>::make (*this, q, z));
  if (e != cudaSuccess)
    return cuda_fail (e, "cooperative launch of the iteration kernel", __FILE__, __LINE__);
  return BMFP_SUCCESS;
}

int WideEngine::launch_phase (int phase, cudaStream_t s)
{
  void *q = jacobi_ ? q_ : p_;
  void *z = jacobi_ ? z_ : s_;
  if (dtype_ == BMFP_R64F)
    {
      Args<double> a
        = ArgsOf<double>::make (*this, q, z);
      if (phase == 2 || phase == 4)
        launch_spmv_dispatch<double> (spmv_kind_, phase, a, s);
      else
        launch_vector_phase<double> (pre_kind_, phase, a, s);
    }
  else
    {
      Args<float> a
        = ArgsOf<float>::make (*this, q, z);
      if (phase == 2 || phase == 4)
        launch_spmv_dispatch<float> (spmv_kind_, phase, a, s);
      else
        launch_vector_phase<float> (pre_kind_, phase, a, s);
    }
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

int WideEngine::capture (cudaStream_t s)
{
  cudaGraph_t g = nullptr;
  BMFP_CUDA (cudaStreamBeginCapture (s, cudaStreamCaptureModeThreadLocal));
  int st = BMFP_SUCCESS;
  for (int it = 0; it < chunk_ && st == BMFP_SUCCESS; it++)
    for (int ph = 1; ph <= 5 && st == BMFP_SUCCESS; ph++)
      st = launch_phase (ph, s);
  cudaError_t e = cudaStreamEndCapture (s, &g);
  if (st != BMFP_SUCCESS)
    {
      if (g)
        cudaGraphDestroy (g);
      return st;
    }
  if (e != cudaSuccess)
    return cuda_fail (e, "cudaStreamEndCapture", __FILE__, __LINE__);
  e = cudaGraphInstantiate (&graph_, g, 0);
  cudaGraphDestroy (g);
  if (e != cudaSuccess)
    return cuda_fail (e, "cudaGraphInstantiate", __FILE__, __LINE__);
  return BMFP_SUCCESS;
}

int WideEngine::start (bool zero, const void *c, double tol, int max_iter, double norm_b, int iter0, bool new_shadow,
                        cudaStream_t s)
{
  void *q = jacobi_ ? q_ : p_;
  void *z = jacobi_ ? z_ : s_;
  const double eps = replace_ ? unit_roundoff (dtype_) : 0.0;
  c_ = c;
  from_zero_ = zero;
  tol_ = tol;
  max_iter_ = max_iter;
  iter0_ = iter0;
  new_shadow_ = new_shadow;
  if (dtype_ == BMFP_R64F)
    {
      const Args<double> a
        = ArgsOf<double>::make (*this, q, z);
      if (zero)
        start_kernel<double, true><<<grid_, kThreads, 0, s>>> (a, (const double *) c, tol, max_iter, norm_b, iter0,
                                                                eps, cA_, new_shadow ? 1 : 0);
      else
        start_kernel<double, false><<<grid_, kThreads, 0, s>>> (a, (const double *) c, tol, max_iter, norm_b,
                                                                 iter0, eps, cA_, new_shadow ? 1 : 0);
    }
  else
    {
      const Args<float> a
        = ArgsOf<float>::make (*this, q, z);
      if (zero)
        start_kernel<float, true><<<grid_, kThreads, 0, s>>> (a, (const float *) c, tol, max_iter, norm_b, iter0,
                                                               eps, cA_, new_shadow ? 1 : 0);
      else
        start_kernel<float, false><<<grid_, kThreads, 0, s>>> (a, (const float *) c, tol, max_iter, norm_b, iter0,
                                                                eps, cA_, new_shadow ? 1 : 0);
    }
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

int WideEngine::start_zero (const void *d_b, double tol, int max_iter, cudaStream_t s)
{
  return start (true, d_b, tol, max_iter, -1.0, 0, false, s);
}

int WideEngine::start_residual (const void *d_r, double tol, int max_iter_total, double norm_b,
                                cudaStream_t s, int iter0, bool new_shadow)
{
  return start (false, d_r, tol, max_iter_total, norm_b, iter0, new_shadow, s);
}

namespace
{
// Stops a run from the host side: the phase kernels of the graphs still to
// come see done and return at once.
__global__ void stop_kernel (DevState *st)
{
  st->done = 1;
  st->status = kStateBreakdown;
}
} // namespace

// A wait of the persistent or resident kernel gave up: its words may hold a
// partial count, so the state (and the partials) are cleared (the next solve
// starts a new run) and the solve fails, unless the mode was the library's choice.
int WideEngine::barrier_fault (cudaStream_t s)
{
  BMFP_CUDA (cudaStreamSynchronize (s));
  BMFP_CUDA (cudaMemsetAsync (state_, 0, sizeof (DevState), s));
  BMFP_CUDA (cudaMemsetAsync (part_, 0, part_bytes_, s));
  if (resident_mem_)
    BMFP_CUDA (cudaMemsetAsync (resident_mem_, 0, resident_zero_, s));
  if (resident_pub_)
    BMFP_CUDA (cudaMemsetAsync (resident_pub_, 0, resident_pub_bytes_, s));
  BMFP_CUDA (cudaStreamSynchronize (s));
  return fail (BMFP_ERROR_TIMEOUT, "a grid barrier of the iteration kernel gave up waiting");
}

// After a wait that gave up under the auto mode: the graphs take this run again
// from its start (x is written at its end only), and all later ones. `last` is a
// state of the run, for what a restart keeps of the runs before it.
int WideEngine::run_again_as_graphs (const DevState &last, cudaStream_t s)
{
  iterate_ = nullptr;
  resident_ = ResidentPlan ();
  cudaFree (resident_mem_);
  cudaFree (resident_pub_);
  resident_mem_ = resident_pub_ = nullptr;
  const int rc = capture (capture_stream_);
  if (rc != BMFP_SUCCESS)
    return rc;
  if (from_zero_)
    return start (true, c_, tol_, max_iter_, -1.0, 0, new_shadow_, s);
  return start (false, c_, tol_, max_iter_, last.norm_b, iter0_ >= 0 ? iter0_ : last.iter, new_shadow_, s);
}

int WideEngine::run (cudaStream_t s, DevState *out, void *d_snap, double *snap_rr, int stall)
{
  // Keep one graph in flight while the host inspects the previous one.
  long k = 0;
  const long limit = 1 + (long) 1e9 / chunk_;
  double best = INFINITY;                              // smallest (r, r) polled
  const double snap_in = snap_rr ? *snap_rr : INFINITY;
  double snap_at = snap_in;                            // (r, r) of the last copy
  long snap_k = -1;                                    // graph whose end the copy holds
  double mark = INFINITY;                              // best (r, r) at the last halving
  int mark_it = 0;                                     // iteration of that halving
  bool stopping = false;
  for (;; k++)
    {
      if (iterate_)
        {
          const int rc = launch_iterations (s);
          if (rc != BMFP_SUCCESS)
            return rc;
        }
      else
        BMFP_CUDA (cudaGraphLaunch (graph_, s));
      BMFP_CUDA (cudaMemcpyAsync (&h_state_[k & 1], state_, sizeof (DevState), cudaMemcpyDeviceToHost, s));
      BMFP_CUDA (cudaEventRecord (ev_[k & 1], s));
      if (k > 0)
        {
          BMFP_CUDA (cudaEventSynchronize (ev_[(k - 1) & 1]));
          const DevState &h = h_state_[(k - 1) & 1];
          if (h.fault)
            {
              const DevState last = h;
              int rc = barrier_fault (s);
              if (rc == BMFP_ERROR_TIMEOUT && auto_)
                rc = run_again_as_graphs (last, s);
              if (rc != BMFP_SUCCESS)
                return rc;
              best = snap_at = mark = INFINITY; // no copy of the aborted run counts
              if (snap_rr)
                *snap_rr = INFINITY;
              snap_k = -1;
              mark_it = 0;
              stopping = false;
              k = -1;
              continue;
            }
          if (snap_k == k - 1)
            *snap_rr = snap_at = h.rr;
          if (h.done)
            break;
          if (h.rr < best)
            best = h.rr;
          // The iterate after graph k (queued behind it); its (r, r) is read
          // at the next poll.
          if (d_snap && snap_rr && h.rr < 0.25 * snap_at && snap_k != k - 1)
            {
              if (dtype_ == BMFP_R64F)
                snapshot_kernel<double><<<grid_, kThreads, 0, s>>> (n_, (const double *) g_, (const double *) xp_,
                                                                     (double *) d_snap);
              else
                snapshot_kernel<float><<<grid_, kThreads, 0, s>>> (n_, (const float *) g_, (const float *) xp_,
                                                                    (float *) d_snap);
              BMFP_LAUNCH_CHECK ();
              snap_k = k;
              snap_at = h.rr;
            }
          if (mark == INFINITY)
            mark = h.norm_b * h.norm_b;
          if (best <= 0.25 * mark)
            {
              mark = best;
              mark_it = h.iter;
            }
          const bool stalled = stall > 0 && h.iter - mark_it >= stall;
          if (!stopping && (!(h.rr <= 1e16 * best) || stalled))
            {
              stop_kernel<<<1, 1, 0, s>>> (state_);
              BMFP_LAUNCH_CHECK ();
              stopping = true;
            }
        }
      if (k > limit)
        return fail (BMFP_ERROR_TIMEOUT, "solver did not stop");
    }
  BMFP_CUDA (cudaStreamSynchronize (s));
  *out = h_state_[k & 1];
  if (out->fault)
    return barrier_fault (s);
  if (snap_k == k && snap_rr)
    *snap_rr = out->rr;
  // The run's result into x: the snapshot when the run ended above the best
  // point it passed (and that point is a copy of this run), else g + x'.
  const bool restore = d_snap && snap_rr && snap_k >= 0 && out->status != kStateConverged && *snap_rr < snap_in
                       && !(out->rr <= *snap_rr);
  if (restore)
    out->rr = *snap_rr;
  const int add = from_zero_ ? 0 : 1;
  if (dtype_ == BMFP_R64F)
    finish_kernel<double><<<grid_, kThreads, 0, s>>> (n_, (double *) x_, (const double *) g_, (const double *) xp_,
                                                       restore ? (const double *) d_snap : nullptr, add);
  else
    finish_kernel<float><<<grid_, kThreads, 0, s>>> (n_, (float *) x_, (const float *) g_, (const float *) xp_,
                                                      restore ? (const float *) d_snap : nullptr, add);
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

int WideEngine::true_residual (const void *d_b, void *d_r, double *rr, double *bb, cudaStream_t s)
{
  if (dtype_ == BMFP_R64F)
    {
      Args<double> a
        = ArgsOf<double>::make (*this, p_, s_);
      launch_residual<double> (spmv_kind_, a, (const double *) x_, (const double *) d_b, (double *) d_r,
                               (double *) t_, s);
    }
  else
    {
      Args<float> a
        = ArgsOf<float>::make (*this, p_, s_);
      launch_residual<float> (spmv_kind_, a, (const float *) x_, (const float *) d_b, (float *) d_r,
                              (float *) t_, s);
    }
  BMFP_LAUNCH_CHECK ();
  std::vector<double> h (2 * (size_t) grid_);
  BMFP_CUDA (cudaMemcpyAsync (h.data (), part_ + (size_t) kResRR * grid_, sizeof (double) * 2 * grid_,
                              cudaMemcpyDeviceToHost, s));
  BMFP_CUDA (cudaStreamSynchronize (s));
  double a = 0.0, b = 0.0;
  for (int i = 0; i < grid_; i++)
    {
      a += h[i];
      b += h[grid_ + i];
    }
  *rr = a;
  *bb = b;
  return BMFP_SUCCESS;
}
// ------------------------------------------------------------ raw buffers
// Launchers over caller-provided buffers, for the entry point that
// allocates nothing (noalloc.cu). They run the same phase kernels as
// WideEngine, without graphs, and without residual replacement (the
// reference's plain recurrences).

namespace
{
// One cooperative launch of a self-test kernel, a CTA per SM.
cudaError_t launch_selftest (const void *fn, void **args, int sms, cudaStream_t s)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3 ((unsigned) sms);
  cfg.blockDim = dim3 (kThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC (&cfg, fn, args);
}

int selftest_limits (double limit_s, int *sms)
{
  if (!(limit_s > 0.0 && limit_s <= 1.0))
    return fail (BMFP_ERROR_INVALID_VALUE, "the self-test waits between 0 and 1 s (got %g)", limit_s);
  int dev = 0, coop = 0;
  BMFP_CUDA (cudaGetDevice (&dev));
  BMFP_CUDA (cudaDeviceGetAttribute (sms, cudaDevAttrMultiProcessorCount, dev));
  BMFP_CUDA (cudaDeviceGetAttribute (&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop)
    return fail (BMFP_ERROR_NOT_SUPPORTED, "no cooperative launch on this device");
  return BMFP_SUCCESS;
}
} // namespace

int barrier_selftest (double limit_s, int *fault, double *elapsed_s, cudaStream_t s)
{
  int sms = 0;
  const int rc = selftest_limits (limit_s, &sms);
  if (rc != BMFP_SUCCESS)
    return rc;
  DevState *st = nullptr;
  BMFP_CUDA (cudaMalloc (&st, sizeof (DevState)));
  cudaEvent_t a = nullptr, b = nullptr;
  cudaError_t e = cudaMemsetAsync (st, 0, sizeof (DevState), s);
  if (e == cudaSuccess)
    e = cudaEventCreate (&a);
  if (e == cudaSuccess)
    e = cudaEventCreate (&b);
  if (e == cudaSuccess)
    e = cudaEventRecord (a, s);
  if (e == cudaSuccess)
    {
      unsigned long long limit_ns = (unsigned long long) (limit_s * 1e9);
      void *args[] = { &st, &limit_ns };
      e = launch_selftest ((const void *) barrier_selftest_kernel, args, sms, s);
    }
  DevState h{};
  if (e == cudaSuccess)
    e = cudaEventRecord (b, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync (&h, st, sizeof (DevState), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize (s);
  float ms = 0.0f;
  if (e == cudaSuccess)
    e = cudaEventElapsedTime (&ms, a, b);
  if (a)
    cudaEventDestroy (a);
  if (b)
    cudaEventDestroy (b);
  cudaFree (st);
  if (e != cudaSuccess)
    return cuda_fail (e, "barrier self-test", __FILE__, __LINE__);
  if (fault)
    *fault = h.fault;
  if (elapsed_s)
    *elapsed_s = ms * 1e-3;
  return BMFP_SUCCESS;
}

int resident_selftest (double limit_s, int *faults, cudaStream_t s)
{
  int sms = 0;
  const int rc = selftest_limits (limit_s, &sms);
  if (rc != BMFP_SUCCESS)
    return rc;
  const size_t words = sizeof (Word) * 2 * kSlotKinds * 2 * kCopies * (size_t) (sms + 1);
  const size_t flags = sizeof (unsigned) * kFlagStride * (size_t) (sms + 1);
  char *mem = nullptr;
  BMFP_CUDA (cudaMalloc (&mem, words + flags + sizeof (DevState)));
  DevState *st = (DevState *) (mem + words + flags);
  cudaError_t e = cudaSuccess;
  int bits = 0;
  for (int which = 0; which < 3 && e == cudaSuccess; which++)
    {
      e = cudaMemsetAsync (mem, 0, words + flags + sizeof (DevState), s);
      unsigned long long limit_ns = (unsigned long long) (limit_s * 1e9);
      Word *slots = (Word *) mem;
      unsigned *f = (unsigned *) (mem + words);
      void *args[] = { &st, &slots, &f, &which, &limit_ns };
      if (e == cudaSuccess)
        e = launch_selftest ((const void *) resident_selftest_kernel, args, sms, s);
      DevState h{};
      if (e == cudaSuccess)
        e = cudaMemcpyAsync (&h, st, sizeof (DevState), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess)
        e = cudaStreamSynchronize (s);
      // the first CTA's write-back counts only if it did come after the fault
      if (e == cudaSuccess && h.fault && (which != 2 || h.gen == 1))
        bits |= 1 << which;
    }
  cudaFree (mem);
  if (e != cudaSuccess)
    return cuda_fail (e, "self-test of the resident kernel's waits", __FILE__, __LINE__);
  if (faults)
    *faults = bits;
  return BMFP_SUCCESS;
}

int raw_solve_grid (int64_t n, int *grid)
{
  int dev = 0, sms = 0;
  BMFP_CUDA (cudaGetDevice (&dev));
  BMFP_CUDA (cudaDeviceGetAttribute (&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t want = std::max<int64_t> (1, (n + kThreads - 1) / kThreads);
  *grid = (int) std::min<int64_t> ((int64_t) sms * 4, want);
  return BMFP_SUCCESS;
}

namespace
{
int raw_kind (const RawSolve &b)
{
  const int kind = spmv_kind_for (&b.A);
  if (b.aligned)
    return kind;
  // The vectorised row routine needs 16-byte aligned values; fall back to
  // scalar loads for caller arrays that are not.
  return (kind == kCsr8 || kind == kTpr3) ? kind : kTprAny;
}

template <typename T> Args<T> raw_args (const RawSolve &b)
{
  void *q = b.jacobi ? b.q : b.p;
  void *z = b.jacobi ? b.z : b.s;
  return make_args<T> (&b.A, b.n, b.x, b.r, b.rh, b.p, b.v, q, b.s, z, b.t, b.P, b.g, b.xp, b.part, b.grid, b.st);
}
} // namespace

int raw_jacobi (const RawSolve &b, cudaStream_t s)
{
  const int bs = b.A.bs ? b.A.bs : 1;
  if (b.A.dtype == BMFP_R64F)
    jacobi_kernel<double><<<b.grid, kThreads, 0, s>>> (b.A.n_rows, bs, b.A.d_row_ptr, b.A.d_cols,
                                                       (const double *) b.A.d_vals, (double *) b.P);
  else
    jacobi_kernel<float><<<b.grid, kThreads, 0, s>>> (b.A.n_rows, bs, b.A.d_row_ptr, b.A.d_cols,
                                                      (const float *) b.A.d_vals, (float *) b.P);
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

int raw_start (const RawSolve &b, const void *d_rhs, double tol, int max_iter, cudaStream_t s)
{
  if (b.A.dtype == BMFP_R64F)
    start_kernel<double, true><<<b.grid, kThreads, 0, s>>> (raw_args<double> (b), (const double *) d_rhs,
                                                            tol, max_iter, -1.0, 0, 0.0, 0.0, 0);
  else
    start_kernel<float, true><<<b.grid, kThreads, 0, s>>> (raw_args<float> (b), (const float *) d_rhs,
                                                           tol, max_iter, -1.0, 0, 0.0, 0.0, 0);
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

int raw_phase (const RawSolve &b, int phase, cudaStream_t s)
{
  const int kind = raw_kind (b);
  if (b.A.dtype == BMFP_R64F)
    {
      const Args<double> a = raw_args<double> (b);
      if (phase == 2 || phase == 4)
        launch_spmv_dispatch<double> (kind, phase, a, s);
      else
        launch_vector_phase<double> (b.jacobi ? kPrePoint : kPreNone, phase, a, s);
    }
  else
    {
      const Args<float> a = raw_args<float> (b);
      if (phase == 2 || phase == 4)
        launch_spmv_dispatch<float> (kind, phase, a, s);
      else
        launch_vector_phase<float> (b.jacobi ? kPrePoint : kPreNone, phase, a, s);
    }
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

int raw_finish (const RawSolve &b, cudaStream_t s)
{
  if (b.A.dtype == BMFP_R64F)
    finish_kernel<double><<<b.grid, kThreads, 0, s>>> (b.n, (double *) b.x, (const double *) b.g,
                                                       (const double *) b.xp, nullptr, 0);
  else
    finish_kernel<float><<<b.grid, kThreads, 0, s>>> (b.n, (float *) b.x, (const float *) b.g, (const float *) b.xp,
                                                      nullptr, 0);
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}
} // namespace bmfp
