// The iteration kernel of systems whose Krylov vectors fit the SMs' shared
// memory (included by bicgstab.cu, whose Args, DevState helpers and sliced
// matrix it uses).
//
// One cooperative launch runs up to `iters` iterations. Each CTA owns a run of
// consecutive scalar rows and keeps r, rh, p, v, s, t and x' of them in shared
// memory (with room for it, its rows of the sliced matrix too), so that an
// iteration moves the matrix, p and s and nothing else. What one CTA needs
// from others goes round as self-validating 64-bit words, 32 data bits beside
// the number of the exchange: a word with the right number is the value, and
// neither a fence nor a flag stands behind it.
//
//  * p (or q) and s (or z): a row's owner writes its words, and the products
//    look again until every word they gather carries the number. A CTA waits
//    for the rows it reads and for nothing else. Where the matrix is too large
//    for shared memory, the gathers' traffic counts more than the wait: the
//    vector goes out as it is, each CTA releases a flag behind its rows, and
//    waits for the flags of the CTAs its columns belong to.
//  * the three sets of dot products: each CTA writes its partial sums, every
//    CTA reads all of them, a warp to a kind, and each derives the same scalars
//    from the same sums. Nothing is left to a last CTA, and no counter is
//    contended.
//
// What bounds it: small systems, the latency of five one-way trips through L2
// (about 0.6 us each), three divides and the dependent FP64 adds (64 cycles
// each); large ones, the FP64 pipe or L2. Successive sums' words alternate between
// two sets: a CTA can only write sum k + 2 when every CTA has written k + 1, that
// is, has read k. The same holds for p, s and g: the sum after a product tells
// everyone that its words have been read.
//
// us per iteration on the Q4 operator, as graphs and here: FP64 2 048 rows
// 18 / 13, 20 000 22 / 15, 80 000 28 / 23, 180 000 39 / 32, 500 000 66 / 57;
// FP32 2 048 rows 17 / 11, 20 000 20 / 13.5, 80 000 23 / 16.5, 180 000
// 31 / 20, 500 000 41 / 26.5. Whole solves (K + 0.01 I): 200x50 FP64
// 4.38 -> 2.73 ms, 1000x250 mixed 9.06 -> 5.07 ms. Of an iteration's 30 000
// cycles at 20 000 rows the three sums take 17 000, the products 6 600, the
// scalars 4 400.
#pragma once

// Threads per CTA at most: products from global memory live on the loads in
// flight, and in FP32 nine steps of them fit 64 registers.
constexpr int resident_threads (int bytes, bool staged) { return bytes == 4 && !staged ? 1024 : 512; }
constexpr int kSlotKinds = 3;
// A word that all CTAs look at again and again is slow for all of them: the
// looks queue at its line. So every CTA writes its sums in kCopies places, of
// which a reader looks at one, and a flag has a line to itself. us per
// iteration with one copy, 4, 8, 16 and 32: FP64 20 000 rows 19.5 / 17.4 / 16.5 /
// 16.2 / 16.0, FP32 80 000 rows 19.8 / 18.1 / 17.7 / 17.8 / 17.9; a line to a
// flag: FP32 500 000 rows 37.8 -> 30.8, FP64 65.8 -> 59.0.
constexpr int kCopies = 16;
constexpr int kFlagStride = 32; // 4-byte words

using Word = unsigned long long;

__device__ __forceinline__ Word tag_of (unsigned epoch) { return (Word) epoch << 32; }
__device__ __forceinline__ bool tagged (Word w, unsigned epoch) { return (unsigned) (w >> 32) == epoch; }
__device__ __forceinline__ void st_word (Word *p, Word a)
{
  asm volatile ("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}
__device__ __forceinline__ void st_words (Word *p, Word a, Word b)
{
  asm volatile ("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ Word ld_word (const Word *p)
{
  Word a;
  asm volatile ("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return a;
}
__device__ __forceinline__ void ld_words (const Word *p, Word &a, Word &b)
{
  asm volatile ("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

__device__ __forceinline__ void put_value (Word *p, double v, unsigned epoch)
{
  const Word b = (Word) __double_as_longlong (v);
  st_words (p, tag_of (epoch) | (b & 0xffffffffull), tag_of (epoch) | (b >> 32));
}
__device__ __forceinline__ void put_value (Word *p, float v, unsigned epoch)
{
  st_word (p, tag_of (epoch) | __float_as_uint (v));
}
__device__ __forceinline__ double value_of (Word lo, Word hi)
{
  return __hiloint2double ((int) (unsigned) hi, (int) (unsigned) lo);
}

// Words of one element of a published vector.
template <typename T> constexpr int kWords = (int) sizeof (T) / 4;

// Columns c of a published vector (c * B .. c * B + B - 1); false when a word
// does not carry the number yet.
template <int B> __device__ __forceinline__ bool get_vec (const Word *x, int c, unsigned epoch, double (&v)[B])
{
  bool ok = true;
#pragma unroll
  for (int j = 0; j < B; j++)
    {
      Word lo, hi;
      ld_words (x + ((size_t) c * B + j) * 2, lo, hi);
      ok = ok && tagged (lo, epoch) && tagged (hi, epoch);
      v[j] = value_of (lo, hi);
    }
  return ok;
}
__device__ __forceinline__ bool get_vec (const Word *x, int c, unsigned epoch, float (&v)[2])
{
  Word a, b;
  ld_words (x + (size_t) c * 2, a, b);
  v[0] = __uint_as_float ((unsigned) a);
  v[1] = __uint_as_float ((unsigned) b);
  return tagged (a, epoch) && tagged (b, epoch);
}
__device__ __forceinline__ bool get_vec (const Word *x, int c, unsigned epoch, float (&v)[1])
{
  const Word a = ld_word (x + c);
  v[0] = __uint_as_float ((unsigned) a);
  return tagged (a, epoch);
}

__device__ __forceinline__ void put_flag (unsigned *f, unsigned epoch)
{
  asm volatile ("st.release.gpu.global.u32 [%0], %1;" ::"l"(f), "r"(epoch) : "memory");
}
__device__ __forceinline__ bool get_flag (const unsigned *f, unsigned epoch)
{
  unsigned v;
  asm volatile ("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
  return (int) (v - epoch) >= 0;
}

// Looks until `ready`, for at most limit_ns; false when it gave up.
template <class F>
__device__ __forceinline__ bool wait_for (F ready, unsigned long long limit_ns = kBarrierLimitNs)
{
  if (ready ())
    return true;
  unsigned long long t0 = 0; // of the 256th look
  for (unsigned polls = 1; !ready (); polls++)
    if ((polls & 255u) == 0)
      {
        const unsigned long long now = global_ns ();
        if (t0 == 0)
          t0 = now;
        else if (now - t0 > limit_ns)
          return false;
      }
  return true;
}

// This CTA's part of a vector is stored (in place): releases its flag and
// waits for the parts its rows read. False when a wait gave up.
__device__ __forceinline__ bool publish (unsigned *flags, int2 need, unsigned epoch,
                                         unsigned long long limit_ns = kBarrierLimitNs)
{
  __syncthreads ();
  if (threadIdx.x == 0)
    put_flag (flags + blockIdx.x * kFlagStride, epoch);
  bool ok = true;
  for (int j = need.x + (int) threadIdx.x; j <= need.y; j += blockDim.x)
    ok = wait_for ([&] () { return get_flag (flags + j * kFlagStride, epoch); }, limit_ns) && ok;
  return __syncthreads_or (!ok) == 0;
}

// Sum NK per-thread values over the grid as exchange `epoch`, through set
// `turn` of the words (successive sums take the two sets in turn); warp k
// (k < NK <= 4 <= the CTA's warps) returns kind k's sum on every lane (other
// warps 0). False when a wait gave up.
template <int NK>
__device__ bool exchange_sum (Word *slots, int grid, unsigned epoch, int &turn, bool ok, double (&v)[NK], double &out,
                              unsigned long long limit_ns = kBarrierLimitNs)
{
  __shared__ double sh[NK][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double ws[NK];
  warp_sums<NK> (v, ws);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NK; k++)
      sh[k][w] = ws[k];
  __syncthreads ();
  // [copy][kind][CTA], so that a warp reads 512 consecutive bytes
  Word *set = slots + (size_t) turn * kSlotKinds * grid * 2 * kCopies;
  turn ^= 1;
  double sum = 0.0;
  if (w < NK)
    {
      const double a = warp_sum (lane < nw ? sh[w][lane] : 0.0);
      if (lane < kCopies)
        put_value (set + (((size_t) lane * kSlotKinds + w) * grid + blockIdx.x) * 2, a, epoch);
      const Word *mine = set + ((size_t) (blockIdx.x % kCopies) * kSlotKinds + w) * grid * 2;
      constexpr int M = 5; // loads in flight: 160 CTAs
      for (int j0 = 0; j0 < grid; j0 += 32 * M)
        {
          double got[M];
          bool have[M];
#pragma unroll
          for (int m = 0; m < M; m++)
            {
              got[m] = 0.0;
              have[m] = j0 + m * 32 + lane >= grid;
            }
          ok = wait_for ([&] () {
                 bool all = true;
#pragma unroll
                 for (int m = 0; m < M; m++)
                   if (!have[m])
                     {
                       Word lo, hi;
                       ld_words (mine + (size_t) (j0 + m * 32 + lane) * 2, lo, hi);
                       got[m] = value_of (lo, hi);
                       have[m] = tagged (lo, epoch) && tagged (hi, epoch);
                       all = all && have[m];
                     }
                 return all;
               }, limit_ns)
               && ok;
          __syncwarp ();
          const double part = warp_sum_of<M> (got);
          sum = j0 == 0 ? part : sum + part;
        }
    }
  out = sum;
  return __syncthreads_or (!ok) == 0;
}

// B consecutive values of the sliced matrix, staged (SM) or in global memory.
template <typename T, int B, bool SM> __device__ __forceinline__ void ld_values (const T *p, T (&v)[B])
{
  if constexpr (B == 1)
    v[0] = SM ? *p : __ldg (p);
  else if constexpr (sizeof (T) == 8)
    {
      const double2 *q = reinterpret_cast<const double2 *> (p);
      const double2 d = SM ? *q : __ldg (q);
      v[0] = d.x;
      v[1] = d.y;
    }
  else
    {
      const float2 *q = reinterpret_cast<const float2 *> (p);
      const float2 d = SM ? *q : __ldg (q);
      v[0] = d.x;
      v[1] = d.y;
    }
}

// Elements c * B .. of a vector published in place, from L2.
__device__ __forceinline__ void ld_vec (const double *x, int c, double (&v)[2])
{
  asm volatile ("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(x + (size_t) c * 2) : "memory");
}
__device__ __forceinline__ void ld_vec (const float *x, int c, float (&v)[2])
{
  asm volatile ("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(x + (size_t) c * 2) : "memory");
}
__device__ __forceinline__ void ld_vec (const double *x, int c, double (&v)[1])
{
  asm volatile ("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v[0]) : "l"(x + c) : "memory");
}
__device__ __forceinline__ void ld_vec (const float *x, int c, float (&v)[1])
{
  asm volatile ("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v[0]) : "l"(x + c) : "memory");
}

// The CTA's rows times a vector published in place: f (local row, sum) for
// every row, by the thread that owns it, nine steps (a whole row of a Q4 grid)
// in flight.
template <typename T, int B, class F>
__device__ __forceinline__ void global_product (const T *vals, const int *cols, const int *off, int slices, int rows,
                                                const T *x, F f)
{
  constexpr int U = 9;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int s = threadIdx.x >> 5; s < slices; s += nw)
    {
      const int beg = __ldg (off + s), n = __ldg (off + s + 1) - beg;
      const T *v = vals + ((size_t) beg * kSlice + lane) * B;
      const int *c = cols + (size_t) beg * (kSlice / B) + lane / B;
      T acc = 0;
      int k = 0;
      for (; k + U <= n; k += U)
        {
          T av[U][B], xv[U][B];
          int cc[U];
#pragma unroll
          for (int u = 0; u < U; u++)
            cc[u] = __ldg (c + (size_t) (k + u) * (kSlice / B));
#pragma unroll
          for (int u = 0; u < U; u++)
            ld_values<T, B, false> (v + (size_t) (k + u) * kSlice * B, av[u]);
#pragma unroll
          for (int u = 0; u < U; u++)
            ld_vec (x, cc[u], xv[u]);
#pragma unroll
          for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < B; j++)
              acc = fma (av[u][j], xv[u][j], acc);
        }
      for (; k < n; k++)
        {
          T av[B], xv[B];
          ld_vec (x, __ldg (c + (size_t) k * (kSlice / B)), xv);
          ld_values<T, B, false> (v + (size_t) k * kSlice * B, av);
#pragma unroll
          for (int j = 0; j < B; j++)
            acc = fma (av[j], xv[j], acc);
        }
      const int i = s * kSlice + lane;
      if (i < rows)
        f (i, acc);
    }
}

// The CTA's rows, staged in shared memory, times the vector published as
// exchange `epoch`: f (local row, sum) for every row, by the thread that owns
// it, nine steps (a whole row of a Q4 grid) in flight. False when a wait gave
// up.
template <typename T, int B, class F>
__device__ __forceinline__ bool staged_product (const T *vals, const int *cols, const int *off, int base, int slices,
                                                int rows, const Word *x, unsigned epoch, F f)
{
  constexpr int U = 9;
  bool ok = true;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int s = threadIdx.x >> 5; s < slices; s += nw)
    {
      const int beg = __ldg (off + s) - base, n = __ldg (off + s + 1) - base - beg;
      const T *v = vals + (beg * kSlice + lane) * B;
      const int *c = cols + beg * (kSlice / B) + lane / B;
      T acc = 0;
      int k = 0;
      for (; k + U <= n; k += U)
        {
          T xv[U][B];
          int cc[U];
#pragma unroll
          for (int u = 0; u < U; u++)
            cc[u] = c[(k + u) * (kSlice / B)];
          ok = wait_for ([&] () {
                 bool all = true;
#pragma unroll
                 for (int u = 0; u < U; u++)
                   all = get_vec (x, cc[u], epoch, xv[u]) && all;
                 return all;
               })
               && ok;
#pragma unroll
          for (int u = 0; u < U; u++)
            {
              T av[B];
              ld_values<T, B, true> (v + (k + u) * kSlice * B, av);
#pragma unroll
              for (int j = 0; j < B; j++)
                acc = fma (av[j], xv[u][j], acc);
            }
        }
      for (; k < n; k++)
        {
          T av[B], xv[B];
          const int cc = c[k * (kSlice / B)];
          ok = wait_for ([&] () { return get_vec (x, cc, epoch, xv); }) && ok;
          ld_values<T, B, true> (v + k * kSlice * B, av);
#pragma unroll
          for (int j = 0; j < B; j++)
            acc = fma (av[j], xv[j], acc);
        }
      const int i = s * kSlice + lane;
      if (i < rows)
        f (i, acc);
    }
  return ok;
}

// The decision at the end of an iteration from the three sums that warps 0 to
// 2 hold (each takes its sum's divide or square root, the fourth alpha /
// omega); every thread sees the new state on return.
__device__ __forceinline__ void resident_decide (DevState *S, double sum, bool rep)
{
  __shared__ double sh[6];
  const double rho_prev = rep ? S->rho_prev : S->rho;
  if (threadIdx.x == 0)
    {
      sh[0] = sum;
      sh[3] = sum / rho_prev;
    }
  else if (threadIdx.x == 32)
    {
      sh[1] = sum;
      sh[4] = sqrt (sum);
    }
  else if (threadIdx.x == 64)
    sh[5] = S->eps > 0.0 ? sqrt (sum) : 0.0;
  else if (threadIdx.x == 96)
    sh[2] = S->alpha / S->omega;
  __syncthreads ();
  if (threadIdx.x == 0)
    {
      if (!rep)
        {
          S->rho_prev = rho_prev;
          S->iter = S->iter + 1;
        }
      decide_scalars (S, sh[0], sh[1], sh[3], sh[2], sh[4], sh[5], rep);
    }
  __syncthreads ();
}

// A wait gave up. Only the host clears the word: a CTA that ends its launch
// well may do so after this one (store_state).
__device__ __forceinline__ void record_fault (DevState *st)
{
  cuda::atomic_ref<int, cuda::thread_scope_device> (st->fault).store (1, cuda::memory_order_relaxed);
}

// The state at the end of a launch, by one thread: all but the fault word.
__device__ __forceinline__ void store_state (DevState *st, const DevState &S)
{
  static_assert (offsetof (DevState, pad) == offsetof (DevState, fault) + 4
                   && sizeof (DevState) == offsetof (DevState, fault) + 8,
                 "nothing but padding behind the fault word");
  memcpy (__builtin_assume_aligned (st, 8), __builtin_assume_aligned (&S, 8), offsetof (DevState, fault));
}

template <typename T, int B, int PK, bool SM>
__global__ void __launch_bounds__ (resident_threads (sizeof (T), SM), 1) resident_kernel (Args<T> a, ResidentPlan P, int iters)
{
  extern __shared__ __align__ (16) unsigned char smem[];
  __shared__ DevState S;
  const int t = threadIdx.x, nt = blockDim.x;
  const int64_t row0 = (int64_t) blockIdx.x * P.rows;
  const int rows = (int) min ((int64_t) P.rows, a.n - row0);
  const int slices = (rows + kSlice - 1) / kSlice;
  const int slice0 = (int) (row0 / kSlice);
  if (t == 0)
    S = *a.st;
  __syncthreads ();
  if (S.done || S.fault)
    return; // every CTA reads the same words: they were written before this launch
  unsigned epoch = S.gen; // number of the last exchange
  int turn = 0;          // set of the next sum's words
  const int grid = P.grid;
  constexpr int W = kWords<T>;

  T *r = reinterpret_cast<T *> (smem), *rh = r + P.rows, *p = rh + P.rows, *v = p + P.rows, *s = v + P.rows,
    *tt = s + P.rows, *xp = tt + P.rows;
  for (int i = t; i < rows; i += nt)
    {
      r[i] = a.r[row0 + i];
      rh[i] = a.rh[row0 + i];
      p[i] = a.p[row0 + i];
      v[i] = a.v[row0 + i];
      xp[i] = a.xp[row0 + i];
    }
  const int *off = a.soff + slice0;
  int base = 0; // step that vals and cols start at
  const T *vals = a.svals;
  const int *cols = a.scols;
  if constexpr (SM)
    {
      base = __ldg (off);
      const int steps = __ldg (off + slices) - base;
      T *sv = reinterpret_cast<T *> (smem + P.o_vals);
      int *sc = reinterpret_cast<int *> (smem + P.o_cols);
      const int4 *gv = reinterpret_cast<const int4 *> (vals + (size_t) base * kSlice * B);
      const int4 *gc = reinterpret_cast<const int4 *> (cols + (size_t) base * (kSlice / B));
      for (int i = t; i < steps * (kSlice * B * (int) sizeof (T) / 16); i += nt)
        reinterpret_cast<int4 *> (sv)[i] = __ldg (gv + i);
      for (int i = t; i < steps * (kSlice / B * 4 / 16); i += nt)
        reinterpret_cast<int4 *> (sc)[i] = __ldg (gc + i);
      vals = sv;
      cols = sc;
    }
  // The vectors the products read, in place or as words.
  T *gq = PK == kPreNone ? a.p : a.q, *gz = PK == kPreNone ? a.s : a.z;
  Word *pq = P.pub[0], *pz = P.pub[1];
  const int2 need = P.need[blockIdx.x];
  bool ok = true;
  // Rows times the vector published last, f (local row, sum) for each.
  auto product = [&] (const T *x, const Word *words, auto f) {
    if constexpr (SM)
      ok = staged_product<T, B> (vals, cols, off, base, slices, rows, words, epoch, f);
    else if ((ok = publish (P.flags, need, epoch)))
      global_product<T, B> (vals, cols, off, slices, rows, x, f);
  };
  __syncthreads ();
  for (int it = 0; it < iters && !S.done; it++)
    {
      const bool rep = S.rep_now != 0;
      double gg = 0.0;
      ++epoch;
      if (rep)
        {
          for (int i = t; i < rows; i += nt)
            {
              const T gi = a.g[row0 + i] + xp[i];
              a.g[row0 + i] = gi;
              if (SM)
                put_value (pq + (row0 + i) * W, gi, epoch);
              xp[i] = 0;
              gg = fma ((double) gi, (double) gi, gg);
            }
        }
      else
        {
          const T tb = (T) S.beta, tw = (T) S.omega;
          for (int i = t; i < rows; i += nt)
            {
              const T pn = r[i] + tb * (p[i] - tw * v[i]);
              p[i] = pn;
              const T qi = PK == kPreNone ? pn : a.P[row0 + i] * pn;
              if (PK != kPreNone || !SM)
                gq[row0 + i] = qi;
              if (SM)
                put_value (pq + (row0 + i) * W, qi, epoch);
            }
        }
      double sum = 0.0;
      if (rep)
        {
          const T *c = static_cast<const T *> (S.c);
          T rhr = 0, rr = 0;
          product (a.g, pq, [&] (int i, T y) {
            const T ri = c[row0 + i] - y;
            r[i] = ri;
            rhr = fma (rh[i], ri, rhr);
            rr = fma (ri, ri, rr);
          });
          double in[3] = { (double) rhr, (double) rr, gg };
          ++epoch;
          if (!(ok = exchange_sum<3> (P.slots, grid, epoch, turn, ok, in, sum)))
            break;
          resident_decide (&S, sum, true);
          continue;
        }
      T dot = 0;
      product (gq, pq, [&] (int i, T y) {
        v[i] = y;
        dot = fma (rh[i], y, dot);
      });
      double d1[1] = { (double) dot };
      ++epoch;
      if (!(ok = exchange_sum<1> (P.slots, grid, epoch, turn, ok, d1, sum)))
        break;
      if (t == 0)
        {
          const double alpha = S.rho / sum; // gpu/bicgstab.cu:466
          if (!is_zero (sum) && is_finite (alpha))
            S.alpha = alpha;
          else
            {
              S.status = kStateBreakdown;
              S.done = 1;
            }
        }
      __syncthreads ();
      if (S.done)
        break;
      const T ta = (T) S.alpha;
      ++epoch;
      for (int i = t; i < rows; i += nt)
        {
          const T si = r[i] - ta * v[i];
          s[i] = si;
          const T zi = PK == kPreNone ? si : a.P[row0 + i] * si;
          if (PK != kPreNone || !SM)
            gz[row0 + i] = zi;
          if (SM)
            put_value (pz + (row0 + i) * W, zi, epoch);
        }
      T ts = 0, t2 = 0;
      product (gz, pz, [&] (int i, T y) {
        tt[i] = y;
        ts = fma (s[i], y, ts);
        t2 = fma (y, y, t2);
      });
      double d2[2] = { (double) ts, (double) t2 };
      ++epoch;
      if (!(ok = exchange_sum<2> (P.slots, grid, epoch, turn, ok, d2, sum)))
        break;
      __shared__ double sh2[2];
      if (t == 0 || t == 32)
        sh2[t >> 5] = sum;
      __syncthreads ();
      if (t == 0)
        {
          const double omega = is_zero (sh2[1]) ? 0.0 : sh2[0] / sh2[1]; // :488
          if (is_finite (omega))
            S.omega = omega;
          else
            {
              S.status = kStateBreakdown;
              S.done = 1;
            }
        }
      __syncthreads ();
      if (S.done)
        break;
      const T tw = (T) S.omega;
      const bool track = S.eps > 0.0;
      T rhr = 0, rr = 0, xx = 0;
      for (int i = t; i < rows; i += nt)
        {
          const T qi = PK == kPreNone ? p[i] : gq[row0 + i], zi = PK == kPreNone ? s[i] : gz[row0 + i];
          const T xn = xp[i] + ta * qi + tw * zi;
          xp[i] = xn;
          const T ri = s[i] - tw * tt[i]; // :340-357
          r[i] = ri;
          rhr = fma (rh[i], ri, rhr);
          rr = fma (ri, ri, rr);
          if (track)
            xx = fma (xn, xn, xx);
        }
      double d3[3] = { (double) rhr, (double) rr, (double) xx };
      ++epoch;
      if (!(ok = exchange_sum<3> (P.slots, grid, epoch, turn, ok, d3, sum)))
        break;
      resident_decide (&S, sum, false);
    }
  if (!ok)
    {
      if (t == 0)
        record_fault (a.st);
      return;
    }
  __syncthreads ();
  for (int i = t; i < rows; i += nt)
    {
      a.r[row0 + i] = r[i];
      a.p[row0 + i] = p[i];
      a.v[row0 + i] = v[i];
      a.xp[row0 + i] = xp[i];
    }
  if (blockIdx.x == 0 && t == 0)
    {
      S.gen = epoch;
      S.arrive = 0;
      store_state (a.st, S);
    }
}

// First and last CTA that each CTA's columns belong to; need[grid].x: the most
// steps of any CTA's rows.
__global__ void resident_need_kernel (int64_t n, int rows, int b, const int *soff, const int *scols, int2 *need)
{
  __shared__ int lo, hi;
  if (threadIdx.x == 0)
    {
      lo = INT_MAX;
      hi = 0;
    }
  __syncthreads ();
  const int64_t row0 = (int64_t) blockIdx.x * rows, row1 = min (n, row0 + rows);
  const int s0 = soff[row0 / kSlice], s1 = soff[(row1 + kSlice - 1) / kSlice];
  const int64_t e1 = (int64_t) s1 * (kSlice / b);
  int mn = INT_MAX, mx = 0;
  for (int64_t e = (int64_t) s0 * (kSlice / b) + threadIdx.x; e < e1; e += blockDim.x)
    {
      mn = min (mn, scols[e]);
      mx = max (mx, scols[e]);
    }
  atomicMin (&lo, mn);
  atomicMax (&hi, mx);
  __syncthreads ();
  if (threadIdx.x == 0)
    {
      const int self = blockIdx.x;
      need[self].x = lo == INT_MAX ? self : (int) ((int64_t) lo * b / rows);
      need[self].y = lo == INT_MAX ? self : (int) (((int64_t) hi * b + b - 1) / rows);
      atomicMax (&need[gridDim.x].x, s1 - s0);
    }
}

// The waits above run out on purpose, which = 0: a sum over one CTA more than
// the grid holds; 1: a flag that nothing releases; 2: the same in all CTAs but
// the first, which ends its launch after one of them has recorded its fault.
__global__ void resident_selftest_kernel (DevState *st, Word *slots, unsigned *flags, int which,
                                          unsigned long long limit_ns)
{
  __shared__ DevState S;
  const int grid = (int) gridDim.x;
  if (threadIdx.x == 0)
    S = *st;
  __syncthreads ();
  bool ok;
  if (which == 0)
    {
      int turn = 0;
      double in[3] = { 1.0, 1.0, 1.0 }, sum;
      ok = exchange_sum<3> (slots, grid + 1, 1, turn, true, in, sum, limit_ns);
    }
  else if (which == 1 || blockIdx.x > 0)
    ok = publish (flags, make_int2 (0, grid), 1, limit_ns);
  else
    {
      if (threadIdx.x == 0)
        {
          cuda::atomic_ref<int, cuda::thread_scope_device> fault (st->fault);
          wait_for ([&] () { return fault.load (cuda::memory_order_relaxed) != 0; }, 4 * limit_ns);
          S.gen = 1;
          store_state (st, S);
        }
      return;
    }
  if (!ok && threadIdx.x == 0)
    record_fault (st);
}
