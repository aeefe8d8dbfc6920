// Row-tile sparse products: y = A x for BCSR at block sizes from 3 to 32 that are no
// power of two.
//
// A CTA owns a tile of consecutive block rows, whose values and block columns
// are two contiguous runs. It copies them into shared memory with 16-byte
// cp.async (every byte of the run once, whatever the block size or the row
// lengths) and then cuts the tile's blocks into chunks of K, one chunk to bs
// threads (thread r of them takes scalar row r of each block): every lane has
// the same number of multiply-adds however uneven the rows are, and none idles
// because 32 is not a multiple of the block size. A chunk leaves one partial
// sum per block row it meets; the sum of a row's partials, in chunk order, is
// its result.
//
// It serves the block sizes for which a warp per block row (bcsr_tpr_kernel)
// leaves most of the memory system idle. What bounds it: FP64, the FP64 pipe
// (50-70 % busy) and the latency of x; FP32, the latency of the two round trips
// a tile makes (values and columns, then x). us, before (warp per block row)
// and now: rows of 0-15 blocks, 150 000 block rows, bs 3 FP64 77.7 -> 35.2,
// FP32 26.2 -> 21.1; 50 000 block rows of 6 blocks, bs 12 FP32 40.4 -> 34.5,
// FP64 102 -> 97, bs 17 FP64 279 -> 202, FP32 96 -> 69, bs 24 FP64 558 -> 411.
#include "device_common.cuh"
#include "internal.h"

#include <algorithm>

namespace bmfp
{
namespace
{
constexpr int kThreads = 128;
constexpr int kMaxRows = 1024; // block rows per CTA at most

template <typename T, int V> struct Pack
{
  T v[V];
};

template <typename T, int V> __device__ __forceinline__ Pack<T, V> ld_x (const T *p)
{
  Pack<T, V> r;
  if constexpr (V * sizeof (T) == 16)
    {
      const auto t = dev::ld_cached16 (p);
#pragma unroll
      for (int i = 0; i < V; i++)
        r.v[i] = t.v[i];
    }
  else if constexpr (V == 2)
    dev::ld_cached2 (p, r.v[0], r.v[1]);
  else
    r.v[0] = __ldg (p);
  return r;
}

template <typename T, int V> __device__ __forceinline__ Pack<T, V> ld_s (const T *p)
{
  Pack<T, V> r;
  if constexpr (V * sizeof (T) == 16 && sizeof (T) == 4)
    {
      const float4 t = *reinterpret_cast<const float4 *> (p);
      r.v[0] = t.x, r.v[1] = t.y, r.v[2] = t.z, r.v[3] = t.w;
    }
  else if constexpr (V * sizeof (T) == 16)
    {
      const double2 t = *reinterpret_cast<const double2 *> (p);
      r.v[0] = t.x, r.v[1] = t.y;
    }
  else if constexpr (V == 2)
    {
      const float2 t = *reinterpret_cast<const float2 *> (p);
      r.v[0] = t.x, r.v[1] = t.y;
    }
  else
    r.v[0] = *p;
  return r;
}

// With PAD, staged values sit 16 bytes further on after every 128 (block lines
// of a multiple of 64 bytes would otherwise meet in the same banks).
template <typename T, bool PAD> __device__ __forceinline__ int at (int e)
{
  constexpr int L = 128 / (int) sizeof (T), P = 16 / (int) sizeof (T);
  return PAD ? e + e / L * P : e;
}

struct TilePlan
{
  int rows;  // block rows per CTA
  int chunk; // blocks per chunk
  int cap;   // blocks staged at once (a whole number of chunks)
  // shared memory: staged values, then from these byte offsets the block
  // columns, the partial sums, the sums of rows cut by a piece's end, the row
  // offsets and the chunks' first rows
  int o_cols, o_part, o_sum, o_rp, o_first, smem;
};

// Blocks whose x segments a thread has in flight at once.
constexpr int blocks_in_flight (int bs, int bytes)
{
  return bs <= 3 ? 3 : bs <= 6 ? 2 : bs <= 12 && bytes == 4 ? 2 : 1;
}

// One pass over nr rows from r0 on, n blocks from block B0 on, by the whole CTA.
template <typename T, int BSC, int V, bool PAD>
__device__ __forceinline__ void tile_pass (int nbr, int bs_rt, const TilePlan &P, const int *__restrict__ row_ptr,
                                           const int *__restrict__ cols, const T *__restrict__ vals,
                                           const T *__restrict__ x, T *__restrict__ y, int r0, int nr, int B0, int n)
{
  extern __shared__ __align__ (16) unsigned char smem[];
  constexpr int VS = 16 / (int) sizeof (T);
  const int bs = BSC ? BSC : bs_rt;
  const int E = bs * bs;
  const int t = threadIdx.x;
  const int64_t total_cols = __ldg (row_ptr + nbr), total_vals = total_cols * E;
  T *sv = reinterpret_cast<T *> (smem);
  int *sc = reinterpret_cast<int *> (smem + P.o_cols);
  T *part = reinterpret_cast<T *> (smem + P.o_part);
  T *sum = reinterpret_cast<T *> (smem + P.o_sum);
  int *rp = reinterpret_cast<int *> (smem + P.o_rp); // relative to B0
  int *first = reinterpret_cast<int *> (smem + P.o_first);
  const uint32_t sv_a = (uint32_t) __cvta_generic_to_shared (sv), sc_a = (uint32_t) __cvta_generic_to_shared (sc);
  const int K = P.chunk;
  const int slot = t / bs, r = t - slot * bs;
  const int slots = kThreads / bs;

  for (int p0 = 0; p0 == 0 || p0 < n; p0 += P.cap)
    {
      const int nb = min (n - p0, P.cap); // blocks of this piece
      if (nb > 0)
        {
          const int64_t b0 = (int64_t) B0 + p0;
          const int64_t e0 = b0 * E, ea = e0 & ~(int64_t) (VS - 1);
          const int nv = (int) ((e0 + (int64_t) nb * E - ea + VS - 1) / VS);
          for (int j = t; j < nv; j += kThreads)
            {
              const int64_t e = ea + (int64_t) j * VS;
              const int left = (int) min ((int64_t) VS, total_vals - e);
              dev::cp_async16 (sv_a + (PAD ? j + j / 8 : j) * 16, vals + e, left * (int) sizeof (T));
            }
          const int64_t ca = b0 & ~(int64_t) 3;
          const int nc = (int) ((b0 + nb - ca + 3) / 4);
          for (int j = t; j < nc; j += kThreads)
            {
              const int64_t e = ca + j * 4;
              dev::cp_async16 (sc_a + j * 16, cols + e, (int) min ((int64_t) 4, total_cols - e) * 4);
            }
        }
      if (p0 == 0)
        {
          for (int i = t; i <= nr; i += kThreads)
            rp[i] = __ldg (row_ptr + r0 + i) - B0;
          __syncthreads ();
        }
      // which block row each chunk of the piece starts in
      for (int i = t; i < nr; i += kThreads)
        {
          const int lo = max (rp[i], p0) - p0, hi = min (rp[i + 1] - p0, nb);
          if (lo < hi)
            for (int q = (lo + K - 1) / K; q * K < hi; q++)
              first[q] = i;
        }
      dev::cp_async_commit ();
      dev::cp_async_wait<0> ();
      __syncthreads ();
      const int off = (int) ((((int64_t) B0 + p0) * E) & (VS - 1));
      const int *scb = sc + ((B0 + p0) & 3);
      if (slot < slots)
        for (int q = slot; q * K < nb; q += slots)
          {
            int b = q * K;
            const int be = min (b + K, nb);
            int row = first[q];
            int row_end = rp[row + 1] - p0;
            T acc = 0;
            // block b is done: leave the partial sum where its row or the
            // chunk ends
            auto done = [&] () {
              b++;
              if (b == row_end || b == be)
                {
                  part[(q + row) * bs + r] = acc;
                  acc = 0;
                  if (b < be)
                    do
                      {
                        row++;
                        row_end = rp[row + 1] - p0;
                      }
                    while (row_end == b);
                }
            };
            if constexpr (BSC != 0)
              {
                constexpr int UB = blocks_in_flight (BSC, sizeof (T));
                while (b < be)
                  {
                    Pack<T, V> xv[UB][BSC / V];
                    const int left = be - b;
#pragma unroll
                    for (int u = 0; u < UB; u++)
                      if (u == 0 || u < left)
                        {
                          const T *xb = x + (size_t) scb[b + u] * BSC;
#pragma unroll
                          for (int c = 0; c < BSC / V; c++)
                            xv[u][c] = ld_x<T, V> (xb + c * V);
                        }
                    // the lines of two long-lined blocks before the first
                    // flush: the branches in done () would keep them apart
                    constexpr bool kAhead = UB > 1 && BSC > 6;
                    Pack<T, V> av[UB][BSC / V];
                    auto lines = [&] (int u, int at_block) {
                      const int line = off + at_block * E + r * BSC;
#pragma unroll
                      for (int c = 0; c < BSC / V; c++)
                        av[u][c] = ld_s<T, V> (sv + at<T, PAD> (line + c * V));
                    };
                    if (kAhead)
#pragma unroll
                      for (int u = 0; u < UB; u++)
                        lines (u, b + min (u, left - 1));
#pragma unroll
                    for (int u = 0; u < UB; u++)
                      if (u == 0 || u < left)
                        {
                          if (!kAhead)
                            lines (u, b);
#pragma unroll
                          for (int c = 0; c < BSC / V; c++)
#pragma unroll
                            for (int k = 0; k < V; k++)
                              acc = fma (av[u][c].v[k], xv[u][c].v[k], acc);
                          done ();
                        }
                  }
              }
            else
              {
                constexpr int UC = 8;
                while (b < be)
                  {
                    const T *xb = x + (size_t) scb[b] * bs;
                    const int line = off + b * E + r * bs;
                    int c = 0;
                    for (; c + UC * V <= bs; c += UC * V)
                      {
                        Pack<T, V> xv[UC];
#pragma unroll
                        for (int u = 0; u < UC; u++)
                          xv[u] = ld_x<T, V> (xb + c + u * V);
#pragma unroll
                        for (int u = 0; u < UC; u++)
                          {
                            const Pack<T, V> av = ld_s<T, V> (sv + at<T, PAD> (line + c + u * V));
#pragma unroll
                            for (int k = 0; k < V; k++)
                              acc = fma (av.v[k], xv[u].v[k], acc);
                          }
                      }
#pragma unroll 4
                    for (; c < bs; c += V)
                      {
                        const Pack<T, V> xv = ld_x<T, V> (xb + c);
                        const Pack<T, V> av = ld_s<T, V> (sv + at<T, PAD> (line + c));
#pragma unroll
                        for (int k = 0; k < V; k++)
                          acc = fma (av.v[k], xv.v[k], acc);
                      }
                    done ();
                  }
              }
          }
      __syncthreads ();
      for (int s = t; s < nr * bs; s += kThreads)
        {
          const int i = s / bs, rr = s - i * bs;
          const int beg = rp[i], end = rp[i + 1];
          const int lo = max (beg, p0) - p0, hi = min (end - p0, nb);
          if (lo < hi)
            {
              T a = beg < p0 ? sum[s] : (T) 0;
              for (int q = lo / K; q * K < hi; q++)
                a += part[(q + i) * bs + rr];
              if (end - p0 <= nb)
                y[(int64_t) (r0 + i) * bs + rr] = a;
              else
                sum[s] = a;
            }
          else if (p0 == 0 && beg == end)
            y[(int64_t) (r0 + i) * bs + rr] = 0;
        }
      __syncthreads ();
    }
}

// A tile with more than kFullTile times the blocks that a CTA stages at once holds
// rows far above the average. Where such rows lie together, as in a bordered
// system, one CTA would walk them all, 4 us for every CTA's fill. So the full tiles
// of a window of kWindow CTAs are shared out among these by blocks, whole rows at
// a time; each CTA looks at the window's offsets, which its neighbours read too.
// At block size 3 only. us, warp per row / a CTA its own tile / shared, FP64, 20 000 rows of
// 7 with 64 rows of 1000 blocks at the end: bs 3 91 / 435 / 60, bs 5 259 / 343 / 107, bs 6
// 322 / 355 / 132, bs 7 480 / 332 / -, more at larger sizes; 8 rows of 4000, bs 3 294 / 599 / 101.
// Other matrices pay for it (us, own tile / shared: bs 3 FP64, 150 001 rows of 0-15 37.1 /
// 38.1, 100 000 rows of 7 22.6 / 23.0, 20 000 rows of 7 9.1 / 9.9, FP32 within 2 %; bs 5, 42 000
// rows of 6, 21.4 / 22.2), which a loss of 4.8 times is worth and one of a
// third at most is not. (Cutting all tiles by blocks, by a search of the offsets: 40.9, and
// bs 12 36.9 -> 39.7.)
constexpr int kFullTile = 4, kWindow = 32;
constexpr bool shares_tiles (int bs) { return bs == 3; }

// Its CTAs: the last window takes the rest too, up to 2 kWindow - 1.
__device__ __forceinline__ int2 window ()
{
  const int last = max (1, (int) gridDim.x / kWindow) - 1, w = min ((int) blockIdx.x / kWindow, last);
  return make_int2 (w * kWindow, w == last ? (int) gridDim.x : (w + 1) * kWindow);
}

__device__ __forceinline__ int tile_blocks (const TilePlan &P, int nbr, const int *__restrict__ row_ptr, int tile)
{
  const int r0 = min (nbr, tile * P.rows), r1 = min (nbr, r0 + P.rows);
  return __ldg (row_ptr + r1) - __ldg (row_ptr + r0);
}

template <typename T, int BSC, int V, bool PAD>
__device__ __noinline__ void full_tiles (int nbr, int bs_rt, const TilePlan &P, const int *__restrict__ row_ptr,
                                         const int *__restrict__ cols, const T *__restrict__ vals,
                                         const T *__restrict__ x, T *__restrict__ y)
{
  const int w0 = window ().x, w1 = window ().y;
  const int me = blockIdx.x - w0, many = w1 - w0;
  int64_t total = 0;
  for (int q = w0; q < w1; q++)
    if (const int n = tile_blocks (P, nbr, row_ptr, q); n > kFullTile * P.cap)
      total += n;
  // this CTA's share, counted over the blocks of the window's full tiles
  const int64_t lo = (total * me + many - 1) / many;
  const int64_t hi = me + 1 == many ? INT64_MAX : (total * (me + 1) + many - 1) / many;
  int64_t before = 0;
  for (int q = w0; q < w1; q++)
    {
      const int n = tile_blocks (P, nbr, row_ptr, q);
      if (n <= kFullTile * P.cap)
        continue;
      const int r0 = q * P.rows, nr = min (nbr - r0, P.rows), B0 = __ldg (row_ptr + r0);
      int beg = 0, end = 0; // rows that begin before the share's ends
      for (int i0 = 0; i0 < nr; i0 += kThreads)
        {
          const int i = i0 + threadIdx.x;
          const int64_t at = i < nr ? before + __ldg (row_ptr + r0 + i) - B0 : INT64_MAX;
          beg += __syncthreads_count (i < nr && at < lo);
          end += __syncthreads_count (i < nr && at < hi);
        }
      if (beg < end)
        {
          const int b = __ldg (row_ptr + r0 + beg);
          tile_pass<T, BSC, V, PAD> (nbr, bs_rt, P, row_ptr, cols, vals, x, y, r0 + beg, end - beg, b,
                                     __ldg (row_ptr + r0 + end) - b);
        }
      before += n;
    }
}

template <typename T, int BSC, int V, bool PAD>
__global__ void __launch_bounds__ (kThreads, 8)
  tile_kernel (int nbr, int bs_rt, TilePlan P, const int *__restrict__ row_ptr, const int *__restrict__ cols,
               const T *__restrict__ vals, const T *__restrict__ x, T *__restrict__ y)
{
  const int r0 = blockIdx.x * P.rows;
  const int nr = min (nbr - r0, P.rows);
  const int B0 = __ldg (row_ptr + r0), B1 = __ldg (row_ptr + r0 + nr);
  tile_pass<T, BSC, V, PAD> (nbr, bs_rt, P, row_ptr, cols, vals, x, y, r0, nr, B0, B1 - B0);
}

// The same with full tiles shared out (P stays where it is: full_tiles takes its
// address).
template <typename T, int BSC, int V, bool PAD>
__global__ void __launch_bounds__ (kThreads, 10)
  shared_tile_kernel (int nbr, int bs_rt, const __grid_constant__ TilePlan P, const int *__restrict__ row_ptr,
                      const int *__restrict__ cols, const T *__restrict__ vals, const T *__restrict__ x,
                      T *__restrict__ y)
{
  const int r0 = blockIdx.x * P.rows;
  const int nr = min (nbr - r0, P.rows);
  const int B0 = __ldg (row_ptr + r0), n = __ldg (row_ptr + r0 + nr) - B0;
  const int2 w = window ();
  const int tile = min (w.x + (int) threadIdx.x, w.y - 1);
  const int a0 = __ldg (row_ptr + tile * P.rows), a1 = __ldg (row_ptr + min (nbr, (tile + 1) * P.rows));
  if (n <= kFullTile * P.cap)
    tile_pass<T, BSC, V, PAD> (nbr, bs_rt, P, row_ptr, cols, vals, x, y, r0, nr, B0, n);
  if (__syncthreads_or (a1 - a0 > kFullTile * P.cap))
    full_tiles<T, BSC, V, PAD> (nbr, bs_rt, P, row_ptr, cols, vals, x, y);
}

template <typename T, int BSC, int V>
int launch (int nbr, int bs, TilePlan P, const int *rp, const int *c, const T *v, const T *x, T *y, cudaStream_t s)
{
  constexpr bool PAD = BSC > 0 && (BSC * sizeof (T)) % 64 == 0;
  const int S = (int) sizeof (T);
  const size_t raw = (size_t) P.cap * bs * bs * S;
  auto up = [] (size_t v) { return (int) ((v + 15) / 16 * 16); };
  P.o_cols = PAD ? (int) ((raw + 16 + 127) / 128 * 144) : up (raw + 16);
  P.o_part = P.o_cols + up (P.cap * 4 + 16);
  P.o_sum = P.o_part + up ((size_t) ((P.cap + P.chunk - 1) / P.chunk + P.rows) * bs * S);
  P.o_rp = P.o_sum + up ((size_t) P.rows * bs * S);
  P.o_first = P.o_rp + up ((P.rows + 1) * 4);
  P.smem = P.o_first + up ((size_t) (P.cap + P.chunk - 1) / P.chunk * 4);
  const unsigned grid = (unsigned) ((nbr + P.rows - 1) / P.rows);
  if constexpr (shares_tiles (BSC))
    shared_tile_kernel<T, BSC, V, PAD><<<grid, kThreads, P.smem, s>>> (nbr, bs, P, rp, c, v, x, y);
  else
    tile_kernel<T, BSC, V, PAD><<<grid, kThreads, P.smem, s>>> (nbr, bs, P, rp, c, v, x, y);
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}

template <typename T>
int tile_typed (int nbr, int bs, int64_t nnzb, const int *rp, const int *c, const T *v, const T *x, T *y, bool *took,
                cudaStream_t s)
{
  const double avg = std::max (0.5, (double) nnzb / nbr);
  const double block = (double) bs * bs * sizeof (T) + 4;
  // About 24 KB of values and columns per CTA (20 KB for the smallest blocks,
  // whose partial sums take more room): eight CTAs an SM hide one another's
  // copies. Measured at 12 to 52 KB and with 256 threads per CTA; larger tiles
  // and room kept for rows above the average were slower.
  const double room = (bs <= (sizeof (T) == 4 ? 8 : 5) ? 20 : 24) * 1024;
  TilePlan P{};
  const int slots = kThreads / bs;
  P.chunk = std::max (1, (int) (room / (block * slots) + 0.5));
  P.cap = P.chunk * slots;
  P.rows = std::max (1, std::min ((int) (P.cap / avg), std::min (kMaxRows, 8 * kThreads / bs)));
  // Below three tiles an SM the warp-per-row kernel is faster: FP32 bs 3,
  // 20 000 rows (294 tiles) 4.8 against 7.1 us; FP64 bs 3, 20 000 rows (555
  // tiles) 12.9 against 8.6 us.
  *took = (nbr + P.rows - 1) / P.rows >= 3 * 152;
  if (!*took)
    return BMFP_SUCCESS;
  const bool x16 = ((uintptr_t) x & 15) == 0;
  constexpr int VS = 16 / (int) sizeof (T);
#define BMFP_TILE(B)                                                                                                 \
  case B:                                                                                                            \
    {                                                                                                                \
      constexpr int W = B % VS == 0 ? VS : (B % 2 == 0 && VS == 4) ? 2 : 1;                                          \
      return x16 ? launch<T, B, W> (nbr, bs, P, rp, c, v, x, y, s) : launch<T, B, 1> (nbr, bs, P, rp, c, v, x, y, s); \
    }
  switch (bs)
    {
      BMFP_TILE (3) BMFP_TILE (5) BMFP_TILE (6) BMFP_TILE (7) BMFP_TILE (9) BMFP_TILE (10) BMFP_TILE (11)
      BMFP_TILE (12) BMFP_TILE (13) BMFP_TILE (14) BMFP_TILE (15) BMFP_TILE (17) BMFP_TILE (18) BMFP_TILE (20)
      BMFP_TILE (24)
    }
#undef BMFP_TILE
  if (bs % VS == 0 && x16)
    return launch<T, 0, VS> (nbr, bs, P, rp, c, v, x, y, s);
  return launch<T, 0, 1> (nbr, bs, P, rp, c, v, x, y, s);
}
} // namespace

int spmv_tile (int dtype, int nbr, int bs, int64_t nnzb, const int *rp, const int *c, const void *v, const void *x,
               void *y, bool *took, cudaStream_t s)
{
  if (dtype == BMFP_R64F)
    return tile_typed<double> (nbr, bs, nnzb, rp, c, (const double *) v, (const double *) x, (double *) y, took, s);
  return tile_typed<float> (nbr, bs, nnzb, rp, c, (const float *) v, (const float *) x, (float *) y, took, s);
}
} // namespace bmfp
