// FP64 product for block sizes 16 and 32 on row-major blocks, staged per warp.
//
// The owner mapping (one lane per scalar row, every FP64 instruction a useful
// multiply-add) reads a block line per lane: 32 lines per load, and the load
// pipe falls behind the FP64 pipe it feeds. Here a group of BS lanes owns a run
// of consecutive block rows, whose blocks are one contiguous run; the warp
// copies them, and their x, into a ring in shared memory with 16-byte cp.async,
// coalesced and some blocks ahead whatever row they belong to, and the lanes
// read their lines there. An exclusive-or on the 16-byte pieces' places keeps
// eight lanes off each other's banks. So it needs no column-major copy to run
// at the FP64 pipe's rate, which bounds it: an FP64 multiply-add starts every
// 64 cycles per warp and SM quarter, 1.25 TFLOP/s in all.
//
// Measured against the owner mapping (us): bs 32, 100 000 rows of 8 blocks,
// 1499 -> 1341 (97 % of the FP64 rate); rows of 0-15 blocks (30 000) 463 -> 397;
// 1000 rows 33 -> 24. bs 16: 100 000 rows 390 -> 352, rows of 0-15 154 -> 114,
// 1000 rows 13.6 -> 8.9. At bs 8 a row's eight lanes leave the copies too
// short: 92 -> 109, so it keeps the owner mapping. One row per group and as
// many CTAs as that takes, without the runs: 1437 at bs 32, 364 at bs 16.
#include "device_common.cuh"
#include "internal.h"

#include <algorithm>

namespace bmfp
{
namespace
{
constexpr int kThreads = 128;

// Stages of the ring, and bytes of one warp's stage: its 32 / BS blocks, then
// their x. Two CTAs of four warps per SM: two warps to an FP64 pipe.
template <int BS> constexpr int ring_depth () { return BS == 32 ? 3 : 6; }
template <int BS> constexpr int stage_bytes () { return 32 * BS * 8 + 32 * 8; }
constexpr int kCtasPerSm = 2;

// Place of piece k (16 bytes) of line r in its block.
template <int BS> __device__ __forceinline__ int place (int r, int k) { return r * (BS / 2) + (k ^ (r & 7)); }

// First row i with row_ptr[i] + i at `target` or later, by the whole warp (a
// 32-way search).
__device__ __forceinline__ int first_row (const int *__restrict__ row_ptr, int n_rows, int64_t target)
{
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = n_rows; // the answer lies in [lo, hi]
  while (lo < hi)
    {
      const int step = (hi - lo + 31) / 32;
      const int at = lo + lane * step; // ascending, so the lanes below target come first
      const unsigned below = __ballot_sync (0xffffffffu, at < hi && (int64_t) __ldg (row_ptr + at) + at < target);
      const int k = __popc (below);
      if (k == 0)
        return lo;
      const int last = lo + (k - 1) * step; // below target
      hi = min (hi, last + step);
      lo = last + 1;
    }
  return lo;
}

template <int BS>
__global__ void __launch_bounds__ (kThreads)
  ring_kernel (int nbr, const int *__restrict__ row_ptr, const int *__restrict__ cols, const double *__restrict__ vals,
               const double *__restrict__ x, double *__restrict__ y)
{
  extern __shared__ __align__ (16) unsigned char smem[];
  constexpr int D = ring_depth<BS> (), P = BS / 2, Q = 32 / BS; // pieces per line, groups per warp
  const int lane = threadIdx.x & 31, g = lane / BS, r = lane % BS;
  unsigned char *ring = smem + (size_t) (threadIdx.x >> 5) * D * stage_bytes<BS> ();
  const uint32_t ring_a = (uint32_t) __cvta_generic_to_shared (ring);
  // Runs of nearly equal numbers of blocks and rows together, so that a stretch
  // of empty rows is shared out too (a group per row where there are no more
  // rows than groups).
  const int groups = gridDim.x * (kThreads / BS);
  const int first = (int) ((blockIdx.x * kThreads + threadIdx.x) / 32) * Q; // the warp's first group
  const int base = __ldg (row_ptr);
  const int64_t work = (int64_t) __ldg (row_ptr + nbr) - base + nbr;
  int r0 = 0, r1 = 0;
  if (nbr <= groups)
    {
      r0 = min (nbr, first + g);
      r1 = min (nbr, r0 + 1);
    }
  else
    for (int q = 0; q <= Q; q++)
      {
        const int k = first + q;
        const int at = k >= groups ? nbr : k == 0 ? 0 : first_row (row_ptr, nbr, base + work * k / groups);
        if (q == g)
          r0 = at;
        if (q == g + 1)
          r1 = at;
      }
  if (r0 >= r1)
    r0 = r1 = 0;
  const int beg = __ldg (row_ptr + r0), n = __ldg (row_ptr + r1) - beg;
  const int *c = cols + beg;
  const double *a = vals + (size_t) beg * BS * BS;
  const int steps = (int) __reduce_max_sync (0xffffffffu, (unsigned) n);
  int col = n > 0 ? __ldg (c) : 0; // of the next block to copy
  auto copy = [&] (int j) {
    if (j < n)
      {
        const uint32_t s = ring_a + (uint32_t) (j % D * stage_bytes<BS> ());
        const double *b = a + (size_t) j * BS * BS;
#pragma unroll
        for (int i = 0; i < P; i++)
          {
            const int q = i * BS + r; // the group reads BS pieces side by side
            dev::cp_async16 (s + (uint32_t) ((g * BS * P + place<BS> (q / P, q % P)) * 16), b + q * 2, 16);
          }
        if (r < P)
          dev::cp_async16 (s + (uint32_t) (32 * BS * 8 + (g * P + r) * 16), x + (size_t) col * BS + r * 2, 16);
        if (j + 1 < n)
          col = __ldg (c + j + 1);
      }
    dev::cp_async_commit ();
  };
#pragma unroll
  for (int j = 0; j < D - 1; j++)
    copy (j);
  int row = r0;
  int end = row < r1 ? __ldg (row_ptr + row + 1) - beg : 0;
  int next_end = row + 1 < r1 ? __ldg (row_ptr + row + 2) - beg : 0;
  double acc0 = 0, acc1 = 0;
  // Rows that end at block j: the first with its sum, empty ones after it with 0.
  auto finish = [&] (int j) {
    while (row < r1 && end == j)
      {
        y[(int64_t) row * BS + r] = acc0 + acc1;
        acc0 = acc1 = 0;
        row++;
        end = next_end;
        next_end = row + 1 < r1 ? __ldg (row_ptr + row + 2) - beg : 0;
      }
  };
  finish (0);
  for (int j = 0; j < steps; j++)
    {
      copy (j + D - 1);
      dev::cp_async_wait<D - 1> ();
      __syncwarp ();
      if (j < n)
        {
          const double2 *s = reinterpret_cast<const double2 *> (ring + j % D * stage_bytes<BS> ());
          const double2 *line = s + g * BS * P, *xs = s + 32 * P + g * P;
#pragma unroll
          for (int k = 0; k < P; k++)
            {
              const double2 v = line[place<BS> (r, k)], xv = xs[k];
              acc0 = fma (v.x, xv.x, acc0);
              acc1 = fma (v.y, xv.y, acc1);
            }
          finish (j + 1);
        }
      __syncwarp ();
    }
}

template <int BS> constexpr int group_count () { return 152 * kCtasPerSm * (kThreads / BS); }

template <int BS>
int launch (int nbr, const int *rp, const int *c, const double *v, const double *x, double *y, cudaStream_t s)
{
  constexpr int smem = kThreads / 32 * ring_depth<BS> () * stage_bytes<BS> ();
  const int64_t want = ((int64_t) nbr * BS + kThreads - 1) / kThreads;
  const unsigned grid = (unsigned) std::min<int64_t> (want, 152 * kCtasPerSm);
  BMFP_CUDA (cudaFuncSetAttribute (ring_kernel<BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ring_kernel<BS><<<grid, kThreads, smem, s>>> (nbr, rp, c, v, x, y);
  BMFP_LAUNCH_CHECK ();
  return BMFP_SUCCESS;
}
} // namespace

// At bs 16 a group would have one or two rows between these bounds, and the
// last of them run alone: 4000 rows of 9 blocks 27.5 us, owner 25.8 (2600 rows
// 25.0 and 24.6; but 1800 rows 13.2 and 17.4, 5500 rows 34.8 and 35.6). At
// bs 32 the ring was ahead at every size (1300 rows 37.9 and 46.0, 2600 rows
// 56.5 and 66.4, 4000 rows 75.0 and 87.7).
bool spmv_ring_wins (int bs, int nbr)
{
  return bs == 32 || (bs == 16 && (nbr <= group_count<16> () || nbr > 2 * group_count<16> ()));
}

int spmv_ring (int nbr, int bs, const int *rp, const int *c, const double *v, const double *x, double *y,
               cudaStream_t s)
{
  switch (bs)
    {
    case 16: return launch<16> (nbr, rp, c, v, x, y, s);
    case 32: return launch<32> (nbr, rp, c, v, x, y, s);
    default: return fail (BMFP_ERROR_INVALID_VALUE, "no ring kernel for bs %d", bs);
    }
}
} // namespace bmfp
