// spiffe_b200/csrc/compact.cuh -- removal of the particles lost in a push: by
// one block, the common part of the two forms' compaction kernels, and a burst
// by every block of a grid.
#pragma once

#include <cub/block/block_radix_sort.cuh>

constexpr int CT = 1024, CT_ITEMS = 4, CT_SCAN = 16;

// Appends value(i) of the i in [0, span) with take(i), in index order, to
// out[]; returns their number.  Each of the CT threads looks at ITEMS
// neighbouring i per pass, a block-wide prefix count places them.
template <int ITEMS, class Take, class Value>
__device__ __forceinline__ int collect(long long span, int32_t *out, Take take, Value value)
{
  __shared__ int warp_tot[CT / 32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int base = 0;
  for (long long c0 = 0; c0 < span; c0 += (long long)CT * ITEMS) {
    const long long i0 = c0 + (long long)tid * ITEMS;
    unsigned mask = 0;
#pragma unroll
    for (int q = 0; q < ITEMS; q++)
      if (i0 + q < span && take(i0 + q))
        mask |= 1u << q;
    int upto = __popc(mask); // of this and the lower lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, d);
      upto += lane >= d ? v : 0;
    }
    if (lane == 31)
      warp_tot[wid] = upto;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < CT / 32; w++) {
      before += w < wid ? warp_tot[w] : 0;
      total += warp_tot[w];
    }
    int at = base + before + upto - __popc(mask);
    for (; mask; mask &= mask - 1)
      out[at++] = value(i0 + __ffs(mask) - 1);
    base += total;
    __syncthreads();
  }
  return base;
}

// Refills the lost slots below the new count np - n_lost from the survivors
// above it: the k-th hole in ascending index order takes the k-th survivor
// in ascending order, or in descending order with REVERSE (the reference's
// intended swap with the last).  So the result does not depend on the order
// the push appended the losses, which follows the timing of its blocks.  The
// holes, collected from the push's list, are put in order by a block radix
// sort when there are at most CT * CT_ITEMS of them, else collected again from
// all slots, CT_SCAN a thread (one block takes 4 to 35 ns a loss of a burst: the
// split form, whose particle is lost once; the FP64 form shares a burst among
// blocks, below).  is_lost(i): slot i was lost in this push; move(dst, src)
// copies a particle.  Called by all CT threads of one block.
template <bool REVERSE, class Lost, class Move>
__device__ __forceinline__ void compact_block(long long n_lost, long long np, const int32_t *lost_list, int32_t *holes,
                                              int32_t *donors, Lost is_lost, Move move)
{
  typedef cub::BlockRadixSort<int, CT, CT_ITEMS> HoleSort;
  __shared__ typename HoleSort::TempStorage sort_tmp;
  const long long new_np = np - n_lost;
  const int tid = threadIdx.x;
  const int n_holes = collect<1>(
      n_lost, holes, [&](long long i) { return lost_list[i] < new_np; }, [&](long long i) { return lost_list[i]; });
  if (n_holes <= CT * CT_ITEMS) {
    // the holes in ascending order (INT_MAX pads sort last)
    int k[CT_ITEMS];
#pragma unroll
    for (int q = 0; q < CT_ITEMS; q++) {
      const int at = tid * CT_ITEMS + q;
      k[q] = at < n_holes ? holes[at] : 0x7fffffff;
    }
    HoleSort(sort_tmp).Sort(k);
#pragma unroll
    for (int q = 0; q < CT_ITEMS; q++) {
      const int at = tid * CT_ITEMS + q;
      if (at < n_holes)
        holes[at] = k[q];
    }
  } else {
    collect<CT_SCAN>(
        new_np, holes, [&](long long i) { return is_lost((int)i); }, [](long long i) { return (int)i; });
  }
  // as many survivors above the new count as holes below it
  collect<1>(
      n_lost, donors, [&](long long i) { return !is_lost((int)(new_np + i)); },
      [&](long long i) { return (int)(new_np + i); });
  __syncthreads();
  for (int k = tid; k < n_holes; k += CT)
    move(holes[k], donors[REVERSE ? n_holes - 1 - k : k]);
}

// ---- a burst of losses, by every block of a grid
//
// The same pairing from the flags lost[] (bytes 0 or 1, readable to the end of
// the 16-byte word that holds the last).  A block takes the holes of a chunk of
// slots; it counts for itself the holes before and after its chunk and finds the
// survivors of its holes' ranks in the tail, so no block waits for another: the
// flags of a million particles are 1 MB from L2, some 10 us a block.

// Which of the slots i .. i+15 (i a multiple of 16) that lie in [lo, hi) have lost[] == want: bits 0 .. 15
__device__ __forceinline__ unsigned flags16(const uint8_t *lost, int i, int lo, int hi, bool want)
{
  const uint4 x = *reinterpret_cast<const uint4 *>(lost + i);
  auto four = [](unsigned v) { return ((v & 0x01010101u) * 0x01020408u) >> 24 & 15u; }; // a bit a byte
  unsigned m = four(x.x) | four(x.y) << 4 | four(x.z) << 8 | four(x.w) << 12;
  if (!want)
    m ^= 0xffffu;
  if (i < lo)
    m &= 0xffffu << (lo - i);
  if (i + 16 > hi)
    m &= (1u << max(hi - i, 0)) - 1;
  return m;
}

// the calling thread's share of the number of lost in [lo, hi)
__device__ __forceinline__ int count_lost(const uint8_t *lost, int lo, int hi)
{
  int n = 0;
#pragma unroll 4
  for (int i = (lo & ~15) + 16 * (int)threadIdx.x; i < hi; i += 16 * CT)
    n += __popc(flags16(lost, i, lo, hi, true));
  return n;
}

// out[rank] = slot for the slots of [lo, hi) with lost[] == want that have ranks
// r0 .. r1-1; the first of them all has rank `rank`.  A warp takes a run of slots.
__device__ __forceinline__ void place(const uint8_t *lost, int lo, int hi, bool want, int rank, int r0, int r1, int32_t *out)
{
  __shared__ int found[CT / 32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = lo >> 4, last = (hi + 15) >> 4, per = ((last - first + CT / 32 - 1) / (CT / 32) + 31) & ~31;
  const int k0 = first + w * per, k1 = min(k0 + per, last);
  int n = 0;
#pragma unroll 4
  for (int k = k0 + lane; k < k1; k += 32)
    n += __popc(flags16(lost, 16 * k, lo, hi, want));
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0)
    found[w] = n;
  __syncthreads();
  for (int v = 0; v < w; v++)
    rank += found[v];
  __syncthreads(); // found[] is used again
  if (rank >= r1 || rank + n <= r0)
    return;
  for (int k = k0 + lane; k - lane < k1 && rank < r1; k += 32) {
    unsigned m = k < k1 ? flags16(lost, 16 * k, lo, hi, want) : 0u;
    int upto = __popc(m);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, d);
      upto += lane >= d ? v : 0;
    }
    for (int at = rank + upto - __popc(m); m; m &= m - 1, at++)
      if (at >= r0 && at < r1)
        out[at] = 16 * k + __ffs(m) - 1;
    rank += __shfl_sync(0xffffffffu, upto, 31);
  }
}

template <bool REVERSE, class Move>
__device__ __forceinline__ void compact_burst(int n_lost, int np, const uint8_t *lost, int32_t *holes, int32_t *donors, Move move)
{
  __shared__ int sum[3];
  const int new_np = np - n_lost, tid = threadIdx.x;
  const int chunk = ((new_np + (int)gridDim.x - 1) / (int)gridDim.x + 15) & ~15;
  const int a0 = (int)min((long long)blockIdx.x * chunk, (long long)new_np), a1 = (int)min((long long)a0 + chunk, (long long)new_np);
  if (tid < 3)
    sum[tid] = 0;
  __syncthreads();
  int n[3] = {count_lost(lost, 0, a0), count_lost(lost, a0, a1), count_lost(lost, a1, new_np)};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    n[k] = __reduce_add_sync(0xffffffffu, n[k]);
    if ((tid & 31) == 0 && n[k])
      atomicAdd(sum + k, n[k]);
  }
  __syncthreads();
  const int h0 = sum[0], own = sum[1], n_holes = h0 + own + sum[2];
  if (!own)
    return;
  const int d0 = REVERSE ? n_holes - h0 - own : h0;
  place(lost, a0, a1, true, h0, h0, h0 + own, holes);
  place(lost, new_np, np, false, 0, d0, d0 + own, donors);
  __syncthreads();
  for (int k = h0 + tid; k < h0 + own; k += CT)
    move(holes[k], donors[REVERSE ? n_holes - 1 - k : k]);
}

// The end of a push: its particle-steps, the counts it changed, and the
// counters that the next push begins with.  `removed` particles leave the
// array; oa: no on-axis fields, so the push met none (advance_particles.c
// :113-114; with fields the push's reset does this first).
__device__ __forceinline__ void end_push(DevCounts *cnt, long long removed, long long new_np, int oa)
{
  cnt->pushed += cnt->npActive;
  cnt->npActive += cnt->new_active - removed;
  cnt->np = new_np;
  cnt->first_lost = 0x7fffffffffffffffLL;
  cnt->n_lost = 0;
  cnt->new_active = 0;
  if (oa) {
    cnt->oa_min = INFINITY; // HUGE
    cnt->oa_max = -INFINITY;
  }
}
