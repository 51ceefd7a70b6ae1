// spiffe_b200/csrc/compact.cuh -- removal of the particles lost in a push, by
// one block: the common part of the two forms' compaction kernels.
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
// all slots, CT_SCAN a thread (a burst of losses: a particle is lost once, so
// what one block takes longer for it than the grid would, about a nanosecond
// a loss, is little beside the particle's pushes).  is_lost(i): slot i was
// lost in this push; move(dst, src) copies a particle.  Called by all CT
// threads of one block.
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
