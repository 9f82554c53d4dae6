// otg_order.cuh — canonical order of query results, (query << 32 | id) items with an optional
// distance, in CSR form: ids ascending per query, or (distance, id) ascending per query.
//
// By runs: a counting pass places every item in its query's run, and each run is sorted on the chip
// (one warp up to kRunSortMax items, one block up to kBlockRunMax). Bound by the passes over the
// items (about 40 bytes each) where the radix sorts it replaces move 24 bytes of every item per
// 8-bit digit (13 passes for distances: three keys of 20, 64 and 15 bits).
// By bits: dense id results as one row of bits per query; see order_by_bits.
#pragma once

#include "otg_query.cuh"

namespace otg
{

// the count of every query and each item's slot in its query's run (the lanes of a warp that hold
// the same query take their slots with one atomic)
__global__ void query_slots_kernel(const u64* __restrict__ items, u64 m, u32* __restrict__ cnt, u32* __restrict__ slot)
{
  const u32 lane = threadIdx.x & 31;
  const u64 stride = u64(gridDim.x) * blockDim.x;
  for (u64 base = blockIdx.x * u64(blockDim.x) + (threadIdx.x & ~31u); base < m; base += stride)
  {
    const u64 i = base + lane;
    const bool v = i < m;
    const u32 q = v ? u32(items[i] >> 32) : 0xffffffffu;
    const u32 peers = __match_any_sync(~0u, q);
    const int leader = __ffs(int(peers)) - 1;
    u32 b = 0;
    if (v && int(lane) == leader)
      b = atomicAdd(&cnt[q], u32(__popc(peers)));
    b = __shfl_sync(~0u, b, leader);
    if (v)
      slot[i] = b + __popc(peers & ((1u << lane) - 1u));
  }
}
__global__ void query_scatter_kernel(const u64* __restrict__ items, const double* __restrict__ dist, const u32* __restrict__ slot, u64 m,
                                     const u64* __restrict__ off, u32* __restrict__ ids, double* __restrict__ distOut)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < m; i += u64(gridDim.x) * blockDim.x)
  {
    const u64 it = items[i];
    const u64 to = off[u32(it >> 32)] + slot[i];
    ids[to] = u32(it);
    if (dist)
      distOut[to] = dist[i];
  }
}

// offsets (nq + 1 of them) from the counts in one block: up to kScanOneBlock queries this is one launch where
// the scan over tiles takes three
constexpr u64 kScanOneBlock = 16384;
__global__ void __launch_bounds__(1024) scan_one_block_kernel(const u32* __restrict__ cnt, u32 nq, u64* __restrict__ off)
{
  __shared__ u64 warpSums[32];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u32 per = (nq + 1023) / 1024; // counts per thread
  const u32 b = min(nq, threadIdx.x * per), e = min(nq, b + per);
  u64 sum = 0;
  for (u32 i = b; i < e; ++i)
    sum += cnt[i];
  u64 incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const u64 y = __shfl_up_sync(~0u, incl, o);
    if (lane >= u32(o))
      incl += y;
  }
  if (lane == 31)
    warpSums[w] = incl;
  __syncthreads();
  u64 at = incl - sum;
  for (u32 i = 0; i < w; ++i)
    at += warpSums[i];
  for (u32 i = b; i < e; ++i)
  {
    off[i] = at;
    at += cnt[i];
  }
  if (threadIdx.x == 1023)
    off[nq] = at;
}

// sort key of an item: the distance's bits (distances are >= 0, so bit order is value order), then
// the id; without distances the id alone
template<bool DIST>
struct RunKey
{
  u64 d;
  u32 id;
  __device__ __forceinline__ bool less(const RunKey& o) const { return DIST ? (d < o.d || (d == o.d && id < o.id)) : id < o.id; }
};

template<bool DIST>
__device__ __forceinline__ RunKey<DIST> run_load(const u32* ids, const double* dist, u64 i)
{
  RunKey<DIST> k;
  k.id = ids[i];
  k.d = DIST ? u64(__double_as_longlong(dist[i])) : 0;
  return k;
}

// ascending bitonic sort of one key per lane
template<bool DIST>
__device__ __forceinline__ void run_sort_lanes(RunKey<DIST>& v, u32 lane)
{
#pragma unroll
  for (u32 k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (u32 j = k >> 1; j > 0; j >>= 1)
    {
      RunKey<DIST> o;
      o.id = __shfl_xor_sync(~0u, v.id, j);
      o.d = DIST ? __shfl_xor_sync(~0u, v.d, j) : 0;
      const bool up = (lane & k) == 0, lower = (lane & j) == 0;
      const bool take = (lower == up) ? o.less(v) : v.less(o);
      if (take)
        v = o;
    }
}

// ascending bitonic sort of R words per lane, word r of a lane at r * 32 + lane, of which the first n are not ~0
template<int R>
__device__ __forceinline__ void run_sort_words(u32 (&x)[R], u32 n, u32 lane)
{
#pragma unroll
  for (u32 size = 2; size <= u32(R) * 32; size <<= 1)
  {
    if (R == 1 && size >= 2 * n)
      break;
#pragma unroll
    for (u32 stride = size >> 1; stride > 0; stride >>= 1)
    {
      if (stride >= 32)
      {
#pragma unroll
        for (u32 r = 0; r < u32(R); ++r)
        {
          const u32 o = r ^ (stride >> 5);
          if (o > r)
          {
            const bool up = ((r * 32) & size) == 0;
            const u32 a = min(x[r], x[o]), b = max(x[r], x[o]);
            x[r] = up ? a : b;
            x[o] = up ? b : a;
          }
        }
      }
      else
      {
#pragma unroll
        for (u32 r = 0; r < u32(R); ++r)
        {
          const u32 o = __shfl_xor_sync(~0u, x[r], stride);
          const bool up = ((r * 32 + lane) & size) == 0, lower = (lane & stride) == 0;
          x[r] = (lower == up) ? min(x[r], o) : max(x[r], o);
        }
      }
    }
  }
}
// ascending order of n (at most R * 32) ids
template<int R>
__device__ __forceinline__ void run_order_ids(u32* ids, u32 n, u32 lane)
{
  u32 x[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    x[r] = r * 32 + lane < n ? ids[r * 32 + lane] : ~0u;
  run_sort_words<R>(x, n, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r * 32 + lane < n)
      ids[r * 32 + lane] = x[r];
}

// (distance, id) order of n (2 to R * 32) items in shared memory by one warp; false if they need the general
// order (run_order_general). Distances first become 24 bits, their place between the least and the greatest, with
// their index below, and are sorted as one 32-bit word each: a bitonic step takes 4 instructions, on the 96-bit
// items about 25. What the 24 bits leave in the wrong order (ties, of which a ray that starts inside several
// boxes has a few at zero) shows when neighbours are compared, and a few odd-even rounds mend it.
constexpr u32 kRunFixRounds = 6;
template<int R>
__device__ __forceinline__ bool run_order_packed(u64* sd, u32* si, u32 n, u32 lane)
{
  float f[R];
  u32 mn = 0x7f800000u, mx = 0;
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    f[r] = i < n ? __double2float_rn(__longlong_as_double((long long)sd[i])) : 0.f;
    if (i < n)
    {
      mn = min(mn, __float_as_uint(f[r]));
      mx = max(mx, __float_as_uint(f[r]));
    }
  }
  mn = __reduce_min_sync(~0u, mn);
  mx = __reduce_max_sync(~0u, mx);
  const float f0 = __uint_as_float(mn), scale = 16777215.f / fmaxf(__uint_as_float(mx) - f0, 0x1p-100f);
  u32 x[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    x[r] = i < n ? (min(u32((f[r] - f0) * scale), 0xffffffu) << 8) | i : ~0u;
  }
  run_sort_words<R>(x, n, lane);
  u64 d[R];
  u32 id[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane, from = x[r] & 255u;
    d[r] = i < n ? sd[from] : 0;
    id[r] = i < n ? si[from] : 0;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    if (i < n)
    {
      sd[i] = d[r];
      si[i] = id[r];
    }
  }
  __syncwarp();
  for (u32 round = 0; round < kRunFixRounds; ++round)
  {
    u32 wrong = 0;
    for (u32 i = lane; i + 1 < n; i += 32)
    {
      const RunKey<true> a{ sd[i], si[i] }, b{ sd[i + 1], si[i + 1] };
      wrong += b.less(a);
    }
    wrong = __reduce_add_sync(~0u, wrong);
    if (!wrong)
      return true;
    if (wrong > 2 * kRunFixRounds) // more ties than the rounds are likely to mend
      return false;
    for (u32 parity = 0; parity < 2; ++parity)
    {
      for (u32 i = 2 * lane + parity; i + 1 < n; i += 64)
      {
        const RunKey<true> a{ sd[i], si[i] }, b{ sd[i + 1], si[i + 1] };
        if (b.less(a))
        {
          sd[i] = b.d;
          si[i] = b.id;
          sd[i + 1] = a.d;
          si[i + 1] = a.id;
        }
      }
      __syncwarp();
    }
  }
  return false;
}

constexpr u32 kRunSortMax = 256;
constexpr int kRunSortWarps = 8;
// The general order of a run of at most kRunSortMax items: each 32 items in registers, then every item's place is
// its place among its 32 plus the counts of smaller items in the other sorted groups (binary searches in shared memory).
__device__ __forceinline__ void run_order_general(u32* ids, double* dist, u64* sd, u32* si, u32 len, u32 lane)
{
  const u32 groups = (len + 31) >> 5;
  for (u32 g = 0; g < groups; ++g)
  {
    const u32 i = g * 32 + lane;
    RunKey<true> v{ ~0ull, ~0u };
    if (i < len)
      v = run_load<true>(ids, dist, i);
    run_sort_lanes<true>(v, lane);
    si[i] = v.id;
    sd[i] = v.d;
  }
  __syncwarp();
  for (u32 i = lane; i < len; i += 32) // the padding of the last group sorts last in it
  {
    const RunKey<true> v{ sd[i], si[i] };
    u32 rank = lane;
    for (u32 h = 0; h < groups; ++h)
    {
      if (h == i >> 5)
        continue;
      u32 lo = 0;
#pragma unroll
      for (u32 s = 16; s > 0; s >>= 1)
      {
        const u32 j = h * 32 + lo + s - 1;
        const RunKey<true> o{ sd[j], si[j] };
        if (o.less(v))
          lo += s;
      }
      const RunKey<true> o{ sd[h * 32 + lo], si[h * 32 + lo] };
      rank += lo + (o.less(v) ? 1u : 0u);
    }
    ids[rank] = v.id;
    dist[rank] = __longlong_as_double((long long)v.d);
  }
}

// a run that a warp does not sort: into the list for run_sort_block_kernel, or only counted (longCount[1]) where it is too
// long for that: the caller then orders everything another way and spares the block sorts (64 views of 500k
// boxes, 89k ids of which one view has more than 8192: 58 us of 0.36 ms)
constexpr u32 kBlockRunMax = 8192;
__device__ __forceinline__ void list_long_run(u32 run, u64 len, u32* longCount, u32* longRuns, u32 longCap)
{
  if (len > kBlockRunMax)
  {
    atomicAdd(longCount + 1, 1u);
    return;
  }
  const u32 at = atomicAdd(longCount, 1u);
  if (at < longCap)
    longRuns[at] = run;
}

// One warp per query sorts its run in place: ids as words in registers, distances by packed words, or by the general
// order where those give up. Runs above kRunSortMax go to the list longRuns (longCount[0] counts them)
// for run_sort_block_kernel (list_long_run). Bound by issue: the general order for every run took 0.149 ms for the distances of 60k rays
// (now 0.050), 8.1 us for the ids of 10k ranges of about 60 points (now 4.0) and 38.6 us for those of a forest's 1M ranges
// of a few boxes (33.9; 60 at the occupancy that the compiler's choice of registers for 256 ids left).
template<bool DIST>
__global__ void __launch_bounds__(kRunSortWarps * 32, DIST ? 0 : 8) run_sort_kernel(const u64* __restrict__ off, u64 nq, u32* __restrict__ ids, double* __restrict__ dist,
                                                                    u32* __restrict__ longCount, u32* __restrict__ longRuns, u32 longCap)
{
  __shared__ u64 sd[DIST ? kRunSortWarps : 1][DIST ? kRunSortMax : 1];
  __shared__ u32 si[DIST ? kRunSortWarps : 1][DIST ? kRunSortMax : 1];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u64 warps = u64(gridDim.x) * kRunSortWarps;
  for (u64 q = u64(blockIdx.x) * kRunSortWarps + w; q < nq; q += warps)
  {
    const u64 b = off[q];
    const u64 len64 = off[q + 1] - b;
    if (len64 <= 1)
      continue;
    if (len64 > kRunSortMax)
    {
      if (lane == 0)
        list_long_run(u32(q), len64, longCount, longRuns, longCap);
      continue;
    }
    const u32 len = u32(len64);
    if constexpr (!DIST)
    {
      if (len <= 32)
        run_order_ids<1>(ids + b, len, lane);
      else if (len <= 64)
        run_order_ids<2>(ids + b, len, lane);
      else if (len <= 128)
        run_order_ids<4>(ids + b, len, lane);
      else
        run_order_ids<8>(ids + b, len, lane);
    }
    else
    {
      for (u32 i = lane; i < len; i += 32)
      {
        si[w][i] = ids[b + i];
        sd[w][i] = u64(__double_as_longlong(dist[b + i]));
      }
      __syncwarp();
      const bool done = len <= 32    ? run_order_packed<1>(sd[w], si[w], len, lane)
                        : len <= 64  ? run_order_packed<2>(sd[w], si[w], len, lane)
                        : len <= 128 ? run_order_packed<4>(sd[w], si[w], len, lane)
                                     : run_order_packed<8>(sd[w], si[w], len, lane);
      if (done)
        for (u32 i = lane; i < len; i += 32)
        {
          ids[b + i] = si[w][i];
          dist[b + i] = __longlong_as_double((long long)sd[w][i]);
        }
      else
        run_order_general(ids + b, dist + b, sd[w], si[w], len, lane);
      __syncwarp();
    }
  }
}

// One block per listed run (at most kBlockRunMax items) sorts it in place with a bitonic network in shared memory
// (dynamic: 12 or 4 bytes per item).
constexpr int kBlockSortThreads = 512;
template<bool DIST>
__global__ void __launch_bounds__(kBlockSortThreads) run_sort_block_kernel(const u64* __restrict__ off, u32* __restrict__ ids, double* __restrict__ dist,
                                                                         const u32* __restrict__ longCount, const u32* __restrict__ longRuns, u32 longCap)
{
  extern __shared__ u64 runMem[];
  u64* sd = runMem;
  u32* si = reinterpret_cast<u32*>(runMem + (DIST ? kBlockRunMax : 0));
  const u32 n = min(longCount[0], longCap);
  for (u32 r = blockIdx.x; r < n; r += gridDim.x)
  {
    const u32 q = longRuns[r];
    const u64 b = off[q];
    const u32 len = u32(min(off[q + 1] - b, u64(kBlockRunMax)));
    u32 P = 512;
    while (P < len)
      P <<= 1;
    for (u32 i = threadIdx.x; i < P; i += kBlockSortThreads)
    {
      si[i] = i < len ? ids[b + i] : ~0u;
      if (DIST)
        sd[i] = i < len ? u64(__double_as_longlong(dist[b + i])) : ~0ull;
    }
    __syncthreads();
    for (u32 k = 2; k <= P; k <<= 1)
      for (u32 j = k >> 1; j > 0; j >>= 1)
      {
        for (u32 t = threadIdx.x; t < P / 2; t += kBlockSortThreads)
        {
          const u32 i = ((t & ~(j - 1)) << 1) | (t & (j - 1)), x = i + j;
          const RunKey<DIST> a{ DIST ? sd[i] : 0, si[i] }, c{ DIST ? sd[x] : 0, si[x] };
          const bool swap = (i & k) == 0 ? c.less(a) : a.less(c);
          if (swap)
          {
            si[i] = c.id;
            si[x] = a.id;
            if (DIST)
            {
              sd[i] = c.d;
              sd[x] = a.d;
            }
          }
        }
        __syncthreads();
      }
    for (u32 i = threadIdx.x; i < len; i += kBlockSortThreads)
    {
      ids[b + i] = si[i];
      if (DIST)
        dist[b + i] = __longlong_as_double((long long)sd[i]);
    }
    __syncthreads();
  }
}

// ---- order by bits. A row is a whole number of chunks of kBitChunk bits (256 words, one warp's work).
// Rows of a single tree's queries are all rowChunks long; those of a forest start at rowBase[q].
constexpr u32 kBitChunk = 8192;

__global__ void bit_rows_kernel(const u32* __restrict__ qTree, const u64* __restrict__ treeOff, u64 nq, u32* __restrict__ rowChunks)
{
  for (u64 q = blockIdx.x * u64(blockDim.x) + threadIdx.x; q < nq; q += u64(gridDim.x) * blockDim.x)
  {
    const u32 t = qTree[q];
    rowChunks[q] = u32((treeOff[t + 1] - treeOff[t] + kBitChunk - 1) / kBitChunk);
  }
}
// zeroes the *chunks chunks in use
__global__ void bit_clear_kernel(uint4* __restrict__ bits, const u64* __restrict__ chunks)
{
  const u64 n = *chunks * (kBitChunk / 128);
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < n; i += u64(gridDim.x) * blockDim.x)
    bits[i] = make_uint4(0u, 0u, 0u, 0u);
}
__global__ void bit_mark_kernel(const u64* __restrict__ items, u64 m, const u64* __restrict__ rowBase, u32 rowChunks, u32* __restrict__ bits)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < m; i += u64(gridDim.x) * blockDim.x)
  {
    const u64 it = items[i];
    const u32 q = u32(it >> 32), id = u32(it);
    const u64 row = rowBase ? rowBase[q] : u64(q) * rowChunks;
    atomicOr(&bits[row * (kBitChunk / 32) + (id >> 5)], 1u << (id & 31));
  }
}
// set bits per chunk, one warp each (a chunk past the *used ones counts 0)
__global__ void bit_count_kernel(const uint4* __restrict__ bits, u64 chunks, const u64* __restrict__ used, u32* __restrict__ cnt)
{
  const u32 lane = threadIdx.x & 31;
  const u64 n = used ? *used : chunks;
  for (u64 c = (blockIdx.x * u64(blockDim.x) + threadIdx.x) >> 5; c < chunks; c += (u64(gridDim.x) * blockDim.x) >> 5)
  {
    u32 s = 0;
    if (c < n)
    {
      const uint4 a = bits[c * 64 + lane], b = bits[c * 64 + 32 + lane];
      s = __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w) + __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
    }
    for (int o = 16; o > 0; o >>= 1)
      s += __shfl_xor_sync(~0u, s, o);
    if (lane == 0)
      cnt[c] = s;
  }
}
// one warp per chunk writes its ids; the chunks' offsets at the rows' first chunks are the result's.
// m bounds the ids written (the items marked).
__global__ void bit_write_kernel(const u32* __restrict__ bits, const u64* __restrict__ off, u64 chunks, const u64* __restrict__ rowBase, u64 nq, u32 rowChunks,
                                 u64* __restrict__ offsets, u32* __restrict__ ids, u64 m)
{
  const u32 lane = threadIdx.x & 31;
  const u64 tid = blockIdx.x * u64(blockDim.x) + threadIdx.x, threads = u64(gridDim.x) * blockDim.x;
  for (u64 q = tid; q <= nq; q += threads)
    offsets[q] = off[rowBase ? rowBase[q] : q * rowChunks];
  for (u64 c = tid >> 5; c < chunks; c += threads >> 5)
  {
    u64 at = off[c];
    if (off[c + 1] == at)
      continue;
    // the row that holds chunk c: its first id in this chunk
    u64 row = 0;
    if (rowBase)
    {
      u64 lo = 0, hi = nq; // the last row that starts at or before c (rows are not empty)
      while (hi - lo > 1)
      {
        const u64 mid = (lo + hi) >> 1;
        if (rowBase[mid] <= c)
          lo = mid;
        else
          hi = mid;
      }
      row = rowBase[lo];
    }
    else
      row = c / rowChunks * rowChunks;
    const u32 first = u32(c - row) * kBitChunk;
    for (u32 k = 0; k < kBitChunk / 32; k += 32)
    {
      const u32 word = bits[c * (kBitChunk / 32) + k + lane];
      const u32 n = __popc(word);
      u32 incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
      {
        const u32 y = __shfl_up_sync(~0u, incl, o);
        if (lane >= u32(o))
          incl += y;
      }
      const u32 total = __shfl_sync(~0u, incl, 31);
      if (total >= 256)
      {
        // dense: one word after another, one bit per lane, so that the lanes write neighbours
        for (u32 j = 0; j < 32; ++j)
        {
          const u32 wj = __shfl_sync(~0u, word, j);
          const u64 to = at + __shfl_sync(~0u, incl - n, j) + __popc(wj & ((1u << lane) - 1u));
          if (((wj >> lane) & 1u) && to < m)
            ids[to] = first + (k + j) * 32 + lane;
        }
      }
      else
      {
        u64 to = at + incl - n;
        for (u32 b = word; b; b &= b - 1, ++to)
          if (to < m)
            ids[to] = first + (k + lane) * 32 + u32(__ffs(int(b)) - 1);
      }
      at += total;
    }
  }
}

// ---- pairs: one warp per 32 neighbouring a's sorts their runs of b's and writes (a, b): runs up to kPairRankMax by
// rank (the count of smaller b's in the run: runs average a few items), longer ones up to kRunSortMax as words in
// registers; runs above go to the list longRuns, for run_sort_block_kernel and pair_long_write_kernel. Ranks cost a run's
// length per item: 60k boxes of 178 and 739 pairs each, whole call, 1.90 and 9.97 ms with ranks up to 1024, 1.40 and 5.6 this way.
constexpr u32 kPairRankMax = 64;
constexpr u32 kPairTile = 512;
template<int R>
__device__ __forceinline__ void pair_order_run(const u32* bs, u32 a, u32 n, u32 lane, uint2* out)
{
  u32 x[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    x[r] = r * 32 + lane < n ? bs[r * 32 + lane] : ~0u;
  run_sort_words<R>(x, n, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r * 32 + lane < n)
      out[r * 32 + lane] = make_uint2(a, x[r]);
}
__global__ void __launch_bounds__(256) pair_write_kernel(const u64* __restrict__ off, u64 nA, const u32* __restrict__ bs, uint2* __restrict__ out,
                                                         u32* __restrict__ longCount, u32* __restrict__ longRuns, u32 longCap)
{
  __shared__ u32 sb[8][kPairTile];
  __shared__ u32 so[8][33];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u64 warps = u64(gridDim.x) * 8;
  for (u64 g = u64(blockIdx.x) * 8 + w; g * 32 < nA; g += warps)
  {
    const u64 a0 = g * 32;
    const u64 base = off[a0];
    const u64 at = off[min(a0 + lane + 1, nA)]; // runs past the last one are empty
    const u64 total = __shfl_sync(~0u, at, 31) - base;
    if (total == 0)
      continue;
    const u64 prev = __shfl_up_sync(~0u, at, 1);
    const u32 first = u32((lane ? prev : base) - base), len = u32(at - base) - first;
    if (len > kRunSortMax)
      list_long_run(u32(a0) + lane, len, longCount, longRuns, longCap);
    for (u32 mid = __ballot_sync(~0u, len > kPairRankMax && len <= kRunSortMax); mid; mid &= mid - 1)
    {
      const u32 r = u32(__ffs(int(mid))) - 1;
      const u32 b0 = __shfl_sync(~0u, first, r), n = __shfl_sync(~0u, len, r);
      if (n <= 128)
        pair_order_run<4>(bs + base + b0, u32(a0) + r, n, lane, out + base + b0);
      else
        pair_order_run<8>(bs + base + b0, u32(a0) + r, n, lane, out + base + b0);
    }
    if (!__any_sync(~0u, len > 0 && len <= kPairRankMax))
      continue;
    const u32 T = u32(total); // (below 2^32: all pairs are)
    so[w][lane + 1] = u32(at - base);
    if (lane == 0)
      so[w][0] = 0;
    const bool tile = T <= kPairTile;
    if (tile)
      for (u32 t = lane; t < T; t += 32)
        sb[w][t] = bs[base + t];
    __syncwarp();
    for (u32 t = lane; t < T; t += 32)
    {
      u32 r = 0; // the run of item t: the last one that starts at or before it
#pragma unroll
      for (u32 s = 16; s > 0; s >>= 1)
        if (so[w][r + s] <= t)
          r += s;
      const u32 b0 = so[w][r], b1 = so[w][r + 1];
      if (b1 - b0 > kPairRankMax)
        continue;
      u32 rank = 0;
      u32 v;
      if (tile)
      {
        v = sb[w][t];
        for (u32 x = b0; x < b1; ++x)
          rank += sb[w][x] < v ? 1u : 0u;
      }
      else
      {
        v = bs[base + t];
        for (u32 x = b0; x < b1; ++x)
          rank += bs[base + x] < v ? 1u : 0u;
      }
      out[base + b0 + rank] = make_uint2(u32(a0) + r, v);
    }
    __syncwarp();
  }
}
// the listed runs, once they are sorted in place
__global__ void __launch_bounds__(256) pair_long_write_kernel(const u64* __restrict__ off, const u32* __restrict__ bs, uint2* __restrict__ out,
                                                              const u32* __restrict__ longCount, const u32* __restrict__ longRuns, u32 longCap)
{
  const u32 n = min(longCount[0], longCap);
  for (u32 l = blockIdx.x; l < n; l += gridDim.x)
  {
    const u32 a = longRuns[l];
    const u64 e = off[a + 1];
    for (u64 i = off[a] + threadIdx.x; i < e; i += blockDim.x)
      out[i] = make_uint2(a, bs[i]);
  }
}
// (a << bBits | b) into (a, b)
__global__ void unpack_pairs_kernel(const u64* __restrict__ items, u64 m, u32 bBits, uint2* __restrict__ out)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < m; i += u64(gridDim.x) * blockDim.x)
    out[i] = make_uint2(u32(items[i] >> bBits), u32(items[i] & ((u64(1) << bBits) - 1)));
}

} // namespace otg
