// otg_knn.cu — batched GetNearestNeighbors for point trees: a persistent kernel with one warp per
// query (queries taken from a shared counter, so uneven k and uneven density balance out), an FP32
// outward-rounded distance filter, and an exact recheck of the few candidates near the k-th distance.
//
// Result semantics are those of the reference (core/ot_query.h:1208-1270 with AddEntityDistance
// :1058-1164): with F0 = U(maxDistance) (or the largest scalar when unbounded) and
// U(x) = fmax(tol, x * (1 + tol)) (GetValueWithToleranceUpper, :1033-1036), let S0 be the entities
// with distance d < F0. If |S0| >= k, F = U(d_k) with d_k the k-th smallest distance in S0; otherwise
// F = F0. The result is every entity with d < F, ordered by (d, id).
//
// Filter. Every entity gets FP32 bounds lo2 <= d^2 <= hi2 of the distance that the exact
// arithmetic computes: coordinates are stored as x32 = RN(x) with a per-entity error bound e, the
// query as a directed-rounding interval, and squares and sums use directed rounding; the bounds are
// then widened by a relative margin that covers the rounding of the exact formula itself. The warp
// keeps a shared-memory buffer of candidates with lo2 <= Fc2, where Fc is an FP32 upper bound of the
// final F derived from R2 = k-th smallest hi2 among entities certainly inside S0 (hi2 < F0^2).
// Because F <= U(d_k) <= U(sqrt(R2)) <= Fc, every result entity is a candidate. After the traversal
// only the candidates get the exact distance; they are sorted by (d, id) in shared memory and the
// reference rule is applied to them. Queries whose candidates do not fit the buffer (massive ties,
// or k above the buffer's limit) are answered by the plain one-thread-per-query kernels.
// Bound by instruction issue: a query of k = 32 visits about ten subtrees of the tree's lower levels and
// tests a few hundred points in FP32, then takes k exact distances (FP64 square roots) and orders them.
// 1M queries, k in 1..64, 16M points: 14.2 ms with leaf-by-leaf tests and shared-memory sorts for the bound and
// the order, 10.1 ms with bisection and register sorts, 6.8 ms with small subtrees tested whole,
// 6.55 ms with the pivots of knn_kth_bound and 40 warps per SM.
#include "otg_query.cuh"

#include <cfloat>
#include <cmath>
#include <cstddef>

namespace otg
{

constexpr float kInf = __builtin_huge_valf();
// High bits of a query's start, which otherwise is its slot: its results are in the plain kernels' result, or it has more
// than k and those after the first k start here in the array for them.
constexpr u32 kFromFallback = 1u << 31, kMoreThanK = 1u << 30;

// One warp's part of the shared memory, followed by its stack (stackCap nodes and bounds). The exact
// distances of the final order take the place of the bounds, which are not needed by then.
template<int CAP>
struct KnnWarpMem
{
  union
  {
    unsigned long long key[CAP]; // exact distance bits in the final order
    struct
    {
      float lo2[CAP];
      float hi2[CAP];
    };
  };
  u32 pos[CAP]; // sorted position of a candidate, then its entity id
};
template<int CAP>
__host__ __device__ constexpr size_t knn_warp_bytes(u32 stackCap)
{
  return sizeof(KnnWarpMem<CAP>) + size_t(stackCap) * (sizeof(u32) + sizeof(float)); // stackCap: a multiple of 4
}

struct KnnCounters
{
  unsigned long long out;      // result entries beyond their queries' slots
  unsigned long long tests;    // FP32 filter evaluations
  unsigned long long rechecks; // exact distance evaluations
  u32 work;                    // next query to take
  u32 fallbacks;
  u32 irregular; // queries with other than k results
  u32 err;
};

template<typename T>
struct KnnArgs
{
  const uint4* link;
  const float4* nodeBox32; // 2 per node: {min rounded down, 0}, {max rounded up, 0}
  const float4* geom32;    // per sorted entity: {x, y, z, error bound}
  const T* geom;           // exact coordinates (sorted)
  const u32* ids;
  u32 n, nNodes;
  const T* pts;
  const u32* kArr;
  u32 kAll;
  u32 nq;
  const u32* order; // processing order of the queries (spatially sorted), or null
  T F0, tol;
  float F0hi, F0lo2, tolHi, onePlusTolHi, widenLo, widenHi;
  u32 kLimit;
  u32 direct;   // subtrees of at most this many points are tested without their nodes
  u32 stackCap;
  KnnCounters* ctr;
  u32* fallback;
  u64* start;
  u32* count;
  // slots of k results per query, for the first k of them: query q's at slot[q], or at q * kAll
  const u64* slot;
  u64* evenOffsets; // nq + 1 offsets to write, or null
  u32* slotIds;
  double* slotDist;
  // the results after the first k (ties within the tolerance)
  u32* outIds;
  double* outDist;
  u64 outCap;
};

// ---------------------------------------------------------------- FP32 images
// point: {x, y, z, e} with x = RN(x64) and e >= max |x64 - x| inflated by 2^-20 (the per-entity bound
// arithmetic below relies on that margin); e = +inf and x = 0 for coordinates outside the FP32 range (such
// entities always pass the filter). e is half an ulp of the largest coordinate, in FP32: the exact
// difference took nine more FP64 instructions per point and set the kernel's time (4.26M points: 104 us).
template<typename T>
__global__ void point_image_kernel(const T* __restrict__ geom, u64 n, float4* __restrict__ out)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < n; i += u64(gridDim.x) * blockDim.x)
  {
    float v[3];
    float e = 0.f;
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      const float f = sizeof(T) == 8 ? __double2float_rn(double(geom[i * 3 + c])) : float(geom[i * 3 + c]);
      ok &= fabsf(f) < kInf;
      v[c] = f;
      e = fmaxf(e, fabsf(f));
    }
    // |x64 - x| <= 2^-24 |x| (1 + 2^-24), or 2^-150 in the subnormal range
    e = sizeof(T) == 8 ? fmaf(e, 0x1p-24f * (1.f + 0x1p-18f), 0x1p-148f) : 0.f;
    out[i] = ok ? make_float4(v[0], v[1], v[2], e) : make_float4(0.f, 0.f, 0.f, kInf);
  }
}

// Node boxes rounded outward: MinPoint geometry {min, size} (max = min + size), or the exact MBR max.
template<typename T>
__global__ void node_image_kernel(const T* __restrict__ nodeBox, const T* __restrict__ nodeMax, u64 m, float4* __restrict__ out)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < m; i += u64(gridDim.x) * blockDim.x)
  {
    float lo[3], hi[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      const double mn = double(nodeBox[i * 6 + c]);
      const double mx = nodeMax ? double(nodeMax[i * 3 + c]) : mn + double(nodeBox[i * 6 + 3 + c]);
      lo[c] = __double2float_rd(mn);
      hi[c] = __double2float_ru(mx);
    }
    out[2 * i] = make_float4(lo[0], lo[1], lo[2], 0.f);
    out[2 * i + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
  }
}

// ---------------------------------------------------------------- device helpers
// The per-node and per-entity bounds use round-to-nearest FP32 only (directed-rounding FP32
// instructions are much slower on this GPU); every rounding is covered by an explicit margin.
// With u = 2^-24, a round-to-nearest result r of a normal operation is within u|r| of the exact
// value, and sums and products of non-negative values gain at most a factor (1 + u) each.

// lower bound of the squared distance from the query interval [plo, phi] to an outward-rounded
// node box: each positive gap is shrunk by 2^-22 relative (covers its own rounding), the sum of
// squares by 2^-20 (covers four roundings), then by the caller's margin.
__device__ __forceinline__ float node_w2(const float4* __restrict__ nb, u32 node, const float* plo, const float* phi, float widenLo)
{
  const float4 mn = nb[2 * size_t(node)], mx = nb[2 * size_t(node) + 1];
  const float a[3] = { mn.x, mn.y, mn.z }, b[3] = { mx.x, mx.y, mx.z };
  float w2 = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c)
  {
    const float g = fmaxf(fmaxf(a[c] - phi[c], plo[c] - b[c]), 0.f) * (1.f - 0x1p-22f);
    w2 = fmaf(g, g, w2);
  }
  return w2 * ((1.f - 0x1p-20f) * widenLo);
}

// Bounds lo2 <= d^2 <= hi2 of the squared distance between the query (p32 = RN(p), per-coordinate
// error at most Sq, inflated by 2^-20) and an entity image {x32, e} (e inflated by 2^-20):
//   t = RN(x32 - p32) is within u|t| + e + Sq of the exact difference;
//   E = RN(|t| 2^-20 + RN(e + Sq)) >= 15u|t| + (e + Sq)_exact (1 + 12u) covers that error and the
//   rounding of |t| + E and |t| - E; the sums of squares are then widened by the caller's
//   margins, which also cover the rounding of the exact distance formula.
__device__ __forceinline__ void entity_bounds(float4 g, const float* p32, float Sq, float widenLo, float widenHi, float& l2, float& h2)
{
  const float x[3] = { g.x, g.y, g.z };
  const float S = g.w + Sq;
  float L = 0.f, H = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c)
  {
    const float a = fabsf(x[c] - p32[c]);
    const float E = fmaf(a, 0x1p-20f, S);
    const float hi = a + E;
    const float lo = fmaxf(a - E, 0.f);
    L = fmaf(lo, lo, L);
    H = fmaf(hi, hi, H);
  }
  l2 = fmaxf(fmaf(L, widenLo, -0x1p-140f), 0.f);
  h2 = fmaf(H, widenHi, 0x1p-140f);
}

__device__ __forceinline__ u32 pow2_at_least32(u32 v)
{
  return v <= 32 ? 32u : 1u << (32 - __clz(v - 1));
}

// ascending bitonic sort of (key, value) pairs by (key, value)
__device__ __forceinline__ void warp_sort_pairs(unsigned long long* k, u32* v, u32 n2, u32 lane)
{
  for (u32 size = 2; size <= n2; size <<= 1)
    for (u32 stride = size >> 1; stride > 0; stride >>= 1)
    {
      for (u32 t = lane; t < n2 / 2; t += 32)
      {
        const u32 i = ((t & ~(stride - 1)) << 1) | (t & (stride - 1));
        const u32 j = i + stride;
        const bool up = (i & size) == 0;
        const unsigned long long ki = k[i], kj = k[j];
        const u32 vi = v[i], vj = v[j];
        const bool greater = ki > kj || (ki == kj && vi > vj);
        const bool differ = ki != kj || vi != vj;
        if (differ && greater == up)
        {
          k[i] = kj;
          k[j] = ki;
          v[i] = vj;
          v[j] = vi;
        }
      }
      __syncwarp();
    }
}

// Ascending order of n (at most R * 32) distinct (key, value) pairs in shared memory. Keys are first
// reduced to 24 bits (their distance from the least key, as bits, shifted to fit) with their index below, and
// sorted as one 32-bit word each in registers: a bitonic step on a word takes 4 instructions, on the
// 96-bit pairs in shared memory about 25. Pairs that the 24 bits leave in the wrong order (ties and near
// ties) show when neighbours are compared, and then the pairs are sorted in full.
template<int R>
__device__ __forceinline__ void warp_order_pairs(unsigned long long* k, u32* v, u32 n, u32 lane)
{
  unsigned long long key[R];
  unsigned long long mn = ~0ull, mx = 0;
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    key[r] = i < n ? k[i] : ~0ull;
    if (i < n)
    {
      mn = min(mn, key[r]);
      mx = max(mx, key[r]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    mn = min(mn, __shfl_xor_sync(~0u, mn, o));
    mx = max(mx, __shfl_xor_sync(~0u, mx, o));
  }
  const int bits = 64 - __clzll((long long)(mx - mn));
  const int shift = bits > 24 ? bits - 24 : 0;
  u32 x[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    x[r] = i < n ? (u32((key[r] - mn) >> shift) << 8) | i : ~0u;
  }
#pragma unroll
  for (u32 size = 2; size <= u32(R) * 32; size <<= 1)
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
  u32 val[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane, from = x[r] & 255u;
    key[r] = i < n ? k[from] : ~0ull;
    val[r] = i < n ? v[from] : ~0u;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    if (i < n)
    {
      k[i] = key[r];
      v[i] = val[r];
    }
  }
  __syncwarp();
  bool wrong = false;
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const u32 i = r * 32 + lane;
    if (i + 1 < n)
    {
      const unsigned long long k1 = k[i + 1];
      wrong |= key[r] > k1 || (key[r] == k1 && val[r] > v[i + 1]);
    }
  }
  if (__any_sync(~0u, wrong))
  {
    const u32 n2 = pow2_at_least32(n);
    for (u32 i = n + lane; i < n2; i += 32)
    {
      k[i] = ~0ull;
      v[i] = ~0u;
    }
    __syncwarp();
    warp_sort_pairs(k, v, n2, lane);
  }
}

// An upper bound of the k-th least of the bufN <= C * 32 values that are below F0lo2, infinite with fewer than k of
// them: bisection on the float bits (ordered like the values, which are not negative). Squared distances of
// points spread evenly grow with the 2/3 power of their rank, so the first two pivots bracket that
// estimate. Stops once at most k + 1 values lie below, or after `steps` pivots.
template<int C>
__device__ __forceinline__ float knn_kth_bound(const float* hi2, float F0lo2, u32 k, u32 lane, u32 bufN, int steps)
{
  u32 h[C];
  u32 lo = 0x7f800000u, hi = 0, finite = 0;
#pragma unroll
  for (int c = 0; c < C; ++c)
  {
    h[c] = 0x7f800000u;
    const u32 i = c * 32 + lane;
    if (i < bufN)
    {
      const float v = hi2[i];
      if (v < F0lo2)
      {
        h[c] = __float_as_uint(v);
        lo = min(lo, h[c]);
        if (h[c] < 0x7f800000u)
          hi = max(hi, h[c]);
      }
    }
    finite += __popc(__ballot_sync(~0u, h[c] < 0x7f800000u));
  }
  if (finite < k)
    return kInf;
  lo = __reduce_min_sync(~0u, lo);
  hi = __reduce_max_sync(~0u, hi);
  const float guess = __uint_as_float(hi) * exp2f(log2f(float(k) / float(finite)) * (2.f / 3.f));
  // count(<= hi) >= k throughout
  u32 above = finite;
  for (int s = 0; s < steps && above > k + 1 && lo < hi; ++s)
  {
    u32 mid = lo + ((hi - lo) >> 1);
    if (s < 2)
    {
      const u32 g = __float_as_uint(guess * (s == 0 ? 1.1f : 0.9f));
      mid = g > lo && g < hi ? g : mid;
    }
    u32 n = 0;
#pragma unroll
    for (int c = 0; c < C; ++c)
      n += __popc(__ballot_sync(~0u, h[c] <= mid));
    if (n >= k)
    {
      hi = mid;
      above = n;
    }
    else
      lo = mid + 1;
  }
  return __uint_as_float(hi);
}

// Recomputes the candidate bound from the buffer and drops candidates above it.
template<typename T, int CAP>
__device__ __forceinline__ void knn_flush(KnnWarpMem<CAP>& W, const KnnArgs<T>& a, u32 k, u32 lane, u32& bufN, float& Fc2, int steps)
{
  __syncwarp();
  // round-to-nearest with a 2^-20 margin per step keeps every value an upper bound
  // (the buffer's size picks the count of values per lane: 2 or 4 in most queries)
  const float R2 = bufN <= 64    ? knn_kth_bound<2>(W.hi2, a.F0lo2, k, lane, bufN, steps)
                   : bufN <= 128 ? knn_kth_bound<4>(W.hi2, a.F0lo2, k, lane, bufN, steps)
                                 : knn_kth_bound<CAP / 32>(W.hi2, a.F0lo2, k, lane, bufN, steps);
  const float Rhi = sqrtf(R2) * (1.f + 0x1p-20f);
  const float Fc = fmaxf(a.tolHi, fminf(Rhi, a.F0hi) * a.onePlusTolHi);
  const float nFc2 = (Fc * Fc) * (1.f + 0x1p-20f);
  Fc2 = fminf(Fc2, nFc2);
  const u32 lt = (1u << lane) - 1;
  u32 kept = 0;
  for (u32 base = 0; base < bufN; base += 32)
  {
    const u32 i = base + lane;
    bool keep = false;
    u32 pp = 0;
    float l = 0.f, h = 0.f;
    if (i < bufN)
    {
      pp = W.pos[i];
      l = W.lo2[i];
      h = W.hi2[i];
      keep = l <= Fc2;
    }
    const u32 bal = __ballot_sync(~0u, keep);
    __syncwarp();
    if (keep)
    {
      const u32 s = kept + __popc(bal & lt);
      W.pos[s] = pp;
      W.lo2[s] = l;
      W.hi2[s] = h;
    }
    kept += __popc(bal);
    __syncwarp();
  }
  bufN = kept;
}

// The results of a query that has another number of them than k: the first k to its slot, the rest to the array
// for them. Queries with fewer than k (far from everything, or with a tight max distance) leave the rest of their slot
// unused: in that array they would fill it, and an overflow there costs the whole search again (200k queries of k = 16
// with 4.2 results each 1.46 ms, now 0.71). Out of line, as the kernel is short of registers.
template<typename T>
__device__ __noinline__ void knn_other_count(const KnnArgs<T>& a, const u32* ids, const unsigned long long* key, u32 q, u32 k, u32 m, u32 lane)
{
  u64 start = a.slot ? a.slot[q] : u64(q) * a.kAll;
  for (u32 i = lane; i < min(m, k); i += 32)
  {
    a.slotIds[start + i] = ids[i];
    a.slotDist[start + i] = __longlong_as_double((long long)key[i]);
  }
  if (lane == 0)
    atomicAdd(&a.ctr->irregular, 1u);
  if (m > k)
  {
    unsigned long long s0 = 0;
    if (lane == 0)
      s0 = atomicAdd(&a.ctr->out, (unsigned long long)(m - k));
    s0 = __shfl_sync(~0u, s0, 0);
    if (s0 + (m - k) <= a.outCap)
      for (u32 i = k + lane; i < m; i += 32)
      {
        a.outIds[s0 + (i - k)] = ids[i];
        a.outDist[s0 + (i - k)] = __longlong_as_double((long long)key[i]);
      }
    start = s0 | (u64(kMoreThanK) << 32);
  }
  if (lane == 0)
  {
    a.start[q] = start;
    a.count[q] = m;
  }
}

// 40 warps per SM (48 registers, some spills): 1M queries, k in 1..64, 16M points 6.55 ms; 7.22 at 64 to 80 registers and
// 24 to 32 warps, 7.03 with 48 warps.
template<typename T, int CAP, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 40 / WARPS) knn_filtered_kernel(KnnArgs<T> a)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const u32 lane = threadIdx.x & 31;
  unsigned char* mem = smem + (threadIdx.x >> 5) * knn_warp_bytes<CAP>(a.stackCap);
  KnnWarpMem<CAP>& W = *reinterpret_cast<KnnWarpMem<CAP>*>(mem);
  u32* stackNode = reinterpret_cast<u32*>(mem + sizeof(KnnWarpMem<CAP>));
  float* stackW = reinterpret_cast<float*>(stackNode + a.stackCap);
  const u32 lt = (1u << lane) - 1;
  unsigned long long tests = 0, rechecks = 0;
  for (;;)
  {
    u32 item = 0;
    if (lane == 0)
      item = atomicAdd(&a.ctr->work, 1u);
    item = __shfl_sync(~0u, item, 0);
    if (item >= a.nq)
      break;
    const u32 q = a.order ? a.order[item] : item;
    const u32 k = a.kArr ? a.kArr[q] : a.kAll;
    if (a.evenOffsets && lane == 0)
    {
      a.evenOffsets[q] = u64(q) * k;
      if (q == a.nq - 1)
        a.evenOffsets[a.nq] = u64(a.nq) * k;
    }
    if (k == 0) // ot_query.h:1217-1219: no neighbour requested -> empty result
    {
      if (lane == 0)
      {
        a.count[q] = 0;
        a.start[q] = 0;
      }
      continue;
    }
    if (k > a.kLimit)
    {
      if (lane == 0)
      {
        a.fallback[atomicAdd(&a.ctr->fallbacks, 1u)] = q;
        a.count[q] = 0;
      }
      continue;
    }
    // query: p32 = RN(p) with |p - p32| <= 2^-24 |p32| + 2^-150 <= Sq / 2 (doubled margin);
    // [plo, phi] = p32 -/+ 2 Sq encloses p after its own rounding
    T p[3];
    float plo[3], phi[3], p32[3];
    float ap = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      p[c] = a.pts[u64(q) * 3 + c];
      p32[c] = float(p[c]);
      ap = fmaxf(ap, fabsf(p32[c]));
    }
    float Sq = sizeof(T) == 4 ? 0.f : fmaf(ap, 0x1p-23f, 0x1p-140f);
    if (!(ap < kInf))
    {
      // a query outside the FP32 range: every entity is a candidate
      p32[0] = p32[1] = p32[2] = 0.f;
      Sq = kInf;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      plo[c] = p32[c] - 2.f * Sq;
      phi[c] = p32[c] + 2.f * Sq;
    }
    u32 bufN = 0;
    float Fc2;
    {
      const float Fc = fmaxf(a.tolHi, a.F0hi * a.onePlusTolHi);
      Fc2 = (Fc * Fc) * (1.f + 0x1p-20f);
    }
    u32 flushAt = min(u32(CAP), max(64u, 2 * k + 32));
    bool overflow = false;
    u32 sp = 1;
    if (lane == 0)
    {
      stackNode[0] = 0;
      stackW[0] = node_w2(a.nodeBox32, 0, plo, phi, a.widenLo);
    }
    __syncwarp();
    u32 visits = 0;
    while (sp > 0)
    {
      // The topmost of the last 32 nodes that the bound has not passed since they were pushed. The walk is bound
      // by issue: taking the stack's nodes one by one, and weighing children with two compares each, 6.92 ms for the
      // 1M queries below, now 6.64; keeping the link of the next node at hand instead cost 15% (more registers).
      const u32 open = __ballot_sync(~0u, lane < sp && !(stackW[sp - 1 - lane] > Fc2));
      if (!open)
      {
        sp -= min(sp, 32u);
        continue;
      }
      sp -= u32(__ffs(int(open)));
      const u32 node = stackNode[sp];
      __syncwarp();
      if (++visits > a.nNodes)
      {
        overflow = true;
        break;
      }
      const uint4 L = a.link[node];
      if (L.z > a.n || L.y > L.z || L.w > a.n)
      {
        overflow = true;
        break;
      }
      // A subtree of few points is one run of the tree order: its points are tested as they come, 32 at a
      // time, instead of its nodes (a leaf holds 6 points on average in a tree of 20 per node, its
      // parent about 50: the leaves' tests left four of five lanes idle).
      const bool whole = L.w - L.y <= a.direct;
      const u32 end = whole ? L.w : L.z;
      for (u32 base = L.y; base < end; base += 32)
      {
        if (bufN + 32 > flushAt)
        {
          knn_flush<T, CAP>(W, a, k, lane, bufN, Fc2, 10);
          if (bufN + 32 > flushAt)
          {
            flushAt = CAP;
            if (bufN + 32 > flushAt)
            {
              overflow = true;
              break;
            }
          }
        }
        const u32 e = base + lane;
        float l2 = kInf, h2 = kInf;
        bool keep = false;
        if (e < end)
        {
          entity_bounds(a.geom32[e], p32, Sq, a.widenLo, a.widenHi, l2, h2);
          keep = l2 <= Fc2;
        }
        const u32 bal = __ballot_sync(~0u, keep);
        if (keep)
        {
          const u32 s = bufN + __popc(bal & lt);
          W.pos[s] = e;
          W.lo2[s] = l2;
          W.hi2[s] = h2;
        }
        bufN += __popc(bal);
        tests += min(32u, end - base);
      }
      if (overflow)
        break;
      const u32 fc = L.x & kFirstChildMask, cc = whole ? 0u : L.x >> kChildShift;
      if (cc)
      {
        if (u64(fc) + cc > a.nNodes || cc > 8u || sp + cc > a.stackCap)
        {
          overflow = true;
          break;
        }
        float cw = kInf;
        bool ok = false;
        if (lane < cc)
        {
          cw = node_w2(a.nodeBox32, fc + lane, plo, phi, a.widenLo);
          ok = cw <= Fc2;
        }
        const u32 bal = __ballot_sync(~0u, ok);
        // farthest first: a child's place is the number of open children farther away (ties: the higher lane); the bits
        // of a weight order as it does, with the lane in the lowest three
        const u32 wk = (__float_as_uint(cw) & ~7u) | lane;
        u32 rank = 0;
        for (u32 left = bal; left; left &= left - 1)
          rank += __shfl_sync(~0u, wk, __ffs(int(left)) - 1) > wk;
        if (ok)
        {
          stackNode[sp + rank] = fc + lane;
          stackW[sp + rank] = cw;
        }
        sp += __popc(bal);
        __syncwarp();
      }
    }
    if (!overflow)
      knn_flush<T, CAP>(W, a, k, lane, bufN, Fc2, 26);
    if (overflow)
    {
      if (lane == 0)
      {
        a.fallback[atomicAdd(&a.ctr->fallbacks, 1u)] = q;
        a.count[q] = 0;
      }
      __syncwarp();
      continue;
    }
    // exact distances of the candidates, then (distance, id) order
    for (u32 i = lane; i < bufN; i += 32)
    {
      const u32 e = W.pos[i];
      const T d = GeoD<T>::distance(p, a.geom + u64(e) * 3);
      W.key[i] = (unsigned long long)__double_as_longlong(double(d)); // lo2 and hi2 end here
      W.pos[i] = a.ids[e];
    }
    __syncwarp();
    if (bufN <= 32)
      warp_order_pairs<1>(W.key, W.pos, bufN, lane);
    else if (bufN <= 64)
      warp_order_pairs<2>(W.key, W.pos, bufN, lane);
    else if (bufN <= 128)
      warp_order_pairs<4>(W.key, W.pos, bufN, lane);
    else
    {
      const u32 n2 = pow2_at_least32(bufN);
      for (u32 i = bufN + lane; i < n2; i += 32)
      {
        W.key[i] = ~0ull;
        W.pos[i] = ~0u;
      }
      __syncwarp();
      warp_sort_pairs(W.key, W.pos, n2, lane);
    }
    rechecks += bufN;
    // distances are non-negative: comparing bit patterns as integers orders them like values
    const unsigned long long F0bits = (unsigned long long)__double_as_longlong(double(a.F0));
    u32 below0 = 0;
    for (u32 base = 0; base < bufN; base += 32)
    {
      const u32 i = base + lane;
      below0 += __popc(__ballot_sync(~0u, i < bufN && W.key[i] < F0bits));
    }
    const T F = below0 >= k ? upper_tol(T(__longlong_as_double((long long)W.key[k - 1])), a.tol) : a.F0;
    const unsigned long long Fbits = (unsigned long long)__double_as_longlong(double(F));
    u32 m = 0;
    for (u32 base = 0; base < bufN; base += 32)
    {
      const u32 i = base + lane;
      m += __popc(__ballot_sync(~0u, i < bufN && W.key[i] < Fbits));
    }
    // k results go to the query's slot, which is their place in the result if every query has k
    if (m != k)
      knn_other_count<T>(a, W.pos, W.key, q, k, m, lane);
    else
    {
      const u64 s0 = a.slot ? a.slot[q] : u64(q) * a.kAll;
      for (u32 i = lane; i < m; i += 32)
      {
        a.slotIds[s0 + i] = W.pos[i];
        a.slotDist[s0 + i] = __longlong_as_double((long long)W.key[i]);
      }
      if (lane == 0)
      {
        a.start[q] = s0;
        a.count[q] = m;
      }
    }
    __syncwarp();
  }
  if (lane == 0)
  {
    atomicAdd(&a.ctr->tests, tests);
    atomicAdd(&a.ctr->rechecks, rechecks);
  }
}

// ---------------------------------------------------------------- query order, k statistics
// Morton order of the query points in the tree's space (10 bits per dimension): neighbouring
// queries then walk the same nodes, which keeps the traversal in L2.
template<typename T>
__global__ void query_key_kernel(const T* __restrict__ pts, u64 nq, const Space<T>* __restrict__ sp, u32* __restrict__ keys, u32* __restrict__ idx)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < nq; i += u64(gridDim.x) * blockDim.x)
  {
    u32 c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
      const float ext = float(sp->max[d] - sp->min[d]);
      const float rel = ext > 0.f ? float(pts[i * 3 + d] - sp->min[d]) / ext : 0.f;
      const float v = rel * 1024.f;
      c[d] = v <= 0.f ? 0u : (v >= 1023.f ? 1023u : u32(v));
    }
    keys[i] = u32(encode3(c[0], c[1], c[2]));
    idx[i] = u32(i);
  }
}

__global__ void k_stats_kernel(const u32* __restrict__ k, u64 nq, u32* __restrict__ kmax, unsigned long long* __restrict__ ksum)
{
  u32 mx = 0;
  unsigned long long s = 0;
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < nq; i += u64(gridDim.x) * blockDim.x)
  {
    mx = max(mx, k[i]);
    s += k[i];
  }
  for (int o = 16; o > 0; o >>= 1)
  {
    mx = max(mx, __shfl_xor_sync(~0u, mx, o));
    s += __shfl_xor_sync(~0u, s, o);
  }
  if ((threadIdx.x & 31) == 0)
  {
    atomicMax(kmax, mx);
    atomicAdd(ksum, s);
  }
}

// ---------------------------------------------------------------- CSR assembly

__global__ void fallback_points_kernel(const u32* __restrict__ fb, u32 nfb, const void* __restrict__ pts, u32 ptBytes, const u32* __restrict__ kArr,
                                       u32 kAll, unsigned char* __restrict__ outPts, u32* __restrict__ outK)
{
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < nfb; i += gridDim.x * blockDim.x)
  {
    const u32 q = fb[i];
    const unsigned char* src = static_cast<const unsigned char*>(pts) + u64(q) * ptBytes;
    for (u32 b = 0; b < ptBytes; ++b)
      outPts[u64(i) * ptBytes + b] = src[b];
    outK[i] = kArr ? kArr[q] : kAll;
  }
}

__global__ void fallback_slots_kernel(const u32* __restrict__ fb, u32 nfb, const u64* __restrict__ off, u64* __restrict__ start, u32* __restrict__ count)
{
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < nfb; i += gridDim.x * blockDim.x)
  {
    const u32 q = fb[i];
    start[q] = off[i] | (u64(kFromFallback) << 32);
    count[q] = u32(off[i + 1] - off[i]);
  }
}


__device__ __forceinline__ u64 block_scan_u64(u64 v, u64* warpSums, u64& total)
{
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u64 x = v;
  for (int o = 1; o < 32; o <<= 1)
  {
    const u64 y = __shfl_up_sync(~0u, x, o);
    if (lane >= u32(o))
      x += y;
  }
  if (lane == 31)
    warpSums[w] = x;
  __syncthreads();
  if (w == 0)
  {
    u64 s = lane < kScanThreads / 32 ? warpSums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1)
    {
      const u64 y = __shfl_up_sync(~0u, s, o);
      if (lane >= u32(o))
        s += y;
    }
    if (lane < kScanThreads / 32)
      warpSums[lane] = s;
  }
  __syncthreads();
  total = warpSums[kScanThreads / 32 - 1];
  const u64 before = w ? warpSums[w - 1] : 0;
  __syncthreads();
  return before + x - v; // exclusive
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const u32* __restrict__ cnt, u64 n, u64* __restrict__ tileSums)
{
  __shared__ u64 ws[kScanThreads / 32];
  const u64 base = u64(blockIdx.x) * kScanTile + u64(threadIdx.x) * kScanItems;
  u64 s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)
    if (base + j < n)
      s += cnt[base + j];
  u64 total;
  block_scan_u64(s, ws, total);
  if (threadIdx.x == 0)
    tileSums[blockIdx.x] = total;
}

// one block: exclusive scan of the tile sums in place; tileSums[tiles] = grand total
__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(u64* __restrict__ tileSums, u64 tiles)
{
  __shared__ u64 ws[kScanThreads / 32];
  u64 carry = 0;
  for (u64 base = 0; base < tiles; base += kScanThreads)
  {
    const u64 i = base + threadIdx.x;
    const u64 v = i < tiles ? tileSums[i] : 0;
    u64 total;
    const u64 ex = block_scan_u64(v, ws, total);
    if (i < tiles)
      tileSums[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0)
    tileSums[tiles] = carry;
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const u32* __restrict__ cnt, u64 n, const u64* __restrict__ tileSums, u64* __restrict__ off)
{
  __shared__ u64 ws[kScanThreads / 32];
  const u64 base = u64(blockIdx.x) * kScanTile + u64(threadIdx.x) * kScanItems;
  u32 v[kScanItems];
  u64 s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)
  {
    v[j] = base + j < n ? cnt[base + j] : 0u;
    s += v[j];
  }
  u64 total;
  u64 ex = block_scan_u64(s, ws, total) + tileSums[blockIdx.x];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)
    if (base + j < n)
    {
      off[base + j] = ex;
      ex += v[j];
    }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
    off[n] = tileSums[gridDim.x];
}

// warp per query: copies its entries from where they are (its slot and the results after the first k, or the
// plain kernels' result) to CSR order
__global__ void csr_move_kernel(const u64* __restrict__ start, const u32* __restrict__ count, const u64* __restrict__ off, u64 nq,
                                const u64* __restrict__ slot, const u32* __restrict__ kArr, u32 kAll, const u32* __restrict__ slotIds,
                                const double* __restrict__ slotDist, const u32* __restrict__ ids, const double* __restrict__ dist,
                                const u32* __restrict__ fbIds, const double* __restrict__ fbDist, u32* __restrict__ outIds, double* __restrict__ outDist)
{
  const u32 lane = threadIdx.x & 31;
  for (u64 q = (blockIdx.x * u64(blockDim.x) + threadIdx.x) >> 5; q < nq; q += (u64(gridDim.x) * blockDim.x) >> 5)
  {
    const u32 c = count[q];
    if (!c)
      continue;
    const u64 s = start[q], d = off[q];
    const u32 from = u32(s >> 32) & (kFromFallback | kMoreThanK);
    const u64 at = s & ~(u64(kFromFallback | kMoreThanK) << 32);
    const bool more = from == kMoreThanK;
    const u64 src = more ? (slot ? slot[q] : q * kAll) : at;
    const u32 k = more ? (kArr ? kArr[q] : kAll) : c;
    const u32* si = from == kFromFallback ? fbIds : slotIds;
    const double* sd = from == kFromFallback ? fbDist : slotDist;
    for (u32 i = lane; i < c; i += 32)
    {
      outIds[d + i] = i < k ? si[src + i] : ids[at + (i - k)];
      outDist[d + i] = i < k ? sd[src + i] : dist[at + (i - k)];
    }
  }
}

// ---------------------------------------------------------------- host
static void host_bounds(double v, float& lo, float& hi)
{
  float f = float(v);
  lo = f;
  hi = f;
  if (double(f) > v)
    lo = std::nextafter(f, -kInf);
  if (double(f) < v)
    hi = std::nextafter(f, kInf);
}

// box entities rounded outward: {min rounded down, 0}, {max rounded up, 0}
template<typename T>
__global__ void entity_box_image_kernel(const T* __restrict__ geom, u64 n, float4* __restrict__ out)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < n; i += u64(gridDim.x) * blockDim.x)
  {
    float v[6];
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      v[c] = __double2float_rd(double(geom[i * 6 + c]));
      v[3 + c] = __double2float_ru(double(geom[i * 6 + 3 + c]));
    }
    out[2 * i] = make_float4(v[0], v[1], v[2], 0.f);
    out[2 * i + 1] = make_float4(v[3], v[4], v[5], 0.f);
  }
}

template<typename T>
static int ensure_image32_impl(TreeState& t, cudaStream_t st, bool boxes)
{
  const bool isBox = t.kind != OTG_KIND_POINTS;
  boxes = boxes && isBox;
  std::lock_guard<std::mutex> g(t.imageMutex);
  cudaError_t e;
  const bool build = !t.image32 || (boxes && !t.boxImage32);
  // the stream that builds orders itself after the streams that built or use the earlier images
  if (t.imageReady && (e = cudaStreamWaitEvent(st, t.imageReady, 0)))
    return cuda_status(e, "waiting for the FP32 tree image");
  if (!build)
    return OTG_OK;
  if (!t.imageReady && (e = cudaEventCreateWithFlags(&t.imageReady, cudaEventDisableTiming)))
    return cuda_status(e, "creating the image event");
  if (!t.image32)
  {
    if ((!isBox && (e = t.geom32.ensure(sizeof(float4) * std::max<u64>(t.n, 1)))) || (e = t.nodeBox32.ensure(sizeof(float4) * 2 * std::max<u64>(t.nodeCount, 1))))
      return cuda_status(e, "allocating the FP32 tree image");
    if (!isBox && t.n)
      point_image_kernel<T><<<blocks_for(t.n), 256, 0, st>>>(t.sortedGeom.as<T>(), t.n, t.geom32.as<float4>());
    node_image_kernel<T><<<blocks_for(t.nodeCount), 256, 0, st>>>(t.nodeBox.as<T>(), isBox ? t.nodeMax.as<T>() : nullptr, t.nodeCount,
                                                                   t.nodeBox32.as<float4>());
  }
  if (boxes && !t.boxImage32)
  {
    if ((e = t.boxImg32.ensure(sizeof(float4) * 2 * std::max<u64>(t.n, 1))))
      return cuda_status(e, "allocating the FP32 box image");
    if (t.n)
      entity_box_image_kernel<T><<<blocks_for(t.n), 256, 0, st>>>(t.sortedGeom.as<T>(), t.n, t.boxImg32.as<float4>());
  }
  if ((e = cudaGetLastError()) || (e = cudaEventRecord(t.imageReady, st)))
    return cuda_status(e, "building the FP32 tree image");
  t.image32 = true;
  t.boxImage32 = t.boxImage32 || boxes;
  return OTG_OK;
}

template<typename T, int CAP, int WARPS>
static int launch_filtered_w(const KnnArgs<T>& a, cudaStream_t st)
{
  const size_t smem = knn_warp_bytes<CAP>(a.stackCap) * WARPS;
  cudaError_t e = cudaFuncSetAttribute(knn_filtered_kernel<T, CAP, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  int dev = 0, sms = 0, per = 0;
  if (!e)
    e = cudaGetDevice(&dev);
  if (!e)
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!e)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, knn_filtered_kernel<T, CAP, WARPS>, WARPS * 32, smem);
  if (e)
    return cuda_status(e, "configuring the kNN kernel");
  const u64 want = (u64(a.nq) + WARPS - 1) / WARPS;
  const u32 grid = u32(std::max<u64>(1, std::min<u64>(u64(sms) * std::max(per, 1), want)));
  knn_filtered_kernel<T, CAP, WARPS><<<grid, WARPS * 32, smem, st>>>(a);
  return cuda_status(cudaGetLastError(), "launching the kNN kernel");
}

// Subtrees of at most this many points are tested without their nodes. 1M queries, k in 1..64, on 16M points
// of 20 per node (whole call): 10.7 ms at 0 and 16, 10.4 at 32, 8.2 at 48, 7.5 at 64, 7.2 at 96, 7.1 at 128; 10k queries of
// k = 8 on 1M points: 0.152, 0.155, 0.137, 0.120, 0.118, 0.117, 0.118 ms. Above 96 the points tested in vain
// take what the nodes cost.
constexpr u32 kDirectPoints = 96;

// shape: warps per block (2, 4 or 8)
template<typename T, int CAP>
static int launch_filtered(const KnnArgs<T>& a, int shape, cudaStream_t st)
{
  if (shape == 2)
    return launch_filtered_w<T, CAP, 2>(a, st);
  if (shape == 8)
    return launch_filtered_w<T, CAP, 8>(a, st);
  return launch_filtered_w<T, CAP, 4>(a, st);
}

template<typename T>
static int knn_filtered_impl(TreeState& t, const T* pts, const u32* dk, u64 nq, u32 kAll, double maxDist, double tol, ResultState& r, cudaStream_t st)
{
  cudaError_t e;
  if (int rc = ensure_image32(t, st))
    return rc;
  const T tl = tol_of<T>(tol);
  const T F0 = maxDist < 0 ? Lim<T>::max() : upper_tol_host(T(maxDist), tl);
  // k statistics: the buffer size follows the largest k, the output guess the sum of k
  u32 kmax = kAll;
  u64 ksum = u64(kAll) * nq;
  TmpBuf stats;
  if (dk)
  {
    if ((e = stats.ensure(16, st)))
      return cuda_status(e, "allocating k statistics");
    cudaMemsetAsync(stats.p, 0, 16, st);
    k_stats_kernel<<<blocks_for(nq), 256, 0, st>>>(dk, nq, stats.as<u32>(), reinterpret_cast<unsigned long long*>(stats.as<unsigned char>() + 8));
    unsigned long long h[2] = { 0, 0 };
    if ((e = read_back(h, stats.p, 16, st)))
      return cuda_status(e, "reading k statistics");
    kmax = u32(h[0]);
    ksum = h[1];
  }
  const bool big = kmax > 112;
  // spatial order of the queries
  TmpBuf qkeys, order;
  // below 64k queries the batch takes the queries in input order: four radix passes over a few
  // tiles cost more than the locality gains, the tree's upper levels sitting in L2 anyway
  const bool sortQueries = nq >= (u64(1) << 16);
  if (sortQueries)
  {
    if ((e = qkeys.ensure(sizeof(u32) * nq, st)) || (e = order.ensure(sizeof(u32) * nq, st)))
      return cuda_status(e, "allocating the query order");
    query_key_kernel<T><<<blocks_for(nq), 256, 0, st>>>(pts, nq, t.space.as<Space<T>>(), qkeys.as<u32>(), order.as<u32>());
  }
  // one block: the counters, the queries' starts and counts, the list of fallbacks
  TmpBuf perQuery, irregular;
  if ((e = perQuery.ensure(64 + (sizeof(u64) + 2 * sizeof(u32)) * nq, st)))
    return cuda_status(e, "allocating kNN buffers");
  static_assert(sizeof(KnnCounters) <= 64, "the starts follow the counters");
  KnnCounters* ctr = perQuery.as<KnnCounters>();
  u64* start = reinterpret_cast<u64*>(perQuery.as<unsigned char>() + 64);
  u32* cnt = reinterpret_cast<u32*>(start + nq);
  u32* fb = cnt + nq;
  if (sortQueries)
  {
    cudaMemsetAsync(ctr, 0, sizeof(KnnCounters), st); // (the sort's error bits)
    if (int rc = sort_pairs_u32(qkeys.as<u32>(), order.as<u32>(), nq, 30, st, &ctr->err))
      return rc;
  }
  qkeys.release();
  KnnArgs<T> a{};
  a.link = t.nodeLink.as<uint4>();
  a.nodeBox32 = t.nodeBox32.as<float4>();
  a.geom32 = t.geom32.as<float4>();
  a.geom = t.sortedGeom.as<T>();
  a.ids = t.sortedIds.as<u32>();
  a.n = u32(t.n);
  a.nNodes = u32(t.nodeCount);
  a.pts = pts;
  a.kArr = dk;
  a.kAll = kAll;
  a.nq = u32(nq);
  a.order = sortQueries ? order.as<u32>() : nullptr;
  a.F0 = F0;
  a.tol = tl;
  float lo, hi;
  host_bounds(double(F0), lo, hi);
  a.F0hi = hi;
  {
    float l2, h2;
    host_bounds(double(lo) * double(lo), l2, h2);
    a.F0lo2 = l2;
  }
  host_bounds(double(tl), lo, hi);
  a.tolHi = hi;
  host_bounds(double(T(T(1) + tl)), lo, hi);
  host_bounds(double(hi) * (1.0 + 0x1p-20), lo, hi); // margin for the rounding of one product
  a.onePlusTolHi = hi;
  // relative margins that cover the rounding of the exact distance formula
  a.widenLo = sizeof(T) == 8 ? 1.f - 0x1p-18f : 1.f - 0x1p-16f;
  a.widenHi = sizeof(T) == 8 ? 1.f + 0x1p-18f : 1.f + 0x1p-16f;
  a.kLimit = big ? 240u : 112u;
  a.ctr = ctr;
  a.fallback = fb;
  a.start = start;
  a.count = cnt;
  a.direct = t.respanned ? 0u : kDirectPoints; // (points may lie outside their nodes)
  a.stackCap = (7 * (t.D + 1) + 9 + 3) & ~3u; // depth first: at most 7 entries per level beside the current node's 8 children
  // a slot of k per query: the result itself if every query has k (no ties within the tolerance, enough
  // points in reach); then nothing is moved and the call waits for the GPU once
  const u64 tiles = (nq + kScanTile - 1) / kScanTile;
  TmpBuf tileSums;
  if ((dk && (e = tileSums.ensure(sizeof(u64) * (tiles + 1), st))) ||
      (e = result_alloc(r, sizeof(u64) * (nq + 1), sizeof(u32) * std::max<u64>(ksum, 1), sizeof(double) * std::max<u64>(ksum, 1), st)))
    return cuda_status(e, "allocating the kNN result");
  if (dk)
  {
    scan_reduce_kernel<<<u32(tiles), kScanThreads, 0, st>>>(dk, nq, tileSums.as<u64>());
    scan_tiles_kernel<<<1, kScanThreads, 0, st>>>(tileSums.as<u64>(), tiles);
    scan_apply_kernel<<<u32(tiles), kScanThreads, 0, st>>>(dk, nq, tileSums.as<u64>(), r.offsets.as<u64>());
    a.slot = r.offsets.as<u64>();
  }
  else
    a.evenOffsets = r.offsets.as<u64>(); // written by the search
  a.slotIds = r.ids.as<u32>();
  a.slotDist = r.dist.as<double>();
  u64 cap = ksum / 8 + 4096;
  KnnCounters h{};
  for (int attempt = 0; attempt < 2; ++attempt)
  {
    if ((e = irregular.ensure((sizeof(u32) + sizeof(double)) * cap, st)))
      return cuda_status(e, "allocating the kNN output");
    a.outDist = irregular.as<double>();
    a.outIds = reinterpret_cast<u32*>(a.outDist + cap);
    a.outCap = cap;
    int rc = tune_run(tune_key("knn", sizeof(T) == 8, int(t.kind), t.n, nq), { { 2, "warp x2" }, { 4, "warp x4" }, { 8, "warp x8" } }, 4, st,
                      [&](int shape) {
                        // (keeps the sort's error bits, the last word)
                        cudaMemsetAsync(ctr, 0, sortQueries ? offsetof(KnnCounters, err) : sizeof(KnnCounters), st);
                        return big ? launch_filtered<T, 512>(a, shape, st) : launch_filtered<T, 256>(a, shape, st);
                      });
    if (rc)
      return rc;
    if ((e = read_back(&h, ctr, sizeof(h), st)))
      return cuda_status(e, "running the kNN kernel");
    if (h.out <= cap)
      break;
    cap = h.out + h.out / 16 + 4096;
  }
  if (h.err & kErrTimeout)
  {
    set_error("a bounded device wait ran out");
    return OTG_ERR_TIMEOUT;
  }
  if (h.out > cap)
  {
    set_error("kNN output sizing did not converge");
    return OTG_ERR_OUT_OF_MEMORY;
  }
  r.nq = nq;
  r.nids = ksum;
  r.hasDist = true;
  r.filterTests = h.tests;
  r.rechecks = h.rechecks;
  if (h.irregular == 0 && h.fallbacks == 0)
    return OTG_OK;
  // queries the filter handed over to the plain kernels
  ResultState fbr;
  if (h.fallbacks)
  {
    TmpBuf fpts, fk;
    if ((e = fpts.ensure(sizeof(T) * 3 * h.fallbacks, st)) || (e = fk.ensure(sizeof(u32) * h.fallbacks, st)))
      return cuda_status(e, "allocating fallback queries");
    fallback_points_kernel<<<blocks_for(h.fallbacks), 256, 0, st>>>(fb, h.fallbacks, pts, u32(sizeof(T) * 3), dk, kAll,
                                                                   fpts.as<unsigned char>(), fk.as<u32>());
    if (int rc = query_knn(t, fpts.p, h.fallbacks, fk.as<u32>(), 0, maxDist, tol, OTG_ALGO_PLAIN_FP64, fbr, OTG_MEM_DEVICE, st))
      return rc;
    fallback_slots_kernel<<<blocks_for(h.fallbacks), 256, 0, st>>>(fb, h.fallbacks, fbr.offsets.as<u64>(), start, cnt);
  }
  // CSR: offsets by scan of the counts, then entries moved into query order
  u64 total = 0;
  if ((e = tileSums.ensure(sizeof(u64) * (tiles + 1), st)))
    return cuda_status(e, "allocating the kNN result");
  scan_reduce_kernel<<<u32(tiles), kScanThreads, 0, st>>>(cnt, nq, tileSums.as<u64>());
  scan_tiles_kernel<<<1, kScanThreads, 0, st>>>(tileSums.as<u64>(), tiles);
  if ((e = read_back(&total, tileSums.as<u64>() + tiles, sizeof(u64), st)))
    return cuda_status(e, "counting the kNN result");
  ResultState moved;
  if ((e = result_alloc(moved, sizeof(u64) * (nq + 1), sizeof(u32) * std::max<u64>(total, 1), sizeof(double) * std::max<u64>(total, 1), st)))
    return cuda_status(e, "allocating the result");
  scan_apply_kernel<<<u32(tiles), kScanThreads, 0, st>>>(cnt, nq, tileSums.as<u64>(), moved.offsets.as<u64>());
  csr_move_kernel<<<blocks_for(nq * 32), 256, 0, st>>>(start, cnt, moved.offsets.as<u64>(), nq, a.slot, dk, kAll, r.ids.as<u32>(), r.dist.as<double>(),
                                                        a.outIds, a.outDist, fbr.ids.as<u32>(), fbr.dist.as<double>(), moved.ids.as<u32>(),
                                                        moved.dist.as<double>());
  std::swap(r.offsets.p, moved.offsets.p);
  std::swap(r.offsets.bytes, moved.offsets.bytes);
  std::swap(r.ids.p, moved.ids.p);
  std::swap(r.ids.bytes, moved.ids.bytes);
  std::swap(r.dist.p, moved.dist.p);
  std::swap(r.dist.bytes, moved.dist.bytes);
  r.nids = total;
  e = cudaStreamSynchronize(st);
  if (e || (e = cudaGetLastError()))
    return cuda_status(e, "assembling the kNN result");
  return OTG_OK;
}

int ensure_image32(TreeState& t, cudaStream_t st, bool boxes)
{
  return t.scalar == OTG_SCALAR_F64 ? ensure_image32_impl<double>(t, st, boxes) : ensure_image32_impl<float>(t, st, boxes);
}

int use_images(TreeState& t, TreeView<double>& tv, u64 tests, cudaStream_t st)
{
  const bool isBox = t.kind != OTG_KIND_POINTS;
  {
    // building the images moves 80 bytes of every box (40 of a point) and a test that they spare reads 48
    // and takes some 30 FP64 operations: worth it from about one test per entity on, so that a tree
    // rebuilt for a few queries does not pay for them (1M boxes built anew, then 2000, 4000, 8000 and 64000 ranges of 128
    // estimated tests: 114, 143, 213 and 1070 us by exact tests, 114, 127, 142 and 310 with the images built by the call)
    std::lock_guard<std::mutex> g(t.imageMutex);
    t.imageTests += tests;
    if (!(isBox ? t.boxImage32 : t.image32) && t.imageTests < t.n)
      return OTG_OK;
  }
  if (int rc = ensure_image32(t, st, isBox))
    return rc == OTG_ERR_OUT_OF_MEMORY ? OTG_OK : rc; // without room for them the exact tests answer as they are
  tv.nodeImg = t.nodeBox32.as<float4>();
  if (isBox)
    tv.boxImg = t.boxImg32.as<float4>();
  else
    tv.pointImg = t.geom32.as<float4>();
  return OTG_OK;
}

int knn_filtered(TreeState& t, const void* dpts, const u32* dk, u64 nq, u32 kAll, double maxDist, double tol, ResultState& r, cudaStream_t st)
{
  return t.scalar == OTG_SCALAR_F64 ? knn_filtered_impl<double>(t, (const double*)dpts, dk, nq, kAll, maxDist, tol, r, st)
                                    : knn_filtered_impl<float>(t, (const float*)dpts, dk, nq, kAll, maxDist, tol, r, st);
}

} // namespace otg
