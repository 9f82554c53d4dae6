// otg_batch.cu — batched RangeSearch, FrustumCulling, RayIntersectedAll, PlaneSearch and
// PlanePositiveSegmentation: persistent kernels in
// which each warp takes the next query from a shared counter (queries of uneven cost balance out,
// in one tree or across the trees of a forest) and answers it cooperatively:
//   * the node's own entities are tested by the 32 lanes in parallel (coalesced reads of the
//     tree-ordered geometry), hits compacted with a ballot into a per-warp shared buffer that is
//     flushed to the result with one atomic per flush;
//   * the node's children are tested by one lane each before they are pushed, so the depth-first
//     stack (in shared memory) only ever holds nodes the query enters.
// Every node and entity test is the reference predicate in the tree's scalar type, applied to the
// same nodes as the one-query-per-thread kernels of otg_query.cu, so the id sets are identical:
//   RangeSearch         core/ot_query.h:476-583
//   FrustumCulling      core/ot_query.h:767-833
//   RayIntersectedAll   core/ot_query.h:1928-2022
//   PlaneSearch         core/ot_query.h:612-636
//   PlanePositiveSegmentation core/ot_query.h:687-744
//   Query<And / Or>     core/ot_query.h:864-1026
//   PickSearch          core/ot_query.h:425-466
#include "otg_query.cuh"
#include "otg_ray.cuh"

namespace otg
{

constexpr u32 kItemBuf = 128;
constexpr u32 kContained = 1u << 31; // stack entry flag: the range contains the node (emit its subtree)
// Per-warp node stack. A step pops up to 32 nodes and pushes at most 8 children each, so it runs
// only while that cannot pass kWideStack - kWideReserve; beyond, one node per step (depth first)
// adds at most 7 entries per level over at most 19 levels.
constexpr int kWideStack = 768;
constexpr int kWideReserve = 160;

struct WarpSink
{
  u64* items;
  double* dist;
  u32 n;
};

// flushes the warp's buffered results to the appender (all lanes)
__device__ __forceinline__ void sink_flush(WarpSink& s, Appender& out, u32 lane)
{
  if (s.n == 0)
    return;
  unsigned long long base = 0;
  if (lane == 0)
    base = out.reserve(s.n);
  base = __shfl_sync(~0u, base, 0);
  for (u32 t = lane; t < s.n; t += 32)
    if (base + t < out.capacity)
    {
      out.items[base + t] = s.items[t];
      if (out.dist)
        out.dist[base + t] = s.dist[t];
    }
  __syncwarp();
  s.n = 0;
}

// appends the lanes with hit set (all lanes call)
__device__ __forceinline__ void sink_put(WarpSink& s, Appender& out, u32 lane, bool hit, u32 q, u32 id, double d)
{
  const u32 bal = __ballot_sync(~0u, hit);
  if (!bal)
    return;
  if (s.n + 32 > kItemBuf)
    sink_flush(s, out, lane);
  if (hit)
  {
    const u32 slot = s.n + __popc(bal & ((1u << lane) - 1));
    s.items[slot] = (u64(q) << 32) | id;
    if (out.dist)
      s.dist[slot] = d;
  }
  s.n += __popc(bal);
  __syncwarp();
}

// query kinds
constexpr int kRange = 0, kFrustum = 1, kRayAll = 2, kPlane = 3, kPlanePositive = 4, kQuery = 5, kPick = 6;

// ---- FP32 pre-tests of RangeSearch on FP64 point trees
// The FP64 tests (core/ot_query.h:476-583 with internal_geometry_module.h:190-252, :398-422):
//   node pruned  : some d with  maxL <= RN(nmin - tol)  or  maxR <= P        (overlap_by_min_point)
//   node inside  : every d with P <= nmin and maxR <= Q                      (range_contains_min_size)
//   point inside : every d with P < x < Q (tol != 0), or rmin <= x <= rmax (tol == 0)
// with P = RN(rmin - tol), Q = RN(rmax + tol), maxL = RN(rmin + RN(rmax - rmin)) per query and
// maxR = RN(nmin + nsize) per node. The images bound the FP64 values: a node's image holds
// lo = rd(nmin) and hi = ru(maxR), so nmin lies in [lo, succ(lo)) and maxR in (pred(hi), hi]; a
// point's image holds x32 = RN32(x), so x lies in (pred(x32), succ(x32)). Because floats are
// discrete, "succ(a) <= b" is "a < b" and "pred(a) >= b" is "a > b" for floats a, b, and each test
// below is decided where these bounds settle it, with per-query thresholds rounded down (lo) and up
// (hi) from the exact FP64 values:
//   P < x  : true if x32 > P.hi, false if x32 < P.lo      x < Q  : true if x32 < Q.lo, false if x32 > Q.hi
//   (the same for rmin <= x and x <= rmax with P = rmin, Q = rmax when tol == 0)
//   maxR <= P : true if hi <= P.lo, false if hi > P.hi   maxR <= Q : true if hi <= Q.lo, false if hi > Q.hi
//   P <= nmin : true if P.hi <= lo, false if lo < P.lo
//   maxL <= RN(nmin - tol) : true if ru(W + g) <= lo, false if lo < rd(W - g), W = RN(maxL + tol),
//     where the slack g = 2^-46 (M + tol) exceeds every FP64 rounding involved (M bounds the range's
//     and the root box's coordinates, so also every node's). RN is monotone, so maxL + tol <= nmin
//     gives maxL <= RN(nmin - tol); and nmin + g/2 < maxL + tol gives RN(nmin - tol) < maxL.
// Undecided tests run in FP64, so every answer is the FP64 answer.
//
// Box trees. A node's image holds the exact MBR max where the tests use maxR = RN(nmin + nsize), within the
// slack g of it: their P and Q thresholds are widened by g. An entity's image holds lo = rd(bmin) and
// hi = ru(bmax), so bmin lies in [lo, succ(lo)) and bmax in (pred(hi), hi], and its test is decided by four
// thresholds per dimension (e0 .. e3, boxes that lie in the root box, tol >= 0):
//   inside (rmin <= bmin, bmax <= rmax and both on the other side too, contains_box_no_tol), with
//     e0 = rd(rmin), e1 = ru(rmin), e2 = rd(rmax), e3 = ru(rmax):
//     in  if e1 <= lo < e2 and e1 < hi <= e2 in every dimension; out if lo or hi < e0 or > e3 in some dimension
//   overlap (GetBoxRelation == Overlapped), with e0 = rd(rmin - tol - g), e1 = ru(rmin + tol),
//     e2 = rd(rmax - tol - g), e3 = ru(rmax + tol + g):
//     in  if hi > e1 and lo < e2 in every dimension (its "overlapped" branch); out if hi < e0 or lo > e3 in some
//     dimension (then "separated" or "adjacent")
struct RangeF32
{
  float w[3], s[3], plo[3], phi[3], qlo[3], qhi[3];
  float e0[3], e1[3], e2[3], e3[3]; // box entities
};

__device__ __forceinline__ void range_thresholds(const double* r, const double* rsize, const double* rootBox, double tol, bool isBox, int mode, RangeF32& f)
{
  double M = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    M = fmax(M, fmax(fabs(r[d]), fabs(r[3 + d])));
    M = fmax(M, fmax(fabs(rootBox[d]), fabs(rootBox[d] + rootBox[3 + d])));
  }
  const double g = (M + fabs(tol)) * 0x1p-46;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    const double maxL = r[d] + rsize[d];
    const double P = r[d] - tol, Q = r[3 + d] + tol;
    const double W = maxL + tol;
    f.w[d] = __double2float_ru(W + g);
    f.s[d] = __double2float_rd(W - g);
    const double wide = isBox ? g : 0.0;
    f.plo[d] = __double2float_rd(P - wide);
    f.phi[d] = __double2float_ru(P + wide);
    f.qlo[d] = __double2float_rd(Q - wide);
    f.qhi[d] = __double2float_ru(Q + wide);
    const bool over = mode == OTG_RANGE_OVERLAP;
    f.e0[d] = __double2float_rd(over ? r[d] - tol - g : r[d]);
    f.e1[d] = __double2float_ru(over ? r[d] + tol : r[d]);
    f.e2[d] = __double2float_rd(over ? r[3 + d] - tol - g : r[3 + d]);
    f.e3[d] = __double2float_ru(over ? r[3 + d] + tol + g : r[3 + d]);
  }
}

// The FP64 tests of the undecided cases, out of line: inlined, the compiler may evaluate them for
// every node and point beside the FP32 tests (predicated), which kept the FP64 pipe busy.
// the query's range as the caller passed it (6 doubles), and its size
__device__ __forceinline__ void range_load(const double* q, double r[6], double rsize[3])
{
#pragma unroll
  for (int c = 0; c < 6; ++c)
    r[c] = q[c];
#pragma unroll
  for (int c = 0; c < 3; ++c)
    rsize[c] = r[3 + c] - r[c];
}
__device__ __noinline__ bool range_node_enters_fp64(const double* q, const double* nb, double tol)
{
  double r[6], rsize[3];
  range_load(q, r, rsize);
  return GeoD<double>::overlap_by_min_point(r, rsize, nb, nb + 3, tol);
}
__device__ __noinline__ bool range_node_inside_fp64(const double* q, const double* nb, double tol)
{
  double r[6], rsize[3];
  range_load(q, r, rsize);
  return GeoD<double>::range_contains_min_size(r, nb, nb + 3, tol);
}
__device__ __noinline__ bool range_point_inside_fp64(const double* q, const double* p, double tol)
{
  double r[6], rsize[3];
  range_load(q, r, rsize);
  return GeoD<double>::box_contains_point(r, p, tol);
}

// One query's FP64 setup, done beforehand by one thread per query (an FP64 instruction of a warp
// occupies this GPU's FP64 pipe for many cycles, so a warp doing one query's setup costs 32 times as
// much): the FP32 thresholds, and the flags of the root shortcut and of an empty range.
constexpr u32 kRangeAll = 1u, kRangeEmpty = 2u;
struct RangeQ
{
  RangeF32 f;
  u32 flags, pad;
};
constexpr u32 kRangeWords = 30; // of the thresholds
static_assert(sizeof(RangeQ) == 128, "RangeQ: 32 words");

__global__ void __launch_bounds__(128) range_prepare_kernel(TreeView<double> tv, const double* __restrict__ ranges, u32 nq, int mode, double tol,
                                                            RangeQ* __restrict__ out)
{
  using G = GeoD<double>;
  for (u32 q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x)
  {
    const u32 root = query_root(tv, q);
    double r[6], rsize[3], rb[6];
    range_load(ranges + u64(q) * 6, r, rsize);
    const double* nb = tv.nodeBox + u64(root) * 6;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      rb[c] = nb[c];
      rb[3 + c] = nb[c] + nb[3 + c];
    }
    RangeQ o;
    o.flags = G::range_contains_box(r, rb, tol) ? kRangeAll : 0u; // root shortcut (:488-511)
    double vol = 1.0;                                             // zero-volume range -> empty (:514-519)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      vol *= rsize[c];
    if (vol <= 0.0)
      o.flags |= kRangeEmpty;
    range_thresholds(r, rsize, nb, tol, tv.isBox != 0, mode, o.f);
    o.pad = 0;
    out[q] = o;
  }
}

// node: enter 0 (pruned) / 1 (entered) / 2 (undecided); inside 0 / 1 / 2 likewise
__device__ __forceinline__ void range_node_f32(const float4* __restrict__ img, u32 node, const RangeF32& f, int& enter, int& inside)
{
  const float4 mn = img[2 * size_t(node)], mx = img[2 * size_t(node) + 1];
  const float lo[3] = { mn.x, mn.y, mn.z }, hi[3] = { mx.x, mx.y, mx.z };
  bool anyPrune = false, allKeep = true, allIn = true, anyOut = false;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    anyPrune |= (f.w[d] <= lo[d]) | (hi[d] <= f.plo[d]);
    allKeep &= (lo[d] < f.s[d]) & (hi[d] > f.phi[d]);
    allIn &= (f.phi[d] <= lo[d]) & (hi[d] <= f.qlo[d]);
    anyOut |= (lo[d] < f.plo[d]) | (hi[d] > f.qhi[d]);
  }
  enter = anyPrune ? 0 : (allKeep ? 1 : 2);
  inside = anyOut ? 0 : (allIn ? 1 : 2);
}

// box entity: 0 out, 1 in, 2 undecided
__device__ __forceinline__ int range_box_f32(const float4* __restrict__ img, u32 e, const RangeF32& f, bool over)
{
  const float4 mn = img[2 * size_t(e)], mx = img[2 * size_t(e) + 1];
  const float lo[3] = { mn.x, mn.y, mn.z }, hi[3] = { mx.x, mx.y, mx.z };
  bool allIn = true, anyOut = false;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    if (over)
    {
      allIn &= (hi[d] > f.e1[d]) & (lo[d] < f.e2[d]);
      anyOut |= (hi[d] < f.e0[d]) | (lo[d] > f.e3[d]);
    }
    else
    {
      allIn &= (f.e1[d] <= lo[d]) & (lo[d] < f.e2[d]) & (f.e1[d] < hi[d]) & (hi[d] <= f.e2[d]);
      anyOut |= (lo[d] < f.e0[d]) | (hi[d] < f.e0[d]) | (lo[d] > f.e3[d]) | (hi[d] > f.e3[d]);
    }
  }
  return anyOut ? 0 : (allIn ? 1 : 2);
}
__device__ __noinline__ bool range_box_fp64(const double* q, const double* box, int mode, double tol)
{
  double r[6], rsize[3], b[6];
  range_load(q, r, rsize);
  load_box(box, b);
  return mode == OTG_RANGE_OVERLAP ? GeoD<double>::box_relation(r, b, tol) == -1 : GeoD<double>::contains_box_no_tol(r, b);
}

// ---- FP32 pre-tests of PickSearch on FP64 trees. A node or box holds the point p if
// min - tol < p < max + tol in every dimension (node_contains_point compares |p - min - half| with half + tol,
// box_contains_point the two sides; with tol = 0 the sides belong to it), up to roundings far below
// g = 2^-46 (M + tol), M bounding the point's and the root box's coordinates:
//   in  if lo < rd(p + tol - g) and hi > ru(p - tol + g) in every dimension
//   out if lo > ru(p + tol + g) or hi < rd(p - tol - g) in some dimension
// A point entity equals p within tol only if it is not out (lo = hi = its image, RN).
struct PickF32
{
  float inLo[3], inHi[3], outLo[3], outHi[3];
};
struct PickQ
{
  PickF32 f;
  u32 skip, pad[3]; // skip: outside the tree's box (:430-431)
};
static_assert(sizeof(PickQ) == 64, "PickQ: 16 words");

__global__ void __launch_bounds__(128) pick_prepare_kernel(TreeView<double> tv, const double* __restrict__ pts, u32 nq, double tol, PickQ* __restrict__ out)
{
  for (u32 q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x)
  {
    const double* nb = tv.nodeBox + u64(query_root(tv, q)) * 6;
    double rb[6], p[3];
    double M = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      rb[c] = nb[c];
      rb[3 + c] = nb[c] + nb[3 + c];
      p[c] = pts[u64(q) * 3 + c];
      M = fmax(M, fmax(fabs(p[c]), fmax(fabs(rb[c]), fabs(rb[3 + c]))));
    }
    const double g = (M + fabs(tol)) * 0x1p-46;
    PickQ o;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      o.f.inLo[c] = __double2float_rd(p[c] + tol - g);
      o.f.inHi[c] = __double2float_ru(p[c] - tol + g);
      o.f.outLo[c] = __double2float_ru(p[c] + tol + g);
      o.f.outHi[c] = __double2float_rd(p[c] - tol - g);
    }
    o.skip = GeoD<double>::box_contains_point(rb, p, tol) ? 0u : 1u;
    o.pad[0] = o.pad[1] = o.pad[2] = 0;
    out[q] = o;
  }
}
// 0 out, 1 in, 2 undecided
__device__ __forceinline__ int pick_f32(float4 mn, float4 mx, const PickF32& f)
{
  const float lo[3] = { mn.x, mn.y, mn.z }, hi[3] = { mx.x, mx.y, mx.z };
  bool allIn = true, anyOut = false;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    allIn &= (lo[d] < f.inLo[d]) & (hi[d] > f.inHi[d]);
    anyOut |= (lo[d] > f.outLo[d]) | (hi[d] < f.outHi[d]);
  }
  return anyOut ? 0 : (allIn ? 1 : 2);
}
__device__ __noinline__ bool pick_node_fp64(const double* nb, const double* p, double tol) { return GeoD<double>::node_contains_point(nb, nb + 3, p, tol); }
__device__ __noinline__ bool pick_entity_fp64(const double* g, int isBox, const double* p, double tol)
{
  return isBox ? GeoD<double>::box_contains_point(g, p, tol) : GeoD<double>::points_equal(g, p, tol);
}

// point: 0 outside, 1 inside, 2 undecided (also for a point without a finite image)
__device__ __forceinline__ int range_point_f32(const float4 p, const RangeF32& f)
{
  if (!(p.w < INFINITY))
    return 2;
  const float x[3] = { p.x, p.y, p.z };
  bool allIn = true, anyOut = false;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    allIn &= (x[d] > f.phi[d]) & (x[d] < f.qlo[d]);
    anyOut |= (x[d] < f.plo[d]) | (x[d] > f.qhi[d]);
  }
  return anyOut ? 0 : (allIn ? 1 : 2);
}

// ---- FP32 tests of boxes and points against planes (frustum and plane kinds)
// The exact test (GetBoxPlaneRelationAD, internal_geometry_module.h:254-280) compares the projections of
// the box's farthest and nearest corner, smax and smin, with dist -+ tol. Here both are summed in FP32
// over the box's corners (outward-rounded images of FP64 trees, the values themselves in FP32 trees).
// With M_d the largest coordinate of the root box, E = 2^-19 (sum |n_d| M_d + |dist| + tol) is 32
// units of roundoff of the largest sum possible, which covers the images, the products and sums here
// (under 12 units) and the exact test's own rounding, in FP32 trees too (under 10). Each plane keeps
// the four thresholds
//   smax < a: certainly negative   smax > b: certainly not   smin > c: certainly positive   smin < d: certainly not
// and what they leave undecided takes the exact test. Values outside the FP32 range make E infinite or
// NaN, which decides nothing.
// A node certainly positive for every plane of a frustum holds only entities that pass (they lie in the
// node, and E also spans their own tests' rounding): its subtree is taken untested. 64 frusta, 64
// planes and 8 half-spaces on 1M FP64 boxes: kernels 4.27 ms with exact tests, every entity of a frustum
// tested and contained runs copied one by one, 0.35 ms now.
struct PlaneF32
{
  float n[3], a, b, c, d, pad;
};
// planes per query that the FP32 tests take, one made by each lane; the ones after them are tested exactly
constexpr u32 kMaxPlanes = 32;

__device__ __forceinline__ void plane_f32(const PlaneF32& p, const float lo[3], const float hi[3], float& smin, float& smax)
{
  smin = smax = 0.f;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    const float x = p.n[d] * lo[d], y = p.n[d] * hi[d];
    smin += fminf(x, y);
    smax += fmaxf(x, y);
  }
}

// An entity against more than eight planes: 0 negative for some, 1 for none, 2 undecided. Leaving at the first negative
// one gains with many planes (16 views of 36 on 500k regular FP32 boxes 1.96 ms, now 1.22) and costs with
// the six of a view (96 views 1.33 ms, 1.43 with it), whose loop stands in the kernel without it.
__device__ __noinline__ u32 planes_many_f32(const PlaneF32* planes, u32 n, float3 l, float3 h)
{
  const float lo[3] = { l.x, l.y, l.z }, hi[3] = { h.x, h.y, h.z };
  bool sure = true;
  for (u32 i = 0; i < n; ++i)
  {
    float smin, smax;
    plane_f32(planes[i], lo, hi, smin, smax);
    if (smax < planes[i].a)
      return 0;
    sure &= smax > planes[i].b;
  }
  return sure ? 1 : 2;
}

// planes {dist, n} of one query, lanes 0 .. np - 1; rootBox: {min, size}
template<typename T>
__device__ __forceinline__ void plane_thresholds(const T* pl, u32 np, const T* rootBox, T tol, u32 lane, PlaneF32* out)
{
  if (lane < np)
  {
    PlaneF32 p;
    const float d = float(pl[4 * lane]), t = float(tol);
    float e = fabsf(d) + fabsf(t);
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
      p.n[c] = float(pl[4 * lane + 1 + c]);
      const float lo = float(rootBox[c]), hi = float(T(rootBox[c] + rootBox[3 + c]));
      e += fabsf(p.n[c]) * fmaxf(fabsf(lo), fabsf(hi));
    }
    e = e * 0x1p-19f + 0x1p-120f;
    p.a = (d - t) - e;
    p.b = (d - t) + e;
    p.c = (d + t) + e;
    p.d = (d + t) - e;
    p.pad = 0.f;
    out[lane] = p;
  }
}

// the exact tests of undecided nodes and entities, out of line (see range_node_enters_fp64)
template<typename T>
__device__ __noinline__ bool frustum_node_exact(const T* nb, const T* pl, u32 np, T tol)
{
  for (u32 i = 0; i < np; ++i) // :779-795 first Hit selects, first Negative prunes
  {
    const int rel = GeoD<T>::box_plane(nb, nb + 3, pl[4 * i], pl + 4 * i + 1, tol);
    if (rel == 1)
      return true;
    if (rel == 0)
      return false;
  }
  return true;
}
// an entity passes unless it is negative for some plane. All planes in one call: 64 frusta of 9 planes on 500k FP32
// boxes, tested exactly, 0.66 ms with a call for each and 0.45 this way (with the FP32 tests 0.37).
template<typename T>
__device__ __noinline__ bool frustum_entity_exact(const T* g, int isBox, const T* pl, u32 np, T tol)
{
  if (!isBox)
  {
    for (u32 i = 0; i < np; ++i)
      if (GeoD<T>::point_plane(g, pl[4 * i], pl + 4 * i + 1, tol) == 0)
        return false;
    return true;
  }
  T b[6];
  load_box(g, b);
  const T bsize[3] = { T(b[3] - b[0]), T(b[4] - b[1]), T(b[5] - b[2]) };
  for (u32 i = 0; i < np; ++i)
    if (GeoD<T>::box_plane(b, bsize, pl[4 * i], pl + 4 * i + 1, tol) == 0)
      return false;
  return true;
}
// GetEntityPlaneRelation (ot_query.h:586-602) of a point or box
template<typename T>
__device__ __noinline__ int entity_plane_exact(const T* g, int isBox, const T* pl, T tol)
{
  if (!isBox)
    return GeoD<T>::point_plane(g, pl[0], pl + 1, tol);
  T bsize[3] = { T(g[3] - g[0]), T(g[4] - g[1]), T(g[5] - g[2]) };
  return GeoD<T>::box_plane(g, bsize, pl[0], pl + 1, tol);
}
template<typename T>
__device__ __noinline__ int node_plane_exact(const T* nb, const T* pl, T tol)
{
  return GeoD<T>::box_plane(nb, nb + 3, pl[0], pl + 1, tol);
}

template<typename T, int KIND>
struct BatchArgs
{
  TreeView<T> tv;
  const T* q;   // ranges (6 per query), planes (4 * np per query, 4 for the plane kinds), rays (6 per query) or points (3 per query)
  u32 np;       // planes per query
  u32 nq;
  int mode;     // RangeSearchMode
  T tol, tolInc, maxDist;
  Appender out;
  u32* work;          // counters (see batch_work_bytes), then the split items
  u32* err;
  QueryProgram<T> qp; // combined queries
  int phase;          // 0: whole queries; 1: top levels, deeper subtrees become items; 2: the items
  u32 splitCap;       // item capacity of the work buffer
  u32 splitDepth;     // depth of the subtrees that become items
  // FP64 trees with FP32 images, one record per query of its setup. Ranges: RangeQ; set only where
  // out.count has three slots (the item count, then the pre-tests and the undecided ones, added at the
  // end). Rays on box trees: RayPrep. Picks: PickQ.
  const void* prep = nullptr;
  float tolUp = 0.f, tolIncUp = 0.f; // tol and tolInc rounded up (rays)
  bool planeF32 = false;             // FP32 plane tests: images (FP64 trees), entities in their nodes
};

constexpr u32 kCandBuf = 64;

// Rays on FP64 trees take 94 registers by themselves, which leaves 16 warps per SM; 32 are asked for (64 registers, a
// few spills on the exact path): 30k rays through 1M FP64 boxes 0.53 ms, now 0.44; 40 warps give 0.52. The other
// kinds take what they need: bounds of 8, 40 or 48 warps made them 3 to 30% slower.
template<typename T, int KIND, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, KIND == kRayAll && sizeof(T) == 8 ? 32 / WARPS : 0) batch_query_kernel(BatchArgs<T, KIND> a)
{
  static_assert(KIND >= kRange && KIND <= kPick, "every query kind has its own setup, node test and entity test below");
  using G = GeoD<T>;
  constexpr bool kRangeF32 = KIND == kRange && sizeof(T) == 8;
  constexpr bool kRayPre = KIND == kRayAll && sizeof(T) == 8;
  constexpr bool kPickPre = KIND == kPick && sizeof(T) == 8;
  __shared__ PickF32 pickF[kPickPre ? WARPS : 1];
  constexpr bool kPlanes = KIND == kFrustum || KIND == kPlane || KIND == kPlanePositive;
  // kinds that take whole subtrees untested
  constexpr bool kWhole = KIND == kRange || KIND == kPlanePositive || KIND == kFrustum;
  __shared__ PlaneF32 planeF[kPlanes ? WARPS : 1][KIND == kFrustum ? kMaxPlanes : 1];
  __shared__ RayF32 rayF[kRayPre ? WARPS : 1];
  __shared__ u32 candMem[kRayPre ? WARPS : 1][kRayPre ? kCandBuf : 1];
  __shared__ RangeF32 rangeF[kRangeF32 ? WARPS : 1];
  __shared__ u32 runMem[WARPS][3][32]; // flat runs: entity bases, child bases, child runs' lanes
  __shared__ u32 stackMem[WARPS][kWideStack];
  __shared__ u64 itemMem[WARPS][kItemBuf];
  __shared__ double distMem[KIND == kRayAll ? WARPS : 1][KIND == kRayAll ? kItemBuf : 1];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u32* stack = stackMem[w];
  WarpSink sink{ itemMem[w], KIND == kRayAll ? distMem[w] : nullptr, 0 };
  const TreeView<T>& tv = a.tv;
  u64* items = reinterpret_cast<u64*>(a.work + 4);
  u32 f32Tests = 0, f32Undecided = 0; // FP32 pre-tests of this lane (range on FP64 point trees)
  for (;;)
  {
    u32 q = 0, start = 0;
    if (a.phase == 2)
    {
      // the next (query, subtree) item left by the first phase
      u32 idx = 0;
      if (lane == 0)
        idx = atomicAdd(a.work + 1, 1u);
      idx = __shfl_sync(~0u, idx, 0);
      if (idx >= min(a.work[2], a.splitCap))
        break;
      const u64 item = items[idx];
      q = u32(item >> 32);
      start = u32(item);
      if (q >= a.nq)
        break;
    }
    else
    {
      if (lane == 0)
        q = atomicAdd(a.work, 1u);
      q = __shfl_sync(~0u, q, 0);
      if (q >= a.nq)
        break;
    }
    const u32 root = query_root(tv, q);
    const u32 idBase = id_base(tv, root);
    // ---- query setup (identical on all lanes)
    T r[6], rsize[3];
    const T* pl = nullptr;
    RayD<T> ray;
    bool skip = false;
    bool useF32 = false;
    if constexpr (kRangeF32)
    {
      if (a.prep)
      {
        // the query's prepared thresholds into the warp's shared copy, its flags to every lane
        const u32* src = reinterpret_cast<const u32*>(static_cast<const RangeQ*>(a.prep) + q);
        __syncwarp(); // the previous query's thresholds are read by every lane before they change
        if (lane < kRangeWords)
          reinterpret_cast<u32*>(&rangeF[w])[lane] = src[lane];
        const u32 flags = src[kRangeWords];
        __syncwarp();
        useF32 = true;
        if (a.phase != 2 && (flags & kRangeAll))
        {
          const u32 nt = tv.qTree ? u32(tv.treeOff[root + 1] - tv.treeOff[root]) : tv.n;
          unsigned long long base = 0;
          if (lane == 0)
            base = a.out.reserve(nt);
          base = __shfl_sync(~0u, base, 0);
          for (u32 i = lane; i < nt; i += 32)
            if (base + i < a.out.capacity)
              a.out.items[base + i] = (u64(q) << 32) | i;
          continue;
        }
        skip = (flags & kRangeEmpty) != 0;
      }
    }
    if constexpr (KIND == kRange)
    {
      if (!useF32)
      {
      load_box(a.q + u64(q) * 6, r);
      if (a.phase != 2) // items continue queries that passed this setup in the first phase
      {
        T rb[6];
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
          rb[c] = tv.nodeBox[u64(root) * 6 + c];
          rb[3 + c] = tv.nodeBox[u64(root) * 6 + c] + tv.nodeBox[u64(root) * 6 + 3 + c];
        }
        if (G::range_contains_box(r, rb, a.tol)) // root shortcut (:488-511): every id of the tree
        {
          const u32 nt = tv.qTree ? u32(tv.treeOff[root + 1] - tv.treeOff[root]) : tv.n;
          unsigned long long base = 0;
          if (lane == 0)
            base = a.out.reserve(nt);
          base = __shfl_sync(~0u, base, 0);
          for (u32 i = lane; i < nt; i += 32)
            if (base + i < a.out.capacity)
              a.out.items[base + i] = (u64(q) << 32) | i;
          continue;
        }
      }
      T vol = T(1); // zero-volume range -> empty (:514-519)
#pragma unroll
      for (int c = 0; c < 3; ++c)
      {
        rsize[c] = T(r[3 + c] - r[c]);
        vol *= rsize[c];
      }
      skip = vol <= T(0);
      }
    }
    else if constexpr (KIND == kFrustum)
    {
      pl = a.q + u64(q) * a.np * 4;
      skip = a.np == 0;
    }
    else if constexpr (KIND == kPlane || KIND == kPlanePositive)
      pl = a.q + u64(q) * 4;
    else if constexpr (KIND == kPick)
    {
      pl = a.q + u64(q) * 3; // the point
      bool made = false;
      if constexpr (kPickPre)
        if (a.prep)
        {
          const u32* src = reinterpret_cast<const u32*>(static_cast<const PickQ*>(a.prep) + q);
          __syncwarp(); // the previous query's thresholds are read by every lane before they change
          if (lane < 12)
            reinterpret_cast<u32*>(&pickF[w])[lane] = src[lane];
          skip = a.phase != 2 && src[12] != 0;
          __syncwarp();
          made = true;
        }
      if (!made && a.phase != 2)
      {
        T rb[6];
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
          rb[c] = tv.nodeBox[u64(root) * 6 + c];
          rb[3 + c] = tv.nodeBox[u64(root) * 6 + c] + tv.nodeBox[u64(root) * 6 + 3 + c];
        }
        skip = !G::box_contains_point(rb, pl, a.tol); // :430-431 the point outside the tree's box
      }
    }
    else if constexpr (KIND == kRayAll)
    {
      bool made = false;
      if constexpr (kRayPre)
        if (a.prep)
        {
          const RayPrep* p = static_cast<const RayPrep*>(a.prep) + q;
          const u32 flags = p->flags;
          __syncwarp(); // the previous ray's setup is read by every lane before it changes
          if (lane == 0)
            ray_f32_of(*p, rayF[w]);
          __syncwarp();
          skip = !(flags & kRayValid);
          useF32 = (flags & kRayF32) != 0;
          made = true;
        }
      if (!made)
      {
        ray.make(a.q + u64(q) * 6, a.q + u64(q) * 6 + 3, a.tol, a.tolInc);
        skip = !ray.valid;
      }
    }
    if (skip)
      continue;
    bool planeTests = false;
    if constexpr (kPlanes)
      if (a.planeF32)
      {
        planeTests = true;
        __syncwarp(); // the previous query's planes are read by every lane before they change
        plane_thresholds<T>(pl, min(a.np, kMaxPlanes), tv.nodeBox + u64(root) * 6, a.tol, lane, planeF[w]);
        __syncwarp();
      }
    // the FP32 corners of a node or entity for the plane tests
    auto corners = [&](bool isNode, u32 i, float lo[3], float hi[3]) {
      if constexpr (sizeof(T) == 8)
      {
        if (!isNode && !tv.isBox)
        {
          const float4 p = tv.pointImg[i];
          lo[0] = hi[0] = p.w < INFINITY ? p.x : NAN; // a point without a finite image decides nothing
          lo[1] = hi[1] = p.y, lo[2] = hi[2] = p.z;
          return;
        }
        const float4* img = isNode ? tv.nodeImg : tv.boxImg;
        const float4 x = img[2 * size_t(i)], y = img[2 * size_t(i) + 1];
        lo[0] = x.x, lo[1] = x.y, lo[2] = x.z;
        hi[0] = y.x, hi[1] = y.y, hi[2] = y.z;
      }
      else
      {
        const bool point = !isNode && !tv.isBox;
        const T* g = isNode ? tv.nodeBox + u64(i) * 6 : tv.geom + u64(i) * (point ? 3 : 6);
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
          lo[c] = g[c];
          hi[c] = point ? g[c] : (isNode ? g[c] + g[3 + c] : g[3 + c]);
        }
      }
    };
    u32 nCand = 0; // entities of this ray that may be hit, not yet tested exactly
    // the exact test of the last min(32, nCand) buffered entities, one per lane: candidates of many
    // nodes fill the lanes (an FP64 instruction costs the same for one lane as for 32)
    auto test_cands = [&]() {
      if constexpr (kRayPre)
      {
        const u32 take = min(nCand, 32u);
        nCand -= take;
        bool hit = false;
        double en = 0.0, ex = 0.0;
        u32 id = 0;
        if (lane < take)
        {
          const u32 e = candMem[w][nCand + lane];
          hit = ray_box_exact(a.q + u64(q) * 6, static_cast<const RayPrep*>(a.prep) + q, tv.geom + u64(e) * 6, a.tol, a.tolInc, en, ex) &&
                (a.maxDist == T(0) || en <= a.maxDist);
          if (hit)
            id = tv.ids[e] - idBase;
        }
        __syncwarp();
        sink_put(sink, a.out, lane, hit, q, id, en);
      }
    };
    // ---- node test of one node (run by one lane per child)
    auto enters = [&](u32 node, bool& contained) -> bool {
      const T* nb = tv.nodeBox + u64(node) * 6;
      contained = false;
      if constexpr (KIND == kRange)
      {
        if constexpr (kRangeF32)
        {
          if (useF32)
          {
            int en, in;
            range_node_f32(tv.nodeImg, node, rangeF[w], en, in);
            ++f32Tests;
            f32Undecided += (en == 2 || (en != 0 && in == 2)) ? 1u : 0u;
            if (en == 0)
              return false;
            if (en == 2 && !range_node_enters_fp64(a.q + u64(q) * 6, nb, a.tol))
              return false;
            contained = in == 1;
            if (in == 2)
              contained = range_node_inside_fp64(a.q + u64(q) * 6, nb, a.tol);
            return true;
          }
          // FP64 trees without the pre-tests (box trees): the same tests, out of line, so that none of
          // their FP64 arithmetic is evaluated beside the FP32 path
          if (!range_node_enters_fp64(a.q + u64(q) * 6, nb, a.tol))
            return false;
          contained = range_node_inside_fp64(a.q + u64(q) * 6, nb, a.tol);
          return true;
        }
        T nmin[3] = { nb[0], nb[1], nb[2] }, nsize[3] = { nb[3], nb[4], nb[5] };
        if (!G::overlap_by_min_point(r, rsize, nmin, nsize, a.tol))
          return false;
        contained = G::range_contains_min_size(r, nmin, nsize, a.tol);
        return true;
      }
      else if constexpr (kPlanes)
      {
        const u32 np = KIND == kFrustum ? a.np : 1u;
        if (planeTests)
        {
          float lo[3], hi[3];
          corners(true, node, lo, hi);
          const u32 nf = min(np, kMaxPlanes);
          bool decided = nf == np, positive = true;
          for (u32 i = 0; i < nf; ++i)
          {
            const PlaneF32& p = planeF[w][i];
            float smin, smax;
            plane_f32(p, lo, hi, smin, smax);
            if (smax < p.a)
              return false; // (of a frustum: the planes before this one are positive)
            if (smin > p.c)
              continue;
            positive = false;
            decided = (smax > p.b) & (smin < p.d); // certainly hit
            break;
          }
          if (decided)
          {
            contained = positive && KIND != kPlane;
            return KIND == kPlane ? !positive : true; // :620-621 PlaneSearch enters only nodes the plane hits
          }
        }
        if constexpr (KIND == kFrustum)
          return frustum_node_exact<T>(nb, pl, np, a.tol);
        const int rel = node_plane_exact<T>(nb, pl, a.tol);
        if (KIND == kPlane)
          return rel == 1;
        contained = rel == 2; // :702-710 negative prunes, positive takes the subtree
        return rel != 0;
      }
      else if constexpr (KIND == kQuery)
        return cond_combine(a.qp, q, a.err, [&](const QueryCond& c) { return cond_node(a.qp, c, nb, a.tol); });
      else if constexpr (KIND == kPick)
      {
        if constexpr (kPickPre)
        {
          if (a.prep)
          {
            const int dec = pick_f32(tv.nodeImg[2 * size_t(node)], tv.nodeImg[2 * size_t(node) + 1], pickF[w]);
            if (dec != 2)
              return dec == 1;
          }
          return pick_node_fp64(nb, pl, a.tol);
        }
        return G::node_contains_point(nb, nb + 3, pl, a.tol);
      }
      else if constexpr (KIND == kRayAll)
      {
        T en, ex;
        if constexpr (kRayPre)
          if (a.prep)
          {
            const int rel = useF32 ? ray_box_f32(rayF[w], a.tolUp, a.tolIncUp, tv.nodeImg[2 * size_t(node)], tv.nodeImg[2 * size_t(node) + 1]).rel : 2;
            if (rel != 2)
              return rel == 1;
            return ray_node_exact(a.q + u64(q) * 6, static_cast<const RayPrep*>(a.prep) + q, nb, a.tol, a.tolInc, en, ex);
          }
        return ray.hit_node(nb, nb + 3, en, ex);
      }
    };
    u32 sp = 0;
    if (lane == 0)
    {
      bool contained;
      if (a.phase == 2)
      {
        stack[0] = start; // entered (its node test passed) in the first phase
        sp = 1;
      }
      else if (enters(root, contained))
      {
        stack[0] = root | (contained ? kContained : 0u);
        sp = 1;
      }
    }
    sp = __shfl_sync(~0u, sp, 0);
    __syncwarp();
    u32 visits = 0;
    bool bad = false;
    // the lane holding flat item f of a run of per-lane counts with inclusive prefix `incl`
    auto owner = [&](u32 incl, u32 f) -> u32 {
      u32 o = 0;
#pragma unroll
      for (u32 s = 16; s >= 1; s >>= 1)
        if (__shfl_sync(~0u, incl, o + s - 1) <= f)
          o += s;
      return o;
    };
    while (sp > 0)
    {
      // up to 32 nodes per step, one per lane; one at a time (depth first) near the stack's end. The
      // entities and children of the popped nodes are spread over the lanes as one flat run, so
      // consecutive lanes read consecutive entities of a node.
      const u32 take = (sp + 7u * 32u <= u32(kWideStack - kWideReserve)) ? min(sp, 32u) : 1u;
      sp -= take;
      const bool act = lane < take;
      const u32 entry = act ? stack[sp + lane] : 0u;
      __syncwarp();
      const u32 node = entry & ~kContained;
      uint4 L = make_uint4(0u, 0u, 0u, 0u);
      if (act)
        L = tv.link[node];
      visits += take;
      const bool badLane = act && (L.z > tv.n || L.w > tv.n || L.y > L.z || (L.x >> kChildShift) > 8u ||
                                   u64(L.x & kFirstChildMask) + (L.x >> kChildShift) > tv.nNodes);
      if (__any_sync(~0u, badLane) || visits > tv.nNodes)
      {
        bad = true;
        break;
      }
      // Contained nodes: whole subtrees without entity tests (range :549-567, positive side :711-726); a
      // subtree is one run of sortedIds. The runs of the popped nodes are copied together, with one
      // reservation. In the first launch of a
      // split batch a large one is left to its children, which become items: one warp copying half
      // of a tree would be the last to end.
      bool whole = false, expand = false;
      if constexpr (kWhole)
      {
        const bool cont = act && (entry & kContained);
        if (__any_sync(~0u, cont))
        {
          expand = cont && a.phase == 1 && (L.x >> kChildShift) != 0u && L.w - L.y > 1024u;
          whole = cont;
          const u32 len = cont ? (expand ? L.z : L.w) - L.y : 0u;
          u32 incl = len;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1)
          {
            const u32 y = __shfl_up_sync(~0u, incl, o);
            if (lane >= u32(o))
              incl += y;
          }
          const u32 total = __shfl_sync(~0u, incl, 31);
          unsigned long long base = 0;
          if (lane == 0 && total)
            base = a.out.reserve(total);
          base = __shfl_sync(~0u, base, 0);
          const u64 room = base < a.out.capacity ? a.out.capacity - base : 0;
          const u32 end = u32(min(u64(total), room));
          const u32* __restrict__ src = tv.ids;
          u64* __restrict__ dst = a.out.items + base;
          for (u32 f0 = 0; f0 < end; f0 += 128)
          {
            u32 id[4];
#pragma unroll
            for (u32 k = 0; k < 4; ++k)
            {
              const u32 f = f0 + k * 32 + lane;
              const u32 o = owner(incl, min(f, total - 1));
              const u32 oy = __shfl_sync(~0u, L.y, o), oex = __shfl_sync(~0u, incl - len, o);
              id[k] = f < end ? src[oy + (f - oex)] : 0u;
            }
#pragma unroll
            for (u32 k = 0; k < 4; ++k)
              if (f0 + k * 32 + lane < end)
                dst[f0 + k * 32 + lane] = (u64(q) << 32) | (id[k] - idBase);
          }
        }
      }
      const bool tests = act && !whole;
      // The entities and the children of the popped nodes as flat runs: the items of the lanes before (excl),
      // of both kinds from one scan where the counts fit one word (23 and 9 bits), and for the r-th lane
      // that has any, its first item minus its place in the flat order, in shared memory.
      const u32 cntE = tests ? L.z - L.y : 0u;
      const u32 cntC = (tests || expand) ? (L.x >> kChildShift) : 0u;
      u32 inclE = cntE, inclC = cntC;
      if (!__any_sync(~0u, cntE >= (1u << 17)))
      {
        u32 incl = cntE | (cntC << 23);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
          const u32 y = __shfl_up_sync(~0u, incl, o);
          if (lane >= u32(o))
            incl += y;
        }
        inclE = incl & ((1u << 23) - 1);
        inclC = incl >> 23;
      }
      else
      {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
          const u32 y = __shfl_up_sync(~0u, inclE, o), z = __shfl_up_sync(~0u, inclC, o);
          if (lane >= u32(o))
          {
            inclE += y;
            inclC += z;
          }
        }
      }
      const u32 totalE = __shfl_sync(~0u, inclE, 31), totalC = __shfl_sync(~0u, inclC, 31);
      const u32 exclE = inclE - cntE, exclC = inclC - cntC;
      const u32 lt = (1u << lane) - 1u;
      {
        const u32 nzE = __ballot_sync(~0u, cntE != 0u), nzC = __ballot_sync(~0u, cntC != 0u);
        if (cntE)
          runMem[w][0][__popc(nzE & lt)] = L.y - exclE;
        if (cntC)
        {
          runMem[w][1][__popc(nzC & lt)] = (L.x & kFirstChildMask) - exclC;
          runMem[w][2][__popc(nzC & lt)] = lane;
        }
        __syncwarp();
      }
      // The run of item f0 + lane (`before`: the runs that start before f0): the runs that start in the window
      // of 32 items up to it, by one reduction and a population count. A binary search over the lanes'
      // sums takes five dependent shuffles: 10k ranges on 1M FP64 points 54 us, now 48; 1M ranges and 1M rays
      // on 4096 FP32 trees 1.49 and 2.12 ms, now 1.38 and 1.95.
      auto flat_run = [&](u32 excl, u32 cnt, u32 f0, u32& before) -> u32 {
        const u32 at = excl - f0;
        const u32 starts = __reduce_or_sync(~0u, (cnt && at < 32u) ? 1u << at : 0u);
        const u32 run = before + __popc(starts & (lt | (1u << lane))) - 1u;
        before += __popc(starts);
        return run;
      };
      const u32 expandMask = kWhole ? __ballot_sync(~0u, expand) : 0u;
      // entities of the popped nodes
      {
        const u32 total = totalE;
        u32 before = 0;
        for (u32 f0 = 0; f0 < total; f0 += 32)
        {
          const u32 f = f0 + lane;
          const u32 run = flat_run(exclE, cntE, f0, before);
          const u32 e = runMem[w][0][run] + f;
          const bool v = f < total;
          bool hit = false;
          double d = 0.0;
          if constexpr (kRayPre)
            if (a.prep)
            {
              const bool may = v && (!useF32 || ray_box_f32(rayF[w], a.tolUp, a.tolIncUp, tv.boxImg[2 * size_t(e)], tv.boxImg[2 * size_t(e) + 1]).rel != 0);
              const u32 bal = __ballot_sync(~0u, may);
              if (may)
                candMem[w][nCand + __popc(bal & ((1u << lane) - 1))] = e;
              nCand += __popc(bal);
              __syncwarp();
              if (nCand >= 32)
                test_cands();
              continue;
            }
          if (v)
          {
            if constexpr (KIND == kRange)
            {
              if (!tv.isBox)
              {
                int dec = 2;
                if constexpr (kRangeF32)
                  if (useF32)
                  {
                    dec = range_point_f32(tv.pointImg[e], rangeF[w]);
                    ++f32Tests;
                    f32Undecided += dec == 2 ? 1u : 0u;
                  }
                hit = dec == 1;
                if (dec == 2)
                {
                  if constexpr (kRangeF32)
                    hit = range_point_inside_fp64(a.q + u64(q) * 6, tv.geom + u64(e) * 3, a.tol);
                  else
                    hit = G::box_contains_point(r, tv.geom + u64(e) * 3, a.tol);
                }
              }
              else if (kRangeF32)
              {
                if constexpr (kRangeF32)
                {
                  int dec = 2;
                  if (useF32)
                  {
                    dec = range_box_f32(tv.boxImg, e, rangeF[w], a.mode == OTG_RANGE_OVERLAP);
                    ++f32Tests;
                    f32Undecided += dec == 2 ? 1u : 0u;
                  }
                  hit = dec == 2 ? range_box_fp64(a.q + u64(q) * 6, tv.geom + u64(e) * 6, a.mode, a.tol) : dec == 1;
                }
              }
              else
              {
                T bx[6];
                load_box(tv.geom + u64(e) * 6, bx);
                hit = (a.mode == OTG_RANGE_OVERLAP) ? (G::box_relation(r, bx, a.tol) == -1) : G::contains_box_no_tol(r, bx);
              }
            }
            else if constexpr (kPlanes)
            {
              const u32 np = KIND == kFrustum ? a.np : 1u;
              const T* g = tv.geom + u64(e) * (tv.isBox ? 6 : 3);
              bool decided = false;
              u32 passed = 0; // leading planes that the entity is certainly not negative for
              if (planeTests)
              {
                float lo[3], hi[3];
                corners(false, e, lo, hi);
                bool neg = false, sure = true, cut = true;
                // an entity with a NaN (the root may hold some) takes the exact test: the corners' sums pass a NaN over
                const bool plain = (lo[0] <= hi[0]) & (lo[1] <= hi[1]) & (lo[2] <= hi[2]);
                const u32 nf = min(np, kMaxPlanes);
                if (KIND == kFrustum && nf > 8u)
                {
                  const u32 rel = planes_many_f32(planeF[w], nf, make_float3(lo[0], lo[1], lo[2]), make_float3(hi[0], hi[1], hi[2]));
                  neg = rel == 0;
                  sure = rel == 1;
                }
                else
                  for (u32 i = 0; i < nf; ++i)
                  {
                    const PlaneF32& p = planeF[w][i];
                    float smin, smax;
                    plane_f32(p, lo, hi, smin, smax);
                    neg |= smax < p.a;
                    sure &= smax > p.b;
                    if (KIND == kPlane)
                    {
                      cut = smin < p.d;
                      neg |= smin > p.c; // not hit
                    }
                  }
                decided = plain & (neg | (sure & cut & (nf == np)));
                hit = !neg;
                passed = plain && sure ? nf : 0u;
              }
              if (!decided)
              {
                if constexpr (KIND == kFrustum)
                  hit = frustum_entity_exact<T>(g, tv.isBox, pl + 4 * passed, np - passed, a.tol);
                else
                {
                  const int rel = entity_plane_exact<T>(g, tv.isBox, pl, a.tol);
                  hit = KIND == kPlane ? rel == 1 : rel != 0;
                }
              }
            }
            else if constexpr (KIND == kQuery)
            {
              const T* g = tv.geom + u64(e) * (tv.isBox ? 6 : 3);
              hit = cond_combine(a.qp, q, a.err, [&](const QueryCond& c) { return cond_entity(a.qp, c, g, tv.isBox != 0, a.tol); });
            }
            else if constexpr (kPickPre)
            {
              int dec = 2;
              if (a.prep)
              {
                float4 lo, hi;
                if (tv.isBox)
                {
                  lo = tv.boxImg[2 * size_t(e)];
                  hi = tv.boxImg[2 * size_t(e) + 1];
                }
                else
                  lo = hi = tv.pointImg[e];
                dec = pick_f32(lo, hi, pickF[w]);
                if (!tv.isBox) // a point within reach is tested exactly, and so is one without a finite image
                  dec = dec != 0 || !(lo.w < INFINITY) ? 2 : 0;
              }
              hit = dec == 2 ? pick_entity_fp64(tv.geom + u64(e) * (tv.isBox ? 6 : 3), tv.isBox, pl, a.tol) : dec == 1;
            }
            else if constexpr (KIND == kPick)
              hit = tv.isBox ? G::box_contains_point(tv.geom + u64(e) * 6, pl, a.tol) : G::points_equal(tv.geom + u64(e) * 3, pl, a.tol);
            else if constexpr (KIND == kRayAll)
            {
              T en, ex;
              hit = (tv.isBox ? ray.hit_box(tv.geom + u64(e) * 6, en, ex) : ray.hit_point(tv.geom + u64(e) * 3, en, ex)) &&
                    (a.maxDist == T(0) || en <= a.maxDist);
              d = double(en);
            }
          }
          sink_put(sink, a.out, lane, hit, q, hit ? tv.ids[e] - idBase : 0u, d);
        }
      }
      // children of the popped nodes, tested before they are pushed
      {
        const u32 total = totalC;
        u32 before = 0;
        for (u32 f0 = 0; f0 < total; f0 += 32)
        {
          const u32 f = f0 + lane;
          const u32 run = flat_run(exclC, cntC, f0, before);
          bool keep = false, contained = false;
          const u32 child = runMem[w][1][run] + f;
          bool free = false; // a contained node's child
          if constexpr (kWhole)
            if (expandMask)
              free = (expandMask >> runMem[w][2][run]) & 1u;
          if (f < total)
          {
            keep = contained = free;
            if (!free)
              keep = enters(child, contained);
          }
          if (a.phase == 1)
          {
            // subtrees at the split depth become items for any warp
            const bool defer = keep && tv.nodeDepth[child] >= a.splitDepth;
            const u32 dbal = __ballot_sync(~0u, defer);
            if (dbal)
            {
              u32 ibase = 0;
              if (lane == 0)
                ibase = atomicAdd(a.work + 2, u32(__popc(dbal)));
              ibase = __shfl_sync(~0u, ibase, 0);
              if (defer)
              {
                const u32 slot = ibase + __popc(dbal & ((1u << lane) - 1));
                if (slot < a.splitCap)
                  items[slot] = (u64(q) << 32) | child | (contained ? kContained : 0u);
                else
                  atomicOr(a.err, kErrStack);
              }
            }
            keep = keep && !defer;
          }
          const u32 bal = __ballot_sync(~0u, keep);
          if (sp + __popc(bal) > u32(kWideStack))
          {
            bad = true;
            break;
          }
          if (keep)
            stack[sp + __popc(bal & ((1u << lane) - 1))] = child | (contained ? kContained : 0u);
          sp += __popc(bal);
        }
      }
      __syncwarp();
      if (bad)
        break;
    }
    if constexpr (kRayPre)
      if (nCand)
        test_cands();
    if (bad && lane == 0)
      atomicOr(a.err, kErrStack);
    sink_flush(sink, a.out, lane);
  }
  if constexpr (kRangeF32)
  {
    if (a.prep)
    {
      // the warp's counts, after the item count of the appender
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
      {
        f32Tests += __shfl_xor_sync(~0u, f32Tests, o);
        f32Undecided += __shfl_xor_sync(~0u, f32Undecided, o);
      }
      if (lane == 0)
      {
        atomicAdd(a.out.count + 1, (unsigned long long)f32Tests);
        atomicAdd(a.out.count + 2, (unsigned long long)f32Undecided);
      }
    }
  }
}

template<typename T, int KIND, int WARPS>
static int launch_batch_w(const BatchArgs<T, KIND>& a, cudaStream_t st)
{
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (!e)
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!e)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, batch_query_kernel<T, KIND, WARPS>, WARPS * 32, 0);
  if (!e && !a.out.cleared)
    e = cudaMemsetAsync(a.work, 0, 16, st);
  if (e)
    return cuda_status(e, "configuring the batched query kernel");
  const u64 resident = u64(sms) * std::max(per, 1);
  const u64 want = (u64(a.nq) + WARPS - 1) / WARPS;
  const u32 grid = u32(std::max<u64>(1, std::min<u64>(resident, want)));
  if (a.splitCap == 0)
  {
    batch_query_kernel<T, KIND, WARPS><<<grid, WARPS * 32, 0, st>>>(a);
    return cuda_status(cudaGetLastError(), "launching the batched query kernel");
  }
  // a small batch: the top levels of every query, then its subtrees spread over every resident warp
  BatchArgs<T, KIND> b = a;
  b.phase = 1;
  batch_query_kernel<T, KIND, WARPS><<<grid, WARPS * 32, 0, st>>>(b);
  b.phase = 2;
  batch_query_kernel<T, KIND, WARPS><<<u32(resident), WARPS * 32, 0, st>>>(b);
  return cuda_status(cudaGetLastError(), "launching the batched query kernel");
}

// shape: warps per block (2, 4 or 8) | split code << 8 (otg_query.cuh: shape_split_depth), autotuned
// workBytes: size of the work buffer; a batch is split only when the buffer holds its items
template<typename T, int KIND>
static int launch_batch(const BatchArgs<T, KIND>& a0, int shape, cudaStream_t st, size_t workBytes)
{
  if (workBytes < 16)
  {
    set_error("batched query work buffer below its 16 bytes of counters");
    return OTG_ERR_INVALID_ARGUMENT;
  }
  BatchArgs<T, KIND> a = a0;
  a.phase = 0;
  a.splitDepth = shape_split_depth(shape, a.nq);
  const u64 items = a.splitDepth ? u64(a.nq) * split_items_per_query(a.splitDepth) : 0;
  a.splitCap = (items && a.tv.nodeDepth && workBytes >= 16 + sizeof(u64) * items) ? u32(items) : 0u;
  const int warps = shape & 0xff;
  if (warps == 2)
    return launch_batch_w<T, KIND, 2>(a, st);
  if (warps == 8)
    return launch_batch_w<T, KIND, 8>(a, st);
  return launch_batch_w<T, KIND, 4>(a, st);
}

template<typename T>
int batch_range(const TreeView<T>& tv, const T* ranges, u32 nq, int mode, T tol, Appender out, u32* work, u32* err, cudaStream_t st, int shape, size_t workBytes)
{
  BatchArgs<T, kRange> a{ tv, ranges, 0, nq, mode, tol, T(0), T(0), out, work, err };
  TmpBuf prep;
  if constexpr (sizeof(T) == 8)
  {
    // FP64 trees with FP32 images: the per-query setup by one thread per query
    if (tv.nodeImg && (tv.isBox ? tv.boxImg && tv.inNodes && tol >= T(0) : tv.pointImg != nullptr) && nq)
    {
      if (cudaError_t e = prep.ensure(sizeof(RangeQ) * nq, st))
        return cuda_status(e, "allocating the range setup");
      range_prepare_kernel<<<u32((nq + 127) / 128), 128, 0, st>>>(tv, ranges, nq, mode, double(tol), prep.as<RangeQ>());
      a.prep = prep.p;
    }
  }
  return launch_batch<T, kRange>(a, shape, st, workBytes);
}
// whether the plane kinds test in FP32: FP64 trees need their images, and every entity lies in its node
template<typename T>
static bool plane_filter(const TreeView<T>& tv)
{
  if (sizeof(T) == 8)
    return tv.inNodes && tv.nodeImg && (tv.isBox ? tv.boxImg : tv.pointImg);
  return tv.inNodes;
}
template<typename T>
int batch_frustum(const TreeView<T>& tv, const T* planes, u32 np, u32 nq, T tol, Appender out, u32* work, u32* err, cudaStream_t st, int shape, size_t workBytes)
{
  BatchArgs<T, kFrustum> a{ tv, planes, np, nq, 0, tol, T(0), T(0), out, work, err };
  a.planeF32 = plane_filter(tv);
  return launch_batch<T, kFrustum>(a, shape, st, workBytes);
}
template<typename T>
int batch_plane(const TreeView<T>& tv, const T* planes, u32 nq, bool positive, T tol, Appender out, u32* work, u32* err, cudaStream_t st, int shape, size_t workBytes)
{
  if (positive)
  {
    BatchArgs<T, kPlanePositive> a{ tv, planes, 1, nq, 0, tol, T(0), T(0), out, work, err };
    a.planeF32 = plane_filter(tv);
    return launch_batch<T, kPlanePositive>(a, shape, st, workBytes);
  }
  BatchArgs<T, kPlane> a{ tv, planes, 1, nq, 0, tol, T(0), T(0), out, work, err };
  a.planeF32 = plane_filter(tv);
  return launch_batch<T, kPlane>(a, shape, st, workBytes);
}
template<typename T>
int batch_query_program(const TreeView<T>& tv, const QueryProgram<T>& qp, u32 nq, T tol, Appender out, u32* work, u32* err, cudaStream_t st, int shape, size_t workBytes)
{
  BatchArgs<T, kQuery> a{ tv, nullptr, 0, nq, 0, tol, T(0), T(0), out, work, err };
  a.qp = qp;
  return launch_batch<T, kQuery>(a, shape, st, workBytes);
}
template<typename T>
int batch_pick(const TreeView<T>& tv, const T* pts, u32 nq, T tol, Appender out, u32* work, u32* err, cudaStream_t st, int shape, size_t workBytes)
{
  BatchArgs<T, kPick> a{ tv, pts, 0, nq, 0, tol, T(0), T(0), out, work, err };
  TmpBuf prep;
  if constexpr (sizeof(T) == 8)
  {
    if (tv.nodeImg && (tv.isBox ? tv.boxImg : tv.pointImg) && tv.inNodes && tol >= T(0) && nq)
    {
      if (cudaError_t e = prep.ensure(sizeof(PickQ) * nq, st))
        return cuda_status(e, "allocating the pick setup");
      pick_prepare_kernel<<<u32((nq + 127) / 128), 128, 0, st>>>(tv, pts, nq, double(tol), prep.as<PickQ>());
      a.prep = prep.p;
    }
  }
  return launch_batch<T, kPick>(a, shape, st, workBytes);
}
template<typename T>
int batch_ray_all(const TreeView<T>& tv, const T* rays, u32 nq, T tol, T tolInc, T maxDist, Appender out, u32* work, u32* err, cudaStream_t st,
                  int shape, size_t workBytes)
{
  BatchArgs<T, kRayAll> a{ tv, rays, 0, nq, 0, tol, tolInc, maxDist, out, work, err };
  TmpBuf prep;
  if constexpr (sizeof(T) == 8)
  {
    // FP64 box trees with FP32 images: the setup by one thread per ray, most tests in FP32
    if (tv.nodeImg && tv.boxImg && tv.isBox && nq)
    {
      if (cudaError_t e = prep.ensure(sizeof(RayPrep) * nq, st))
        return cuda_status(e, "allocating the ray setup");
      if (int rc = ray_prepare(rays, nq, double(tol), double(tolInc), prep.as<RayPrep>(), st))
        return rc;
      a.prep = prep.p;
      a.tolUp = float_ru_host(double(tol));
      a.tolIncUp = float_ru_host(double(tolInc));
    }
  }
  return launch_batch<T, kRayAll>(a, shape, st, workBytes);
}

template int batch_range<double>(const TreeView<double>&, const double*, u32, int, double, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_range<float>(const TreeView<float>&, const float*, u32, int, float, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_frustum<double>(const TreeView<double>&, const double*, u32, u32, double, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_frustum<float>(const TreeView<float>&, const float*, u32, u32, float, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_plane<double>(const TreeView<double>&, const double*, u32, bool, double, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_plane<float>(const TreeView<float>&, const float*, u32, bool, float, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_query_program<double>(const TreeView<double>&, const QueryProgram<double>&, u32, double, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_query_program<float>(const TreeView<float>&, const QueryProgram<float>&, u32, float, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_pick<double>(const TreeView<double>&, const double*, u32, double, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_pick<float>(const TreeView<float>&, const float*, u32, float, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_ray_all<double>(const TreeView<double>&, const double*, u32, double, double, double, Appender, u32*, u32*, cudaStream_t, int, size_t);
template int batch_ray_all<float>(const TreeView<float>&, const float*, u32, float, float, float, Appender, u32*, u32*, cudaStream_t, int, size_t);

} // namespace otg
