// otg_collide.cu — candidate search of CollisionDetection (core/ot_query.h:1308-1497 two trees,
// :1690-1914 one tree) with an FP32 filter.
//
// One warp walks the other tree for a packet of up to 32 entities of the first tree that follow each other
// in it at the same depth, and so lie close together. A stack entry is a node and the mask of the
// entities whose boxes may meet it. The node's own entities are tested by the lanes in parallel
// against each box of the mask (read from shared memory), its children against the packet's common
// box first and then box by box. Entities of shallow nodes (large boxes, long walks, little in common)
// come first, one to a packet; packets are taken from a shared counter.
// Bound by instruction issue and by the latency of the node loads. One entity per warp spends a walk of
// the upper levels on every box: 4M clustered FP64 boxes with themselves took 6.67 ms and now take 1.55 ms,
// 8M against 16M 9.39 and 1.89 ms.
//
// The test runs on FP32 images of the second tree's boxes, lo = rd(min) and hi = ru(max). With M the
// largest coordinate of the two root boxes and of the first box, and G = 2^-20 (M + tol), four bounds per dimension of the
// first box decide GetBoxRelation (general.h:262-289) for all but a few pairs:
//   certainly not         hi < a.min - tol - G or lo > a.max + tol + G in some dimension
//   certainly overlapped  hi > a.min + tol + G and lo < a.max - tol - G in every dimension
// G is eight times the images' rounding and, in FP32 trees, the rounding of the predicate itself: the
// first makes that dimension "separated" or "adjacent" in its arithmetic, either of which excludes
// "overlapped", the second is its "overlapped" branch. The rest is re-tested with the exact predicate
// in the tree's scalar type, so the candidate set equals {pairs with GetBoxRelation == Overlapped}.
// A certain overlap is also deeper than any rounding in the reference's tree walk, which prunes by
// node boxes that hold the two: such pairs are marked (kPairSure) and spared the walk's rules in
// collide_filter_kernel. In a single tree only pairs whose second position follows the first are
// searched, so each pair is tested once.
#include "otg_query.cuh"

#include <cmath>

namespace otg
{

constexpr u32 kPairBuf = 128;
// Subtrees of at most this many entities are tested without their nodes. 4M clustered boxes of 32 per node with
// themselves: 1.98 ms at 0, 1.83 at 64, 1.73 at 128 (searches of 16M boxes of 16 per node stay within 1%).
constexpr u32 kDirectBoxes = 128;

// Entities to a packet: 32 where that gives every resident warp a packet (about 156k entities), else as many
// as do. 1000, 20k and 60k boxes that overlap most or some 1500 of the others, whole call: 2.57, 3.48 and 5.18 ms with 32
// always, 0.34, 1.17 and 2.87 this way; 20k, 60k and 150k with 3 each 0.228, 0.257 and 0.255, now 0.210, 0.230 and 0.261.
constexpr u64 kPacketsWanted = 152 * 32;

struct CollideCounters
{
  unsigned long long tests;
  unsigned long long rechecks;
  u32 work;
  u32 pad;
};

template<typename T>
struct CollideArgs
{
  const T* geomA;
  u32 nA;
  const u32* order;    // processing order of the A entities
  const u32* ownerA;   // node holding each A entity (kNoOwner: none reachable, skipped)
  const u32* singles;  // entities at the front of the order that are walked one by one
  const T* rootA;      // root boxes {min, size}
  const T* rootB;
  const float4* imgB;  // per entity {min rounded down}, {max rounded up}
  const T* geomB;
  const uint4* linkB;
  const float4* nodeB; // per node {min rounded down}, {max rounded up}
  u32 nB, nNodesB;
  u32 direct;          // subtrees of at most this many entities are tested without their nodes
  u32 stackCap;        // entries of a warp's stack
  u32 packet;          // entities to a packet
  T tol;
  int selfMode;
  int swapOut; // two trees searched from the second tree's entities: emit (walked position, entity position)
  // Entities lie in their nodes. If not (set_entities), which pairs are found depends on the nodes that a
  // box enters: node boxes are then tested without G (tolHi: tol rounded up), and no overlap is marked.
  int sure;
  float tolHi;
  Appender out;
  CollideCounters* ctr;
  u32* err;
};

// a warp's shared memory: the packet's bounds (a.min - tol - G, position; a.max + tol + G; a.min + tol + G;
// a.max - tol - G), the children's boxes, the pair buffer, the stack (a multiple of 4 entries, so that
// every warp's part starts on 16 bytes)
struct CollideWarpMem
{
  float4 box[32][4];
  float4 child[8][2];
  float4 common[2]; // the packet's common bounds
  u64 pairs[kPairBuf];
};
static_assert(sizeof(CollideWarpMem) % 16 == 0, "warps' parts start on 16 bytes");
__host__ __device__ constexpr size_t collide_warp_bytes(u32 stackCap) { return sizeof(CollideWarpMem) + size_t(stackCap) * (sizeof(uint4) + sizeof(u32)); }

__device__ __forceinline__ bool apart(float4 a0, float4 a1, float4 lo, float4 hi)
{
  return (hi.x < a0.x) | (hi.y < a0.y) | (hi.z < a0.z) | (a1.x < lo.x) | (a1.y < lo.y) | (a1.z < lo.z);
}

template<typename T>
__device__ __noinline__ bool boxes_overlap_exact(const T* a, const T* b, T tol)
{
  T ea[6], eb[6];
  load_box(a, ea);
  load_box(b, eb);
  return GeoD<T>::box_relation(ea, eb, tol) == -1;
}

// 64 registers and 32 warps per SM, with the children's boxes loaded after the entities and the common box in shared
// memory: 1.55 and 1.89 ms on the two workloads above. The children on their way during the entities: 1.73 and
// 2.17 ms; at 80 to 96 registers and 24 warps 1.76 and 2.20; 40 warps spill (1.88 and 2.17).
template<typename T, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 32 / WARPS) collide_packet_kernel(CollideArgs<T> a)
{
  extern __shared__ __align__(16) unsigned char collideMem[];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned char* mem = collideMem + w * collide_warp_bytes(a.stackCap);
  CollideWarpMem& W = *reinterpret_cast<CollideWarpMem*>(mem);
  uint4* stackL = reinterpret_cast<uint4*>(mem + sizeof(CollideWarpMem));
  u32* stackM = reinterpret_cast<u32*>(stackL + a.stackCap);
  const u32 lt = (1u << lane) - 1;
  u32 tests = 0, rechecks = 0;
  const u32 singles = min(*a.singles, a.nA);
  const u32 items = singles + (a.nA - singles + a.packet - 1) / a.packet;
  float M = 0.f; // of the header comment
#pragma unroll
  for (int c = 0; c < 3; ++c)
  {
    M = fmaxf(M, fmaxf(fabsf(float(a.rootA[c])), fabsf(float(T(a.rootA[c] + a.rootA[3 + c])))));
    M = fmaxf(M, fmaxf(fabsf(float(a.rootB[c])), fabsf(float(T(a.rootB[c] + a.rootB[3 + c])))));
  }
  const float tolf = float(a.tol);
  const uint4 root = a.linkB[0];
  auto flush = [&](u32 n) {
    unsigned long long b0 = 0;
    if (lane == 0)
      b0 = a.out.reserve(n);
    b0 = __shfl_sync(~0u, b0, 0);
    for (u32 t = lane; t < n; t += 32)
      if (b0 + t < a.out.capacity)
        a.out.items[b0 + t] = W.pairs[t];
    __syncwarp();
  };
  for (;;)
  {
    u32 item = 0;
    if (lane == 0)
      item = atomicAdd(&a.ctr->work, 1u);
    item = __shfl_sync(~0u, item, 0);
    if (item >= items)
      break;
    const u32 first = item < singles ? item : singles + (item - singles) * a.packet;
    const u32 count = item < singles ? 1u : min(a.packet, a.nA - first);
    u32 i = 0xffffffffu;
    bool valid = false;
    float4 a0 = make_float4(INFINITY, INFINITY, INFINITY, 0.f), a1 = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
    float4 n0 = a0, n1 = a1; // the bounds for node boxes
    if (lane < count)
    {
      i = a.order[first + lane];
      // an entity that no node reachable from the root holds takes part in no pair
      valid = a.ownerA[i] != kNoOwner;
      T e[6];
      load_box(a.geomA + u64(i) * 6, e);
      // round-to-nearest: G is many times the roundings here (this box may lie outside the root box
      // after set_entities)
      const float mn[3] = { float(e[0]), float(e[1]), float(e[2]) }, mx[3] = { float(e[3]), float(e[4]), float(e[5]) };
      float far = M;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        far = fmaxf(far, fmaxf(fabsf(mn[c]), fabsf(mx[c])));
      const float up = tolf + ((far + tolf) * 0x1p-20f + 0x1p-140f);
      // a bound that is no finite number excludes nothing
      auto below = [](float v) { return fabsf(v) < INFINITY ? v : -INFINITY; };
      auto above = [](float v) { return fabsf(v) < INFINITY ? v : INFINITY; };
      if (valid)
      {
        a0 = make_float4(below(mn[0] - up), below(mn[1] - up), below(mn[2] - up), 0.f);
        a1 = make_float4(above(mx[0] + up), above(mx[1] + up), above(mx[2] + up), 0.f);
      }
      n0 = a0;
      n1 = a1;
      if (valid && !a.sure)
      {
        n0 = make_float4(__double2float_rd(double(e[0])), __double2float_rd(double(e[1])), __double2float_rd(double(e[2])), 0.f);
        n1 = make_float4(__fadd_ru(__double2float_ru(double(e[3])), a.tolHi), __fadd_ru(__double2float_ru(double(e[4])), a.tolHi),
                         __fadd_ru(__double2float_ru(double(e[5])), a.tolHi), 0.f);
      }
      a0.w = __uint_as_float(i);
      W.box[lane][0] = a0;
      W.box[lane][1] = a1;
      W.box[lane][2] = make_float4(mn[0] + up, mn[1] + up, mn[2] + up, 0.f);
      W.box[lane][3] = make_float4(mx[0] - up, mx[1] - up, mx[2] - up, 0.f);
    }
    // the packet's common box and first position
    float4 u0 = a0, u1 = a1;
    u32 iMin = valid ? i : 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
      u0.x = fminf(u0.x, __shfl_xor_sync(~0u, u0.x, o));
      u0.y = fminf(u0.y, __shfl_xor_sync(~0u, u0.y, o));
      u0.z = fminf(u0.z, __shfl_xor_sync(~0u, u0.z, o));
      u1.x = fmaxf(u1.x, __shfl_xor_sync(~0u, u1.x, o));
      u1.y = fmaxf(u1.y, __shfl_xor_sync(~0u, u1.y, o));
      u1.z = fmaxf(u1.z, __shfl_xor_sync(~0u, u1.z, o));
      iMin = min(iMin, __shfl_xor_sync(~0u, iMin, o));
    }
    const u32 all = __ballot_sync(~0u, valid);
    if (!all)
      continue;
    if (lane == 0)
    {
      W.common[0] = u0;
      W.common[1] = u1;
    }
    u32 sp = 1, visits = 0, nbuf = 0;
    bool bad = false;
    if (lane == 0)
    {
      stackL[0] = root;
      stackM[0] = all;
    }
    __syncwarp();
    while (sp > 0)
    {
      --sp;
      const uint4 L = stackL[sp];
      const u32 mask = stackM[sp];
      __syncwarp();
      // A subtree of few entities is one run of the tree order, tested as it comes instead of by its nodes
      // (boxes that overlap also overlap each other's nodes, so this adds no pair).
      const bool whole = L.w - L.y <= a.direct;
      const u32 end = whole ? L.w : L.z;
      const u32 fc = L.x & kFirstChildMask, cc = whole ? 0u : L.x >> kChildShift;
      if (L.z > a.nB || L.y > L.z || L.w > a.nB || ++visits > a.nNodesB || cc > 8u || u64(fc) + cc > a.nNodesB || sp + cc > a.stackCap)
      {
        bad = true;
        break;
      }
      const u32 jb = a.selfMode ? max(L.y, iMin + 1) : L.y;
      for (u32 base = jb; base < end; base += 32)
      {
        const u32 j = base + lane;
        bool in = false;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (j < end)
        {
          lo = a.imgB[2 * size_t(j)];
          hi = a.imgB[2 * size_t(j) + 1];
          in = !apart(W.common[0], W.common[1], lo, hi);
        }
        if (!__any_sync(~0u, in))
          continue;
        for (u32 mm = mask; mm; mm &= mm - 1)
        {
          const u32 l = u32(__ffs(int(mm))) - 1;
          const float4 b0 = W.box[l][0], b1 = W.box[l][1];
          const u32 il = __float_as_uint(b0.w);
          const bool cand = in && !apart(b0, b1, lo, hi) && (!a.selfMode || j > il);
          ++tests;
          if (!__any_sync(~0u, cand))
            continue;
          bool hit = false, sure = false;
          if (cand)
          {
            const float4 c0 = W.box[l][2], c1 = W.box[l][3];
            sure = (hi.x > c0.x) & (hi.y > c0.y) & (hi.z > c0.z) & (lo.x < c1.x) & (lo.y < c1.y) & (lo.z < c1.z);
            hit = sure;
            if (!sure)
            {
              hit = boxes_overlap_exact<T>(a.geomA + u64(il) * 6, a.geomB + u64(j) * 6, a.tol);
              ++rechecks;
            }
          }
          const u32 bal = __ballot_sync(~0u, hit);
          if (!bal)
            continue;
          if (nbuf + 32 > kPairBuf)
          {
            flush(nbuf);
            nbuf = 0;
          }
          if (hit)
          {
            const u64 mark = sure && a.sure ? kPairSure : 0;
            W.pairs[nbuf + __popc(bal & lt)] = (a.swapOut ? ((u64(j) << 32) | il) : ((u64(il) << 32) | j)) | mark;
          }
          nbuf += __popc(bal);
          __syncwarp();
        }
      }
      if (cc)
      {
        // the children's boxes and links
        float4 cl = make_float4(0.f, 0.f, 0.f, 0.f), ch = cl;
        uint4 cL = make_uint4(0u, 0u, 0u, 0u);
        if (lane < cc)
        {
          cl = a.nodeB[2 * size_t(fc + lane)];
          ch = a.nodeB[2 * size_t(fc + lane) + 1];
          cL = a.linkB[fc + lane];
          if (!a.sure)
            ch = make_float4(__fadd_ru(ch.x, a.tolHi), __fadd_ru(ch.y, a.tolHi), __fadd_ru(ch.z, a.tolHi), 0.f);
        }
        // the subtree must reach the packet's box, and in a single tree hold a position after its first
        const bool ok = lane < cc && !apart(W.common[0], W.common[1], cl, ch) && (!a.selfMode || cL.w > iMin + 1);
        u32 bal = __ballot_sync(~0u, ok);
        if (ok)
        {
          cl.w = __uint_as_float(cL.w);
          W.child[lane][0] = cl;
          W.child[lane][1] = ch;
        }
        __syncwarp();
        while (bal)
        {
          const u32 k = u32(__ffs(int(bal))) - 1;
          bal &= bal - 1;
          const float4 nl = W.child[k][0], nh = W.child[k][1];
          const bool keep = ((mask >> lane) & 1u) && !apart(n0, n1, nl, nh) && (!a.selfMode || __float_as_uint(nl.w) > i + 1);
          const u32 m = __ballot_sync(~0u, keep);
          if (m)
          {
            if (lane == k)
            {
              stackL[sp] = cL;
              stackM[sp] = m;
            }
            ++sp;
          }
        }
        __syncwarp();
      }
    }
    if (bad && lane == 0)
      atomicOr(a.err, kErrStack);
    if (nbuf)
      flush(nbuf);
    __syncwarp();
  }
  // a box test is one lane's: every lane counts the tests it took part in
  unsigned long long t = tests, r = rechecks;
  for (int o = 16; o > 0; o >>= 1)
  {
    t += __shfl_xor_sync(~0u, t, o);
    r += __shfl_xor_sync(~0u, r, o);
  }
  if (lane == 0)
  {
    atomicAdd(&a.ctr->tests, t);
    atomicAdd(&a.ctr->rechecks, r);
  }
}

// entities of nodes above depth `cut` come first in the order (sorted owner depths)
__global__ void collide_singles_kernel(const u32* __restrict__ keys, u32 n, u32 cut, u32* __restrict__ singles)
{
  u32 lo = 0, hi = n;
  while (lo < hi)
  {
    const u32 mid = (lo + hi) >> 1;
    if (keys[mid] < cut)
      lo = mid + 1;
    else
      hi = mid;
  }
  *singles = lo;
}

// processing order: entities of shallow nodes (large boxes, long walks) first
__global__ void owner_depth_key_kernel(const u32* __restrict__ owner, const unsigned char* __restrict__ depth, u64 n, u32* __restrict__ keys,
                                       u32* __restrict__ idx)
{
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < n; i += u64(gridDim.x) * blockDim.x)
  {
    const u32 o = owner[i];
    keys[i] = o == kNoOwner ? 31u : depth[o]; // entities in no node last (the collision skips them)
    idx[i] = u32(i);
  }
}

template<typename T, int WARPS>
static int launch_collide(const CollideArgs<T>& a, cudaStream_t st)
{
  const size_t smem = collide_warp_bytes(a.stackCap) * WARPS;
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (!e)
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!e)
    e = cudaFuncSetAttribute(collide_packet_kernel<T, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (!e)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, collide_packet_kernel<T, WARPS>, WARPS * 32, smem);
  if (e)
    return cuda_status(e, "configuring the collision kernel");
  const u32 grid = u32(std::max<u64>(1, std::min<u64>(u64(sms) * std::max(per, 1), (u64(a.nA) + WARPS - 1) / WARPS)));
  collide_packet_kernel<T, WARPS><<<grid, WARPS * 32, smem, st>>>(a);
  return cuda_status(cudaGetLastError(), "launching the collision kernel");
}

static u32 collide_packet_size(u64 n)
{
  u32 p = 32;
  while (p > 1 && n / p < kPacketsWanted)
    p >>= 1;
  return p;
}

template<typename T>
static int collide_search_impl(TreeState& A, TreeState& B, bool self, bool swapOut, double tol, Appender out, u32* err, CollideSearch& s,
                               cudaStream_t st)
{
  cudaError_t e;
  if (!s.ready)
  {
    if (int rc = ensure_image32(B, st, true))
      return rc;
    TmpBuf keys;
    if ((e = s.ctr.ensure(sizeof(CollideCounters) + sizeof(u32), st)) || (e = keys.ensure(sizeof(u32) * std::max<u64>(A.n, 1), st)) ||
        (e = s.order.ensure(sizeof(u32) * std::max<u64>(A.n, 1), st)))
      return cuda_status(e, "allocating the collision order");
    owner_depth_key_kernel<<<blocks_for(A.n), 256, 0, st>>>(A.ownerNode.as<u32>(), A.nodeDepth.as<unsigned char>(), A.n, keys.as<u32>(), s.order.as<u32>());
    if (int rc = sort_pairs_u32(keys.as<u32>(), s.order.as<u32>(), A.n, 5, st, err))
      return rc;
    // One to a packet above the depth whose cells hold 256 nodes of the walked tree on average: the
    // walks of such boxes are long, and 32 of them in one warp would end last.
    u32 cut = 0;
    while (cut < 19 && (B.nodeCount >> (3 * cut)) > 256)
      ++cut;
    collide_singles_kernel<<<1, 1, 0, st>>>(keys.as<u32>(), u32(A.n), cut, reinterpret_cast<u32*>(s.ctr.as<CollideCounters>() + 1));
    s.ready = true;
  }
  CollideArgs<T> a{};
  a.order = s.order.as<u32>();
  a.ownerA = A.ownerNode.as<u32>();
  a.singles = reinterpret_cast<const u32*>(s.ctr.as<CollideCounters>() + 1);
  a.rootA = A.nodeBox.as<T>();
  a.rootB = B.nodeBox.as<T>();
  a.geomA = A.sortedGeom.as<T>();
  a.nA = u32(A.n);
  a.imgB = B.boxImg32.as<float4>();
  a.geomB = B.sortedGeom.as<T>();
  a.linkB = B.nodeLink.as<uint4>();
  a.nodeB = B.nodeBox32.as<float4>();
  a.nB = u32(B.n);
  a.nNodesB = u32(B.nodeCount);
  // depth first: at most 7 entries per level beside the current node's 8 children
  a.stackCap = (7 * (B.D + 1) + 9 + 3) & ~3u;
  a.packet = collide_packet_size(A.n);
  a.tol = tol < 0 ? base_tol<T>() : T(tol);
  a.selfMode = self ? 1 : 0;
  a.swapOut = swapOut ? 1 : 0;
  a.sure = !A.respanned && !B.respanned;
  a.direct = a.sure ? kDirectBoxes : 0u;
  a.tolHi = float(a.tol);
  if (double(a.tolHi) < double(a.tol))
    a.tolHi = std::nextafter(a.tolHi, __builtin_huge_valf());
  a.out = out;
  a.ctr = s.ctr.as<CollideCounters>();
  a.err = err;
  return tune_run(tune_key(self ? "collide self" : "collide pair", sizeof(T) == 8, 1, B.n, A.n), { { 2, "warp x2" }, { 4, "warp x4" }, { 8, "warp x8" } }, 4,
                  st, [&](int shape) {
                    cudaMemsetAsync(s.ctr.p, 0, sizeof(CollideCounters), st);
                    cudaMemsetAsync(out.count, 0, sizeof(unsigned long long), st);
                    if (shape == 2)
                      return launch_collide<T, 2>(a, st);
                    if (shape == 8)
                      return launch_collide<T, 8>(a, st);
                    return launch_collide<T, 4>(a, st);
                  });
}

int collide_search_filtered(TreeState& A, TreeState& B, bool self, double tol, Appender out, u32* err, CollideSearch& s, cudaStream_t st)
{
  const bool swap = !self && B.n < A.n;
  TreeState& Q = swap ? B : A;
  TreeState& W = swap ? A : B;
  return A.scalar == OTG_SCALAR_F64 ? collide_search_impl<double>(Q, W, self, swap, tol, out, err, s, st)
                                    : collide_search_impl<float>(Q, W, self, swap, tol, out, err, s, st);
}

int collide_search_stats(const CollideSearch& s, u64& tests, u64& rechecks, cudaStream_t st)
{
  CollideCounters h{};
  if (cudaError_t e = read_back(&h, s.ctr.p, sizeof(h), st))
    return cuda_status(e, "reading collision statistics");
  tests = h.tests;
  rechecks = h.rechecks;
  return OTG_OK;
}

} // namespace otg
