// otg_ray.cu — RayIntersectedFirst (core/ot_query.h:2035-2146), one warp per ray, and the per-ray
// setup of the ray kernels.
//
// The result of a ray is every entity hit with enter <= M. M starts at maxDistance; walking the hit
// nodes depth first and their entities in tree order, each hit with enter <= M and exit < M sets
// M = f(exit), f(x) = (1 + tolInc) x + tol'. Where no other hit's exit lies in [x0, f(x0)), x0 the
// smallest exit among the hits with enter <= maxDistance and exit < maxDistance, the walk ends with
// M = f(x0) in any order. The two kernels:
//   ray_first_near_kernel  walks nearest node first with a shrinking bound, so a ray sees the few
//                          nodes before its first hits instead of every node it meets. It finds x0,
//                          and checks that no other exit lies in [x0, f(x0)) (such a hit also has
//                          enter < f(x0), so it is among the candidates). Rays that fail the check,
//                          or whose candidates overflow the buffer, go to a list.
//   ray_first_walk_kernel  the walk itself, in its order, for the listed rays (or for every ray of a
//                          tree that the first kernel does not take): nodes and entities are tested
//                          32 at a time, and the updates of M are applied one after another.
// Bound by the latency of dependent node loads and by issue, on data that sits in L2. 30k rays through
// 1M FP64 boxes: 0.16 ms for the near kernel and 4 us for the (empty) list, where the two kernels with
// one ray per thread, which OTG_ALGO_PLAIN_FP64 keeps, take 24.8 + 1.9 ms: their walk meets the nodes
// in tree order, so the bound comes late, and each lane reads its own node.
#include "otg_ray.cuh"

#include <cmath>

namespace otg
{

__global__ void __launch_bounds__(128) ray_prepare_kernel(const double* __restrict__ rays, u64 nq, double tol, double tolInc, RayPrep* __restrict__ out)
{
  for (u64 q = blockIdx.x * u64(blockDim.x) + threadIdx.x; q < nq; q += u64(gridDim.x) * blockDim.x)
  {
    RayD<double> r;
    r.make(rays + q * 6, rays + q * 6 + 3, tol, tolInc);
    RayPrep p;
    bool ok = tol >= 0.0 && tol < 1e30 && tolInc >= 0.0 && tolInc <= 1.0;
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
      p.inv[d] = r.inv[d];
      p.o[d] = __double2float_rn(r.origin[d]);
      p.invf[d] = __double2float_rn(r.inv[d]);
      p.S[d] = fmaf(fabsf(p.o[d]), 0x1p-21f, 0x1p-140f);
      ok &= isfinite(p.o[d]) && isfinite(p.invf[d]);
    }
    p.flags = r.sign | (r.zero << 3) | (r.valid ? kRayValid : 0u) | (ok ? kRayF32 : 0u);
    out[q] = p;
  }
}

int ray_prepare(const double* rays, u64 nq, double tol, double tolInc, RayPrep* out, cudaStream_t st)
{
  ray_prepare_kernel<<<u32(std::min<u64>((nq + 127) / 128, 152 * 16)), 128, 0, st>>>(rays, nq, tol, tolInc, out);
  return cuda_status(cudaGetLastError(), "preparing rays");
}

constexpr int kFirstWarps = 4;
constexpr u32 kFirstCand = 128;

template<typename T>
struct RayFirstArgs
{
  TreeView<T> tv;
  const T* rays;
  const RayPrep* prep; // FP64 trees with images; null: exact tests only
  u32 nq;
  T tol, tolInc, maxDist;
  float tolUp, tolIncUp;
  float maxLo, maxHi; // maxDist rounded down and up
  Appender out;
  u32* work;       // {next ray, listed rays, next listed ray, 0}, then the list
  const u32* list; // null: every ray
  u32* err;
};

// f(exit) of an upper bound of the exit, rounded up (0 <= tolInc <= 1, x >= 0)
__device__ __forceinline__ float bound_up(float x, float tolIncUp, float appliedUp)
{
  const float v = fmaf(x, tolIncUp, x) + appliedUp;
  return x < INFINITY ? v + v * 0x1p-20f : INFINITY; // (INFINITY times 0 is not a number)
}

// bounds of a ray's enter and exit for node or entity `i`: FP32 on the images (FP64 trees), else exact
template<typename T, bool NODE>
__device__ __forceinline__ RayBounds first_bounds(const RayFirstArgs<T>& a, const RayF32& f, const RayD<T>& ray, u32 i)
{
  if constexpr (sizeof(T) == 8)
  {
    const float4* img = NODE ? a.tv.nodeImg : a.tv.boxImg;
    return ray_box_f32(f, a.tolUp, a.tolIncUp, img[2 * size_t(i)], img[2 * size_t(i) + 1]);
  }
  else
  {
    T en = 0, ex = 0;
    const T* g = (NODE ? a.tv.nodeBox : a.tv.geom) + u64(i) * 6;
    const bool hit = NODE ? ray.hit_node(g, g + 3, en, ex) : ray.hit_box(g, en, ex);
    return RayBounds{ hit ? 1 : 0, float(en), float(en), float(ex) };
  }
}

template<typename T>
__global__ void __launch_bounds__(kFirstWarps * 32) ray_first_near_kernel(RayFirstArgs<T> a)
{
  constexpr bool kF32 = sizeof(T) == 8;
  __shared__ u32 stackNode[kFirstWarps][kStack];
  __shared__ float stackEn[kFirstWarps][kStack];
  __shared__ u32 candPos[kFirstWarps][kFirstCand];
  __shared__ float candEn[kFirstWarps][kFirstCand];
  __shared__ T hitEn[kFirstWarps][kFirstCand];
  __shared__ RayF32 rayF[kF32 ? kFirstWarps : 1];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u32 lt = (1u << lane) - 1u;
  const TreeView<T>& tv = a.tv;
  const T applied = a.tol == T(0) ? Lim<T>::eps() : a.tol;
  const float appliedUp = fmaxf(a.tolUp, float(Lim<T>::eps()) * (1.f + 0x1p-20f));
  for (;;)
  {
    u32 q = 0;
    if (lane == 0)
      q = atomicAdd(a.work, 1u);
    q = __shfl_sync(~0u, q, 0);
    if (q >= a.nq)
      break;
    RayD<T> ray;
    bool usable;
    if constexpr (kF32)
    {
      const u32 flags = a.prep[q].flags;
      if (!(flags & kRayValid))
        continue;
      usable = (flags & kRayF32) != 0;
      __syncwarp(); // the previous ray's setup is read by every lane before it changes
      if (lane == 0)
        ray_f32_of(a.prep[q], rayF[w]);
      __syncwarp();
    }
    else
    {
      ray.make(a.rays + u64(q) * 6, a.rays + u64(q) * 6 + 3, a.tol, a.tolInc);
      if (!ray.valid)
        continue;
      usable = a.tol >= T(0) && a.tolInc >= T(0) && a.tolInc <= T(1);
    }
    const RayF32& f = rayF[kF32 ? w : 0];
    const u32 root = query_root(tv, q), idBase = id_base(tv, root);
    // an upper bound of the final M: maxDistance, or f of an exit below it
    float Mf = bound_up(a.maxHi, a.tolIncUp, appliedUp);
    u32 nc = 0, visits = 0;
    int sp = 0;
    bool give = !usable, bad = false; // give: this ray to the walk kernel
    if (!give)
    {
      const RayBounds b = first_bounds<T, true>(a, f, ray, root);
      bool in = b.rel != 0;
      if constexpr (kF32)
        if (b.rel == 2)
        {
          double en, ex;
          in = ray_node_exact(a.rays + u64(q) * 6, a.prep + q, tv.nodeBox + u64(root) * 6, a.tol, a.tolInc, en, ex);
        }
      if (in && b.enLo <= Mf)
      {
        if (lane == 0)
        {
          stackNode[w][0] = root;
          stackEn[w][0] = b.enLo;
        }
        sp = 1;
      }
    }
    __syncwarp();
    while (sp > 0)
    {
      --sp;
      const u32 node = stackNode[w][sp];
      const float nodeEn = stackEn[w][sp];
      __syncwarp();
      if (nodeEn > Mf)
        continue;
      const uint4 L = tv.link[node];
      const u32 fc = L.x & kFirstChildMask, cc = L.x >> kChildShift;
      if (L.z > tv.n || L.w > tv.n || L.y > L.z || ++visits > tv.nNodes || cc > 8u || u64(fc) + cc > tv.nNodes || sp + int(cc) > kStack)
      {
        bad = true;
        break;
      }
      for (u32 base = L.y; base < L.z; base += 32)
      {
        const u32 e = base + lane;
        RayBounds b{ 0, 0.f, 0.f, 0.f };
        if (e < L.z)
          b = first_bounds<T, false>(a, f, ray, e);
        // a certain hit bounds M
        float up = INFINITY;
        if (b.rel == 1 && b.enHi <= a.maxLo && b.exHi < a.maxLo)
          up = bound_up(fmaxf(b.exHi, 0.f), a.tolIncUp, appliedUp);
        if (__any_sync(~0u, up < Mf))
        {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
            up = fminf(up, __shfl_xor_sync(~0u, up, o));
          Mf = fminf(Mf, up);
        }
        const bool keep = b.rel != 0 && b.enLo <= Mf;
        const u32 bal = __ballot_sync(~0u, keep);
        if (!bal)
          continue;
        if (nc + __popc(bal) > kFirstCand)
        {
          // drop the candidates that the bound has passed
          u32 kept = 0;
          for (u32 i0 = 0; i0 < nc; i0 += 32)
          {
            const u32 i = i0 + lane;
            const u32 p = i < nc ? candPos[w][i] : 0u;
            const float en = i < nc ? candEn[w][i] : INFINITY;
            const bool k = i < nc && en <= Mf;
            const u32 kb = __ballot_sync(~0u, k);
            if (k)
            {
              candPos[w][kept + __popc(kb & lt)] = p;
              candEn[w][kept + __popc(kb & lt)] = en;
            }
            kept += __popc(kb);
            __syncwarp();
          }
          nc = kept;
          if (nc + __popc(bal) > kFirstCand)
          {
            give = true;
            break;
          }
        }
        if (keep)
        {
          candPos[w][nc + __popc(bal & lt)] = e;
          candEn[w][nc + __popc(bal & lt)] = b.enLo;
        }
        nc += __popc(bal);
        __syncwarp();
      }
      if (give)
        break;
      if (cc)
      {
        // the children that the ray enters before the bound, the nearest on top of the stack
        bool in = false;
        float en = INFINITY;
        if (lane < cc)
        {
          const RayBounds b = first_bounds<T, true>(a, f, ray, fc + lane);
          in = b.rel != 0 && b.enLo <= Mf;
          en = b.enLo;
          if constexpr (kF32)
            if (in && b.rel == 2)
            {
              double x, y;
              in = ray_node_exact(a.rays + u64(q) * 6, a.prep + q, tv.nodeBox + u64(fc + lane) * 6, a.tol, a.tolInc, x, y);
            }
        }
        const u32 bal = __ballot_sync(~0u, in);
        u32 rank = 0;
        for (u32 j = 0; j < cc; ++j)
        {
          const float ej = __shfl_sync(~0u, en, j);
          if (((bal >> j) & 1u) && (ej > en || (ej == en && j > lane)))
            ++rank;
        }
        if (in)
        {
          stackNode[w][sp + rank] = fc + lane;
          stackEn[w][sp + rank] = en;
        }
        sp += __popc(bal);
        __syncwarp();
      }
    }
    if (bad)
    {
      if (lane == 0)
        atomicOr(a.err, kErrStack);
      __syncwarp();
      continue;
    }
    if (!give)
    {
      // the candidates' exact enter and exit, 32 at a time; a candidate the exact test misses gets
      // an enter above every bound
      T x0 = Lim<T>::max(), x1 = Lim<T>::max(); // the least exit that counts; the least other exit above it
      bool any = false;
      T exs[kFirstCand / 32];
#pragma unroll
      for (u32 k = 0; k < kFirstCand / 32; ++k)
      {
        exs[k] = Lim<T>::max();
        const u32 i = k * 32 + lane;
        if (i < nc)
        {
          T en = 0, ex = 0;
          bool hit;
          const T* g = tv.geom + u64(candPos[w][i]) * 6;
          if constexpr (kF32)
            hit = ray_box_exact(a.rays + u64(q) * 6, a.prep + q, g, a.tol, a.tolInc, en, ex);
          else
            hit = ray.hit_box(g, en, ex);
          hitEn[w][i] = hit ? en : T(INFINITY);
          if (hit)
          {
            exs[k] = ex;
            if (en <= a.maxDist && ex < a.maxDist)
            {
              any = true;
              x0 = ex < x0 ? ex : x0;
            }
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
      {
        const T y = __shfl_xor_sync(~0u, x0, o);
        x0 = y < x0 ? y : x0;
      }
      any = __any_sync(~0u, any);
      const T M = any ? (T(1) + a.tolInc) * x0 + applied : a.maxDist;
      if (any)
      {
#pragma unroll
        for (u32 k = 0; k < kFirstCand / 32; ++k)
          if (exs[k] != x0 && exs[k] < x1)
            x1 = exs[k];
        give = __any_sync(~0u, x1 < M);
      }
      if (!give)
      {
        __syncwarp();
        u32 total = 0;
        for (u32 i0 = 0; i0 < nc; i0 += 32)
          total += __popc(__ballot_sync(~0u, i0 + lane < nc && hitEn[w][i0 + lane] <= M));
        unsigned long long at = 0;
        if (lane == 0 && total)
          at = a.out.reserve(total);
        at = __shfl_sync(~0u, at, 0);
        for (u32 i0 = 0; i0 < nc; i0 += 32)
        {
          const bool k = i0 + lane < nc && hitEn[w][i0 + lane] <= M;
          const u32 bal = __ballot_sync(~0u, k);
          const u64 to = at + __popc(bal & lt);
          if (k && to < a.out.capacity)
          {
            a.out.items[to] = (u64(q) << 32) | (tv.ids[candPos[w][i0 + lane]] - idBase);
            a.out.dist[to] = double(hitEn[w][i0 + lane]);
          }
          at += __popc(bal);
        }
      }
    }
    if (give && lane == 0)
      a.work[4 + atomicAdd(a.work + 1, 1u)] = q; // at most nq rays are listed
    __syncwarp();
  }
}

// the exact enter and exit of node or entity `i`, with the FP32 tests sparing the certain misses
template<typename T, bool NODE>
__device__ __forceinline__ bool walk_hit(const RayFirstArgs<T>& a, const RayF32& f, bool useF32, const RayD<T>& ray, u32 q, u32 i, T& en, T& ex)
{
  if constexpr (sizeof(T) == 8)
    if (a.prep)
    {
      if (useF32)
      {
        const float4* img = NODE ? a.tv.nodeImg : a.tv.boxImg;
        if (ray_box_f32(f, a.tolUp, a.tolIncUp, img[2 * size_t(i)], img[2 * size_t(i) + 1]).rel == 0)
          return false;
      }
      return NODE ? ray_node_exact(a.rays + u64(q) * 6, a.prep + q, a.tv.nodeBox + u64(i) * 6, a.tol, a.tolInc, en, ex)
                  : ray_box_exact(a.rays + u64(q) * 6, a.prep + q, a.tv.geom + u64(i) * 6, a.tol, a.tolInc, en, ex);
    }
  if (NODE)
    return ray.hit_node(a.tv.nodeBox + u64(i) * 6, a.tv.nodeBox + u64(i) * 6 + 3, en, ex);
  return a.tv.isBox ? ray.hit_box(a.tv.geom + u64(i) * 6, en, ex) : ray.hit_point(a.tv.geom + u64(i) * 3, en, ex);
}

template<typename T>
__global__ void __launch_bounds__(kFirstWarps * 32) ray_first_walk_kernel(RayFirstArgs<T> a)
{
  constexpr bool kF32 = sizeof(T) == 8;
  __shared__ u32 stackNode[kFirstWarps][kStack];
  __shared__ T stackEn[kFirstWarps][kStack];
  __shared__ RayF32 rayF[kF32 ? kFirstWarps : 1];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u32 lt = (1u << lane) - 1u;
  const TreeView<T>& tv = a.tv;
  const T applied = a.tol == T(0) ? Lim<T>::eps() : a.tol;
  const u32 total = a.list ? min(a.work[1], a.nq) : a.nq;
  for (;;)
  {
    u32 item = 0;
    if (lane == 0)
      item = atomicAdd(a.work + 2, 1u);
    item = __shfl_sync(~0u, item, 0);
    if (item >= total)
      break;
    const u32 q = a.list ? a.list[item] : item;
    RayD<T> ray;
    bool useF32 = false, made = false;
    if constexpr (kF32)
      if (a.prep)
      {
        const u32 flags = a.prep[q].flags;
        if (!(flags & kRayValid))
          continue;
        useF32 = (flags & kRayF32) != 0;
        __syncwarp(); // the previous ray's setup is read by every lane before it changes
        if (lane == 0)
          ray_f32_of(a.prep[q], rayF[w]);
        __syncwarp();
        made = true;
      }
    if (!made)
    {
      ray.make(a.rays + u64(q) * 6, a.rays + u64(q) * 6 + 3, a.tol, a.tolInc);
      if (!ray.valid)
        continue;
    }
    const RayF32& f = rayF[kF32 ? w : 0];
    const u32 root = query_root(tv, q), idBase = id_base(tv, root);
    T M = a.maxDist;
    bool bad = false;
    // two walks: the updates of M, then every hit with enter <= M
    for (int pass = 0; pass < 2 && !bad; ++pass)
    {
      u32 visits = 0;
      int sp = 0;
      {
        T en = 0, ex = 0;
        const bool in = walk_hit<T, true>(a, f, useF32, ray, q, root, en, ex) && !(en > M);
        if (in && lane == 0)
        {
          stackNode[w][0] = root;
          stackEn[w][0] = en;
        }
        sp = in ? 1 : 0;
      }
      __syncwarp();
      while (sp > 0)
      {
        --sp;
        const u32 node = stackNode[w][sp];
        const T nodeEn = stackEn[w][sp];
        __syncwarp();
        if (nodeEn > M)
          continue;
        const uint4 L = tv.link[node];
        const u32 fc = L.x & kFirstChildMask, cc = L.x >> kChildShift;
        if (L.z > tv.n || L.w > tv.n || L.y > L.z || ++visits > tv.nNodes || cc > 8u || u64(fc) + cc > tv.nNodes || sp + int(cc) > kStack)
        {
          bad = true;
          break;
        }
        for (u32 base = L.y; base < L.z; base += 32)
        {
          const u32 e = base + lane;
          T en = 0, ex = 0;
          const bool hit = e < L.z && walk_hit<T, false>(a, f, useF32, ray, q, e, en, ex);
          if (pass == 0)
          {
            // the updates of these entities, in their order
            u32 rest = ~0u;
            for (;;)
            {
              const u32 bal = __ballot_sync(~0u, hit && !(en > M) && !(ex >= M)) & rest;
              if (!bal)
                break;
              const int first = __ffs(int(bal)) - 1;
              M = (T(1) + a.tolInc) * __shfl_sync(~0u, ex, first) + applied;
              rest = first == 31 ? 0u : ~0u << (first + 1);
            }
          }
          else
          {
            const bool k = hit && !(en > M);
            const u32 bal = __ballot_sync(~0u, k);
            if (bal)
            {
              unsigned long long at = 0;
              if (lane == 0)
                at = a.out.reserve(__popc(bal));
              at = __shfl_sync(~0u, at, 0) + __popc(bal & lt);
              if (k && at < a.out.capacity)
              {
                a.out.items[at] = (u64(q) << 32) | (tv.ids[e] - idBase);
                a.out.dist[at] = double(en);
              }
            }
          }
        }
        if (cc)
        {
          T en = 0, ex = 0;
          const bool in = lane < cc && walk_hit<T, true>(a, f, useF32, ray, q, fc + lane, en, ex) && !(en > M && pass == 1);
          const u32 bal = __ballot_sync(~0u, in);
          if (in)
          {
            stackNode[w][sp + __popc(bal & lt)] = fc + lane;
            stackEn[w][sp + __popc(bal & lt)] = en;
          }
          sp += __popc(bal);
          __syncwarp();
        }
      }
    }
    if (bad && lane == 0)
      atomicOr(a.err, kErrStack);
    __syncwarp();
  }
}

template<typename K>
static int first_grid(K kernel, u64 nq, u32& grid)
{
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (!e)
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!e)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kFirstWarps * 32, 0);
  if (e)
    return cuda_status(e, "configuring the ray kernel");
  grid = u32(std::max<u64>(1, std::min<u64>(u64(sms) * std::max(per, 1), (nq + kFirstWarps - 1) / kFirstWarps)));
  return OTG_OK;
}

size_t ray_first_work_bytes(u64 nq) { return sizeof(u32) * (4 + nq); }

template<typename T>
int ray_first(const TreeView<T>& tv, bool near, const T* rays, u32 nq, T tol, T tolInc, T maxDist, Appender out, u32* work, u32* err, cudaStream_t st)
{
  RayFirstArgs<T> a{ tv, rays, nullptr, nq, tol, tolInc, maxDist, float_ru_host(double(tol)), float_ru_host(double(tolInc)) };
  a.maxHi = float_ru_host(double(maxDist));
  a.maxLo = -float_ru_host(-double(maxDist));
  a.out = out;
  a.work = work;
  a.err = err;
  TmpBuf prep;
  if constexpr (sizeof(T) == 8)
  {
    if (tv.nodeImg && tv.boxImg)
    {
      if (cudaError_t e = prep.ensure(sizeof(RayPrep) * nq, st))
        return cuda_status(e, "allocating the ray setup");
      if (int rc = ray_prepare(rays, nq, double(tol), double(tolInc), prep.as<RayPrep>(), st))
        return rc;
      a.prep = prep.as<RayPrep>();
    }
    near = near && a.prep;
  }
  if (!out.cleared)
    cudaMemsetAsync(work, 0, sizeof(u32) * 4, st);
  u32 grid = 0;
  if (near)
  {
    if (int rc = first_grid(ray_first_near_kernel<T>, nq, grid))
      return rc;
    ray_first_near_kernel<T><<<grid, kFirstWarps * 32, 0, st>>>(a);
    a.list = work + 4;
  }
  if (int rc = first_grid(ray_first_walk_kernel<T>, nq, grid))
    return rc;
  ray_first_walk_kernel<T><<<grid, kFirstWarps * 32, 0, st>>>(a);
  return cuda_status(cudaGetLastError(), "launching the first-hit kernels");
}

template int ray_first<double>(const TreeView<double>&, bool, const double*, u32, double, double, double, Appender, u32*, u32*, cudaStream_t);
template int ray_first<float>(const TreeView<float>&, bool, const float*, u32, float, float, float, Appender, u32*, u32*, cudaStream_t);

} // namespace otg
