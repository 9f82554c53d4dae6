// otg_ray.cuh — FP32 tests of rays against boxes of FP64 trees.
//
// The exact test (RayD, detail/internal_geometry_module.h:536-723) takes about 30 FP64 operations per
// box, and this GPU's FP64 rate is a sixtieth of its FP32 rate. The tests below bound its enter and
// exit values in FP32 on outward-rounded box images and decide most boxes; only undecided nodes, and
// entities that may be hit (their distance is a result), take the exact test. RayIntersectedAll, 30k
// rays through 1M FP64 boxes (2.25M hits): 3.45 ms with exact tests only, 0.44 ms with these.
//
// Bounds. With u = 2^-24: the image holds lo = rd(min) and hi = ru(max); o32 = RN(o) and inv32 = RN(inv)
// are within u of their values; S = 2^-21 |o| + 2^-140 per dimension. The near face moved out by S,
//   tn = RN(RN(RN(near -+ S) - o32) inv32),
// is within 8u |tn| of a bound of the exact near distance: the rounding of near -+ S is at most
// u(|near - o32| + |o32| + S), of which the last two terms are below S / 2, and the rest are relative
// roundings. (A node's max is RN(min + size) in the exact test, within 2^-52 (|o| + |max - o|) of the
// image's exact max: also covered.) So tn - 2^-19 |tn| is a lower bound of the exact near distance, and
// with K = (4 S + 2^-21 max(|near|, |far|)) |inv32|, which spans the move and the image's own rounding
// twice, tn + 2^-19 |tn| + K is an upper bound; the far face likewise. The tolerance terms
// 0.5 (max(0, x) tolInc + tol) are monotone for 0 <= tolInc <= 1 and are rounded outward; other
// tolerances (and rays outside the FP32 range) leave every box undecided.
// NaN coordinates drop out of fminf / fmaxf as they drop out of the exact test's comparisons.
#pragma once

#include "otg_query.cuh"

namespace otg
{

// one ray's setup, made by one thread (an FP64 instruction of a warp costs the same for one lane)
struct RayPrep
{
  double inv[3];
  float o[3], invf[3], S[3];
  u32 flags; // bits 0-2: direction < 0; 3-5: direction treated as zero; 6: normalised; 7: FP32 tests usable
};
static_assert(sizeof(RayPrep) == 64, "RayPrep: 16 words");
constexpr u32 kRayValid = 1u << 6, kRayF32 = 1u << 7;

struct RayF32
{
  float o[3], inv[3], S[3];
  u32 flags;
};

// the exact ray from its setup (hit_box and hit_node; the direction itself is only read by hit_point)
__device__ __forceinline__ RayD<double> ray_exact(const double* __restrict__ q, const RayPrep& p, double tol, double tolInc)
{
  RayD<double> r;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    r.origin[d] = q[d];
    r.dir[d] = q[3 + d];
    r.inv[d] = p.inv[d];
  }
  r.minTol = tol;
  r.tolInc = tolInc;
  r.sign = p.flags & 7u;
  r.zero = (p.flags >> 3) & 7u;
  r.valid = (p.flags & kRayValid) != 0;
  return r;
}

struct RayBounds
{
  int rel; // 0 certainly missed, 1 certainly hit, 2 undecided
  float enLo, enHi, exHi; // of the exact enter and exit where the box is hit
};

// tolf, tif: tol and tolInc rounded up
__device__ __forceinline__ RayBounds ray_box_f32(const RayF32& r, float tolf, float tif, float4 lo4, float4 hi4)
{
  constexpr float c = 0x1p-19f;
  const float lo[3] = { lo4.x, lo4.y, lo4.z }, hi[3] = { hi4.x, hi4.y, hi4.z };
  float enL = -INFINITY, enH = -__FLT_MAX__, exH = INFINITY, exL = __FLT_MAX__;
  float zA = -INFINITY, zB = INFINITY;
  bool zIn = true;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    const bool neg = (r.flags >> d) & 1u;
    const float S = r.S[d], o = r.o[d];
    const float W = fmaf(fmaxf(fabsf(lo[d]), fabsf(hi[d])), 0x1p-21f, 4.f * S);
    if ((r.flags >> (3 + d)) & 1u)
    {
      const float a = (lo[d] - S) - o, b = (hi[d] + S) - o;
      zA = fmaxf(zA, fmaf(-fabsf(a), c, a));
      zB = fminf(zB, fmaf(fabsf(b), c, b));
      zIn &= (a + W <= 0.f) & (b - W >= 0.f);
      continue;
    }
    const float inv = r.inv[d];
    const float K = W * fabsf(inv);
    const float tn = ((neg ? hi[d] + S : lo[d] - S) - o) * inv;
    const float tf = ((neg ? lo[d] - S : hi[d] + S) - o) * inv;
    const float en = fabsf(tn) * c, ef = fabsf(tf) * c;
    enL = fmaxf(enL, tn - en);
    enH = fmaxf(enH, (tn + en) + K);
    exH = fminf(exH, tf + ef);
    exL = fminf(exL, (tf - ef) - K);
  }
  const float g = fmaf(fmaxf(enL, 0.f), tif, tolf), x = fmaf(fmaxf(exH, 0.f), tif, tolf);
  const float L = (enL - 0.5f * g) - (fabsf(enL) + g) * 0x1p-20f;
  const float X = (exH + 0.5f * x) + (fabsf(exH) + x) * 0x1p-20f;
  const float xt = x + x * 0x1p-20f;
  const bool miss = (L >= X) | (X <= 0.f) | (zA > xt) | (zB < -xt);
  const bool hit = (enH < exL) & (exL > 0.f) & zIn;
  return RayBounds{ miss ? 0 : (hit ? 1 : 2), fmaxf(L, 0.f), fmaxf(enH, 0.f), X };
}

__device__ __forceinline__ void ray_f32_of(const RayPrep& p, RayF32& f)
{
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    f.o[d] = p.o[d];
    f.inv[d] = p.invf[d];
    f.S[d] = p.S[d];
  }
  f.flags = p.flags;
}

// The exact tests, out of line: inlined, the compiler may evaluate their FP64 arithmetic beside the
// FP32 tests.
static __device__ __noinline__ bool ray_node_exact(const double* q, const RayPrep* p, const double* nb, double tol, double tolInc, double& en, double& ex)
{
  return ray_exact(q, *p, tol, tolInc).hit_node(nb, nb + 3, en, ex);
}
static __device__ __noinline__ bool ray_box_exact(const double* q, const RayPrep* p, const double* box, double tol, double tolInc, double& en, double& ex)
{
  return ray_exact(q, *p, tol, tolInc).hit_box(box, en, ex);
}

// the setup of nq rays (device pointers), one thread each (otg_ray.cu)
int ray_prepare(const double* rays, u64 nq, double tol, double tolInc, RayPrep* out, cudaStream_t st);
// RayIntersectedFirst (otg_ray.cu). near: the entities lie in their nodes (a box tree with the geometry
// that it was built from). work: ray_first_work_bytes(nq) of device memory.
template<typename T>
int ray_first(const TreeView<T>& tv, bool near, const T* rays, u32 nq, T tol, T tolInc, T maxDist, Appender out, u32* work, u32* err, cudaStream_t st);
size_t ray_first_work_bytes(u64 nq);
// a double as a float that is not below it
static inline float float_ru_host(double v)
{
  float f = float(v);
  if (double(f) < v)
    f = std::nextafter(f, __builtin_huge_valf());
  return f;
}

} // namespace otg
