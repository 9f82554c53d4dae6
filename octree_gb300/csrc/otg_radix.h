// otg_radix.h — which key bits each pass of the radix sort (otg_sort.cuh) takes.
#pragma once

namespace otg
{
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kRadixWide = 2 * kRadix; // digits of the wide passes
constexpr u32 kMaxPasses = 8;

// A pass's digit of a key: a shifted field, and (GAP, a first pass only) the key's lowest bits kept in place below it.
struct SortDigit
{
  u32 keep, shift;
  template<int RADIX, bool GAP, typename K>
  __host__ __device__ __forceinline__ u32 of(K k) const
  {
    const u32 f = u32(k >> shift) & u32(RADIX - 1);
    return GAP ? (u32(k) & keep) | (f & ~keep) : f;
  }
};
struct RadixPlan
{
  u32 radix, passes; // digits per pass; every pass's digits are below radix
  SortDigit digit[kMaxPasses];
};

// The digits of a sort by `bits` key bits of which bits [low, low + gap) say nothing (gap 0: none). A box key
// ends in a depth of five bits that is at most D, so only its lowest bits are sorted by: 26 key bits of
// depth 6 are 24, three passes instead of four (8M FP64 boxes: 0.24 ms of passes, then 0.19). Nine-bit digits (wide)
// where they save a pass: a pass of them costs a tenth more (512 counters per warp instead of 256, more
// statuses, and three blocks still fit an SM): 65.8M boxes of a forest of depth 4, 18 bits, 1.13 ms in three passes, 0.78 in two.
inline RadixPlan radix_plan(u32 bits, u32 low, u32 gap, bool wideAllowed)
{
  RadixPlan r = {};
  const u32 left = bits - gap;
  const u32 narrow = (left + kRadixBits - 1) / kRadixBits, wide = (left + kRadixBits) / (kRadixBits + 1);
  const bool w = wideAllowed && wide < narrow;
  r.radix = w ? kRadixWide : kRadix;
  r.passes = w ? wide : narrow;
  u32 at = 0; // first sorted bit of the pass
  for (u32 p = 0; p < r.passes; ++p)
  {
    r.digit[p].keep = p == 0 && gap ? (1u << low) - 1 : 0u;
    r.digit[p].shift = at + gap;
    at += w ? kRadixBits + 1 : kRadixBits;
  }
  return r;
}
} // namespace otg
