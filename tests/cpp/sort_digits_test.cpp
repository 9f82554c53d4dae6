// The digits of radix_plan put keys in the order of their values: the passes' digits, last pass
// first, compare as the keys do, for box keys of every depth (with the cells outside the grid and
// the depth -1 of a box larger than its space) and for plain keys of every width.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline
namespace otg
{
using u32 = std::uint32_t;
using u64 = std::uint64_t;
}
#include "otg_radix.h"
using namespace otg;

template<typename K, bool GAP>
static u64 rank_value(const RadixPlan& p, K k)
{
  u64 v = 0;
  for (u32 i = p.passes; i-- > 0;)
  {
    const bool g = GAP && p.digit[i].keep != 0;
    const u32 d = p.radix == u32(kRadix) ? (g ? p.digit[i].of<kRadix, true>(k) : p.digit[i].of<kRadix, false>(k))
                                         : (g ? p.digit[i].of<kRadixWide, true>(k) : p.digit[i].of<kRadixWide, false>(k));
    if (d >= p.radix)
      std::printf("digit out of range\n"), std::exit(1);
    v = v * p.radix + d;
  }
  return v;
}

template<typename K, bool GAP>
static int check(const RadixPlan& p, std::vector<K> keys)
{
  std::sort(keys.begin(), keys.end());
  for (size_t i = 1; i < keys.size(); ++i)
  {
    const u64 a = rank_value<K, GAP>(p, keys[i - 1]), b = rank_value<K, GAP>(p, keys[i]);
    if (keys[i - 1] == keys[i] ? a != b : a >= b)
      return 1;
  }
  return 0;
}

int main()
{
  std::mt19937_64 g(7);
  for (u32 D = 1; D <= 8; ++D)
  {
    u32 low = 1;
    while ((D >> low) != 0)
      ++low;
    const u32 bits = std::min(3 * D + 8, 32u);
    const RadixPlan p = radix_plan(bits, low, 5 - low, true);
    std::vector<u32> keys;
    for (int i = 0; i < 20000; ++i)
    {
      const u64 cells = i % 2 ? u64(1) << (3 * D) : u64(1) << std::min(3 * D + 3, 27u);
      // no cell has all bits above the grid's and all bits of the grid
      const u64 loc = std::min<u64>(g() % cells, (u64(1) << std::min(3 * D + 3, 27u)) - 2);
      keys.push_back(u32(loc << 5 | g() % (D + 1)));
    }
    keys.push_back(0xffffffffu);
    if (check<u32, true>(p, keys))
      return std::printf("box keys of depth %u\n", D), 1;
  }
  for (u32 bits = 1; bits <= 64; ++bits)
  {
    const u64 all = bits == 64 ? ~u64(0) : (u64(1) << bits) - 1;
    std::vector<u64> keys{ 0, all };
    std::vector<u32> narrow{ 0, u32(all) };
    for (int i = 0; i < 5000; ++i)
    {
      keys.push_back(g() & all);
      narrow.push_back(u32(g() & all));
    }
    const RadixPlan p = radix_plan(bits, 0, 0, false);
    if (bits <= 63 && check<u64, false>(p, keys))
      return std::printf("64-bit keys of %u bits\n", bits), 1;
    if (bits <= 32 && check<u32, false>(radix_plan(bits, 0, 0, true), narrow))
      return std::printf("32-bit keys of %u bits\n", bits), 1;
  }
  std::printf("ok\n");
  return 0;
}
