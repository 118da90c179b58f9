// Which levels' block ILU substitutions run in one thread-block cluster
// (k_ilu_cluster), and on how many CTAs: plain host rules, without CUDA, so that
// they can be checked at their limits without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace gb {

constexpr size_t kIluClusterBytes = 216 * 1024; // of y in a CTA's shared memory
constexpr size_t kIluZeroBytes = 32;            // and of the zeros behind the CTA's rows
constexpr int kIluRowsPerLevel = 32;            // a CTA's share of an average level
constexpr int kIluOwnerShift = 24;
constexpr int kIluPlaceMask = (1 << kIluOwnerShift) - 1;

// CTA r of `ctas` owns the rows [r chunk, (r + 1) chunk); ctas 0: the level's rows
// do not fit a cluster. fp64: FP64 substitutions fit it too; FP32 ones always do.
// The packed factors are made for what fits, and only that is launched.
struct IluPlan
{
  int ctas = 0, chunk = 0;
  bool fp64 = false;
  size_t value_bytes() const { return fp64 ? 8 : 4; } // of the widest that fits
};

// n rows of B components in nlev dependency levels, clusters of up to `most`
// CTAs: the smallest power of two whose shared memory holds y and in which a level
// of average width gives each CTA at most kIluRowsPerLevel rows.
inline IluPlan
ilu_plan(int64_t n, int B, int nlev, int most)
{
  IluPlan P;
  if ((n + 1) * B >= (int64_t(1) << kIluOwnerShift))
    return P;
  auto bytes = [&](int ctas, size_t size) { return size_t((n + ctas - 1) / ctas) * B * size; };
  P.fp64 = bytes(most, 8) <= kIluClusterBytes;
  const size_t size = P.value_bytes();
  if (bytes(most, size) > kIluClusterBytes)
    return IluPlan();
  int ctas = 1;
  while (ctas < most && (bytes(ctas, size) > kIluClusterBytes ||
                         n > int64_t(ctas) * nlev * kIluRowsPerLevel))
    ctas *= 2;
  P.ctas = ctas;
  P.chunk = static_cast<int>((n + ctas - 1) / ctas);
  return P;
}

// Whether a CTA's copies of other CTAs' rows fit behind its own rows and zeros.
inline bool
ilu_copies_fit(const IluPlan& P, int B, int64_t copies)
{
  const int64_t places = (int64_t(P.chunk) + 1 + copies) * B;
  return size_t(places) * P.value_bytes() <= kIluClusterBytes &&
         places < (int64_t(1) << kIluOwnerShift);
}

// Whether the packed factors are worth their memory: `slots` places for a block
// in both directions together, padding included, for `entries` blocks of the
// factors. Every (CTA, level) pair takes whole groups of 32 rows, and a row whole
// chunks of entries: 2 to 3 slots per entry on 3D meshes, up to about 10 on long
// narrow 2D ones, but 170 for a chain of rows that depend on each other one by
// one, which at the largest size that fits would be 3.6 GB for 21 MB of factors.
// Such levels keep the level launches, once the packed form passes 64 MB.
constexpr int64_t kIluPackBytes = int64_t(64) << 20;
constexpr int kIluPackRatio = 16;
inline bool
ilu_padding_ok(const IluPlan& P, int B, int64_t slots, int64_t entries)
{
  const int64_t B2 = int64_t(B) * B;
  const int64_t packed = slots * (4 + B2 * (P.fp64 ? 12 : 4)); // column, values
  return packed <= std::max(kIluPackBytes, kIluPackRatio * entries * (4 + B2 * 12));
}

} // namespace gb
