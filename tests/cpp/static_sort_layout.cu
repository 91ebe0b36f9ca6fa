// Where the look-back words of kifi_radix_sort_pairs_u32_static lie in its
// static scratch, by the addresses that a digit pass forms (sort_pass_body):
// compiling this file is the check, it needs no GPU.
#include "../../merge_fusion_gb300/csrc/kifi_sort_body.cuh"
#include "../../merge_fusion_gb300/csrc/kifi_sort_static.cu"

namespace kifi {
namespace {

// one past the last look-back word that the four passes of a sort of `tiles` tiles touch
constexpr size_t words_end(size_t max_tiles, size_t tiles) {
    constexpr size_t kR = 256;
    size_t end = 0;
    for (size_t pass = 0; pass < 4; ++pass)
        for (size_t t = 0; t < tiles; ++t) {
            const size_t lb = pass * sort_detail::lookback_rows(max_tiles) * kR;
            const size_t tile_end = lb + (t + 1) * kR;
            const size_t group_end = lb + (max_tiles + t / sort_detail::kGroup + 1) * kR;
            if (tile_end > end) end = tile_end;
            if (group_end > end) end = group_end;
        }
    return end;
}

// all tiles of the largest n, whose last group may be partial
constexpr size_t kLimitTiles = (kMaxKeys + sort_detail::kTile - 1) / sort_detail::kTile;
static_assert(kLookback + words_end(kTiles, kLimitTiles) * sizeof(unsigned long long) <= kAltKeys,
              "look-back words lie on the spare keys");
static_assert(kAltKeys + (kMaxKeys + 64) * sizeof(uint32_t) <= kAltVals, "spare keys lie on the spare values");
static_assert(kAltVals + (kMaxKeys + 64) * sizeof(uint32_t) <= kScratchBytes, "spare values leave the scratch");
static_assert(kLookback % 8 == 0 && kAltKeys % 256 == 0 && kAltVals % 256 == 0, "alignment");

// the allocating scratch: one pass's rows hold every tile's and every group's, for any tile count
constexpr bool rows_hold(size_t most) {
    for (size_t m = 1; m <= most; ++m)
        if (m + (m - 1) / sort_detail::kGroup + 1 > sort_detail::lookback_rows(m)) return false;
    return true;
}
static_assert(rows_hold(4096), "a pass's rows reach into the next pass's");

}  // namespace
}  // namespace kifi
