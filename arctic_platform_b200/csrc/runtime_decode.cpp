// Host runtime: which form of decode attention over shared prompts takes less time at the lengths at hand.
//
// The one launch (decode_attention.cu) saves two ramps, has two threads per row of a node and hides short private pages behind the
// nodes.  But it reads private pages with four warps an SM, each one page (8 KB) ahead, and leaves sequences whole where there are more
// of them than warps; paged_decode_mma_kernel of the three launches keeps four times as many bytes under way and runs at the copy
// rate.  The last part of a node joins all its rows in eight warps, and every warp looks through all slots for its own pages.  So it
// loses where a warp's chain of pages is long against the saving, and where small nodes or many slots repeat the fixed work.
//
// A layer in us on a B200, 32 / 8 heads, three launches against one: 8 prompts of 2048 tokens x 16 samples with 17 own tokens 47 / 27,
// with 512 84 / 74, with 1024 121 / 120, with 2048 194 / 210, with 1 to 1024 83 / 101, with 1 to 2048 124 / 175; 40 prompts of 512 x
// 4 with 17 own 65 / 57, with 128 74 / 77, with 1024 156 / 234; one of 8192 x 2 with 2048 own 55 / 29; 64 of 256 x 16 (1024 slots)
// with 17 own, 16 / 8 heads, 153 / 251; one of 416 x 32 with 8 own, 16 / 4 heads, 17 / 24.
//
// The sums below are in us, fitted to both times at 1600 sizes: 2 to 1024 slots, 64 to 8192 shared and 8 to 2500 own tokens, equal or
// not, all or a fifth of the slots live, 2 to 8 heads a key head, 2 to 8 key heads, one shared level.  At 1892 other sizes of these
// ranges they are within 7 and 6 % in the mean, and what they choose takes 0.4 % more than the better of the two: 14 % less than three
// launches and 12 % less than one up to 256 slots, 8 % and 24 % less for more slots.  With a header above the prompts (959 sizes, none of
// them fitted to): 0.9 % more than the better of the two, 17 % less than three launches and 4 % less than one.
#include <algorithm>
#include <cstdint>
#include <vector>

namespace {

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Blocks of the given times, in turn on `places`: the longest of each round.
double rounds(const std::vector<double>& times, int64_t places) {
  double all = 0;
  for (size_t i = 0; i < times.size(); i += places)
    all += *std::max_element(times.begin() + i, times.begin() + std::min(times.size(), i + static_cast<size_t>(places)));
  return all;
}

}  // namespace

extern "C" {

// node_tokens, node_slots [nodes]: of each row of the node tables in use, of which `node_rows` are launched; own_tokens [B]: private
// tokens of every slot, 0 for idle ones; splits, own_parts: parts of a node and of a sequence (at most) in one launch, of at least
// own_chunk pages; pass_splits, seq_splits: in three.  1: one launch takes no longer, 0: three do less, -1: bad arguments.
int32_t apb_rt_one_launch_pays(const int32_t* node_tokens, const int32_t* node_slots, int32_t nodes, const int32_t* own_tokens, int32_t B,
                               int32_t node_rows, int32_t Hq, int32_t Hkv, int32_t splits, int32_t own_parts, int32_t own_chunk,
                               int32_t pass_splits, int32_t seq_splits, int32_t sms) try {
  if (B < 1 || nodes < 0 || node_rows < nodes || Hkv < 1 || Hq < Hkv || splits < 1 || own_parts < 1 || own_chunk < 1 || pass_splits < 1 ||
      seq_splits < 1 || sms < 1)
    return -1;
  std::vector<int64_t> pages(B);
  int64_t sum = 0, most = 0;
  for (int e = 0; e < B; ++e) {
    pages[e] = ceil_div(std::max(own_tokens[e], 0), 16);
    sum += pages[e];
    most = std::max(most, pages[e]);
  }
  const double per_sm = static_cast<double>(sum) * Hkv / sms;
  const double heads = static_cast<double>(B) * Hq / 4096, units_own = static_cast<double>(B) * Hkv / 1024;
  const int64_t head_rounds = ceil_div(Hq, 4 * Hkv);

  std::vector<double> tiles;
  tiles.reserve(static_cast<size_t>(nodes) * Hkv * pass_splits);
  for (int s = 0; s < pass_splits; ++s)
    for (int g = 0; g < nodes; ++g)
      tiles.insert(tiles.end(), Hkv, 3.9 + 2.25 * ceil_div(ceil_div(node_tokens[g], 128), pass_splits));
  const double three = 7.9 + rounds(tiles, sms) + 0.162 * per_sm + 0.103 * most / seq_splits + 3.9 * units_own + 6.6 * heads;

  // the chains of the one launch, as its kernel cuts them: nothing is a part too
  const int64_t units = static_cast<int64_t>(node_rows) * Hkv * splits;
  const int64_t grid = std::max<int64_t>(units, std::min<int64_t>(ceil_div(static_cast<int64_t>(B) * Hkv, 4), sms)), warps = 4 * grid;
  sum = 0;
  for (auto& n : pages) sum += n = std::max<int64_t>(n, 1);
  most = std::max<int64_t>(most, 1);
  int64_t chunk = std::max({static_cast<int64_t>(own_chunk), ceil_div(most, own_parts), ceil_div(sum * Hkv, warps)});
  for (int i = 0; i < 12 && B <= 256 && chunk < most; ++i) {
    int64_t n = 0;
    for (auto p : pages) n += ceil_div(p, chunk);
    if (n * Hkv <= warps) break;
    chunk += std::max<int64_t>(1, chunk >> 4);
  }
  std::vector<double> chain(warps, 0.0);
  int64_t item = 0, parts = 1;
  for (auto p : pages) {
    const int64_t n = ceil_div(p, chunk);
    parts = std::max(parts, n);
    for (int64_t k = 0; k < n * Hkv; ++k, ++item) chain[item % warps] += 4.1 + 0.63 * ceil_div(p, n);
  }
  const double look = 0.85 * ceil_div(B, 32);
  std::vector<double> blocks(grid);
  for (int64_t c = 0; c < grid; ++c) {
    const double own = look + std::max({chain[c], chain[c + grid], chain[c + 2 * grid], chain[c + 3 * grid]});
    const int64_t g = c < units ? c % (static_cast<int64_t>(node_rows) * Hkv) / Hkv : nodes;
    const double node = g < nodes ? 1.6 * ceil_div(ceil_div(node_tokens[g], 128), splits) +
                                        0.77 * head_rounds * ceil_div(node_slots[g], 8) * (0.5 * splits + 1)
                                  : 0.0;
    blocks[c] = 3.1 + std::max(node, own) + 0.31 * std::min(node, own);
  }
  const double one = rounds(blocks, sms) + 0.61 * head_rounds * parts + 0.041 * per_sm + 2.6 * heads;
  return one <= three ? 1 : 0;
} catch (...) {
  return -1;
}
}
