// Host runtime: which form of decode attention over shared prompts takes less time for the responses ahead.
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
//
// A rollout keeps to one form until sequences join it: the first steps of another form are captured in a graph of their own, which took
// 0.9 s in the middle of a rollout of the 4B model (128 sequences, 36 layers) -- more than the better form gives back behind the crossing
// (2048 steps of 8 x 16 samples: 14.86 s with one launch, 15.29 with three, 14.99 with the better of the two at each step once both are
// captured).
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

struct Launch {
  const int32_t *node_tokens, *node_slots;
  int64_t nodes, B, node_rows, Hq, Hkv, splits, own_parts, own_chunk, pass_splits, seq_splits, sms;
};

// Times of the two forms for `pages` private pages of every slot (0: idle).
void both(const Launch& p, std::vector<int64_t> pages, double* three, double* one) {
  int64_t sum = 0, most = 0;
  for (auto n : pages) {
    sum += n;
    most = std::max(most, n);
  }
  const double per_sm = static_cast<double>(sum) * p.Hkv / p.sms;
  const double heads = static_cast<double>(p.B) * p.Hq / 4096, rows = static_cast<double>(p.B) * p.Hkv / 1024;
  const int64_t head_rounds = ceil_div(p.Hq, 4 * p.Hkv);

  std::vector<double> tiles;
  tiles.reserve(p.nodes * p.Hkv * p.pass_splits);
  for (int64_t s = 0; s < p.pass_splits; ++s)
    for (int64_t g = 0; g < p.nodes; ++g)
      tiles.insert(tiles.end(), p.Hkv, 2.84 + 2.28 * ceil_div(ceil_div(p.node_tokens[g], 128), p.pass_splits));
  *three = 9.0 + rounds(tiles, p.sms) + 0.163 * per_sm + 0.08 * most / p.seq_splits + 6.6 * rows + 6.1 * heads;

  // the chains of the one launch, as its kernel cuts them: nothing is a part too
  const int64_t units = p.node_rows * p.Hkv * p.splits;
  const int64_t grid = std::max(units, std::min(ceil_div(p.B * p.Hkv, 4), p.sms)), warps = 4 * grid;
  sum = 0;
  for (auto& n : pages) sum += n = std::max<int64_t>(n, 1);
  most = std::max<int64_t>(most, 1);
  int64_t chunk = std::max({p.own_chunk, ceil_div(most, p.own_parts), ceil_div(sum * p.Hkv, warps)});
  for (int i = 0; i < 12 && p.B <= 256 && chunk < most; ++i) {
    int64_t n = 0;
    for (auto g : pages) n += ceil_div(g, chunk);
    if (n * p.Hkv <= warps) break;
    chunk += std::max<int64_t>(1, chunk >> 4);
  }
  std::vector<double> chain(warps, 0.0);
  int64_t at = 0, parts = 1;
  for (auto g : pages) {
    const int64_t n = ceil_div(g, chunk);
    parts = std::max(parts, n);
    const double item = 4.9 + 0.63 * ceil_div(g, n);
    for (int64_t k = 0; k < n * p.Hkv; ++k) {
      chain[at] += item;
      if (++at == warps) at = 0;
    }
  }
  const double look = 0.81 * ceil_div(p.B, 32);
  std::vector<double> blocks(grid);
  for (int64_t c = 0; c < grid; ++c) {
    const double own = look + std::max({chain[c], chain[c + grid], chain[c + 2 * grid], chain[c + 3 * grid]});
    const int64_t g = c < units ? c % (p.node_rows * p.Hkv) / p.Hkv : p.nodes;
    const double node = g < p.nodes ? 1.6 * ceil_div(ceil_div(p.node_tokens[g], 128), p.splits) +
                                          0.77 * head_rounds * ceil_div(p.node_slots[g], 8) * (0.5 * p.splits + 1)
                                    : 0.0;
    blocks[c] = 2.5 + std::max(node, own) + 0.37 * std::min(node, own);
  }
  *one = rounds(blocks, p.sms) + 0.6 * head_rounds * parts + 0.034 * per_sm + 2.3 * heads;
}

constexpr int kStretches = 4;

}  // namespace

extern "C" {

// node_tokens, node_slots [nodes]: of each row of the node tables in use, of which `node_rows` are launched; own_tokens [B]: private
// tokens of every slot, 0 for idle ones; left [B]: steps that a slot still has before it, one token each; splits, own_parts: parts of a node and of a
// sequence (at most) in one launch, of at least own_chunk pages; pass_splits, seq_splits: in three.  The times are those in the
// middle of four equal stretches of the longest `left`.  1: one launch takes no longer over all of them, 0: three do less, -1: bad
// arguments.
int32_t apb_rt_one_launch_pays(const int32_t* node_tokens, const int32_t* node_slots, int32_t nodes, const int32_t* own_tokens,
                               const int32_t* left, int32_t B, int32_t node_rows, int32_t Hq, int32_t Hkv, int32_t splits, int32_t own_parts,
                               int32_t own_chunk, int32_t pass_splits, int32_t seq_splits, int32_t sms) try {
  if (B < 1 || nodes < 0 || node_rows < nodes || Hkv < 1 || Hq < Hkv || splits < 1 || own_parts < 1 || own_chunk < 1 || pass_splits < 1 ||
      seq_splits < 1 || sms < 1)
    return -1;
  const Launch p{node_tokens, node_slots, nodes, B, node_rows, Hq, Hkv, splits, own_parts, own_chunk, pass_splits, seq_splits, sms};
  int64_t longest = 0;                    // of the slots in use: one whose sequence has ended early may have steps left
  for (int e = 0; e < B; ++e)
    if (own_tokens[e] > 0) longest = std::max<int64_t>(longest, left[e]);
  double three = 0, one = 0;
  std::vector<int64_t> pages(B);
  for (int k = 0; k < kStretches && (k == 0 || longest > 16); ++k) {
    const int64_t t = longest > 16 ? longest * (2 * k + 1) / (2 * kStretches) : longest / 2;
    for (int e = 0; e < B; ++e) pages[e] = own_tokens[e] > 0 && t <= std::max(left[e], 0) ? ceil_div(own_tokens[e] + t, 16) : 0;
    double a, b;
    both(p, pages, &a, &b);
    three += a;
    one += b;
  }
  return one <= three ? 1 : 0;
} catch (...) {
  return -1;
}
}
