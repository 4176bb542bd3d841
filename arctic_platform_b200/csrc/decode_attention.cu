// Attention of a decode step (one query token per sequence) over a paged cache, in one launch.
//
// Shared nodes.  All decode queries that share one node of the prefix forest (the rollouts of one prompt, or all rollouts of all
// prompts under a common header) attend to the node's KV pages TOGETHER: the query rows of up to 128/R sequences x R query heads of
// one KV head form one 128-row UMMA tile, the node's K/V pages are streamed once by TMA (one 16-token page per copy, straight out of
// the paged cache), S = Q K^T and P V run on the tensor core with S/P in tensor memory.  KV of a shared prompt is therefore read once
// per step for all of its rollouts instead of once per rollout.  The reference obtains this behaviour from ArcticInference's forest
// cascade attention (`use_fca`, arctic_platform/common/utils/server_models.py:123-132).
//
// Own pages.  What a sequence does not share it reads by itself, a warp per (sequence, KV head, part of its pages) on m16n8k16 MMAs.
//
// Everything leaves an un-normalised partial (max, sum, numerator) per query row; whoever is the last to arrive at a row's counter
// joins its partials, in the order of their places, not of their arrival.
//
// A CTA of the shared form: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 softmax (a row belongs to two threads, each with 64 of a
// block's 128 columns), warps 10-13 own pages.  As three launches -- shared pass with one thread per row, a pass of 96 KB CTAs over
// the own pages that could not start beside it, a merge -- a layer of 8 prompts x 16 samples (2048 shared tokens, 17 own, 8 key heads)
// took 24 + 19 + 6 us behind each other; 17 own tokens are a few KB per warp and hide behind the shared ones here: 27 us together.
// Long own contexts do not: four warps with one page ahead keep 32 KB under way per SM where paged_decode_mma_kernel has 128 KB, and at
// 2048 own tokens the three launches take 194 us, this one 210 (lengths from 1 to 2048: 124 and 175).  The rollout engine takes the
// one that is faster for the responses ahead (runtime_decode.cpp).  (Sequences that share nothing are left to
// paged_decode_mma_kernel, whose clusters join their parts sooner than counters in memory do: 7 us against 10 for one sequence of 400
// tokens, 33 against 36 for 41 of 500 to 1500.)
// Compiled for up to 8 query heads a key head it spills nothing, for 16 the walk over own pages spills 224 bytes (128 registers a
// thread are all that 448 threads leave).
//
// The KV blocks of a node are software-pipelined: tensor memory holds TWO score buffers, the MMA warp issues Q K^T of block j+1 before
// it waits for the probabilities of block j, and P V accumulates over all blocks in ONE output buffer in tensor memory that the
// softmax warps read only once, at the end.  The running maximum is therefore a REFERENCE maximum: a row rescales its output (read,
// multiply, write back -- after the previous P V has landed) only when its true maximum, or that of another row of its warp, has moved
// more than 2^8 above the reference; otherwise the probabilities are taken against the stale reference (at most 256, harmless in bf16
// / fp32) and nothing is rescaled.
#include "common.cuh"
#include "host_utils.cuh"
#include "paged_mma.cuh"

namespace apb {

struct DecodeAttnParams {
  const __nv_bfloat16* q;       // [B, Hq, 128]
  const __nv_bfloat16* kcache;  // [pages, Hkv, 16, 128]
  const __nv_bfloat16* vcache;
  __nv_bfloat16* out;           // [B, Hq, 128]
  int* arrived;                 // [2][B * Hkv] zeros, left as zeros: arrivals at a row, arrivals of its own parts
  int* status;
  int B, Hq, Hkv;
  float scale_log2;
  // shared nodes
  int G, splits, n_levels;
  const int* q_start;           // [G] first sequence (query row) of the node
  const int* q_count;           // [G] sequences below the node (R * count <= 128)
  const int* pages;             // [G, max_pages]
  int max_pages;
  const int* kv_len;            // [G] tokens in the node
  const int* level;             // [G] tree level of the node (selects the partials' buffer) or null (all level 0)
  const int* row_mask;          // [B] bit l: the row has a node at level l; bit n_levels: its own pages count
  float* sh_o[3];               // per level: [B, Hq, splits, 128] fp32 un-normalised numerators
  float* sh_ml[3];              // per level: [B, Hq, splits, 2] (max in base-2 scaled units, sum)
  // own pages
  const int* own_row;           // [B] row of the entry
  const int* own_active;        // [B] 0: nothing to read
  const int* own_pages;         // [B, own_max_pages]
  int own_max_pages;
  const int* own_len;           // [B]
  int own_chunk, own_parts;     // pages a part has at least (unless there are fewer), parts at most
  float* own_o;                 // [B, Hq, own_parts, 128]
  float* own_ml;                // [B, Hq, own_parts, 2]
};

constexpr int kDaThreads = 448;
constexpr int kDaSoftWarps = 8;
constexpr int kDaOwnWarps = 4;
constexpr int kDaOwnStages = 2;
constexpr int kDaOwnRing = kDaOwnStages * 2 * kMmaPageBytes;     // 16 KB per warp
constexpr int kDaSlots = 4;
constexpr int kDaTile = 128 * 128 * 2;  // one Q / K / V tile (D = 128)
constexpr int kDaBarBytes = 128;
constexpr int kDaExtra = kDaBarBytes + 2 * 2 * 128 * 4 /*maxima*/;
constexpr int kDaSmem = kDaTile + kDaSlots * kDaTile + kDaOwnWarps * kDaOwnRing + kDaExtra + 896 /*from 128- to 1024-byte alignment*/;
constexpr int kDaTmemCols = 512;        // S0 | S1 | O (128 fp32 columns each); 384 used, the allocation is a power of 2
constexpr int kDaOutStride = 132;       // floats between staged output rows
constexpr float kDaRescaleSlack = 8.f;  // log2 units the true row maximum may exceed the reference before a rescale
static_assert(kDaSmem <= 227 * 1024, "shared memory of one CTA");
static_assert(128 * kDaOutStride * 4 <= kDaSlots * kDaTile, "output rows are staged in the ring");

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Joins the partials of the query heads of one (row, key head), in the order of their places; a whole warp, four columns a lane.  KB
// parts of four heads are requested at a time: one part of one head after the other took longer than the attention itself.
template <int KB>
__device__ __forceinline__ void join_heads(const DecodeAttnParams& p, int row, int kvh, int n_own, int lane) {
  const int R = p.Hq / p.Hkv;
  const int levels = p.n_levels;
  const int mask = p.row_mask[row];
#pragma unroll 1
  for (int r0 = 0; r0 < R; r0 += 4) {
    const long long at = static_cast<long long>(row) * p.Hq + kvh * R + r0;
    float m[4], l[4], a[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      m[r] = -INFINITY;
      l[r] = a[r][0] = a[r][1] = a[r][2] = a[r][3] = 0.f;
    }
#pragma unroll 1
    for (int src = 0; src <= levels; ++src) {
      if (!((mask >> src) & 1)) continue;
      const bool own = src == levels;
      const float* o = own ? p.own_o : src == 0 ? p.sh_o[0] : src == 1 ? p.sh_o[1] : p.sh_o[2];
      const float* ml = own ? p.own_ml : src == 0 ? p.sh_ml[0] : src == 1 ? p.sh_ml[1] : p.sh_ml[2];
      const int n = own ? n_own : p.splits, places = own ? p.own_parts : p.splits;
#pragma unroll 1
      for (int k0 = 0; k0 < n; k0 += KB) {
        float4 v[KB][4];
        float2 s[KB][4];
#pragma unroll
        for (int k = 0; k < KB; ++k)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const bool there = k0 + k < n && r0 + r < R;
            const long long i = (at + r) * places + k0 + k;
            s[k][r] = there ? __ldcg(reinterpret_cast<const float2*>(ml + i * 2)) : make_float2(-INFINITY, 0.f);
            v[k][r] = there ? __ldcg(reinterpret_cast<const float4*>(o + i * 128 + lane * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float mn = m[r];
#pragma unroll
          for (int k = 0; k < KB; ++k) mn = fmaxf(mn, s[k][r].x);
          const float mu = mn == -INFINITY ? 0.f : mn, f0 = exp2f(m[r] - mu);
          l[r] *= f0;
#pragma unroll
          for (int e = 0; e < 4; ++e) a[r][e] *= f0;
#pragma unroll
          for (int k = 0; k < KB; ++k) {
            if (s[k][r].x == -INFINITY) continue;          // an empty part left no numerators
            const float f = exp2f(s[k][r].x - mu);
            l[r] += s[k][r].y * f;
            a[r][0] += v[k][r].x * f;
            a[r][1] += v[k][r].y * f;
            a[r][2] += v[k][r].z * f;
            a[r][3] += v[k][r].w * f;
          }
          m[r] = mn;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r0 + r >= R) break;
      const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
      *reinterpret_cast<uint2*>(p.out + (at + r) * 128 + lane * 4) =
          make_uint2(pack_bf16x2(a[r][0] * inv, a[r][1] * inv), pack_bf16x2(a[r][2] * inv, a[r][3] * inv));
    }
  }
}

// One more arrival at a row's counter: a node's part (add 1) or all of its own parts (add 1 and their number in the upper half).
// Returns the number of own parts when nothing is missing any more, else 0.  The caller's partials are written and fenced.
__device__ __forceinline__ int arrive_row(const DecodeAttnParams& p, int row, int kvh, int add) {
  int* c = p.arrived + static_cast<long long>(row) * p.Hkv + kvh;
  const int now = atomicAdd(c, add) + add;
  const int expected = 1 + __popc(p.row_mask[row] & ((1 << p.n_levels) - 1)) * p.splits;
  if ((now & 0xffff) != expected) return 0;
  *c = 0;
  __threadfence();
  return now >> 16;
}

// Own pages: warp `w` of `warps` takes every warps-th (sequence, part, key head).  A key head has 8 H query heads or less.
// Parts are as long as the work divided by the warps, a little longer until they are no more than the warps; where there are more
// (sequence, key head) pairs than warps nothing is cut, and warps walk one or two whole sequences (16 % over an even split at 1024
// pairs of equal length, more if lengths differ).  Which parts a row has thus depends on the lengths of all rows of the batch, and
// with them its last bits.
template <int H>
__device__ __forceinline__ void own_pass(const DecodeAttnParams& p, uint32_t ring, int w, int warps, int lane) {
  const int R = p.Hq / p.Hkv, units = p.B * p.Hkv;
  auto tokens = [&](int e) { return e < p.B && p.own_active[e] > 0 ? max(0, p.own_len[e]) : 0; };
  auto in_pages = [&](int e) { return e < p.B ? max(1, (tokens(e) + kPage - 1) / kPage) : 0; };      // nothing is a part too
  int sum = 0, most = 0;
  for (int e = lane; e < p.B; e += 32) {
    const int n = in_pages(e);
    sum += n;
    most = max(most, n);
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  most = __reduce_max_sync(0xffffffffu, most);
  const long long all = static_cast<long long>(sum) * p.Hkv;
  int chunk = max(max(p.own_chunk, (most + p.own_parts - 1) / p.own_parts), static_cast<int>((all + warps - 1) / warps));
  for (int i = 0; i < 12 && p.B <= 256 && chunk < most; ++i) {
    int n = 0;
    for (int e = lane; e < p.B; e += 32) n += (in_pages(e) + chunk - 1) / chunk;
    if (__reduce_add_sync(0xffffffffu, n) * p.Hkv <= warps) break;
    chunk += max(1, chunk >> 4);
  }
  long long before = 0;                // items of the entries in front of these 32
  long long item = w;
  for (int e0 = 0; e0 < p.B; e0 += 32) {
    const int c_len = tokens(e0 + lane), c_pages = in_pages(e0 + lane);
    const int c_parts = (c_pages + chunk - 1) / chunk;
    int end = c_parts * p.Hkv;         // inclusive sums
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += t;
    }
    const int here = __shfl_sync(0xffffffffu, end, 31);
    for (; item < before + here; item += warps) {
      const int local = static_cast<int>(item - before);
      const int from = __ffs(__ballot_sync(0xffffffffu, local < end)) - 1;
      const int e = e0 + from, parts = __shfl_sync(0xffffffffu, c_parts, from), len = __shfl_sync(0xffffffffu, c_len, from);
      const int inside = local - (__shfl_sync(0xffffffffu, end, from) - parts * p.Hkv);
      const int part = inside / p.Hkv, kvh = inside - part * p.Hkv;
      const int pages = (len + kPage - 1) / kPage;
      const int per = (pages + parts - 1) / parts, p0 = part * per, n = min(pages, p0 + per) - p0;     // n <= 0: nothing
      const int row = p.own_row[e];
      if (row < 0 || row >= p.B) {       // also of an entry that is not active: its row's arrivals are counted
        if (lane == 0 && p.status) atomicCAS(p.status, 0, kBadTable);
        continue;
      }
      const int* table = p.own_pages + static_cast<long long>(e) * p.own_max_pages + p0;
      int ids = lane < n ? table[lane] : 0;            // of pages [j & ~31, + 32)
      PagedHeads<H> acc;
      acc.start(p.q + (static_cast<long long>(row) * p.Hq + kvh * R) * 128, n > 0 ? R : 0, lane);
      auto issue = [&](int j, int id) {
        const long long at = (static_cast<long long>(id) * p.Hkv + kvh) * (kPage * 128);
        decode_issue_page(ring + (j % kDaOwnStages) * 2 * kMmaPageBytes, p.kcache + at, p.vcache + at, lane);
      };
      for (int j = 0; j < kDaOwnStages - 1; ++j) {
        const int id = __shfl_sync(0xffffffffu, ids, j);
        if (j < n) issue(j, id);
        cp_async_commit();
      }
#pragma unroll 1
      for (int j = 0; j < n; ++j) {
        const int jn = j + kDaOwnStages - 1;
        if ((jn & 31) == 0) ids = jn + lane < n ? table[jn + lane] : 0;
        const int id = __shfl_sync(0xffffffffu, ids, jn & 31);
        if (jn < n) issue(jn, id);
        cp_async_commit();
        cp_async_wait<kDaOwnStages - 1>();
        __syncwarp();
        acc.page(ring + (j % kDaOwnStages) * 2 * kMmaPageBytes, len - (p0 + j) * kPage, p.scale_log2, lane);
        __syncwarp();
      }
      cp_async_wait<0>();
      acc.finish();

      // nobody else contributes to the row: it is done here
      const bool alone = parts == 1 && (p.row_mask[row] & ((1 << p.n_levels) - 1)) == 0;
      const long long head0 = static_cast<long long>(row) * p.Hq + kvh * R;
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int head = 8 * h + (lane & 3) * 2 + e, d = lane >> 2;
          if (head >= R) continue;
          if (alone) {
            const float inv = acc.l[h][e] > 0.f ? 1.f / acc.l[h][e] : 0.f;
            __nv_bfloat16* dst = p.out + (head0 + head) * 128 + d;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              dst[i * 16] = __float2bfloat16(acc.o[h][i][e] * inv);
              dst[i * 16 + 8] = __float2bfloat16(acc.o[h][i][2 + e] * inv);
            }
          } else {
            const long long at = (head0 + head) * p.own_parts + part;
            if (n > 0) {
              float* dst = p.own_o + at * 128 + d;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                dst[i * 16] = acc.o[h][i][e];
                dst[i * 16 + 8] = acc.o[h][i][2 + e];
              }
            }
            if (d == 0) *reinterpret_cast<float2*>(p.own_ml + at * 2) = make_float2(acc.m[h][e], acc.l[h][e]);
          }
        }
      if (alone) continue;
      __threadfence();
      __syncwarp();
      int n_own = 0;
      if (lane == 0) {
        int* c = p.arrived + units + row * p.Hkv + kvh;
        if (parts == 1 || atomicAdd(c, 1) == parts - 1) {
          if (parts > 1) *c = 0;
          __threadfence();
          n_own = arrive_row(p, row, kvh, 1 + (parts << 16));
        }
      }
      n_own = __shfl_sync(0xffffffffu, n_own, 0);
      if (n_own > 0) join_heads<1>(p, row, kvh, n_own, lane);
    }
    before += here;
  }
}

template <int H>
__global__ void __launch_bounds__(kDaThreads, 1)
decode_cascade_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                      const __grid_constant__ CUtensorMap tma_v, const DecodeAttnParams p) {
  constexpr int D = 128;
  extern __shared__ __align__(128) uint8_t da_smem[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(da_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_q = smem;
  uint8_t* smem_kv = smem + kDaTile;
  uint8_t* smem_own = smem_kv + kDaSlots * kDaTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_own + kDaOwnWarps * kDaOwnRing);
  uint64_t* kv_full = bars;
  uint64_t* kv_empty = bars + kDaSlots;
  uint64_t* q_full = bars + 2 * kDaSlots;
  uint64_t* s_full = q_full + 1;    // [2] MMA -> softmax: scores of block j are in S[j & 1]
  uint64_t* p_full = s_full + 2;    // [2] softmax -> MMA: probabilities of block j are in S[j & 1]
  // [2] MMA -> softmax: P V of block j has been added to O.  A barrier for even blocks and one for odd ones: when the last block is
  // waited for, no more is known than that the products up to the third last have landed (they are ahead of the last scores in
  // the tensor core's order), and one barrier with a phase per block would take the third last's parity for the last one's.
  uint64_t* o_full = p_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(o_full + 2);
  static_assert((2 * kDaSlots + 7) * 8 + 4 <= kDaBarBytes, "barriers");
  float* halves = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + kDaBarBytes);      // [2][2][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = p.G * p.Hkv * p.splits;
  const bool has_unit = static_cast<int>(blockIdx.x) < units;
  const int unit = has_unit ? blockIdx.x : 0;
  const int node_heads = max(1, p.G * p.Hkv);
  const int split = unit / node_heads;
  const int g = unit % node_heads / p.Hkv;
  const int kvh = unit % p.Hkv;
  const int R = p.Hq / p.Hkv;
  // what a table asks for beyond the tile or the batch is left out and reported: the output rows are staged for 128 and no more
  const int asked = has_unit ? p.q_count[g] : 0;
  const int qs = has_unit ? p.q_start[g] : 0;
  const int nq = qs < 0 ? 0 : min(min(asked, 128 / R), p.B - qs);
  if (asked > 0 && nq != asked && threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, kBadTable);
  const int len = has_unit ? p.kv_len[g] : 0;
  const int n_blocks_all = (len + 127) / 128;
  const int per = (n_blocks_all + p.splits - 1) / p.splits;
  const int b0 = split * per;
  const int b1 = min(n_blocks_all, b0 + per);
  const int n_blocks = nq > 0 ? max(0, b1 - b0) : 0;

  if (nq > 0) {         // uniform across the CTA
    if (threadIdx.x == 0) {
      for (int s = 0; s < kDaSlots; ++s) {
        mbar_init(&kv_full[s], 1);
        mbar_init(&kv_empty[s], 1);
      }
      mbar_init(q_full, 1);
      for (int b = 0; b < 2; ++b) {
        mbar_init(&s_full[b], 1);
        mbar_init(&p_full[b], kDaSoftWarps * 32);
        mbar_init(&o_full[b], 1);
      }
      mbar_fence_init();
    }
    if (warp == 1) {
      tmem_alloc(tmem_holder, kDaTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = nq > 0 ? *tmem_holder : 0u;
  // chained launch: barriers and TMEM are set up.  The pages of a shared node are never written while its
  // sequences decode (new tokens go to private pages), so the first K and V tiles are requested BEFORE
  // the wait for the previous kernel; q, which that kernel produces, is loaded after it.
  pdl_launch_dependents();

  if (warp == 0) {
    // the whole warp: 16 lanes issue the 16 boxes (8 pages, two halves of the head) of a tile.  Pages past the end of the node are
    // replaced by its last page: finite data, masked by `limit`
    const int* table = p.pages + static_cast<long long>(g) * p.max_pages;
    const int last_page = (len + 15) / 16 - 1, pg = (lane & 15) >> 1, half = lane & 1;
    auto page_of = [&](int j) { return j < n_blocks ? table[min((b0 + j) * 8 + pg, last_page)] : 0; };
    int page = page_of(0);
    bool ok = true;
    for (int j = 0; j < n_blocks && ok; ++j) {
      const int next = page_of(j + 1);
      for (int v = 0; v < 2; ++v) {
        const int n = 2 * j + v, slot = n % kDaSlots;
        if (n >= kDaSlots) ok = __all_sync(0xffffffffu, mbar_wait(&kv_empty[slot], ((n / kDaSlots) & 1) ^ 1, p.status, kTimeoutEmpty));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&kv_full[slot], kDaTile);
        __syncwarp();
        if (lane < 16)
          tma_load_2d(smem_kv + slot * kDaTile + half * 16384 + pg * 2048, v ? &tma_v : &tma_k, &kv_full[slot], half * 64,
                      (page * p.Hkv + kvh) * 16);
      }
      page = next;
    }
    pdl_wait();
    if (!ok) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 100000ull) {
      }
    }
  } else if (warp == 1) {
    pdl_wait();
    // the whole warp walks the loop and one elected lane issues, so that descriptors are uniform (see gemm_tcgen05_2cta.cu)
    if (n_blocks > 0) {
      if (elect_one()) {
        mbar_expect_tx(q_full, kDaTile);
        for (int c = 0; c < 2; ++c) tma_load_4d(smem_q + c * 16384, &tma_q, q_full, c * 64, 0, kvh, qs);
      }
      __syncwarp();
      const uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = umma_idesc_bf16(128, D, 0, 1);
      const uint64_t desc_q = umma_smem_desc(smem_u32(smem_q), 0, 1024), desc_k = umma_smem_desc(smem_u32(smem_kv), 0, 1024);
      const uint64_t desc_v = umma_smem_desc(smem_u32(smem_kv), 16384, 1024);
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
        const bool r = __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, code));
        tc_fence_after();
        return r;
      };
      bool ok = wait(q_full, 0, kTimeoutFull);
      // S(j) = Q K(j)^T into score buffer j & 1
      auto issue_qk = [&](int j) -> bool {
        const uint32_t slot = (2 * j) % kDaSlots;
        if (!wait(&kv_full[slot], ((2 * j) / kDaSlots) & 1, kTimeoutFull)) return false;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k)
            umma_bf16_ss(tmem_base + (j & 1) * 128, desc_q + (k / 4) * 1024 + (k % 4) * 2,
                         desc_k + slot * (kDaTile >> 4) + (k / 4) * 1024 + (k % 4) * 2, idesc_s, k > 0 ? 1u : 0u);
          tc_commit(&s_full[j & 1]);
          tc_commit(&kv_empty[slot]);
        }
        __syncwarp();
        return true;
      };
      if (ok) ok = issue_qk(0);
      for (int j = 0; j < n_blocks && ok; ++j) {
        // the scores of the NEXT block first: they are ready when the softmax warps finish this one.  Its buffer
        // held the probabilities of block j-1, whose P V was issued before this point (the pipe runs in order).
        if (j + 1 < n_blocks && !issue_qk(j + 1)) {
          ok = false;
          break;
        }
        const uint32_t slot = (2 * j + 1) % kDaSlots, b = j & 1;
        if (!wait(&kv_full[slot], ((2 * j + 1) / kDaSlots) & 1, kTimeoutFull) || !wait(&p_full[b], (j >> 1) & 1, kTimeoutTmemEmpty)) {
          ok = false;
          break;
        }
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 128 / 16; ++k)
            umma_bf16_ts(tmem_base + 256, tmem_base + b * 128 + k * 8, desc_v + slot * (kDaTile >> 4) + k * 128, idesc_o,
                         (j > 0 || k > 0) ? 1u : 0u);
          tc_commit(&o_full[b]);
          tc_commit(&kv_empty[slot]);
        }
        __syncwarp();
      }
    }
  } else if (warp < 2 + kDaSoftWarps) {
    pdl_wait();                    // the partial buffers may still be read by the previous layer's join
    if (nq > 0) {
      const int quarter = warp & 3, half = (warp - 2) >> 2;      // two warps per quarter of the rows, 64 columns of a block each
      const int row = quarter * 32 + lane, pair = 1 + quarter;
      const bool live = quarter * 32 < nq * R;                   // a quarter of padding rows only keeps the barriers going
      const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
      // m_ref: the maximum the exponentials are taken against (see the header); l_run: sum of this half in the same units
      float m_ref = -INFINITY, l_run = 0.f;
      bool ok = true;                                            // uniform in the warp; barriers are met either way
      const uint32_t t_o = tmem_base + lane_off + 256 + half * 64;
      for (int j = 0; j < n_blocks; ++j) {
        const int b = j & 1;
        ok = ok && __all_sync(0xffffffffu, mbar_wait(&s_full[b], (j >> 1) & 1, p.status, kTimeoutTmemFull));
        tc_fence_after();
        const uint32_t t_s = tmem_base + lane_off + b * 128;
        const int limit = min(128, len - (b0 + j) * 128) - half * 64;
        float* mine = halves + (b * 2 + half) * 128;
        uint32_t sc[2][32];
        float mx = -INFINITY;
        if (ok && live) {
#pragma unroll
          for (int c = 0; c < 2; ++c) tmem_ld_32x32(t_s + half * 64 + c * 32, sc[c]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i < limit) mx = fmaxf(mx, __uint_as_float(sc[c][i]));
          mine[row] = mx;
        }
        tc_fence_before();
        bar_sync(pair, 64);        // both halves are in registers: probabilities may go over the scores
        tc_fence_after();
        if (ok && live) {
          mx = fmaxf(mx, halves[(b * 2 + (half ^ 1)) * 128 + row]);
          const float m_new = fmaxf(m_ref, mx * p.scale_log2);
          // one row that is behind moves the references of its quarter: tensor-memory loads and stores are warp collectives
          if (__any_sync(0xffffffffu, m_new > m_ref + kDaRescaleSlack || m_ref == -INFINITY)) {
            // move the reference.  Everything accumulated so far is in the old units: the row sum here, the output
            // row in tensor memory (once the previous block's P V has landed; block 0 has nothing to rescale)
            const float alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - m_new);
            if (j > 0) {
              ok = __all_sync(0xffffffffu, mbar_wait(&o_full[b ^ 1], ((j - 1) >> 1) & 1, p.status, kTimeoutTmemFull));
              tc_fence_after();
              if (ok) {
#pragma unroll 1
                for (int c = 0; c < 2; ++c) {
                  uint32_t r[32];
                  tmem_ld_32x32(t_o + c * 32, r);
                  tmem_ld_wait();
#pragma unroll
                  for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                  tmem_st_32x32(t_o + c * 32, r);
                }
              }
            }
            l_run *= alpha;
            m_ref = m_new;
          }
          const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
          float rowsum = 0.f;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float p0 = exp2f(__uint_as_float(sc[c][2 * i]) * p.scale_log2 - m_use);
              float p1 = exp2f(__uint_as_float(sc[c][2 * i + 1]) * p.scale_log2 - m_use);
              if (c * 32 + 2 * i >= limit) p0 = 0.f;
              if (c * 32 + 2 * i + 1 >= limit) p1 = 0.f;
              rowsum += p0 + p1;
              pk[i] = pack_bf16x2(p0, p1);
            }
            tmem_st_32x16(t_s + half * 32 + c * 16, pk);
          }
          tmem_st_wait();
          l_run += rowsum;
        }
        tc_fence_before();
        mbar_arrive(&p_full[b]);
      }
      // the output row: one read after the last P V, staged in the ring (all its tiles have been used) so that rows leave in 512
      // bytes each
      float* stage = reinterpret_cast<float*>(smem_kv);
      if (n_blocks > 0) {
        const int last = n_blocks - 1;
        ok = ok && __all_sync(0xffffffffu, mbar_wait(&o_full[last & 1], (last >> 1) & 1, p.status, kTimeoutTmemFull));
        tc_fence_after();
        if (ok && live) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(t_o + c * 32, r);
            tmem_ld_wait();
            float4* dst = reinterpret_cast<float4*>(stage + row * kDaOutStride + half * 64 + c * 32);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              dst[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                                   __uint_as_float(r[4 * i + 3]));
          }
        }
      }
      float* sums = halves;                                           // [2][128], once the last maxima have been read
      uint8_t* joins = reinterpret_cast<uint8_t*>(halves + 2 * 128);  // [128] own parts of a row that is to be joined here, else 0
      bar_sync(5, kDaSoftWarps * 32);
      sums[half * 128 + row] = l_run;
      bar_sync(5, kDaSoftWarps * 32);
      int lvl = p.level ? p.level[g] : 0;
      lvl = lvl < 0 ? 0 : (lvl >= p.n_levels ? p.n_levels - 1 : lvl);
      float* sh_o = lvl == 0 ? p.sh_o[0] : (lvl == 1 ? p.sh_o[1] : p.sh_o[2]);
      float* sh_ml = lvl == 0 ? p.sh_ml[0] : (lvl == 1 ? p.sh_ml[1] : p.sh_ml[2]);
      const int rows = nq * R;
      auto place = [&](int r) {
        return ((static_cast<long long>(qs) + r / R) * p.Hq + kvh * R + r % R) * p.splits + split;
      };
      if (half == 0 && row < rows)
        *reinterpret_cast<float2*>(sh_ml + place(row) * 2) = make_float2(m_ref, sums[row] + sums[128 + row]);
      if (n_blocks > 0)
        for (int r = warp - 2; r < rows; r += kDaSoftWarps)
          *reinterpret_cast<float4*>(sh_o + place(r) * D + lane * 4) = *reinterpret_cast<const float4*>(stage + r * kDaOutStride + lane * 4);
      __threadfence();
      bar_sync(5, kDaSoftWarps * 32);
      const int t = threadIdx.x - 64;
      if (t < nq) joins[t] = static_cast<uint8_t>(arrive_row(p, qs + t, kvh, 1));
      bar_sync(5, kDaSoftWarps * 32);
      for (int i = warp - 2; i < nq; i += kDaSoftWarps)
        if (joins[i]) join_heads<2>(p, qs + i, kvh, joins[i], lane);
    }
  } else {
    pdl_wait();
    const int w = warp - 2 - kDaSoftWarps;
    own_pass<H>(p, smem_u32(smem_own) + w * kDaOwnRing, w * gridDim.x + blockIdx.x, gridDim.x * kDaOwnWarps, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1 && nq > 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kDaTmemCols);
  }
}

}  // namespace apb

extern "C" {

// Decode attention over a prefix forest: q, out [B, Hq, 128] bf16, caches [num_pages, Hkv, 16, 128] bf16.
//   nodes (G of them, 0: none; q_count 0: unused): q_start, q_count, pages [G, max_pages], kv_len, level (or null), row_mask [B];
//   `splits` parts per node, partials per level sh_o[l] [B, Hq, splits, 128], sh_ml[l] [B, Hq, splits, 2]; R * max(q_count) <= 128,
//   rows of the same level are below one node at most;
//   what a table asks for beyond that, or beyond the batch, is left out and recorded in the status word;
//   own pages: entry e < B is row own_row[e] (each row once, active or not), read when own_active[e] > 0: own_pages [B, own_max_pages], own_len, in
//   parts of at least own_chunk pages, at most own_parts of them; own_o [B, Hq, own_parts, 128], own_ml [B, Hq, own_parts, 2].
// arrived: 2 * B * Hkv zeros, which are zeros again afterwards (unless the tables broke these rules: then the caller clears them).
// Rows without anything to attend to are zeros.
int apb_decode_attention(const void* q, const void* kcache, const void* vcache, void* out, int* arrived, long long num_pages, int B,
                         int Hq, int Hkv, int D, float scale, int G, int splits, int n_levels, const int* q_start, const int* q_count,
                         const int* pages, int max_pages, const int* kv_len, const int* level, const int* row_mask,
                         float* const* sh_o, float* const* sh_ml, const int* own_row, const int* own_active, const int* own_pages,
                         int own_max_pages, const int* own_len, int own_chunk, int own_parts, float* own_o, float* own_ml,
                         cudaStream_t s) {
  using namespace apb;
  if (B <= 0) return 0;
  if (D != 128 || Hkv <= 0 || Hq % Hkv || !arrived || !out || own_chunk < 1 || own_parts < 1 || own_parts > 255 || !own_o || !own_ml)
    return kBadArgument;
  const int R = Hq / Hkv;
  if (16 % R) return kBadArgument;
  DecodeAttnParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.kcache = static_cast<const __nv_bfloat16*>(kcache);
  p.vcache = static_cast<const __nv_bfloat16*>(vcache);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.arrived = arrived;
  p.status = status_device_ptr();
  p.B = B;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.own_row = own_row;
  p.own_active = own_active;
  p.own_pages = own_pages;
  p.own_max_pages = own_max_pages;
  p.own_len = own_len;
  p.own_chunk = own_chunk;
  p.own_parts = own_parts;
  p.own_o = own_o;
  p.own_ml = own_ml;
  const bool tall = R > 8;
  auto* kernel = tall ? decode_cascade_kernel<2> : decode_cascade_kernel<1>;
  static bool configured[2][64] = {{false}};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[tall][dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDaSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[tall][dev & 63] = true;
  }
  const long long own = static_cast<long long>(B) * Hkv;
  const int sms = sm_count();
  if (G < 0) G = 0;
  if (splits < 1 || splits > 255 || n_levels < 1 || n_levels > 3 || !sh_o || !sh_ml || !row_mask) return kBadArgument;
  for (int l = 0; l < n_levels; ++l)
    if (!sh_o[l] || !sh_ml[l]) return kBadArgument;
  if (n_levels > 1 && !level) return kBadArgument;
  CUtensorMap tq, tk, tv;
  {
    const uint64_t dims[4] = {128, static_cast<uint64_t>(R), static_cast<uint64_t>(Hkv), static_cast<uint64_t>(B)};
    const uint64_t strides[3] = {128 * 2ull, static_cast<uint64_t>(R) * 128 * 2ull, static_cast<uint64_t>(Hq) * 128 * 2ull};
    const uint32_t box[4] = {64, static_cast<uint32_t>(R), 1, static_cast<uint32_t>(128 / R)};
    int rc = make_tmap_nd(&tq, q, 2, 4, dims, strides, box);
    if (rc) return 1000 + rc;
  }
  const uint64_t rows = static_cast<uint64_t>(num_pages) * Hkv * 16;
  int rc = make_tmap_2d(&tk, kcache, 2, rows, 128, 128, 64, 16);
  if (rc) return 2000 + rc;
  rc = make_tmap_2d(&tv, vcache, 2, rows, 128, 128, 64, 16);
  if (rc) return 3000 + rc;
  p.G = G;
  p.splits = splits;
  p.n_levels = n_levels;
  p.q_start = q_start;
  p.q_count = q_count;
  p.pages = pages;
  p.max_pages = max_pages;
  p.kv_len = kv_len;
  p.level = level;
  p.row_mask = row_mask;
  for (int l = 0; l < 3; ++l) {
    // levels beyond n_levels alias the last valid buffer: a level id out of range can never reach a null pointer
    p.sh_o[l] = sh_o[l < n_levels ? l : n_levels - 1];
    p.sh_ml[l] = sh_ml[l < n_levels ? l : n_levels - 1];
  }
  const long long units = static_cast<long long>(G) * Hkv * splits;
  const long long for_own = (own + kDaOwnWarps - 1) / kDaOwnWarps;
  const long long want = for_own < sms ? for_own : sms;
  const int grid = static_cast<int>(units > want ? units : want);
  return static_cast<int>(launch_kernel(kernel, dim3(grid), dim3(kDaThreads), kDaSmem, s, tq, tk, tv, p));
}
}
