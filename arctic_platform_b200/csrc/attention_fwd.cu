// Segment attention forward on tcgen05 tensor cores.
//
// One kernel covers plain packed varlen causal attention, ZoRRo prompt-to-prompt
// attention and ZoRRo response-to-(shared prompt + own response) attention: every
// query tile attends to a "prefix" key range that is fully visible (the group's
// shared prompt, stored ONCE in the packed K/V) followed by its "own" key range
// under a bottom-right aligned causal mask.  The reference reaches the same result
// by materialising per-sample [prompt || response] K/V copies with torch.cat and
// two flash_attn_varlen calls per layer
// (arctic_platform/rl/zorro_train/qwen_attention_patcher.py:1197-1231,
//  arctic_platform/rl/zorro_train/zorro_train.py:857-912); here the key tile index
// is resolved in the kernel and nothing is replicated.
//
// CTA = 384 threads, one per SM, walking its share of the work table (longest tiles first): warp 0 TMA producer,
// warp 1 MMA issuer, warps 4-7 and 8-11 two softmax groups.  The two groups hold two query heads of the same KV head
// (same 128 query rows), so they walk the same K/V tiles and ping-pong on the tensor
// core: while one group does softmax on S_j the other group's P*V and next S run.
// S (fp32) lives in TMEM, P (bf16) overwrites it in place and feeds the P*V MMA as
// the TMEM A operand, the P*V product is read back and accumulated in registers
// with the usual online-softmax rescale.
//
// What bounds it: 2048 tensor cycles per pair of 128 x 128 blocks, and as many of the exponential unit (16 per
// cycle and SM).  A group's other instructions (maxima, packed fp32 arithmetic, the read of the previous P*V) hide
// behind the other group's products; loads from tensor memory are 32 columns at a time, the next one on its way
// while one is worked on, because 128 registers hold O.  P*V of block j - 1 is read when S_j is there (it was issued
// before S_j), so nobody waits for it.  Masks are applied only where a block has any.  Reading O behind every block,
// masks everywhere, unpacked arithmetic and one CTA per tile took 7200 cycles per pair of blocks (8 x 4096 tokens,
// 32 / 8 heads: 1.74 ms, 630 TFLOP/s), this 5500 (1.34 ms, 820; 32768 tokens 860 TFLOP/s).  Adding the previous P*V
// between the exponentials instead, 16 columns at a time, spilled and took 1.46 ms.
//
// With TMEM_O, O stays in tensor memory, where the products add themselves up: it is rescaled only when the running maximum of one of a
// warp's 32 rows has moved (nearly always in the first 32 blocks, in a tenth of them behind 256) and read once per tile, scores are read
// once.  8 x 4096 tokens 1.11 ms instead of 1.33, one sequence of 32768 8.3 instead of 9.9 (1060 TFLOP/s), 12 x 300 46 us instead of 56.
// Weights, row sums and maxima are those of the other form; O is added up by the tensor core, in fp32 as there, but it cuts off what
// does not fit.  Errors of O against 64 bits, scores of standard deviation 0.3, 1 and 3: 4096 tokens 1.780e-3, 1.780e-3 and 1.707e-3 with
// either form (1e-5 of that apart), 32768 tokens 1.785e-3, 1.785e-3 and 1.719e-3 against 1.784e-3, 1.784e-3 and 1.718e-3 with O in
// registers; the rounding of the result to bf16 is nearly all of it.  Other last bits make routers downstream choose other experts now and
// then: models with experts keep O in registers.  Moving the reference only when it lags by 2^8 takes 1.03 ms, but rounds the
// largest weight, which is 1 otherwise (error 2.05e-3 instead of 1.77e-3 at a deviation of 3).  140 bytes of a softmax thread spill
// (280 with O in registers).  Two buffers of 32 columns for the
// rescaling spilled (1.25 ms); a polynomial on the FMA pipe for 1/8 to 1/2 of the exponentials gained nothing.
#include "attention_common.cuh"
#include "host_utils.cuh"

namespace apb {

struct AttnFwdParams {
  const int* work;  // [num_work][8]: q_row0, q_valid, pre_start, pre_len, own_start, own_len, diag, head|(pair<<16)
  int num_work;
  int Hq, Hkv;
  float scale_log2;  // softmax scale * log2(e)
  __nv_bfloat16* O;  // [T, Hq*D]
  long long ldo;
  float* lse;        // [Hq, T] natural-log LSE
  int T;
  int* status;
};

// Three warpgroups: issue and two of softmax.  Registers move from the first to the others: 56 + 2 * 224 = 3 * 168, what the block
// was launched with.
constexpr int kAttnThreads = 384;
constexpr int kAttnRegsIssue = 56, kAttnRegsSoftmax = 224;
constexpr int kKvBlock = 128;

template <int D>
struct AttnCfg {
  static constexpr int kChunks = D / 64;
  static constexpr int kTileBytes = 128 * D * 2;      // one Q, K or V tile
  static constexpr int kSlots = 4;                    // K/V ring
  static constexpr int kSmemBytes = 2 * kTileBytes + kSlots * kTileBytes + 1024 + 256;
};

struct AttnItem {
  int q_row0, q_valid, pre_start, pre_len, own_start, own_len, diag, head0, n_groups, n_pre, n_blocks;
  __device__ __forceinline__ explicit AttnItem(const int* w) {
    const int4 a = *reinterpret_cast<const int4*>(w), b = *reinterpret_cast<const int4*>(w + 4);
    q_row0 = a.x, q_valid = a.y, pre_start = a.z, pre_len = a.w;
    own_start = b.x, own_len = b.y, diag = b.z;
    head0 = b.w & 0xFFFF;
    n_groups = (b.w >> 16) ? 2 : 1;
    n_pre = (pre_len + kKvBlock - 1) / kKvBlock;
    n_blocks = n_pre + (own_len + kKvBlock - 1) / kKvBlock;
  }
};

template <int D, bool TMEM_O>
__global__ void __launch_bounds__(kAttnThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                const __grid_constant__ CUtensorMap tma_v, const AttnFwdParams p) {
  using Cfg = AttnCfg<D>;
  constexpr int kSlots = Cfg::kSlots;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_q = smem;                              // 2 tiles
  uint8_t* smem_kv = smem + 2 * Cfg::kTileBytes;       // ring
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_kv + kSlots * Cfg::kTileBytes);
  uint64_t* kv_full = bars;                 // [kSlots]
  uint64_t* kv_empty = bars + kSlots;       // [kSlots]
  uint64_t* q_full = bars + 2 * kSlots;
  uint64_t* q_empty = q_full + 1;
  uint64_t* s_full = q_empty + 1;  // [2]
  uint64_t* p_full = s_full + 2;   // [2]
  uint64_t* o_full = p_full + 2;   // [2]  once per work item
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(o_full + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int g = 0; g < 2; ++g) {
      mbar_init(&s_full[g], 1);
      mbar_init(&p_full[g], 128);
      mbar_init(&o_full[g], 1);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // TMEM map: S/P of group g at columns [g*128, g*128+128), O of group g at [256 + g*128, ...+D)

  // This CTA's items: one of every gridDim.x, from the front and from the back in turn, so that the CTA with the longest item
  // of one round gets the shortest of the next.
  const int rounds = (p.num_work + gridDim.x - 1) / gridDim.x;
  auto item_at = [&](int round) {
    const int i = round * gridDim.x + ((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    return i < p.num_work ? i : -1;
  };
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {      // of a whole warp
    const bool r = __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, code));
    tc_fence_after();
    return r;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kAttnRegsIssue));
    if (warp == 0) {
      // ---------------------------------------------------------------- producer
      if (lane == 0) {
        bool ok = true;
        int slot = 0;
        uint32_t phase = 0, items = 0;
        for (int round = 0; round < rounds && ok; ++round) {
          const int at = item_at(round);
          if (at < 0) continue;
          const AttnItem w(p.work + static_cast<long long>(at) * 8);
          if (w.n_blocks == 0) continue;
          const int kvh = w.head0 / (p.Hq / p.Hkv);
          ok = mbar_wait(q_empty, (items & 1) ^ 1, p.status, kTimeoutEmpty);
          if (!ok) break;
          ++items;
          mbar_expect_tx(q_full, w.n_groups * Cfg::kTileBytes);
          for (int g = 0; g < w.n_groups; ++g)
            for (int c = 0; c < Cfg::kChunks; ++c)
              tma_load_2d(smem_q + g * Cfg::kTileBytes + c * 16384, &tma_q, q_full, (w.head0 + g) * D + c * 64, w.q_row0);
          for (int n = 0; n < 2 * w.n_blocks; ++n) {
            ok = mbar_wait(&kv_empty[slot], phase ^ 1, p.status, kTimeoutEmpty);
            if (!ok) break;
            const int b = n >> 1;
            const int row = b < w.n_pre ? w.pre_start + b * kKvBlock : w.own_start + (b - w.n_pre) * kKvBlock;
            uint8_t* dst = smem_kv + slot * Cfg::kTileBytes;
            mbar_expect_tx(&kv_full[slot], Cfg::kTileBytes);
            const CUtensorMap* map = (n & 1) ? &tma_v : &tma_k;
            for (int c = 0; c < Cfg::kChunks; ++c) tma_load_2d(dst + c * 16384, map, &kv_full[slot], kvh * D + c * 64, row);
            if (++slot == kSlots) {
              slot = 0;
              phase ^= 1;
            }
          }
        }
        if (!ok) {
          const uint64_t t0 = global_timer_ns();
          while (global_timer_ns() - t0 < 100000ull) {
          }
        }
      }
    } else if (warp == 1) {
      // -------------------------------------------------------------- MMA issuer (whole warp, one elected lane issues: see
      // gemm_tcgen05_2cta.cu)
      const uint32_t idesc_s = umma_idesc_bf16(128, kKvBlock, 0, 0);
      const uint32_t idesc_o = umma_idesc_bf16(128, D, 0, 1);
      const uint64_t desc_q = umma_smem_desc(smem_u32(smem_q), 0, 1024), desc_k = umma_smem_desc(smem_u32(smem_kv), 0, 1024);
      const uint64_t desc_v = umma_smem_desc(smem_u32(smem_kv), 16384, 1024);
      constexpr uint32_t kTile = Cfg::kTileBytes >> 4;
      auto issue_s = [&](uint32_t g, uint32_t slot) {      // by the elected lane
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_bf16_ss(tmem_base + g * 128, desc_q + g * kTile + (k / 4) * 1024 + (k % 4) * 2,
                       desc_k + slot * kTile + (k / 4) * 1024 + (k % 4) * 2, idesc_s, k > 0 ? 1u : 0u);
        tc_commit(&s_full[g]);
      };
      auto issue_o = [&](uint32_t g, uint32_t slot, bool first) {
#pragma unroll
        for (int k = 0; k < kKvBlock / 16; ++k)
          umma_bf16_ts(tmem_base + 256 + g * 128, tmem_base + g * 128 + k * 8, desc_v + slot * kTile + k * 128, idesc_o,
                       (!first || k > 0) ? 1u : 0u);
      };
      uint32_t slot = 0, phase = 0, items = 0, done[2] = {0, 0};       // done: blocks of each group whose P has been awaited
      auto wait_slot = [&]() {         // the ring's next tile; its slot
        const uint32_t s = slot;
        const bool r = wait(&kv_full[s], phase, kTimeoutFull);
        if (++slot == kSlots) {
          slot = 0;
          phase ^= 1;
        }
        return r;
      };
      bool ok = true;
      for (int round = 0; round < rounds && ok; ++round) {
        const int at = item_at(round);
        if (at < 0) continue;
        const AttnItem w(p.work + static_cast<long long>(at) * 8);
        if (w.n_blocks == 0) continue;
        uint32_t sk = slot;
        ok = wait(q_full, items & 1, kTimeoutFull) && wait_slot();
        if (!ok) break;
        ++items;
        if (elect_one()) {
          for (int g = 0; g < w.n_groups; ++g) issue_s(g, sk);
          tc_commit(&kv_empty[sk]);
          if (w.n_blocks == 1) tc_commit(q_empty);
        }
        __syncwarp();
        for (int j = 0; j < w.n_blocks && ok; ++j) {
          const bool more = j + 1 < w.n_blocks;
          const uint32_t sv = slot;
          ok = wait_slot();
          sk = slot;
          if (ok && more) ok = wait_slot();
          if (!ok) break;
          for (int g = 0; g < w.n_groups && ok; ++g) {
            ok = wait(&p_full[g], done[g] & 1, kTimeoutTmemEmpty);
            if (!ok) break;
            ++done[g];
            if (elect_one()) {
              issue_o(g, sv, !TMEM_O || j == 0);
              if (more)
                issue_s(g, sk);      // over P, which the product above reads first: the tensor core keeps the order of issue
              else
                tc_commit(&o_full[g]);
              if (g == w.n_groups - 1) {
                tc_commit(&kv_empty[sv]);
                if (more) tc_commit(&kv_empty[sk]);
                if (j + 2 == w.n_blocks) tc_commit(q_empty);
              }
            }
            __syncwarp();
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax groups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kAttnRegsSoftmax));
    const int g = (warp >> 2) - 1;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;  // row inside the query tile
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t t_s = tmem_base + lane_off + g * 128;
    const uint32_t t_o = tmem_base + lane_off + 256 + g * 128;
    const uint64_t c2 = xtc_pair(p.scale_log2, p.scale_log2);
    uint32_t blocks = 0, items = 0;       // of this group so far
    bool ok = true;
    uint64_t o[TMEM_O ? 1 : D / 2];          // pairs of columns
    uint32_t buf[2][32];
    for (int round = 0; round < rounds && ok; ++round) {
      const int at = item_at(round);
      if (at < 0) continue;
      const AttnItem w(p.work + static_cast<long long>(at) * 8);
      if (w.n_blocks == 0 || g >= w.n_groups) continue;
      float m_run = -INFINITY, l_run = 0.f, alpha = 0.f;       // TMEM_O: l_run is the sum when all is done
      uint64_t l2 = 0;                // its sum so far, in two halves
#pragma unroll
      for (int i = 0; i < D / 2 && !TMEM_O; ++i) o[i] = 0;
      // o = o * alpha + P*V, 32 columns that are in `v`
      auto add = [&](int c, const uint32_t (&v)[32]) {
        const uint64_t a2 = xtc_pair(alpha, alpha);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          o[c * 16 + i] = xtc_fma2(o[c * 16 + i], a2, xtc_pair(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
      };
      for (int j = 0; j < w.n_blocks; ++j) {
        ok = wait(&s_full[g], blocks & 1, kTimeoutTmemFull);
        if (!ok) break;
        ++blocks;
        // visible key columns of this block: of this row, and of the tile's first row
        int limit, least;
        if (j < w.n_pre) {
          limit = least = w.pre_len - j * kKvBlock;
        } else {
          const int b0 = (j - w.n_pre) * kKvBlock;
          least = min(w.own_len - b0, w.diag - b0 + 1);
          limit = min(w.own_len - b0, row + w.diag - b0 + 1);
        }
        const bool masked = least < kKvBlock;
        if constexpr (TMEM_O) {
          uint32_t v[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, v[c]);
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_wait(v[c]);
          if (masked) {
#pragma unroll
            for (int c = 0; c < kKvBlock; ++c)
              if (c >= limit) v[c / 32][c % 32] = 0xff800000u;        // its weight is 2^-inf: the scale is positive here
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < kKvBlock; c += 2)
            mx[(c >> 1) & 3] = fmaxf(fmaxf(mx[(c >> 1) & 3], __uint_as_float(v[c / 32][c % 32])), __uint_as_float(v[c / 32][c % 32 + 1]));
          const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
          if (__any_sync(0xffffffffu, m_new > m_run)) {
            if (j > 0) {           // O holds the blocks before this one: their product was issued ahead of this S
              alpha = m_run == -INFINITY ? 0.f : xtc_ex2(m_run - m_new);
              l2 = xtc_mul2(l2, xtc_pair(alpha, alpha));
              const uint64_t a2 = xtc_pair(alpha, alpha);
              uint32_t r[2][16];
              tmem_ld_32x16(t_o, r[0]);
              tmem_ld_wait(r[0]);
#pragma unroll
              for (int c = 0; c < D / 16; ++c) {
                if (c + 1 < D / 16) tmem_ld_32x16(t_o + (c + 1) * 16, r[(c + 1) & 1]);
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                  const float2 f = xtc_unpair(xtc_mul2(xtc_pair(__uint_as_float(r[c & 1][i]), __uint_as_float(r[c & 1][i + 1])), a2));
                  r[c & 1][i] = __float_as_uint(f.x);
                  r[c & 1][i + 1] = __float_as_uint(f.y);
                }
                tmem_st_32x16(t_o + c * 16, r[c & 1]);
                if (c + 1 < D / 16) tmem_ld_wait(r[(c + 1) & 1]);
              }
            }
            m_run = m_new;
          }
          const float m_use = m_run == -INFINITY ? 0.f : m_run;
          const uint64_t nm2 = xtc_pair(-m_use, -m_use);
          uint64_t sum[2] = {0, 0};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float2 f = xtc_unpair(
                  xtc_fma2(xtc_pair(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), c2, nm2));
              f.x = xtc_ex2(f.x);
              f.y = xtc_ex2(f.y);
              sum[i & 1] = xtc_add2(sum[i & 1], xtc_pair(f.x, f.y));
              pk[i] = pack_bf16x2(f.x, f.y);
            }
            tmem_st_32x16(t_s + c * 16, pk);
          }
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(&p_full[g]);
          l2 = xtc_add2(l2, xtc_add2(sum[0], sum[1]));
          continue;
        }
        auto mask = [&](int c, uint32_t (&v)[32]) {
          if (masked) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= limit) v[i] = 0xff800000u;
          }
        };
        // the product of the block before, which was issued ahead of this S
        if (j > 0) {
          tmem_ld_32x32(t_o, buf[0]);
          tmem_ld_wait(buf[0]);
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            if (c + 1 < D / 32) tmem_ld_32x32(t_o + (c + 1) * 32, buf[(c + 1) & 1]);
            else tmem_ld_32x32(t_s, buf[(c + 1) & 1]);
            add(c, buf[c & 1]);
            tmem_ld_wait(buf[(c + 1) & 1]);
          }
        } else {
          tmem_ld_32x32(t_s, buf[0]);
          tmem_ld_wait(buf[0]);
        }
        // pass 1: row maximum (buf[c & 1] holds columns [32 c, +32) at the start of step c: D / 32 is even)
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_ld_32x32(t_s + ((c + 1) & 3) * 32, buf[(c + 1) & 1]);
          mask(c, buf[c & 1]);
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            mx[(i >> 1) & 3] = fmaxf(fmaxf(mx[(i >> 1) & 3], __uint_as_float(buf[c & 1][i])), __uint_as_float(buf[c & 1][i + 1]));
          tmem_ld_wait(buf[(c + 1) & 1]);
        }
        const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        alpha = xtc_ex2(m_run - m_use);  // m_run = -inf -> 0
        // pass 2: probabilities, written over S as packed bf16 (two per 32-bit column)
        const uint64_t nm2 = xtc_pair(-m_use, -m_use);
        float rowsum = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c < 3) tmem_ld_32x32(t_s + (c + 1) * 32, buf[(c + 1) & 1]);
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float2 f = xtc_unpair(
                xtc_fma2(xtc_pair(__uint_as_float(buf[c & 1][2 * i]), __uint_as_float(buf[c & 1][2 * i + 1])), c2, nm2));
            f.x = xtc_ex2(f.x);
            f.y = xtc_ex2(f.y);
            if (masked) {            // the weight itself: a masked score times a scale of zero is no number
              if (c * 32 + 2 * i >= limit) f.x = 0.f;
              if (c * 32 + 2 * i + 1 >= limit) f.y = 0.f;
            }
            rowsum += f.x + f.y;
            pk[i] = pack_bf16x2(f.x, f.y);
          }
          if (c < 3) tmem_ld_wait(buf[(c + 1) & 1]);
          tmem_st_32x16(t_s + c * 16, pk);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&p_full[g]);
        l_run = fmaf(l_run, alpha, rowsum);
        m_run = m_new;
      }
      if (!ok) break;
      ok = wait(&o_full[g], items & 1, kTimeoutTmemFull);
      if (!ok) break;
      ++items;
      if constexpr (TMEM_O) {
        const float2 l = xtc_unpair(l2);
        l_run = l.x + l.y;
      } else {
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          tmem_ld_32x32(t_o + c * 32, buf[0]);
          tmem_ld_wait(buf[0]);
          add(c, buf[0]);
        }
        tc_fence_before();
      }
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const long long t = static_cast<long long>(w.q_row0) + row;
      __nv_bfloat16* dst = p.O + t * p.ldo + static_cast<long long>(w.head0 + g) * D;
      if constexpr (TMEM_O) {
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(t_o + c * 32, r);
          tmem_ld_wait(r);
          if (row < w.q_valid) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 x;
              x.x = pack_bf16x2(__uint_as_float(r[q * 8 + 0]) * inv, __uint_as_float(r[q * 8 + 1]) * inv);
              x.y = pack_bf16x2(__uint_as_float(r[q * 8 + 2]) * inv, __uint_as_float(r[q * 8 + 3]) * inv);
              x.z = pack_bf16x2(__uint_as_float(r[q * 8 + 4]) * inv, __uint_as_float(r[q * 8 + 5]) * inv);
              x.w = pack_bf16x2(__uint_as_float(r[q * 8 + 6]) * inv, __uint_as_float(r[q * 8 + 7]) * inv);
              *reinterpret_cast<uint4*>(dst + c * 32 + q * 8) = x;
            }
          }
        }
        tc_fence_before();
      } else if (row < w.q_valid) {
#pragma unroll
        for (int q = 0; q < D / 8; ++q) {
          float2 f[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) f[i] = xtc_unpair(o[q * 4 + i]);
          uint4 x;
          x.x = pack_bf16x2(f[0].x * inv, f[0].y * inv);
          x.y = pack_bf16x2(f[1].x * inv, f[1].y * inv);
          x.z = pack_bf16x2(f[2].x * inv, f[2].y * inv);
          x.w = pack_bf16x2(f[3].x * inv, f[3].y * inv);
          *reinterpret_cast<uint4*>(dst + q * 8) = x;
        }
      }
      if (p.lse && row < w.q_valid)
        p.lse[static_cast<long long>(w.head0 + g) * p.T + t] =
            l_run > 0.f ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace apb

extern "C" {

// q [T, Hq*D] (row stride ldq), k/v [T, Hkv*D] (ldk/ldv), o [T, Hq*D] (ldo), lse [Hq, T] fp32 or null.
// work: device int32 [num_work][8] (see AttnFwdParams).  scale is the softmax scale (1/sqrt(D)).
// tmem_o: O may be added up in tensor memory (see the header); scales that are not positive, which change the place of the maximum among
// the scores, take the other form either way.
int apb_attn_fwd_form(const void* q, const void* k, const void* v, void* o, float* lse, const int* work, int num_work,
                     int T, int Hq, int Hkv, int D, long long ldq, long long ldk, long long ldv, long long ldo,
                     float scale, int tmem_o, cudaStream_t stream) {
  using namespace apb;
  if (num_work <= 0) return 0;
  if ((D != 128 && D != 64) || (ldq % 8) || (ldk % 8) || (ldv % 8) || (ldo % 8) || Hq % Hkv) return kBadArgument;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_2d(&tq, q, 2, T, static_cast<uint64_t>(Hq) * D, ldq, 64, 128);
  if (rc) return 1000 + rc;
  rc = make_tmap_2d(&tk, k, 2, T, static_cast<uint64_t>(Hkv) * D, ldk, 64, 128);
  if (rc) return 2000 + rc;
  rc = make_tmap_2d(&tv, v, 2, T, static_cast<uint64_t>(Hkv) * D, ldv, 64, 128);
  if (rc) return 3000 + rc;
  AttnFwdParams p;
  p.work = work;
  p.num_work = num_work;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.O = static_cast<__nv_bfloat16*>(o);
  p.ldo = ldo;
  p.lse = lse;
  p.T = T;
  p.status = status_device_ptr();
  const int grid = num_work < sm_count() ? num_work : sm_count();
  const bool in_tmem = tmem_o && scale > 0.f;
  auto* kernel = D == 128 ? (in_tmem ? attn_fwd_kernel<128, true> : attn_fwd_kernel<128, false>)
                          : (in_tmem ? attn_fwd_kernel<64, true> : attn_fwd_kernel<64, false>);
  const int smem = D == 128 ? AttnCfg<128>::kSmemBytes : AttnCfg<64>::kSmemBytes;
  static bool configured[4][64] = {{false}};
  const int variant = (D == 128 ? 0 : 2) + (in_tmem ? 1 : 0);
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[variant][dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[variant][dev & 63] = true;
  }
  kernel<<<grid, kAttnThreads, smem, stream>>>(tq, tk, tv, p);
  return static_cast<int>(cudaGetLastError());
}
}
