// bf16 GEMM on CTA pairs: two SMs work on one output tile of 256 x 256 or 256 x 512 with tcgen05.mma.cta_group::2.
//
// What bounds it: the card's power limit.  With real operands the clock falls until it fits, and every byte moved costs clock: a
// 256 x 512 tile moves a quarter less from L2 than a 256 x 256 tile, whose 64 B per SM and tensor cycle are also close to what L2
// delivers.  With all-zero operands, where power does not matter, it runs at 2090 TFLOP/s; products issued by a lone lane (see the
// issuer) stopped at 1290, real operands at 1100 to 1360, now 1270 to 1560 (Qwen3-4B shapes, 8192 to 18432 rows).
// It fills all 512 columns of tensor memory, so the two accumulators cannot belong to two tiles; they are the two halves of one
// (see "Halves").
//
// Layout of the protocol (cluster of 2 CTAs, rank 0 = leader):
//   warp 0   TMA producer of ITS CTA: A rows [m0 + 128*rank, +128) and, of every 256 columns of the tile, 128 rows of B per
//            k-block.  Loads are plain per-CTA copies (no multicast qualifier); the peer's copies signal the LEADER's
//            "full" barrier (cp.async.bulk.tensor ... cta_group::2), which expects the bytes of both CTAs.
//   warp 1   leader only: issues the MMAs, then commits to the "empty" barrier of the stage in BOTH CTAs and,
//            at the end of an accumulator, to its "full" barrier in both CTAs.  Owns the TMEM allocation
//            (both CTAs execute the paired alloc / dealloc).
//   warps 2-9 epilogue of ITS CTA, two warps per 32 accumulator rows: each takes 128 of the accumulator's 256 columns into
//            registers at once and gives the accumulator back (16 arrivals on the leader's barrier: 8 warps x 2 CTAs) before
//            it computes and stores.  Results leave through 4 KB of shared memory per warp and TMA stores (or TMA additions,
//            carried out by L2, for "+="): a row per thread would cost one L1 wavefront per 16 bytes, four times the main loop of a
//            weight gradient over 549 tokens.
// Halves.  NT = 256: a tile uses one of two accumulators in turn, its epilogue overlaps the next tile's main loop.  NT = 512: the
// columns [0, 256) and [256, 512) of a tile are accumulator 0 and 1.  The last k-blocks of a tile are multiplied for half 0
// first, then for half 1, and so are the first ones of the next tile: half 0 is read out while half 1 is finished, half 1 while the
// next tile's half 0 is begun, and the tensor cores do not wait for either.
// Every mbarrier wait is bounded; a CTA whose wait runs out records a status code and unwinds, its partner's
// waits then run out as well, and both meet at the cluster barrier before TMEM is released.
//
// Stands in for the cuBLAS GEMMs behind every nn.Linear of the reference
// (arctic_platform/model/patches/liger.py:25-36 keeps them on cuBLAS).
#include "common.cuh"
#include "gemm_common.cuh"
#include "host_utils.cuh"

namespace apb {

constexpr int kPairBK = 64;
constexpr int kPairBoxBytes = 128 * kPairBK * 2;   // 128 rows of A, or of one half of B
constexpr int kPairEpiWarps = 8;
constexpr int kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr int kPairTmemCols = 512;                 // two fp32 accumulators of 256 columns
constexpr int kPairGroupM = 16;                    // row tiles that are walked before the next column tile

template <int NT>
struct PairCfg {
  static constexpr int kHalves = NT / 256;
  static constexpr int kStageBytes = (1 + kHalves) * kPairBoxBytes;
  static constexpr int kStages = NT == 256 ? 6 : 4;
  static constexpr int kSmem = kStages * kStageBytes + kPairEpiWarps * kStagedBoxBytes + 1024 /*align*/ + 256 /*barriers*/;
};
static_assert(PairCfg<256>::kSmem <= 227 * 1024 && PairCfg<512>::kSmem <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Per-CTA tiled load whose completion bytes are counted on a barrier that may live in the partner CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];"
      ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_holder, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_holder)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on one mbarrier (cluster address: this CTA's or the partner's) once every MMA issued so far is done.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr)
               : "memory");
}

// What a variant of the kernel does with its accumulators.  A kernel holds one of them: with all in one kernel the unrolled code of
// the untaken ones pushed the taken one out of the instruction cache (gate/up of 18432 tokens: 2.6 ms against 0.9).
enum PairEpi : int { kPairBf16, kPairF32, kPairSwiGLU, kPairGeGLU, kPairClampGLU, kPairPartial, kPairDlogits };

// 128 accumulator columns from `nb` on of the rows [row0, row0 + 32), this lane's row in `acc`.  Columns and rows outside the
// output are clipped by the tensor maps; a box that would begin outside is not sent.
template <int EPI>
__device__ __forceinline__ void pair_epilogue(const GemmParams& p, const CUtensorMap& tma_c, const CUtensorMap& tma_c2,
                                              const StagedBox& out, int row0, int nb, const uint32_t (&acc)[4][32]) {
  const int row = row0 + out.lane;
  const bool row_ok = row < p.M;
  if constexpr (EPI == kPairPartial) {
    lmhead_partial_128(p, row, row_ok, acc, nb);
  } else if constexpr (EPI == kPairF32) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (nb + c * 32 >= p.N) break;
      out.begin();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float4 f;
        f.x = __uint_as_float(acc[c][u * 4]) * p.alpha;
        f.y = __uint_as_float(acc[c][u * 4 + 1]) * p.alpha;
        f.z = __uint_as_float(acc[c][u * 4 + 2]) * p.alpha;
        f.w = __uint_as_float(acc[c][u * 4 + 3]) * p.alpha;
        out.put(u, *reinterpret_cast<const uint4*>(&f));
      }
      out.send(&tma_c, nb + c * 32, row0, p.epi != kEpiF32);
    }
  } else {
    constexpr bool glu = EPI == kPairSwiGLU || EPI == kPairGeGLU || EPI == kPairClampGLU;
    if (!glu || p.C != nullptr) {
      LmheadRow lm;
      if constexpr (EPI == kPairDlogits) lm = lmhead_row(p, row, row_ok);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int col0 = nb + c * 64;
        if (col0 >= p.N) break;
        out.begin();
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float a = __uint_as_float(acc[c * 2 + u / 4][(u % 4) * 8 + j]);
            v[j] = EPI == kPairDlogits ? lmhead_dlogit(lm, a, col0 + u * 8 + j) : a * p.alpha;
          }
          if (EPI != kPairDlogits && p.bias && col0 + u * 8 < p.N) {     // N is a multiple of 8
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] += __bfloat162float(p.bias[col0 + u * 8 + j]);
          }
          out.put(u, make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7])));
        }
        out.send(&tma_c, col0, row0, false);
      }
    }
    if constexpr (glu) {
      out.begin();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int i = u * 16 + 2 * j;
          float g = __uint_as_float(acc[i / 32][i % 32]) * p.alpha, x = __uint_as_float(acc[i / 32][i % 32 + 1]) * p.alpha;
          if (p.C && p.bias && nb + i < p.N) {
            g += __bfloat162float(p.bias[nb + i]);
            x += __bfloat162float(p.bias[nb + i + 1]);
          }
          a[j] = EPI == kPairSwiGLU ? silu_f(g) * x : EPI == kPairGeGLU ? gelu_tanh_f(g) * x : clamped_glu_f(g, x, p.glu_limit);
        }
        out.put(u, make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7])));
      }
      out.send(&tma_c2, nb / 2, row0, false);
    }
  }
}

template <int NT, int EPI>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                      const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_c2, const GemmParams p) {
  using Cfg = PairCfg<NT>;
  constexpr int kStages = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_out = smem + kStages * Cfg::kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_out + kPairEpiWarps * kStagedBoxBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tfull_bar = empty_bar + kStages;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_cta_rank();      // 0 = leader
  const bool leader = cta == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  const int tiles_m = (p.M + 255) / 256;
  const int tiles_n = (p.N + NT - 1) / NT;
  const int mn_tiles = tiles_m * tiles_n;
  const int total_tiles = mn_tiles * p.splits;   // work units: output tiles x K splits (split-K adds into C)
  const int k_blocks = (p.K + kPairBK - 1) / kPairBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);    // the leader's arrive.expect_tx; bytes come from both CTAs
      mbar_init(&empty_bar[s], 1);   // one commit by the leader's MMA thread
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);                    // one commit by the leader's MMA thread
      mbar_init(&tempty_bar[b], 2 * kPairEpiWarps);   // the epilogue warps of both CTAs (used in the leader only)
    }
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_holder, kPairTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                // both CTAs' barriers are initialised before anybody signals the partner
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  // Tile order: kPairGroupM m-tiles of one n-band at a time, so pairs running together share B in L2.
  auto decode = [&](int unit, int& m0, int& n0, int& kb0, int& kb1) {
    const int split = unit / mn_tiles;
    const int t = unit - split * mn_tiles;
    kb0 = static_cast<int>((static_cast<long long>(k_blocks) * split) / p.splits);
    kb1 = static_cast<int>((static_cast<long long>(k_blocks) * (split + 1)) / p.splits);
    const int per_group = kPairGroupM * tiles_n;
    const int g = t / per_group;
    const int first_m = g * kPairGroupM;
    const int gsize = min(tiles_m - first_m, kPairGroupM);
    const int r = t - g * per_group;
    m0 = (first_m + r % gsize) * 256;
    n0 = (r / gsize) * NT;
  };
  // accumulators of a tile: its second half may lie outside the output
  auto halves_of = [&](int n0) { return NT == 512 && n0 + 256 < p.N ? 2 : 1; };

  if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += num_pairs) {
        int m0, n0, kb0, kb1;
        decode(t, m0, n0, kb0, kb1);
        const int halves = halves_of(n0);
        const int my_m = m0 + static_cast<int>(cta) * 128;
        const int my_n = n0 + static_cast<int>(cta) * 128;
        // All tiles walk K in the same order: pairs that share a row or a column of tiles in one wave then hit the
        // same operand tiles close together in time, which is what keeps them in L2 (starting every tile at a
        // different k-block was measured: it helps short K and costs up to 10 % at K >= 9728).
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, kTimeoutEmpty)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * Cfg::kStageBytes;
          const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
          if (leader) mbar_expect_tx(&full_bar[stage], 2 * (1 + halves) * kPairBoxBytes);
          if (!p.a_mn) {
            tma_load_2d_pair(sa, &tma_a, bar, kb * kPairBK, my_m);
          } else {
#pragma unroll
            for (int c = 0; c < 2; ++c)
              tma_load_2d_pair(sa + c * (64 * kPairBK * 2), &tma_a, bar, my_m + c * 64, kb * kPairBK);
          }
          for (int h = 0; h < halves; ++h) {
            uint8_t* sb = sa + (1 + h) * kPairBoxBytes;
            if (!p.b_mn) {
              tma_load_2d_pair(sb, &tma_b, bar, kb * kPairBK, my_n + h * 256);
            } else {
#pragma unroll
              for (int c = 0; c < 2; ++c)
                tma_load_2d_pair(sb + c * (64 * kPairBK * 2), &tma_b, bar, my_n + h * 256 + c * 64, kb * kPairBK);
            }
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        // Give copies already issued time to land before shared memory is released.
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 100000ull) {
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    // The whole warp walks the loop and one elected lane issues: stage numbers and descriptors are then uniform, and an MMA
    // costs two additions in front of it.  Built by a lone lane in a divergent branch, every operand went through a copy into
    // uniform registers, and the issue took longer than the 128 cycles of the MMA.
    if (leader) {
      const uint32_t idesc = umma_idesc_bf16(256, 256, p.a_mn, p.b_mn);
      const uint32_t base = smem_u32(smem) >> 4;
      const uint64_t desc_a = umma_smem_desc(0, p.a_mn ? 64 * kPairBK * 2 : 0, 1024) + base;
      const uint64_t desc_b = umma_smem_desc(0, p.b_mn ? 64 * kPairBK * 2 : 0, 1024) + base + (kPairBoxBytes >> 4);
      const uint32_t step_a = (p.a_mn ? 2048 : 32) >> 4, step_b = (p.b_mn ? 2048 : 32) >> 4;
      const uint32_t peer_bars = map_to_cta(smem_u32(full_bar), 1) - smem_u32(full_bar);
      uint32_t stage = 0, phase = 0;
      uint32_t used[2] = {0, 0};      // times that each accumulator has been filled
      int it = 0;
      bool ok = true;
      auto wait_full = [&](uint32_t s, uint32_t ph) {
        const bool r = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, kTimeoutFull));
        tc_fence_after();
        return r;
      };
      auto wait_acc = [&](int slot) {
        const bool r = __all_sync(0xffffffffu, mbar_wait(&tempty_bar[slot], (used[slot] & 1) ^ 1, p.status, kTimeoutTmemEmpty));
        ++used[slot];
        tc_fence_after();
        return r;
      };
      // the MMAs of one stage; `release`: the stage is free in both CTAs once they have read it; `publish`: so is the accumulator
      auto mma = [&](uint32_t s, int half, int slot, bool first, bool release, bool publish) {
        const uint64_t da = desc_a + s * (Cfg::kStageBytes >> 4);
        const uint64_t db = desc_b + s * (Cfg::kStageBytes >> 4) + half * (kPairBoxBytes >> 4);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kPairBK / 16; ++k)
            umma_bf16_ss_pair(tmem_base + slot * 256, da + k * step_a, db + k * step_b, idesc, (!first || k > 0) ? 1u : 0u);
          if (release) {
            const uint32_t eb = smem_u32(&empty_bar[s]);
            tc_commit_pair(eb);
            tc_commit_pair(eb + peer_bars);
          }
          if (publish) {
            const uint32_t tb = smem_u32(&tfull_bar[slot]);
            tc_commit_pair(tb);
            tc_commit_pair(tb + peer_bars);
          }
        }
        __syncwarp();
      };
      for (int t = pair; t < total_tiles && ok; t += num_pairs, ++it) {
        int m0, n0, kb0, kb1;
        decode(t, m0, n0, kb0, kb1);
        const int n = kb1 - kb0, halves = halves_of(n0);
        const int slot0 = NT == 512 ? 0 : (it & 1);
        if (!wait_acc(slot0)) {
          ok = false;
          break;
        }
        // runs of k-blocks: the first and the last kStages of them are walked once per half, the others once
        for (int b = 0; b < n && ok;) {
          const int last = max(kStages, n - kStages);
          const int run = halves == 1 ? 1 : b == 0 ? min(n, kStages) : b >= last ? n - b : 1;
          const bool end = b + run == n;
          uint32_t s = stage, ph = phase;
          for (int i = 0; i < run && ok; ++i) {
            ok = wait_full(s, ph);
            if (!ok) break;
            mma(s, 0, slot0, b + i == 0, halves == 1, end && i == run - 1);
            if (++s == kStages) {
              s = 0;
              ph ^= 1;
            }
          }
          if (!ok) break;
          if (halves == 2) {
            if (b == 0 && !wait_acc(1)) {
              ok = false;
              break;
            }
            uint32_t s1 = stage;
            for (int i = 0; i < run; ++i) {
              mma(s1, 1, 1, b + i == 0, true, end && i == run - 1);
              if (++s1 == kStages) s1 = 0;
            }
          }
          stage = s;
          phase = ph;
          b += run;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs)
    const int quarter = warp & 3;              // TMEM lanes this warp may read
    const int part = (warp - 2) >> 2;          // columns [128 part, +128) of every accumulator
    const StagedBox out{smem_out + (warp - 2) * kStagedBoxBytes, lane};
    uint32_t used[2] = {0, 0};
    int it = 0;
    bool ok = true;
    for (int t = pair; t < total_tiles && ok; t += num_pairs, ++it) {
      int m0, n0, kb0, kb1;
      decode(t, m0, n0, kb0, kb1);
      const int row0 = m0 + static_cast<int>(cta) * 128 + quarter * 32;
      const int halves = halves_of(n0);
      for (int h = 0; h < halves; ++h) {
        const int slot = NT == 512 ? h : (it & 1);
        ok = mbar_wait(&tfull_bar[slot], used[slot] & 1, p.status, kTimeoutTmemFull);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        ++used[slot];
        tc_fence_after();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + slot * 256 + part * 128;
        uint32_t acc[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(taddr + c * 32, acc[c]);
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_wait(acc[c]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[slot]), 0));
        const int nb = n0 + h * 256 + part * 128;
        if (row0 < p.M && nb < p.N) pair_epilogue<EPI>(p, tma_c, tma_c2, out, row0, nb, acc);
      }
    }
    if (lane == 0) tma_out_wait_all();
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // nobody's shared memory or TMEM is still a target of the partner
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kPairTmemCols);
  }
}

// Pairs that can be resident at once (SMs of a pair must sit in one cluster-capable group, so this can be fewer than half the
// SM count).  The grid never exceeds it: a pair that had to wait for a second wave would still take a full share of the tiles.
template <int NT, int EPI>
static int pair_capacity(cudaLaunchConfig_t cfg) {
  static int resident[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!resident[dev & 63]) {
    if (cudaFuncSetAttribute(gemm_bf16_pair_kernel<NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<NT>::kSmem) != cudaSuccess)
      return -static_cast<int>(cudaGetLastError());
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_bf16_pair_kernel<NT, EPI>, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = sm_count() / 2 - 4;        // conservative when the query is unavailable
    }
    resident[dev & 63] = n < sm_count() / 2 ? n : sm_count() / 2;
  }
  return resident[dev & 63];
}

template <int NT, int EPI>
static int launch_pair_as(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tc2,
                       const GemmParams& p, cudaStream_t stream) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = PairCfg<NT>::kSmem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int room = pair_capacity<NT, EPI>(cfg);
  if (room <= 0) return room < 0 ? -room : kBadArgument;
  const long long total = static_cast<long long>((p.M + 255) / 256) * ((p.N + NT - 1) / NT) * p.splits;
  cfg.gridDim = dim3(2 * static_cast<int>(total < room ? total : room));
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_bf16_pair_kernel<NT, EPI>, ta, tb, tc, tc2, p);
  if (e != cudaSuccess) return static_cast<int>(e);
  return static_cast<int>(cudaGetLastError());
}

template <int NT>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tc2,
                       const GemmParams& p, cudaStream_t s) {
  switch (p.epi) {
    case kEpiBf16: return launch_pair_as<NT, kPairBf16>(ta, tb, tc, tc2, p, s);
    case kEpiF32:
    case kEpiF32Accum:
    case kEpiF32Atomic: return launch_pair_as<NT, kPairF32>(ta, tb, tc, tc2, p, s);
    case kEpiSwiGLU: return launch_pair_as<NT, kPairSwiGLU>(ta, tb, tc, tc2, p, s);
    case kEpiGeGLU: return launch_pair_as<NT, kPairGeGLU>(ta, tb, tc, tc2, p, s);
    case kEpiClampGLU: return launch_pair_as<NT, kPairClampGLU>(ta, tb, tc, tc2, p, s);
    case kEpiLogprobPartial: return launch_pair_as<NT, kPairPartial>(ta, tb, tc, tc2, p, s);
    case kEpiDlogits: return launch_pair_as<NT, kPairDlogits>(ta, tb, tc, tc2, p, s);
    default: return kBadArgument;
  }
}

// Launches the kernel on filled-in operands: A and B as boxes of 64 x 128 (64 x 64 transposed).
int launch_gemm_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t stream) {
  CUtensorMap tc = ta, tc2 = ta;               // outputs that the epilogue does not write keep a valid map
  const bool f32 = p.epi == kEpiF32 || p.epi == kEpiF32Accum || p.epi == kEpiF32Atomic;
  if (p.C) {
    const int rc = make_tmap_2d(&tc, p.C, f32 ? 4 : 2, p.M, p.N, p.ldc, f32 ? 32 : 64, 32);
    if (rc) return 3000 + rc;
  }
  if (p.C2) {
    const int rc = make_tmap_2d(&tc2, p.C2, 2, p.M, p.N / 2, p.ldc2, 64, 32);
    if (rc) return 4000 + rc;
  }
  // The width whose waves take less time.  Twice as wide is 0.9 of twice as long where the main loop is long or the weights'
  // gradient is formed (under the power limit, 18432 x 2560 x 19456: 1.40 ms against 1.54; 151936 x 2560 x 16384: 10.8 against
  // 12.4), and a few percent more than twice where its start and end show (18432 x 6144 x 2560: 0.448 ms against 0.427).
  const long long pairs = sm_count() / 2, tm = (p.M + 255) / 256;
  auto waves = [&](int nt) { return (tm * ((p.N + nt - 1) / nt) * p.splits + pairs - 1) / pairs; };
  const bool steady = (p.K + kPairBK - 1) / kPairBK / p.splits >= 96 || (f32 && p.a_mn && p.M >= 4 * p.K);
  if (waves(512) * (steady ? 1.8 : 2.1) < waves(256)) return launch_pair<512>(ta, tb, tc, tc2, p, stream);
  return launch_pair<256>(ta, tb, tc, tc2, p, stream);
}

}  // namespace apb

extern "C" {

// D[M,N] = alpha * op(A) * op(B)^T with the CTA-pair kernel.  Same operand conventions as apb_gemm_bf16
// (a_mn / b_mn, leading dimensions multiples of 8, 16-byte aligned bases).  Epilogues: bf16 (+bias), f32,
// f32 accumulate (split along K by the kernel's own choice when that fills the last wave), the GLU kinds (glu_limit:
// kEpiClampGLU).  No tile table.  Returns kBadArgument for anything else so that the caller can fall back to the one-CTA
// kernel.
int apb_gemm_bf16_pair_glu(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                           long long ldc, int a_mn, int b_mn, int epi, float alpha, const void* bias, void* C2,
                           long long ldc2, float glu_limit, cudaStream_t stream) {
  using namespace apb;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const bool glu = is_glu_epilogue(epi);
  if (epi != kEpiBf16 && epi != kEpiF32 && epi != kEpiF32Accum && !glu) return kBadArgument;
  if ((lda % 8) || (ldb % 8) || (N % 8) || (reinterpret_cast<uintptr_t>(A) & 15) ||
      (reinterpret_cast<uintptr_t>(B) & 15) || (reinterpret_cast<uintptr_t>(C) & 15))
    return kBadArgument;
  if (epi == kEpiBf16 || glu) {
    if (C && (ldc % 8)) return kBadArgument;
    if (epi == kEpiBf16 && !C) return kBadArgument;
  } else if (!C || (ldc % 4)) {
    return kBadArgument;
  }
  if (glu && (!C2 || (ldc2 % 8) || (N % 16))) return kBadArgument;

  CUtensorMap ta, tb;
  int rc;
  if (!a_mn)
    rc = make_tmap_2d(&ta, A, 2, static_cast<uint64_t>(M), static_cast<uint64_t>(K), lda, 64, 128);
  else
    rc = make_tmap_2d(&ta, A, 2, static_cast<uint64_t>(K), static_cast<uint64_t>(M), lda, 64, 64);
  if (rc) return 1000 + rc;
  if (!b_mn)
    rc = make_tmap_2d(&tb, B, 2, static_cast<uint64_t>(N), static_cast<uint64_t>(K), ldb, 64, 128);
  else
    rc = make_tmap_2d(&tb, B, 2, static_cast<uint64_t>(K), static_cast<uint64_t>(N), ldb, 64, 64);
  if (rc) return 2000 + rc;

  GemmParams p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.a_mn = a_mn;
  p.b_mn = b_mn;
  p.epi = epi;
  p.splits = 1;
  p.C = C;
  // Accumulating products (weight gradients: few output tiles, very long K) whose tile count leaves much of the
  // last wave of pairs idle are cut along K; the parts add into C with red.add, which is what "+=" asks for.
  if (epi == kEpiF32Accum) {
    const int k_blocks = (K + kPairBK - 1) / kPairBK;
    const long long tiles = static_cast<long long>((M + 255) / 256) * ((N + 255) / 256);
    const int pairs_hint = sm_count() / 2;
    auto wave_eff = [&](int s) {
      const long long units = tiles * s;
      const long long waves = (units + pairs_hint - 1) / pairs_hint;
      return static_cast<double>(units) / static_cast<double>(waves * pairs_hint);
    };
    int best = 1;
    double best_eff = wave_eff(1);
    for (int s = 2; s <= 16; ++s) {
      if (k_blocks / s < 32) break;
      const double e = wave_eff(s);
      if (e > best_eff + 0.04) {
        best = s;
        best_eff = e;
      }
    }
    if (best > 1) {
      p.splits = best;
      p.epi = kEpiF32Atomic;
    }
  }
  p.ldc = ldc;
  p.C2 = C2;
  p.ldc2 = ldc2;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.alpha = alpha;
  p.glu_limit = glu_limit;
  p.status = status_device_ptr();

  return launch_gemm_pair(ta, tb, p, stream);
}

int apb_gemm_bf16_pair(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                       long long ldc, int a_mn, int b_mn, int epi, float alpha, const void* bias, void* C2,
                       long long ldc2, cudaStream_t stream) {
  if (epi == apb::kEpiClampGLU) return apb::kBadArgument;      // needs its limit
  return apb_gemm_bf16_pair_glu(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, alpha, bias, C2, ldc2, 0.f, stream);
}
}
