// Segment attention backward on tcgen05 tensor cores (see attention_fwd.cu for
// the segment model).  One CTA owns one key block (128 rows of one KV head) and
// walks every 128-row query tile that can see it -- all query heads of the KV
// head, and under ZoRRo all rollouts that share the prompt the block belongs to
// -- so dK and dV of a shared prompt are accumulated in tensor memory and written
// once.  The reference gets these sums from autograd through torch.cat copies of
// the prompt K/V (arctic_platform/rl/zorro_train/zorro_train.py:857-912).
//
// Per query tile, with S and dP transposed so that TMEM lanes are key rows:
//   S^T  = K  Q^T          dP^T = V dO^T                     (tensor core)
//   P^T  = exp2(S^T*c - lse[q])     dS^T = P^T*(dP^T - delta[q])     (two groups of 128 threads, 64 columns each)
//   dV  += P^T dO          dK  += dS^T Q        dQ = dS K          (tensor core)
// P^T overwrites S^T in TMEM and is the TMEM A operand of the dV product; dS^T goes
// to shared memory once and is read by two products (K-major for dK, M-major for
// dQ).  The softmax scale that dS lacks is applied to dK and dQ where they leave.
//
// What bounds it: five products of 128 x 128 x 128, 2560 tensor cycles per tile.  Tensor memory (512 columns) holds S^T / P^T,
// dP^T, dK and dV; dQ takes dP^T's place once dS^T has been formed.  The products are issued in the order
//   S(i+1)  dQ(i)  dK(i)  dP(i+1)  dV(i+1)
// so that each waits for something that was ready earlier: the exponentials of tile i+1 have the time of three products, dS(i) that
// of dV(i) and S(i+1), the read-out of dQ(i) that of dK(i).  dQ is read by a group of its own and leaves as TMA additions of
// 32 x 32 boxes.  One sequence of 16384 tokens, 32 query and 8 key heads: 5.7 ms (960 TFLOP/s; the products alone 4.3).  Before:
// 64-row tiles (their 64-wide products alone 6.8 ms, since the operands saturate shared memory) 10.3 with dQ added by TMA, 13 with
// red.add of one float per lane.
#include "attention_common.cuh"
#include "host_utils.cuh"

namespace apb {

struct AttnBwdParams {
  const int* cta;   // [n_cta][8]  kv_row0, kv_valid, kvh, list_off, list_cnt
  const int* list;  // [n_list][4] q_row0, q_valid, diag_rel
  int Hq, Hkv, T;
  float scale, scale_log2;
  const float* lse;    // [Hq, T]
  const float* delta;  // [Hq, T]
  __nv_bfloat16* dk;   // [T, Hkv*D]
  __nv_bfloat16* dv;
  long long ld_dk, ld_dv;
  int* status;
};

// Four warpgroups: producer and MMA issuer; two for P and dS; one for dQ.  Registers are moved from the first to the others:
// 56 + 3 * 152 = 4 * 128, what the block was launched with.
constexpr int kBwdThreads = 512;
constexpr int kBwdRegsIssue = 56, kBwdRegsWork = 152;
constexpr int kBwdTile = 128;            // query rows and key rows
constexpr int kBigDiag = 1 << 27;

template <int D>
struct AttnBwdCfg {
  static_assert(D == 128, "tensor memory and the dQ boxes are laid out for heads of 128");
  static constexpr int kTileBytes = kBwdTile * D * 2;
  static constexpr int kHeadBytes = 2 * 128 * 4 + 2 * 128 * 4 + 128;   // -lse and -delta of two tiles, barriers
  // statistics and barriers lie in front, the tiles from the next multiple of 1024 on
  static constexpr int kSmemBytes = 3072 + 6 * kTileBytes /*K, V, 2 Q, dO, dS*/ + 8 * kStagedBoxBytes;
  static_assert(kHeadBytes <= 3072 - 896 && kSmemBytes <= 227 * 1024, "shared memory of one CTA");
};

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_do,
                const __grid_constant__ CUtensorMap tma_k, const __grid_constant__ CUtensorMap tma_v,
                const __grid_constant__ CUtensorMap tma_dq, const AttnBwdParams p) {
  using Cfg = AttnBwdCfg<D>;
  constexpr int kTileBytes = Cfg::kTileBytes;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  float* smem_lse = reinterpret_cast<float*>(smem_raw);        // [2][128]
  float* smem_delta = smem_lse + 256;                          // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_delta + 256);
  uint64_t* q_full = bars;            // [2]  copy and statistics
  uint64_t* q_empty = bars + 2;       // [2]
  uint64_t* do_full = bars + 4;       // copy and statistics
  uint64_t* do_empty = bars + 5;
  uint64_t* kv_full = bars + 6;
  uint64_t* s_full = bars + 7;        // S^T of a tile is there
  uint64_t* p_full = bars + 8;        // (256 arrivals) P^T written
  uint64_t* dp_full = bars + 9;       // dP^T is there
  uint64_t* ds_full = bars + 10;      // (256 arrivals) dS^T in shared memory, dP^T read
  uint64_t* dq_full = bars + 11;      // dQ is there
  uint64_t* dq_read = bars + 12;      // (128 arrivals) dQ has been read
  uint64_t* dkv_full = bars + 13;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 14);
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + Cfg::kHeadBytes + 1023) & ~uintptr_t(1023));
  uint8_t* smem_k = smem;
  uint8_t* smem_v = smem + kTileBytes;
  uint8_t* smem_q = smem + 2 * kTileBytes;       // [2]
  uint8_t* smem_do = smem + 4 * kTileBytes;
  uint8_t* smem_ds = smem + 5 * kTileBytes;      // [column half][128 key rows][64 bf16]
  uint8_t* smem_out = smem + 6 * kTileBytes;     // [warp][2] boxes of dQ on their way out

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int* c = p.cta + static_cast<long long>(blockIdx.x) * 8;
  const int kv_row0 = c[0], kv_valid = c[1], kvh = c[2], list_off = c[3], list_cnt = c[4];
  const int ratio = p.Hq / p.Hkv;
  const int n_iter = list_cnt * ratio;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 2);
      mbar_init(&q_empty[s], 1);
    }
    mbar_init(do_full, 2);
    mbar_init(do_empty, 1);
    mbar_init(kv_full, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 256);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, 256);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, 128);
    mbar_init(dkv_full, 1);
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
  constexpr uint32_t kColS = 0, kColDP = 128, kColDK = 256, kColDV = 384;

  // a wait of a whole warp
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
    const bool r = __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, code));
    tc_fence_after();
    return r;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kBwdRegsIssue));
    if (warp == 0 && n_iter > 0) {
      // ---------------------------------------------------------------- producer (whole warp)
      if (lane == 0) {
        mbar_expect_tx(kv_full, 2 * kTileBytes);
        for (int ch = 0; ch < D / 64; ++ch) {
          tma_load_2d(smem_k + ch * 16384, &tma_k, kv_full, kvh * D + ch * 64, kv_row0);
          tma_load_2d(smem_v + ch * 16384, &tma_v, kv_full, kvh * D + ch * 64, kv_row0);
        }
      }
      bool ok = true;
      int hd = 0;
      const int* e = p.list + static_cast<long long>(list_off) * 4;
      for (int i = 0; i < n_iter && ok; ++i) {
        const int s = i & 1;
        const int q_row0 = e[0];
        const int head = kvh * ratio + hd;
        if (++hd == ratio) {
          hd = 0;
          e += 4;
        }
        // the statistics are on their way while the buffers are waited for
        const float* lse = p.lse + static_cast<long long>(head) * p.T + q_row0;
        const float* delta = p.delta + static_cast<long long>(head) * p.T + q_row0;
        float a[4], d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = q_row0 + lane + 32 * j < p.T;
          a[j] = in ? -lse[lane + 32 * j] * 1.4426950408889634f : 0.f;
          d[j] = in ? -delta[lane + 32 * j] : 0.f;
        }
        ok = wait(&q_empty[s], ((i >> 1) & 1) ^ 1, kTimeoutEmpty);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(&q_full[s], kTileBytes);
          for (int ch = 0; ch < D / 64; ++ch)
            tma_load_2d(smem_q + s * kTileBytes + ch * 16384, &tma_q, &q_full[s], head * D + ch * 64, q_row0);
        }
        // (tile i - 2's -lse and -delta were read before its P^T and dS^T were published, and dK(i - 2) came after both)
#pragma unroll
        for (int j = 0; j < 4; ++j) smem_lse[s * 128 + lane + 32 * j] = a[j];
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full[s]);
        ok = wait(do_empty, (i & 1) ^ 1, kTimeoutEmpty);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(do_full, kTileBytes);
          for (int ch = 0; ch < D / 64; ++ch) tma_load_2d(smem_do + ch * 16384, &tma_do, do_full, head * D + ch * 64, q_row0);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) smem_delta[s * 128 + lane + 32 * j] = d[j];
        __syncwarp();
        if (lane == 0) mbar_arrive(do_full);
      }
      if (!ok && lane == 0) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 100000ull) {
        }
      }
    } else if (warp == 1 && n_iter > 0) {
      // -------------------------------------------------------------- MMA issuer (whole warp, one elected lane issues: see
      // gemm_tcgen05_2cta.cu)
      const uint32_t idesc_kk = umma_idesc_bf16(128, 128, 0, 0);        // S^T, dP^T : A K-major, B K-major
      const uint32_t idesc_kn = umma_idesc_bf16(128, 128, 0, 1);        // dV, dK    : A K-major, B N-major
      const uint32_t idesc_mn = umma_idesc_bf16(128, 128, 1, 1);        // dQ        : A M-major, B N-major
      auto kmajor = [&](const uint8_t* t) { return umma_smem_desc(smem_u32(t), 0, 1024); };
      auto nmajor = [&](const uint8_t* t) { return umma_smem_desc(smem_u32(t), 16384, 1024); };
      const uint64_t k_k = kmajor(smem_k), v_k = kmajor(smem_v), k_n = nmajor(smem_k), q_k = kmajor(smem_q), q_n = nmajor(smem_q),
                     do_k = kmajor(smem_do), do_n = nmajor(smem_do), ds_k = kmajor(smem_ds), ds_m = nmajor(smem_ds);
      constexpr uint32_t kTile = kTileBytes >> 4;
      // by the elected lane: one product, eight steps of 16; a K-major operand advances within 64-column chunks, an M- or
      // N-major one by 16 rows
      auto product = [&](uint32_t col, uint64_t a, bool a_rows, uint64_t b, bool b_rows, uint32_t idesc, bool first) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + col, a + (a_rows ? k * 128 : (k / 4) * 1024 + (k % 4) * 2),
                       b + (b_rows ? k * 128 : (k / 4) * 1024 + (k % 4) * 2), idesc, (!first || k > 0) ? 1u : 0u);
      };
      auto scores_of = [&](uint32_t s) {
        if (elect_one()) {
          product(kColS, k_k, false, q_k + s * kTile, false, idesc_kk, true);
          tc_commit(s_full);
        }
        __syncwarp();
      };
      auto dp_of = [&]() {
        if (elect_one()) {
          product(kColDP, v_k, false, do_k, false, idesc_kk, true);
          tc_commit(dp_full);
        }
        __syncwarp();
      };
      auto dv_of = [&](bool first) {       // P^T: columns [0, 64) in TMEM columns [0, 32), columns [64, 128) in [64, 96)
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_bf16_ts(tmem_base + kColDV, tmem_base + kColS + (k / 4) * 64 + (k % 4) * 8, do_n + k * 128, idesc_kn,
                         (!first || k > 0) ? 1u : 0u);
          tc_commit(do_empty);
        }
        __syncwarp();
      };
      bool ok = wait(kv_full, 0, kTimeoutFull) && wait(&q_full[0], 0, kTimeoutFull);
      if (ok) {
        scores_of(0);
        ok = wait(do_full, 0, kTimeoutFull);
      }
      if (ok) {
        dp_of();
        ok = wait(p_full, 0, kTimeoutTmemEmpty);
      }
      if (ok) dv_of(true);
      for (int i = 0; i < n_iter && ok; ++i) {
        const uint32_t par = i & 1, s = i & 1;
        const bool next = i + 1 < n_iter;
        // S(i+1) over P(i), which dV(i) has read: the tensor core executes one CTA's MMAs in issue order
        if (next) {
          ok = wait(&q_full[s ^ 1], ((i + 1) >> 1) & 1, kTimeoutFull);
          if (!ok) break;
          scores_of(s ^ 1);
        }
        ok = wait(ds_full, par, kTimeoutTmemEmpty);
        if (!ok) break;
        if (elect_one()) {
          product(kColDP, ds_m, true, k_n, true, idesc_mn, true);
          tc_commit(dq_full);
          product(kColDK, ds_k, false, q_n + s * kTile, true, idesc_kn, i == 0);
          tc_commit(&q_empty[s]);
          if (!next) tc_commit(dkv_full);
        }
        __syncwarp();
        if (next) {
          ok = wait(do_full, par ^ 1, kTimeoutFull) && wait(dq_read, par, kTimeoutTmemEmpty);
          if (!ok) break;
          dp_of();
          ok = wait(p_full, par ^ 1, kTimeoutTmemEmpty);
          if (!ok) break;
          dv_of(false);
        }
      }
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ P and dS: 64 columns of every tile per group
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kBwdRegsWork));
    const int quarter = warp & 3;
    const int grp = (warp >> 2) - 1;
    const int r = quarter * 32 + lane;  // key row of the block
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const bool row_ok = r < kv_valid;
    const uint32_t t_s = tmem_base + lane_off + kColS + grp * 64, t_dp = tmem_base + lane_off + kColDP + grp * 64;
    uint8_t* ds_row = smem_ds + grp * 16384 + r * 128;
    const uint64_t c2 = xtc_pair(p.scale_log2, p.scale_log2);
    bool ok = true;
    int hd = 0;
    const int4* e = reinterpret_cast<const int4*>(p.list) + list_off;
    for (int i = 0; i < n_iter; ++i) {
      const int s = i & 1;
      const uint32_t par = i & 1;
      const int q_valid = e->y - grp * 64, diag = e->z + grp * 64;      // of this group's columns
      if (++hd == ratio) {
        hd = 0;
        ++e;
      }
      // Columns that some rows do not see (the diagonal, the block's and the tile's end) take the masked form
      const bool all = kv_valid == kBwdTile && q_valid >= 64 && diag >= 127;
      const int c_min = !row_ok ? 64 : diag >= kBigDiag ? 0 : r - diag;
      ok = wait(&q_full[s], (i >> 1) & 1, kTimeoutFull) && wait(s_full, par, kTimeoutTmemFull);
      if (!ok) break;
      uint64_t pr[32];                  // P^T in pairs of columns
      {
        const ulonglong2* nlse = reinterpret_cast<const ulonglong2*>(smem_lse + s * 128 + grp * 64);
        uint32_t v[2][32], pk[32];
        tmem_ld_32x32(t_s, v[0]);
        tmem_ld_32x32(t_s + 32, v[1]);
        tmem_ld_wait(v[0]);
        tmem_ld_wait(v[1]);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const ulonglong2 n = nlse[u];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = 4 * u + 2 * h;
            float2 f = xtc_unpair(xtc_fma2(xtc_pair(__uint_as_float(v[col / 32][col % 32]), __uint_as_float(v[col / 32][col % 32 + 1])),
                                           c2, h ? n.y : n.x));
            f.x = xtc_ex2(f.x);
            f.y = xtc_ex2(f.y);
            if (!all) {
              if (col < c_min || col >= q_valid) f.x = 0.f;
              if (col + 1 < c_min || col + 1 >= q_valid) f.y = 0.f;
            }
            pr[col / 2] = xtc_pair(f.x, f.y);
            pk[col / 2] = pack_bf16x2(f.x, f.y);
          }
        }
        tmem_st_32x32(t_s, pk);
        tmem_st_wait();
      }
      // dO (and -delta, which comes with it) is seen before P^T is published: dV(i), which needs P^T alone of this group, gives dO's
      // buffer back, and its barrier may then pass tile i + 1's phase before a warp that was held up here has looked at tile i's.
      ok = wait(do_full, par, kTimeoutFull);
      if (!ok) break;
      tc_fence_before();
      mbar_arrive(p_full);
      ok = wait(dp_full, par, kTimeoutTmemFull);
      if (!ok) break;
      const ulonglong2* ndelta = reinterpret_cast<const ulonglong2*>(smem_delta + s * 128 + grp * 64);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        tmem_ld_32x32(t_dp + half * 32, v);
        tmem_ld_wait(v);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint32_t o[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const ulonglong2 n = ndelta[half * 8 + u * 2 + h];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int col = u * 8 + h * 4 + j * 2;
              const uint64_t w = pr[half * 16 + col / 2];
              float2 f = xtc_unpair(
                  xtc_mul2(w, xtc_add2(xtc_pair(__uint_as_float(v[col]), __uint_as_float(v[col + 1])), j ? n.y : n.x)));
              if (!all) {                            // whatever dP^T holds where a row does not see the column
                const float2 q = xtc_unpair(w);
                if (q.x == 0.f) f.x = 0.f;
                if (q.y == 0.f) f.y = 0.f;
              }
              o[h * 2 + j] = pack_bf16x2(f.x, f.y);
            }
          }
          *reinterpret_cast<uint4*>(ds_row + (((half * 4 + u) ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(ds_full);
    }
    // dK (first group) and dV (second) of this block.  The TMEM loads are warp collectives: every lane runs them, only the
    // global stores are predicated on the row being inside the block.
    if (ok && n_iter > 0) ok = wait(dkv_full, 0, kTimeoutTmemFull);
    if (ok) {
      __nv_bfloat16* dst = grp ? p.dv + (static_cast<long long>(kv_row0) + r) * p.ld_dv : p.dk + (static_cast<long long>(kv_row0) + r) * p.ld_dk;
      dst += static_cast<long long>(kvh) * D;
      const float scale = grp ? 1.f : p.scale;
#pragma unroll 1
      for (int h = 0; h < D / 32; ++h) {
        uint32_t v[32];
        if (n_iter > 0) {  // uniform across the CTA
          tmem_ld_32x32(tmem_base + lane_off + (grp ? kColDV : kColDK) + h * 32, v);
          tmem_ld_wait(v);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(v[q * 8 + 0]) * scale, __uint_as_float(v[q * 8 + 1]) * scale);
            o.y = pack_bf16x2(__uint_as_float(v[q * 8 + 2]) * scale, __uint_as_float(v[q * 8 + 3]) * scale);
            o.z = pack_bf16x2(__uint_as_float(v[q * 8 + 4]) * scale, __uint_as_float(v[q * 8 + 5]) * scale);
            o.w = pack_bf16x2(__uint_as_float(v[q * 8 + 6]) * scale, __uint_as_float(v[q * 8 + 7]) * scale);
            *reinterpret_cast<uint4*>(dst + h * 32 + q * 8) = o;
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dQ: one query row per thread
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kBwdRegsWork));
    const int quarter = warp & 3;
    const uint32_t t_dq = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + kColDP;
    uint8_t* boxes = smem_out + quarter * 2 * kStagedBoxBytes;
    int hd = 0;
    const int4* e = reinterpret_cast<const int4*>(p.list) + list_off;
    for (int i = 0; i < n_iter; ++i) {
      const int q_row0 = e->x, rows = e->y - quarter * 32;      // rows of this warp that belong to the tile
      const int head = kvh * ratio + hd;
      if (++hd == ratio) {
        hd = 0;
        ++e;
      }
      if (!wait(dq_full, i & 1, kTimeoutTmemFull)) break;
      uint32_t v[4][32];
#pragma unroll
      for (int b = 0; b < 4; ++b) tmem_ld_32x32(t_dq + b * 32, v[b]);
#pragma unroll
      for (int b = 0; b < 4; ++b) tmem_ld_wait(v[b]);
      tc_fence_before();
      mbar_arrive(dq_read);
      if (rows <= 0) continue;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const StagedBox out{boxes + (b & 1) * kStagedBoxBytes, lane};
        out.begin<1>();
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          float4 f = make_float4(__uint_as_float(v[b][u * 4]) * p.scale, __uint_as_float(v[b][u * 4 + 1]) * p.scale,
                                 __uint_as_float(v[b][u * 4 + 2]) * p.scale, __uint_as_float(v[b][u * 4 + 3]) * p.scale);
          if (lane >= rows) f = make_float4(0.f, 0.f, 0.f, 0.f);       // rows of another segment: whatever dS holds there
          out.put(u, *reinterpret_cast<const uint4*>(&f));
        }
        out.send(&tma_dq, head * D + b * 32, q_row0 + quarter * 32, true);
      }
    }
    if (lane == 0) tma_out_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[h, t] = sum_d dO[t,h,d] * O[t,h,d] for heads of 128; 16 lanes per (t, h), 16 bytes of each per lane.
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, long long ldo, const __nv_bfloat16* __restrict__ d_o, long long lddo,
                  float* __restrict__ delta, int T, int Hq) {
  const long long gw = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 4;
  const int lane = threadIdx.x & 15;
  const bool ok = gw < static_cast<long long>(T) * Hq;
  const int t = ok ? static_cast<int>(gw / Hq) : 0, h = ok ? static_cast<int>(gw % Hq) : 0;
  const uint4 x = *reinterpret_cast<const uint4*>(o + t * ldo + static_cast<long long>(h) * 128 + lane * 8);
  const uint4 y = *reinterpret_cast<const uint4*>(d_o + t * lddo + static_cast<long long>(h) * 128 + lane * 8);
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xs[i]));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ys[i]));
    acc += a.x * b.x + a.y * b.y;
  }
#pragma unroll
  for (int s = 8; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (ok && lane == 0) delta[static_cast<long long>(h) * T + t] = acc;
}

}  // namespace apb

extern "C" {

// Backward of apb_attn_fwd_form for head_dim 128.
//   q/o/d_o [T, Hq*D], k/v [T, Hkv*D] bf16 with row strides ld*; lse [Hq,T] from the forward.
//   delta [Hq,T] fp32 scratch (written here); dq_acc [T, Hq*D] fp32 accumulator, zeroed by the caller;
//   dk/dv [T, Hkv*D] bf16 outputs.  cta/list are the tables of apb_rt_attn_bwd_work.
int apb_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                 float* delta, float* dq_acc, void* dk, void* dv, const int* cta, int n_cta, const int* list, int T,
                 int Hq, int Hkv, int D, long long ldq, long long ldk, long long ldv, long long ldo, long long lddo,
                 long long ld_dq, long long ld_dk, long long ld_dv, float scale, cudaStream_t stream) {
  using namespace apb;
  if (n_cta <= 0 || T <= 0) return 0;
  if (D != 128 || (ld_dq % 4) || (ldq % 8) || (ldk % 8) || (ldv % 8) || (ldo % 8) || (lddo % 8) || (ld_dk % 8) || (ld_dv % 8) || Hq % Hkv ||
      ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(d_o)) & 15))
    return kBadArgument;
  {
    const int grid = static_cast<int>((static_cast<long long>(T) * Hq * 16 + 255) / 256);
    attn_delta_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(o), ldo,
                                                static_cast<const __nv_bfloat16*>(d_o), lddo, delta, T, Hq);
  }
  CUtensorMap tq, tdo, tk, tv, tdq;
  int rc = make_tmap_2d(&tq, q, 2, T, static_cast<uint64_t>(Hq) * D, ldq, 64, kBwdTile);
  if (rc) return 1000 + rc;
  rc = make_tmap_2d(&tdo, d_o, 2, T, static_cast<uint64_t>(Hq) * D, lddo, 64, kBwdTile);
  if (rc) return 2000 + rc;
  rc = make_tmap_2d(&tk, k, 2, T, static_cast<uint64_t>(Hkv) * D, ldk, 64, 128);
  if (rc) return 3000 + rc;
  rc = make_tmap_2d(&tv, v, 2, T, static_cast<uint64_t>(Hkv) * D, ldv, 64, 128);
  if (rc) return 4000 + rc;
  rc = make_tmap_2d(&tdq, dq_acc, 4, T, static_cast<uint64_t>(Hq) * D, ld_dq, 32, 32);
  if (rc) return 5000 + rc;
  AttnBwdParams p;
  p.cta = cta;
  p.list = list;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.T = T;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = lse;
  p.delta = delta;
  p.dk = static_cast<__nv_bfloat16*>(dk);
  p.dv = static_cast<__nv_bfloat16*>(dv);
  p.ld_dk = ld_dk;
  p.ld_dv = ld_dv;
  p.status = status_device_ptr();
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         AttnBwdCfg<128>::kSmemBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev & 63] = true;
  }
  attn_bwd_kernel<128><<<n_cta, kBwdThreads, AttnBwdCfg<128>::kSmemBytes, stream>>>(tq, tdo, tk, tv, tdq, p);
  return static_cast<int>(cudaGetLastError());
}
}
