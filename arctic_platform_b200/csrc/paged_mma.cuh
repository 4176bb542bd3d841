// Warp-level pieces of decode attention over a paged cache on m16n8k16 MMAs: a page's K and V come through a shared-memory ring of
// the warp (cp.async, 16-byte chunks XOR-swizzled so that the 8 rows of an ldmatrix tile hit 8 different bank groups), the 16 rows of
// a tile hold the query heads of one key head.
#pragma once
#include "common.cuh"

namespace apb {

constexpr int kPage = 16;
constexpr int kMmaPageBytes = kPage * 128 * 2;                    // one K or V page of one head

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One page (K and V, 4 KB each, contiguous in the cache) -> one ring stage; chunk c of row t lands at
// t * 256 + ((c ^ (t & 7)) * 16) so that the 8 rows of an ldmatrix tile hit 8 different bank groups.
__device__ __forceinline__ void decode_issue_page(uint32_t stage_addr, const __nv_bfloat16* kpage,
                                                  const __nv_bfloat16* vpage, int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = i * 32 + lane;  // 16-byte chunk 0..255 of the page
    const int t = c >> 4, col = c & 15;
    const uint32_t off = static_cast<uint32_t>(t * 256 + ((col ^ (t & 7)) << 4));
    cp_async16(stage_addr + off, reinterpret_cast<const uint8_t*>(kpage) + c * 16);
    cp_async16(stage_addr + kMmaPageBytes + off, reinterpret_cast<const uint8_t*>(vpage) + c * 16);
  }
}

// [8][8] bf16, a row per four lanes, to its transpose
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// Running softmax of the 8 H query heads of a key head over the pages that a warp walks.  Both products are taken transposed, S^T =
// K Q^T and O^T += V^T P^T: the 16 rows of a tile are tokens or dimensions and its 8 columns the heads, so nothing is spent on
// rows that a group of 8 heads or less does not have (with the heads as rows a page took twice the MMAs and 40 more registers).
// A lane has heads 2 (lane % 4) and the next one, and of them tokens or dimensions lane / 4 and lane / 4 + 8 of a tile.
template <int H>
struct PagedHeads {
  uint32_t qb[H][8][2];     // Q as B fragments
  float o[H][8][4];         // numerators, a tile per 16 dimensions
  float m[H][2], l[H][2];   // maximum and sum of a head, in units of 2^x

  // q: the first head's row, 128 apart; heads from `heads` on are zeros
  __device__ __forceinline__ void start(const __nv_bfloat16* q, int heads, int lane) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int head = 8 * h + (lane >> 2);
      const bool ok = head < heads;
      const __nv_bfloat16* qp = q + head * 128 + (lane & 3) * 2;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        qb[h][ks][0] = ok ? *reinterpret_cast<const uint32_t*>(qp + ks * 16) : 0u;
        qb[h][ks][1] = ok ? *reinterpret_cast<const uint32_t*>(qp + ks * 16 + 8) : 0u;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) o[h][i][0] = o[h][i][1] = o[h][i][2] = o[h][i][3] = 0.f;
      m[h][0] = m[h][1] = -INFINITY;
      l[h][0] = l[h][1] = 0.f;
    }
  }

  // K and V of one page in a ring stage; `left` of its tokens count (16 or more: all)
  __device__ __forceinline__ void page(uint32_t k_addr, int left, float scale_log2, int lane) {
    const uint32_t v_addr = k_addr + kMmaPageBytes;
    const int mat = lane >> 3, rowin = lane & 7;
    float s[H][4];
#pragma unroll
    for (int h = 0; h < H; ++h) s[h][0] = s[h][1] = s[h][2] = s[h][3] = 0.f;
    {
      const int tok = rowin + 8 * (mat & 1);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const int chunk = ks * 2 + (mat >> 1);
        uint32_t a[4];
        ldsm_x4(k_addr + tok * 256 + ((chunk ^ (tok & 7)) << 4), a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int h = 0; h < H; ++h) mma_16816(s[h], a, qb[h][ks][0], qb[h][ks][1]);
      }
    }
    const bool in0 = (lane >> 2) < left, in1 = (lane >> 2) + 8 < left;
    uint32_t pb[H][2];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      float pr[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float x0 = in0 ? s[h][e] * scale_log2 : -INFINITY, x1 = in1 ? s[h][2 + e] * scale_log2 : -INFINITY;
        float mx = fmaxf(x0, x1);
#pragma unroll
        for (int k = 4; k < 32; k <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, k));
        const float m_new = fmaxf(m[h][e], mx);
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        const float alpha = exp2f(m[h][e] - m_use);       // -inf -> 0
        pr[e] = exp2f(x0 - m_use);
        pr[2 + e] = exp2f(x1 - m_use);
        // sums stay with the lane until the walk ends
        l[h][e] = l[h][e] * alpha + (pr[e] + pr[2 + e]);
        m[h][e] = m_new;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          o[h][i][e] *= alpha;
          o[h][i][2 + e] *= alpha;
        }
      }
      pb[h][0] = transpose_8x8(pack_bf16x2(pr[0], pr[1]));
      pb[h][1] = transpose_8x8(pack_bf16x2(pr[2], pr[3]));
    }
    {
      const int tok = rowin + 8 * (mat >> 1);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int chunk = i * 2 + (mat & 1);
        uint32_t a[4];
        ldsm_x4_t(v_addr + tok * 256 + ((chunk ^ (tok & 7)) << 4), a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int h = 0; h < H; ++h) mma_16816(o[h][i], a, pb[h][0], pb[h][1]);
      }
    }
  }

  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int k = 4; k < 32; k <<= 1) l[h][e] += __shfl_xor_sync(0xffffffffu, l[h][e], k);
  }
};

}  // namespace apb
