// Rows added into a table at given places: the gradients of row look-ups.
//
// Bound by memory: the source is read once (16 bytes per thread) and leaves as vector reductions that the L2 carries out, so
// nothing is sorted, no dense gradient of the table is formed, and rows that nobody names are not touched.  18432 rows of 2560
// into a 151936-row fp32 embedding gradient: 0.10 ms (94 MB read, 189 MB added) against 3.6 ms of the sort, the dense bf16 gradient, its
// fp32 copy and the sum with the accumulated gradient.  Rows that repeat are added in any order: their last bits vary from run to run.
#include "common.cuh"
#include "host_utils.cuh"

namespace apb {

__device__ __forceinline__ void red_add_bf16x8(__nv_bfloat16* dst, const uint4& v) {
  asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}

// dst[index[r], :] += src[r, :], eight columns per thread.
template <typename Dst>
__global__ void __launch_bounds__(256)
rows_add_kernel(const __nv_bfloat16* __restrict__ src, long long ld_src, const long long* __restrict__ index, Dst* __restrict__ dst,
                long long ld_dst, long long dst_rows, int rows, int units) {
  const long long total = static_cast<long long>(rows) * units;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / units), c = static_cast<int>(i - static_cast<long long>(r) * units) * 8;
    const long long to = index[r];
    if (to < 0 || to >= dst_rows) continue;
    const uint4 v = *reinterpret_cast<const uint4*>(src + r * ld_src + c);
    Dst* d = dst + to * ld_dst + c;
    if constexpr (sizeof(Dst) == 2) {
      red_add_bf16x8(d, v);
    } else {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      float2 f[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) f[k] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[k]));
      atomicAdd(reinterpret_cast<float4*>(d), make_float4(f[0].x, f[0].y, f[1].x, f[1].y));
      atomicAdd(reinterpret_cast<float4*>(d) + 1, make_float4(f[2].x, f[2].y, f[3].x, f[3].y));
    }
  }
}

// ---------------------------------------------------------------- rows to experts and back
// Places of the routed (token, expert) pairs in expert-major order: expert e's pairs, in the order of the tokens, from
// sum(roundup(count[e'], pad), e' < e) on.  One CTA per expert; each counts all pairs for itself, so there is one launch and
// nothing to clear, and ranks them with ballots.  35000 pairs over 128 experts: 25 us where sorting took 113.
constexpr int kPlaceThreads = 1024;
constexpr int kPlaceMaxExperts = 512;

__global__ void __launch_bounds__(kPlaceThreads)
moe_place_kernel(const long long* __restrict__ expert, int pairs, int experts, int pad, int* __restrict__ counts,
                 int* __restrict__ place) {
  pdl_entry();
  __shared__ int hist[kPlaceMaxExperts];
  __shared__ int per_warp[kPlaceThreads / 32];
  __shared__ int begin;
  const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < experts; i += kPlaceThreads) hist[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < pairs; i += kPlaceThreads) {
    const long long x = expert[i];
    if (x >= 0 && x < experts) atomicAdd(&hist[x], 1);
    else if (e == 0) place[i] = -1;
  }
  __syncthreads();
  if (warp == 0) {
    int before = 0;
    for (int i = lane; i < e; i += 32) before += (hist[i] + pad - 1) / pad * pad;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) begin = before;
  }
  if (threadIdx.x == 0) counts[e] = hist[e];
  __syncthreads();
  if (hist[e] == 0) return;
  int next = begin;
  for (int base = 0; base < pairs; base += kPlaceThreads) {
    const int i = base + threadIdx.x;
    const bool mine = i < pairs && expert[i] == e;
    const unsigned votes = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) per_warp[warp] = __popc(votes);
    __syncthreads();
    const int n = per_warp[lane];
    int before = lane < warp ? n : 0, all = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, o);
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (mine) place[i] = next + before + __popc(votes & ((1u << lane) - 1));
    next += all;
    __syncthreads();
  }
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// dst[place[t, j]] = src[t] for all j: a token's row is read once.  Memory bound, eight columns per thread.
__global__ void __launch_bounds__(256)
moe_spread_kernel(const __nv_bfloat16* __restrict__ src, long long ld_src, const int* __restrict__ place, int tokens, int k, int units,
                  __nv_bfloat16* __restrict__ dst, long long ld_dst) {
  pdl_entry();
  const long long total = static_cast<long long>(tokens) * units;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(i / units), c = static_cast<int>(i - static_cast<long long>(t) * units) * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(src + t * ld_src + c);
    for (int j = 0; j < k; ++j) {
      const int to = place[t * k + j];
      if (to >= 0) *reinterpret_cast<uint4*>(dst + to * ld_dst + c) = v;
    }
  }
}

// dst[t] = sum_j weight[t, j] src[place[t, j]] (weight null: 1), the rows of a token taken in the order of j, summed in fp32.  Weights
// and weighted rows are rounded to bf16 as an element-wise product of bf16 tensors rounds them: a later layer's router turns last bits
// into other experts, so they are those of the product and sum that this kernel took the place of.
__global__ void __launch_bounds__(256)
moe_collect_kernel(const __nv_bfloat16* __restrict__ src, long long ld_src, const int* __restrict__ place,
                   const float* __restrict__ weight, int tokens, int k, int units, __nv_bfloat16* __restrict__ dst, long long ld_dst) {
  pdl_entry();
  const long long total = static_cast<long long>(tokens) * units;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(i / units), c = static_cast<int>(i - static_cast<long long>(t) * units) * 8;
    float sum[8] = {};
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
      const int from = place[t * k + j];
      if (from < 0) continue;
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(src + from * ld_src + c), f);
      if (weight) {
        const float w = __bfloat162float(__float2bfloat16(weight[t * k + j]));
#pragma unroll
        for (int q = 0; q < 8; ++q) f[q] = __bfloat162float(__float2bfloat16(w * f[q]));
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) sum[q] += f[q];
    }
    *reinterpret_cast<uint4*>(dst + t * ld_dst + c) = pack8(sum);
  }
}

// Gradient of moe_collect: d_src[place[t, j]] = weight[t, j] d[t], d_weight[t, j] = <d[t], src[place[t, j]]>.  One warp per pair.
__global__ void __launch_bounds__(256)
moe_collect_bwd_kernel(const __nv_bfloat16* __restrict__ d, long long ld_d, const __nv_bfloat16* __restrict__ src, long long ld_src,
                       const int* __restrict__ place, const float* __restrict__ weight, int tokens, int k, int units,
                       __nv_bfloat16* __restrict__ d_src, float* __restrict__ d_weight) {
  const int lane = threadIdx.x & 31;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5, pairs = static_cast<long long>(tokens) * k;
  for (long long p = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5; p < pairs; p += warps) {
    const int at = place[p];
    const float w = weight[p];
    float dot = 0.f;
    if (at >= 0) {
      const __nv_bfloat16* a = d + (p / k) * ld_d;
      const __nv_bfloat16* b = src + at * ld_src;
      __nv_bfloat16* o = d_src + at * ld_src;
      for (int u = lane; u < units; u += 32) {
        float f[8], g[8];
        unpack8(*reinterpret_cast<const uint4*>(a + u * 8), f);
        unpack8(*reinterpret_cast<const uint4*>(b + u * 8), g);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          dot += f[q] * g[q];
          f[q] *= w;
        }
        *reinterpret_cast<uint4*>(o + u * 8) = pack8(f);
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) d_weight[p] = dot;
  }
}

static int row_blocks(long long threads, int per_sm) {
  const long long blocks = (threads + 255) / 256, cap = static_cast<long long>(per_sm) * sm_count();
  return static_cast<int>(blocks < cap ? blocks : cap);
}
static bool row_args_ok(int cols, long long ld_a, long long ld_b, const void* a, const void* b) {
  return cols > 0 && cols % 8 == 0 && ld_a % 8 == 0 && ld_b % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}

}  // namespace apb

extern "C" {

// See moe_place_kernel.  expert [pairs] int64 (others than 0..experts-1 get place -1), counts [experts], place [pairs] int32.
int apb_moe_place(const void* expert, int pairs, int experts, int pad, int* counts, int* place, cudaStream_t stream) {
  using namespace apb;
  if (experts <= 0 || experts > kPlaceMaxExperts || pad < 1 || pairs < 0) return kBadArgument;
  return static_cast<int>(launch_kernel(moe_place_kernel, dim3(experts), dim3(kPlaceThreads), 0, stream,
                                        static_cast<const long long*>(expert), pairs, experts, pad, counts, place));
}

// dst[place[t, j]] = src[t]; rows bf16, place [tokens, k].
int apb_moe_spread(const void* src, long long ld_src, const int* place, int tokens, int k, int cols, void* dst, long long ld_dst,
                   cudaStream_t stream) {
  using namespace apb;
  if (tokens <= 0 || k <= 0) return 0;
  if (!row_args_ok(cols, ld_src, ld_dst, src, dst)) return kBadArgument;
  return static_cast<int>(launch_kernel(moe_spread_kernel, dim3(row_blocks(static_cast<long long>(tokens) * (cols / 8), 16)), dim3(256), 0,
                                        stream, static_cast<const __nv_bfloat16*>(src), ld_src, place, tokens, k, cols / 8,
                                        static_cast<__nv_bfloat16*>(dst), ld_dst));
}

// dst[t] = sum_j weight[t, j] src[place[t, j]]; weight fp32 or null.
int apb_moe_collect(const void* src, long long ld_src, const int* place, const float* weight, int tokens, int k, int cols, void* dst,
                    long long ld_dst, cudaStream_t stream) {
  using namespace apb;
  if (tokens <= 0 || k <= 0) return 0;
  if (!row_args_ok(cols, ld_src, ld_dst, src, dst)) return kBadArgument;
  return static_cast<int>(launch_kernel(moe_collect_kernel, dim3(row_blocks(static_cast<long long>(tokens) * (cols / 8), 16)), dim3(256), 0,
                                        stream, static_cast<const __nv_bfloat16*>(src), ld_src, place, weight, tokens, k, cols / 8,
                                        static_cast<__nv_bfloat16*>(dst), ld_dst));
}

// Gradients of the above: d_src rows like src's, d_weight [tokens, k].
int apb_moe_collect_bwd(const void* d, long long ld_d, const void* src, long long ld_src, const int* place, const float* weight,
                        int tokens, int k, int cols, void* d_src, float* d_weight, cudaStream_t stream) {
  using namespace apb;
  if (tokens <= 0 || k <= 0) return 0;
  if (!row_args_ok(cols, ld_d, ld_src, d, src) || (reinterpret_cast<uintptr_t>(d_src) & 15)) return kBadArgument;
  moe_collect_bwd_kernel<<<row_blocks(static_cast<long long>(tokens) * k * 32, 16), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(d), ld_d, static_cast<const __nv_bfloat16*>(src), ld_src, place, weight, tokens, k, cols / 8,
      static_cast<__nv_bfloat16*>(d_src), d_weight);
  return static_cast<int>(cudaGetLastError());
}

// dst[index[r], 0..cols) += src[r, 0..cols) for r < rows; src bf16, dst bf16 or fp32 (dst_f32), index int64.  Places outside
// [0, dst_rows) are left out.  cols and the row strides are multiples of 8, the bases 16-byte aligned.
int apb_rows_add(const void* src, long long ld_src, const void* index, void* dst, long long ld_dst, long long dst_rows, int dst_f32,
                 int rows, int cols, cudaStream_t stream) {
  using namespace apb;
  if (rows <= 0 || cols <= 0) return 0;
  if ((cols % 8) || (ld_src % 8) || (ld_dst % 8) || ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) ||
      (reinterpret_cast<uintptr_t>(index) & 7))
    return kBadArgument;
  const long long blocks = (static_cast<long long>(rows) * (cols / 8) + 255) / 256;
  const long long cap = 16ll * sm_count();
  const int grid = static_cast<int>(blocks < cap ? blocks : cap);
  const auto* s = static_cast<const __nv_bfloat16*>(src);
  const auto* ix = static_cast<const long long*>(index);
  if (dst_f32)
    rows_add_kernel<float><<<grid, 256, 0, stream>>>(s, ld_src, ix, static_cast<float*>(dst), ld_dst, dst_rows, rows, cols / 8);
  else
    rows_add_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(s, ld_src, ix, static_cast<__nv_bfloat16*>(dst), ld_dst, dst_rows, rows,
                                                             cols / 8);
  return static_cast<int>(cudaGetLastError());
}
}
