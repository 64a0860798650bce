// y[M, N] = x[M, K] W[N, K]^T for up to 8 rows of x in bf16, fp32 accumulation: the smaller products of
// decode steps.  What such a product costs is not its bytes (8 MB: 1.3 us) but the way from the release
// of the kernel ahead to its own end.  So weights go from memory straight into the registers that
// mma.sync reads: W's rows are its 16-row operand, x's rows the 8-column one, k is a summed index, so a
// lane may hold any k as long as both operands agree (a lane takes 16 bytes of a row; 4 lanes a 64-byte
// run; two runs a step of 64 k).  A warp loads the first four steps of its weights (8 KB) BEFORE it waits
// for the kernel ahead: a matrix of up to 9.7 MB (eight warps on each of 148 SMs) is then in registers
// when x arrives, and what is left is one trip to L2 for x, the products, the sum over the block's warps
// and the store.  The tcgen05 kernel of gemm_bf16.cu stages both operands through TMA and shared memory,
// reads its accumulator back from tensor memory and sums K splits over a cluster.
//
// A warp owns 16 rows of W and a share of K (PARTS warps of the block's eight a row group); lane group g
// has rows 2 g and 2 g + 1 (a gate and its up value meet in one lane).
// Measured on a B200, weights from HBM, 8 rows, in a graph of products (here / tcgen05 kernel, us): 1024 x
// 1024 2.3 / 3.3, 3200 x 1024 2.8 / 4.0, 2048 x 1536 2.7 / 3.9, 2048 x 2048 3.1 / 4.3.  Larger matrices
// stream better through the other kernel's ring: 1536 x 8960 10.9 / 8.9; and with 9 to 16 rows
// (two column tiles, twice the reads of x) 2048 x 2048 took 5.1 / 4.3, so neither comes here.
#include "common.cuh"

namespace gf {

constexpr int WARPS = 8, RING = 4;                           // steps of 64 k under way a warp
enum { ST_STORE = 0, ST_RELU2 = 1, ST_GATED = 2, ST_XIELU = 4 };

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Weights are read once: past L1, and without a claim on it.
__device__ __forceinline__ uint4 load_weights(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

struct StreamArgs {
  const bf16* x;
  const bf16* w;
  const float* bias;       // [N] or null; ST_GATED: {limit, alpha, shift} or null
  void* out;
  int ldx, ldo, M, N, K;
  float a, b;              // ST_XIELU
};

template <int PARTS, int EPI, typename OUT>
__global__ void __launch_bounds__(WARPS * 32, 2)
gemm_stream_kernel(const StreamArgs args) {
  __shared__ float sums[PARTS > 1 ? WARPS : 1][4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int part = warp % PARTS;
  const int M = args.M, N = args.N, K = args.K;
  const int n = (blockIdx.x * (WARPS / PARTS) + warp / PARTS) * 16 + 2 * g;
  const int units = (K + 63) / 64, u0 = units * part / PARTS, u1 = units * (part + 1) / PARTS;
  const bf16* w0 = args.w + (size_t)(n < N ? n : 0) * K + 8 * t;
  const int next = n + 1 < N ? K : 0;                        // to the second row
  const int k_end = min(u1 * 64, K) - 8 * t;                 // this lane's runs start before it
  uint4 wa[RING][2], wb[RING][2];
  auto load_w = [&](int slot, int u) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = u * 64 + h * 32;
      wa[slot][h] = wb[slot][h] = make_uint4(0u, 0u, 0u, 0u);
      if (k < k_end) wa[slot][h] = load_weights(w0 + k), wb[slot][h] = load_weights(w0 + k + next);
    }
  };
#pragma unroll
  for (int i = 0; i < RING; ++i) load_w(i, u0 + i);
  float b0 = 0.f, b1 = 0.f;
  if (EPI != ST_GATED && args.bias) b0 = n < N ? args.bias[n] : 0.f, b1 = n + 1 < N ? args.bias[n + 1] : 0.f;
  // The kernel behind may only start now: earlier, its own loads (a large product's ring) compete with
  // those that this chain waits for (8 requests, 32 experts: 30.7 -> 28.6 ms for the whole batch).
  pdl_wait();
  pdl_trigger();

  // x from L2: this block may have shared its SM with readers of what the buffer held before, and no two
  // warps read the same of it.
  uint4 xs[2][2];
  const bf16* xr = args.x + (size_t)(g < M ? g : 0) * args.ldx + 8 * t;
  auto load_x = [&](int slot, int u) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = u * 64 + h * 32;
      xs[slot][h] = make_uint4(0u, 0u, 0u, 0u);
      if (g < M && k < k_end) xs[slot][h] = __ldcg(reinterpret_cast<const uint4*>(xr + k));
    }
  };
  load_x(0, u0);
  load_x(1, u0 + 1);
  float acc[4] = {0.f, 0.f, 0.f, 0.f};                       // rows 2 t, 2 t + 1 of x by rows n | n + 1 of W
  for (int u = u0; u < u1; u += RING)
#pragma unroll
    for (int i = 0; i < RING; ++i) {                         // (steps behind u1 multiply zeros)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 a = wa[i][h], c = wb[i][h], v = xs[i & 1][h];
        mma_16816(acc, a.x, c.x, a.y, c.y, v.x, v.y);
        mma_16816(acc, a.z, c.z, a.w, c.w, v.z, v.w);
      }
      load_w(i, u + i + RING);
      load_x(i & 1, u + i + 2);
    }
  if (PARTS > 1) {                                           // the first of a group's warps adds up
#pragma unroll
    for (int e = 0; e < 4; ++e) sums[warp][e][lane] = acc[e];
    __syncthreads();
    if (part) return;
#pragma unroll
    for (int p = 1; p < PARTS; ++p)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] += sums[warp + p][e][lane];
  }
  if (n >= N) return;
  OUT* out = reinterpret_cast<OUT*>(args.out);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = 2 * t + i;
    if (m >= M) continue;
    float v0 = acc[i], v1 = acc[2 + i];
    if constexpr (EPI == ST_GATED) {
      out[(size_t)m * args.ldo + (n >> 1)] = from_f32<OUT>(gated_activation(v0, v1, args.bias));
    } else {
      v0 += b0, v1 += b1;
      if (EPI == ST_RELU2) v0 = fmaxf(v0, 0.f), v1 = fmaxf(v1, 0.f), v0 *= v0, v1 *= v1;
      if (EPI == ST_XIELU) v0 = xielu(v0, args.a, args.b), v1 = xielu(v1, args.a, args.b);
      OUT* dst = out + (size_t)m * args.ldo + n;
      if (n + 1 < N && (args.ldo & 1) == 0) {
        if constexpr (sizeof(OUT) == 2)
          *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(v0, v1);
        else
          *reinterpret_cast<float2*>(dst) = make_float2(v0, v1);
      } else {
        dst[0] = from_f32<OUT>(v0);
        if (n + 1 < N) dst[1] = from_f32<OUT>(v1);
      }
    }
  }
}

template <int EPI, typename OUT> int start_stream(const StreamArgs& a, int parts, cudaStream_t st) {
  const int groups = (a.N + 15) / 16;
#define GF_GO(PARTS)                                                                                   \
  if (parts == PARTS)                                                                                  \
    return launch_kernel(gemm_stream_kernel<PARTS, EPI, OUT>,                                          \
                         dim3((groups + WARPS / PARTS - 1) / (WARPS / PARTS)), dim3(WARPS * 32), 0, st, a);
  GF_GO(1) GF_GO(2) GF_GO(4) GF_GO(8)
#undef GF_GO
  return -6;
}

}  // namespace gf

using namespace gf;

GF_DEFINE_PDL_SWITCH

// x [M <= 8, K] (rows ldx apart), w [N, K] bf16; bias fp32 [N] or null; epi: 0 (+ bias), 1 relu(.)^2, 2 gated
// (weight rows gate, up, gate, up, ...; out [M, N / 2]; bias: {limit, alpha, shift} or null), 4 xIELU.
// parts: warps that share a row's reduction (1, 2, 4, 8), 0 picks.  Returns -6 for what it does not take.
GF_EXPORT int gf_gemm_stream(const void* x, int ldx, const void* w, const float* bias, void* out, int ldo,
                             int M, int N, int K, int epi, int out_f32, float act_a, float act_b,
                             int parts, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 8 || K <= 0 || K % 8 || ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) ||
      ((uintptr_t)out & 7) || (epi == ST_GATED && ((N & 1) || out_f32)))
    return -6;
  if (parts == 0) {
    // about 8 warps an SM at least, and no share of less than two steps: measured, the most parts that
    // leave every warp two steps are the best up to matrices of 10 MB
    parts = 1;
    while (parts < 8 && (long long)((N + 15) / 16) * parts < 148 * 8 && K >= parts * 256) parts *= 2;
  }
  const StreamArgs a{(const bf16*)x, (const bf16*)w, bias, out, ldx, ldo, M, N, K, act_a, act_b};
  auto st = (cudaStream_t)stream;
  if (epi == ST_GATED) return start_stream<ST_GATED, bf16>(a, parts, st);
  if (epi == ST_STORE)
    return out_f32 ? start_stream<ST_STORE, float>(a, parts, st) : start_stream<ST_STORE, bf16>(a, parts, st);
  if (epi == ST_RELU2)
    return out_f32 ? start_stream<ST_RELU2, float>(a, parts, st) : start_stream<ST_RELU2, bf16>(a, parts, st);
  if (epi == ST_XIELU)
    return out_f32 ? start_stream<ST_XIELU, float>(a, parts, st) : start_stream<ST_XIELU, bf16>(a, parts, st);
  return -6;
}
