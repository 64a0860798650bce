// C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) in true fp32: FMA on the CUDA cores, no tensor-core
// mode of reduced precision.  This is the matrix product of the 32-bit path.  The reference has no
// fp32 product at all (ginfer/core/op/kernels/cuda/gemm_kernel/gemm_kernel.cu:166 registers f16 and
// bf16 only).
//
// The order of every sum is fixed by N and K alone, so a row's result does not depend on what else is
// in the batch, nor on which of the two kernels below computes it: K is cut into 2, 4 or 8 segments, a
// segment is two chains of FMAs in ascending k (even and odd k) and their sum, and the segments are
// added in pairs, pairs of pairs, and so on.  The two chains are the halves of fma.rn.f32x2: pairs of
// neighbouring k are what a 16-byte load of either operand holds, and half as many instructions issue.
// (It is not the pipes' rate that asks for pairs: tiles of 64 rows with one FMA an instruction measured the
// same 37 TFLOP/s, half of what the pipes of 148 SMs can do.)
//
//   rows_kernel   up to 16 rows of A, as a decode step has them: bound by reading W once.  A block is
//                 one warp: 32 rows of W and two segments of K, which half a warp each takes; the
//                 segments of a row meet in a cluster.  A lane owns two rows of W, so that what it
//                 reads of A (a 16-byte shared-memory read costs four cycles whether the lanes read
//                 the same or not) is used twice.  cp.async in a ring of its own, three stages deep
//                 where every SM has five such warps, six where it has fewer.
//   tile_kernel   more rows: bound by the FMA pipes and the shared-memory reads alike (8 x 8 outputs a
//                 thread: 64 cycles of either for a warp's step of four k), and with two warps a scheduler,
//                 as many as the accumulators allow, by what either waits for the other.  So the next four
//                 k of A and the next column of W are read ahead, stages are 32 k long (half the barriers),
//                 and a short last tile multiplies the rows that are there only.  Block tiles of 32 or 64
//                 rows by 128 columns, a segment of K (of 128 rows, one block an SM: 128 rows of 17,920 x
//                 1,536 take 231 us, in two tiles 180).
// Measured on a B200 (floor: W's bytes at 6.54 TB/s, or FMAs at 74 TFLOP/s), 3 rows: 17,920 x
// 1,536 in 30 us (floor 17), 1,536 x 8,960 in 23 (8.4), 151,936 x 1,536 in 155 (143); 164 rows, against
// stages of 16 k read as they are multiplied in tiles of 64 whole rows: 17,920 x 1,536 in 233 us (290; floor
// 122), 1,536 x 8,960 in 157 (202; 61), 2,048 x 1,536 in 41 (53); 1,000 rows of the last 174 (240).
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace gf {

namespace cg = cooperative_groups;

constexpr int KS = 8;                                     // segments are multiples of this
constexpr int KU = 32;                                    // k of a stage of the rows kernel

// Segments of K, a function of the matrix alone (it fixes the order of the sums): enough for a few
// blocks an SM; eight where each has 32 k at least, four where each has 8 (short reductions are cut too,
// for shorter chains of roundings).
inline int k_segments(int N, int K) {
  int s = N <= 4096 ? 8 : N <= 32768 ? 4 : 2;
  while (s > 2 && s * (s > 4 ? 4 * KS : KS) > K) s >>= 1;
  return s;
}

// VEC floats to shared memory; zeros where !in (nothing is read then).
template <int VEC>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool in) {
  const uint32_t d = smem_u32(dst);
  const int bytes = in ? VEC * 4 : 0;
  if constexpr (VEC == 4)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two FMAs, of the low and of the high halves.
using f32x2 = unsigned long long;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float halves_sum(f32x2 v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// ---------------------------------------------------------------------------------- few rows
constexpr int RP = KU + 4;                                // pitch of a row of W: 9 x 16 bytes, no conflicts

template <int MT, int STAGES> struct RowsShared {
  float w[STAGES][2][32][RP];
  float x[STAGES][2][MT][KU];
  float sum[2][MT][32];
};

template <int MT, int VEC, int STAGES>
__global__ void __launch_bounds__(32)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W,
                     const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldc, int seg, int ranks) {
  extern __shared__ __align__(16) uint8_t raw[];
  auto& sm = *reinterpret_cast<RowsShared<MT, STAGES>*>(raw);
  const int lane = threadIdx.x, half = lane >> 4, row = lane & 15;
  const int rank = blockIdx.x % ranks, n0 = blockIdx.x / ranks * 32;     // (x: the grid's long side)
  const int kbase = 2 * rank * seg;                       // seg: a multiple of KS
  const int steps = max(0, min(seg, K - kbase) + KU - 1) / KU;
  pdl_trigger();
  pdl_wait();

  auto fetch = [&](int step) {
    if (step < steps) {
      const int st = step % STAGES;
      constexpr int PER = KU / VEC;                       // copies a row
#pragma unroll 16
      for (int e = lane; e < 64 * PER; e += 32) {
        const int h = e / (32 * PER), r = e / PER % 32, kk = (e % PER) * VEC;
        const int at = step * KU + kk, k = kbase + h * seg + at;
        const bool in = n0 + r < N && at < seg && k < K;
        copy_async<VEC>(&sm.w[st][h][r][kk], in ? W + (size_t)(n0 + r) * K + k : W, in);
      }
#pragma unroll
      for (int e = lane; e < 2 * MT * PER; e += 32) {
        const int h = e / (MT * PER), r = e / PER % MT, kk = (e % PER) * VEC;
        const int at = step * KU + kk, k = kbase + h * seg + at;
        const bool in = r < M && at < seg && k < K;
        copy_async<VEC>(&sm.x[st][h][r][kk], in ? A + (size_t)r * lda + k : A, in);
      }
    }
    copy_commit();
  };

  f32x2 acc[2][MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[0][m] = acc[1][m] = 0;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  for (int step = 0; step < steps; ++step) {
    copy_wait<STAGES - 2>();
    __syncwarp();                                         // this step is there, the last one is read
    fetch(step + STAGES - 1);
    const auto& w = sm.w[step % STAGES][half];
    const auto& x = sm.x[step % STAGES][half];
#pragma unroll
    for (int kk = 0; kk < KU; kk += 4) {
      const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&w[row][kk]);
      const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(&w[row + 16][kk]);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&x[m][kk]);
        fma2(acc[0][m], v.x, w0.x);
        fma2(acc[1][m], v.x, w1.x);
        fma2(acc[0][m], v.y, w0.y);
        fma2(acc[1][m], v.y, w1.y);
      }
    }
  }
  copy_wait<0>();
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    sm.sum[half][m][row] = halves_sum(acc[0][m]);
    sm.sum[half][m][row + 16] = halves_sum(acc[1][m]);
  }
  __syncwarp();
  const int n = n0 + lane;
  const float add = bias && n < N ? bias[n] : 0.f;
  if (ranks == 1) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
      if (m < M && n < N) C[(size_t)m * ldc + n] = (sm.sum[0][m][lane] + sm.sum[1][m][lane]) + add;
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int m = rank; m < M; m += ranks) {
    float p[4] = {0.f, 0.f, 0.f, 0.f};                    // (adding the zeros of ranks that are not there is exact)
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (r < ranks) {
        const float* part = cluster.map_shared_rank(&sm.sum[0][m][lane], r);
        p[r] = part[0] + part[MT * 32];
      }
    if (n < N) C[(size_t)m * ldc + n] = ((p[0] + p[1]) + (p[2] + p[3])) + add;
  }
  cluster.sync();                                         // nobody leaves while its sums are read
}

// ---------------------------------------------------------------------------------- more rows
constexpr int BN = 128, OP = BN + 16;
// k of a stage and stages: long stages where a block has enough warps to fill them with 16-byte copies
template <int BM, int VEC> struct TileRing {
  static constexpr int BK = BM >= 64 && VEC == 4 ? 32 : 16, BP = BK + 4, STAGES = BK == 32 ? 3 : 4;
};

template <int BM, int VEC> constexpr size_t tile_shared() {
  using R = TileRing<BM, VEC>;
  const size_t ring = (size_t)R::STAGES * (BM + BN) * R::BP, out = (size_t)BM * OP;
  return (ring > out ? ring : out) * sizeof(float);
}

template <int BM, int VEC>
__global__ void __launch_bounds__(BM * 2, BM == 64 ? 2 : 3)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W,
                     const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldc, int seg, int ranks) {
  extern __shared__ __align__(16) float ring[];           // TILE_STAGES x (BM + BN) rows of BP
  constexpr int THREADS = BM * 2, TY = BM / 8;
  constexpr int BK = TileRing<BM, VEC>::BK, BP = TileRing<BM, VEC>::BP, TILE_STAGES = TileRing<BM, VEC>::STAGES;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int rank = blockIdx.x % ranks, n0 = blockIdx.x / ranks * BN, m0 = blockIdx.y * BM;
  const int kbase = rank * seg;
  const int steps = max(0, min(seg, K - kbase) + BK - 1) / BK;
  pdl_trigger();
  pdl_wait();

  auto fetch = [&](int step) {
    if (step < steps) {
      float* st = ring + (size_t)(step % TILE_STAGES) * (BM + BN) * BP;
      const int k0 = kbase + step * BK, k_end = min(kbase + seg, K);
      constexpr int PER = BK / VEC;
#pragma unroll 8
      for (int e = tid; e < BM * PER; e += THREADS) {
        const int r = e / PER, kk = (e % PER) * VEC, k = k0 + kk;
        const bool in = m0 + r < M && k < k_end;
        copy_async<VEC>(st + r * BP + kk, in ? A + (size_t)(m0 + r) * lda + k : A, in);
      }
#pragma unroll 8
      for (int e = tid; e < BN * PER; e += THREADS) {
        const int r = e / PER, kk = (e % PER) * VEC, k = k0 + kk;
        const bool in = n0 + r < N && k < k_end;
        copy_async<VEC>(st + (BM + r) * BP + kk, in ? W + (size_t)(n0 + r) * K + k : W, in);
      }
    }
    copy_commit();
  };

  f32x2 acc[8][8];                                        // rows ty + TY i, columns tx + 16 j
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;
#pragma unroll
  for (int s = 0; s < TILE_STAGES - 1; ++s) fetch(s);
  // NI: rows a thread has at most (the last tile of rows may be short).  The next four k of A, and the next
  // column of W, are read while the ones at hand are multiplied.
  auto products = [&](auto rows_of) {
    constexpr int NI = decltype(rows_of)::value;
    for (int step = 0; step < steps; ++step) {
      copy_wait<TILE_STAGES - 2>();
      __syncthreads();                                    // this step is there, the last one is read
      fetch(step + TILE_STAGES - 1);
      const float* as = ring + (size_t)(step % TILE_STAGES) * (BM + BN) * BP + ty * BP;
      const float* ws = ring + (size_t)(step % TILE_STAGES) * (BM + BN) * BP + (BM + tx) * BP;
      ulonglong2 a[2][NI], w[2];
#pragma unroll
      for (int i = 0; i < NI; ++i) a[0][i] = *reinterpret_cast<const ulonglong2*>(as + TY * i * BP);
      w[0] = *reinterpret_cast<const ulonglong2*>(ws);
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
        const int now = kk / 4 & 1;
        if (kk + 4 < BK) {
#pragma unroll
          for (int i = 0; i < NI; ++i)
            a[now ^ 1][i] = *reinterpret_cast<const ulonglong2*>(as + TY * i * BP + kk + 4);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (j < 7) w[(j & 1) ^ 1] = *reinterpret_cast<const ulonglong2*>(ws + 16 * (j + 1) * BP + kk);
          else if (kk + 4 < BK) w[(j & 1) ^ 1] = *reinterpret_cast<const ulonglong2*>(ws + kk + 4);
#pragma unroll
          for (int i = 0; i < NI; ++i) fma2(acc[i][j], a[now][i].x, w[j & 1].x);
#pragma unroll
          for (int i = 0; i < NI; ++i) fma2(acc[i][j], a[now][i].y, w[j & 1].y);
        }
      }
    }
  };
  const int most = min(8, (M - m0 + TY - 1) / TY);
  if (BM > 32 && most > 6) products(std::integral_constant<int, 8>{});     // (24 rows at most in tiles of 32)
  else if (most == 6) products(std::integral_constant<int, 6>{});
  else if (most == 5) products(std::integral_constant<int, 5>{});
  else if (most > 2) products(std::integral_constant<int, 4>{});
  else products(std::integral_constant<int, 2>{});
  copy_wait<0>();
  __syncthreads();                                        // the ring becomes the segment's sums
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) ring[(ty + TY * i) * OP + tx + 16 * j] = halves_sum(acc[i][j]);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int rows = BM / ranks;                            // 2, 4 or 8 ranks
  for (int e = tid; e < rows * BN; e += THREADS) {
    const int r = rank * rows + e / BN, m = m0 + r, n = n0 + e % BN;
    if (m >= M || n >= N) continue;
    float p[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < ranks) p[s] = *cluster.map_shared_rank(ring + r * OP + e % BN, s);
    const float v = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
    C[(size_t)m * ldc + n] = v + (bias ? bias[n] : 0.f);
  }
  cluster.sync();
}

struct F32Args {
  const float *A, *W, *bias;
  float* C;
  int M, N, K, lda, ldc, segments, seg;
  cudaStream_t stream;
};

template <typename Kernel>
int start(Kernel* kernel, OncePerDevice& once, int ranks, int columns, int rows, int threads, size_t smem,
          const F32Args& a) {
  const int rc = once.run([&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (rc) return rc;
  return launch_kernel_cluster_dims(kernel, dim3(ranks * columns, rows), dim3(threads), smem, a.stream, ranks,
                                    true, a.A, a.W, a.bias, a.C, a.M, a.N, a.K, a.lda, a.ldc, a.seg, ranks);
}

template <int MT, int VEC, int STAGES> int start_rows_staged(const F32Args& a) {
  static OncePerDevice once;
  return start(gemm_f32_rows_kernel<MT, VEC, STAGES>, once, a.segments / 2, (a.N + 31) / 32, 1, 32,
               sizeof(RowsShared<MT, STAGES>), a);
}

template <int MT, int VEC> int start_rows(const F32Args& a) {
  const long warps = (long)((a.N + 31) / 32) * (a.segments / 2);
  return warps >= 5 * 148 ? start_rows_staged<MT, VEC, 3>(a) : start_rows_staged<MT, VEC, 6>(a);
}

template <int BM, int VEC> int start_tile(const F32Args& a) {
  static OncePerDevice once;
  return start(gemm_f32_tile_kernel<BM, VEC>, once, a.segments, (a.N + BN - 1) / BN, (a.M + BM - 1) / BM,
               BM * 2, tile_shared<BM, VEC>(), a);
}

template <int VEC> int start_by_rows(const F32Args& a) {
  if (a.M <= 1) return start_rows<1, VEC>(a);
  if (a.M <= 2) return start_rows<2, VEC>(a);
  if (a.M <= 4) return start_rows<4, VEC>(a);
  if (a.M <= 8) return start_rows<8, VEC>(a);
  if (a.M <= 16) return start_rows<16, VEC>(a);
  // 25 rows and more leave half of the rows of a tile of 64 out and still gain: its stages are longer and its blocks have
  // four warps.  28 rows, tiles of 32 / 64 (20 rows): 8192 x 2048 54.7 / 37.4 us (40.0 / 37.1), 1536 x 8960 72.9 / 53.9 (51.4 /
  // 53.8), 2048 x 1536 18.2 / 16.4 (14.6 / 16.4), 37888 x 3584 244 / 220 (173 / 216), 17920 x 1536 58.0 / 59.3 (43.3 / 59.1).
  return a.M <= 24 ? start_tile<32, VEC>(a) : start_tile<64, VEC>(a);
}

}  // namespace gf

using namespace gf;

GF_DEFINE_PDL_SWITCH

GF_EXPORT int gf_gemm_f32(const float* A, int lda, const float* W, const float* bias, float* C,
                          int ldc, int M, int N, int K, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  const int segments = k_segments(N, K), units = (K + KS - 1) / KS;
  const F32Args a{A, W, bias, C, M, N, K, lda, ldc, segments, (units + segments - 1) / segments * KS,
                  (cudaStream_t)stream};
  const bool whole = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
  return whole ? start_by_rows<4>(a) : start_by_rows<1>(a);
}
