// Routed feed-forward (mixture of experts) without a host round trip: every kernel reads the
// routing from device memory, so a step can be captured in a CUDA graph.
//
//   moe_route_kernel    a warp a token: scores = softmax(router logits) in fp32 over all experts
//                       (or the sigmoid of each logit), the `top` largest chosen (lowest index
//                       among equals), their scores kept as weights (optionally renormalised over
//                       the chosen ones).
//   moe_route_grouped_kernel  the same over groups of neighbouring experts, chosen by scores that a
//                       correction shifts: only experts of the groups with the largest best score can be
//                       chosen; the last outputs may be experts without matrices (identity), whose
//                       weights are added up per token; the row may hold a gate's logit as well.
//   moe_plan_kernel     a block an expert: (token, choice) pairs counted per expert, the experts' ranges in
//                       the sorted order, each pair's place, and the list of row tiles (expert,
//                       first row) that the grouped products walk over.
//   moe_stream_kernel   the grouped products of decode steps: an expert's weights streamed once (see there).
//   moe_ring_kernel     those of one to two and a half pairs an expert, where that grid takes more than a round.
//   moe_gemv_kernel     those of a handful of pairs for layers that stay off it (see there).
//   moe_gemm_mma_kernel those of more pairs, in tiles of 64 rows (see there).
//   moe_gemm_kernel     (32-bit path, and sizes the other refuses) grouped product over the sorted pairs, a block a (row tile, column tile):
//                       FIRST: rows gathered from the tokens, W = the expert's row-interleaved
//                       gate/up matrix, epilogue = clamped sigmoid-gated GLU (MODE 1), or W = the
//                       expert's up matrix, epilogue = relu(w * acc)^2 with the pair's routing
//                       weight w, which is the product of the row scaled by w (MODE 2); else
//                       (MODE 0) rows = the first product's output, W = the expert's down matrix,
//                       fp32 out.  The reduction runs in a fixed order, so a pair's result does
//                       not depend on the batch.
//   moe_combine_kernel  out[t] = sum over the token's choices, in the order chosen, of weight *
//                       the pair's row.
#include <cmath>
#include <type_traits>

#include "common.cuh"

namespace gf {

constexpr int kMaxExperts = 256;
constexpr int kRouteSlots = kMaxExperts / 32;

__global__ void moe_route_kernel(const float* __restrict__ logits, int T, int E, int top,
                                 int renorm, int sigmoid, int* __restrict__ idx,
                                 float* __restrict__ wgt) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  if (t >= T) return;
  float s[kRouteSlots];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < kRouteSlots; ++i) {
    const int e = lane + 32 * i;
    s[i] = e < E ? logits[(size_t)t * E + e] : -INFINITY;
    mx = fmaxf(mx, s[i]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kRouteSlots; ++i) {
    const float sc = sigmoid ? 1.f / (1.f + expf(-s[i])) : expf(s[i] - mx);
    s[i] = lane + 32 * i < E ? sc : -1.f;                    // -1: no expert, or taken
    sum += s[i] > 0.f ? s[i] : 0.f;
  }
  sum = sigmoid ? 1.f : warp_sum(sum);
  float chosen_sum = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -1.f;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < kRouteSlots; ++i)
      if (s[i] > best) best = s[i], be = lane + 32 * i;       // ascending e: lowest index wins
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ob > best || (ob == best && oe < be)) best = ob, be = oe;
    }
#pragma unroll
    for (int i = 0; i < kRouteSlots; ++i)
      if (lane + 32 * i == be) s[i] = -1.f;
    chosen_sum += best;
    if (lane == 0) {
      idx[(size_t)t * top + k] = be;
      wgt[(size_t)t * top + k] = best / sum;
    }
  }
  if (renorm) {
    __syncwarp();
    if (lane < top) wgt[(size_t)t * top + lane] *= sum / chosen_sum;
  }
}

// logits: rows of ld floats, E router outputs first: E - identity experts with matrices, then the
// identity ones.  Scores s = softmax over all E; choice scores c = s + correction (null: s).  groups > 1:
// equal groups of E / groups neighbours, a group's score the largest c in it, the `keep` best groups
// stay (lowest index among equals).  Of their experts the `top` with the largest c are chosen (lowest
// index among equals).  idx: the expert, or -1 for an identity one; wgt: its s (0 for an identity one);
// identity_w[t]: the sum of the identity ones' s (null: not wanted).  gate[t] = sigmoid(row[gate_col])
// (null: no gate).  always > 0: every token has that many more pairs behind its choices, of the experts
// E - identity, E - identity + 1, ..., with its gate as weight (rows of idx and wgt are top + always long).
// SLOTS: router outputs a lane.
template <int SLOTS>
__global__ void moe_route_grouped_kernel(const float* __restrict__ logits, int ld, int T, int E,
                                         int identity, int top, int groups, int keep,
                                         const float* __restrict__ correction, int gate_col,
                                         int always, int* __restrict__ idx, float* __restrict__ wgt,
                                         float* __restrict__ identity_w,
                                         float* __restrict__ gate) {
  constexpr int kW = 4;                                       // warps a block
  __shared__ float gscore[kW][kMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * kW + warp;
  pdl_trigger();
  pdl_wait();
  if (t >= T) return;                                         // (warps are independent)
  const float* row = logits + (size_t)t * ld;
  float s[SLOTS], c[SLOTS];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    const int e = lane + 32 * i;
    s[i] = e < E ? row[e] : -INFINITY;
    mx = fmaxf(mx, s[i]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    s[i] = expf(s[i] - mx);                                   // 0 past the last expert
    sum += s[i];
  }
  sum = warp_sum(sum);
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    const int e = lane + 32 * i;
    s[i] = s[i] / sum;
    c[i] = e < E ? s[i] + (correction ? correction[e] : 0.f) : -INFINITY;
  }
  if (groups > 1 && keep < groups) {
    const int gs = E / groups;
    float* gsc = gscore[warp];
    for (int g = 0; g < groups; ++g) {
      float best = -INFINITY;
#pragma unroll
      for (int i = 0; i < SLOTS; ++i) {
        const int e = lane + 32 * i;
        if (e >= g * gs && e < (g + 1) * gs) best = fmaxf(best, c[i]);
      }
      best = warp_max(best);
      if (lane == 0) gsc[g] = best;
    }
    __syncwarp();
    // a group stays if fewer than `keep` groups come before it (larger, or equal with a lower index)
#pragma unroll
    for (int i = 0; i < SLOTS; ++i) {
      const int e = lane + 32 * i;
      if (e >= E) continue;
      const int g = e / gs;
      int ahead = 0;
      for (int o = 0; o < groups; ++o) ahead += gsc[o] > gsc[g] || (gsc[o] == gsc[g] && o < g);
      if (ahead >= keep) c[i] = -INFINITY;
    }
  }
  const int E0 = E - identity, ldk = top + always;
  float id_sum = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < SLOTS; ++i)
      if (c[i] > best) best = c[i], be = lane + 32 * i;       // ascending e: lowest index wins
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ob > best || (ob == best && oe < be)) best = ob, be = oe;
    }
    float w = 0.f;
#pragma unroll
    for (int i = 0; i < SLOTS; ++i)
      if (lane + 32 * i == be) w = s[i], c[i] = -INFINITY;
    w = __shfl_sync(0xffffffffu, w, be & 31);
    const bool none = be >= E0;                               // an identity expert (or none is left)
    if (none) id_sum += w;
    if (lane == 0) {
      idx[(size_t)t * ldk + k] = none ? -1 : be;
      wgt[(size_t)t * ldk + k] = none ? 0.f : w;
    }
  }
  if (lane == 0 && identity_w) identity_w[t] = id_sum;
  if (gate_col >= 0) {
    const float gt = 1.f / (1.f + expf(-row[gate_col]));
    if (lane == 0 && gate) gate[t] = gt;
    if (lane < always) {
      idx[(size_t)t * ldk + top + lane] = E0 + lane;
      wgt[(size_t)t * ldk + top + lane] = gt;
    }
  }
}

// Pairs p = t * top + k.  offsets[E + 1]; pos_of_pair[P]; pair_of_pos[P]; tiles: tile_expert[],
// tile_row0[] (first sorted row of the tile), num_tiles[0].  A pair whose expert is -1 has no place
// (pos_of_pair -1): the sorted order then holds offsets[E] < P pairs.
// A block an expert (one SM could not keep up: 8,192 pairs took 29 us in one block).  Every block
// counts all experts' pairs for itself, so that it knows where its expert's rows and tiles begin
// without waiting for another block; then its warps take equal runs of the pairs, count their
// expert's pairs in them, and place them behind the runs before: a pair's place is the number of
// earlier pairs of the same expert, whatever the grid.
constexpr int kPlanThreads = 256, kPlanWarps = kPlanThreads / 32;
__global__ void __launch_bounds__(kPlanThreads)
moe_plan_kernel(const int* __restrict__ idx, int P, int E, int tile_rows, int stage,
                int* __restrict__ offsets, int* __restrict__ pos_of_pair,
                int* __restrict__ pair_of_pos, int* __restrict__ tile_expert,
                int* __restrict__ tile_row0, int* __restrict__ num_tiles) {
  __shared__ int count[kMaxExperts], run_count[kPlanWarps], base[2];
  extern __shared__ int held[];                    // the pairs' experts, if they fit
  const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  for (int i = threadIdx.x; i < E; i += blockDim.x) count[i] = 0;
  if (stage)
#pragma unroll 8
    for (int p = threadIdx.x; p < P; p += blockDim.x) held[p] = fresh_index(idx + p);
  __syncthreads();
  auto expert_of = [&](int p) { return stage ? held[p] : fresh_index(idx + p); };
  // this block's expert by ballots over the warps' runs; the others by shared atomics
  const int run = (((P + kPlanWarps - 1) / kPlanWarps) + 31) & ~31;
  const int p_lo = warp * run, p_hi = min(P, p_lo + run);
  int mine_in_run = 0;
  for (int p0 = p_lo; p0 < p_hi; p0 += 32) {
    const int p = p0 + lane;
    const int g = p < p_hi ? expert_of(p) : -1;
    if (g >= 0 && g != e) atomicAdd(&count[g], 1);
    mine_in_run += __popc(__ballot_sync(0xffffffffu, g == e));
  }
  if (lane == 0) run_count[warp] = mine_in_run;
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int w = 0; w < kPlanWarps; ++w) n += run_count[w];
    count[e] = n;
    int at = 0, nt = 0;
    for (int i = 0; i < e; ++i) {
      at += count[i];
      nt += (count[i] + tile_rows - 1) / tile_rows;
    }
    base[0] = at;
    base[1] = nt;
    offsets[e] = at;
    if (e == E - 1) {
      offsets[E] = at + n;
      num_tiles[0] = nt + (n + tile_rows - 1) / tile_rows;
    }
  }
  __syncthreads();
  const int start = base[0], n_mine = count[e];
  for (int r = threadIdx.x * tile_rows; r < n_mine; r += blockDim.x * tile_rows) {
    tile_expert[base[1] + r / tile_rows] = e;
    tile_row0[base[1] + r / tile_rows] = start + r;
  }
  int at = start;
  for (int w = 0; w < warp; ++w) at += run_count[w];
  for (int p0 = p_lo; p0 < p_hi; p0 += 32) {
    const int p = p0 + lane;
    const int g = p < p_hi ? expert_of(p) : e + 1;
    const bool mine = g == e;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (mine) {
      const int pos = at + __popc(m & ((1u << lane) - 1));
      pos_of_pair[p] = pos;
      pair_of_pos[pos] = p;
    }
    at += __popc(m);
    if (e == 0 && g < 0) pos_of_pair[p] = -1;
  }
}

__device__ __forceinline__ float clamped_glu(float g, float u, float limit, float alpha,
                                             float up_shift) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  if (alpha < 0.f) return fmaxf(g, 0.f) * (u + up_shift);   // the sigmoid sharpened to a step: relu
  return g / (1.f + expf(-alpha * g)) * (u + up_shift);
}

constexpr int kBM = 32, kBN = 64, kBK = 32;

// MODE 1: a [T, K] tokens (row of sorted place s = pair_of_pos[s] / top), w [E, 2F, K] (gate row,
// up row, ...), out [P, F] of type T.  MODE 2: the same rows, w [E, F, K], out [P, F] of type T =
// relu(row_w[pair] * acc)^2 (row_w null: 1).  MODE 0: a [P, K] (T), w [E, N, K], out [P, N] fp32.
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
moe_gemm_kernel(const T* __restrict__ a, int lda, const T* __restrict__ w, int N, int K,
                const int* __restrict__ offsets, const int* __restrict__ pair_of_pos, int top,
                const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                const int* __restrict__ num_tiles, void* __restrict__ out_, float limit,
                float alpha, float up_shift, const float* __restrict__ row_w) {
  constexpr bool FIRST = MODE != 0;
  __shared__ float As[kBM][kBK + 1], Ws[kBN][kBK + 1];
  __shared__ int src_row[kBM];
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= fresh_index(num_tiles)) return;
  const int e = fresh_index(tile_expert + blockIdx.x), row0 = fresh_index(tile_row0 + blockIdx.x);
  const int rows = min(kBM, fresh_index(offsets + e + 1) - row0);
  const int n0 = blockIdx.y * kBN;
  const T* we = w + (size_t)e * N * K;
  if (threadIdx.x < kBM) {
    const int s = row0 + threadIdx.x;
    src_row[threadIdx.x] = threadIdx.x < rows ? (FIRST ? fresh_index(pair_of_pos + s) / top : s) : -1;
  }
  __syncthreads();
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;    // rows 2 ty, 2 ty + 1; cols 4 tx ..
  float acc[2][4] = {};
  for (int k0 = 0; k0 < K; k0 += kBK) {
    for (int i = threadIdx.x; i < kBM * kBK; i += 256) {
      const int r = i / kBK, k = i - r * kBK;
      const int sr = src_row[r];
      As[r][k] = (sr >= 0 && k0 + k < K) ? to_f32(a[(size_t)sr * lda + k0 + k]) : 0.f;
    }
    for (int i = threadIdx.x; i < kBN * kBK; i += 256) {
      const int n = i / kBK, k = i - n * kBK;
      Ws[n][k] = (n0 + n < N && k0 + k < K) ? to_f32(we[(size_t)(n0 + n) * K + k0 + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kBK; ++k) {
      const float a0 = As[2 * ty][k], a1 = As[2 * ty + 1][k];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float b = Ws[4 * tx + j][k];
        acc[0][j] = fmaf(a0, b, acc[0][j]);
        acc[1][j] = fmaf(a1, b, acc[1][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = 2 * ty + i;
    if (r >= rows) continue;
    const size_t s = (size_t)(row0 + r);
    if (MODE == 2) {
      T* out = (T*)out_;
      const float rw = row_w ? row_w[pair_of_pos[s]] : 1.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + 4 * tx + j;
        if (n < N) {
          const float u = fmaxf(to_f32(from_f32<T>(acc[i][j] * rw)), 0.f);
          out[s * N + n] = from_f32<T>(u * u);
        }
      }
    } else if (MODE == 1) {
      T* out = (T*)out_;
      const int F = N / 2;
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const int n = n0 + 4 * tx + j;
        if (n < N) {
          // gate and up are rounded to the activation type as a plain product would store them
          const float gt = to_f32(from_f32<T>(acc[i][j])), up = to_f32(from_f32<T>(acc[i][j + 1]));
          out[s * F + n / 2] = from_f32<T>(clamped_glu(gt, up, limit, alpha, up_shift));
        }
      }
    } else {
      float* out = (float*)out_;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + 4 * tx + j;
        if (n < N) out[s * N + n] = acc[i][j];
      }
    }
  }
}


// ---- the same grouped products on the tensor cores (bf16 operands, fp32 accumulation) -----------
// Tile 64 rows x 128 columns x 32 of the reduction; 8 warps as 2 x 4, a warp 32 x 32 (2 x 4
// mma.sync.m16n8k16 a k-step).  Operand tiles come through three stages of shared memory by 16-byte
// cp.async (rows 40 halves apart: fragment loads meet every bank once); rows past an expert's range
// are zero-filled.  Needs K and the row strides to be multiples of 8 and 16-byte aligned bases.
constexpr int kTM = 64, kTN = 128, kTK = 32, kTStages = 3, kTLd = kTK + 8;

__device__ __forceinline__ void cp_async_16(void* dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3,
                                        const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_u32(p)));
}

template <int MODE>
__global__ void __launch_bounds__(256)
moe_gemm_mma_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w,
                    int N, int K, const int* __restrict__ offsets,
                    const int* __restrict__ pair_of_pos, int top,
                    const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                    const int* __restrict__ num_tiles, void* __restrict__ out_, float limit,
                    float alpha, float up_shift, const float* __restrict__ row_w) {
  constexpr bool FIRST = MODE != 0;
  __shared__ __align__(16) __nv_bfloat16 As[kTStages][kTM][kTLd];
  __shared__ __align__(16) __nv_bfloat16 Ws[kTStages][kTN][kTLd];
  __shared__ int src_row[kTM];
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= fresh_index(num_tiles)) return;
  const int e = fresh_index(tile_expert + blockIdx.x), row0 = fresh_index(tile_row0 + blockIdx.x);
  const int rows = min(kTM, fresh_index(offsets + e + 1) - row0);
  const int n0 = blockIdx.y * kTN;
  const __nv_bfloat16* we = w + (size_t)e * N * K;
  if (threadIdx.x < kTM) {
    const int s = row0 + threadIdx.x;
    src_row[threadIdx.x] = threadIdx.x < rows ? (FIRST ? fresh_index(pair_of_pos + s) / top : s) : -1;
  }
  __syncthreads();
  const int nk = (K + kTK - 1) / kTK;
  auto ask = [&](int kb) {
    const int st = kb % kTStages, k0 = kb * kTK;
    {                                              // A: 64 rows x 4 pieces of 8
      const int r = threadIdx.x >> 2, c = (threadIdx.x & 3) * 8;
      const int sr = src_row[r];
      const bool ok = sr >= 0 && k0 + c < K;
      cp_async_16(&As[st][r][c], ok ? a + (size_t)sr * lda + k0 + c : a, ok);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {                  // W: 128 rows x 4 pieces of 8
      const int id = threadIdx.x + 256 * i;
      const int r = id >> 2, c = (id & 3) * 8;
      const bool ok = n0 + r < N && k0 + c < K;
      cp_async_16(&Ws[st][r][c], ok ? we + (size_t)(n0 + r) * K + k0 + c : we, ok);
    }
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp >> 2, wn = warp & 3;         // the warp's 32 x 32 part
  const int g = lane >> 2, t = lane & 3;
  float acc[2][4][4] = {};
  for (int s = 0; s < kTStages - 1; ++s) {
    if (s < nk) ask(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kb = 0; kb < nk; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kTStages - 2) : "memory");
    __syncthreads();                               // stage kb has landed; stage kb - 1 is free
    if (kb + kTStages - 1 < nk) ask(kb + kTStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int st = kb % kTStages;
#pragma unroll
    for (int kk = 0; kk < kTK; kk += 16) {
      uint32_t af[2][4], bfr[4][2];
      // ldmatrix: A 16 x 16 (lanes 0-15 the rows, lanes 16-31 the second 8 of k); B two column
      // tiles at once (lanes 0-7 / 8-15: the first tile's rows at k / k + 8, lanes 16-31 the second's)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        ldsm_x4(af[i][0], af[i][1], af[i][2], af[i][3],
                &As[st][wm * 32 + i * 16 + (lane & 15)][kk + ((lane >> 4) << 3)]);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
        ldsm_x4(bfr[2 * jj][0], bfr[2 * jj][1], bfr[2 * jj + 1][0], bfr[2 * jj + 1][1],
                &Ws[st][wn * 32 + jj * 16 + (lane & 7) + ((lane >> 4) << 3)]
                   [kk + (((lane >> 3) & 1) << 3)]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], af[i], bfr[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // c0, c1: row g, columns 2t, 2t + 1; c2, c3: row g + 8
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int r = wm * 32 + i * 16 + g + 8 * hh;
      if (r >= rows) continue;
      const size_t s = (size_t)(row0 + r);
      const float rw = (MODE == 2 && row_w) ? row_w[pair_of_pos[s]] : 1.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + wn * 32 + j * 8 + 2 * t;
        const float c0 = acc[i][j][2 * hh], c1 = acc[i][j][2 * hh + 1];
        if (MODE == 2) {
          __nv_bfloat16* out = (__nv_bfloat16*)out_ + s * N;
          const float u0 = fmaxf(to_f32(from_f32<__nv_bfloat16>(c0 * rw)), 0.f);
          const float u1 = fmaxf(to_f32(from_f32<__nv_bfloat16>(c1 * rw)), 0.f);
          if (n < N) out[n] = from_f32<__nv_bfloat16>(u0 * u0);
          if (n + 1 < N) out[n + 1] = from_f32<__nv_bfloat16>(u1 * u1);
        } else if (MODE == 1) {
          if (n < N) {
            const float gt = to_f32(from_f32<__nv_bfloat16>(c0)), up = to_f32(from_f32<__nv_bfloat16>(c1));
            ((__nv_bfloat16*)out_)[s * (N / 2) + n / 2] =
                from_f32<__nv_bfloat16>(clamped_glu(gt, up, limit, alpha, up_shift));
          }
        } else {
          float* out = (float*)out_ + s * N;
          if (n < N) out[n] = c0;
          if (n + 1 < N) out[n + 1] = c1;
        }
      }
    }
}

// ---- the same grouped products where the experts' weight bytes are the work (decode steps) --------
// Up to some hundred pairs every expert that is reached has a few rows, and its matrix is read once for
// them: the time is the stream of weights.  The weights are the 16-row operand of mma.sync and go from
// memory straight into its registers (k is a summed index, so a lane may hold any k as long as both
// operands agree: a lane takes 16 bytes of a row, 4 lanes a 64-byte run, two runs a step of 64 k);
// the pairs' rows, at most 16 of one expert, are staged in shared memory and are the 8-column operand.
// No weight is staged, so a warp keeps 8 loads of 16 bytes a lane under way whatever the other warps do.
// A warp owns 16 weight rows; `parts` warps (1, 2, 4 or 8 of the block's eight) split its reduction
// where the rows alone give too few warps.  `parts` is the order of a pair's sums, so it follows from the
// matrices and from a step's range (up to 20 pairs, up to 16 an expert, more), not from its pairs'
// number: within a range a pair's result does not depend on the batch.  (Steps that ring_serves() takes, from a number
// of pairs on that follows from the matrices up to two and a half an expert, are a range of their own.)  Against `parts` from the number
// itself (both products, weights from HBM, us): 32 experts of 2048 x 2112, 8 pairs 69.6 -> 63.6, 20 pairs 107
// -> 109; 8 of 2048 x 1408, 24 pairs 45 -> 49, 64 pairs 61.5 -> 57.4; elsewhere within 3 %, or faster.  Lane group g has weight rows 2 g and 2 g + 1: a gate and
// its up value meet in one lane.
// Measured on a B200 (both products of a layer, 32 experts of 2048 x 2112, 4 choices; floor = the
// reached experts' bytes at 6.54 TB/s), against a kernel that kept eight rows in shared memory and
// multiplied on the FMA pipes (up to 20 pairs) and the 64-row tiles below (from 21 on): 4 pairs 26.5
// us (29.5; floor 10.6), 20 pairs 53.5 (97.5; 39.6), 64 pairs 91.6 (120; 60.8), 256 pairs 113.5 (172; 82),
// 512 pairs 144.5 (182; 84.6), 1,020 pairs 214 (209: the line lies at 768).
constexpr int kStRows = 16, kStWarps = 8, kStUnroll = 2;
constexpr int kStMaxShared = 160 * 1024;                     // K up to 5,056
// The tiles of rows that `parts` reckons with: for a handful of pairs, at most otherwise.
constexpr int kStHandful = 20, kStHandfulTiles = 12, kStTiles = 32;

__host__ __device__ inline size_t stream_pitch(int K) {      // of a staged row, bytes: 64 mod 128
  return ((size_t)K * 2 + 127) / 128 * 128 + 64;
}

template <int MODE>
__global__ void __launch_bounds__(kStWarps * 32, 2)
moe_stream_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w,
                  int N, int K, const int* __restrict__ offsets, const int* __restrict__ pair_of_pos,
                  int top, const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                  const int* __restrict__ num_tiles, void* __restrict__ out_, float limit,
                  float alpha, float up_shift, const float* __restrict__ row_w, int parts) {
  extern __shared__ __align__(16) uint8_t staged[];          // [kStRows] rows of stream_pitch(K)
  __shared__ float sums[kStWarps][32][8];
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= fresh_index(num_tiles)) return;
  const int e = fresh_index(tile_expert + blockIdx.x), row0 = fresh_index(tile_row0 + blockIdx.x);
  const int rows = min(kStRows, fresh_index(offsets + e + 1) - row0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int part = warp % parts, n0 = (blockIdx.y * (kStWarps / parts) + warp / parts) * 16;
  const size_t pitch = stream_pitch(K);
  const int units = (K + 63) / 64;
  const int u0 = units * part / parts, u1 = units * (part + 1) / parts;
  const int n = n0 + 2 * g;                                  // N is even: both rows are there, or none
  const __nv_bfloat16* w0 = w + ((size_t)e * N + (n < N ? n : 0)) * K + 8 * t;
  const __nv_bfloat16* w1 = w0 + K;
  uint4 ra[kStUnroll][2], rb[kStUnroll][2];                  // rows 2 g and 2 g + 1
  auto load = [&](int u) {
#pragma unroll
    for (int i = 0; i < kStUnroll; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = (u + i) * 64 + h * 32;
        ra[i][h] = rb[i][h] = make_uint4(0u, 0u, 0u, 0u);
        if (u + i < u1 && k + 8 * t < K) {
          ra[i][h] = __ldg(reinterpret_cast<const uint4*>(w0 + k));
          rb[i][h] = __ldg(reinterpret_cast<const uint4*>(w1 + k));
        }
      }
  };
  load(u0);
  {                                                          // the rows, zeros up to whole steps
    const int k8 = units * 8, staged_rows = rows <= 8 ? 8 : 16;
    for (int i = threadIdx.x; i < staged_rows * k8; i += kStWarps * 32) {
      const int r = i / k8, c = (i - r * k8) * 8;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < rows && c < K) {
        const int src = MODE != 0 ? fresh_index(pair_of_pos + row0 + r) / top : row0 + r;
        v = __ldcg(reinterpret_cast<const uint4*>(a + (size_t)src * lda + c));
      }
      *reinterpret_cast<uint4*>(staged + r * pitch + (size_t)c * 2) = v;
    }
  }
  __syncthreads();
  float acc[2][4] = {};                                      // pairs 8 j + 2 t, + 1 of rows 2 g | 2 g + 1
  const uint8_t* x0 = staged + g * pitch + 16 * t;
  const bool second = rows > 8;
  for (int u = u0; u < u1; u += kStUnroll) {
    uint4 ca[kStUnroll][2], cb[kStUnroll][2];
#pragma unroll
    for (int i = 0; i < kStUnroll; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) ca[i][h] = ra[i][h], cb[i][h] = rb[i][h];
    load(u + kStUnroll);
#pragma unroll
    for (int i = 0; i < kStUnroll; ++i) {
      if (u + i >= u1) break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint8_t* x = x0 + (size_t)(u + i) * 128 + h * 64;
        const uint32_t lo[4] = {ca[i][h].x, cb[i][h].x, ca[i][h].y, cb[i][h].y};
        const uint32_t hi[4] = {ca[i][h].z, cb[i][h].z, ca[i][h].w, cb[i][h].w};
        const uint4 v = *reinterpret_cast<const uint4*>(x);
        const uint32_t b0[2] = {v.x, v.y}, b1[2] = {v.z, v.w};
        mma_bf16(acc[0], lo, b0);
        mma_bf16(acc[0], hi, b1);
        if (second) {
          const uint4 y = *reinterpret_cast<const uint4*>(x + 8 * pitch);
          const uint32_t d0[2] = {y.x, y.y}, d1[2] = {y.z, y.w};
          mma_bf16(acc[1], lo, d0);
          mma_bf16(acc[1], hi, d1);
        }
      }
    }
  }
  if (parts > 1) {                                           // the first of a group's warps adds up
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) sums[warp][lane][j * 4 + i] = acc[j][i];
    __syncthreads();
    if (part) return;
    for (int p = 1; p < parts; ++p)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] += sums[warp + p][lane][j * 4 + i];
  }
  if (n >= N) return;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 8 * j + 2 * t + i;
      if (r >= rows) continue;
      const size_t s = (size_t)(row0 + r);
      const float c0 = acc[j][i], c1 = acc[j][2 + i];        // weight rows n, n + 1
      if (MODE == 2) {
        const float rw = row_w ? fresh(row_w + fresh_index(pair_of_pos + s)) : 1.f;
        const float v0 = fmaxf(to_f32(from_f32<__nv_bfloat16>(c0 * rw)), 0.f);
        const float v1 = fmaxf(to_f32(from_f32<__nv_bfloat16>(c1 * rw)), 0.f);
        *reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)out_ + s * N + n) =
            __floats2bfloat162_rn(v0 * v0, v1 * v1);
      } else if (MODE == 1) {
        const float gt = to_f32(from_f32<__nv_bfloat16>(c0)), up = to_f32(from_f32<__nv_bfloat16>(c1));
        ((__nv_bfloat16*)out_)[s * (N / 2) + n / 2] =
            from_f32<__nv_bfloat16>(clamped_glu(gt, up, limit, alpha, up_shift));
      } else {
        *reinterpret_cast<float2*>((float*)out_ + s * N + n) = make_float2(c0, c1);
      }
    }
}

// ---- the same for more pairs of large experts ------------------------------------------------------
// The grid above is (tile, weight rows) blocks, about one and a half rounds of them: while the last round runs
// half of the places are empty.  Here one block an SM takes an equal run of the step's (tile of pairs, 16 weight
// rows) items, one list.  Its sixteen warps share an item's reduction: step f of a matrix (16-row groups in
// order, steps of 64 k inside) belongs to warp f mod 16, whatever block has it, so that a pair's sums follow from
// the matrix alone.  A warp's steps come through a ring of its own in shared memory, each lane with its own
// 16-byte copies (nobody else reads them: no barrier), which runs on across items and tiles; after every two
// items the warps' sums meet, two warps add them up in order and store.
// Whole batches on a B200 (ms, the grid above / here), 32 experts of 2048 x 2112, 4 choices: 9 requests 35.7 / 30.8,
// 16 requests 42.5 / 34.2, 32 requests 29.18 / 29.16, 64 requests 24.4 / 24.9; 29 of 2048 x 1408, 5 choices: 8
// requests 28.5 / 27.9, 30 requests 26.5 / 27.3.  See ring_serves() for the line.
constexpr int kRgWarps = 16, kRgRing = 3, kRgItems = 2;
constexpr int kRgSlot = 2048;                                // a step: 16 rows x 64 k
constexpr int kRgHead = 128;                                 // the rows' weights
constexpr int kRgSums = kRgItems * kRgWarps * 2 * 32 * 16;
constexpr int kRgMaxShared = 227 * 1024;
constexpr int kRgMinExperts = 16, kRgMinK = 1280;
constexpr size_t kRgMinBytes = 4 << 20;
__host__ __device__ inline size_t ring_shared(int K) {
  return kRgHead + (size_t)kRgWarps * kRgRing * kRgSlot + kRgSums + kStRows * stream_pitch(K);
}
// Steps of one to two and a half pairs an expert, where the grid above would come to more than one round of blocks:
// a grid that fits at once has nothing to gain, and the second round costs what a full one does.  The
// grid's blocks follow from the experts that P pairs reach of E, about E (1 - (1 - 1 / E)^P); at 0.95 rounds nearly as
// many steps have an expert more as have one less, and the second round costs more than the ring.  In us a product on a
// B200, weights from HBM, grid / ring, by rounds: 2112 x 2048, 24 experts, 24 pairs (0.88) 27.8 / 29.9, 28 pairs (0.96,
// one expert more than that reached) 41.6 / 34.4, 36 pairs (1.08) 41.8 / 34.0, 32 experts, 64 pairs (1.60) 48.1 / 45.9, 80 (1.70)
// 50.2 / 49.2; 64 experts, 96 pairs (2.9) 76.7 / 72.6; 2816 x 2048, 32 experts, 48 pairs (1.86) 50.4 / 51.6; 1280 x 2048, 32
// experts, 40 pairs (0.78) 25.7 / 29.0, 80 pairs (1.00) 43.1 / 35.5; 1536 x 2048 28.3 / 30.3 (0.93), 44.9 / 38.2 (1.2); 2048 x
// 1408, 32 experts, 32 pairs (1.1) 29.6 / 25.6, 80 (1.6) 34.4 / 35.4; 2048 x 3072 (a block an SM), 24 experts, 28 pairs 89 /
// 45.  A shorter reduction leaves warps without a step in an item: 4096 x 512, 24 experts, 28 pairs (1.8) 15.3 / 18.7, 3072 x 1024
// (1.4) 25.7 / 28.3.  From 1,280 to 1,536 columns the second round has to be at least half empty, and an expert less costs
// more than one more gains.  Ring over grid, sums over 16 to 64 experts: 4096 x 1280 0.99 at 1 to 1.5 rounds, 1.05 from there
// to 1.9, 0.97 behind; 2048 x 1408 0.96, 1.02, 0.96 and 1.09 at 0.95 to 1; 3072 x 1408 0.94, 1.03, 0.96; 2048 x 1536 0.94, 1.01,
// 0.95 and 1.06; 2048 x 2112 0.90, 0.96, 0.91 and 1.01; 2816 x 2048 0.90, 0.99, 0.94 and 0.82.  Fewer experts: 16 of 2816 x 2048, 24 pairs 41.9 / 34.7; 8, 16 pairs (1.05) 18.9 / 20.9, 20 pairs 26.2 /
// 23.5.  Small matrices: 1536 x 1024, 24 experts, 60 pairs 18.6 / 22.7.
inline bool ring_serves(int pairs, int experts, int N, int K, int span, size_t grid_shared, int sms) {
  if (experts < kRgMinExperts || pairs <= kStHandful || pairs < experts || 2 * pairs > 5 * experts || K < kRgMinK ||
      (size_t)N * K * sizeof(__nv_bfloat16) < kRgMinBytes || ring_shared(K) > kRgMaxShared)
    return false;
  const double reached = experts * (1.0 - pow(1.0 - 1.0 / experts, pairs));
  const int places = sms * (2 * (grid_shared + 9 * 1024) < 204 * 1024 ? 2 : 1);   // (2,816 columns are the last with two)
  const double rounds = reached * ((N + span - 1) / span) / places;
  return K < 2048 ? rounds >= 1.0 && (rounds < 1.5 || rounds >= 1.9) : rounds >= 0.95;
}
__device__ __forceinline__ void ring_copy(uint32_t dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(kRgWarps * 32, 1)
moe_ring_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w,
                int N, int K, const int* __restrict__ offsets, const int* __restrict__ pair_of_pos,
                int top, const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                const int* __restrict__ num_tiles, void* __restrict__ out_, float limit,
                float alpha, float up_shift, const float* __restrict__ row_w) {
  extern __shared__ __align__(128) uint8_t shared[];         // head | rings | sums | [kStRows] rows of stream_pitch(K)
  float* weight_of = reinterpret_cast<float*>(shared);       // [kStRows]
  float4* sums = reinterpret_cast<float4*>(shared + kRgHead + kRgWarps * kRgRing * kRgSlot);
  uint8_t* staged = shared + kRgHead + kRgWarps * kRgRing * kRgSlot + kRgSums;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int units = (K + 63) / 64, groups = (N + 15) / 16;
  pdl_wait();
  pdl_trigger();
  const long long items = (long long)fresh_index(num_tiles) * groups;
  const long long i0 = items * blockIdx.x / gridDim.x, i1 = items * (blockIdx.x + 1) / gridDim.x;
  if (i0 >= i1) return;
  const int first_tile = (int)(i0 / groups), first_group = (int)(i0 % groups);
  const int last_tile = (int)((i1 - 1) / groups), last_group = (int)((i1 - 1) % groups);

  // the warp's next step to ask for: step pu of group pg of tile pt; from group `pend` on the block has no more
  // of this tile
  int pt = first_tile, pg, pu, pend;
  const __nv_bfloat16* pw;
  auto enter = [&](int tile, int group) {                    // the warp's first step at or behind `group`
    const int ahead = (warp - group * units) & (kRgWarps - 1);
    pg = group + ahead / units, pu = ahead % units;
    pend = tile == last_tile ? last_group + 1 : groups;
    pw = w + (size_t)fresh_index(tile_expert + tile) * N * K + 8 * t;
  };
  enter(pt, first_group);
  const uint32_t ring = smem_u32(shared) + kRgHead + warp * kRgRing * kRgSlot + lane * 16;
  auto ask = [&](int slot) {
    while (pg >= pend && pt < last_tile) {
      ++pt;
      enter(pt, 0);
    }
    if (pg < pend) {
      const int n = pg * 16 + 2 * g;                         // N is even: both rows are there, or none
      const __nv_bfloat16* src = pw + (size_t)n * K + pu * 64;
      const uint32_t dst = ring + slot * kRgSlot;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool there = n < N && pu * 64 + h * 32 + 8 * t < K;
        ring_copy(dst + h * 1024, there ? src + h * 32 : w, there);
        ring_copy(dst + h * 1024 + 512, there ? src + h * 32 + K : w, there);
      }
      pu += kRgWarps;
      while (pu >= units) pu -= units, ++pg;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kRgRing; ++i) ask(i);

  int slot = 0;
  const size_t pitch = stream_pitch(K);
  const uint8_t* x0 = staged + g * pitch + 16 * t;
  const uint8_t* mine = shared + kRgHead + warp * kRgRing * kRgSlot + lane * 16;
  for (int tile = first_tile; tile <= last_tile; ++tile) {
    const int e = fresh_index(tile_expert + tile), row0 = fresh_index(tile_row0 + tile);
    const int rows = min(kStRows, fresh_index(offsets + e + 1) - row0);
    const bool second = rows > 8;
    if (MODE == 2 && (int)threadIdx.x < rows)
      weight_of[threadIdx.x] = row_w ? fresh(row_w + fresh_index(pair_of_pos + row0 + threadIdx.x)) : 1.f;
    {                                                        // the rows, zeros up to whole steps
      const int k8 = units * 8, staged_rows = second ? 16 : 8;
      for (int i = threadIdx.x; i < staged_rows * k8; i += kRgWarps * 32) {
        const int r = i / k8, c = (i - r * k8) * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows && c < K) {
          const int src = MODE != 0 ? fresh_index(pair_of_pos + row0 + r) / top : row0 + r;
          v = __ldcg(reinterpret_cast<const uint4*>(a + (size_t)src * lda + c));
        }
        *reinterpret_cast<uint4*>(staged + r * pitch + (size_t)c * 2) = v;
      }
    }
    __syncthreads();
    const int g0 = tile == first_tile ? first_group : 0, g1 = tile == last_tile ? last_group + 1 : groups;
    for (int from = g0; from < g1; from += kRgItems) {
      const int many = min(kRgItems, g1 - from);
      for (int b = 0; b < many; ++b) {
        float acc[2][2][4] = {};                             // [run][8 j ..]: pairs 8 j + 2 t, + 1 of rows 2 g | 2 g + 1
        for (int u = (warp - (from + b) * units) & (kRgWarps - 1); u < units; u += kRgWarps) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kRgRing - 1) : "memory");
          const uint8_t *x = x0 + (size_t)u * 128, *at = mine + slot * kRgSlot;
          uint4 wa[2], wb[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            wa[h] = *reinterpret_cast<const uint4*>(at + h * 1024);
            wb[h] = *reinterpret_cast<const uint4*>(at + h * 1024 + 512);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t lo[4] = {wa[h].x, wb[h].x, wa[h].y, wb[h].y};
            const uint32_t hi[4] = {wa[h].z, wb[h].z, wa[h].w, wb[h].w};
            const uint4 v = *reinterpret_cast<const uint4*>(x + h * 64);
            const uint32_t b0[2] = {v.x, v.y}, b1[2] = {v.z, v.w};
            mma_bf16(acc[h][0], lo, b0);
            mma_bf16(acc[h][0], hi, b1);
            if (second) {
              const uint4 y = *reinterpret_cast<const uint4*>(x + 8 * pitch + h * 64);
              const uint32_t d0[2] = {y.x, y.y}, d1[2] = {y.z, y.w};
              mma_bf16(acc[h][1], lo, d0);
              mma_bf16(acc[h][1], hi, d1);
            }
          }
          ask(slot);                                         // its old contents are in registers
          slot = slot + 1 == kRgRing ? 0 : slot + 1;
        }
        float4* to = sums + (b * kRgWarps + warp) * 64 + lane;
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (j == 0 || second)
            to[j * 32] = make_float4(acc[0][j][0] + acc[1][j][0], acc[0][j][1] + acc[1][j][1],
                                     acc[0][j][2] + acc[1][j][2], acc[0][j][3] + acc[1][j][3]);
      }
      __syncthreads();
      const int n = (from + warp) * 16 + 2 * g;
      if (warp < many && n < N) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (j == 1 && !second) break;
          const float4* of = sums + warp * kRgWarps * 64 + j * 32 + lane;
          float4 s = of[0];
#pragma unroll
          for (int p = 1; p < kRgWarps; ++p) {
            const float4 v = of[p * 64];
            s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = 8 * j + 2 * t + i;
            if (r >= rows) continue;
            const size_t at = (size_t)(row0 + r);
            const float c0 = i ? s.y : s.x, c1 = i ? s.w : s.z;    // weight rows n, n + 1
            if (MODE == 2) {
              const float rw = weight_of[r];
              const float v0 = fmaxf(to_f32(from_f32<__nv_bfloat16>(c0 * rw)), 0.f);
              const float v1 = fmaxf(to_f32(from_f32<__nv_bfloat16>(c1 * rw)), 0.f);
              *reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)out_ + at * N + n) =
                  __floats2bfloat162_rn(v0 * v0, v1 * v1);
            } else if (MODE == 1) {
              const float gt = to_f32(from_f32<__nv_bfloat16>(c0)), up = to_f32(from_f32<__nv_bfloat16>(c1));
              ((__nv_bfloat16*)out_)[at * (N / 2) + n / 2] =
                  from_f32<__nv_bfloat16>(clamped_glu(gt, up, limit, alpha, up_shift));
            } else {
              *reinterpret_cast<float2*>((float*)out_ + at * N + n) = make_float2(c0, c1);
            }
          }
        }
      }
      __syncthreads();                                       // the sums (and the rows) may be written again
    }
  }
}

// ---- the same for a handful of pairs on the FMA pipes ----------------------------------------------
// For layers that stay off moe_stream_kernel (their routers' close calls ask for sums in one order).  The
// work is the experts' weight bytes.  A tile is up to 8 rows of one expert, kept in shared memory; the (tile,
// two neighbouring weight rows) items of the step, one list, are cut into one equal run a block, two blocks
// an SM, and of a block's run every warp takes every eighth item (a gate and its up value in the gated form).
// A warp reads its items' weights once, with 16-byte loads, in batches of 1,024 k of both rows, each lane a
// strided share of the reduction; while one batch is multiplied the next one, of the same item or of the next,
// is under way, so that the stream does not stop at an item's end.  A warp sum ends an item.  The order of the
// sums depends on K alone, so a pair's result does not depend on the batch.
// The loops over a tile's rows are most of the instructions, so their number is the compiler's; tiles of
// three rows and more hold each batch's code once (kernels alternate, and code that is not there is waited for).
// On a B200, weights from HBM, both products, us (floor in brackets), against a grid of (tile, 16 to 64 weight
// rows) blocks whose warps waited for each batch and branched for each row: 32 experts of 2048 x 1408, 4 choices, 1
// token 21.6 / 31.8 (10.7), 2 tokens 33.6 / 50.2 (18.8), 4 tokens 60 / 75 (34.9), 5 tokens 66 / 94 (40.2); 16 of 1024 x 704,
// 2 choices, 4 tokens 16.2 / 19.0, 8 tokens 27.3 / 26.7, 10 tokens 33.6 / 31.1.
constexpr int kFewRows = 8, kFewWarps = 8, kFewBlocks = 2, kFewSteps = 4;
constexpr int kFewMaxShared = 64 * 1024;                     // K up to 4,096

__device__ __forceinline__ void bf16x8_to_f32(const uint4& raw, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x, v[2 * i + 1] = f.y;
  }
}

// Weights are read once: past L1, and without a claim on it.
__device__ __forceinline__ uint4 load_once(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

template <int MODE>
__global__ void __launch_bounds__(kFewWarps * 32, kFewBlocks)
moe_gemv_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w,
                int N, int K, const int* __restrict__ offsets, const int* __restrict__ pair_of_pos,
                int top, const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                const int* __restrict__ num_tiles, void* __restrict__ out_, float limit,
                float alpha, float up_shift) {
  extern __shared__ __align__(16) __nv_bfloat16 xrows[];           // [kFewRows][K]
  pdl_wait();
  pdl_trigger();
  const int items = N >> 1;                                        // of a tile; N is even
  const long long all = (long long)fresh_index(num_tiles) * items;
  const int i0 = (int)(all * blockIdx.x / gridDim.x), i1 = (int)(all * (blockIdx.x + 1) / gridDim.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k8 = K >> 3;
  for (int at = i0; at < i1;) {
    const int tile = at / items, p0 = at - tile * items, p1 = min(items, p0 + (i1 - at));
    const int e = fresh_index(tile_expert + tile), row0 = fresh_index(tile_row0 + tile);
    const int rows = min(kFewRows, fresh_index(offsets + e + 1) - row0);
    const __nv_bfloat16* we = w + (size_t)e * N * K + lane * 8;
    int ask_item = p0 + warp, ask_k = 0;
    auto load = [&](uint4 (&wa)[kFewSteps], uint4 (&wb)[kFewSteps]) {
      if (ask_item >= p1) return;
      const __nv_bfloat16* src = we + (size_t)(2 * ask_item) * K + ask_k;
#pragma unroll
      for (int u = 0; u < kFewSteps; ++u)
        if (ask_k + lane * 8 + u * 256 < K) wa[u] = load_once(src + u * 256), wb[u] = load_once(src + u * 256 + K);
      ask_k += kFewSteps * 256;
      if (ask_k >= K) ask_k = 0, ask_item += kFewWarps;
    };
    uint4 wa[kFewSteps], wb[kFewSteps], va[kFewSteps], vb[kFewSteps];
    load(wa, wb);
    load(va, vb);
    for (int i = threadIdx.x; i < rows * k8; i += kFewWarps * 32) {
      const int r = i / k8, c = (i - r * k8) * 8;
      const int src = MODE != 0 ? fresh_index(pair_of_pos + row0 + r) / top : row0 + r;
      *reinterpret_cast<uint4*>(xrows + (size_t)r * K + c) =
          __ldcg(reinterpret_cast<const uint4*>(a + (size_t)src * lda + c));
    }
    __syncthreads();
    // ROWS: of the tile, known to the compiler (its loops over them are most of the instructions)
    auto run = [&](auto rows_of) {
      constexpr int ROWS = decltype(rows_of)::value;
      int item = p0 + warp, k = 0;
      float acc0[ROWS], acc1[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc0[r] = acc1[r] = 0.f;
      auto multiply = [&](const uint4 (&pa)[kFewSteps], const uint4 (&pb)[kFewSteps]) {
#pragma unroll
        for (int u = 0; u < kFewSteps; ++u) {
          const int c = k + lane * 8 + u * 256;
          if (c >= K) break;
          float f0[8], f1[8];
          bf16x8_to_f32(pa[u], f0);
          bf16x8_to_f32(pb[u], f1);
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            if (ROWS > 4 && r >= rows) break;
            float x[8];
            bf16x8_to_f32(*reinterpret_cast<const uint4*>(xrows + (size_t)r * K + c), x);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              acc0[r] = fmaf(f0[j], x[j], acc0[r]);
              acc1[r] = fmaf(f1[j], x[j], acc1[r]);
            }
          }
        }
      };
      auto finish = [&]() {                                        // behind a batch: the item's end, if it is
        k += kFewSteps * 256;
        if (k < K) return;
        const int n = 2 * item;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)                           // (warp_sum, all rows side by side)
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            acc0[r] += __shfl_xor_sync(0xffffffffu, acc0[r], o);
            acc1[r] += __shfl_xor_sync(0xffffffffu, acc1[r], o);
          }
        if (lane == 0) {
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            if (r >= rows) break;
            const size_t s = (size_t)(row0 + r);
            if (MODE == 1) {
              const float gt = to_f32(from_f32<__nv_bfloat16>(acc0[r])), up = to_f32(from_f32<__nv_bfloat16>(acc1[r]));
              ((__nv_bfloat16*)out_)[s * (N / 2) + n / 2] =
                  from_f32<__nv_bfloat16>(clamped_glu(gt, up, limit, alpha, up_shift));
            } else {
              float* to = (float*)out_ + s * N + n;                // (aligned to four bytes is enough)
              to[0] = acc0[r];
              to[1] = acc1[r];
            }
          }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc0[r] = acc1[r] = 0.f;
        k = 0, item += kFewWarps;
      };
      while (item < p1) {
        multiply(wa, wb);
        if (ROWS > 2) {                                            // (once in the code: there is much of it)
#pragma unroll
          for (int u = 0; u < kFewSteps; ++u) wa[u] = va[u], wb[u] = vb[u];
          load(va, vb);
          finish();
          continue;
        }
        load(wa, wb);
        finish();
        if (item >= p1) break;
        multiply(va, vb);
        load(va, vb);
        finish();
      }
    };
    if (rows == 1) run(std::integral_constant<int, 1>{});
    else if (rows == 2) run(std::integral_constant<int, 2>{});
    else if (rows == 3) run(std::integral_constant<int, 3>{});
    else if (rows == 4) run(std::integral_constant<int, 4>{});
    else run(std::integral_constant<int, 8>{});
    at += p1 - p0;
    if (at < i1) __syncthreads();                                  // the rows are free for the next tile's
  }
}

// xs[s, :] = x[pair_of_pos[s] / top, :]: the tokens' rows in sorted order, 16 bytes an access, for
// the grouped product that reads its rows by TMA (K % 8 == 0, 16-byte aligned rows).
__global__ void moe_gather_rows_kernel(const __nv_bfloat16* __restrict__ x, int ldx,
                                       const int* __restrict__ pair_of_pos,
                                       const int* __restrict__ placed, int top, int P, int K,
                                       __nv_bfloat16* __restrict__ xs) {
  pdl_trigger();
  pdl_wait();
  const int k8 = K >> 3;
  P = min(P, fresh_index(placed));                  // pairs that have a place
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)P * k8;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t s = i / k8;
    const int c = (int)(i - s * k8) * 8;
    const size_t src = (size_t)(fresh_index(pair_of_pos + s) / top) * ldx + c;
    *reinterpret_cast<uint4*>(xs + s * K + c) = *reinterpret_cast<const uint4*>(x + src);
  }
}

// A thread has VEC channels (4, or 1 for widths that are no multiple of four) of a token; the places of four
// choices are asked for together, then their rows.  A decode step of 4 tokens with 4 choices (2,048
// channels, B200): 10.9 us with a block a token whose threads asked for every place again for each of their
// channels, below 3 now; 2,251 tokens 39 us and 18.
constexpr int kCombineThreads = 128;
template <typename T, int VEC>
__global__ void __launch_bounds__(kCombineThreads)
moe_combine_kernel(const float* __restrict__ y, const int* __restrict__ pos_of_pair,
                   const float* __restrict__ wgt, int top, int N, T* __restrict__ out) {
  const size_t t = blockIdx.x;
  const int n = (blockIdx.y * kCombineThreads + threadIdx.x) * VEC;
  pdl_trigger();
  pdl_wait();
  if (n >= N) return;
  float acc[VEC] = {};
  for (int k0 = 0; k0 < top; k0 += 4) {
    int p[4];
    float w[4], v[4][VEC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[i] = k0 + i < top ? fresh_index(pos_of_pair + t * top + k0 + i) : -1;
      w[i] = wgt && k0 + i < top ? fresh(wgt + t * top + k0 + i) : 1.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (p[i] >= 0) {
        if constexpr (VEC == 4) Quad<float>::fresh(y + (size_t)p[i] * N + n, v[i]);
        else v[i][0] = fresh(y + (size_t)p[i] * N + n);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)                      // in the order chosen
      if (p[i] >= 0)
#pragma unroll
        for (int x = 0; x < VEC; ++x) acc[x] = fmaf(w[i], v[i][x], acc[x]);
  }
  if constexpr (VEC == 4) Quad<T>::store(out + t * N + n, acc);
  else out[t * N + n] = from_f32<T>(acc[0]);
}

}  // namespace gf

using namespace gf;
using bf = __nv_bfloat16;

GF_DEFINE_PDL_SWITCH

// Streaming multiprocessors of the current device, asked of it once.
static int sm_count(int* sms) {
  static OncePerDevice once;
  static int count[OncePerDevice::kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= OncePerDevice::kMaxDevices) return -9;
  const int rc = once.run([&] { return cudaDeviceGetAttribute(&count[dev], cudaDevAttrMultiProcessorCount, dev); });
  *sms = count[dev];
  return rc;
}

// Rows of a tile: of the plain kernel (tensor_cores == 0), of the tensor-core kernel (1), of the
// weight-streaming kernel (2) or of the one with FMAs for a handful of pairs (3).
GF_EXPORT int gf_moe_tile_rows(int tensor_cores) {
  return tensor_cores == 3 ? kFewRows : tensor_cores == 2 ? kStRows : tensor_cores ? kTM : kBM;
}

// sigmoid != 0: a score is the sigmoid of its logit instead of the softmax over all experts.
GF_EXPORT int gf_moe_route(const float* logits, int T, int E, int top, int renorm, int sigmoid,
                           int* idx, float* wgt, void* stream) {
  if (T <= 0) return 0;
  if (E > kMaxExperts || top > E || top > 32) return -3;
  return launch_kernel(moe_route_kernel, dim3((T + 3) / 4), dim3(128), 0, (cudaStream_t)stream,
                       logits, T, E, top, renorm, sigmoid, idx, wgt);
}

// See moe_route_grouped_kernel.
GF_EXPORT int gf_moe_route_grouped(const float* logits, int ld, int T, int E, int identity, int top,
                                   int groups, int keep, const float* correction, int gate_col,
                                   int always, int* idx, float* wgt, float* identity_w, float* gate,
                                   void* stream) {
  if (T <= 0) return 0;
  if (E <= 0 || E > kMaxExperts || identity < 0 || identity > E || top < 1 || groups < 1 ||
      E % groups || keep < 1 || keep > groups || top > E / groups * keep || ld < E ||
      gate_col >= ld || ((gate || always) && gate_col < 0) || always < 0 || always > 32)
    return -3;
#define GF_GO(SLOTS)                                                                              \
  return launch_kernel(moe_route_grouped_kernel<SLOTS>, dim3((T + 3) / 4), dim3(128), 0,          \
                       (cudaStream_t)stream, logits, ld, T, E, identity, top, groups, keep,       \
                       correction, gate_col, always, idx, wgt, identity_w, gate)
  if (E <= 32) GF_GO(1);
  if (E <= 64) GF_GO(2);
  GF_GO(kRouteSlots);
#undef GF_GO
}

GF_EXPORT int gf_moe_plan(const int* idx, int P, int E, int tile_rows, int* offsets,
                          int* pos_of_pair, int* pair_of_pos, int* tile_expert, int* tile_row0,
                          int* num_tiles, void* stream) {
  if (P <= 0) return 0;
  if (E > kMaxExperts || tile_rows <= 0) return -3;
  const size_t held = (size_t)P * sizeof(int);     // staged where it fits without asking for more
  const int stage = held <= 40 * 1024;
  return launch_kernel(moe_plan_kernel, dim3(E), dim3(kPlanThreads), stage ? held : 0,
                       (cudaStream_t)stream, idx, P, E, tile_rows, stage, offsets, pos_of_pair, pair_of_pos, tile_expert, tile_row0,
                       num_tiles);
}

// first 1: gate/up product with the clamped GLU; out [P, N / 2] (dtype).  first 2: up product with
// relu(row_w * .)^2; out [P, N] (dtype); row_w [P] by pair, or null.  first 0: down; out fp32.
GF_EXPORT int gf_moe_gemm(const void* a, int lda, const void* w, int N, int K, const int* offsets,
                          const int* pair_of_pos, int top, const int* tile_expert,
                          const int* tile_row0, const int* num_tiles, int max_tiles, void* out,
                          int first, float limit, float alpha, float up_shift,
                          const float* row_w, int dtype, int tensor_cores, void* stream,
                          int pairs, int experts) {
  if (max_tiles <= 0) return 0;
  auto st = (cudaStream_t)stream;
  if (tensor_cores == 2) {                     // the weight-streaming kernel
    const size_t smem = kStRows * stream_pitch(K);
    if (dtype != GF_BF16 || K % 8 || lda % 8 || N % 2 || (uintptr_t)a % 16 || (uintptr_t)w % 16 ||
        (uintptr_t)out % 8 || smem > kStMaxShared)
      return -3;
    // about 16 warps an SM should be busy
    const int each = pairs <= kStRows * experts ? 2 : 4;       // tiles an expert
    const int most = pairs <= kStHandful ? kStHandfulTiles : kStTiles;
    const int busy = most < each * experts ? most : each * experts;
    int parts = 1;
    while (parts < kStWarps && (long long)busy * (N / 16 + 1) * parts < 16 * 148 && K >= parts * 256) parts *= 2;
    const int span = 16 * (kStWarps / parts);
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    if (ring_serves(pairs, experts, N, K, span, smem, sms)) {
#define GF_RING(MODE)                                                                             \
  {                                                                                               \
    static OncePerDevice attrs;                                                                   \
    if (int rc = attrs.run([&] {                                                                  \
          return cudaFuncSetAttribute(moe_ring_kernel<MODE>,                                      \
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, kRgMaxShared); \
        }))                                                                                       \
      return rc;                                                                                  \
    return launch_kernel(moe_ring_kernel<MODE>, dim3(sms), dim3(kRgWarps * 32), ring_shared(K), st, \
                         (const bf*)a, lda, (const bf*)w, N, K, offsets, pair_of_pos, top,        \
                         tile_expert, tile_row0, num_tiles, out, limit, alpha, up_shift, row_w);  \
  }
      if (first == 2) GF_RING(2)
      if (first) GF_RING(1)
      GF_RING(0)
#undef GF_RING
    }
    const dim3 sgrid(max_tiles, (N + span - 1) / span), sblock(kStWarps * 32);
#define GF_ST(MODE)                                                                               \
  {                                                                                               \
    static OncePerDevice attrs;                                                                   \
    if (int rc = attrs.run([&] {                                                                  \
          return cudaFuncSetAttribute(moe_stream_kernel<MODE>,                                    \
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, kStMaxShared); \
        }))                                                                                       \
      return rc;                                                                                  \
    return launch_kernel(moe_stream_kernel<MODE>, sgrid, sblock, smem, st, (const bf*)a, lda,     \
                         (const bf*)w, N, K, offsets, pair_of_pos, top, tile_expert, tile_row0,   \
                         num_tiles, out, limit, alpha, up_shift, row_w, parts);                   \
  }
    if (first == 2) GF_ST(2)
    if (first) GF_ST(1)
    GF_ST(0)
#undef GF_ST
  }
  if (tensor_cores == 3) {                     // a handful of pairs with plain multiply-adds
    const size_t smem = (size_t)kFewRows * K * sizeof(bf);
    if (dtype != GF_BF16 || K % 8 || lda % 8 || N % 2 || (uintptr_t)a % 16 || (uintptr_t)w % 16 ||
        smem > kFewMaxShared || first == 2)
      return -3;
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    const dim3 fgrid(sms * kFewBlocks), fblock(kFewWarps * 32);
#define GF_FEW(MODE)                                                                              \
  {                                                                                               \
    static OncePerDevice attrs;                                                                   \
    if (int rc = attrs.run([&] {                                                                  \
          return cudaFuncSetAttribute(moe_gemv_kernel<MODE>,                                      \
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, kFewMaxShared);\
        }))                                                                                       \
      return rc;                                                                                  \
    return launch_kernel(moe_gemv_kernel<MODE>, fgrid, fblock, smem, st, (const bf*)a, lda,       \
                         (const bf*)w, N, K, offsets, pair_of_pos, top, tile_expert, tile_row0,   \
                         num_tiles, out, limit, alpha, up_shift);                                 \
  }
    if (first) GF_FEW(1)
    GF_FEW(0)
#undef GF_FEW
  }
  if (tensor_cores) {
    if (dtype != GF_BF16 || K % 8 || lda % 8 || (uintptr_t)a % 16 || (uintptr_t)w % 16) return -3;
    const dim3 tgrid(max_tiles, (N + kTN - 1) / kTN), tblock(256);
#define GF_TC(MODE)                                                                               \
  return launch_kernel(moe_gemm_mma_kernel<MODE>, tgrid, tblock, 0, st, (const bf*)a, lda,          \
                       (const bf*)w, N, K, offsets, pair_of_pos, top, tile_expert, tile_row0,       \
                       num_tiles, out, limit, alpha, up_shift, row_w)
    if (first == 2) GF_TC(2);
    if (first) GF_TC(1);
    GF_TC(0);
#undef GF_TC
  }
  const dim3 grid(max_tiles, (N + kBN - 1) / kBN), block(256);
#define GF_GO(T, MODE)                                                                           \
  return launch_kernel(moe_gemm_kernel<T, MODE>, grid, block, 0, st, (const T*)a, lda,           \
                       (const T*)w, N, K, offsets, pair_of_pos, top, tile_expert, tile_row0,      \
                       num_tiles, out, limit, alpha, up_shift, row_w)
  if (dtype == GF_F32) {
    if (first == 2) GF_GO(float, 2);
    if (first) GF_GO(float, 1);
    GF_GO(float, 0);
  }
  if (first == 2) GF_GO(bf, 2);
  if (first) GF_GO(bf, 1);
  GF_GO(bf, 0);
#undef GF_GO
}

// placed: how many pairs have a place in the sorted order (offsets + E of the plan).
GF_EXPORT int gf_moe_gather_rows(const void* x, int ldx, const int* pair_of_pos, const int* placed,
                                 int top, int P, int K, void* xs, void* stream) {
  if (P <= 0) return 0;
  if (K % 8 || ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)xs & 15)) return -3;
  const size_t want = ((size_t)P * (K / 8) + 255) / 256;
  const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
  return launch_kernel(moe_gather_rows_kernel, dim3(blocks), dim3(256), 0, (cudaStream_t)stream,
                       (const bf*)x, ldx, pair_of_pos, placed, top, P, K, (bf*)xs);
}

GF_EXPORT int gf_moe_combine(const float* y, const int* pos_of_pair, const float* wgt, int T,
                             int top, int N, void* out, int dtype, void* stream) {
  if (T <= 0) return 0;
  auto st = (cudaStream_t)stream;
  const bool quads = N % 4 == 0 && ((uintptr_t)y | (uintptr_t)out) % 16 == 0;
  const int per = kCombineThreads * (quads ? 4 : 1);
  const dim3 grid(T, (N + per - 1) / per), block(kCombineThreads);
#define GF_GO(E)                                                                                       \
  return quads ? launch_kernel(moe_combine_kernel<E, 4>, grid, block, 0, st, y, pos_of_pair, wgt, top, N, \
                               (E*)out)                                                                \
               : launch_kernel(moe_combine_kernel<E, 1>, grid, block, 0, st, y, pos_of_pair, wgt, top, N, \
                               (E*)out)
  if (dtype == GF_F32) GF_GO(float);
  GF_GO(bf);
#undef GF_GO
}
