// Gated delta rule with one decay per head and key channel, or one per head, over packed tokens of
// several requests.
// A request's state lives in a slot: S [heads, D, Vd] in fp32 and the last (taps - 1) inputs of the
// short convolutions, fp32 as well.
//
//   delta_prepare_kernel     a warp a (token, head): causal convolution over time (taps from the rows of
//                            this step, or from the slot where the step's portion starts later than
//                            the tap reaches) + SiLU on the q | k | v channels; q and k made unit
//                            vectors per head (q also times D^-1/2); decay g = exp(-exp(A_log_h) *
//                            softplus(a + dt_bias)); beta = sigmoid(b).  Everything leaves in fp32.
//   delta_prepare_heads_kernel  the same with one decay a head, four channels a lane, a warp walking
//                            over a run of tokens with the convolution's inputs in registers.
//   delta_conv_state_kernel  a thread a (request, channel): the slot's last inputs after the step.
//   delta_recurrence_kernel  per (request, head): S <- g * S (rows); u = beta (v - S^T k);
//                            S <- S + k u^T; o = S^T q, token after token.  The columns of S are
//                            independent: four lanes or a warp share a column (a share of the rows
//                            each, in registers).  The tokens' operands come through two stages of
//                            shared memory, a chunk ahead (cp.async).
//   delta_tree_kernel        the same with eight or sixteen lanes for two columns (see there).
//   delta_chunk_coef_kernel, linear_chunk_coef_kernel, delta_chunk_recurrence_kernel   the recurrence of
//                            long portions, eight tokens at a time: the delta rule with one decay a head,
//                            plain linear attention with a decay a key channel (see there).
//   delta_output_kernel      a warp a (token, head): o / rms(o) * w * sigmoid(gate).
#include "common.cuh"

namespace gf {

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

struct DeltaDims {
  int H, G, D, Vd, taps;
  int channels;          // 2 G D + H Vd: the convolved columns q | k | v of a projection row
  int state_stride;      // floats a slot
  int conv_off;          // where the convolution inputs start in a slot
  int a_ld;              // one decay a head: floats between two tokens of its pre-activations
};

// ONE_DECAY: `a` holds a pre-activation a head (rows of a_ld floats), and one unit makes all heads'
// decays.  A warp a (token, unit): units 0 .. G-1 are q heads, G .. 2G-1 k heads, then H v heads, then H
// decay rows, then one unit for the betas.  No warp waits for another.
template <typename T>
__device__ __forceinline__ float conv_silu_at(const T* __restrict__ proj, int ld, int r, int i,
                                              const float* __restrict__ cs,
                                              const float* __restrict__ conv_w, int taps, int CH,
                                              int ch) {
  float acc = 0.f;
  for (int j = 0; j < taps; ++j) {
    const int off = i - (taps - 1 - j);           // place of the tap's input in the portion
    const float x = off >= 0 ? to_f32(proj[(size_t)(r - (taps - 1 - j)) * ld + ch])
                             : cs[(size_t)(taps - 1 + off) * CH + ch];
    acc = fmaf(conv_w[(size_t)ch * taps + j], x, acc);
  }
  return acc * sigmoid_f(acc);
}

constexpr int kPrepareWarps = 8;
constexpr int kPrepareMaxPerLane = 8;              // head sizes up to 256

template <typename T, bool ONE_DECAY>
__global__ void delta_prepare_kernel(const T* __restrict__ proj, int ld, int b_off,
                                     const float* __restrict__ a, const float* __restrict__ conv_w,
                                     const float* __restrict__ dt_bias,
                                     const float* __restrict__ A_log,
                                     const float* __restrict__ state,
                                     const int* __restrict__ seq_of_token,
                                     const int* __restrict__ cu_seqlens,
                                     const int* __restrict__ slot_ids, DeltaDims dm,
                                     float* __restrict__ qn, float* __restrict__ kn,
                                     float* __restrict__ v, float* __restrict__ g,
                                     float* __restrict__ beta) {
  const int r = blockIdx.x;
  const int unit = blockIdx.y * kPrepareWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  const int G = dm.G, H = dm.H, D = dm.D, Vd = dm.Vd;
  if (unit >= 2 * G + H + (ONE_DECAY ? 0 : H) + 1) return;
  const int b = seq_of_token[r];
  const int i = r - cu_seqlens[b];                // place in this step's portion
  const float* cs = state + (size_t)slot_ids[b] * dm.state_stride + dm.conv_off;
  const int taps = dm.taps, CH = dm.channels, GD = G * D;
  if (unit < 2 * G) {                             // a q or k head: convolve, activate, unit vector
    const int ch0 = unit * D;                     // q heads and k heads follow one another
    float y[kPrepareMaxPerLane];
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < kPrepareMaxPerLane; ++u) {
      const int d = lane + 32 * u;
      y[u] = d < D ? conv_silu_at(proj, ld, r, i, cs, conv_w, taps, CH, ch0 + d) : 0.f;
      ss += y[u] * y[u];
    }
    ss = warp_sum(ss);
    const bool is_q = unit < G;
    const float f = (is_q ? rsqrtf((float)D) : 1.f) / sqrtf(ss + 1e-6f);
    float* dst = (is_q ? qn : kn) + (size_t)r * GD + (size_t)(is_q ? unit : unit - G) * D;
#pragma unroll
    for (int u = 0; u < kPrepareMaxPerLane; ++u) {
      const int d = lane + 32 * u;
      if (d < D) dst[d] = y[u] * f;
    }
  } else if (unit < 2 * G + H) {                  // a v head
    const int h = unit - 2 * G;
    for (int j = lane; j < Vd; j += 32)
      v[((size_t)r * H + h) * Vd + j] =
          conv_silu_at(proj, ld, r, i, cs, conv_w, taps, CH, 2 * GD + h * Vd + j);
  } else if (!ONE_DECAY && unit < 2 * G + 2 * H) {              // a head's decays
    const int h = unit - 2 * G - H;
    const float rate = expf(A_log[h]);
    for (int d = lane; d < D; d += 32) {
      const size_t at = ((size_t)r * H + h) * D + d;
      g[at] = expf(-rate * softplus_f(a[at] + dt_bias[h * D + d]));
    }
  } else {
    for (int h = lane; h < H; h += 32)
      beta[(size_t)r * H + h] = sigmoid_f(to_f32(proj[(size_t)r * ld + b_off + h]));
    if (ONE_DECAY)
      for (int h = lane; h < H; h += 32)
        g[(size_t)r * H + h] =
            expf(-expf(A_log[h]) * softplus_f(a[(size_t)r * dm.a_ld + h] + dt_bias[h]));
  }
}

// One decay a head, the projection's row in fp32 (q | k | v first, decay and beta columns at a_off
// and b_off).  Units: G q heads, G k heads, H v heads, one for decays and betas.  A warp takes a unit
// and `run` consecutive tokens; lanes own four channels (NQ times); the last TAPS - 1 inputs stay in
// registers from token to token and come from the slot at a portion's start.  update_state (every
// portion of the step is one token): the same lanes bring the slot's inputs up to date.
// D, Vd, ld and the offsets are multiples of 4.
template <int TAPS, int NQ>
__global__ void __launch_bounds__(128)
delta_prepare_heads_kernel(const float* __restrict__ proj, int ld, int a_off, int b_off,
                           const float* __restrict__ conv_w, const float* __restrict__ dt_bias,
                           const float* __restrict__ A_log, float* __restrict__ state,
                           const int* __restrict__ seq_of_token,
                           const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids,
                           DeltaDims dm, int T, int run, int update_state, float* __restrict__ qn,
                           float* __restrict__ kn, float* __restrict__ v, float* __restrict__ g,
                           float* __restrict__ beta) {
  constexpr int KEEP = TAPS - 1;
  const int lane = threadIdx.x & 31;
  const int G = dm.G, H = dm.H, D = dm.D, Vd = dm.Vd, GD = G * D;
  const int unit = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int r0 = blockIdx.x * run, r1 = min(r0 + run, T);
  const bool convolves = unit < 2 * G + H;
  const int size = unit < 2 * G ? D : Vd;
  const int ch0 = unit < 2 * G ? unit * D : 2 * GD + (unit - 2 * G) * Vd;
  float w[NQ][4][TAPS];
  if (convolves) {                                  // weights: before the wait
#pragma unroll
    for (int u = 0; u < NQ; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = 4 * (lane + 32 * u) + i;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) w[u][i][j] = d < size ? conv_w[(size_t)(ch0 + d) * TAPS + j] : 0.f;
      }
  }
  // few tokens: the recurrence may start early.  In a prompt its long-lived blocks would land several
  // to an SM on the first SMs that drain.
  if (run == 1) pdl_trigger();
  pdl_wait();
  if (unit > 2 * G + H) return;
  if (!convolves) {
    for (int e = lane; e < (r1 - r0) * H; e += 32) {
      const int r = r0 + e / H, h = e % H;
      const float* row = proj + (size_t)r * ld;
      beta[(size_t)r * H + h] = sigmoid_f(row[b_off + h]);
      g[(size_t)r * H + h] = expf(-expf(A_log[h]) * softplus_f(row[a_off + h] + dt_bias[h]));
    }
    return;
  }
  float past[NQ][4][KEEP > 0 ? KEEP : 1];           // inputs of the tokens before, oldest first
  for (int r = r0; r < r1; ++r) {
    const int b = seq_of_token[r], start = cu_seqlens[b];
    float* cs = state + (size_t)slot_ids[b] * dm.state_stride + dm.conv_off;
    if (r == r0 || r == start) {
#pragma unroll
      for (int m = 0; m < KEEP; ++m) {
        const int at = r - KEEP + m;                // the row of this input, if the step has it
#pragma unroll
        for (int u = 0; u < NQ; ++u) {
          const int d = 4 * (lane + 32 * u);
          float x[4] = {0.f, 0.f, 0.f, 0.f};
          if (d < size)
            Quad<float>::load(at >= start ? proj + (size_t)at * ld + ch0 + d
                                          : cs + (size_t)(KEEP + at - start) * dm.channels + ch0 + d,
                              x);
#pragma unroll
          for (int i = 0; i < 4; ++i) past[u][i][m] = x[i];
        }
      }
    }
    float y[NQ][4];
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      const int d = 4 * (lane + 32 * u);
      float x[4] = {0.f, 0.f, 0.f, 0.f};
      if (d < size) Quad<float>::load(proj + (size_t)r * ld + ch0 + d, x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float acc = 0.f;
#pragma unroll
        for (int m = 0; m < KEEP; ++m) acc = fmaf(w[u][i][m], past[u][i][m], acc);
        acc = fmaf(w[u][i][KEEP], x[i], acc);
        y[u][i] = acc * sigmoid_f(acc);
        ss += y[u][i] * y[u][i];
#pragma unroll
        for (int m = 0; m + 1 < KEEP; ++m) past[u][i][m] = past[u][i][m + 1];
        if (KEEP > 0) past[u][i][KEEP > 0 ? KEEP - 1 : 0] = x[i];
      }
      if (update_state && d < size) {
#pragma unroll
        for (int m = 0; m < KEEP; ++m) {
          const float s4[4] = {past[u][0][m], past[u][1][m], past[u][2][m], past[u][3][m]};
          Quad<float>::store(cs + (size_t)m * dm.channels + ch0 + d, s4);
        }
      }
    }
    float f = 1.f;
    float* dst;
    if (unit < 2 * G) {
      const bool is_q = unit < G;
      ss = warp_sum(ss);
      f = (is_q ? rsqrtf((float)D) : 1.f) / sqrtf(ss + 1e-6f);
      dst = (is_q ? qn : kn) + (size_t)r * GD + (size_t)(is_q ? unit : unit - G) * D;
    } else {
      dst = v + ((size_t)r * H + (unit - 2 * G)) * Vd;
    }
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      const int d = 4 * (lane + 32 * u);
      if (d < size) {
        const float o4[4] = {y[u][0] * f, y[u][1] * f, y[u][2] * f, y[u][3] * f};
        Quad<float>::store(dst + d, o4);
      }
    }
  }
}

template <typename T>
__global__ void delta_conv_state_kernel(const T* __restrict__ proj, int ld,
                                        float* __restrict__ state,
                                        const int* __restrict__ cu_seqlens,
                                        const int* __restrict__ slot_ids, DeltaDims dm) {
  const int b = blockIdx.y;
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (ch >= dm.channels) return;
  const int start = cu_seqlens[b], n = cu_seqlens[b + 1] - start;
  float* cs = state + (size_t)slot_ids[b] * dm.state_stride + dm.conv_off;
  const int keep = dm.taps - 1;
  // entry m holds the input (keep - m) tokens before the next one; ascending m reads entries that
  // are not yet overwritten
  for (int m = 0; m < keep; ++m) {
    const int i = n - keep + m;
    cs[(size_t)m * dm.channels + ch] =
        i >= 0 ? to_f32(proj[(size_t)(start + i) * ld + ch]) : cs[(size_t)(m + n) * dm.channels + ch];
  }
}

constexpr int kRecurrenceThreads = 128;
constexpr int kMaxColumnsPerBlock = 32;
constexpr int kStages = 3;             // chunks of tokens in shared memory

__device__ __forceinline__ void copy_async_4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// What a block of the recurrence stages of a token: q, k, decay and v rows and beta of its head (and columns),
// GD, GD, HD, HV and H floats from one token to the next.  vec: 16-byte copies.
struct DeltaStage {
  const float *q, *k, *v, *g, *beta;
  size_t GD, HD, HV;
  int H, D, ncols;
  bool vec;
};
// Tokens ta .. ta + n - 1 into a stage: k | q | g rows of Dp floats (g only with a decay a channel), v columns,
// beta, the head's decay.  Of a row, quad x (four neighbours) lies at quad x / QL + x % QL * (Dp / 4 / QL): where
// a lane has QL quads in a row, its lanes' reads of one of them are then neighbours and meet every bank once.
// RUN > 0: runs of RUN quads lie a quad apart (four lanes share a run, four runs a sum).
template <int Dp, bool ONE_DECAY, int QL, int RUN = 0>
__device__ __forceinline__ void ask_tokens(const DeltaStage& src, float* st, int ta, int n, int tid,
                                           int threads) {
  constexpr int kV = (ONE_DECAY ? 2 : 3) * Dp, kB = kV + kMaxColumnsPerBlock, kTok = kB + 4;
  const int D = src.D;
  auto quad = [](int x) {
    return 4 * (RUN > 0 ? x + x / (RUN > 0 ? RUN : 1) : QL == 1 ? x : x / QL + x % QL * (Dp / 4 / QL));
  };
  auto place = [&](int d) { return quad(d >> 2) + (d & 3); };
  if (src.vec) {                                   // (a thread keeps the same piece of every token)
    const int dq = D >> 2, nd = (ONE_DECAY ? 2 : 3) * dq, pieces = nd + (src.ncols >> 2);
    for (int e = tid; e < pieces; e += threads) {
      const float* from;
      int dst, step;                               // source floats from one token to the next
      if (e < dq) from = src.k + (size_t)ta * src.GD + 4 * e, dst = quad(e), step = (int)src.GD;
      else if (e < 2 * dq)
        from = src.q + (size_t)ta * src.GD + 4 * (e - dq), dst = Dp + quad(e - dq), step = (int)src.GD;
      else if (!ONE_DECAY && e < nd)
        from = src.g + (size_t)ta * src.HD + 4 * (e - 2 * dq), dst = 2 * Dp + quad(e - 2 * dq),
        step = (int)src.HD;
      else from = src.v + (size_t)ta * src.HV + 4 * (e - nd), dst = kV + 4 * (e - nd), step = (int)src.HV;
      for (int tt = 0; tt < n; ++tt)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(st + (size_t)tt * kTok + dst)),
                     "l"(from + (size_t)tt * step)
                     : "memory");
    }
    if (tid < n) {
      copy_async_4(st + (size_t)tid * kTok + kB, src.beta + (size_t)(ta + tid) * src.H);
      if (ONE_DECAY) copy_async_4(st + (size_t)tid * kTok + kB + 1, src.g + (size_t)(ta + tid) * src.H);
    }
    return;
  }
  const int rd = (ONE_DECAY ? 2 : 3) * D;
  const int per = rd + src.ncols + (ONE_DECAY ? 2 : 1);
  for (int i = tid; i < n * per; i += threads) {
    const int tt = i / per, e = i - tt * per;
    const size_t t = (size_t)(ta + tt);
    float* dst = st + (size_t)tt * kTok;
    if (e < D) copy_async_4(dst + place(e), src.k + t * src.GD + e);
    else if (e < 2 * D) copy_async_4(dst + Dp + place(e - D), src.q + t * src.GD + (e - D));
    else if (!ONE_DECAY && e < rd) copy_async_4(dst + 2 * Dp + place(e - 2 * D), src.g + t * src.HD + (e - 2 * D));
    else if (e < rd + src.ncols) copy_async_4(dst + kV + (e - rd), src.v + t * src.HV + (e - rd));
    else if (e == rd + src.ncols) copy_async_4(dst + kB, src.beta + t * src.H);
    else copy_async_4(dst + kB + 1, src.g + t * src.H);
  }
}

// A block = (request, head, 128 / LP columns of S); LP lanes share a column, DPER rows each.  The
// tokens' k, q, g rows (padded to Dp = LP * DPER floats, the padding zero), the block's v columns and
// beta come through three stages of shared memory, CHUNK tokens each, asked for two chunks ahead
// with cp.async.  LP = 4 where requests x heads x columns fill the device (decode batches); LP = 32
// (a warp a column, eight columns a block) where they do not (one long prompt): a token is a chain
// of dependent instructions for a warp, and with eight times the lanes a column the chain is short
// and eight times as many warps share an SM's schedulers.
// ONE_DECAY: g holds a decay a head; it travels beside beta.
template <int DPER, int LP, int CHUNK, int THREADS, bool ONE_DECAY>
__global__ void __launch_bounds__(THREADS)
delta_recurrence_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                        const float* __restrict__ v, const float* __restrict__ g,
                        const float* __restrict__ beta, float* __restrict__ state,
                        const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids,
                        DeltaDims dm, float* __restrict__ o) {
  constexpr int Dp = LP * DPER;
  constexpr int kV = (ONE_DECAY ? 2 : 3) * Dp;                 // where a token's v columns start
  constexpr int kB = kV + kMaxColumnsPerBlock;                 // beta (and the head's decay)
  constexpr int kTok = kB + 4;                                 // floats a token in a stage
  extern __shared__ __align__(16) float stage[];               // [kStages][CHUNK][kTok]
  constexpr int cols = THREADS / LP;
  const int b = blockIdx.x / dm.H, h = blockIdx.x - b * dm.H;
  const int part = threadIdx.x % LP, lc = threadIdx.x / LP;
  const int col0 = blockIdx.y * cols, col = col0 + lc;
  pdl_trigger();
  const int D = dm.D, Vd = dm.Vd;
  for (int i = threadIdx.x; i < kStages * CHUNK * kTok; i += blockDim.x) stage[i] = 0.f;
  __syncthreads();
  pdl_wait();
  const int row0 = part * DPER;
  const bool col_ok = col < Vd;
  const int cj = col_ok ? col : 0;
  const int kvh = h / (dm.H / dm.G);
  float* Sg = state + (size_t)slot_ids[b] * dm.state_stride + ((size_t)h * D) * Vd + cj;
  float S[DPER];
#pragma unroll
  for (int i = 0; i < DPER; ++i) S[i] = (row0 + i < D) ? Sg[(size_t)(row0 + i) * Vd] : 0.f;
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  const size_t GD = (size_t)dm.G * D, HD = (size_t)dm.H * D, HV = (size_t)dm.H * Vd;
  const int ncols = min(cols, Vd - col0);
  const DeltaStage src{qn + (size_t)kvh * D, kn + (size_t)kvh * D, v + (size_t)h * Vd + col0,
                       ONE_DECAY ? g + h : g + (size_t)h * D, beta + h, GD, HD, HV, dm.H, D, ncols,
                       (D & 3) == 0 && (Vd & 3) == 0 && (ncols & 3) == 0};
  auto ask = [&](int chunk) {                      // the chunk's tokens into stage chunk % kStages
    const int ta = t0 + chunk * CHUNK;
    ask_tokens<Dp, ONE_DECAY, 1>(src, stage + (size_t)(chunk % kStages) * CHUNK * kTok, ta,
                                 min(CHUNK, t1 - ta), threadIdx.x, THREADS);
    copy_async_commit();
  };
  const int nchunks = (t1 - t0 + CHUNK - 1) / CHUNK;
  // two chunks are under way while a third is worked on (a group is committed every turn, empty
  // ones too, so that "all but the last two" always means "chunk c has landed")
  for (int c = 0; c < kStages - 1; ++c) {
    if (c < nchunks) ask(c);
    else copy_async_commit();
  }
  for (int c = 0; c < nchunks; ++c) {
    // the stage of chunk c + 2 held chunk c - 1, which every warp left at the last barrier
    if (c + kStages - 1 < nchunks) ask(c + kStages - 1);
    else copy_async_commit();
    copy_async_wait<kStages - 1>();
    __syncthreads();
    const float* st = stage + (size_t)(c % kStages) * CHUNK * kTok;
    const int ta = t0 + c * CHUNK, n = min(CHUNK, t1 - ta);
    // The chunk's tokens, unrolled: the read-out o = S^T q of a token is off the chain that the
    // next token waits for (only u is on it), so its lane reduction is left until the chunk is
    // done and the eight reductions run side by side.
    float outp[CHUNK];
#pragma unroll
    for (int tt = 0; tt < CHUNK; ++tt) {
      outp[tt] = 0.f;
      if (tt < n) {
        const float* tok = st + (size_t)tt * kTok;
        const float4* k4 = reinterpret_cast<const float4*>(tok + row0);
        const float4* q4 = reinterpret_cast<const float4*>(tok + Dp + row0);
        const float4* g4 = reinterpret_cast<const float4*>(tok + 2 * Dp + row0);   // (not ONE_DECAY)
        const float vc = tok[kV + lc], bc = tok[kB], g1 = tok[kB + 1];
        float kc[DPER];
#pragma unroll
        for (int i = 0; i < DPER / 4; ++i) {
          const float4 kk = k4[i];
          const float4 gg = ONE_DECAY ? make_float4(g1, g1, g1, g1) : g4[i];
          kc[4 * i] = kk.x, kc[4 * i + 1] = kk.y, kc[4 * i + 2] = kk.z, kc[4 * i + 3] = kk.w;
          S[4 * i] *= gg.x, S[4 * i + 1] *= gg.y, S[4 * i + 2] *= gg.z, S[4 * i + 3] *= gg.w;
        }
        float d4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < DPER; ++i) d4[i & 3] = fmaf(S[i], kc[i], d4[i & 3]);
        float dot = (d4[0] + d4[1]) + (d4[2] + d4[3]);
#pragma unroll
        for (int sh = 1; sh < LP; sh <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, sh);
        const float u = bc * (vc - dot);
        float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < DPER / 4; ++i) {
          const float4 qq = q4[i];
          S[4 * i] = fmaf(kc[4 * i], u, S[4 * i]);
          S[4 * i + 1] = fmaf(kc[4 * i + 1], u, S[4 * i + 1]);
          S[4 * i + 2] = fmaf(kc[4 * i + 2], u, S[4 * i + 2]);
          S[4 * i + 3] = fmaf(kc[4 * i + 3], u, S[4 * i + 3]);
          o4[0] = fmaf(S[4 * i], qq.x, o4[0]);
          o4[1] = fmaf(S[4 * i + 1], qq.y, o4[1]);
          o4[2] = fmaf(S[4 * i + 2], qq.z, o4[2]);
          o4[3] = fmaf(S[4 * i + 3], qq.w, o4[3]);
        }
        outp[tt] = (o4[0] + o4[1]) + (o4[2] + o4[3]);
      }
    }
#pragma unroll
    for (int sh = 1; sh < LP; sh <<= 1) {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) outp[tt] += __shfl_xor_sync(0xffffffffu, outp[tt], sh);
    }
    if (part == 0 && col_ok) {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt)
        if (tt < n) o[(size_t)(ta + tt) * HV + (size_t)h * Vd + col] = outp[tt];
    }
    __syncthreads();                               // the stage is free for the chunk after next
  }
  if (col_ok) {
#pragma unroll
    for (int i = 0; i < DPER; ++i)
      if (row0 + i < D) Sg[(size_t)(row0 + i) * Vd] = S[i];
  }
}

// ---- portions of many tokens ----------------------------------------------------------------------------
// Where requests x heads x columns do not fill the device (one long prompt, a small decode batch) the time
// is the longest portion's chain from token to token, and behind that what shared memory gives an SM a
// cycle: with a warp a column a token took three 16-byte reads a lane and ten shuffles for every column.
// Here LP lanes share two neighbouring columns, DPER rows each: a read of k, q and g serves both, and most of
// a sum's tree lies in registers.  While a token's sum goes through the lanes, the warp reads the next
// token's operands and multiplies the state that the token before left by that token's q.
// The orders of the sums over the rows are older than this kernel, and a router behind the layer makes close
// calls, so they stay.  Where the triples are few: one binary tree over LP * DPER products in the rows' order
// (a lane's rows, then lanes 1, 2, 4, 8 apart).  Where they are many (CHAIN): four runs of D / 4 rows; of a
// run four chains of multiply-adds, over every fourth row, a lane each; chains, then runs, added in pairs.
// A block is up to four groups of 128 threads that share nothing but the SM, each with a request of its own,
// long and short ones together: blocks of one request each are placed two and more to an SM while others are
// empty (1,201 tokens beside three single ones: 423 us; alone 298).
// On a B200, prompts of 150, 300, 600 and 1,201 tokens, 16 heads of 128 x 128: 420 us a layer (a warp a column:
// 740); one of 1,201 tokens 288 (446); eight of 200
// 202 (four lanes a column: 680), seven of 1 to 900 375 (1,620).
// Up to kTreeSorted requests are sorted by length, in every block (B^2 / 128 comparisons a thread: 512 requests of 5 tokens
// 7.9 ms so, 0.8 as they come); more of them fill the device in any order.
constexpr int kTreeThreads = 128, kTreeChunk = 8, kTreeGroups = 4, kTreeSorted = 64;

template <int N> __device__ __forceinline__ float tree_sum(const float* p) {
  if constexpr (N == 1) return p[0];
  else return tree_sum<N / 2>(p) + tree_sum<N / 2>(p + N / 2);
}

template <int DPER, int LP, bool ONE_DECAY, bool CHAIN>
__global__ void __launch_bounds__(kTreeThreads * kTreeGroups, 1)
delta_tree_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                  const float* __restrict__ v, const float* __restrict__ g,
                  const float* __restrict__ beta, float* __restrict__ state,
                  const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids,
                  DeltaDims dm, int B, int by_length, int whole, float* __restrict__ o) {
  constexpr int D4 = LP * DPER, Dp = D4 + (CHAIN ? 16 : 0), CHUNK = kTreeChunk, COLS = 2;
  constexpr int kV = (ONE_DECAY ? 2 : 3) * Dp;                 // where a token's v columns start
  constexpr int kB = kV + kMaxColumnsPerBlock;                 // beta (and the head's decay)
  constexpr int kTok = kB + 4;                                 // floats a token in a stage
  constexpr int cols = kTreeThreads / LP * COLS;
  static_assert(cols <= kMaxColumnsPerBlock && DPER % 4 == 0 && CHUNK * COLS >= LP && (!CHAIN || LP == 16));
  extern __shared__ __align__(16) float stages[];              // a group: [kStages][CHUNK][kTok]
  __shared__ int request[kTreeGroups];
  const int tid = threadIdx.x % kTreeThreads, group = threadIdx.x / kTreeThreads;
  float* stage = stages + (size_t)group * kStages * CHUNK * kTok;
  auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kTreeThreads) : "memory"); };
  const int part = tid % LP, lc = tid / LP * COLS;
  const int of = blockIdx.x / dm.H, h = blockIdx.x - of * dm.H, nz = gridDim.x / dm.H;
  const int col0 = blockIdx.y * cols, col = col0 + lc;
  pdl_trigger();
  const int D = dm.D, Vd = dm.Vd;
  if (D != D4) {                                               // the rows that are not there are zero
    for (int i = tid; i < kStages * CHUNK * kTok; i += kTreeThreads) stage[i] = 0.f;
    group_sync();
  }
  pdl_wait();
  // the group's request: the b-th longest portion's; groups of odd number take theirs from the other end
  int b = group * nz + (group & 1 ? nz - 1 - of : of);
  if (b >= B) return;
  if (by_length) {
    for (int i = tid; i < B; i += kTreeThreads) {
      const int mine = cu_seqlens[i + 1] - cu_seqlens[i];
      int before = 0;
      for (int j = 0; j < B; ++j) {
        const int its = cu_seqlens[j + 1] - cu_seqlens[j];
        before += its > mine || (its == mine && j < i);
      }
      if (before == b) request[group] = i;
    }
    group_sync();
    b = request[group];
  }
  // the lane's i-th row
  auto row = [&](int i) { return CHAIN ? part / 4 * (4 * DPER) + 4 * i + part % 4 : part * DPER + i; };
  const int kvh = h / (dm.H / dm.G);
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  const size_t GD = (size_t)dm.G * D, HD = (size_t)dm.H * D, HV = (size_t)dm.H * Vd;
  const int ncols = min(cols, Vd - col0);
  const DeltaStage src{qn + (size_t)kvh * D, kn + (size_t)kvh * D, v + (size_t)h * Vd + col0,
                       ONE_DECAY ? g + h : g + (size_t)h * D, beta + h, GD, HD, HV, dm.H, D, ncols,
                       (D & 3) == 0 && (Vd & 3) == 0 && (ncols & 3) == 0};
  auto ask = [&](int chunk) {                      // the chunk's tokens into stage chunk % kStages
    const int ta = t0 + chunk * CHUNK;
    ask_tokens<Dp, ONE_DECAY, DPER / 4, CHAIN ? DPER : 0>(src, stage + (size_t)(chunk % kStages) * CHUNK * kTok, ta,
                                        min(CHUNK, t1 - ta), tid, kTreeThreads);
    copy_async_commit();
  };
  const int nchunks = (t1 - t0 + CHUNK - 1) / CHUNK;
  for (int c = 0; c < kStages - 1; ++c) {
    if (c < nchunks) ask(c);
    else copy_async_commit();
  }
  // the state, while the first chunks come: both columns at once where rows are whole and aligned
  float* Sg = state + (size_t)slot_ids[b] * dm.state_stride + (size_t)h * D * Vd + col;
  float S[DPER][COLS];
#pragma unroll
  for (int i = 0; i < DPER; ++i) {
    S[i][0] = S[i][1] = 0.f;
    if (row(i) < D) {
      const float* at = Sg + (size_t)row(i) * Vd;
      if (whole) {
        if (col < Vd) {
          const float2 two = *reinterpret_cast<const float2*>(at);
          S[i][0] = two.x, S[i][1] = two.y;
        }
      } else {
#pragma unroll
        for (int c = 0; c < COLS; ++c)
          if (col + c < Vd) S[i][c] = at[c];
      }
    }
  }
  for (int ch = 0; ch < nchunks; ++ch) {
    if (ch + kStages - 1 < nchunks) ask(ch + kStages - 1);     // (the stage that chunk ch - 1 left)
    else copy_async_commit();
    copy_async_wait<kStages - 1>();
    group_sync();
    const float* tok = stage + (size_t)(ch % kStages) * CHUNK * kTok;
    const int ta = t0 + ch * CHUNK, n = min(CHUNK, t1 - ta);
    float outp[CHUNK * COLS];                                  // summed over the lanes behind the chunk
    float k[DPER], gd[DPER], q[DPER], vb[COLS + 1], before[DPER][COLS];
    auto quads = [&](const float* from, float (&to)[DPER]) {
      if constexpr (CHAIN) {
#pragma unroll
        for (int i = 0; i < DPER; ++i) to[i] = from[part / 4 * (4 * DPER + 4) + part % 4 + 4 * i];
        return;
      }
#pragma unroll
      for (int i = 0; i < DPER; i += 4) {
        const float4 x = *reinterpret_cast<const float4*>(from + (i / 4 * LP + part) * 4);
        to[i] = x.x, to[i + 1] = x.y, to[i + 2] = x.z, to[i + 3] = x.w;
      }
    };
    auto operands = [&](const float* t) {                      // all but q
      quads(t, k);
      if (!ONE_DECAY) quads(t + 2 * Dp, gd);
      else gd[0] = t[kB + 1];
      const float2 vv = *reinterpret_cast<const float2*>(t + kV + lc);
      vb[0] = vv.x, vb[1] = vv.y, vb[2] = t[kB];
    };
    auto read_out = [&](int tt) {
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        float p[DPER];
#pragma unroll
        for (int i = 0; i < DPER; ++i) p[i] = fmaf(before[i][c], q[i], CHAIN && i ? p[i - (i > 0)] : 0.f);
        outp[tt * COLS + c] = CHAIN ? p[DPER - 1] : tree_sum<DPER>(p);
      }
    };
    auto token = [&](int tt, bool more) {
      float dot[COLS], kc[DPER];
#pragma unroll
      for (int i = 0; i < DPER; ++i) kc[i] = k[i];
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        float p[DPER];
#pragma unroll
        for (int i = 0; i < DPER; ++i) {
          S[i][c] *= gd[ONE_DECAY ? 0 : i];
          p[i] = fmaf(S[i][c], kc[i], CHAIN && i ? p[i - (i > 0)] : 0.f);
        }
        dot[c] = CHAIN ? p[DPER - 1] : tree_sum<DPER>(p);
      }
      const float vc[COLS] = {vb[0], vb[1]}, bc = vb[2];
#pragma unroll
      for (int c = 0; c < COLS; ++c) dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], 1);
      if (more) operands(tok + kTok);
#pragma unroll
      for (int c = 0; c < COLS; ++c) dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], 2);
      if (tt > 0) read_out(tt - 1);
#pragma unroll
      for (int sh = 4; sh < LP; sh <<= 1) {
#pragma unroll
        for (int c = 0; c < COLS; ++c) dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], sh);
        if (sh == 4) quads(tok + Dp, q);
      }
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        const float u = bc * (vc[c] - dot[c]);
#pragma unroll
        for (int i = 0; i < DPER; ++i) before[i][c] = S[i][c] = fmaf(kc[i], u, S[i][c]);
      }
      tok += kTok;
    };
    operands(tok);
    if (n == CHUNK) {                                          // (no branch between tokens)
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) token(tt, tt + 1 < CHUNK);
      read_out(CHUNK - 1);
    } else {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) {
        outp[tt * COLS] = outp[tt * COLS + 1] = 0.f;
        if (tt < n) token(tt, tt + 1 < n);
        if (tt == n - 1) read_out(tt);
      }
    }
    // add up across the lanes; every halving of the list leaves a lane the half that its bit names
    int first = 0;
    constexpr int kAll = CHUNK * COLS;
#pragma unroll
    for (int sh = 1; sh < LP; sh <<= 1) {
      const int half = kAll / (2 * sh);
      const bool up = part & sh;
#pragma unroll
      for (int m = 0; m < half; ++m) {
        const float got = __shfl_xor_sync(0xffffffffu, up ? outp[m] : outp[m + half], sh);
        outp[m] = (up ? outp[m + half] : outp[m]) + got;
      }
      if (up) first += half;
    }
#pragma unroll
    for (int m = 0; m < kAll / LP; ++m) {
      const int tt = (first + m) / COLS, c = (first + m) % COLS;
      if (tt < n && col + c < Vd) o[(size_t)(ta + tt) * HV + (size_t)h * Vd + col + c] = outp[m];
    }
    group_sync();                                  // the stage is free for the chunk after next
  }
#pragma unroll
  for (int i = 0; i < DPER; ++i)
    if (row(i) < D) {
      float* at = Sg + (size_t)row(i) * Vd;
      if (whole) {
        if (col < Vd) *reinterpret_cast<float2*>(at) = make_float2(S[i][0], S[i][1]);
      } else {
#pragma unroll
        for (int c = 0; c < COLS; ++c)
          if (col + c < Vd) at[c] = S[i][c];
      }
    }
}

// ---- eight tokens at a time ---------------------------------------------------------------------
// With one decay a head the recurrence over a chunk of tokens 0 .. 7 that starts from S needs S only
// in products that do not wait for one another.  With G_i = g_0 .. g_i, R(j, i) = g_(j+1) .. g_i:
//
//   u_i = beta_i (v_i - G_i S^T k_i) - sum_(j<i) L_ij u_j,   L_ij = beta_i R(j, i) k_j.k_i
//   o_i = G_i S^T q_i + sum_(j<=i) M_ij u_j,                 M_ij = R(j, i) k_j.q_i
//   S  <- G_7 S + sum_j R(j, 7) k_j u_j^T
//
// (ratios of decays are products of the factors between the two tokens, never quotients).  The chain
// from token to token is then eight multiply-adds in registers a chunk, instead of a pass over S and a
// reduction across lanes a token.  Everything is 32-bit multiply-adds.
constexpr int CT = 8;                                          // tokens a chunk
constexpr int kCoefL = 0, kCoefM = 64, kCoefG = 128, kCoefE = 136, kCoefBeta = 144, kCoefs = 152;

// Chunks of request b start at the packed number cu[b] / CT + b; no two requests' chunks meet.
__device__ __forceinline__ int chunk_number(int first_row, int b, int c) { return first_row / CT + b + c; }

// A warp a (chunk, kv head): the 64 dot products k_j.k_i (j < i) and k_j.q_i (j <= i), then for every
// head of the group L, M, G, E (E_j = R(j, 7)) and beta.  Tokens behind the portion's end count as
// k = q = 0, g = 1, beta = 0.
__global__ void __launch_bounds__(128)
delta_chunk_coef_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                        const float* __restrict__ g, const float* __restrict__ beta,
                        const int* __restrict__ cu_seqlens, DeltaDims dm, float* __restrict__ coef) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 4 + (threadIdx.x >> 5), b = blockIdx.y, kvh = blockIdx.z;
  pdl_wait();
  const int t0 = cu_seqlens[b], ta = t0 + c * CT, n = min(CT, cu_seqlens[b + 1] - ta);
  if (n <= 0) return;
  const int D = dm.D, H = dm.H, per = H / dm.G;
  const size_t GD = (size_t)dm.G * D;
  // pair (a, e) = (m / 8, m % 8): k_e.k_a for a > e, k_a.q_e for a <= e
  float val[64];
#pragma unroll
  for (int m = 0; m < 64; ++m) val[m] = 0.f;
  for (int d = 4 * lane; d < D; d += 128) {
    float k[CT][4], q[CT][4];
#pragma unroll
    for (int i = 0; i < CT; ++i) {
#pragma unroll
      for (int x = 0; x < 4; ++x) k[i][x] = q[i][x] = 0.f;
      if (i < n) {
        const size_t at = (size_t)(ta + i) * GD + (size_t)kvh * D + d;
        Quad<float>::load(kn + at, k[i]);
        Quad<float>::load(qn + at, q[i]);
      }
    }
#pragma unroll
    for (int m = 0; m < 64; ++m) {
      const int a = m >> 3, e = m & 7;
#pragma unroll
      for (int x = 0; x < 4; ++x) val[m] = fmaf(k[a > e ? e : a][x], a > e ? k[a][x] : q[e][x], val[m]);
    }
  }
  // add up across the lanes, halving the values each lane carries: lane l ends with m = l, l + 32
#pragma unroll
  for (int half = 16; half >= 1; half >>= 1) {
    const bool up = lane & half;
    // values that differ in this bit of m are neighbours at distance `half`; what is left of the
    // list is indexed by m with the higher bits already fixed to the lane's
#pragma unroll
    for (int hi = 0; hi < 2; ++hi)
#pragma unroll
      for (int m = 0; m < half; ++m) {
        const float lo_v = val[32 * hi + m], hi_v = val[32 * hi + m + half];
        const float got = __shfl_xor_sync(0xffffffffu, up ? lo_v : hi_v, half);
        val[32 * hi + m] = (up ? hi_v : lo_v) + got;
      }
  }
  const float mine[2] = {val[0], val[32]};
  float* base = coef + ((size_t)chunk_number(t0, b, c) * H + (size_t)kvh * per) * kCoefs;
  for (int hh = 0; hh < per; ++hh) {
    const int h = kvh * per + hh;
    const bool real = lane < n;
    const float gl = real ? g[(size_t)(ta + lane) * H + h] : 1.f;
    const float bl = real ? beta[(size_t)(ta + lane) * H + h] : 0.f;
    float* dst = base + (size_t)hh * kCoefs;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int m = lane + 32 * x, a = m >> 3, e = m & 7;
      const int i = a > e ? a : e, j = a > e ? e : a;          // j <= i
      float r = 1.f;
#pragma unroll
      for (int s = 1; s < CT; ++s) {
        const float gs = __shfl_sync(0xffffffffu, gl, s);
        if (s > j && s <= i) r *= gs;
      }
      const float bi = __shfl_sync(0xffffffffu, bl, i);
      if (a > e) {
        dst[kCoefL + i * CT + j] = bi * r * mine[x];
        dst[kCoefM + j * CT + i] = 0.f;                         // (M is read as whole rows)
      } else {
        dst[kCoefM + i * CT + j] = r * mine[x];
        if (i == j) dst[kCoefL + i * CT + j] = 0.f;
      }
    }
    float G = 1.f, E = 1.f;
#pragma unroll
    for (int s = 0; s < CT; ++s) {
      const float gs = __shfl_sync(0xffffffffu, gl, s);
      if (s <= lane) G *= gs;
      if (s > lane) E *= gs;
    }
    if (lane < CT) {
      dst[kCoefG + lane] = G;
      dst[kCoefE + lane] = E;
      dst[kCoefBeta + lane] = bl;
    }
  }
}

// The same for a plain linear attention with a decay a key channel, S <- diag(g) S + k v^T: its u is v, so
// there is no L and no beta.  G_i, R and G_7 are vectors: R stands inside the dot products M is made of,
// and the recurrence reads G_i q_i and R(j, 7) k_j (elementwise) in the places of q_i and k_j.  A warp a
// (chunk, head): those two for every token, [T, H, D] each, M, and the chunk's G_7.  On a B200, two
// prompts of 1,500 and 1,700 tokens, 16 heads of 128 x 128: 20 us, and 360 for the recurrence behind it.
// (The delta rule itself with a decay a channel goes token by token in steps of every length: a router
// behind it makes close calls, so its sums keep one order.)  ld_q, ld_k, ld_g: floats between two tokens.
// The launch takes `heads` heads from number `head0` on, so that what it leaves is bounded: [T, heads, D].
__global__ void __launch_bounds__(128)
linear_chunk_coef_kernel(const float* __restrict__ qn, int ld_q, const float* __restrict__ kn,
                         int ld_k, const float* __restrict__ g, int ld_g,
                         const int* __restrict__ cu_seqlens, DeltaDims dm, int head0, int heads,
                         float* __restrict__ coef, float* __restrict__ total,
                         float* __restrict__ qg, float* __restrict__ ke) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 4 + (threadIdx.x >> 5), b = blockIdx.y, hl = blockIdx.z, h = head0 + hl;
  pdl_wait();
  const int t0 = cu_seqlens[b], ta = t0 + c * CT, n = min(CT, cu_seqlens[b + 1] - ta);
  if (n <= 0) return;
  const int D = dm.D, kvh = h / (dm.H / dm.G);
  const size_t HD = (size_t)heads * D;
  const size_t chunk = (size_t)chunk_number(t0, b, c) * heads + hl;
  float val[64];                                             // pairs as above
#pragma unroll
  for (int m = 0; m < 64; ++m) val[m] = 0.f;
  for (int d = 4 * lane; d < D; d += 128) {
    float k[CT][4], q[CT][4], gd[CT][4];
#pragma unroll
    for (int i = 0; i < CT; ++i) {
#pragma unroll
      for (int x = 0; x < 4; ++x) k[i][x] = q[i][x] = 0.f, gd[i][x] = 1.f;
      if (i < n) {
        const size_t r = ta + i;
        Quad<float>::fresh(kn + r * ld_k + (size_t)kvh * D + d, k[i]);
        Quad<float>::fresh(qn + r * ld_q + (size_t)kvh * D + d, q[i]);
        Quad<float>::fresh(g + r * ld_g + (size_t)h * D + d, gd[i]);
      }
    }
#pragma unroll
    for (int j = 0; j < CT; ++j) {
      float kr[4];                                           // R(j, i) k_j
#pragma unroll
      for (int x = 0; x < 4; ++x) kr[x] = k[j][x], val[9 * j] = fmaf(kr[x], q[j][x], val[9 * j]);
#pragma unroll
      for (int i = j + 1; i < CT; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          kr[x] *= gd[i][x];
          val[8 * j + i] = fmaf(kr[x], q[i][x], val[8 * j + i]);
        }
      if (j < n) Quad<float>::store(ke + (size_t)(ta + j) * HD + (size_t)hl * D + d, kr);
    }
    float G[4] = {1.f, 1.f, 1.f, 1.f};
#pragma unroll
    for (int i = 0; i < CT; ++i) {
      float e[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) G[x] *= gd[i][x], e[x] = G[x] * q[i][x];
      if (i < n) Quad<float>::store(qg + (size_t)(ta + i) * HD + (size_t)hl * D + d, e);
    }
    Quad<float>::store(total + chunk * D + d, G);
  }
#pragma unroll
  for (int half = 16; half >= 1; half >>= 1) {               // lane l ends with m = l, l + 32, as above
    const bool up = lane & half;
#pragma unroll
    for (int hi = 0; hi < 2; ++hi)
#pragma unroll
      for (int m = 0; m < half; ++m) {
        const float lo_v = val[32 * hi + m], hi_v = val[32 * hi + m + half];
        const float got = __shfl_xor_sync(0xffffffffu, up ? lo_v : hi_v, half);
        val[32 * hi + m] = (up ? hi_v : lo_v) + got;
      }
  }
  const float mine[2] = {val[0], val[32]};
  float* dst = coef + chunk * kCoefs;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int m = lane + 32 * x, a = m >> 3, e = m & 7;
    dst[kCoefM + e * CT + a] = a > e ? 0.f : mine[x];        // (M is read as whole rows)
  }
}

// A block = (request, head, 16 CP columns of S); LANES (8 or 16) lanes a column, CP columns a lane (a read
// of k or q serves them all: shared-memory reads bound a block, and two columns a lane halve them where
// there are blocks enough without).  Lane p of a column owns
// the rows 4 (p + LANES i) .. + 3, i < DPER / 4, so that the lanes' reads of a token's k and q are one run of
// shared memory.  Stages as in the kernel above, one barrier a chunk.
// HEADS: the delta rule with a decay a head; ke and total are not read.  PLAIN: linear attention with a
// decay a key channel (u = v; kn is not read; eight lanes a column); qn and ke are [T, heads, D] as
// linear_chunk_coef_kernel leaves them, total the chunks' G_7.  The launch takes `heads` heads from number
// `head0` on (HEADS: all).
enum { HEADS = 0, PLAIN = 1 };
template <int DPER, int LANES, int CP, int MODE>
__global__ void __launch_bounds__(16 * LANES)
delta_chunk_recurrence_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                              const float* __restrict__ ke, const float* __restrict__ total,
                              const float* __restrict__ v, int ld_v, const float* __restrict__ coef,
                              float* __restrict__ state, const int* __restrict__ cu_seqlens,
                              const int* __restrict__ slot_ids, DeltaDims dm, int head0, int heads,
                              float* __restrict__ o) {
  constexpr int Dp = LANES * DPER, COLS = 16 * CP, NQ = DPER / 4;
  static_assert(MODE != PLAIN || LANES == CT, "a lane a token of a chunk");
  // two sets of [CT][Dp]: k | q, or q | ke
  constexpr int kQ = MODE == PLAIN ? 0 : CT * Dp, kE = MODE == HEADS ? 0 : CT * Dp, kG = 2 * CT * Dp;
  constexpr int kVc = kG + (MODE == HEADS ? 0 : Dp), kC = kVc + CT * COLS, kStage = kC + kCoefs;
  constexpr int DOTS = MODE == PLAIN ? CT : 2 * CT;            // with S: the chunk's q, and k in front of them
  extern __shared__ __align__(16) float stage[];               // [kStages][kStage]
  const int b = blockIdx.x / heads, hl = blockIdx.x - b * heads, h = head0 + hl;
  const int p = threadIdx.x % LANES, lc = threadIdx.x / LANES;
  const int col0 = blockIdx.y * COLS;                          // a lane's columns: col0 + lc + 16 c
  pdl_trigger();
  const int D = dm.D, Vd = dm.Vd;
  for (int i = threadIdx.x; i < kStages * kStage; i += blockDim.x) stage[i] = 0.f;
  __syncthreads();
  pdl_wait();
  const int kvh = MODE == HEADS ? h / (dm.H / dm.G) : hl;
  float* Sg = state + (size_t)slot_ids[b] * dm.state_stride + ((size_t)h * D) * Vd;
  float S[CP][NQ][4];
#pragma unroll
  for (int y = 0; y < CP; ++y)
#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int row = 4 * (p + LANES * i) + x, col = col0 + lc + 16 * y;
        S[y][i][x] = row < D ? Sg[(size_t)row * Vd + (col < Vd ? col : 0)] : 0.f;
      }
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  const size_t KD = (size_t)(MODE == HEADS ? dm.G : heads) * D, HV = (size_t)dm.H * Vd;
  const int vq = min(COLS, Vd - col0) >> 2, dq = D >> 2;
  const int nchunks = (t1 - t0 + CT - 1) / CT;
  const int chunk0 = chunk_number(t0, b, 0);
  const float* coef0 = coef + ((size_t)chunk0 * heads + hl) * kCoefs;
  auto copy16 = [](float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  };
  auto ask = [&](int c) {
    float* st = stage + (size_t)(c % kStages) * kStage;
    const int ta = t0 + c * CT, n = min(CT, t1 - ta);
    for (int e = threadIdx.x; e < n * dq; e += blockDim.x) {
      const int t = e / dq, d = 4 * (e - t * dq);
      const size_t at = (size_t)(ta + t) * KD + (size_t)kvh * D + d;
      if (MODE != PLAIN) copy16(st + t * Dp + d, kn + at);
      copy16(st + kQ + t * Dp + d, qn + at);
      if (MODE != HEADS) copy16(st + kE + t * Dp + d, ke + at);
    }
    if (MODE != HEADS)
      for (int e = threadIdx.x; e < dq; e += blockDim.x)
        copy16(st + kG + 4 * e, total + ((size_t)(chunk0 + c) * heads + hl) * D + 4 * e);
    for (int e = threadIdx.x; e < n * vq; e += blockDim.x) {
      const int t = e / vq, d = 4 * (e - t * vq);
      copy16(st + kVc + t * COLS + d, v + (size_t)(ta + t) * ld_v + (size_t)h * Vd + col0 + d);
    }
    if (n < CT) {                    // behind the portion's end: zeros, not an older chunk's tokens
      for (int e = threadIdx.x; e < (CT - n) * Dp; e += blockDim.x)
        st[n * Dp + e] = st[CT * Dp + n * Dp + e] = 0.f;
      for (int e = threadIdx.x; e < (CT - n) * COLS; e += blockDim.x) st[kVc + n * COLS + e] = 0.f;
    }
    for (int e = threadIdx.x; e < kCoefs / 4; e += blockDim.x)
      copy16(st + kC + 4 * e, coef0 + (size_t)c * heads * kCoefs + 4 * e);
  };
  for (int c = 0; c < kStages - 1; ++c) {
    if (c < nchunks) ask(c);
    copy_async_commit();
  }
  for (int c = 0; c < nchunks; ++c) {
    copy_async_wait<kStages - 2>();
    __syncthreads();                 // chunk c has landed for all, and all have left chunk c - 1
    if (c + kStages - 1 < nchunks) ask(c + kStages - 1);       // into the stage of chunk c - 1
    copy_async_commit();
    const float* st = stage + (size_t)(c % kStages) * kStage;
    const float* cf = st + kC;
    // this lane's share of S^T k_i (x[i]) and S^T q_i (x[8 + i]; PLAIN: x[i])
    float x[CP][DOTS];
#pragma unroll
    for (int y = 0; y < CP; ++y)
#pragma unroll
      for (int i = 0; i < DOTS; ++i) x[y][i] = 0.f;
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const float* at = st + 4 * (p + LANES * i);
#pragma unroll
      for (int t = 0; t < DOTS; ++t) {
        const float4 a = *reinterpret_cast<const float4*>(at + t * Dp);
#pragma unroll
        for (int y = 0; y < CP; ++y) {
          const float(&s)[4] = S[y][i];
          x[y][t] = fmaf(s[0], a.x, fmaf(s[1], a.y, fmaf(s[2], a.z, fmaf(s[3], a.w, x[y][t]))));
        }
      }
    }
    // add up across the column's lanes: of eight, lane p ends with both sums of token p; of sixteen,
    // lane p with S^T k of token p or S^T q of token p - 8
#pragma unroll
    for (int half = LANES / 2; half >= 1; half >>= 1) {
      const bool up = p & half;
#pragma unroll
      for (int y = 0; y < CP; ++y)
#pragma unroll
        for (int hi = 0; hi < DOTS / LANES; ++hi)
#pragma unroll
          for (int m = 0; m < half; ++m) {
            const float lo_v = x[y][LANES * hi + m], hi_v = x[y][LANES * hi + m + half];
            const float got = __shfl_xor_sync(0xffffffffu, up ? lo_v : hi_v, half);
            x[y][LANES * hi + m] = (up ? hi_v : lo_v) + got;
          }
    }
    const int tok = p % CT;                                     // the token this lane looks after
    const float Gp = MODE == HEADS ? cf[kCoefG + tok] : 1.f;
    float u[CP][CT];
    if constexpr (MODE == PLAIN) {
#pragma unroll
      for (int y = 0; y < CP; ++y)
#pragma unroll
        for (int i = 0; i < CT; ++i) u[y][i] = st[kVc + i * COLS + lc + 16 * y];
    } else {
#pragma unroll
    for (int y = 0; y < CP; ++y) {
      const float rp = cf[kCoefBeta + tok] * (st[kVc + tok * COLS + lc + 16 * y] - Gp * x[y][0]);
#pragma unroll
      for (int i = 0; i < CT; ++i) u[y][i] = __shfl_sync(0xffffffffu, rp, i, LANES);
    }
#pragma unroll
    for (int j = 0; j < CT - 1; ++j)
#pragma unroll
      for (int i = j + 1; i < CT; ++i) {
        const float l = -cf[kCoefL + i * CT + j];
#pragma unroll
        for (int y = 0; y < CP; ++y) u[y][i] = fmaf(l, u[y][j], u[y][i]);
      }
    }
    {
      const float4* Mp = reinterpret_cast<const float4*>(cf + kCoefM + tok * CT);
      const float4 m0 = Mp[0], m1 = Mp[1];
      const int row = t0 + c * CT + tok;
      const float m[CT] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
      float out[CP], all = 0.f;
#pragma unroll
      for (int y = 0; y < CP; ++y) {
        out[y] = Gp * x[y][LANES == CT && MODE != PLAIN ? CT : 0];
#pragma unroll
        for (int j = 0; j < CT; ++j) out[y] = fmaf(m[j ^ 3], u[y][j ^ 3], out[y]);
        all += out[y];
      }
      if (isnan(all)) {          // M is 0 for later tokens, but 0 times what is no number would reach back
#pragma unroll
        for (int y = 0; y < CP; ++y) {
          out[y] = Gp * x[y][LANES == CT && MODE != PLAIN ? CT : 0];
#pragma unroll
          for (int j = 0; j < CT; ++j)
            if ((j ^ 3) <= tok) out[y] = fmaf(m[j ^ 3], u[y][j ^ 3], out[y]);
        }
      }
#pragma unroll
      for (int y = 0; y < CP; ++y) {
        const int col = col0 + lc + 16 * y;
        if (col < Vd && row < t1 && p >= LANES - CT) o[(size_t)row * HV + (size_t)h * Vd + col] = out[y];
      }
    }
    const float Gc = MODE == HEADS ? cf[kCoefG + CT - 1] : 1.f;
    if (MODE == HEADS)
#pragma unroll
      for (int j = 0; j < CT; ++j) {
        const float e = cf[kCoefE + j];
#pragma unroll
        for (int y = 0; y < CP; ++y) u[y][j] *= e;
      }
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const float* at = st + kE + 4 * (p + LANES * i);
      float4 g4 = make_float4(Gc, Gc, Gc, Gc);
      if (MODE != HEADS) g4 = *reinterpret_cast<const float4*>(st + kG + 4 * (p + LANES * i));
#pragma unroll
      for (int y = 0; y < CP; ++y)
        S[y][i][0] *= g4.x, S[y][i][1] *= g4.y, S[y][i][2] *= g4.z, S[y][i][3] *= g4.w;
#pragma unroll
      for (int t = 0; t < CT; ++t) {
        const float4 a = *reinterpret_cast<const float4*>(at + t * Dp);
#pragma unroll
        for (int y = 0; y < CP; ++y) {
          S[y][i][0] = fmaf(a.x, u[y][t], S[y][i][0]);
          S[y][i][1] = fmaf(a.y, u[y][t], S[y][i][1]);
          S[y][i][2] = fmaf(a.z, u[y][t], S[y][i][2]);
          S[y][i][3] = fmaf(a.w, u[y][t], S[y][i][3]);
        }
      }
    }
  }
#pragma unroll
  for (int y = 0; y < CP; ++y)
#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int row = 4 * (p + LANES * i) + x, col = col0 + lc + 16 * y;
        if (row < D && col < Vd) Sg[(size_t)row * Vd + col] = S[y][i][x];
      }
}

struct ChunkArgs {
  const float *q, *k, *ke, *total, *v;
  int ld_v;
  const float* coef;
  float* state;
  const int *cu_seqlens, *slot_ids;
  int head0, heads;
  float* o;
};

template <int DPER, int LANES, int CP, int MODE>
static int launch_chunk_columns(int B, const DeltaDims& dm, const ChunkArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)kStages * sizeof(float) *
                      ((2 * CT + (MODE == HEADS ? 0 : 1)) * LANES * DPER + CT * 16 * CP + kCoefs);
  static OncePerDevice attrs;
  if (int rc = attrs.run([&] {
        return cudaFuncSetAttribute(delta_chunk_recurrence_kernel<DPER, LANES, CP, MODE>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      }))
    return rc;
  return launch_kernel(delta_chunk_recurrence_kernel<DPER, LANES, CP, MODE>,
                       dim3(B * a.heads, (dm.Vd + 16 * CP - 1) / (16 * CP)), dim3(16 * LANES), smem, st, a.q,
                       a.k, a.ke, a.total, a.v, a.ld_v, a.coef, a.state, a.cu_seqlens, a.slot_ids, dm, a.head0,
                       a.heads, a.o);
}

template <int DPER, int LANES, int MODE>
static int launch_chunks(int B, const DeltaDims& dm, const ChunkArgs& a, cudaStream_t st) {
  // two blocks an SM of 16 columns: then one of 32 each does the same work with half the reads (16 heads of 128
  // x 128, coefficients and this, 16 / 32 columns, us: eight portions of 500 tokens, delta rule 530 / 335,
  // linear 483 / 248; four of up to 1,201, 432 / 378 and 359 / 311)
  if (LANES * DPER <= 128 && (long long)B * a.heads * ((dm.Vd + 15) / 16) >= 2 * 148 && dm.Vd > 16)
    return launch_chunk_columns<DPER, LANES, LANES * DPER <= 128 ? 2 : 1, MODE>(B, dm, a, st);
  return launch_chunk_columns<DPER, LANES, 1, MODE>(B, dm, a, st);
}

template <typename T>
__global__ void delta_output_kernel(const float* __restrict__ o, const T* __restrict__ gate,
                                    int gate_ld, const float* __restrict__ w, float eps,
                                    T* __restrict__ out, int pairs, int H, int Vd) {
  const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  if (pair >= pairs) return;
  const int t = pair / H, h = pair - t * H;
  const float* src = o + (size_t)pair * Vd;
  float ss = 0.f;
  for (int j = lane; j < Vd; j += 32) ss += src[j] * src[j];
  ss = warp_sum(ss);
  const float rms = sqrtf(ss / (float)Vd + eps);
  for (int j = lane; j < Vd; j += 32) {
    const float gt = sigmoid_f(to_f32(gate[(size_t)t * gate_ld + (size_t)h * Vd + j]));
    out[(size_t)pair * Vd + j] = from_f32<T>(src[j] / rms * w[j] * gt);
  }
}

}  // namespace gf

using namespace gf;
using bf = __nv_bfloat16;

GF_DEFINE_PDL_SWITCH

static DeltaDims dims_of(int H, int G, int D, int Vd, int taps, int state_stride, int conv_off) {
  DeltaDims dm;
  dm.H = H, dm.G = G, dm.D = D, dm.Vd = Vd, dm.taps = taps;
  dm.channels = 2 * G * D + H * Vd;
  dm.state_stride = state_stride, dm.conv_off = conv_off, dm.a_ld = 0;
  return dm;
}

// proj: [T, ld] with the columns q | k | v first and the H beta columns at b_off.
GF_EXPORT int gf_delta_prepare(const void* proj, int ld, int b_off, const float* a,
                               const float* conv_w, const float* dt_bias, const float* A_log,
                               float* state, const int* seq_of_token, const int* cu_seqlens,
                               const int* slot_ids, int T, int B, int H, int G, int D, int Vd,
                               int taps, int state_stride, int conv_off, float* qn, float* kn,
                               float* v, float* g, float* beta, int dtype, void* stream) {
  if (T <= 0) return 0;
  if (H % G || taps < 1) return -3;
  const DeltaDims dm = dims_of(H, G, D, Vd, taps, state_stride, conv_off);
  if (D > 32 * kPrepareMaxPerLane) return -3;
  auto st = (cudaStream_t)stream;
  const int units = 2 * G + 2 * H + 1;
  const dim3 pgrid(T, (units + kPrepareWarps - 1) / kPrepareWarps), pblock(kPrepareWarps * 32);
  int rc;
  if (dtype == GF_F32)
    rc = launch_kernel(delta_prepare_kernel<float, false>, pgrid, pblock, 0, st, (const float*)proj, ld,
                       b_off, a, conv_w, dt_bias, A_log, (const float*)state, seq_of_token,
                       cu_seqlens, slot_ids, dm, qn, kn, v, g, beta);
  else
    rc = launch_kernel(delta_prepare_kernel<bf, false>, pgrid, pblock, 0, st, (const bf*)proj, ld, b_off,
                       a, conv_w, dt_bias, A_log, (const float*)state, seq_of_token, cu_seqlens,
                       slot_ids, dm, qn, kn, v, g, beta);
  if (rc || taps == 1) return rc;
  const dim3 grid((dm.channels + 127) / 128, B);
  if (dtype == GF_F32)
    return launch_kernel(delta_conv_state_kernel<float>, grid, dim3(128), 0, st,
                         (const float*)proj, ld, state, cu_seqlens, slot_ids, dm);
  return launch_kernel(delta_conv_state_kernel<bf>, grid, dim3(128), 0, st, (const bf*)proj, ld,
                       state, cu_seqlens, slot_ids, dm);
}

// One decay a head.  proj: [T, ld] fp32 with the columns q | k | v first and the heads' decay
// pre-activations and betas at a_off and b_off.  max_q_len: the step's longest portion.
GF_EXPORT int gf_delta_prepare_heads(const float* proj, int ld, int a_off, int b_off,
                                     const float* conv_w, const float* dt_bias, const float* A_log,
                                     float* state, const int* seq_of_token, const int* cu_seqlens,
                                     const int* slot_ids, int T, int B, int max_q_len, int H, int G,
                                     int D, int Vd, int taps, int state_stride, int conv_off,
                                     float* qn, float* kn, float* v, float* g, float* beta,
                                     void* stream) {
  if (T <= 0) return 0;
  if (H % G || taps < 1 || D > 32 * kPrepareMaxPerLane) return -3;
  DeltaDims dm = dims_of(H, G, D, Vd, taps, state_stride, conv_off);
  dm.a_ld = ld;
  auto st = (cudaStream_t)stream;
  const int units = 2 * G + H + 1;
  const bool al = (((uintptr_t)proj | (uintptr_t)state | (uintptr_t)qn | (uintptr_t)kn |
                    (uintptr_t)v) & 15) == 0;
  bool updated = false;
  int rc = 1;
  if (D % 4 == 0 && Vd % 4 == 0 && ld % 4 == 0 && state_stride % 4 == 0 && conv_off % 4 == 0 && al &&
      D <= 256 && Vd <= 256 && taps <= 4) {
    // few tokens: one each a warp; many: runs, so that a token's inputs are loaded once
    const int run = T <= 256 ? 1 : 8;
    updated = max_q_len == 1;
    const dim3 grid((T + run - 1) / run, (units + 3) / 4), block(128);
#define GF_GO(TAPS, NQ)                                                                            \
  if (taps == TAPS && D <= 128 * NQ && Vd <= 128 * NQ && rc == 1)                                  \
    rc = launch_kernel(delta_prepare_heads_kernel<TAPS, NQ>, grid, block, 0, st, proj, ld, a_off,  \
                       b_off, conv_w, dt_bias, A_log, state, seq_of_token, cu_seqlens, slot_ids,   \
                       dm, T, run, updated ? 1 : 0, qn, kn, v, g, beta);
    GF_GO(1, 1) GF_GO(2, 1) GF_GO(3, 1) GF_GO(4, 1)
    GF_GO(1, 2) GF_GO(2, 2) GF_GO(3, 2) GF_GO(4, 2)
#undef GF_GO
  } else {
    const dim3 grid(T, (units + kPrepareWarps - 1) / kPrepareWarps), block(kPrepareWarps * 32);
    rc = launch_kernel(delta_prepare_kernel<float, true>, grid, block, 0, st, proj, ld, b_off,
                       proj + a_off, conv_w, dt_bias, A_log, (const float*)state, seq_of_token,
                       cu_seqlens, slot_ids, dm, qn, kn, v, g, beta);
  }
  if (rc || taps == 1 || updated) return rc;
  return launch_kernel(delta_conv_state_kernel<float>, dim3((dm.channels + 127) / 128, B), dim3(128),
                       0, st, proj, ld, state, cu_seqlens, slot_ids, dm);
}

// fp32 words of scratch with which a step of `heads` heads goes eight tokens at a time: gf_delta_recurrence
// (one_decay 1), gf_decay_channels_chunked (0).
GF_EXPORT long long gf_delta_chunk_words(int T, int B, int heads, int D, int one_decay) {
  const long long chunks = (long long)(T / CT + B + 1) * heads;
  return one_decay ? chunks * kCoefs : chunks * (kCoefs + D) + 2ll * T * heads * D;
}

// Many (request, head, column) triples: whether T tokens of B requests take the kernel of portions of many tokens
// instead of four lanes a column, which give the same bits.  A request costs that kernel more before its first
// token (one block of up to four requests an SM), a token less.  Its time over that of four lanes on a B200, 8 to
// 512 requests of equal portions: 16 heads of 128 x 128, 2 tokens 1.3 to 1.75, 4 tokens 0.95 to 1.2, 6 tokens 0.84 to 0.95, 8 tokens
// 0.62 to 0.75, 16 tokens 0.5; with a decay a head 6 tokens 1.1, 8 tokens 0.79 to 0.95; 64 x 64, 16 tokens 1.0 to 1.26,
// 32 tokens 0.8 to 1.0, 64 tokens 0.7 to 0.9.
inline bool tree_pays(long long T, int B, int D, bool one_decay) {
  return D > 32 && T >= (long long)(D <= 64 ? 32 : one_decay ? 8 : 5) * B;
}

// one_decay: g is [T, H] (a decay a head), else [T, H, D].  scratch (gf_delta_chunk_words; null: token by
// token) is for steps with one decay a head; max_q_len: the longest portion (0: not known); singles: how many
// requests in front have one token.  *launches: kernels launched.
GF_EXPORT int gf_delta_recurrence(const float* qn, const float* kn, const float* v, const float* g,
                                  const float* beta, float* state, const int* cu_seqlens,
                                  const int* slot_ids, int B, int H, int G, int D, int Vd,
                                  int state_stride, float* o, int one_decay, float* scratch,
                                  int max_q_len, int T, int singles, int* launches, void* stream) {
  *launches = 0;
  if (B <= 0) return 0;
  *launches = 1;
  if (H % G) return -3;
  const DeltaDims dm = dims_of(H, G, D, Vd, 1, state_stride, 0);
  auto st = (cudaStream_t)stream;
  if (one_decay && scratch && D % 4 == 0 && Vd % 4 == 0 && D <= 256 && B <= 65535 && G <= 65535 &&
      (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)v | (uintptr_t)scratch) & 15) == 0) {
    const int chunks = (max_q_len + CT - 1) / CT;
    if (int rc = launch_kernel(delta_chunk_coef_kernel, dim3((chunks + 3) / 4, B, G), dim3(128), 0, st,
                               qn, kn, g, beta, cu_seqlens, dm, scratch))
      return rc;
    ++*launches;
    const ChunkArgs a{qn, kn, nullptr, nullptr, v, H * Vd, scratch, state, cu_seqlens, slot_ids, 0, H, o};
#define GF_GO(DPER, LANES)                                                                         \
  if (D <= DPER * LANES) return launch_chunks<DPER, LANES, HEADS>(B, dm, a, st);
    GF_GO(4, 8)
    GF_GO(8, 8)
    GF_GO(16, 8)             // (sixteen lanes of 8 rows: 348 us for a prompt that takes 317 so)
    GF_GO(16, 16)
#undef GF_GO
  }
  // few (request, head, column) triples: more lanes a column than four (see the kernels).  Which it is decides
  // the order of the sums, for all requests of the step
  const long long units = (long long)B * H * ((Vd + 31) / 32);
  const bool wide = units < 2 * 148;
  auto lanes = [&](int lp, int n) -> int {         // the first n requests, lp lanes a column
    const int threads = lp == 32 ? 256 : kRecurrenceThreads;
    const int cols = threads / lp;
    const dim3 grid(n * H, (Vd + cols - 1) / cols), block(threads);
#define GF_AS(DPER, LP, CHUNK, THREADS, ONE)                                                       \
  {                                                                                                \
    const size_t smem =                                                                            \
        (size_t)kStages * CHUNK * ((ONE ? 2 : 3) * LP * DPER + kMaxColumnsPerBlock + 4) *          \
        sizeof(float);                                                                             \
    return launch_kernel(delta_recurrence_kernel<DPER, LP, CHUNK, THREADS, ONE>, grid, block,      \
                         smem, st, qn, kn, v, g, beta, state, cu_seqlens, slot_ids, dm, o);        \
  }
#define GF_GO(DPER, LP, CHUNK, THREADS)                                                            \
  if (lp == LP && D <= LP * DPER) {                                                                \
    if (one_decay) GF_AS(DPER, LP, CHUNK, THREADS, true)                                           \
    GF_AS(DPER, LP, CHUNK, THREADS, false)                                                         \
  }
    GF_GO(4, 4, 8, kRecurrenceThreads)
    GF_GO(8, 4, 8, kRecurrenceThreads)
    GF_GO(16, 4, 8, kRecurrenceThreads)
    GF_GO(32, 4, 8, kRecurrenceThreads)
    GF_GO(64, 4, 4, kRecurrenceThreads)
    GF_GO(4, 16, 8, kRecurrenceThreads)
    GF_GO(4, 32, 8, 256)
    GF_GO(8, 32, 4, 256)
#undef GF_GO
#undef GF_AS
    return -3;
  };
  auto tree = [&](int first) -> int {              // the requests from number `first` on
    const int n = B - first;
    const int *cu = cu_seqlens + first, *slots = slot_ids + first;
    const int whole = Vd % 2 == 0 && state_stride % 2 == 0 && ((uintptr_t)state & 7) == 0;
#define GF_TREE(DPER, LP, ONE, CHAIN)                                                              \
  {                                                                                                \
    constexpr int cols = kTreeThreads / LP * 2;                                                    \
    constexpr size_t smem = (size_t)kStages * kTreeChunk *                                         \
                            ((ONE ? 2 : 3) * (LP * DPER + (CHAIN ? 16 : 0)) + kMaxColumnsPerBlock + 4) * \
                            sizeof(float);                                                         \
    const int ny = (Vd + cols - 1) / cols;                                                         \
    if (max_q_len == 1 || n == 1)                                                                  \
      return launch_kernel(delta_tree_kernel<DPER, LP, ONE, CHAIN>, dim3(n * H, ny),               \
                           dim3(kTreeThreads), smem, st, qn, kn, v, g, beta, state, cu, slots, dm, \
                           n, 0, whole, o);                                                        \
    /* the fewest requests a block with which every block has an SM of its own */                  \
    int groups = 1;                                                                                \
    while (groups < kTreeGroups && (long long)H * ny * ((n + groups - 1) / groups) > 148) groups *= 2; \
    const int nz = (n + groups - 1) / groups;                                                      \
    const size_t alone = 120 * 1024, all = smem * groups;                                          \
    static OncePerDevice attrs;                                                                    \
    if (int rc = attrs.run([&] {                                                                   \
          return cudaFuncSetAttribute(delta_tree_kernel<DPER, LP, ONE, CHAIN>,                     \
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);    \
        }))                                                                                        \
      return rc;                                                                                   \
    return launch_kernel_behind(delta_tree_kernel<DPER, LP, ONE, CHAIN>, dim3(nz * H, ny),         \
                                dim3(kTreeThreads * groups),                                       \
                                (long long)H * ny * nz <= 148 && all < alone ? alone : all, st,    \
                                qn, kn, v, g, beta, state, cu, slots, dm, n, n <= kTreeSorted,     \
                                whole, o);                                                         \
  }
    if (D <= 64) {
      if (one_decay && wide) GF_TREE(8, 8, true, false)
      if (one_decay) GF_TREE(4, 16, true, true)
      if (wide) GF_TREE(8, 8, false, false)
      GF_TREE(4, 16, false, true)
    }
    if (one_decay && wide) GF_TREE(8, 16, true, false)
    if (one_decay) GF_TREE(8, 16, true, true)
    if (wide) GF_TREE(8, 16, false, false)
    GF_TREE(8, 16, false, true)
#undef GF_TREE
  };
  if (wide) {
    // Key sizes up to 64: sixteen lanes a column (four rows each: the tree kernel's sums) start sooner, and with few
    // columns nothing waits for shared memory.  On a B200, us, tree kernel / sixteen lanes, 64 x 64: one request of 8
    // heads 1.16 at 1 token, 1.23 at 17, 1.04 at 100; 64 units 1.13 (17 tokens 1.15, 100 0.95); 128 units 0.86 at 1 token, 1.04
    // at 2, 1.06 at 15, 0.91 at 17, 0.69 at 100; 256 units 0.55 to 0.87.
    if (D <= 64 && !(units >= 192 || (units >= 128 && (max_q_len == 1 || T >= 16ll * B)))) return lanes(16, B);
    // Key sizes up to 128: while the blocks of a warp a column are few, it starts sooner, and the tree kernel's shorter
    // token pays from some 60 tokens on.  Tree kernel / a warp a column, on a B200, one request: 16 units, 128 x 128 1.16 at 1
    // token (3.9 us, 3.4), 1.27 at 5, 1.20 at 17, 1.04 at 60, 1.00 at 100, 0.91 at 1,201, 72 x 128 1.15, 1.10, 1.11, 0.99, 0.95,
    // 0.87; 20 units 1.15 at 1, 1.0 at 60; 24 and 28 units 0.8 to 1.2, by the columns; 32 units 0.7 to 0.9.
    const long long longest = max_q_len > 0 ? max_q_len : T;
    const bool warp = D > 128 || (D > 64 && units <= 20 && longest < 64);
    return warp ? lanes(32, B) : tree(0);
  }
  // (many requests of a token each are their states' bytes, which four lanes a column read in longer runs:
  // 16 requests of 16 heads of 128 x 128 19 us against 29)
  if (D > 128 || max_q_len == 1) return lanes(4, B);
  if (tree_pays(T, B, D, one_decay)) return tree(0);
  // a few portions behind many decoding requests: each on the kernel that it would have alone (16 heads of 128 x
  // 128, 127 single tokens and a portion of 64: 157 us, all on four lanes 204, all on the tree kernel 330; 255 and a
  // portion of 300: 386, 751 and 1,340)
  if (singles > 0 && singles < B && tree_pays((long long)T - singles, B - singles, D, one_decay)) {
    if (int rc = lanes(4, singles)) return rc;
    ++*launches;
    return tree(singles);
  }
  return lanes(4, B);
}

// A plain linear attention with a decay a key channel, S <- diag(g) S + k v^T, o = S^T q, eight tokens at a
// time.  Rows of q, k (G heads of D), v (H of Vd) and g (H of D) are ld_* floats apart; `heads` of the H
// from number `head0` on; scratch: gf_delta_chunk_words with one_decay 0; o [T, H, Vd].  Returns -6 for what it does not take (key sizes over
// 128, sizes or rows that are no multiples of four).
GF_EXPORT int gf_decay_channels_chunked(const float* q, int ld_q, const float* k, int ld_k, const float* v,
                                        int ld_v, const float* g, int ld_g, float* state, int state_stride,
                                        const int* cu_seqlens, const int* slot_ids, int T, int B, int H,
                                        int G, int D, int Vd, float* o, float* scratch, int max_q_len,
                                        int head0, int heads, void* stream) {
  if (B <= 0) return 0;
  if (H % G || D > 128 || D % 4 || Vd % 4 || ld_q % 4 || ld_k % 4 || ld_v % 4 || ld_g % 4 || B > 65535 ||
      H > 65535 || head0 < 0 || heads <= 0 || head0 + heads > H ||
      (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)g | (uintptr_t)scratch) & 15))
    return -6;
  const DeltaDims dm = dims_of(H, G, D, Vd, 1, state_stride, 0);
  auto st = (cudaStream_t)stream;
  const size_t chunks = (size_t)(T / CT + B + 1) * heads, HTD = (size_t)T * heads * D;
  float *total = scratch + chunks * kCoefs, *qg = total + chunks * D, *ke = qg + HTD;
  if (int rc = launch_kernel(linear_chunk_coef_kernel, dim3(((max_q_len + CT - 1) / CT + 3) / 4, B, heads),
                             dim3(128), 0, st, q, ld_q, k, ld_k, g, ld_g, cu_seqlens, dm, head0, heads,
                             scratch, total, qg, ke))
    return rc;
  const ChunkArgs a{qg, nullptr, ke, total, v, ld_v, scratch, state, cu_seqlens, slot_ids, head0, heads, o};
  if (D <= 32) return launch_chunks<4, 8, PLAIN>(B, dm, a, st);
  if (D <= 64) return launch_chunks<8, 8, PLAIN>(B, dm, a, st);
  return launch_chunks<16, 8, PLAIN>(B, dm, a, st);
}

GF_EXPORT int gf_delta_output(const float* o, const void* gate, int gate_ld, const float* w,
                              float eps, void* out, int T, int H, int Vd, int dtype, void* stream) {
  const int pairs = T * H;
  if (pairs <= 0) return 0;
  auto st = (cudaStream_t)stream;
  const dim3 grid((pairs + 3) / 4), block(128);
  if (dtype == GF_F32)
    return launch_kernel(delta_output_kernel<float>, grid, block, 0, st, o, (const float*)gate,
                         gate_ld, w, eps, (float*)out, pairs, H, Vd);
  return launch_kernel(delta_output_kernel<bf>, grid, block, 0, st, o, (const bf*)gate, gate_ld, w,
                       eps, (bf*)out, pairs, H, Vd);
}
