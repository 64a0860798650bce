// One token (or none) of every request through the recurrences over per-request state S [H, D, Vd] (decode steps):
//
//   linear   S <- g S + (c k) v^T,                      o = S^T q + skip_h v
//   delta    S <- g S, u = beta (v - S^T k), S <- S + k u^T, o = S^T q      (= S'^T q + u (k . q), S' = g S)
//
// with a decay g a head or a key channel.  The work is the state: read once, written once.  The kernels
// that walk over many tokens (decay_state.cu, delta_rule.cu) give a lane a column, so that a row of S is
// read 32 bytes at a time by single loads, and set up stages for tokens that are not there.  Here a thread
// has four columns of D / (256 / lanes a row) rows: 16 loads of 16 bytes under way, whole rows at a time.
// Then one sum over the block (both of the delta rule's, S'^T k and S'^T q, at once).  fp32 throughout.
// Measured on a B200, 16 heads of 128 x 128: 32 requests 14.0 us (67 MB: 10.3 at 6.54 TB/s), 29.4 with a lane a
// column; 8 requests 7.1 and 9.7.  (Layers with the delta rule and channel decays stay with the kernel that
// walks over tokens, ops/delta.py: recurrence.)
#include "common.cuh"

namespace gf {

constexpr int kStepThreads = 256, kStepMaxD = 256;

struct StepArgs {
  const float *q, *k, *v, *g, *c, *skip, *beta;      // c, skip: null where there is none; beta: delta only
  float *state, *o;
  const int *cu_seqlens, *slot_ids;
  int ld_q, ld_k, ld_v, ld_g, ld_c, ld_o, gD;        // floats between two tokens' rows; gD: 1 or D
  int H, G, D, Vd, state_stride;
};

// CQ lanes share a row (four columns each); NR rows a thread.
template <int CQ, int NR, bool DELTA>
__global__ void __launch_bounds__(kStepThreads, NR <= 16 ? 2 : 1)
state_step_kernel(const StepArgs a) {
  constexpr int RG = kStepThreads / CQ;              // rows at a time
  __shared__ float qs[kStepMaxD], ks[kStepMaxD], gs[kStepMaxD];
  __shared__ __align__(16) float red[DELTA ? 2 : 1][RG][CQ * 4];
  const int b = blockIdx.z, h = blockIdx.y, D = a.D, Vd = a.Vd;
  const int cq = threadIdx.x % CQ, rg = threadIdx.x / CQ, lane = threadIdx.x & 31;
  const int col = blockIdx.x * CQ * 4 + 4 * cq;
  const bool live = col < Vd;
  pdl_trigger();
  pdl_wait();
  const size_t r = a.cu_seqlens[b];
  if (a.cu_seqlens[b + 1] == (int)r) return;         // a request without a token: no row, no change
  const int kvh = h / (a.H / a.G);
  float* S = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)h * D * Vd + col;
  float s[NR][4];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int d = rg + RG * i;
    s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
    if (live && d < D) Quad<float>::load(S + (size_t)d * Vd, s[i]);
  }
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (live) Quad<float>::fresh(a.v + r * a.ld_v + (size_t)h * Vd + col, v);
  for (int d = threadIdx.x; d < D; d += kStepThreads) {
    qs[d] = fresh(a.q + r * a.ld_q + (size_t)kvh * D + d);
    ks[d] = fresh(a.k + r * a.ld_k + (size_t)kvh * D + d);
    gs[d] = fresh(a.g + r * a.ld_g + (a.gD == 1 ? h : h * D + d));
  }
  __syncthreads();
  float dq[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (DELTA) {
    float dk[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int d = rg + RG * i;
      if (d < D) {
        const float gd = gs[d], kd = ks[d], qd = qs[d];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          s[i][x] *= gd;
          dk[x] = fmaf(s[i][x], kd, dk[x]);
          dq[x] = fmaf(s[i][x], qd, dq[x]);
        }
      }
    }
    Quad<float>::store(&red[0][rg][4 * cq], dk);
    Quad<float>::store(&red[DELTA ? 1 : 0][rg][4 * cq], dq);
    float kq = 0.f;                                  // every warp for itself
    for (int d = lane; d < D; d += 32) kq = fmaf(ks[d], qs[d], kq);
    kq = warp_sum(kq);
    __syncthreads();
    const float beta = fresh(a.beta + r * a.H + h);
    float u[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < RG; ++j) {
      float p[4];
      Quad<float>::load(&red[0][j][4 * cq], p);
#pragma unroll
      for (int x = 0; x < 4; ++x) u[x] += p[x];
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) u[x] = beta * (v[x] - u[x]);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int d = rg + RG * i;
      if (d < D) {
        const float kd = ks[d];
#pragma unroll
        for (int x = 0; x < 4; ++x) s[i][x] = fmaf(kd, u[x], s[i][x]);
      }
    }
    if (rg == 0 && live) {
      float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < RG; ++j) {
        float p[4];
        Quad<float>::load(&red[DELTA ? 1 : 0][j][4 * cq], p);
#pragma unroll
        for (int x = 0; x < 4; ++x) out[x] += p[x];
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) out[x] = fmaf(u[x], kq, out[x]);
      Quad<float>::store(a.o + r * a.ld_o + (size_t)h * Vd + col, out);
    }
  } else {
    const float c = a.c ? fresh(a.c + r * a.ld_c + h) : 1.f;
    float cv[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) cv[x] = c * v[x];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int d = rg + RG * i;
      if (d < D) {
        const float gd = gs[d], kd = ks[d], qd = qs[d];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          s[i][x] = fmaf(gd, s[i][x], kd * cv[x]);
          dq[x] = fmaf(s[i][x], qd, dq[x]);
        }
      }
    }
    Quad<float>::store(&red[0][rg][4 * cq], dq);
    __syncthreads();
    if (rg == 0 && live) {
      const float sk = a.skip ? a.skip[h] : 0.f;
      float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < RG; ++j) {
        float p[4];
        Quad<float>::load(&red[0][j][4 * cq], p);
#pragma unroll
        for (int x = 0; x < 4; ++x) out[x] += p[x];
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) out[x] = fmaf(sk, v[x], out[x]);
      Quad<float>::store(a.o + r * a.ld_o + (size_t)h * Vd + col, out);
    }
  }
  if (live)
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int d = rg + RG * i;
      if (d < D) Quad<float>::store(S + (size_t)d * Vd, s[i]);
    }
}

template <bool DELTA> int start_step(const StepArgs& a, int B, cudaStream_t st) {
#define GF_GO(CQ, NR)                                                                                  \
  if ((a.Vd <= CQ * 4 || CQ == 32) && a.D <= NR * (kStepThreads / CQ))                                 \
    return launch_kernel(state_step_kernel<CQ, NR, DELTA>, dim3((a.Vd + CQ * 4 - 1) / (CQ * 4), a.H, B), \
                         dim3(kStepThreads), 0, st, a);
  GF_GO(8, 2) GF_GO(8, 4) GF_GO(8, 8)                // values of up to 32, keys of up to 64, 128, 256
  GF_GO(16, 4) GF_GO(16, 8) GF_GO(16, 16)            // of up to 64
  GF_GO(32, 8) GF_GO(32, 16) GF_GO(32, 32)           // of up to 128 and wider
#undef GF_GO
  return -6;
}

}  // namespace gf

using namespace gf;

GF_DEFINE_PDL_SWITCH

// Rows of q and k: G heads of D; v and o: H of Vd; g: H (gD 1) or H of D (gD D); c: H; beta [B, H] by token
// (null: the linear form, which may have c and skip).  Every request of the step has one token, at row
// cu_seqlens[b], or none (cu_seqlens[b + 1] == cu_seqlens[b]).  Returns -6 for what it does not take (keys over 256, values, rows, slots or addresses that
// are no multiples of four floats).
GF_EXPORT int gf_state_step(const float* q, int ld_q, const float* k, int ld_k, const float* v, int ld_v,
                            const float* g, int ld_g, int gD, const float* c, int ld_c, const float* skip,
                            const float* beta, float* state, int state_stride, const int* cu_seqlens,
                            const int* slot_ids, int B, int H, int G, int D, int Vd, float* o, int ld_o,
                            void* stream) {
  if (B <= 0) return 0;
  if (G <= 0 || H % G || D <= 0 || D > kStepMaxD || Vd <= 0 || Vd % 4 || state_stride % 4 || ld_v % 4 ||
      ld_o % 4 || (gD != 1 && gD != D) || B > 65535 || H > 65535 ||
      (((uintptr_t)state | (uintptr_t)v | (uintptr_t)o) & 15))
    return -6;
  const StepArgs a{q, k, v, g, c, skip, beta, state, o, cu_seqlens, slot_ids, ld_q, ld_k, ld_v, ld_g,
                   ld_c, ld_o, gD, H, G, D, Vd, state_stride};
  return beta ? start_step<true>(a, B, (cudaStream_t)stream) : start_step<false>(a, B, (cudaStream_t)stream);
}
