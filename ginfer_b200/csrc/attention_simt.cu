// Paged grouped-query attention with plain fp32 arithmetic: the kernel of the 32-bit path, and the
// fall-back of the bf16 path for head sizes the tensor-core kernels do not take.
//
// A block owns one (token, query head).  The token's absolute position p decides what it sees:
// keys lo..p with lo = first_visible_key(p, window) (a sliding window, chunks, or everything).
// Keys have hd channels, values vd (the two may differ).  Keys are visited in groups of 32 starting
// at lo; warp w takes groups w, w + 8, ... in order and the warps' results are put together in order,
// so a row's result depends only on (lo, p) and the cache contents, never on how the step was cut or
// what else is in the batch.  Running maximum, sum and the output accumulator are fp32.  Two optional
// shapings of a score s = q.k * scale, in this order: a soft cap (s <- cap * tanh(s / cap)) and a
// distance bias a head (s <- s - slope_n * (p - c)).  A sink (a score without a key and a value) may
// enter the softmax's denominator.
//
// What bounds it is the latency of the cache's rows with few warps at work (a decode step of three
// requests has 36 heads): eight warps a head, and every load of a group independent of the others.
// Scores: eight lanes a key, each 16 bytes of every 128 (hd 128: 16 loads a lane in flight); values: a
// lane owns four channels, a key's row is one load of the warp, eight of them in flight.  3 requests of
// up to 106 keys, 12 heads of 128, fp32, on a B200: 12.5 us, and 128 us with a warp a head that read
// a channel of 32 keys at a time; 164 prompt tokens 38 us, 128 before.
#include "common.cuh"

namespace gf {

constexpr int kMaxHeadDim = 256;
constexpr int kWarps = 8;

// VEC channels as one access: 4, or 1 for sizes and addresses that are no multiples of four elements; from L2
// (the kernel ahead has just rotated q and written this step's keys and values).
template <typename T, int VEC> __device__ __forceinline__ void load_channels(const T* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) Quad<T>::fresh(p, v);
  else v[0] = fresh(p);
}

// QN, VN: steps of eight lanes over a key's channels, of a warp over a value's.
template <typename T, int VEC, int QN, int VN>
__global__ void __launch_bounds__(kWarps * 32, QN * VEC <= 16 ? 2 : 1)
paged_attention_simt_kernel(
    const T* __restrict__ q, int q_row_stride, const T* __restrict__ kpages,
    const T* __restrict__ vpages, const int* __restrict__ block_table, int table_stride,
    const int* __restrict__ seq_of_token, const int* __restrict__ positions, T* __restrict__ out,
    int nh, int nkv, int hd, int vd, int page_size, int window, float scale,
    float softcap, const float* __restrict__ slopes, const Sink sink) {
  __shared__ float part[kWarps][VN * 32 * VEC];
  __shared__ float part_m[kWarps], part_l[kWarps];
  constexpr int QS = 8 * VEC, VS = 32 * VEC;              // channels of eight lanes, of a warp
  constexpr int KB = QN * VEC <= 16 ? 4 : QN * VEC <= 32 ? 2 : 1;   // keys a lane has under way
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & 7, quarter = lane >> 3;
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x / nh, n = blockIdx.x - t * nh;
  const int kvh = n / (nh / nkv);
  const int b = seq_of_token[t];
  const int p = positions[t];
  const int lo = first_visible_key(p, window);
  const float slope = slopes ? slopes[n] : 0.f;
  const int* tbl = block_table + (size_t)b * table_stride;
  const T* qrow = q + (size_t)t * q_row_stride + (size_t)n * hd;
  float qv[QN][VEC];
#pragma unroll
  for (int i = 0; i < QN; ++i) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) qv[i][e] = 0.f;
    const int d = i * QS + sub * VEC;
    if (d < hd) load_channels<T, VEC>(qrow + d, qv[i]);
  }

  float acc[VN][VEC];
#pragma unroll
  for (int i = 0; i < VN; ++i)
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[i][e] = 0.f;
  float m = -INFINITY, l = 0.f;
  const size_t tok_stride = (size_t)nkv * hd, vtok_stride = (size_t)nkv * vd;
  const T* kbase = kpages + (size_t)kvh * hd;
  const T* vbase = vpages + (size_t)kvh * vd;

  for (int c0 = lo + 32 * warp; c0 <= p; c0 += 32 * kWarps) {
    const int c = c0 + lane, nvalid = min(32, p - c0 + 1);
    const bool valid = lane < nvalid;
    const int slot = valid ? tbl[c / page_size] * page_size + c % page_size : 0;
    float s = 0.f;
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += KB) {                  // KB x four keys at a time, their loads first
      float kv[KB][QN][VEC];
#pragma unroll
      for (int j = 0; j < KB; ++j) {
        const int key = 4 * (j0 + j) + quarter;
        const int sj = __shfl_sync(0xffffffffu, slot, key);
        const T* krow = kbase + (size_t)sj * tok_stride + sub * VEC;
#pragma unroll
        for (int i = 0; i < QN; ++i) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) kv[j][i][e] = 0.f;
          if (key < nvalid && i * QS + sub * VEC < hd) load_channels<T, VEC>(krow + i * QS, kv[j][i]);
        }
      }
#pragma unroll
      for (int j = 0; j < KB; ++j) {
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < QN; ++i)
#pragma unroll
          for (int e = 0; e < VEC; ++e) dot = fmaf(qv[i][e], kv[j][i][e], dot);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float mine = __shfl_sync(0xffffffffu, dot, (lane & 3) * 8);
        if ((lane >> 2) == j0 + j) s = mine;              // lane = key from here on
      }
    }
    s *= scale;
    if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    s -= slope * (float)(p - c);
    if (!valid) s = -INFINITY;
    const float m_new = fmaxf(m, warp_max(s));
    // a group of scores of -inf adds nothing (the reference maximum is then any finite one)
    const float ref = m_new == -INFINITY ? 0.f : m_new;
    const float pexp = expf(s - ref);
    const float corr = expf(m - ref);                     // m = -inf on the first group: corr = 0
    l = l * corr + warp_sum(pexp);
#pragma unroll
    for (int i = 0; i < VN; ++i)
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[i][e] *= corr;
    for (int j0 = 0; j0 < nvalid; j0 += 8) {              // eight values at a time, their loads first
      float v[8][VN][VEC];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int sj = __shfl_sync(0xffffffffu, slot, j0 + j);
        const T* vrow = vbase + (size_t)sj * vtok_stride + lane * VEC;
#pragma unroll
        for (int i = 0; i < VN; ++i) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) v[j][i][e] = 0.f;
          if (j0 + j < nvalid && i * VS + lane * VEC < vd) load_channels<T, VEC>(vrow + i * VS, v[j][i]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float pj = __shfl_sync(0xffffffffu, pexp, j0 + j);   // 0 past the last key
#pragma unroll
        for (int i = 0; i < VN; ++i)
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[i][e] = fmaf(pj, v[j][i][e], acc[i][e]);
      }
    }
    m = m_new;
  }
  if (lane == 0) part_m[warp] = m, part_l[warp] = l;
#pragma unroll
  for (int i = 0; i < VN; ++i)
#pragma unroll
    for (int e = 0; e < VEC; ++e) part[warp][i * VS + lane * VEC + e] = acc[i][e];
  __syncthreads();
  float top = part_m[0];                                  // warp 0 has a key: finite
#pragma unroll
  for (int w = 1; w < kWarps; ++w) top = fmaxf(top, part_m[w]);
  float f[kWarps], sum = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    f[w] = expf(part_m[w] - top);                         // no group: exp(-inf) = 0
    sum = fmaf(part_l[w], f[w], sum);
  }
  const float inv = 1.f / (sum + expf(sink.at(n) - top)); // no sink: exp(-inf) = 0
  T* orow = out + ((size_t)t * nh + n) * vd;
  for (int d = threadIdx.x; d < vd; d += kWarps * 32) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v = fmaf(part[w][d], f[w], v);
    orow[d] = from_f32<T>(v * inv);
  }
}

template <typename T, int VEC, int QN, int VN, typename... Args>
int start_simt(int blocks, cudaStream_t st, Args... args) {
  return launch_kernel(paged_attention_simt_kernel<T, VEC, QN, VN>, dim3(blocks), dim3(kWarps * 32), 0, st,
                       args...);
}

}  // namespace gf

using namespace gf;

GF_DEFINE_PDL_SWITCH

// q: rows of q_row_stride elements whose first nh*hd hold the query heads.  kpages/vpages:
// [num_pages, page_size, nkv, hd] and [.., nkv, vd].  out: [T, nh, vd] packed.  window: the mask as
// first_visible_key() reads it.  softcap <= 0: no cap; slopes: nh fp32 slopes or null; sink: the
// sink's score, -inf for none; sinks: nh fp32 scores, one a head, or null.  Returns -3 for head sizes
// it refuses.
GF_EXPORT int gf_paged_attention_simt(const void* q, int q_row_stride, const void* kpages,
                                      const void* vpages, const int* block_table, int table_stride,
                                      const int* seq_of_token, const int* positions, void* out,
                                      int T, int nh, int nkv, int hd, int vd, int page_size,
                                      int window, float scale, float softcap, const float* slopes,
                                      float sink, const float* sinks, int dtype, void* stream) {
  if (T <= 0) return 0;
  if (hd > kMaxHeadDim || hd <= 0 || vd > kMaxHeadDim || vd <= 0 || nh % nkv) return -3;
  auto st = (cudaStream_t)stream;
  const bool four = hd % 4 == 0 && vd % 4 == 0 && q_row_stride % 4 == 0;
  const Sink si{sink, sinks};
  // sizes up to 128 in multiples of four, as models have them; the larger and the odd ones
#define GF_GO(E, VEC, QN, VN)                                                                             \
  return start_simt<E, VEC, QN, VN>(T * nh, st, (const E*)q, q_row_stride, (const E*)kpages,              \
                                    (const E*)vpages, block_table, table_stride, seq_of_token, positions, \
                                    (E*)out, nh, nkv, hd, vd, page_size, window, scale, softcap, slopes, si)
#define GF_GO_TYPE(E)                                                                                     \
  {                                                                                                       \
    const bool vec = four && ((uintptr_t)q | (uintptr_t)kpages | (uintptr_t)vpages) % (4 * sizeof(E)) == 0; \
    if (vec && hd <= 128 && vd <= 128) GF_GO(E, 4, 4, 1);                                                 \
    if (vec) GF_GO(E, 4, 8, 2);                                                                           \
    GF_GO(E, 1, 32, 8);                                                                                   \
  }
  if (dtype == GF_F32) GF_GO_TYPE(float)
  GF_GO_TYPE(__nv_bfloat16)
#undef GF_GO_TYPE
#undef GF_GO
}
