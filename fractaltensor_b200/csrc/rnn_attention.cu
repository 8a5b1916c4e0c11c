// Attention of the attention RNN (examples/rnn_attention/rnn_attention.py:52-70, attn_func):
//
//   scores_j = e_j @ encoder_proj + decoder @ decoder_proj      (one number per encoder position)
//   weights  = softmax over the encoder positions j
//   v        = sum_j weights_j * e_j
//
// for every sequence of the batch and every decoder step.  The decoder state itself,
// tanh(y_t @ W + v_{t-1} @ U + b), is a cell of the wavefront (csrc/cell_gemm.cu / cell_simt.cu);
// this file holds what surrounds it: the scores e_j @ encoder_proj, which do not depend on the
// decoder step and are computed once per call, and the softmax-weighted sums of the encoder rows.
//
// The decoder adds the same number to every score of a step, and a softmax does not change when all
// its scores move by one number: v_t is the softmax-weighted sum over e_j @ encoder_proj alone, one
// vector a sequence.  So the recurrent input of every decoder cell is known as soon as the encoder is
// done, and the decoder, a chain of Lt cells and Lt attention steps as written, is one launch that puts
// the vector of every sequence into the rows of its steps (attn_vector_kernel), one matrix product over
// all steps, and one launch that looks at the decoder's terms (attn_finish_kernel).  Only a term that is
// not finite does not cancel: it makes every weight of its step NaN, and in the chain every later step
// of the sequence.
//
// Layout: time-major padded batches, row (j, n) of `enc` at (j * N + n) * H.  Sequence n attends to
// encoder positions j < src_lens[n] (all Ls when src_lens is NULL).  L2-bound row work: len * H encoder
// elements a sequence in (for the scores by each of its H / 128 CTAs, and once for the sum), Lt * H out; then Lt * H
// decoder elements in.  With the scores in a launch of their own and the weights and sums anew for every step, the whole
// program (H 512, 64 sequences, 50 + 50 positions, bf16) took 155.8 us; as here 114.9 (with the encoder's scan as it was
// then, in both).
#include "../../include/ftb200.h"
#include "ptx.cuh"
#include "tmap.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace ftb {
namespace {

constexpr int kAttnThreads = 256;
constexpr int kAttnCols = 128;  // output columns of a CTA

template <typename T> __device__ __forceinline__ float ld_f32(const T* p);
template <> __device__ __forceinline__ float ld_f32<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ld_f32<__half>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float ld_f32<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void st_f32(T* p, float x);
template <> __device__ __forceinline__ void st_f32<float>(float* p, float x) { *p = x; }
template <> __device__ __forceinline__ void st_f32<__half>(__half* p, float x) { *p = __float2half_rn(x); }
template <> __device__ __forceinline__ void st_f32<__nv_bfloat16>(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// 16 bytes of a row as fp32 numbers.
template <typename T>
struct Piece {
  static constexpr int n = 16 / sizeof(T);
};
__device__ __forceinline__ void ld_piece(const float* p, float (&v)[4]) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
template <typename T>
__device__ __forceinline__ void ld_piece(const T* p, float (&v)[8]) {
  const uint4 x = *reinterpret_cast<const uint4*>(p);
  const T* e = reinterpret_cast<const T*>(&x);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = ld_f32<T>(e + i);
}

// The dot products of up to kDots rows, `stride` elements apart, with proj (of any alignment): a warp's work; every
// lane gets them.
constexpr int kDots = 4;
template <typename T>
__device__ __forceinline__ void row_dots(const T* rows, long long stride, int count, const T* proj, int H, int lane,
                                         float (&s)[kDots]) {
  constexpr int n = Piece<T>::n;
#pragma unroll
  for (int r = 0; r < kDots; ++r) s[r] = 0.f;
  for (int h = lane * n; h < H; h += 32 * n) {
    float p[n];
#pragma unroll
    for (int i = 0; i < n; ++i) p[i] = ld_f32<T>(proj + h + i);
#pragma unroll
    for (int r = 0; r < kDots; ++r) {
      if (r >= count) continue;
      float x[n];
      ld_piece(rows + r * stride + h, x);
#pragma unroll
      for (int i = 0; i < n; ++i) s[r] = fmaf(x[i], p[i], s[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < kDots; ++r) s[r] = warp_sum(s[r]);
}

__device__ __forceinline__ int source_len(const int* src_lens, int n, int Ls) {
  const int len = src_lens ? src_lens[n] : Ls;
  return len < 0 ? 0 : (len > Ls ? Ls : len);
}

// The attention vector of sequence blockIdx.x, columns 128 * blockIdx.y .., into the rows of all Lt steps; the scores
// into `scores` [Ls, N].  The CTAs of a sequence compute its len scores each for itself.  Latency: a chain of reads
// of the encoder's rows for the scores, two reductions over the CTA, and reads of the rows again (from L2) for the sum.
// The scores of positions past a sequence's length, which its vector does not need, are a CTA's own, behind the columns.
template <typename T>
__global__ void __launch_bounds__(kAttnThreads)
attn_vector_kernel(const T* __restrict__ enc, const T* __restrict__ enc_proj, const int* __restrict__ src_lens,
                   float* __restrict__ scores, T* __restrict__ out, int Lt, int Ls, int N, int H) {
  constexpr int kN = Piece<T>::n, kColGroups = kAttnCols / kN, kRowGroups = kAttnThreads / kColGroups;
  constexpr int kWarps = kAttnThreads / 32;
  extern __shared__ float s_w[];  // [Ls] scores, then weights
  __shared__ float s_red[kWarps];
  __shared__ float s_part[kRowGroups][kAttnCols];
  __shared__ __align__(16) T s_out[kAttnCols];
  const int n = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const long long step_elems = static_cast<long long>(N) * H;
  const T* mine = enc + static_cast<long long>(n) * H;
  grid_launch_dependents();
  grid_dependency_wait();
  const int len = source_len(src_lens, n, Ls);

  if (blockIdx.y * kAttnCols >= H) {
    for (int j0 = len + wid * kDots; j0 < Ls; j0 += kWarps * kDots) {
      float s[kDots];
      row_dots(mine + j0 * step_elems, step_elems, Ls - j0, enc_proj, H, lane, s);
#pragma unroll
      for (int r = 0; r < kDots; ++r)
        if (lane == r && j0 + r < Ls) scores[static_cast<long long>(j0 + r) * N + n] = s[r];
    }
    return;
  }
  float mx = -INFINITY;
  for (int j0 = wid * kDots; j0 < len; j0 += kWarps * kDots) {
    float s[kDots];
    row_dots(mine + j0 * step_elems, step_elems, len - j0, enc_proj, H, lane, s);
#pragma unroll
    for (int r = 0; r < kDots; ++r) {
      if (j0 + r >= len) continue;
      mx = fmaxf(mx, s[r]);
      if (lane == r) {
        s_w[j0 + r] = s[r];
        if (blockIdx.y == 0) scores[static_cast<long long>(j0 + r) * N + n] = s[r];
      }
    }
  }
  if (lane == 0) s_red[wid] = mx;
  __syncthreads();
  mx = s_red[0];
#pragma unroll
  for (int w = 1; w < kWarps; ++w) mx = fmaxf(mx, s_red[w]);
  __syncthreads();
  float sum = 0.f;
  for (int j = tid; j < len; j += kAttnThreads) {
    const float e = expf(s_w[j] - mx);
    s_w[j] = e;
    sum += e;
  }
  sum = warp_sum(sum);
  if (lane == 0) s_red[wid] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) sum += s_red[w];
  const float inv = len > 0 ? 1.f / sum : 0.f;

  // weighted sum: a thread takes 16 bytes of every kRowGroups-th row
  const int cg = tid % kColGroups, rg = tid / kColGroups, h = blockIdx.y * kAttnCols + cg * kN;
  float acc[kN];
#pragma unroll
  for (int i = 0; i < kN; ++i) acc[i] = 0.f;
  if (h < H) {
#pragma unroll 4
    for (int j = rg; j < len; j += kRowGroups) {
      float x[kN];
      ld_piece(mine + j * step_elems + h, x);
#pragma unroll
      for (int i = 0; i < kN; ++i) acc[i] = fmaf(s_w[j], x[i], acc[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < kN; ++i) s_part[rg][cg * kN + i] = acc[i];
  __syncthreads();
  if (tid < kAttnCols) {
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < kRowGroups; ++r) v += s_part[r][tid];
    st_f32<T>(s_out + tid, v * inv);
  }
  __syncthreads();
  if (h < H) {
    const uint4 v = *reinterpret_cast<const uint4*>(s_out + cg * kN);
    T* o = out + static_cast<long long>(n) * H + h;
    for (int t = rg; t < Lt; t += kRowGroups) *reinterpret_cast<uint4*>(o + t * step_elems) = v;
  }
}

// The decoder's terms dec_t . dec_proj of sequence blockIdx.x.  The largest score of a step is the largest of the
// encoder's scores plus the term; if that is not finite the step's vector is NaN, and so are the decoder states and
// vectors of the steps behind it.  (Encoder scores that are not finite are in every step's vector already.)
// Latency, 32 steps a round of a CTA: gridDim.y CTAs share the steps of a sequence where the sequences alone do not fill
// the device.  Each writes what follows from the steps it has looked at.  One that meets another's NaNs in `dec` finds a
// step behind that one's, and writes a part of the same.
// (H 512, bf16, 1 sequence, 8 + 4096 positions, the whole program: 412 us with one CTA a sequence, 63 so.)
template <typename T>
__global__ void __launch_bounds__(kAttnThreads)
attn_finish_kernel(T* __restrict__ dec, const T* __restrict__ dec_proj, const float* __restrict__ scores,
                   const int* __restrict__ src_lens, T* __restrict__ out, int Lt, int Ls, int N, int H) {
  constexpr int kWarps = kAttnThreads / 32;
  __shared__ int s_first;
  const int n = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const long long step_elems = static_cast<long long>(N) * H, row = static_cast<long long>(n) * H;
  if (tid == 0) s_first = Lt;
  grid_launch_dependents();
  grid_dependency_wait();
  __syncthreads();
  const int len = source_len(src_lens, n, Ls);
  if (len == 0) return;  // nothing to attend to: zeros
  float mx = -INFINITY;
  for (int j = lane; j < len; j += 32) mx = fmaxf(mx, scores[static_cast<long long>(j) * N + n]);
  mx = warp_max(mx);
  for (int t0 = (blockIdx.y * kWarps + wid) * kDots; t0 < Lt; t0 += gridDim.y * kWarps * kDots) {
    float c[kDots];
    row_dots(dec + t0 * step_elems + row, step_elems, Lt - t0, dec_proj, H, lane, c);
#pragma unroll
    for (int r = 0; r < kDots; ++r)
      if (lane == r && t0 + r < Lt && !isfinite(mx + c[r])) atomicMin(&s_first, t0 + r);
  }
  __syncthreads();
  const float nan = __int_as_float(0x7FFFFFFF);
  for (int t = s_first + wid; t < Lt; t += kWarps)
    for (int h = lane; h < H; h += 32) {
      if (t > s_first) st_f32<T>(dec + t * step_elems + row + h, nan);
      st_f32<T>(out + t * step_elems + row + h, nan);
    }
}

template <typename T>
int attn_vectors_t(const void* enc, const void* enc_proj, const int* src_lens, float* scores, void* out, int Lt, int Ls,
                   int N, int H, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  if (!ensure_dynamic_smem(attn_vector_kernel<T>, 48 * 1024, configured)) return FTB_ERR_LAUNCH;
  const cudaError_t err =
      launch_light(attn_vector_kernel<T>, dim3(N, (H + kAttnCols - 1) / kAttnCols + (src_lens != nullptr)), dim3(kAttnThreads),
                   static_cast<size_t>(Ls) * sizeof(float), stream, static_cast<const T*>(enc),
                   static_cast<const T*>(enc_proj), src_lens, scores, static_cast<T*>(out), Lt, Ls, N, H);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

template <typename T>
int attn_finish_t(void* dec, const void* dec_proj, const float* scores, const int* src_lens, void* out, int Lt, int Ls,
                  int N, int H, cudaStream_t stream) {
  // as many CTAs as there are rounds of steps, up to what is resident at once (8 of 256 threads an SM)
  constexpr int kRound = kAttnThreads / 32 * kDots;
  const int rounds = (Lt + kRound - 1) / kRound, room = (8 * current_sm_count() + N - 1) / N;
  const cudaError_t err =
      launch_light(attn_finish_kernel<T>, dim3(N, rounds < room ? rounds : room), dim3(kAttnThreads), 0, stream,
                   static_cast<T*>(dec), static_cast<const T*>(dec_proj), scores, src_lens, static_cast<T*>(out), Lt, Ls, N, H);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

}  // namespace

// Longest source sequence the attention takes: its scores sit in 48 KB of shared memory.
int rnn_attention_max_src_len() { return 48 * 1024 / static_cast<int>(sizeof(float)); }

// The attention vector of every sequence into its rows of out [Lt, N, H]; the encoder's scores into scores [Ls, N].
int launch_attn_vectors(int dtype, const void* enc, const void* enc_proj, const int* src_lens, float* scores, void* out,
                        int Lt, int Ls, int N, int H, cudaStream_t stream) {
  switch (dtype) {
    case FTB_F32: return attn_vectors_t<float>(enc, enc_proj, src_lens, scores, out, Lt, Ls, N, H, stream);
    case FTB_F16: return attn_vectors_t<__half>(enc, enc_proj, src_lens, scores, out, Lt, Ls, N, H, stream);
    default: return attn_vectors_t<__nv_bfloat16>(enc, enc_proj, src_lens, scores, out, Lt, Ls, N, H, stream);
  }
}

// What decoder terms that are not finite make of the vectors in `out` and the states in `dec`.
int launch_attn_finish(int dtype, void* dec, const void* dec_proj, const float* scores, const int* src_lens, void* out,
                       int Lt, int Ls, int N, int H, cudaStream_t stream) {
  switch (dtype) {
    case FTB_F32: return attn_finish_t<float>(dec, dec_proj, scores, src_lens, out, Lt, Ls, N, H, stream);
    case FTB_F16: return attn_finish_t<__half>(dec, dec_proj, scores, src_lens, out, Lt, Ls, N, H, stream);
    default: return attn_finish_t<__nv_bfloat16>(dec, dec_proj, scores, src_lens, out, Lt, Ls, N, H, stream);
  }
}

}  // namespace ftb
