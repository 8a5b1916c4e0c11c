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
// its scores move by one number: v_t is the softmax-weighted sum over e_j @ encoder_proj alone.  So
// the recurrent input of every decoder cell is known as soon as the encoder is done, and the
// decoder, a chain of Lt cells and Lt attention steps as written, runs as one matrix product over all
// steps followed by one launch of the attention over all steps (ftb_rnn_attention_fwd).  Only a number that
// is not finite does not cancel: it makes every weight of its step NaN, and in the chain every later step
// of the sequence.  carry_nan_kernel, one warp a sequence behind the attention, does that (2 us of the call).
//
// Layout: time-major padded batches, row (j, n) of `enc` at (j * N + n) * H.  Sequence n attends to
// encoder positions j < src_lens[n] (all Ls when src_lens is NULL).  L2-bound row work: per
// decoder step and sequence the kernel reads len * H encoder elements (they stay in L2 across the
// steps) and writes H.
#include "../../include/ftb200.h"
#include "ptx.cuh"
#include "tmap.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace ftb {
namespace {

constexpr int kStepThreads = 128;  // one output column per thread
constexpr int kCarryThreads = 128;

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

// scores[r] = rows[r, :] . proj for r < n_rows: one warp per row.
template <typename T>
__global__ void __launch_bounds__(256)
row_dot_kernel(const T* __restrict__ rows, const T* __restrict__ proj, float* __restrict__ scores, long long n_rows,
               int H) {
  const int lane = threadIdx.x & 31;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  grid_launch_dependents();
  grid_dependency_wait();  // the encoder's last level wrote the rows
  for (long long r = warp; r < n_rows; r += n_warps) {
    float s = 0.f;
    for (int h = lane; h < H; h += 32) s = fmaf(ld_f32<T>(rows + r * H + h), ld_f32<T>(proj + h), s);
    s = warp_sum(s);
    if (lane == 0) scores[r] = s;
  }
}

// Attention vectors.  grid = (N, ceil(H / 128), steps); CTA (n, cb, t) computes columns cb * 128 .. of
// v_t for sequence n from the decoder states dec [Lt, N, H] of its step.  dec == nullptr: the scores
// of the encoder alone, and the one result goes to the rows of `copies` steps (the recurrent inputs of
// the decoder cells).  Every CTA of a sequence recomputes the len weights (a dot product over H and a
// softmax over len numbers: small next to the len x 128 weighted sum).
template <typename T>
__global__ void __launch_bounds__(kStepThreads)
attn_step_kernel(const T* __restrict__ enc, const float* __restrict__ enc_scores, const T* __restrict__ dec,
                 const T* __restrict__ dec_proj, const int* __restrict__ src_lens, T* __restrict__ out, int copies,
                 int Ls, int N, int H) {
  extern __shared__ float s_w[];  // [Ls] scores, then weights
  __shared__ float s_red[kStepThreads / 32];
  const int n = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const long long step_elems = static_cast<long long>(N) * H;
  const T* dec_t = dec == nullptr ? nullptr : dec + blockIdx.z * step_elems + static_cast<long long>(n) * H;
  grid_launch_dependents();
  grid_dependency_wait();
  int len = src_lens ? src_lens[n] : Ls;
  len = len < 0 ? 0 : (len > Ls ? Ls : len);

  // c = decoder . decoder_proj
  float part = 0.f;
  if (dec_t != nullptr)
    for (int h = tid; h < H; h += kStepThreads) part = fmaf(ld_f32<T>(dec_t + h), ld_f32<T>(dec_proj + h), part);
  part = warp_sum(part);
  if (lane == 0) s_red[wid] = part;
  __syncthreads();
  float c = 0.f;
#pragma unroll
  for (int w = 0; w < kStepThreads / 32; ++w) c += s_red[w];
  __syncthreads();

  // scores and their maximum
  float mx = -INFINITY;
  for (int j = tid; j < len; j += kStepThreads) {
    const float s = enc_scores[static_cast<long long>(j) * N + n] + c;
    s_w[j] = s;
    mx = fmaxf(mx, s);
  }
  mx = warp_max(mx);
  if (lane == 0) s_red[wid] = mx;
  __syncthreads();
  mx = s_red[0];
#pragma unroll
  for (int w = 1; w < kStepThreads / 32; ++w) mx = fmaxf(mx, s_red[w]);
  __syncthreads();
  float sum = 0.f;
  for (int j = tid; j < len; j += kStepThreads) {
    const float e = expf(s_w[j] - mx);
    s_w[j] = e;
    sum += e;
  }
  sum = warp_sum(sum);
  if (lane == 0) s_red[wid] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int w = 0; w < kStepThreads / 32; ++w) sum += s_red[w];
  const float inv = len > 0 ? 1.f / sum : 0.f;

  // weighted sum of the encoder rows, one column per thread, four rows in flight
  const int h = blockIdx.y * kStepThreads + tid;
  if (h >= H) return;
  const T* col = enc + static_cast<long long>(n) * H + h;
  float acc = 0.f;
  int j = 0;
  for (; j + 4 <= len; j += 4) {
    const float e0 = ld_f32<T>(col + (j + 0) * step_elems), e1 = ld_f32<T>(col + (j + 1) * step_elems);
    const float e2 = ld_f32<T>(col + (j + 2) * step_elems), e3 = ld_f32<T>(col + (j + 3) * step_elems);
    acc = fmaf(s_w[j], e0, acc);
    acc = fmaf(s_w[j + 1], e1, acc);
    acc = fmaf(s_w[j + 2], e2, acc);
    acc = fmaf(s_w[j + 3], e3, acc);
  }
  for (; j < len; ++j) acc = fmaf(s_w[j], ld_f32<T>(col + j * step_elems), acc);
  T* o = out + blockIdx.z * step_elems + static_cast<long long>(n) * H + h;
  for (int k = 0; k < copies; ++k) st_f32<T>(o + k * step_elems, acc * inv);
}

// Where step t of a sequence has NaN for its vector, so have the steps behind it and their decoder states.
// (Encoder states are at most 1 and weights too: a vector is finite or NaN, and NaN weights make all of its
// columns NaN.  A NaN encoder state alone is in every step's vector already.)
template <typename T>
__global__ void __launch_bounds__(kCarryThreads)
carry_nan_kernel(T* __restrict__ dec, T* __restrict__ out, int Lt, int N, int H) {
  const int n = blockIdx.x * (kCarryThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  grid_launch_dependents();
  grid_dependency_wait();
  if (n >= N) return;
  const long long step_elems = static_cast<long long>(N) * H, row = static_cast<long long>(n) * H;
  int first = Lt;
  for (int t0 = 0; t0 < Lt && first == Lt; t0 += 32) {
    const int t = t0 + lane;
    const bool bad = t < Lt && isnan(ld_f32<T>(out + t * step_elems + row));
    const unsigned who = __ballot_sync(0xffffffffu, bad);
    if (who != 0) first = t0 + __ffs(who) - 1;
  }
  const float nan = __int_as_float(0x7FFFFFFF);
  for (int t = first + 1; t < Lt; ++t)
    for (int h = lane; h < H; h += 32) {
      st_f32<T>(dec + t * step_elems + row + h, nan);
      st_f32<T>(out + t * step_elems + row + h, nan);
    }
}

template <typename T>
int carry_nan_t(void* dec, void* out, int Lt, int N, int H, cudaStream_t stream) {
  constexpr int kRows = kCarryThreads / 32;
  const cudaError_t err = launch_light(carry_nan_kernel<T>, dim3((N + kRows - 1) / kRows), dim3(kCarryThreads), 0, stream,
                                       static_cast<T*>(dec), static_cast<T*>(out), Lt, N, H);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

template <typename T>
int enc_scores_t(const void* enc, const void* proj, float* scores, long long n_rows, int H, cudaStream_t stream) {
  const long long ctas = (n_rows + 7) / 8;
  const long long full = static_cast<long long>(current_sm_count()) * 8;
  const int grid = static_cast<int>(ctas < full ? ctas : full);
  const cudaError_t err = launch_light(row_dot_kernel<T>, dim3(grid), dim3(256), 0, stream, static_cast<const T*>(enc),
                                           static_cast<const T*>(proj), scores, n_rows, H);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

template <typename T>
int attn_steps_t(const void* enc, const float* enc_scores, const void* dec, const void* dec_proj, const int* src_lens,
                 void* out, int steps, int Ls, int N, int H, cudaStream_t stream) {
  const dim3 grid(N, (H + kStepThreads - 1) / kStepThreads, dec == nullptr ? 1 : steps);
  const cudaError_t err = launch_light(attn_step_kernel<T>, grid, dim3(kStepThreads), static_cast<size_t>(Ls) * sizeof(float),
                                           stream, static_cast<const T*>(enc), enc_scores, static_cast<const T*>(dec),
                                           static_cast<const T*>(dec_proj), src_lens, static_cast<T*>(out),
                                           dec == nullptr ? steps : 1, Ls, N, H);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

}  // namespace

// Longest source sequence the step kernel takes: its scores sit in 48 KB of shared memory.
int rnn_attention_max_src_len() { return 48 * 1024 / static_cast<int>(sizeof(float)); }

int launch_enc_scores(int dtype, const void* enc, const void* proj, float* scores, long long n_rows, int H,
                      cudaStream_t stream) {
  switch (dtype) {
    case FTB_F32: return enc_scores_t<float>(enc, proj, scores, n_rows, H, stream);
    case FTB_F16: return enc_scores_t<__half>(enc, proj, scores, n_rows, H, stream);
    default: return enc_scores_t<__nv_bfloat16>(enc, proj, scores, n_rows, H, stream);
  }
}

int launch_carry_nan(int dtype, void* dec, void* out, int Lt, int N, int H, cudaStream_t stream) {
  switch (dtype) {
    case FTB_F32: return carry_nan_t<float>(dec, out, Lt, N, H, stream);
    case FTB_F16: return carry_nan_t<__half>(dec, out, Lt, N, H, stream);
    default: return carry_nan_t<__nv_bfloat16>(dec, out, Lt, N, H, stream);
  }
}

// The attention vectors of `steps` decoder steps (at most 65535) into out [steps, N, H]; dec == nullptr:
// without a decoder term, the same vectors in the rows of every step.
int launch_attn_steps(int dtype, const void* enc, const float* enc_scores, const void* dec, const void* dec_proj,
                      const int* src_lens, void* out, int steps, int Ls, int N, int H, cudaStream_t stream) {
  switch (dtype) {
    case FTB_F32: return attn_steps_t<float>(enc, enc_scores, dec, dec_proj, src_lens, out, steps, Ls, N, H, stream);
    case FTB_F16: return attn_steps_t<__half>(enc, enc_scores, dec, dec_proj, src_lens, out, steps, Ls, N, H, stream);
    default: return attn_steps_t<__nv_bfloat16>(enc, enc_scores, dec, dec_proj, src_lens, out, steps, Ls, N, H, stream);
  }
}

}  // namespace ftb
