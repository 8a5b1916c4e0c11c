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
// For 16-bit states of up to 512 units attn_decode_kernel does all of this, the product with U and the cells in one launch.
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
    // (16-bit only: for fp32 the branch costs more than three loads from L1, H 64, 1 sequence, 8 + 4096 positions 78.0 us without it, 80.0)
    if (sizeof(T) == 2 && (reinterpret_cast<uintptr_t>(proj) & 15) == 0) {
      ld_piece(proj + h, p);
    } else {
#pragma unroll
      for (int i = 0; i < n; ++i) p[i] = ld_f32<T>(proj + h + i);
    }
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

// All that follows the encoder's scan in one launch, where the decoder's input halves y_t W (fp32, `pre` [Lt, N, H]) are there
// already: scores, weights and vector of a sequence, the product of the vector with U, the decoder states of all steps and
// their terms.  A cluster of H / 128 CTAs takes two sequences, a CTA 128 columns of both: U's 128 rows (128 KB at H 512) are
// then read once for the two, which with one sequence a cluster would be 32 MB through L2 for 64.  A warp's score rows are
// shared by the cluster; scores, vectors and partial terms go between its CTAs through shared memory.
// Latency: what the later stages read (the rows for the sum, U, the input halves) depends on no earlier stage and is requested
// behind the score rows; what is left is a trip to L2 and three exchanges over the cluster.  H 512, 64 sequences, 50 + 50 positions, bf16, after
// the scan: 12.5 + 10.7 + 9.2 us as three launches (vector, cells, finish), 15 so, and the product in front of the scan 2 us longer;
// the whole program 105.5 us before, 94.2 so.  (U by 128 row copies of one warp: 99.4; its rows into registers: 98.9.)
constexpr int kDecThreads = 512, kDecWarps = kDecThreads / 64;  // of a sequence
constexpr int kDecMaxH = 512;
constexpr int kDecMaxSource = 256, kDecMaxSteps = 128;  // source positions, target steps
constexpr int kDecAhead = 8;       // steps of a warp, and rows of the sum of a thread over 2, requested ahead

__device__ __forceinline__ void st_cluster_f32(float* p, uint32_t rank, float x) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(smem_u32(p), rank)), "f"(x) : "memory");
}
template <typename T>
__device__ __forceinline__ void st_cluster_16(T* p, uint32_t rank, T x) {
  asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(map_to_cta(smem_u32(p), rank)),
               "h"(*reinterpret_cast<const unsigned short*>(&x)) : "memory");
}
// D += A B of 16 x 8 x 16, A rows of 16-bit numbers, fp32 sums.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, __half) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, __nv_bfloat16) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <typename T>
__global__ void __launch_bounds__(kDecThreads)
attn_decode_kernel(const T* __restrict__ enc, const T* __restrict__ enc_proj, const int* __restrict__ src_lens,
                   float* __restrict__ scores, const float* __restrict__ pre, const T* __restrict__ U, int ldu,
                   const float* __restrict__ bias, const T* __restrict__ dec_proj, T* __restrict__ dec, T* __restrict__ out,
                   int Lt, int Ls, int N, int H, int* __restrict__ status) {
  constexpr int kN = 8, kColGroups = kAttnCols / kN, kRowGroups = kDecThreads / 2 / kColGroups;
  constexpr int kMaxCtas = kDecMaxH / kAttnCols;
  __shared__ float s_score[2][kDecMaxSource], s_w[2][kDecMaxSource];
  __shared__ float s_term[kMaxCtas][2][kDecMaxSteps];  // the CTAs' parts of the decoder's terms
  __shared__ float s_part[2][kRowGroups][kAttnCols];
  __shared__ __align__(16) T s_v[2][kDecMaxH];
  __shared__ __align__(16) float s_z[2][2][kAttnCols];  // [half of K][sequence]: v . U
  __shared__ uint64_t u_full;
  __shared__ int s_first[2], s_abort;
  extern __shared__ __align__(16) unsigned char s_u_raw[];  // this CTA's 128 rows of U, 16 bytes between them
  T* s_u = reinterpret_cast<T*>(s_u_raw);
  const int u_stride = H + 8;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, seq = wid / kDecWarps, w = wid % kDecWarps, gt = tid & 255;
  const uint32_t rank = cluster_ctarank(), ctas = H / kAttnCols;
  const int n = 2 * (blockIdx.x / ctas) + seq, col0 = rank * kAttnCols;
  const bool mine = n < N;
  const long long step_elems = static_cast<long long>(N) * H, row = static_cast<long long>(n) * H;
  const auto group_sync = [&] { asm volatile("bar.sync %0, 256;" ::"r"(1 + seq) : "memory"); };
  if (gt == 0) s_first[seq] = Lt;
  if (tid == 0) {
    mbar_init(&u_full, 1);
    s_abort = 0;
    fence_barrier_init();
    mbar_arrive_expect_tx(&u_full, kAttnCols * H * 2);
  }
  grid_launch_dependents();
  cluster_sync_all();  // nobody stores into a CTA that has not started; u_full is set up
  grid_dependency_wait();
  const int len = mine ? source_len(src_lens, n, Ls) : 0;

  // scores of all source positions, rows dealt to the warps of the cluster
  if (mine)
    for (int j0 = (rank * kDecWarps + w) * kDots; j0 < Ls; j0 += ctas * kDecWarps * kDots) {
      float s[kDots];
      row_dots(enc + row + j0 * step_elems, step_elems, Ls - j0, enc_proj, H, lane, s);
#pragma unroll
      for (int r = 0; r < kDots; ++r)
        if (lane == r && j0 + r < Ls) {
          scores[static_cast<long long>(j0 + r) * N + n] = s[r];
          for (uint32_t k = 0; k < ctas; ++k) st_cluster_f32(&s_score[seq][j0 + r], k, s[r]);
        }
    }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // What later stages read does not depend on the scores: on its way while they come together.  (A copy takes its warp some
  // 60 cycles: every warp issues its share.)
  if (lane < kAttnCols / (2 * kDecWarps)) {
    const int i = wid * (kAttnCols / (2 * kDecWarps)) + lane;
    bulk_load_1d(s_u + i * u_stride, U + static_cast<long long>(col0 + i) * ldu, H * 2, &u_full);
  }
  __syncwarp();
  const int cg = gt % kColGroups, rg = gt / kColGroups, c = col0 + lane * 4;
  uint4 ahead_row[kDecAhead / 2];
  float4 ahead_pre[kDecAhead];
#pragma unroll
  for (int i = 0; i < kDecAhead / 2; ++i) {
    const int j = rg + i * kRowGroups;
    if (j < len) ahead_row[i] = *reinterpret_cast<const uint4*>(enc + row + j * step_elems + col0 + cg * kN);
  }
#pragma unroll
  for (int i = 0; i < kDecAhead; ++i) {
    const int t = w + i * kDecWarps;
    if (mine && t < Lt) ahead_pre[i] = __ldcs(reinterpret_cast<const float4*>(pre + t * step_elems + row + c));
  }
  const float4 b = bias != nullptr ? __ldg(reinterpret_cast<const float4*>(bias + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
  float proj[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) proj[i] = ld_f32<T>(dec_proj + c + i);
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

  float mx = -INFINITY;
  for (int j = lane; j < len; j += 32) mx = fmaxf(mx, s_score[seq][j]);
  mx = warp_max(mx);
  float sum = 0.f;
  for (int j = lane; j < len; j += 32) {
    const float e = expf(s_score[seq][j] - mx);
    if (w == 0) s_w[seq][j] = e;
    sum += e;
  }
  sum = warp_sum(sum);
  const float inv = len > 0 ? 1.f / sum : 0.f;
  group_sync();

  // weighted sum: a thread takes 16 bytes of every kRowGroups-th row
  {
    float acc[kN];
#pragma unroll
    for (int i = 0; i < kN; ++i) acc[i] = 0.f;
    const auto add = [&](int j, const uint4& piece) {
      float x[kN];
      ld_piece(reinterpret_cast<const T*>(&piece), x);
#pragma unroll
      for (int i = 0; i < kN; ++i) acc[i] = fmaf(s_w[seq][j], x[i], acc[i]);
    };
#pragma unroll
    for (int i = 0; i < kDecAhead / 2; ++i)
      if (rg + i * kRowGroups < len) add(rg + i * kRowGroups, ahead_row[i]);
    for (int j = rg + kDecAhead / 2 * kRowGroups; j < len; j += kRowGroups)
      add(j, *reinterpret_cast<const uint4*>(enc + row + j * step_elems + col0 + cg * kN));
#pragma unroll
    for (int i = 0; i < kN; ++i) s_part[seq][rg][cg * kN + i] = acc[i];
  }
  group_sync();
  if (gt < kAttnCols) {
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < kRowGroups; ++r) v += s_part[seq][r][gt];
    T t;
    st_f32<T>(&t, v * inv);
    for (uint32_t r = 0; r < ctas; ++r) st_cluster_16<T>(&s_v[seq][col0 + gt], r, t);
  }
  const bool u_there = mbar_wait(&u_full, 0, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
  __syncwarp();
  cluster_sync_all();

  // The vector into the rows of all steps.
  const uint2 v = *reinterpret_cast<const uint2*>(&s_v[seq][c]);
  if (mine)
    for (int t = w; t < Lt; t += kDecWarps) *reinterpret_cast<uint2*>(out + t * step_elems + row + c) = v;
  // v . U: 16 units and half of K a warp; the two sequences are columns 0 and 1 of 8.
  {
    const int m0 = (wid & 7) * 16, half = wid >> 3, col = lane >> 2;
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    const T* ar = s_u + (m0 + (lane & 15)) * u_stride + (lane >> 4) * 8;
    for (int k = half * (H / 2); k < (half + 1) * (H / 2); k += 16) {
      uint32_t a[4];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(smem_u32(ar + k)) : "memory");
      uint32_t b0 = 0, b1 = 0;
      if (col < 2) {
        b0 = *reinterpret_cast<const uint32_t*>(&s_v[col][k + 2 * (lane & 3)]);
        b1 = *reinterpret_cast<const uint32_t*>(&s_v[col][k + 8 + 2 * (lane & 3)]);
      }
      mma16816(d, a, b0, b1, T());
    }
    if ((lane & 3) == 0) {
      s_z[half][0][m0 + col] = d[0];
      s_z[half][1][m0 + col] = d[1];
      s_z[half][0][m0 + col + 8] = d[2];
      s_z[half][1][m0 + col + 8] = d[3];
    }
  }
  __syncthreads();

  // the steps of the sequence: a warp a step, four units a lane
  if (mine) {
    const float4 z0 = *reinterpret_cast<const float4*>(&s_z[0][seq][lane * 4]);
    const float4 z1 = *reinterpret_cast<const float4*>(&s_z[1][seq][lane * 4]);
    const float zz[4] = {z0.x + z1.x, z0.y + z1.y, z0.z + z1.z, z0.w + z1.w}, bb[4] = {b.x, b.y, b.z, b.w};
    const auto step = [&](int t, const float4& p) {
      const float x[4] = {p.x, p.y, p.z, p.w};
      T d[4];
      float term = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        st_f32<T>(d + i, tanh_fast((t > 0 ? x[i] + zz[i] : x[i]) + bb[i]));  // step 0 starts from nothing
        term = fmaf(ld_f32<T>(d + i), proj[i], term);
      }
      *reinterpret_cast<uint2*>(dec + t * step_elems + row + c) = *reinterpret_cast<const uint2*>(d);
      term = warp_sum(term);
      if (lane < ctas) st_cluster_f32(&s_term[rank][seq][t], lane, term);
    };
#pragma unroll
    for (int i = 0; i < kDecAhead; ++i)
      if (w + i * kDecWarps < Lt) step(w + i * kDecWarps, ahead_pre[i]);
    for (int t = w + kDecAhead * kDecWarps; t < Lt; t += kDecWarps)
      step(t, __ldcs(reinterpret_cast<const float4*>(pre + t * step_elems + row + c)));
  }
  __syncwarp();
  cluster_sync_all();  // (the last access to another CTA's memory lies before it)
  // Steps whose largest score, the encoder's largest plus the term, is not finite: attn_finish_kernel says what they do.
  if (mine && len > 0)
    for (int t = gt; t < Lt; t += 256) {
      float term = 0.f;
      for (uint32_t r = 0; r < ctas; ++r) term += s_term[r][seq][t];
      if (!isfinite(mx + term)) atomicMin(&s_first[seq], t);
    }
  group_sync();
  const float nan = __int_as_float(0x7FFFFFFF);
  if (mine)
    for (int t = s_first[seq] + w; t < Lt; t += kDecWarps)
      for (int h = col0 + lane; h < col0 + kAttnCols; h += 32) {
        if (t > s_first[seq]) st_f32<T>(dec + t * step_elems + row + h, nan);
        st_f32<T>(out + t * step_elems + row + h, nan);
      }
  if (!u_there) {
    // The wait ran out: give the copies of U time to land before the shared memory goes back.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
}

template <typename T>
int attn_decode_t(const void* enc, const void* enc_proj, const int* src_lens, float* scores, const float* pre, const void* U,
                  int ldu, const float* bias, const void* dec_proj, void* dec, void* out, int Lt, int Ls, int N, int H,
                  int* status, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  static std::atomic<unsigned long long> configured{0};
  if (!ensure_dynamic_smem(attn_decode_kernel<T>, kAttnCols * (kDecMaxH + 8) * 2, configured)) return FTB_ERR_LAUNCH;
  cfg.gridDim = dim3((N + 1) / 2 * (H / kAttnCols));
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = kAttnCols * (H + 8) * 2;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = H / kAttnCols;
  attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, attn_decode_kernel<T>, static_cast<const T*>(enc), static_cast<const T*>(enc_proj),
                                             src_lens, scores, pre, static_cast<const T*>(U), ldu, bias, static_cast<const T*>(dec_proj),
                                             static_cast<T*>(dec), static_cast<T*>(out), Lt, Ls, N, H, status);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
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

// Whether launch_attn_decode takes a call (its scratch aside): where all clusters are on the device at once (a CTA an SM; 72
// sequences at H 512) and a sequence has few steps.  us, the whole program as three launches behind the scan / as one, H 512, bf16:
// 50 + 50 positions, 55 sequences 109.0 / 98.4, 256 136.1 / 151.6; 26 + 52, 81 sequences 71.8 / 75.9; 27 + 8, 6 sequences 66.5 / 59.4;
// 20 + 250, 1 sequence 59.1 / 61.7; H 128, 26 + 61, 42 sequences 48.2 / 45.1.
bool attn_decode_supported(int dtype, int Ls, int Lt, int N, int H, int sm_count) {
  return dtype != FTB_F32 && H % kAttnCols == 0 && H <= kDecMaxH && Ls <= kDecMaxSource && Lt <= kDecMaxSteps &&
         (N + 1) / 2 * (H / kAttnCols) <= sm_count - 4;
}

// Everything behind the encoder's scan; pre: the decoder's input halves, U: row u of Wp_trg from its recurrent half on.
int launch_attn_decode(int dtype, const void* enc, const void* enc_proj, const int* src_lens, float* scores, const float* pre,
                       const void* U, int ldu, const float* bias, const void* dec_proj, void* dec, void* out, int Lt, int Ls,
                       int N, int H, int* status, cudaStream_t stream) {
  if (dtype == FTB_F16)
    return attn_decode_t<__half>(enc, enc_proj, src_lens, scores, pre, U, ldu, bias, dec_proj, dec, out, Lt, Ls, N, H, status, stream);
  return attn_decode_t<__nv_bfloat16>(enc, enc_proj, src_lens, scores, pre, U, ldu, bias, dec_proj, dec, out, Lt, Ls, N, H, status, stream);
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
