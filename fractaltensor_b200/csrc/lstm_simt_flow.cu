// fp32 stacked LSTM, I == H, as one persistent launch whose hidden states carry their own arrival
// (examples/stacked_rnn/stacked_lstm1.py:12-76).
//
// A CTA owns TM sequences x 8 units (32 packed gate columns) of one layer for a whole sweep over time,
// weights in shared memory and cell state in registers, as csrc/lstm_simt_static.cu does.  There a step is
// one serial pass (flag, both operands from L2, multiply, reduce, store, fence, flag: 8.2 us at H 256 and
// 32 sequences, 3.2 of them the multiplication).  Here its parts belong to warps of their own:
//   * the output array is filled with 0xFFFFFFFF beforehand, a pattern no hidden state has (NaN is stored as
//     0x7FFFFFFF).  Readers take 16-byte chunks of the rows they need and repeat those with a word that has
//     not arrived: no fence, no flag, one trip through L2;
//   * the input half of step t + 1 is multiplied by the early warps while the state of step t is under way;
//     its operand is loaded by warps of their own, a step ahead.  Only the recurrent half is on the chain;
//   * shared memory gives an SM 128 bytes a cycle however many lanes read the same word, so that what a lane
//     multiplies per word it reads is the rate: 8 rows x 8 columns of one 32-wide K chunk, four products a word;
//   * TM is 8, 16 or 32: small batches multiply no rows that are not there, and small models spread theirs
//     over the device.
// A step of 32 rows in cycles (stamps of one CTA): the recurrent half's multiplication 4840 of 10 450, its sums 850, two cells a thread
// 1080, the pause before the first look 450, the states 2920; of 16 rows 2240 of 5490, 480, 600, 550 and 1430; of 8 rows 1110 of 3930,
// 430, 610, 410 and 1130.  Against one serial pass (us, D x L x N x H): 4 x 64 x 32 x
// 256 550 -> 385, 4 x 64 x 16 x 256 526 -> 218, 2 x 64 x 8 x 256 499 -> 151.
// The sums are the level kernel's (csrc/cell_simt.cu): every chunk of 32 in ascending order, a group's chunks in
// order, the four groups in order; all fp32 schedules give the same bits.
//
// The roles meet at named barriers: warps that wait there take no issue slots, and polling a shared-memory
// barrier instead cost the multiplying warps three quarters of their rate (4.4 cycles an FMA).
//
// Cooperative launch: CTAs wait for each other's states.  That wait is bounded; when it runs out, or another
// CTA has reported an error, the CTA goes through the rest of its steps without waiting for data.
#include "../../include/ftb200.h"
#include "flow_plan.h"
#include "ptx.cuh"
#include "tmap.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>

namespace ftb {

namespace {

constexpr int TN = 32;  // gate columns of a CTA
constexpr int TK = 32;  // K chunk of the level kernel (fixes the summation order)
constexpr int kLdW = TN + 4;
constexpr int kMaxSlots = 2;     // input tiles in shared memory
constexpr int kMaxPause = 4000;  // cycles
constexpr int kMaxSmem = 224 * 1024;
constexpr int kLoadWarps = 4;
constexpr int kMul = 4;  // multiplying warps of a half

// Named barriers (0 is __syncthreads).
enum Bar : int { kInFull = 1, kInEmpty = 1 + kMaxSlots, kPartsTaken = 1 + 2 * kMaxSlots, kEarlyDone, kLateWarpsMeet, kEarlyWarpsMeet };
__device__ __forceinline__ void bar_wait(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_post(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <int TM>
struct SimtFlowCfg {
  // A lane's part of a chunk's TM x 32 products; 16 lanes make up the chunk.
  static constexpr int kRows = TM == 32 ? 8 : 4, kCols = TM == 8 ? 4 : 8;
  static constexpr int kLateWarps = 4;
  static constexpr int kCells = TM == 32 ? 2 : 1;  // of a thread of theirs, 16 rows apart
  // first warp of each role: the input half's multiplication, the recurrent half's and the cells, input tiles
  static constexpr int kLate = kMul, kLoad = kMul + kLateWarps;
  static constexpr int kThreads = 32 * (kLoad + kLoadWarps);
};

struct SimtFlowArgs {
  const float* x;     // [L, N, H]
  const float* w;     // packed [D, 4H, 2H]
  const float* bias;  // packed [D, 4H] or null
  float* hs;          // [D, L, N, H], all 0xFFFFFFFF before the launch
  float* c;           // [D, N, H]
  int* status;
  int D, L, N, H, G;
  int m_tiles, n_tiles;
  int n_slots;        // input tiles in shared memory
};

// Rows of activations in shared memory: a chunk is 36 words long, a row 8 more than a multiple of 32, so that the
// words at the same k of four rows and two chunks, which the lanes of a warp read together, are on 32 banks.
constexpr int kLdChunk = TK + 4;
__host__ __device__ constexpr int row_words(int H) { return (H / TK * kLdChunk + 31 - 8) / 32 * 32 + 8; }

__device__ __forceinline__ float sigmoid_acc(float x) { return 1.f / (1.f + expf(-x)); }

__device__ __forceinline__ uint4 ld_relaxed_gpu_v4(const float* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_gpu32(float* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ bool arrived(const uint4& v) {
  return v.x != 0xFFFFFFFFu && v.y != 0xFFFFFFFFu && v.z != 0xFFFFFFFFu && v.w != 0xFFFFFFFFu;
}

// Rows 0 .. rows-1 of [.., H] at src -> dst[row][row_words(H)], by warp `w` of `warps`: two 16-byte chunks of each of kInFlight
// rows a lane in flight.  With `poll` a chunk is repeated until its four words are states; the others (inputs of the call) are
// taken as they are.  Returns the number of rounds of loads beyond the first.  (Not inlined: beside the multiplications in the
// kernel's body the registers do not suffice and its loops spill.)
template <int kInFlight>
__device__ __noinline__ int load_rows(float* dst, const float* src, int rows, int H, int w, int warps, bool poll,
                                      uint32_t sleep_ns, volatile int* s_abort, int* status) {
  const int lane = threadIdx.x & 31, ld = row_words(H);
  int extra = 0;
  for (int r0 = w; r0 < rows; r0 += kInFlight * warps)
    for (int k0 = 4 * lane; __any_sync(0xffffffffu, k0 < H); k0 += 256) {
      uint4 v[2 * kInFlight];
      uint32_t mine = 0;
#pragma unroll
      for (int i = 0; i < 2 * kInFlight; ++i) {
        v[i] = make_uint4(0, 0, 0, 0);
        if (r0 + (i >> 1) * warps < rows && k0 + (i & 1) * 128 < H) mine |= 1u << i;
      }
      uint32_t missing = mine;
      uint64_t t0 = 0;
      for (uint32_t it = 0;;) {
#pragma unroll
        for (int i = 0; i < 2 * kInFlight; ++i)
          if (missing & (1u << i)) v[i] = ld_relaxed_gpu_v4(src + (r0 + (i >> 1) * warps) * H + k0 + (i & 1) * 128);
#pragma unroll
        for (int i = 0; i < 2 * kInFlight; ++i)
          if ((missing & (1u << i)) && (!poll || arrived(v[i]))) missing &= ~(1u << i);
        if (__all_sync(0xffffffffu, missing == 0) || __any_sync(0xffffffffu, *s_abort != 0)) break;
        ++extra;
        if (sleep_ns != 0) __nanosleep(sleep_ns);
        if ((++it & 0x3F) == 0) {
          if (t0 == 0) t0 = globaltimer_ns();
          if (__any_sync(0xffffffffu, globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS || ld_relaxed_gpu(status) != 0)) {
            if (lane == 0) {
              *s_abort = 1;
              atomicCAS(status, 0, FTB_ERR_TIMEOUT_DEP);
            }
            break;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 2 * kInFlight; ++i)
        if (mine & (1u << i)) {
          const int k = k0 + (i & 1) * 128;
          *reinterpret_cast<uint4*>(dst + (r0 + (i >> 1) * warps) * ld + k + 4 * (k / TK)) = v[i];
        }
    }
  return extra;
}

// The late warps' part of a state, rows w, w + warps, .. (kRows of them) of the next step's operand: what load_rows does, with
// the addresses and masks made once a sweep.  On the chain, beside the early warps' multiplication, every instruction counts:
// as load_rows 450 cycles until the first load, 400 to 650 until the last, 350 to 600 for the stores.
template <int kRows>
struct StateLoad {
  int first, src_row, dst_row, wide;  // (numbers)
  int dst_first;
  uint32_t mine;

  __device__ __forceinline__ StateLoad(int rows, int H, int w, int warps) {
    const int lane = threadIdx.x & 31, ld = row_words(H);
    first = w * H + 4 * lane;
    src_row = warps * H;
    dst_first = w * ld + 4 * lane + 4 * (4 * lane / TK);
    dst_row = warps * ld;
    wide = H;
    mine = 0;
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      if (w + i * warps < rows) mine |= 1u << i;
  }
  __device__ __forceinline__ int load(const float* src, float* dst, volatile int* s_abort, int* status) const {
    const int lane = threadIdx.x & 31;
    int extra = 0;
    src += first;
    dst += dst_first;
    for (int k0 = 4 * lane; k0 - 4 * lane < wide; k0 += 256, src += 256, dst += 256 + 32) {
      uint4 v[2][kRows];
      uint32_t missing[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) missing[j] = k0 + j * 128 < wide ? mine : 0u;
      const uint32_t taken[2] = {missing[0], missing[1]};
      uint64_t t0 = 0;
      for (uint32_t it = 1;; ++it) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < kRows; ++i)
            if (missing[j] & (1u << i)) v[j][i] = ld_relaxed_gpu_v4(src + i * src_row + j * 128);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < kRows; ++i)
            if ((missing[j] & (1u << i)) && arrived(v[j][i])) missing[j] &= ~(1u << i);
        if (__all_sync(0xffffffffu, (missing[0] | missing[1]) == 0)) break;
        ++extra;
        if (__any_sync(0xffffffffu, *s_abort != 0)) break;
        if ((it & 0x3F) == 0) {
          if (t0 == 0) t0 = globaltimer_ns();
          if (__any_sync(0xffffffffu, globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS || ld_relaxed_gpu(status) != 0)) {
            if (lane == 0) {
              *s_abort = 1;
              atomicCAS(status, 0, FTB_ERR_TIMEOUT_DEP);
            }
            break;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < kRows; ++i)
          if (taken[j] & (1u << i)) *reinterpret_cast<uint4*>(dst + i * dst_row + j * (128 + 16)) = v[j][i];
    }
    return extra;
  }
};

// 32 rows: 16 loads a lane in flight leave no registers for addresses kept beside the rest (inlined 383 -> 490 us a call).
template <>
struct StateLoad<8> {
  int rows, H, w, warps;

  __device__ __forceinline__ StateLoad(int rows, int H, int w, int warps) : rows(rows), H(H), w(w), warps(warps) {}
  __device__ __forceinline__ int load(const float* src, float* dst, volatile int* s_abort, int* status) const {
    return load_rows<8>(dst, src, rows, H, w, warps, true, 0, s_abort, status);
  }
};

// Products of the TM rows A[row][lda] with W[k][kLdW], n_chunks (even) chunks of 32 wide; chunk c's sums, in
// ascending order of k, to p[c][TM][32].  Warp w of kMul, a half-warp to a chunk: a lane has rows ry, ry + G, ..
// (neighbouring rows fall on different banks) and kCols columns, two of them to an FMA (fma.rn.f32x2: each
// half rounds as fmaf does).  H 256, 148 CTAs, cycles of four warps alone at TM 8 / 16 / 32, unrolled whole: 1100 / 1750 / 3250 (packed
// FMAs on registers alone would take 650 / 1300 / 2600).  The loop over k is unrolled whole at 8 and 16 rows (4 x 64 x 16 x 256 219 us,
// by eight k 233).  At 32 rows that is 27 KB of code: two SMs share what fetches it, and where their CTAs are not in step, with
// tiles of different heights or layers beside each other, everything on both of them took up to 1.8 times as long.
// Four k at a time, us whole / four: 3 layers of 64 steps, H 192, 36 sequences 455 / 365, 32 350 / 362; 4 of H 128, 43 449 / 352.
template <int TM>
__device__ __forceinline__ void multiply_here(const float* A, const float* W, int lda, int n_chunks, float* p, int w) {
  constexpr int R = SimtFlowCfg<TM>::kRows, C = SimtFlowCfg<TM>::kCols, G = TM / R;
  const int lane = threadIdx.x & 31, cx = lane & (TN / C - 1), ry = (lane & 15) / (TN / C);
  for (int c = 2 * w + (lane >> 4); c < n_chunks; c += 2 * kMul) {
    uint64_t acc[R][C / 2] = {};
    const float* a = A + ry * lda + c * kLdChunk;
    const float* b = W + c * TK * kLdW + C * cx;
    constexpr int kUnroll = TM == 32 ? 2 : TK / 2;
#pragma unroll kUnroll
    for (int k = 0; k < TK; k += 2, a += 2, b += 2 * kLdW) {
      float2 av[R];
#pragma unroll
      for (int i = 0; i < R; ++i) av[i] = *reinterpret_cast<const float2*>(a + i * G * lda);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint64_t wv[C / 2];
#pragma unroll
        for (int h = 0; h < C; h += 4) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(b + q * kLdW + h);
          wv[h / 2] = v.x; wv[h / 2 + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float x = q == 0 ? av[i].x : av[i].y;
          uint64_t xx;
          asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(x));
#pragma unroll
          for (int h = 0; h < C / 2; ++h) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][h]) : "l"(xx), "l"(wv[h]));
        }
      }
    }
    float* out = p + c * TM * TN + C * cx;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int h = 0; h < C / 2; h += 2)
        *reinterpret_cast<ulonglong2*>(out + (ry + i * G) * TN + 2 * h) = make_ulonglong2(acc[i][h], acc[i][h + 1]);
  }
}

// (A call at 16 rows, where inlining it leaves the rest of the kernel too few registers.  At 8 rows 151 us inlined against 155 for
// 2 x 64 x 8 x 256; at 32 rows, with four k at a time, 383 against 426 for 4 x 64 x 32 x 256.)
template <int TM>
__device__ __noinline__ void multiply_call(const float* A, const float* W, int lda, int n_chunks, float* p, int w) {
  multiply_here<TM>(A, W, lda, n_chunks, p, w);
}
template <int TM>
__device__ __forceinline__ void multiply(const float* A, const float* W, int lda, int n_chunks, float* p, int w) {
  if constexpr (TM == 16) multiply_call<TM>(A, W, lda, n_chunks, p, w);
  else multiply_here<TM>(A, W, lda, n_chunks, p, w);
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
// Chunks from .. to-1 of four columns, in order.
__device__ __forceinline__ float4 chunk_sum(const float* q, int stride, int from, int to) {
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int ch = from; ch < to; ++ch) sum = add4(sum, *reinterpret_cast<const float4*>(q + ch * stride));
  return sum;
}
// n chunks in kGroups groups, the groups in order.
template <int kGroups>
__device__ __forceinline__ float4 group_sums(const float* q, int stride, int n) {
  float4 v = chunk_sum(q, stride, 0, n / kGroups);
#pragma unroll
  for (int g = 1; g < kGroups; ++g) v = add4(v, chunk_sum(q, stride, n * g / kGroups, n * (g + 1) / kGroups));
  return v;
}

template <int TM>
__global__ void __launch_bounds__(SimtFlowCfg<TM>::kThreads, 1)
lstm_simt_flow_kernel(const __grid_constant__ SimtFlowArgs a) {
  using C = SimtFlowCfg<TM>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_abort;

  const int H = a.H, K = 2 * H, lda = row_words(H);
  float* sW = reinterpret_cast<float*>(smem_raw);  // [2H][36]
  float* sS = sW + K * kLdW;                       // [TM][lda] state
  float* sI = sS + TM * lda;                       // [n_slots][TM][lda] input
  float* sP = sI + a.n_slots * TM * lda;           // [H / 16][TM][32] sums of chunks
  const int tid = threadIdx.x, warp = tid >> 5;
  int* status = a.status;
  if (tid == 0) s_abort = 0;

  const int tiles = a.m_tiles * a.n_tiles;
  const int j = blockIdx.x / tiles;
  const int tile = blockIdx.x - j * tiles;
  const int n_tile = tile / a.m_tiles;
  const int row0 = (tile - n_tile * a.m_tiles) * TM;
  const int rows = min(TM, a.N - row0);
  const size_t step_elems = static_cast<size_t>(a.N) * H;
  const int chunks = H / TK;  // of a half
  // Threads at the barriers between two roles, and between the late warps.
  constexpr int kWithLoad = 32 * (kMul + kLoadWarps), kWithLate = 32 * (kMul + C::kLateWarps), kLateThreads = 32 * C::kLateWarps;
  const int total = (a.D - j + a.G - 1) / a.G * a.L;  // steps of this CTA

  int pause = 300;  // cycles between a state's store and the first look for the others'
  int k = 0;        // steps since the launch
  for (int l = j; l < a.D; l += a.G) {
    __syncthreads();  // the last sweep's weights have been used
    {
      const float* W = a.w + (static_cast<size_t>(l) * 4 * H + n_tile * TN) * K;
      const int k4s = K / 4;
#pragma unroll 1
      for (int e = tid; e < TN * k4s; e += C::kThreads) {
        const int col = e / k4s, kk = (e - col * k4s) * 4;
        const float4 v = *reinterpret_cast<const float4*>(W + static_cast<size_t>(col) * K + kk);
        sW[(kk + 0) * kLdW + col] = v.x;
        sW[(kk + 1) * kLdW + col] = v.y;
        sW[(kk + 2) * kLdW + col] = v.z;
        sW[(kk + 3) * kLdW + col] = v.w;
      }
      if (l == j)  // rows past the batch are multiplied as zeros
        for (int e = tid; e < (1 + a.n_slots) * TM * lda; e += C::kThreads) sS[e] = 0.f;
    }
    __syncthreads();
    float* hs_l = a.hs + static_cast<size_t>(l) * a.L * step_elems + static_cast<size_t>(row0) * H;

    if (warp < C::kLate) {
      // ------------------------------------------------------------ input half
      for (int t = 0; t < a.L; ++t, ++k) {
        const int slot = a.n_slots == 2 ? (k & 1) : 0;
        bar_wait(kInFull + slot, kWithLoad);
        if (k > 0) bar_wait(kPartsTaken, kWithLate);
        multiply<TM>(sI + slot * TM * lda, sW, lda, chunks, sP, warp);
        if (k + a.n_slots < total) bar_post(kInEmpty + slot, kWithLoad);
        // The sums of the input half, which leaves those of the recurrent half alone on the chain: the first two of the four
        // groups are the input's.  (The first step of a sweep is an input half alone: its chunks make up all four.)
        bar_wait(kEarlyWarpsMeet, 32 * kMul);
#pragma unroll
        for (int i = 0; i < C::kCells; ++i)
          if ((tid >> 3) + 16 * i < TM) {
            float* q = sP + ((tid >> 3) + 16 * i) * TN + 4 * (tid & 7);
            *reinterpret_cast<float4*>(q) = t == 0 ? group_sums<4>(q, TM * TN, chunks) : group_sums<2>(q, TM * TN, chunks);
          }
        bar_post(kEarlyDone, kWithLate);
      }
    } else if (warp < C::kLoad) {
      // -------------------------------- recurrent half, cells, then the layer's whole state for the next step
      const int cell = tid - 32 * C::kLate;
      const int row = cell >> 3, u = cell & 7, unit = n_tile * 8 + u;  // and the row 16 further, TM 32
      float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.bias != nullptr) b = *reinterpret_cast<const float4*>(a.bias + static_cast<size_t>(l) * 4 * H + 4 * unit);
      float c[C::kCells] = {};
      const StateLoad<TM / C::kLateWarps> state(rows, H, warp - C::kLate, C::kLateWarps);
      for (int t = 0; t < a.L; ++t, ++k) {
        if (t > 0) multiply<TM>(sS, sW + H * kLdW, lda, chunks, sP + chunks * TM * TN, warp - C::kLate);
        bar_wait(kEarlyDone, kWithLate);  // (the late warps meet here too)
        float* out = hs_l + t * step_elems;
        float4 v[C::kCells];
#pragma unroll
        for (int i = 0; i < C::kCells; ++i) {
          v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (row + 16 * i < TM) {
            const float* q = sP + (row + 16 * i) * TN + 4 * u;
            v[i] = *reinterpret_cast<const float4*>(q);
            if (t > 0) {
              const float* r = q + chunks * TM * TN;
              v[i] = add4(v[i], chunk_sum(r, TM * TN, 0, chunks / 2));
              v[i] = add4(v[i], chunk_sum(r, TM * TN, chunks / 2, chunks));
            }
          }
        }
        if (row < rows) {
          uint32_t bits[C::kCells];
#pragma unroll
          for (int i = 0; i < C::kCells; ++i) {
            const float gi = sigmoid_acc(v[i].x + b.x);
            const float gf = sigmoid_acc(v[i].y + b.y);
            const float go = sigmoid_acc(v[i].z + b.z);
            const float gc = tanhf(v[i].w + b.w);
            const float cn = gf * c[i] + gi * gc;
            c[i] = cn;
            bits[i] = __float_as_uint(go * tanhf(cn));
            if (bits[i] == 0xFFFFFFFFu) bits[i] = 0x7FFFFFFFu;
          }
#pragma unroll
          for (int i = 0; i < C::kCells; ++i)
            if (row + 16 * i < rows) st_relaxed_gpu32(out + static_cast<size_t>(row + 16 * i) * H + unit, bits[i]);
        }
        __syncwarp();
        // (After the cells, not before: the early warps' multiplication would slow them to a third.)
        if (k + 1 < total) bar_post(kPartsTaken, kWithLate);
        if (t + 1 < a.L) {
          {
            const long long c0 = clock64();
            while (clock64() - c0 < pause) __nanosleep(20);
          }
          const int extra = state.load(out, sS, &s_abort, status);
          // Everything at the first look: a little earlier next time; else later.  (Looks that come too early
          // load the L2 that the states have to pass through.)
          pause = extra > 0 ? min(pause + 100, kMaxPause) : pause - (pause >> 5);
          bar_wait(kLateWarpsMeet, kLateThreads);
        }
      }
#pragma unroll
      for (int i = 0; i < C::kCells; ++i)
        if (row + 16 * i < rows) a.c[(static_cast<size_t>(l) * a.N + row0 + row + 16 * i) * H + unit] = c[i];
    } else {
      // ------------------------------------------------------------ input tiles
      const float* src = l == 0 ? a.x + static_cast<size_t>(row0) * H : hs_l - static_cast<size_t>(a.L) * step_elems;
      for (int t = 0; t < a.L; ++t, ++k) {
        const int slot = a.n_slots == 2 ? (k & 1) : 0;
        if (k >= a.n_slots) bar_wait(kInEmpty + slot, kWithLoad);
        load_rows<4>(sI + slot * TM * lda, src + t * step_elems, rows, H, warp - C::kLoad, kLoadWarps, l > 0, 200, &s_abort,
                  status);
        bar_post(kInFull + slot, kWithLoad);
      }
    }
  }
}

size_t smem_bytes(int tm, int H, int slots) {
  return (static_cast<size_t>(2 * H) * kLdW + static_cast<size_t>(1 + slots) * tm * row_words(H) + H / 16 * tm * TN) *
         sizeof(float);
}

template <int TM>
int launch(const SimtFlowArgs& a, size_t smem, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = lstm_simt_flow_kernel<TM>;
  if (!ensure_dynamic_smem(kfn, kMaxSmem, configured)) return FTB_ERR_LAUNCH;
  // FTB_REFUSE_COOPERATIVE=1 makes this function answer as if the driver had refused the
  // cooperative launch (host-side failure injection for the schedule fallback's tests).
  {
    const char* e = getenv("FTB_REFUSE_COOPERATIVE");
    if (e != nullptr && e[0] == '1') return FTB_ERR_LAUNCH;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.G * a.m_tiles * a.n_tiles);
  cfg.blockDim = dim3(SimtFlowCfg<TM>::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[1];
  int na = 0;
  // FTB_NO_COOPERATIVE=1 drops the cooperative attribute (profilers that cannot replay
  // cooperative launches); residency then rests on grid <= SM count on an otherwise idle device.
  static const bool no_coop = [] {
    const char* e = getenv("FTB_NO_COOPERATIVE");
    return e != nullptr && e[0] == '1';
  }();
  if (!no_coop) {
    attrs[na].id = cudaLaunchAttributeCooperative;
    attrs[na].val.cooperative = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  if (cudaLaunchKernelEx(&cfg, kfn, a) != cudaSuccess) {
    cudaGetLastError();
    return FTB_ERR_LAUNCH;
  }
  count_launch();
  return FTB_OK;
}

}  // namespace

// How the kernel would run a problem; est_us: about what that takes.  False: not for this kernel.  Layers that do not fit on the
// device beside each other cost a sweep each.  Measured steps, us, at H 64 / 128 / 192 / 256 / 320 / 384: 8 rows 1.75 / 1.8 / 1.9 /
// 2.0 / 2.9 / 3.0, 16 rows - / 2.6 / 2.7 / 2.85 / 4.3 / 4.6, 32 rows 4.7 / 4.85 / 5.05 / 5.3.  A row of more than 256 is read in two rounds.
bool lstm_simt_flow_plan(int D, int L, int N, int I, int H, int sm_count, SimtFlowPlan* plan) {
  if (I != H || H % 64 != 0) return false;
  bool found = false;
  for (int tm = 8; tm <= 32; tm *= 2) {
    if (smem_bytes(tm, H, 1) > static_cast<size_t>(kMaxSmem)) continue;
    const long long tiles = static_cast<long long>((N + tm - 1) / tm) * (4 * H / TN);
    if (tiles > sm_count) continue;
    const int per_sweep = std::min<int>(D, static_cast<int>(sm_count / tiles));
    const int sweeps = (D + per_sweep - 1) / per_sweep;
    const double h = H / 256.0;
    const double step = tm == 8    ? 1.65 + 0.35 * h + (H > 256 ? 0.75 : 0.0)
                        : tm == 16 ? 2.2 + 0.68 * h + (H > 256 ? 1.3 : 0.0)
                                   : 4.44 + 0.83 * h;
    const double us = static_cast<double>(sweeps) * (L + per_sweep - 1) * step;
    if (!found || us < plan->est_us) *plan = {tm, us};
    found = true;
  }
  return found;
}

// x: [L,N,H]; Wp: [D,4H,2H] fp32 packed; hs: [D,L,N,H]; c: [D,N,H]; plan: lstm_simt_flow_plan.
int launch_lstm_simt_flow(const float* x, const float* Wp, const float* bias_p, float* hs, float* c, int D, int L, int N,
                          int H, const SimtFlowPlan& plan, int* status, int sm_count, cudaStream_t stream) {
  const int tm = plan.rows;
  SimtFlowArgs a;
  a.x = x;
  a.w = Wp;
  a.bias = bias_p;
  a.hs = hs;
  a.c = c;
  a.status = status;
  a.D = D; a.L = L; a.N = N; a.H = H;
  a.m_tiles = (N + tm - 1) / tm;
  a.n_tiles = 4 * H / TN;
  a.G = std::min(D, sm_count / (a.m_tiles * a.n_tiles));
  if (a.G < 1) return FTB_ERR_ARG;
  a.n_slots = smem_bytes(tm, H, 2) <= static_cast<size_t>(kMaxSmem) ? 2 : 1;
  const size_t smem = smem_bytes(tm, H, a.n_slots);
  if (cudaMemsetAsync(hs, 0xFF, sizeof(float) * static_cast<size_t>(D) * L * N * H, stream) != cudaSuccess)
    return FTB_ERR_LAUNCH;
  if (tm == 8) return launch<8>(a, smem, stream);
  if (tm == 16) return launch<16>(a, smem, stream);
  return launch<32>(a, smem, stream);
}

}  // namespace ftb
