// One-off parameter re-layout for the cell kernels: the reference keeps one
// [in, out] matrix per gate (x @ W orientation, examples/stacked_rnn/rnn_utils.py);
// the kernels want one K-major row per accumulator column with the four gates of
// a unit in adjacent rows, so that a TMEM lane holds i,f,o,c~ of a unit in
// adjacent accumulator columns.
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {

namespace {

// A stack of transposes in one launch: blockIdx.z is (layer, matrix, gate), matrix 0 or 1 (W, U).
//   out[layer][(u * gates + g) * ldo + off + k] = in[layer][g][k][u],  k < K, u < U;  0 for U <= u < u_end
struct TransposeArgs {
  const void* in[2];
  int K[2];    // rows of a matrix
  int off[2];  // where they go in a packed row
  int matrices, gates, U, u_end, ldo;
  void* out;
  size_t out_layer;  // elements
};

// Bound by memory: 64 x 64 tiles through shared memory, 16 bytes a thread on both sides (reads go singly where rows do
// not begin on 16 bytes).  With 32 x 32 tiles moved element by element, a launch for each matrix of each layer, the
// word program's parameters (3 layers of 512, 10000 words, 22.6 MB) took 42 us a pass; so 15.
constexpr int kTile = 64, kPackThreads = 256;
template <typename E>
__global__ void __launch_bounds__(kPackThreads) pack_transpose_kernel(const TransposeArgs a) {
  constexpr int kN = 16 / sizeof(E), kVecs = kTile / kN;
  __shared__ E tile[kTile][kTile + 4 / sizeof(E)];
  const int g = blockIdx.z % a.gates, m = blockIdx.z / a.gates % a.matrices, layer = blockIdx.z / (a.gates * a.matrices);
  const int K = m == 0 ? a.K[0] : a.K[1], k0 = blockIdx.y * kTile, u0 = blockIdx.x * kTile;
  if (k0 >= K) return;
  const E* src = static_cast<const E*>(m == 0 ? a.in[0] : a.in[1]) + (static_cast<size_t>(layer) * a.gates + g) * K * a.U;
  const bool vec_in = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && a.U % kN == 0;
  if (vec_in) {
    for (int e = threadIdx.x; e < kTile * kVecs; e += kPackThreads) {
      const int k = e / kVecs, u = e % kVecs * kN;
      if (k0 + k >= K) continue;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (u0 + u < a.U) v = __ldcs(reinterpret_cast<const uint4*>(src + static_cast<size_t>(k0 + k) * a.U + u0 + u));
      const E* x = reinterpret_cast<const E*>(&v);
#pragma unroll
      for (int i = 0; i < kN; ++i) tile[k][u + i] = x[i];
    }
  } else {
    for (int e = threadIdx.x; e < kTile * kTile; e += kPackThreads) {
      const int k = e / kTile, u = e % kTile;
      if (k0 + k < K) tile[k][u] = u0 + u < a.U ? src[static_cast<size_t>(k0 + k) * a.U + u0 + u] : E(0);
    }
  }
  __syncthreads();
  E* dst = static_cast<E*>(a.out) + layer * a.out_layer + (m == 0 ? a.off[0] : a.off[1]);
  const bool vec_out = ((reinterpret_cast<uintptr_t>(dst) | static_cast<uintptr_t>(a.ldo) * sizeof(E)) & 15) == 0 && K % kN == 0;
  for (int e = threadIdx.x; e < kTile * kVecs; e += kPackThreads) {
    const int u = e / kVecs, k = e % kVecs * kN;
    if (u0 + u >= a.u_end || k0 + k >= K) continue;
    E* row = dst + (static_cast<size_t>(u0 + u) * a.gates + g) * a.ldo + k0 + k;
    uint4 v;
    E* x = reinterpret_cast<E*>(&v);
#pragma unroll
    for (int i = 0; i < kN; ++i) x[i] = tile[k + i][u];
    if (vec_out) {
      *reinterpret_cast<uint4*>(row) = v;
    } else {
      for (int i = 0; i < kN && k0 + k + i < K; ++i) row[i] = x[i];
    }
  }
}

template <typename E>
__global__ void pack_bias_kernel(const E* __restrict__ bias, float* __restrict__ out, int gates, int H, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int layer = i / (gates * H), r = i - layer * gates * H, g = r / H, u = r - g * H;
  out[static_cast<size_t>(layer) * gates * H + u * gates + g] = static_cast<float>(bias[i]);
}

int pack_stack(const TransposeArgs& a, int layers, int dtype, cudaStream_t s) {
  const int K = a.matrices > 1 && a.K[1] > a.K[0] ? a.K[1] : a.K[0], per_layer = a.gates * a.matrices;
  // (gridDim.z is 65535 at most)
  for (int l0 = 0, step = 65535 / per_layer; l0 < layers; l0 += step) {
    TransposeArgs b = a;
    const int n = layers - l0 < step ? layers - l0 : step;
    for (int m = 0; m < a.matrices; ++m)
      b.in[m] = static_cast<const char*>(a.in[m]) + static_cast<size_t>(l0) * a.gates * a.K[m] * a.U * dtype_size(dtype);
    b.out = static_cast<char*>(a.out) + l0 * a.out_layer * dtype_size(dtype);
    const dim3 grid((a.u_end + kTile - 1) / kTile, (K + kTile - 1) / kTile, n * per_layer);
    if (dtype_size(dtype) == 4)
      pack_transpose_kernel<uint32_t><<<grid, kPackThreads, 0, s>>>(b);
    else
      pack_transpose_kernel<uint16_t><<<grid, kPackThreads, 0, s>>>(b);
    count_launch();
    if (cudaGetLastError() != cudaSuccess) return FTB_ERR_LAUNCH;
  }
  return FTB_OK;
}

}  // namespace

int pack_lstm(const void* W, const void* U, const void* bias, void* Wp, float* bias_p, int D, int I, int H, int dtype,
              cudaStream_t s) {
  const int K = I + H;
  const TransposeArgs a = {{W, U}, {I, H}, {0, I}, 2, 4, H, H, K, Wp, static_cast<size_t>(4) * H * K};
  const int rc = pack_stack(a, D, dtype, s);
  if (rc) return rc;
  if (bias != nullptr && bias_p != nullptr) {
    const int n = D * 4 * H, thr = 256, grid = (n + thr - 1) / thr;
    if (dtype == FTB_F32)
      pack_bias_kernel<float><<<grid, thr, 0, s>>>(static_cast<const float*>(bias), bias_p, 4, H, n);
    else if (dtype == FTB_F16)
      pack_bias_kernel<__half><<<grid, thr, 0, s>>>(static_cast<const __half*>(bias), bias_p, 4, H, n);
    else
      pack_bias_kernel<__nv_bfloat16><<<grid, thr, 0, s>>>(static_cast<const __nv_bfloat16*>(bias), bias_p, 4, H, n);
    if (cudaGetLastError() != cudaSuccess) return FTB_ERR_LAUNCH;
    count_launch();
  }
  return FTB_OK;
}

// P: [H, V] (x @ P orientation) -> Pt: [Vp, H] K-major, row v = column v of P, rows V..Vp-1 zero.
int pack_projection(const void* P, void* Pt, int H, int V, int Vp, int dtype, cudaStream_t s) {
  const TransposeArgs a = {{P, nullptr}, {H, 0}, {0, 0}, 1, 1, V, Vp, H, Pt, 0};
  return pack_stack(a, 1, dtype, s);
}

// Grid cell: Wp[u, k] = i2h[k, u] for the 2H states, then h2h for the H inputs.
int pack_grid(const void* i2h, const void* h2h, void* Wp, int H, int dtype, cudaStream_t s) {
  const TransposeArgs a = {{i2h, h2h}, {2 * H, H}, {0, 2 * H}, 2, 1, H, H, 3 * H, Wp, 0};
  return pack_stack(a, 1, dtype, s);
}

// Tanh RNN cell: Wp[u, k] = W[k, u] for k < I, U[k - I, u] for the H recurrent inputs behind them.
int pack_rnn(const void* W, const void* U, void* Wp, int I, int H, int dtype, cudaStream_t s) {
  const TransposeArgs a = {{W, U}, {I, H}, {0, I}, 2, 1, H, H, I + H, Wp, 0};
  return pack_stack(a, 1, dtype, s);
}

}  // namespace ftb
