// How the stacked LSTM kernels whose hidden states carry their own arrival would run a problem, and what they
// would take: shared by the kernels' files and the entry points that choose between schedules (csrc/wavefront.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ftb {

// csrc/lstm_flow.cu (16-bit): batch slices of nb columns, S of them, G layers beside each other, CTAs in pairs or not, weight
// blocks of the ring that input weights pass through (0: all are kept).
struct FlowPlan {
  int nb, S, G;
  bool pair;
  int ring;
  double est_us;
};
bool lstm_flow_plan(int dtype, int D, int L, int N, int64_t T, int I, int H, int sm_count, bool stream, FlowPlan* plan);
bool lstm_flow_form(int dtype, int D, int N, int I, int H, int sm_count, int nb, bool pair, bool ring, FlowPlan* plan);
int launch_lstm_flow(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c, const int* off,
                     int64_t T, int D, int L, int N, int I, int H, const FlowPlan& plan, int* flags, int* status,
                     cudaStream_t stream);

// csrc/lstm_simt_flow.cu (fp32): tiles of `rows` sequences (8, 16 or 32).
struct SimtFlowPlan {
  int rows;
  double est_us;
};
bool lstm_simt_flow_plan(int D, int L, int N, int I, int H, int sm_count, SimtFlowPlan* plan);
int launch_lstm_simt_flow(const float* x, const float* Wp, const float* bias_p, float* hs, float* c, int D, int L, int N,
                          int H, const SimtFlowPlan& plan, int* status, int sm_count, cudaStream_t stream);

// csrc/grid_flow.cu (16-bit grid RNN): batch slices of nb columns, S of them, `groups` (layer, row, slice) chains beside each other.
struct GridFlowPlan {
  int nb, S, groups;
  size_t ints;  // counters
  double est_us;
};
size_t grid_flow_ints(int D, int A, int B, int N);
bool grid_flow_form(int dtype, int D, int A, int B, int N, int H, int sm_count, int nb, GridFlowPlan* plan);
bool grid_flow_plan(int dtype, int D, int A, int B, int N, int H, int sm_count, size_t max_ints, GridFlowPlan* plan);
int launch_grid_flow(int dtype, const void* X, const void* Y, const void* Wpx, const void* Wpy, const float* bias_x,
                     const float* bias_y, void* hx, void* hy, int D, int A, int B, int N, int H, const GridFlowPlan& plan,
                     int* counters, int* status, cudaStream_t stream);

}  // namespace ftb
