// Host side of the RNN hot path: wavefront schedulers that turn the
// fold/scan/map nests of the reference programs into levels of independent
// cells, one kernel launch per level, plus the C-ABI entry points.
//
// The reference derives the same schedules by hand per benchmark
// (benchmarks/rnn/fractaltensor/stacked_lstm/regions/region3.h:11-28 for the
// stacked skew m = d + t, dilated_lstm/regions/region2.h:34-93 for the dilated
// steps, grid_lstm/regions/region8.h:26-53 for m = d + i + j) and executes each
// hyperplane as gather -> batched GEMM -> elementwise -> scatter.  Here a level
// is one launch of a fused cell kernel that addresses the hyperplane in place.
#include <algorithm>
#include <initializer_list>
#include <map>
#include <mutex>
#include <vector>

#include "../../include/ftb200.h"
#include "cell.h"
#include "flow_plan.h"
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {

int launch_cell_gemm(int dtype, int epi, int bn, int pair, const CUtensorMap* maps, const CUtensorMap& mapW,
                     const CUtensorMap& mapC, const CellBatch& batch, int* status, int sm_count,
                     cudaStream_t stream);
int launch_cell_gemm_persistent(int dtype, int epi, int bn, int pair, const CUtensorMap* maps,
                                const CUtensorMap& mapW, const CUtensorMap& mapC, const CellBatch& header,
                                const PlanView& plan, int* status, int sm_count, cudaStream_t stream);
bool lstm_simt_static_supported(int D, int N, int I, int H, int sm_count);
double lstm_simt_static_us(int D, int L, int N, int I, int H, int sm_count);
int launch_lstm_simt_static(const float* x, const float* Wp, const float* bias_p, float* hs, float* c, int D, int L,
                            int N, int I, int H, int* done, int* status, int sm_count, cudaStream_t stream);
bool lstm_static_supported(int dtype, int D, int N, int I, int H, int G, int sm_count);
int launch_lstm_static(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c, int D, int L,
                       int N, int I, int H, int G, int* done, int* status, unsigned long long* trace,
                       cudaStream_t stream);
bool lstm_wmajor_supported(int dtype, int D, int N, int I, int H, int G, int sm_count);
int launch_lstm_wmajor(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c, int D, int L,
                       int N, int I, int H, int G, int resident, int* done, int* status, unsigned long long* trace,
                       cudaStream_t stream);
bool lstm_dilated_cluster_supported(int dtype, int D, int N, int H, int sm_count);
size_t lstm_dilated_cluster_flag_ints(int D, int L);
int launch_lstm_dilated_cluster(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c,
                                const int* dilations, int D, int L, int N, int H, int schedule, int* flags, int* status,
                                int sm_count, cudaStream_t stream);
int launch_cell_simt(int epi, const float* const* act, const int* ld_act, const float* const* w, int ldw,
                     const CellBatch& batch, cudaStream_t stream);
int pack_lstm(const void* W, const void* U, const void* bias, void* Wp, float* bias_p, int D, int I, int H, int dtype,
              cudaStream_t s);
int pack_grid(const void* i2h, const void* h2h, void* Wp, int H, int dtype, cudaStream_t s);
int pack_projection(const void* P, void* Pt, int H, int V, int Vp, int dtype, cudaStream_t s);
int pack_rnn(const void* W, const void* U, void* Wp, int I, int H, int dtype, cudaStream_t s);
int rnn_attention_max_src_len();
// project.cu
bool project_twice_supported(int dtype, long long T, int V, int H, bool unpacked);
size_t project_twice_scratch(long long T, int V);
int launch_project_twice(int dtype, const void* h, const void* P, bool unpacked, float* probs, long long ld, int T, int V,
                         int Vp, int H, void* scratch, int* status, cudaStream_t stream);
bool attn_decode_supported(int dtype, int Ls, int Lt, int N, int H, int sm_count);
int launch_attn_decode(int dtype, const void* enc, const void* enc_proj, const int* src_lens, float* scores, const float* pre,
                       const void* U, int ldu, const float* bias, const void* dec_proj, void* dec, void* out, int Lt, int Ls,
                       int N, int H, int* status, cudaStream_t stream);
int launch_attn_vectors(int dtype, const void* enc, const void* enc_proj, const int* src_lens, float* scores, void* out,
                        int Lt, int Ls, int N, int H, cudaStream_t stream);
int launch_attn_finish(int dtype, void* dec, const void* dec_proj, const float* scores, const int* src_lens, void* out,
                       int Lt, int Ls, int N, int H, cudaStream_t stream);
int launch_ragged_rows(const void* src, void* dst, const int* start, const int* off, int N, int L, long long row_bytes,
                       bool to_time_major, cudaStream_t stream);
bool rnn_chain_supported(int dtype, int H);
int launch_rnn_chain(int dtype, const float* pre, const void* Wp, int ldw, int k0, const float* bias,
                     const void* before, void* out, int steps, int N, int H, int* status, cudaStream_t stream);
int online_softmax_rows(const float* x, float* y, int rows, int width, int ld, int ld_out, cudaStream_t stream);

namespace {

constexpr size_t kWorkspaceBytes = 256;

// Launch context for one family of cells (up to two weight buffers, up to four
// activation buffers).
struct CellLauncher {
  int dtype = FTB_BF16;
  int epi = EPI_STORE;
  int bn = 128;
  int pair = 0;  // 16-bit path: run CTAs as pairs on 256-row blocks
  int n_cols = 0, ld_out = 0, ld_c = 0;
  int sm_count = 0;
  int* status = nullptr;
  cudaStream_t stream = nullptr;
  // 16-bit path
  CUtensorMap maps[kNumActMaps];
  CUtensorMap mapW;
  CUtensorMap mapC;  // fp32 cell state (LSTM); otherwise the second weight buffer's map (or a copy of mapW)
  // fp32 path
  const float* act[kNumActMaps] = {nullptr, nullptr, nullptr, nullptr};
  int ld_act[kNumActMaps] = {0, 0, 0, 0};
  const float* w = nullptr;   // weight buffer 0
  const float* w2 = nullptr;  // weight buffer 1 (cells with w_map == 1), same row length
  int ldw = 0;

  int rows_per_tile() const { return dtype == FTB_F32 ? 32 : 128; }
  int m_tiles_for(int rows) const {
    if (dtype != FTB_F32 && pair) return 2 * ((rows + 255) / 256);
    return (rows + rows_per_tile() - 1) / rows_per_tile();
  }
  int w_box_rows() const { return pair ? bn / 2 : bn; }
  int cols_per_tile() const { return dtype == FTB_F32 ? 32 : bn; }

  // Launches the cells of one level (any number; split into chunks).
  int run(std::vector<CellItem>& items) const {
    const int n_tiles_n = (n_cols + cols_per_tile() - 1) / cols_per_tile();
    for (size_t off = 0; off < items.size(); off += kMaxItems) {
      CellBatch b;
      b.n_items = static_cast<int>(std::min<size_t>(kMaxItems, items.size() - off));
      b.n_cols = n_cols;
      b.ld_out = ld_out;
      b.ld_c = ld_c;
      b.pad_ = 0;
      int tiles = 0;
      for (int i = 0; i < b.n_items; ++i) {
        CellItem it = items[off + i];
        it.m_tiles = m_tiles_for(it.rows);
        it.tile0 = tiles;
        tiles += it.m_tiles * n_tiles_n;
        b.items[i] = it;
      }
      b.total_tiles = tiles;
      int rc;
      if (dtype == FTB_F32) {
        const float* ws[kNumWeightMaps] = {w, w2 ? w2 : w};
        rc = launch_cell_simt(epi, act, ld_act, ws, ldw, b, stream);
      } else {
        rc = launch_cell_gemm(dtype, epi, bn, pair, maps, mapW, mapC, b, status, sm_count, stream);
      }
      if (rc) return rc;
    }
    return FTB_OK;
  }
};

// Runs a whole wavefront as one persistent launch: `items` in an order in which every item
// only depends on earlier ones, `deps[i]` = per segment the inclusive range of item indices the
// segment reads (-1 = external).  Tables go to the workspace with stream-ordered copies.
int run_persistent(const CellLauncher& cl, std::vector<CellItem>& items, const std::vector<int32_t>& deps,
                   char* ws, const struct PlanLayout& lay);

CellItem blank_item() {
  CellItem it;
  it.out = nullptr;
  it.c = nullptr;
  it.bias = nullptr;
  for (int s = 0; s < kMaxSeg; ++s) it.seg_row[s] = it.seg_kb[s] = it.seg_wk[s] = it.seg_map[s] = 0;
  it.nseg = 0;
  it.w_row0 = 0;
  it.rows = 0;
  it.c_zero = 0;
  it.tile0 = 0;
  it.m_tiles = 0;
  it.out_row0 = 0;
  it.c_row0 = 0;
  it.out_map = 1;
  it.w_map = 0;
  it.skip = 0;
  it.pad_ = 0;
  return it;
}

void add_seg(CellItem& it, int map, int64_t row, int k_elems, int wk) {
  const int s = it.nseg++;
  it.seg_map[s] = map;
  it.seg_row[s] = static_cast<int32_t>(row);
  it.seg_kb[s] = k_elems / 64;
  it.seg_wk[s] = wk;
}

int begin_call(void* workspace, size_t workspace_bytes, cudaStream_t stream, int** status) {
  if (workspace == nullptr || workspace_bytes < kWorkspaceBytes) return FTB_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0) return FTB_ERR_ALIGN;
  int rc = check_device_sm100();
  if (rc) return rc;
  if (cudaMemsetAsync(workspace, 0, kWorkspaceBytes, stream) != cudaSuccess) return FTB_ERR_LAUNCH;
  *status = static_cast<int*>(workspace);
  return FTB_OK;
}

bool valid_dtype(int dt) { return dt == FTB_F32 || dt == FTB_F16 || dt == FTB_BF16; }

// Every kernel reads and writes 16 bytes at a time (the fp32 path as float4, the 16-bit path by TMA).
bool aligned16(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return false;
  return true;
}

// Optional tuning knobs of the wavefront entry points (0 = automatic).
struct Tuning {
  int layers_per_group = 0, bn = 0, schedule = 0, skew = 0, pair = 0, fine_deps = 0, resident = 0;
  explicit Tuning(const int* t) {
    if (t != nullptr) {
      layers_per_group = t[0];
      bn = t[1];
      schedule = t[2];
      skew = t[3];
      pair = t[4];
      fine_deps = t[5];
      resident = t[6];
    }
  }
  // pair: 0 = automatic (pairs when a cell has more than 128 rows), 1 = never, 2 = always.
  int use_pair(int rows) const { return pair == 2 || (pair == 0 && rows > 128); }
};

// ---------------------------------------------------------- persistent schedule
// Workspace layout of a persistent stacked-LSTM call: status block, then the
// item table, the dependency table, the completion targets and the counters.
constexpr int kMaxCtas = 1024;  // entries of the per-CTA first-item table
struct PlanLayout {
  size_t items, dep, target, cta_first, done, tile_done, c_done, counters_end, trace, total;
};
PlanLayout plan_layout(size_t n_items, int max_tiles_per_item = 64) {
  PlanLayout p;
  auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  p.items = kWorkspaceBytes;
  p.dep = up(p.items + sizeof(CellItem) * n_items);
  p.target = up(p.dep + sizeof(int32_t) * 2 * kMaxSeg * n_items);
  p.cta_first = up(p.target + sizeof(int32_t) * n_items);
  p.done = up(p.cta_first + sizeof(int32_t) * kMaxCtas);
  const size_t max_tiles = n_items * max_tiles_per_item;
  p.tile_done = up(p.done + sizeof(int32_t) * 2 * n_items);
  p.c_done = up(p.tile_done + sizeof(int32_t) * max_tiles);
  p.counters_end = up(p.c_done + sizeof(int32_t) * max_tiles);
  p.trace = p.counters_end;
#ifdef FTB_TRACE
  p.total = up(p.trace + 8 * 4 * max_tiles);
#else
  p.total = p.trace;
#endif
  return p;
}

int run_persistent(const CellLauncher& cl, std::vector<CellItem>& items, const std::vector<int32_t>& deps,
                   char* ws, const PlanLayout& lay, size_t ws_bytes = 0) {
  const int n = static_cast<int>(items.size());
  const int n_tiles_n = (cl.n_cols + cl.cols_per_tile() - 1) / cl.cols_per_tile();
  std::vector<int32_t> target(n);
  int tiles = 0;
  for (int i = 0; i < n; ++i) {
    items[i].m_tiles = cl.m_tiles_for(items[i].rows);
    items[i].tile0 = tiles;
    tiles += items[i].m_tiles * n_tiles_n;
    target[i] = 8 * items[i].m_tiles * n_tiles_n;  // eight epilogue warps per tile
  }
  // Tile -> item lookups without a table walk on the device (the grid size computed here is
  // the one launch_cell_gemm_persistent uses): for every item the item that holds the tile one
  // grid stride further, and for every CTA the item of its first tile.
  int grid = std::min(tiles, cl.sm_count);
  if (cl.pair) grid &= ~1;
  if (grid <= 0) return FTB_OK;
  if (grid > kMaxCtas) return FTB_ERR_ARG;
  {
    int j = 0;
    for (int i = 0; i < n; ++i) {
      const int t = items[i].tile0 + grid;
      while (j + 1 < n && t >= items[j + 1].tile0) ++j;
      items[i].skip = j;
    }
  }
  std::vector<int32_t> cta_first(grid);
  {
    int j = 0;
    for (int c = 0; c < grid; ++c) {
      while (j + 1 < n && c >= items[j + 1].tile0) ++j;
      cta_first[c] = j;
    }
  }
  // The host vectors die with this call; cudaMemcpyAsync from pageable memory returns once the
  // bytes are staged.
  if (cudaMemcpyAsync(ws + lay.items, items.data(), sizeof(CellItem) * n, cudaMemcpyHostToDevice, cl.stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(ws + lay.dep, deps.data(), sizeof(int32_t) * 2 * kMaxSeg * n, cudaMemcpyHostToDevice,
                      cl.stream) != cudaSuccess ||
      cudaMemcpyAsync(ws + lay.target, target.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, cl.stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(ws + lay.cta_first, cta_first.data(), sizeof(int32_t) * grid, cudaMemcpyHostToDevice,
                      cl.stream) != cudaSuccess ||
      cudaMemsetAsync(ws + lay.done, 0, sizeof(int32_t) * 2 * n, cl.stream) != cudaSuccess)
    return FTB_ERR_LAUNCH;
  CellBatch header;
  header.n_items = n;
  header.n_cols = cl.n_cols;
  header.ld_out = cl.ld_out;
  header.ld_c = cl.ld_c;
  header.total_tiles = tiles;
  header.pad_ = 0;
  PlanView pv = {reinterpret_cast<const CellItem*>(ws + lay.items), reinterpret_cast<const int32_t*>(ws + lay.dep),
                 reinterpret_cast<const int32_t*>(ws + lay.target), reinterpret_cast<int32_t*>(ws + lay.done),
                 nullptr, nullptr, 0, 0, 0, 0, reinterpret_cast<const int32_t*>(ws + lay.cta_first), nullptr};
#ifdef FTB_TRACE
  // Debug build: four time stamps per tile behind the tables, when the caller left room.
  if (ws_bytes >= lay.total + static_cast<size_t>(32) * tiles)
    pv.trace = reinterpret_cast<unsigned long long*>(ws + lay.total);
#endif
  return launch_cell_gemm_persistent(cl.dtype, cl.epi, cl.bn, cl.pair, cl.maps, cl.mapW, cl.mapC, header, pv,
                                     cl.status, cl.sm_count, cl.stream);
}

struct StackedPlanArgs {
  int D, L, N, I, H, G, skew, es, tiles_per_item, m_tiles;
  char* hs;
  float* c;
  const float* bias_p;
  CellItem* items;
  int32_t* dep;
  int32_t* target;
};

// Position of cell (l, t) in the launch order: groups of G layers one after the
// other; inside a group level by level, level m = skew * j + t with j the layer's
// index in the group, lower layers first.  A cell reads (l, t-1), one level back,
// and (l-1, t), `skew` levels back (or in an earlier group): with skew >= 2 the
// input half of a cell's K loop can run while the cells of the previous level,
// which feed its recurrent half, are still finishing.
__device__ int stacked_item_index(const StackedPlanArgs& a, int l, int t) {
  const int g0 = (l / a.G) * a.G;
  const int Lg = min(a.G, a.D - g0);
  const int j = l - g0;
  const int m = a.skew * j + t;
  int before = 0;
  for (int q = 0; q < m; ++q) {
    const int j_lo = (max(0, q - a.L + 1) + a.skew - 1) / a.skew;
    const int j_hi = min(Lg - 1, q / a.skew);
    before += max(0, j_hi - j_lo + 1);
  }
  const int j_min = (max(0, m - a.L + 1) + a.skew - 1) / a.skew;
  return g0 * a.L + before + (j - j_min);
}

__global__ void plan_stacked_kernel(const StackedPlanArgs a) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= a.D * a.L) return;
  const int l = id / a.L, t = id - l * a.L;
  const int pos = stacked_item_index(a, l, t);
  CellItem it;
  for (int s = 0; s < kMaxSeg; ++s) it.seg_row[s] = it.seg_kb[s] = it.seg_wk[s] = it.seg_map[s] = 0;
  int32_t dep[kMaxSeg][2] = {{-1, -1}, {-1, -1}, {-1, -1}};
  int ns = 0;
  if (l == 0) {
    it.seg_map[ns] = 0; it.seg_row[ns] = t * a.N; it.seg_kb[ns] = a.I / 64; it.seg_wk[ns] = 0;
  } else {
    it.seg_map[ns] = 1; it.seg_row[ns] = ((l - 1) * a.L + t) * a.N; it.seg_kb[ns] = a.H / 64; it.seg_wk[ns] = 0;
    dep[ns][0] = dep[ns][1] = stacked_item_index(a, l - 1, t);
  }
  ++ns;
  if (t > 0) {
    it.seg_map[ns] = 2; it.seg_row[ns] = (l * a.L + t - 1) * a.N; it.seg_kb[ns] = a.H / 64; it.seg_wk[ns] = a.I;
    dep[ns][0] = dep[ns][1] = stacked_item_index(a, l, t - 1);
    ++ns;
  }
  it.nseg = ns;
  it.w_row0 = l * 4 * a.H;
  it.rows = a.N;
  it.c_zero = (t == 0);
  it.out = a.hs + (static_cast<size_t>(l) * a.L + t) * a.N * a.H * a.es;
  it.out_row0 = (l * a.L + t) * a.N;
  it.out_map = 1;
  it.w_map = 0;
  it.skip = 0;
  it.pad_ = 0;
  it.c = a.c + static_cast<size_t>(l) * a.N * a.H;
  it.c_row0 = l * a.N;
  it.bias = a.bias_p ? a.bias_p + static_cast<size_t>(l) * 4 * a.H : nullptr;
  it.m_tiles = a.m_tiles;
  it.tile0 = pos * a.tiles_per_item;
  a.items[pos] = it;
  for (int s = 0; s < kMaxSeg; ++s) {
    a.dep[(pos * kMaxSeg + s) * 2 + 0] = dep[s][0];
    a.dep[(pos * kMaxSeg + s) * 2 + 1] = dep[s][1];
  }
  a.target[pos] = 8 * a.tiles_per_item;  // eight epilogue warps per tile
}

// Accumulator tile width.  The last column tile of a cell may be partial (the
// epilogue skips 32-column groups past n_cols), so n_cols % 32 == 0 is enough.
int pick_bn(int n_cols, int want) {
  if (n_cols % 32 != 0) return 0;
  if (want == 128 || want == 256) return want;
  if (want != 0) return 0;
  return (n_cols % 256 == 0 && n_cols >= 2048) ? 256 : 128;
}

}  // namespace
}  // namespace ftb

using namespace ftb;

extern "C" {

int ftb_version(void) { return 1; }

const char* ftb_status_str(int code) {
  switch (code) {
    case FTB_OK: return "ok";
    case FTB_ERR_ARG: return "bad argument (shape, pointer or dtype)";
    case FTB_ERR_ALIGN: return "pointer or stride not 16-byte aligned";
    case FTB_ERR_WORKSPACE: return "workspace missing or too small";
    case FTB_ERR_DRIVER: return "tensor-map encode failed or driver entry point missing";
    case FTB_ERR_LAUNCH: return "kernel launch failed";
    case FTB_ERR_ARCH: return "device is not sm_100";
    case FTB_ERR_SCRATCH_LIMIT: return "problem needs more scratch than the built-in static buffer holds";
    case FTB_ERR_TIMEOUT_TMA: return "device wait ran out: TMA stage never arrived";
    case FTB_ERR_TIMEOUT_MMA: return "device wait ran out: MMA never committed";
    case FTB_ERR_TIMEOUT_EPI: return "device wait ran out: epilogue never drained";
    case FTB_ERR_TIMEOUT_SLOT: return "device wait ran out: no free pipeline stage";
    case FTB_ERR_TIMEOUT_DEP: return "device wait ran out: a cell's inputs never completed";
    case FTB_ERR_TMEM_LAYOUT: return "the two CTAs of a pair got different TMEM columns";
    case FTB_ERR_INDEX: return "an index was outside its table";
    default: return "unknown status";
  }
}

size_t ftb_workspace_bytes(void) { return kWorkspaceBytes; }

long long ftb_launch_count(void) { return launches_so_far(); }

int ftb_read_status(const void* workspace, int* status_out, void* stream) {
  if (workspace == nullptr || status_out == nullptr) return FTB_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cudaMemcpyAsync(status_out, workspace, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return FTB_ERR_LAUNCH;
  if (cudaStreamSynchronize(s) != cudaSuccess) return FTB_ERR_LAUNCH;
  return FTB_OK;
}

int ftb_lstm_pack_weights(const void* W, const void* U, const void* bias, void* Wp, float* bias_p, int D, int I,
                          int H, int dtype, void* stream) {
  if (!W || !U || !Wp || D <= 0 || I <= 0 || H <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (bias != nullptr && bias_p == nullptr) return FTB_ERR_ARG;
  return pack_lstm(W, U, bias, Wp, bias_p, D, I, H, dtype, static_cast<cudaStream_t>(stream));
}

int ftb_grid_pack_weights(const void* i2h, const void* h2h, void* Wp, int H, int dtype, void* stream) {
  if (!i2h || !h2h || !Wp || H <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  return pack_grid(i2h, h2h, Wp, H, dtype, static_cast<cudaStream_t>(stream));
}

// Upper bound of tiles per cell over the tile shapes the library may pick.
static int stacked_max_tiles_per_cell(int N, int H) { return 2 * ((N + 255) / 256) * ((4 * H + 127) / 128); }

// Arrival counters of the lstm_flow kernel, one per cell and batch slice (of 16 sequences or more).
static size_t flow_flag_bytes(int D, int L, int slices) { return sizeof(int) * D * L * static_cast<size_t>(slices); }
constexpr int kMostFlowSlices = 128;  // of a layer: two CTAs or more each

size_t ftb_lstm_stacked_workspace_bytes(int D, int L, int N, int H) {
  if (D <= 0 || L <= 0 || N <= 0 || H <= 0) return kWorkspaceBytes;
  return plan_layout(static_cast<size_t>(D) * L, stacked_max_tiles_per_cell(N, H)).total + flow_flag_bytes(D, L, (N + 15) / 16);
}

// Layers per group of the static-ownership kernels: at most `G` (what L2 holds) and what fits on the
// device at `ctas` CTAs a layer, evened out over the groups.
static int fit_groups(int D, int G, int ctas, int sm_count) {
  const int most = std::min(std::min(G, D), sm_count / ctas);
  if (most < 1) return G;
  const int groups = (D + most - 1) / most;
  return (D + groups - 1) / groups;
}

// About what the 16-bit kernels that stream weights take (us), by groups of G layers: sweeps * (L + G - 1) steps of
// a length fitted to 504 problems (H 128..1024, D 1..16, N 16..256, L 64; within 20 %, 6 % in the root mean
// square).  Measured, us (generic / static / weights on the M side / everything on chip; * taken): D 8, N 200, H 640 928*
// / 1251 / - / 1339; D 12, N 200, H 512 997* / 1191 / - / 1289; D 16, N 256, H 512 1277 / 1030* / - / 1861; D 4, N 256, H 512
// 681 / 512 / - / 452*; D 12, N 160, H 320 870 / 665 / - / 628*; D 12, N 128, H 512 925 / 962 / 821 / 681*; D 12, N 128, H 128
// 509 / 424 / 292 / 232*; D 7, N 15, H 832 1730 / 1327 / 895 / 345*.
struct StackedEstimate {
  int D, L, N, sm_count, m, n_tiles;
  double h;
  StackedEstimate(int D, int L, int N, int H, int sm_count)
      : D(D), L(L), N(N), sm_count(sm_count), m((N + 255) / 256), n_tiles((4 * H + 255) / 256), h(H / 1024.0) {}
  double steps(int G) const { return static_cast<double>((D + G - 1) / G) * (L + G - 1); }
  // one CTA per 128 gate rows; the batch is the N side of the MMA, 16 to 128 wide
  double wmajor(int G) const {
    const double n = (N <= 16 ? 16 : N <= 32 ? 32 : N <= 64 ? 64 : 128) / 128.0;
    return steps(G) * (1.77 + 5.65 * h + 1.1 * n + 1.15 * n * h + 0.45 * (32 * h * G / sm_count));
  }
  // a CTA pair per 256 sequences x 256 gate columns; without full tiles of 128 sequences it stores row by row
  double static_pairs(int G) const {
    const double busy = static_cast<double>(2 * m * n_tiles * G) / sm_count;
    return steps(G) * (N % 128 == 0 ? 6.4 - 0.9 * h + 6.0 * h * h + 3.2 * h * busy : 8.3 + 5.0 * h * h * h + 2.2 * busy);
  }
  double generic(int G) const { return steps(G) * (11.9 + 1.2 * h + 0.23 * m * G); }
};

// Layers whose packed weights stay within about half of L2.
static int l2_group(int D, int H, int K, size_t es) {
  int dev = 0, l2 = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
  const double per_layer = 4.0 * H * K * es;
  if (per_layer * D <= 0.55 * l2) return D;
  return std::max(1, std::min(static_cast<int>((0.55 * l2) / per_layer), D));
}

// What a 16-bit stacked call may run, and what it takes of that when no schedule is named.
struct StackedChoice {
  int Gw, Gs;  // layers per group
  bool can_wmajor, can_static, take_static, can_flow, on_chip;
  FlowPlan flow;
};
static StackedChoice stacked_choice(int dtype, int D, int L, int N, int I, int H, int G, const Tuning& tune, int sm_count) {
  StackedChoice ch;
  // Static tile ownership (schedule 3, and the automatic choice when it applies): CTA pairs
  // keep their slice of a layer, cell state in registers, for a whole sweep over time.
  // Weights-major static ownership (schedule 4, and the automatic choice for batches of at most
  // 128 sequences): the batch is the N side of the MMA, so a small batch wastes no tensor work.
  const int pair_ctas = 2 * ((N + 255) / 256) * ((4 * H + 255) / 256);
  ch.Gw = tune.layers_per_group > 0 ? G : fit_groups(D, G, 4 * H / 128, sm_count);
  ch.can_wmajor = lstm_wmajor_supported(dtype, D, N, I, H, ch.Gw, sm_count);
  ch.Gs = tune.layers_per_group > 0 ? G : fit_groups(D, G, pair_ctas, sm_count);
  ch.can_static = tune.pair != 1 && (tune.bn == 0 || tune.bn == 256) && !tune.fine_deps &&
                  lstm_static_supported(dtype, D, N, I, H, ch.Gs, sm_count);
  // Everything on chip: schedule 5, and the automatic choice where that is expected to be faster (with a part of the
  // input weights read from L2 every step if need be).
  ch.can_flow = tune.layers_per_group == 0 && lstm_flow_plan(dtype, D, L, N, static_cast<int64_t>(L) * N, I, H, sm_count,
                                                             tune.schedule != 5, &ch.flow);
  const StackedEstimate est(D, L, N, H, sm_count);
  const double wmajor_us = est.wmajor(ch.Gw), static_us = est.static_pairs(ch.Gs), generic_us = est.generic(G);
  // Groups that had to be cut to what fits on the device, for static ownership, are more sweeps than those of the
  // generic kernel, which takes groups of any size.
  ch.take_static = ch.can_static && (pair_ctas * G <= sm_count || static_us < 1.03 * generic_us);
  const double old_us = ch.can_wmajor ? wmajor_us : (ch.take_static ? static_us : generic_us);
  // (Of 5277 calls the choice by these estimates is 0.3 % behind the fastest kernel on average; with the kernel with weights on chip
  // a twentieth behind, as it had to come out while it was estimated too high, 143 calls were more than 10 % behind, now 21.  8 us:
  // the others are estimated a little low on small calls.)
  ch.on_chip = ch.can_flow && ch.flow.est_us < old_us + 8.0;
  return ch;
}

int ftb_lstm_stacked_form(int D, int L, int N, int I, int H, int dtype, int* form) {
  if (!form || D <= 0 || L <= 0 || N <= 0 || H <= 0 || I <= 0 || H % 64 != 0 || I % 64 != 0 || (D > 1 && I != H)) return FTB_ERR_ARG;
  if (dtype != FTB_F16 && dtype != FTB_BF16) return FTB_ERR_ARG;
  const StackedChoice ch = stacked_choice(dtype, D, L, N, I, H, l2_group(D, H, I + H, dtype_size(dtype)), Tuning(nullptr),
                                          current_sm_count());
  form[0] = ch.on_chip ? 5 : (ch.can_wmajor ? 4 : (ch.take_static ? 3 : 2));
  form[1] = ch.on_chip ? ch.flow.nb : 0;
  form[2] = ch.on_chip ? (ch.flow.pair ? 2 : 1) : 0;
  form[3] = ch.on_chip ? ch.flow.ring : 0;
  return FTB_OK;
}

int ftb_lstm_stacked_fwd(const void* x, const void* Wp, const float* bias_p, void* hs, float* c, int D, int L,
                         int N, int I, int H, int dtype, const int* tuning, void* workspace, size_t workspace_bytes,
                         void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const Tuning tune(tuning);
  const int layers_per_group = tune.layers_per_group, bn = tune.bn, schedule = tune.schedule, skew = tune.skew;
  if (!x || !Wp || !hs || !c || D <= 0 || L <= 0 || N <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (H <= 0 || I <= 0 || H % 64 != 0 || I % 64 != 0) return FTB_ERR_ARG;
  if (D > 1 && I != H) return FTB_ERR_ARG;
  if (static_cast<int64_t>(D) * L * N > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({x, Wp, bias_p, hs, c})) return FTB_ERR_ALIGN;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;

  const int K = I + H;
  const size_t es = dtype_size(dtype);
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_LSTM;
  cl.n_cols = 4 * H;
  cl.ld_out = H;
  cl.ld_c = H;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  if (dtype == FTB_F32) {
    cl.act[0] = static_cast<const float*>(x);
    cl.ld_act[0] = I;
    cl.act[1] = cl.act[2] = static_cast<const float*>(hs);
    cl.ld_act[1] = cl.ld_act[2] = H;
    cl.w = static_cast<const float*>(Wp);
    cl.ldw = K;
  } else {
    cl.bn = pick_bn(4 * H, bn);
    if (cl.bn == 0) return FTB_ERR_ARG;
    cl.pair = tune.use_pair(N);
    rc = make_tmap_2d(&cl.maps[0], x, dtype, static_cast<uint64_t>(L) * N, I, I, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[1], hs, dtype, static_cast<uint64_t>(D) * L * N, H, H, 128, 64);
    if (rc) return rc;
    cl.maps[2] = cl.maps[1];
    cl.maps[3] = cl.maps[0];
    rc = make_tmap_2d(&cl.mapW, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, K, K, cl.w_box_rows(), 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapC, c, FTB_F32, static_cast<uint64_t>(D) * N, H, H, 128, 32);
    if (rc) return rc;
  }

  const int G = layers_per_group > 0 ? std::min(layers_per_group, D) : l2_group(D, H, K, es);

  const int n_cells = D * L;
  const PlanLayout lay = plan_layout(n_cells, stacked_max_tiles_per_cell(N, H));
  if (dtype == FTB_F32 && schedule != 1 && (schedule >= 2 || workspace_bytes >= lay.total)) {
    // fp32: one persistent launch, a CTA per accumulator tile with its weights in shared memory
    // (csrc/lstm_simt_static.cu), when a layer's tiles fit on the device.
    if (workspace_bytes < lay.total) return FTB_ERR_WORKSPACE;
    const bool can = lstm_simt_static_supported(D, N, I, H, cl.sm_count);
    if (schedule >= 2 && !can) return FTB_ERR_ARG;
    if (can) {
      // With I == H there is also the kernel whose states carry their own arrival (csrc/lstm_simt_flow.cu; schedule
      // 5 names it, 2 to 4 the other one).  A step of its is shorter, but its tiles need more CTAs where 32 rows do
      // not fit beside the weights (H of 320 and more) or the batch is large, and layers that do not fit beside each
      // other cost a sweep each: the automatic choice takes the one with the smaller estimate (us, this one / the other,
      // L 64: D 3, N 32 at H 256 367 / 517, at H 320 859 / 626; D 3, N 16, H 320 315 / 580; D 3, N 200, H 64 487 / 507).
      SimtFlowPlan flow;
      const bool can_flow = lstm_simt_flow_plan(D, L, N, I, H, cl.sm_count, &flow);
      if (can_flow && (schedule == 5 || (schedule == 0 && flow.est_us < lstm_simt_static_us(D, L, N, I, H, cl.sm_count))))
        rc = launch_lstm_simt_flow(static_cast<const float*>(x), static_cast<const float*>(Wp), bias_p,
                                   static_cast<float*>(hs), c, D, L, N, H, flow, status, cl.sm_count, stream);
      else
        rc = launch_lstm_simt_static(static_cast<const float*>(x), static_cast<const float*>(Wp), bias_p,
                                     static_cast<float*>(hs), c, D, L, N, I, H,
                                     reinterpret_cast<int*>(static_cast<char*>(workspace) + lay.done), status,
                                     cl.sm_count, stream);
      // A refused cooperative launch falls back to one launch per level under the automatic choice.
      if (rc != FTB_ERR_LAUNCH || schedule != 0) return rc;
    }
  }
  const bool persistent = dtype != FTB_F32 && schedule != 1 && (schedule >= 2 || workspace_bytes >= lay.total);
  if (persistent) {
    if (workspace_bytes < lay.total) return FTB_ERR_WORKSPACE;
    char* ws = static_cast<char*>(workspace);
    const StackedChoice ch = stacked_choice(dtype, D, L, N, I, H, G, tune, cl.sm_count);
    const bool can_flow = ch.can_flow && workspace_bytes >= lay.total + flow_flag_bytes(D, L, ch.flow.S);
    if (schedule == 5 && !can_flow) return FTB_ERR_ARG;
    if (schedule == 5 || (schedule == 0 && can_flow && ch.on_chip && tune.pair == 0 && bn == 0 && !tune.fine_deps)) {
      rc = launch_lstm_flow(dtype, x, Wp, bias_p, hs, c, nullptr, static_cast<int64_t>(L) * N, D, L, N, I, H, ch.flow,
                            reinterpret_cast<int*>(ws + lay.total), status, stream);
      if (rc != FTB_ERR_LAUNCH || schedule != 0) return rc;
      goto level_schedule;
    }
    if (schedule == 4 && !ch.can_wmajor) return FTB_ERR_ARG;
    if (schedule == 4 || (schedule == 0 && ch.can_wmajor && tune.pair == 0 && bn == 0 && !tune.fine_deps)) {
      // tuning[6]: 0 = as many recurrent weight blocks on chip as fit, -1 = none, n = n blocks
      const int resident = tune.resident == 0 ? -1 : (tune.resident < 0 ? 0 : tune.resident);
      unsigned long long* trace = nullptr;
#ifdef FTB_TRACE
      trace = reinterpret_cast<unsigned long long*>(ws + lay.trace);
#endif
      // one flag per (cell, tile), in the per-tile counter area (at least 4H/128 ints per cell)
      rc = launch_lstm_wmajor(dtype, x, Wp, bias_p, hs, c, D, L, N, I, H, ch.Gw, resident,
                              reinterpret_cast<int*>(ws + lay.tile_done), status, trace, stream);
      if (rc != FTB_ERR_LAUNCH || schedule != 0) return rc;
      goto level_schedule;
    }
    if (schedule == 3 && !ch.can_static) return FTB_ERR_ARG;
    if (schedule == 3 || (schedule == 0 && ch.take_static)) {
      unsigned long long* trace = nullptr;
#ifdef FTB_TRACE
      trace = reinterpret_cast<unsigned long long*>(ws + lay.trace);
#endif
      rc = launch_lstm_static(dtype, x, Wp, bias_p, hs, c, D, L, N, I, H, ch.Gs,
                              reinterpret_cast<int*>(ws + lay.done), status, trace, stream);
      // A cooperative launch can be refused (device shared through MPS, SMs reserved, ...).
      // With an explicit schedule that is the caller's error to see; the automatic choice
      // falls back to one launch per level, which needs no co-residency.
      if (rc != FTB_ERR_LAUNCH || schedule != 0) return rc;
      goto level_schedule;
    }
    StackedPlanArgs pa;
    pa.D = D; pa.L = L; pa.N = N; pa.I = I; pa.H = H; pa.G = G; pa.es = static_cast<int>(es);
    pa.skew = skew > 0 ? skew : 1;
    pa.m_tiles = cl.m_tiles_for(N);
    pa.tiles_per_item = pa.m_tiles * ((4 * H + cl.bn - 1) / cl.bn);
    pa.hs = static_cast<char*>(hs);
    pa.c = c;
    pa.bias_p = bias_p;
    pa.items = reinterpret_cast<CellItem*>(ws + lay.items);
    pa.dep = reinterpret_cast<int32_t*>(ws + lay.dep);
    pa.target = reinterpret_cast<int32_t*>(ws + lay.target);
    int32_t* done = reinterpret_cast<int32_t*>(ws + lay.done);
    if (cudaMemsetAsync(done, 0, lay.counters_end - lay.done, stream) != cudaSuccess) return FTB_ERR_LAUNCH;
    plan_stacked_kernel<<<(n_cells + 127) / 128, 128, 0, stream>>>(pa);
    if (cudaGetLastError() != cudaSuccess) return FTB_ERR_LAUNCH;
    count_launch();
    CellBatch header;
    header.n_items = n_cells;
    header.n_cols = 4 * H;
    header.ld_out = H;
    header.ld_c = H;
    header.total_tiles = n_cells * pa.tiles_per_item;
    header.pad_ = 0;
    PlanView pv = {pa.items, pa.dep, pa.target, done, reinterpret_cast<int32_t*>(ws + lay.tile_done),
                   reinterpret_cast<int32_t*>(ws + lay.c_done), tune.fine_deps == 1 ? 1 : 0, cl.bn / 4,
                   pa.tiles_per_item, 0, nullptr, nullptr};
#ifdef FTB_TRACE
    pv.trace = reinterpret_cast<unsigned long long*>(ws + lay.trace);
#endif
    rc = launch_cell_gemm_persistent(dtype, EPI_LSTM, cl.bn, cl.pair, cl.maps, cl.mapW, cl.mapC, header, pv,
                                     status, cl.sm_count, stream);
    if (rc != FTB_ERR_LAUNCH || schedule != 0) return rc;
  }

level_schedule:
  std::vector<CellItem> items;
  for (int g0 = 0; g0 < D; g0 += G) {
    const int Lg = std::min(G, D - g0);
    for (int m = 0; m < Lg + L - 1; ++m) {
      items.clear();
      for (int l = g0; l < g0 + Lg; ++l) {
        const int t = m - (l - g0);
        if (t < 0 || t >= L) continue;
        CellItem it = blank_item();
        if (l == 0)
          add_seg(it, 0, static_cast<int64_t>(t) * N, I, 0);
        else
          add_seg(it, 1, (static_cast<int64_t>(l - 1) * L + t) * N, H, 0);
        if (t > 0) add_seg(it, 2, (static_cast<int64_t>(l) * L + t - 1) * N, H, I);
        it.w_row0 = l * 4 * H;
        it.rows = N;
        it.c_zero = (t == 0);
        it.out = static_cast<char*>(hs) + (static_cast<size_t>(l) * L + t) * N * H * es;
        it.out_row0 = static_cast<int32_t>((static_cast<int64_t>(l) * L + t) * N);
        it.out_map = 1;
        it.c = c + static_cast<size_t>(l) * N * H;
        it.c_row0 = l * N;
        it.bias = bias_p ? bias_p + static_cast<size_t>(l) * 4 * H : nullptr;
        items.push_back(it);
      }
      rc = cl.run(items);
      if (rc) return rc;
    }
  }
  return FTB_OK;
}

// first_rows: the first row of every step and their number, [L + 1], on the device already, or nullptr.
static int stacked_varlen(const void* x, const void* Wp, const float* bias_p, void* hs, float* c, const int* active_rows,
                          const int* first_rows, int D, int L, int I, int H, int dtype, const int* tuning, void* workspace,
                          size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const Tuning tune(tuning);
  if (!x || !Wp || !hs || !c || !active_rows || D <= 0 || L <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (H <= 0 || I <= 0 || H % 64 != 0 || I % 64 != 0) return FTB_ERR_ARG;
  if (D > 1 && I != H) return FTB_ERR_ARG;
  // Row offset of every step in the packed buffers; the batch must be sorted by decreasing length.
  std::vector<int64_t> off(L + 1, 0);
  for (int t = 0; t < L; ++t) {
    if (active_rows[t] <= 0 || (t > 0 && active_rows[t] > active_rows[t - 1])) return FTB_ERR_ARG;
    off[t + 1] = off[t] + active_rows[t];
  }
  const int64_t T = off[L];
  const int N = active_rows[0];
  if (static_cast<int64_t>(D) * T > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({x, Wp, bias_p, hs, c})) return FTB_ERR_ALIGN;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;

  const int K = I + H;
  const size_t es = dtype_size(dtype);
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_LSTM;
  cl.n_cols = 4 * H;
  cl.ld_out = H;
  cl.ld_c = H;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  if (dtype == FTB_F32) {
    cl.act[0] = static_cast<const float*>(x);
    cl.ld_act[0] = I;
    cl.act[1] = cl.act[2] = static_cast<const float*>(hs);
    cl.ld_act[1] = cl.ld_act[2] = H;
    cl.w = static_cast<const float*>(Wp);
    cl.ldw = K;
  } else {
    cl.bn = pick_bn(4 * H, tune.bn);
    if (cl.bn == 0) return FTB_ERR_ARG;
    cl.pair = tune.use_pair(N);
    rc = make_tmap_2d(&cl.maps[0], x, dtype, static_cast<uint64_t>(T), I, I, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[1], hs, dtype, static_cast<uint64_t>(D) * T, H, H, 128, 64);
    if (rc) return rc;
    cl.maps[2] = cl.maps[1];
    cl.maps[3] = cl.maps[0];
    rc = make_tmap_2d(&cl.mapW, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, K, K, cl.w_box_rows(), 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapC, c, FTB_F32, static_cast<uint64_t>(D) * N, H, H, 128, 32);
    if (rc) return rc;
  }

  // Layers run in groups whose packed weights stay in L2, as in the rectangular entry point.
  int G = tune.layers_per_group;
  if (G <= 0) {
    int dev = 0, l2 = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
    const double per_layer = 4.0 * H * K * es;
    G = static_cast<int>((0.55 * l2) / per_layer);
    G = std::max(1, G);
  }
  G = std::min(G, D);

  // Cell (l, t) holds the active_rows[t] sequences still running: it reads the layer below (or
  // x) at step t and the first active_rows[t] rows of its own layer's step t-1.
  auto make_item = [&](int l, int t) {
    CellItem it = blank_item();
    if (l == 0)
      add_seg(it, 0, off[t], I, 0);
    else
      add_seg(it, 1, static_cast<int64_t>(l - 1) * T + off[t], H, 0);
    if (t > 0) add_seg(it, 2, static_cast<int64_t>(l) * T + off[t - 1], H, I);
    it.w_row0 = l * 4 * H;
    it.rows = active_rows[t];
    it.c_zero = (t == 0);
    it.out = static_cast<char*>(hs) + (static_cast<size_t>(l) * T + off[t]) * H * es;
    it.out_row0 = static_cast<int32_t>(static_cast<int64_t>(l) * T + off[t]);
    it.out_map = 1;
    it.c = c + static_cast<size_t>(l) * N * H;
    it.c_row0 = l * N;
    it.bias = bias_p ? bias_p + static_cast<size_t>(l) * 4 * H : nullptr;
    return it;
  };

  const int n_cells = D * L;
  const PlanLayout lay = plan_layout(n_cells, 0);
  // Everything on chip (csrc/lstm_flow.cu): the first rows of the steps and the arrival counters sit
  // behind the tables of the generic schedule.
  FlowPlan flow;
  const size_t off_bytes = (sizeof(int) * (L + 1) + 255) & ~static_cast<size_t>(255);
  const bool can_flow = tune.layers_per_group == 0 && tune.pair == 0 && tune.bn == 0 &&
                        lstm_flow_plan(dtype, D, L, N, T, I, H, cl.sm_count, tune.schedule != 5, &flow) &&
                        workspace_bytes >= lay.total + off_bytes + flow_flag_bytes(D, L, flow.S);
  if (tune.schedule == 5 && !can_flow) return FTB_ERR_ARG;
  // the generic schedule takes about 14 us a step and group of layers at any size
  if (tune.schedule == 5 || (tune.schedule == 0 && can_flow && flow.est_us < ((D + G - 1) / G) * (L + G - 1) * 10.0)) {
    char* ws = static_cast<char*>(workspace);
    if (first_rows == nullptr) {
      std::vector<int> first(off.begin(), off.end());
      if (cudaMemcpyAsync(ws + lay.total, first.data(), sizeof(int) * (L + 1), cudaMemcpyHostToDevice, stream) != cudaSuccess)
        return FTB_ERR_LAUNCH;
      first_rows = reinterpret_cast<int*>(ws + lay.total);
    }
    rc = launch_lstm_flow(dtype, x, Wp, bias_p, hs, c, first_rows, T, D, L, N, I, H, flow,
                          reinterpret_cast<int*>(ws + lay.total + off_bytes), status, stream);
    if (rc != FTB_ERR_LAUNCH || tune.schedule != 0) return rc;
  }
  bool persistent = dtype != FTB_F32 && tune.schedule != 1 && (tune.schedule >= 2 || workspace_bytes >= lay.total);
  if (persistent) {
    if (workspace_bytes < lay.total) return FTB_ERR_WORKSPACE;
    // One persistent launch over the steps [t0, t1) of every layer.  Launch order: group by
    // group, level by level (level = layer-in-group + step), so every cell comes after the two
    // it reads; cells of earlier steps belong to an earlier launch on the stream and count as
    // inputs.
    auto run_range = [&](const CellLauncher& launcher, int t0, int t1) -> int {
      const int Lr = t1 - t0;
      std::vector<CellItem> order;
      order.reserve(static_cast<size_t>(D) * Lr);
      std::vector<int> index_of(static_cast<size_t>(D) * Lr, -1);
      for (int g0 = 0; g0 < D; g0 += G) {
        const int Lg = std::min(G, D - g0);
        for (int m = 0; m < Lg + Lr - 1; ++m)
          for (int l = g0; l < g0 + Lg; ++l) {
            const int t = m - (l - g0);
            if (t < 0 || t >= Lr) continue;
            index_of[l * Lr + t] = static_cast<int>(order.size());
            order.push_back(make_item(l, t0 + t));
          }
      }
      std::vector<int32_t> deps(order.size() * kMaxSeg * 2, -1);
      for (int l = 0; l < D; ++l)
        for (int t = 0; t < Lr; ++t) {
          const int me = index_of[l * Lr + t];
          if (l > 0)
            deps[(me * kMaxSeg + 0) * 2 + 0] = deps[(me * kMaxSeg + 0) * 2 + 1] = index_of[(l - 1) * Lr + t];
          if (t > 0) deps[(me * kMaxSeg + 1) * 2 + 0] = deps[(me * kMaxSeg + 1) * 2 + 1] = index_of[l * Lr + t - 1];
        }
      return run_persistent(launcher, order, deps, static_cast<char*>(workspace), lay, workspace_bytes);
    };
    // Once the batch has shrunk to one 128-row tile, a CTA pair would multiply 128 rows of
    // padding with every weight tile.  From that step on the cells run as single CTAs on
    // 128-column tiles (same bytes per CTA and K block, half the tensor work, twice the tiles):
    // the time axis is cut there into two launches.  Only when the caller left the tile shape open.
    int t_split = L;
    if (cl.pair && tune.pair == 0 && tune.bn == 0 && tune.schedule == 0)
      for (int t = 0; t < L; ++t)
        if (active_rows[t] <= 128) {
          t_split = t;
          break;
        }
    rc = FTB_OK;
    if (t_split > 0) rc = run_range(cl, 0, t_split);
    if (rc == FTB_OK && t_split < L) {
      CellLauncher single = cl;
      single.pair = 0;
      single.bn = 128;
      rc = make_tmap_2d(&single.mapW, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, K, K, single.w_box_rows(), 64);
      if (rc) return rc;
      rc = run_range(single, t_split, L);
    }
    if (rc != FTB_ERR_LAUNCH || tune.schedule != 0) return rc;
    // A refused cooperative launch falls back to one launch per level (which recomputes every cell).
  }

  std::vector<CellItem> items;
  for (int g0 = 0; g0 < D; g0 += G) {
    const int Lg = std::min(G, D - g0);
    for (int m = 0; m < Lg + L - 1; ++m) {
      items.clear();
      for (int l = g0; l < g0 + Lg; ++l) {
        const int t = m - (l - g0);
        if (t < 0 || t >= L) continue;
        items.push_back(make_item(l, t));
      }
      rc = cl.run(items);
      if (rc) return rc;
    }
  }
  return FTB_OK;
}

int ftb_lstm_stacked_varlen_fwd(const void* x, const void* Wp, const float* bias_p, void* hs, float* c,
                                const int* active_rows, int D, int L, int I, int H, int dtype, const int* tuning,
                                void* workspace, size_t workspace_bytes, void* stream) {
  return stacked_varlen(x, Wp, bias_p, hs, c, active_rows, nullptr, D, L, I, H, dtype, tuning, workspace, workspace_bytes, stream);
}

int ftb_lstm_flow_form_fwd(const void* x, const void* Wp, const float* bias_p, void* hs, float* c, const int* active_rows,
                           int D, int L, int N, int I, int H, int dtype, int nb, int pair, int ring, void* workspace,
                           size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!x || !Wp || !hs || !c || D <= 0 || L <= 0 || N <= 0 || H <= 0 || I <= 0) return FTB_ERR_ARG;
  if (!aligned16({x, Wp, bias_p, hs, c})) return FTB_ERR_ALIGN;
  std::vector<int> first(L + 1, 0);
  for (int t = 0; t < L; ++t) {
    const int rows = active_rows != nullptr ? active_rows[t] : N;
    if (rows <= 0 || rows > (t > 0 && active_rows != nullptr ? active_rows[t - 1] : N) || (t == 0 && rows != N)) return FTB_ERR_ARG;
    if (static_cast<int64_t>(D) * (first[t] + static_cast<int64_t>(rows)) > 0x7fffffffLL) return FTB_ERR_ARG;
    first[t + 1] = first[t] + rows;
  }
  FlowPlan flow;
  if (!lstm_flow_form(dtype, D, N, I, H, current_sm_count(), nb, pair == 2, ring != 0, &flow)) return FTB_ERR_ARG;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;
  const size_t table = (sizeof(int) * (L + 1) + 255) & ~static_cast<size_t>(255);
  if (workspace_bytes < kWorkspaceBytes + table + flow_flag_bytes(D, L, flow.S)) return FTB_ERR_WORKSPACE;
  int* off = reinterpret_cast<int*>(static_cast<char*>(workspace) + kWorkspaceBytes);
  if (active_rows != nullptr &&
      cudaMemcpyAsync(off, first.data(), sizeof(int) * (L + 1), cudaMemcpyHostToDevice, stream) != cudaSuccess)
    return FTB_ERR_LAUNCH;
  return launch_lstm_flow(dtype, x, Wp, bias_p, hs, c, active_rows != nullptr ? off : nullptr, first[L], D, L, N, I, H, flow,
                          off + table / sizeof(int), status, stream);
}

// Row tables of a ragged batch.
size_t ftb_lstm_stacked_ragged_scratch_bytes(int L, int N) {
  return L <= 0 || N <= 0 ? 0 : sizeof(int) * (static_cast<size_t>(L) + 1 + N);
}

// With no scratch they go behind the workspace of the packed entry point.
size_t ftb_lstm_stacked_ragged_workspace_bytes(int D, int L, int N) {
  if (D <= 0 || L <= 0 || N <= 0) return kWorkspaceBytes;
  return ftb_lstm_stacked_varlen_workspace_bytes(D, L) + ftb_lstm_stacked_ragged_scratch_bytes(L, N) + 16;
}

int ftb_lstm_stacked_ragged_fwd(const void* x, const void* Wp, const float* bias_p, const int* lens, void* xt, void* hs,
                                float* c, void* out, int D, int N, int I, int H, int dtype, void* workspace,
                                size_t workspace_bytes, void* stream) {
  return ftb_lstm_stacked_ragged_fwd_scratch(x, Wp, bias_p, lens, xt, hs, c, out, D, N, I, H, dtype, nullptr, 0, workspace,
                                             workspace_bytes, stream);
}

int ftb_lstm_stacked_ragged_fwd_scratch(const void* x, const void* Wp, const float* bias_p, const int* lens, void* xt,
                                        void* hs, float* c, void* out, int D, int N, int I, int H, int dtype,
                                        void* scratch, size_t scratch_bytes, void* workspace, size_t workspace_bytes,
                                        void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!x || !Wp || !lens || !xt || !hs || !c || !out || D <= 0 || N <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (H <= 0 || I <= 0 || H % 64 != 0 || I % 64 != 0 || (D > 1 && I != H)) return FTB_ERR_ARG;
  int L = 0;
  int64_t T = 0;
  for (int n = 0; n < N; ++n) {
    if (lens[n] <= 0) return FTB_ERR_ARG;
    L = std::max(L, lens[n]);
    T += lens[n];
  }
  if (static_cast<int64_t>(D) * T > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({x, Wp, bias_p, xt, hs, c, out, scratch})) return FTB_ERR_ALIGN;
  const size_t packed_bytes = ftb_lstm_stacked_varlen_workspace_bytes(D, L);
  if (workspace == nullptr ||
      workspace_bytes < (scratch != nullptr ? packed_bytes : ftb_lstm_stacked_ragged_workspace_bytes(D, L, N)))
    return FTB_ERR_WORKSPACE;
  if (scratch != nullptr && scratch_bytes < ftb_lstm_stacked_ragged_scratch_bytes(L, N)) return FTB_ERR_WORKSPACE;
  int rc = check_device_sm100();
  if (rc) return rc;
  // The tables are copied from memory that ends with the call: in a graph every replay would read what is there then,
  // and the rows would go by it.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) {
    cudaGetLastError();
    return FTB_ERR_LAUNCH;
  }
  if (capture != cudaStreamCaptureStatusNone) return FTB_ERR_ARG;
  // Sequences by decreasing length (equal ones in their order): active[t] of them are longer than t, and those of
  // length n go to the places from active[n] on.
  std::vector<int> active(static_cast<size_t>(L) + 1, 0), table(static_cast<size_t>(L) + 1 + N);
  for (int n = 0; n < N; ++n) ++active[lens[n] - 1];
  for (int t = L - 1; t > 0; --t) active[t - 1] += active[t];
  int* off = table.data();
  int* start = off + L + 1;
  off[0] = 0;
  for (int t = 0; t < L; ++t) off[t + 1] = off[t] + active[t];
  {
    std::vector<int> place(active.begin() + 1, active.end());  // [n - 1]: of the next sequence of length n
    int row = 0;
    for (int n = 0; n < N; ++n) {
      start[place[lens[n] - 1]++] = row;
      row += lens[n];
    }
  }
  int* d_off = scratch != nullptr ? static_cast<int*>(scratch)
                                  : reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(workspace) + packed_bytes + 15) &
                                                           ~static_cast<uintptr_t>(15));
  const int* d_start = d_off + L + 1;
  if (cudaMemcpyAsync(d_off, table.data(), sizeof(int) * table.size(), cudaMemcpyHostToDevice, stream) != cudaSuccess)
    return FTB_ERR_LAUNCH;
  const long long es = static_cast<long long>(dtype_size(dtype));
  rc = launch_ragged_rows(x, xt, d_start, d_off, N, L, I * es, true, stream);
  if (rc) return rc;
  rc = stacked_varlen(xt, Wp, bias_p, hs, c, active.data(), d_off, D, L, I, H, dtype, nullptr, workspace, packed_bytes, stream_);
  if (rc) return rc;
  return launch_ragged_rows(static_cast<const char*>(hs) + static_cast<size_t>(D - 1) * T * H * es, out, d_start, d_off, N, L,
                            H * es, false, stream);
}

size_t ftb_lstm_stacked_varlen_workspace_bytes(int D, int L) {
  if (D <= 0 || L <= 0) return kWorkspaceBytes;
  // tables of the generic schedule; first rows of the steps and arrival counters of the on-chip one
  return plan_layout(static_cast<size_t>(D) * L, 0).total + sizeof(int) * (static_cast<size_t>(L) + 1) + 256 + flow_flag_bytes(D, L, kMostFlowSlices);
}

int ftb_lstm_dilated_fwd(const void* x, const void* Wp, const float* bias_p, void* hs, float* c,
                         const int* dilations, int D, int L, int N, int H, int dtype, const int* tuning,
                         void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const Tuning tune(tuning);
  const int bn = tune.bn;
  if (!x || !Wp || !hs || !c || !dilations || D <= 0 || L <= 0 || N <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (H <= 0 || H % 64 != 0) return FTB_ERR_ARG;
  int max_dil = 1;
  for (int l = 0; l < D; ++l) {
    if (dilations[l] <= 0) return FTB_ERR_ARG;
    max_dil = std::max(max_dil, dilations[l]);
  }
  if (static_cast<int64_t>(D) * L * N > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({x, Wp, bias_p, hs, c})) return FTB_ERR_ALIGN;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;

  const int K = 2 * H;
  const size_t es = dtype_size(dtype);
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_LSTM;
  cl.n_cols = 4 * H;
  cl.ld_out = H;
  cl.ld_c = H;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  if (dtype == FTB_F32) {
    cl.act[0] = static_cast<const float*>(x);
    cl.act[1] = cl.act[2] = static_cast<const float*>(hs);
    cl.ld_act[0] = cl.ld_act[1] = cl.ld_act[2] = H;
    cl.w = static_cast<const float*>(Wp);
    cl.ldw = K;
  } else {
    cl.bn = pick_bn(4 * H, bn);
    if (cl.bn == 0) return FTB_ERR_ARG;
    cl.pair = tune.pair == 2;  // cells here are latency-bound: single CTAs measured faster than pairs
    rc = make_tmap_2d(&cl.maps[0], x, dtype, static_cast<uint64_t>(L) * N, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[1], hs, dtype, static_cast<uint64_t>(D) * L * N, H, H, 128, 64);
    if (rc) return rc;
    cl.maps[2] = cl.maps[1];
    cl.maps[3] = cl.maps[0];
    rc = make_tmap_2d(&cl.mapW, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, K, K, cl.w_box_rows(), 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapC, c, FTB_F32, static_cast<uint64_t>(D) * max_dil * N, H, H, 128, 32);
    if (rc) return rc;
  }

  // Schedules 4 and 5, and the automatic choice when one applies: a chain of CTAs per (layer, batch slice), weights
  // resident in tensor memory, the state of a layer with dilation 1 handed on through the shared memory of a
  // thread-block cluster (4) or, without clusters, through the output array (5).  Their counters sit behind the
  // tables of the generic persistent schedule in the workspace.
  {
    const size_t flags_off = plan_layout(D * L, 0).total;
    const size_t need = flags_off + sizeof(int) * lstm_dilated_cluster_flag_ints(D, L);
    const bool can = lstm_dilated_cluster_supported(dtype, D, N, H, cl.sm_count) && tune.pair == 0 && bn == 0;
    if (tune.schedule == 4 && (!can || workspace_bytes < need)) return can ? FTB_ERR_WORKSPACE : FTB_ERR_ARG;
    if ((tune.schedule == 4 || tune.schedule == 5 || tune.schedule == 0) && can && workspace_bytes >= need) {
      rc = launch_lstm_dilated_cluster(dtype, x, Wp, bias_p, hs, c, dilations, D, L, N, H, tune.schedule,
                                       reinterpret_cast<int*>(static_cast<char*>(workspace) + flags_off), status,
                                       cl.sm_count, stream);
      // A refused cooperative launch falls back to the generic wavefront under the automatic choice, as does schedule 5
      // where it does not apply.
      if (rc != (tune.schedule == 5 ? FTB_ERR_ARG : FTB_ERR_LAUNCH) || tune.schedule == 4) return rc;
    }
  }

  // Layer l advances in steps of dilations[l] consecutive timesteps: those
  // timesteps only depend on the step before (same layer) and on the layer
  // below, so one step is one cell of batch dilation*N.  Earliest-start levels.
  std::map<int, std::vector<CellItem>> levels;
  std::map<int, std::vector<std::pair<int, int>>> level_ids;  // (layer, step) of each item, same order
  std::vector<std::vector<int>> level_of(D);
  for (int l = 0; l < D; ++l) {
    const int dl = dilations[l];
    const int steps = (L + dl - 1) / dl;
    level_of[l].resize(steps);
    for (int s = 0; s < steps; ++s) {
      const int t0 = s * dl;
      const int t1 = std::min(L, t0 + dl);
      int lv = 0;
      if (s > 0) lv = level_of[l][s - 1] + 1;
      if (l > 0) {
        const int below = (t1 - 1) / dilations[l - 1];
        lv = std::max(lv, level_of[l - 1][below] + 1);
      }
      level_of[l][s] = lv;
      CellItem it = blank_item();
      if (l == 0)
        add_seg(it, 0, static_cast<int64_t>(t0) * N, H, 0);
      else
        add_seg(it, 1, (static_cast<int64_t>(l - 1) * L + t0) * N, H, 0);
      if (s > 0) add_seg(it, 2, (static_cast<int64_t>(l) * L + t0 - dl) * N, H, H);
      it.w_row0 = l * 4 * H;
      it.rows = (t1 - t0) * N;
      it.c_zero = (s == 0);
      it.out = static_cast<char*>(hs) + (static_cast<size_t>(l) * L + t0) * N * H * es;
      it.out_row0 = static_cast<int32_t>((static_cast<int64_t>(l) * L + t0) * N);
      it.out_map = 1;
      it.c = c + static_cast<size_t>(l) * max_dil * N * H;
      it.c_row0 = l * max_dil * N;
      it.bias = bias_p ? bias_p + static_cast<size_t>(l) * 4 * H : nullptr;
      levels[lv].push_back(it);
      level_ids[lv].push_back(std::make_pair(l, s));
    }
  }
  int n_items = 0;
  for (auto& kv : levels) n_items += static_cast<int>(kv.second.size());
  const PlanLayout lay = plan_layout(n_items, 0);
  const bool persistent = dtype != FTB_F32 && tune.schedule != 1 && (tune.schedule >= 2 || workspace_bytes >= lay.total);
  if (persistent) {
    if (workspace_bytes < lay.total) return FTB_ERR_WORKSPACE;
    // Launch order = level order.  A step of layer l reads the layer below up to the step that
    // holds its last timestep (the steps of a layer complete in order, so waiting for that one
    // is enough) and the step before it in its own layer.
    std::vector<CellItem> order;
    std::vector<std::vector<int>> index_of(D);
    for (int l = 0; l < D; ++l) index_of[l].resize(level_of[l].size());
    for (auto& kv : levels)
      for (size_t i = 0; i < kv.second.size(); ++i) {
        const std::pair<int, int> id = level_ids[kv.first][i];
        index_of[id.first][id.second] = static_cast<int>(order.size());
        order.push_back(kv.second[i]);
      }
    std::vector<int32_t> deps(static_cast<size_t>(n_items) * kMaxSeg * 2, -1);
    for (int l = 0; l < D; ++l)
      for (size_t s = 0; s < index_of[l].size(); ++s) {
        const int me = index_of[l][s];
        const int dl = dilations[l];
        const int t1 = std::min(L, static_cast<int>(s + 1) * dl);
        if (l > 0) {
          const int below = index_of[l - 1][(t1 - 1) / dilations[l - 1]];
          deps[(me * kMaxSeg + 0) * 2 + 0] = deps[(me * kMaxSeg + 0) * 2 + 1] = below;
        }
        if (s > 0) {
          const int prev = index_of[l][s - 1];
          deps[(me * kMaxSeg + 1) * 2 + 0] = deps[(me * kMaxSeg + 1) * 2 + 1] = prev;
        }
      }
    rc = run_persistent(cl, order, deps, static_cast<char*>(workspace), lay, workspace_bytes);
    // A refused cooperative launch falls back to one launch per level, as in the other entries;
    // an explicitly requested persistent schedule reports the refusal.
    if (rc != FTB_ERR_LAUNCH || tune.schedule != 0) return rc;
  }
  for (auto& kv : levels) {
    rc = cl.run(kv.second);
    if (rc) return rc;
  }
  return FTB_OK;
}

size_t ftb_lstm_dilated_workspace_bytes(int D, int L) {
  if (D <= 0 || L <= 0) return kWorkspaceBytes;
  // tables of the generic persistent schedule, then the flags of the cluster schedule
  return plan_layout(static_cast<size_t>(D) * L, 0).total + sizeof(int) * lstm_dilated_cluster_flag_ints(D, L);
}

int ftb_grid_rnn_fwd(const void* X, const void* Y, const void* Wpx, const void* Wpy, const float* bias_x,
                     const float* bias_y, void* hx, void* hy, int D, int A, int B, int N, int H, int dtype,
                     void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!X || !Y || !Wpx || !Wpy || !hx || !hy || D <= 0 || A <= 0 || B <= 0 || N <= 0 || !valid_dtype(dtype))
    return FTB_ERR_ARG;
  if (H <= 0 || H % 64 != 0) return FTB_ERR_ARG;
  if (static_cast<int64_t>(D) * A * B * N > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({X, Y, Wpx, Wpy, bias_x, bias_y, hx, hy})) return FTB_ERR_ALIGN;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;

  const int K = 3 * H;
  const size_t es = dtype_size(dtype);
  // One launch context for both directions: activation buffers 0..3 = X, Y, hx, hy; weight
  // buffer 0 = direction x, 1 = direction y.  Direction x reads (hx | hy | X or hx below),
  // direction y reads (hx | hy | Y or hy below).
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_TANH;
  cl.n_cols = H;
  cl.ld_out = H;
  cl.ld_c = H;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  if (dtype == FTB_F32) {
    cl.act[0] = static_cast<const float*>(X);
    cl.act[1] = static_cast<const float*>(Y);
    cl.act[2] = static_cast<const float*>(hx);
    cl.act[3] = static_cast<const float*>(hy);
    cl.ld_act[0] = cl.ld_act[1] = cl.ld_act[2] = cl.ld_act[3] = H;
    cl.w = static_cast<const float*>(Wpx);
    cl.w2 = static_cast<const float*>(Wpy);
    cl.ldw = K;
  } else {
    cl.bn = pick_bn(H, 128);
    if (cl.bn == 0) return FTB_ERR_ARG;
    const uint64_t grid_rows = static_cast<uint64_t>(A) * B * N;
    rc = make_tmap_2d(&cl.maps[0], X, dtype, grid_rows, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[1], Y, dtype, grid_rows, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[2], hx, dtype, grid_rows * D, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[3], hy, dtype, grid_rows * D, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapW, Wpx, dtype, static_cast<uint64_t>(D) * H, K, K, cl.bn, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapC, Wpy, dtype, static_cast<uint64_t>(D) * H, K, K, cl.bn, 64);
    if (rc) return rc;
  }

  // Cell (d, a, b) of direction dirn, and which earlier cell each of its K segments reads
  // (-1: an input of the call).  Anti-diagonal level = d + a + b.
  auto cell_index = [&](int d, int a, int b) { return (static_cast<int64_t>(d) * A + a) * B + b; };
  auto make_item = [&](int d, int a, int b, int dirn, int64_t (&src)[kMaxSeg]) {
    CellItem it = blank_item();
    const int64_t cell = cell_index(d, a, b);
    for (int s = 0; s < kMaxSeg; ++s) src[s] = -1;
    // The cell's own input first: it is an input of the call (layer 0) or was finished two
    // levels ago, so its K blocks run while the two neighbours of the previous level finish.
    if (d == 0) {
      add_seg(it, dirn, (static_cast<int64_t>(a) * B + b) * N, H, 2 * H);
    } else {
      src[it.nseg] = cell_index(d - 1, a, b) * 2 + dirn;
      add_seg(it, 2 + dirn, cell_index(d - 1, a, b) * N, H, 2 * H);
    }
    if (a > 0) {
      src[it.nseg] = cell_index(d, a - 1, b) * 2 + 0;
      add_seg(it, 2, cell_index(d, a - 1, b) * N, H, 0);
    }
    if (b > 0) {
      src[it.nseg] = (cell - 1) * 2 + 1;
      add_seg(it, 3, (cell - 1) * N, H, H);
    }
    it.w_row0 = d * H;
    it.w_map = dirn;
    it.rows = N;
    it.out = static_cast<char*>(dirn == 0 ? hx : hy) + static_cast<size_t>(cell) * N * H * es;
    const float* bias = dirn == 0 ? bias_x : bias_y;
    it.bias = bias ? bias + static_cast<size_t>(d) * H : nullptr;
    return it;
  };

  const int n_items = 2 * D * A * B;
  const int levels = (D - 1) + (A - 1) + (B - 1) + 1;
  const PlanLayout lay = plan_layout(n_items, 0);
  // Weights on chip, states that carry their own arrival (csrc/grid_flow.cu): the choice where it applies and the workspace has
  // room for its counters behind the tables.
  GridFlowPlan flow;
  if (workspace_bytes > lay.total &&
      grid_flow_plan(dtype, D, A, B, N, H, cl.sm_count, (workspace_bytes - lay.total) / sizeof(int), &flow)) {
    rc = launch_grid_flow(dtype, X, Y, Wpx, Wpy, bias_x, bias_y, hx, hy, D, A, B, N, H, flow,
                          reinterpret_cast<int*>(static_cast<char*>(workspace) + lay.total), status, stream);
    if (rc != FTB_ERR_LAUNCH) return rc;  // a refused cooperative launch falls back to the generic wavefront
  }
  const bool persistent = dtype != FTB_F32 && workspace_bytes >= lay.total;
  if (persistent) {
    // One cooperative launch for the whole grid: items in level order, each K segment waiting
    // for the one earlier cell it reads.
    std::vector<CellItem> order;
    order.reserve(n_items);
    std::vector<int> index_of(n_items, -1);
    std::vector<int64_t> srcs;
    srcs.reserve(static_cast<size_t>(n_items) * kMaxSeg);
    for (int m = 0; m < levels; ++m)
      for (int d = 0; d < D; ++d)
        for (int a = 0; a < A; ++a) {
          const int b = m - d - a;
          if (b < 0 || b >= B) continue;
          for (int dirn = 0; dirn < 2; ++dirn) {
            int64_t src[kMaxSeg];
            index_of[cell_index(d, a, b) * 2 + dirn] = static_cast<int>(order.size());
            order.push_back(make_item(d, a, b, dirn, src));
            for (int s = 0; s < kMaxSeg; ++s) srcs.push_back(src[s]);
          }
        }
    std::vector<int32_t> deps(static_cast<size_t>(n_items) * kMaxSeg * 2, -1);
    for (int i = 0; i < n_items; ++i)
      for (int s = 0; s < kMaxSeg; ++s) {
        const int64_t src = srcs[static_cast<size_t>(i) * kMaxSeg + s];
        if (src >= 0) deps[(i * kMaxSeg + s) * 2 + 0] = deps[(i * kMaxSeg + s) * 2 + 1] = index_of[src];
      }
    rc = run_persistent(cl, order, deps, static_cast<char*>(workspace), lay, workspace_bytes);
    if (rc != FTB_ERR_LAUNCH) return rc;  // a refused cooperative launch falls back to levels
  }

  std::vector<CellItem> items;
  for (int m = 0; m < levels; ++m) {
    items.clear();
    for (int d = 0; d < D; ++d)
      for (int a = 0; a < A; ++a) {
        const int b = m - d - a;
        if (b < 0 || b >= B) continue;
        for (int dirn = 0; dirn < 2; ++dirn) {
          int64_t src[kMaxSeg];
          items.push_back(make_item(d, a, b, dirn, src));
        }
      }
    rc = cl.run(items);
    if (rc) return rc;
  }
  return FTB_OK;
}

int ftb_rnn_pack_weights(const void* W, const void* U, void* Wp, int I, int H, int dtype, void* stream) {
  if (!W || !U || !Wp || I <= 0 || H <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  return pack_rnn(W, U, Wp, I, H, dtype, static_cast<cudaStream_t>(stream));
}

// Scratch of the encoder's chain kernel: fp32 input halves of as many source steps as this allows (a
// longer source is scanned in pieces).
static constexpr size_t kMaxPreBytes = 32u << 20;

size_t ftb_rnn_attention_scratch_bytes(int Ls, int N, int H, int dtype) {
  if (Ls <= 0 || N <= 0 || H <= 0 || !rnn_chain_supported(dtype, H)) return 0;
  const size_t step = static_cast<size_t>(N) * H * sizeof(float);
  return std::min<size_t>(Ls, kMaxPreBytes / step) * step;
}

size_t ftb_rnn_attention_scratch_bytes_all(int Ls, int Lt, int N, int H, int dtype) {
  const size_t encoder = ftb_rnn_attention_scratch_bytes(Ls, N, H, dtype);
  const size_t step = static_cast<size_t>(N > 0 ? N : 0) * (H > 0 ? H : 0) * sizeof(float);
  if (Lt <= 0 || encoder == 0 || encoder < Ls * step || !attn_decode_supported(dtype, Ls, Lt, N, H, current_sm_count())) return encoder;
  return encoder + Lt * step;
}

size_t ftb_rnn_attention_workspace_bytes(int Ls, int N, int H, int dtype) {
  return kWorkspaceBytes + ftb_rnn_attention_scratch_bytes(Ls, N, H, dtype);
}

int ftb_rnn_attention_fwd(const void* src, const void* trg, const void* Wp_src, const void* Wp_trg,
                          const float* bias_src, const float* bias_trg, const void* enc_proj, const void* dec_proj,
                          const int* src_lens, void* enc, float* enc_scores, void* dec, void* out, int Ls, int Lt,
                          int N, int H, int dtype, void* workspace, size_t workspace_bytes, void* stream) {
  const bool room = workspace != nullptr && workspace_bytes > kWorkspaceBytes;
  return ftb_rnn_attention_fwd_scratch(src, trg, Wp_src, Wp_trg, bias_src, bias_trg, enc_proj, dec_proj, src_lens, enc,
                                       enc_scores, dec, out, Ls, Lt, N, H, dtype,
                                       room ? static_cast<char*>(workspace) + kWorkspaceBytes : nullptr,
                                       room ? workspace_bytes - kWorkspaceBytes : 0, workspace, workspace_bytes, stream);
}

int ftb_rnn_attention_fwd_scratch(const void* src, const void* trg, const void* Wp_src, const void* Wp_trg,
                                  const float* bias_src, const float* bias_trg, const void* enc_proj,
                                  const void* dec_proj, const int* src_lens, void* enc, float* enc_scores, void* dec,
                                  void* out, int Ls, int Lt, int N, int H, int dtype, void* scratch,
                                  size_t scratch_bytes, void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!src || !trg || !Wp_src || !Wp_trg || !enc_proj || !dec_proj || !enc || !enc_scores || !dec || !out)
    return FTB_ERR_ARG;
  if (Ls <= 0 || Lt <= 0 || N <= 0 || H <= 0 || H % 64 != 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (Ls > rnn_attention_max_src_len()) return FTB_ERR_ARG;
  if (static_cast<int64_t>(std::max(Ls, Lt)) * N > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({src, trg, Wp_src, Wp_trg, bias_src, bias_trg, enc, dec, out, scratch})) return FTB_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(enc_scores) & 3) != 0 || (reinterpret_cast<uintptr_t>(src_lens) & 3) != 0)
    return FTB_ERR_ALIGN;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;

  const int K = 2 * H;
  const size_t es = dtype_size(dtype);
  // One launch context for both cells: activation buffers 0..3 = src, trg, enc, out (the attention
  // vectors, which are the decoder's recurrent input); weight buffer 0 = encoder, 1 = decoder.
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_TANH;
  cl.n_cols = H;
  cl.ld_out = H;
  cl.ld_c = H;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  if (dtype == FTB_F32) {
    cl.act[0] = static_cast<const float*>(src);
    cl.act[1] = static_cast<const float*>(trg);
    cl.act[2] = static_cast<const float*>(enc);
    cl.act[3] = static_cast<const float*>(out);
    cl.ld_act[0] = cl.ld_act[1] = cl.ld_act[2] = cl.ld_act[3] = H;
    cl.w = static_cast<const float*>(Wp_src);
    cl.w2 = static_cast<const float*>(Wp_trg);
    cl.ldw = K;
  } else {
    cl.bn = pick_bn(H, 128);
    if (cl.bn == 0) return FTB_ERR_ARG;
    const uint64_t src_rows = static_cast<uint64_t>(Ls) * N, trg_rows = static_cast<uint64_t>(Lt) * N;
    rc = make_tmap_2d(&cl.maps[0], src, dtype, src_rows, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[1], trg, dtype, trg_rows, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[2], enc, dtype, src_rows, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.maps[3], out, dtype, trg_rows, H, H, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapW, Wp_src, dtype, H, K, K, cl.bn, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&cl.mapC, Wp_trg, dtype, H, K, K, cl.bn, 64);
    if (rc) return rc;
  }

  std::vector<CellItem> items(1);
  // Encoder: e_j = tanh(x_j W + e_{j-1} U + b).  With room for the fp32 input halves x_j W of at least
  // one step in the scratch: those as one product, then the scan as one launch of the chain kernel
  // (csrc/rnn_chain.cu), piece by piece; else one level per source position.
  const size_t pre_step = static_cast<size_t>(N) * H * sizeof(float);
  const int piece = rnn_chain_supported(dtype, H) && scratch != nullptr
                        ? static_cast<int>(std::min<size_t>(Ls, scratch_bytes / pre_step)) : 0;
  // With room for the decoder's input halves y_t W behind them, those come with the same product, and the rest is one launch.
  const bool decode = piece == Ls && scratch_bytes / pre_step >= static_cast<size_t>(Ls) + Lt &&
                      attn_decode_supported(dtype, Ls, Lt, N, H, cl.sm_count);
  float* pre_trg = static_cast<float*>(scratch) + static_cast<size_t>(Ls) * N * H;
  for (int j = 0; j < Ls && piece > 0; j += piece) {
    const int steps = std::min(piece, Ls - j);
    float* pre = static_cast<float*>(scratch);
    CellLauncher gemm = cl;
    gemm.epi = EPI_STORE_F32;
    // Tiles of 256 columns where those of 128 would be more than one round of the SMs.
    const int rows128 = (steps * N + 127) / 128 + (decode ? (Lt * N + 127) / 128 : 0);
    if (H % 256 == 0 && rows128 * (H / 128) > cl.sm_count) {
      gemm.bn = 256;
      if ((rc = make_tmap_2d(&gemm.mapW, Wp_src, dtype, H, K, K, 256, 64))) return rc;
      if ((rc = make_tmap_2d(&gemm.mapC, Wp_trg, dtype, H, K, K, 256, 64))) return rc;
    }
    items[0] = blank_item();
    add_seg(items[0], 0, static_cast<int64_t>(j) * N, H, 0);
    items[0].rows = steps * N;
    items[0].out = pre;
    if (decode) {
      items.push_back(blank_item());
      add_seg(items[1], 1, 0, H, 0);
      items[1].w_map = 1;
      items[1].rows = Lt * N;
      items[1].out = pre_trg;
    }
    rc = gemm.run(items);
    items.resize(1);
    if (rc) return rc;
    char* enc_j = static_cast<char*>(enc) + static_cast<size_t>(j) * N * H * es;
    rc = launch_rnn_chain(dtype, pre, Wp_src, K, H, bias_src, j > 0 ? enc_j - static_cast<size_t>(N) * H * es : nullptr,
                          enc_j, steps, N, H, status, stream);
    if (rc) return rc;
  }
  for (int j = 0; j < Ls && piece == 0; ++j) {
    CellItem it = blank_item();
    add_seg(it, 0, static_cast<int64_t>(j) * N, H, 0);
    if (j > 0) add_seg(it, 2, static_cast<int64_t>(j - 1) * N, H, H);
    it.rows = N;
    it.w_map = 0;
    it.bias = bias_src;
    it.out = static_cast<char*>(enc) + static_cast<size_t>(j) * N * H * es;
    items[0] = it;
    rc = cl.run(items);
    if (rc) return rc;
  }
  // Decoder.  The attention vector of a step does not depend on the decoder (its term moves all scores
  // of a softmax by one number), so the vectors of all steps are known here: they go to their rows of
  // `out`, where the decoder cells read them as recurrent inputs, all cells run as one level, and a
  // term that is not finite is carried to the steps behind it at the end.
  if (decode)
    return launch_attn_decode(dtype, enc, enc_proj, src_lens, enc_scores, pre_trg, static_cast<const char*>(Wp_trg) + H * es, K,
                              bias_trg, dec_proj, dec, out, Lt, Ls, N, H, status, stream);
  rc = launch_attn_vectors(dtype, enc, enc_proj, src_lens, enc_scores, out, Lt, Ls, N, H, stream);
  if (rc) return rc;
  items.clear();
  for (int t = 0; t < std::min(Lt, 2); ++t) {  // step 0 has no recurrent input; steps 1.. are consecutive rows
    CellItem it = blank_item();
    add_seg(it, 1, static_cast<int64_t>(t) * N, H, 0);
    if (t > 0) add_seg(it, 3, 0, H, H);
    it.rows = t == 0 ? N : (Lt - 1) * N;
    it.w_map = 1;
    it.bias = bias_trg;
    it.out = static_cast<char*>(dec) + static_cast<size_t>(t) * N * H * es;
    items.push_back(it);
  }
  rc = cl.run(items);
  if (rc) return rc;
  return launch_attn_finish(dtype, dec, dec_proj, enc_scores, src_lens, out, Lt, Ls, N, H, stream);
}

int ftb_grid_flow_form_fwd(const void* X, const void* Y, const void* Wpx, const void* Wpy, const float* bias_x,
                           const float* bias_y, void* hx, void* hy, int D, int A, int B, int N, int H, int dtype, int nb,
                           void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!X || !Y || !Wpx || !Wpy || !hx || !hy || D <= 0 || A <= 0 || B <= 0 || N <= 0) return FTB_ERR_ARG;
  if (static_cast<int64_t>(D) * A * B * N > 0x7fffffffLL) return FTB_ERR_ARG;
  if (!aligned16({X, Y, Wpx, Wpy, bias_x, bias_y, hx, hy})) return FTB_ERR_ALIGN;
  GridFlowPlan flow;
  // (a named form has at most 32 slices; the automatic choice counts up to 64)
  if (!grid_flow_form(dtype, D, A, B, N, H, current_sm_count(), nb, &flow) || flow.S > 32) return FTB_ERR_ARG;
  int* status = nullptr;
  const int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;
  if (workspace_bytes < kWorkspaceBytes + sizeof(int) * flow.ints) return FTB_ERR_WORKSPACE;
  return launch_grid_flow(dtype, X, Y, Wpx, Wpy, bias_x, bias_y, hx, hy, D, A, B, N, H, flow,
                          reinterpret_cast<int*>(static_cast<char*>(workspace) + kWorkspaceBytes), status, stream);
}

size_t ftb_grid_rnn_tables_bytes(int D, int A, int B) {
  if (D <= 0 || A <= 0 || B <= 0) return kWorkspaceBytes;
  return plan_layout(static_cast<size_t>(2) * D * A * B, 0).total;
}

size_t ftb_grid_rnn_workspace_bytes(int D, int A, int B) {
  if (D <= 0 || A <= 0 || B <= 0) return kWorkspaceBytes;
  // tables of the generic persistent schedule, then the counters of the one with weights on chip, of any batch
  return plan_layout(static_cast<size_t>(2) * D * A * B, 0).total + sizeof(int) * grid_flow_ints(D, A, B, 0);
}

size_t ftb_grid_rnn_call_workspace_bytes(int D, int A, int B, int N, int H, int dtype) {
  if (D <= 0 || A <= 0 || B <= 0 || N <= 0 || H <= 0 || dtype == FTB_F32) return kWorkspaceBytes;
  return plan_layout(static_cast<size_t>(2) * D * A * B, 0).total + (H <= 256 ? sizeof(int) * grid_flow_ints(D, A, B, N) : 0);
}

int ftb_gemm_nt(const void* A, const void* Bt, void* out, int M, int N, int K, int dtype, const int* tuning,
                void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const Tuning tune(tuning);
  if (!A || !Bt || !out || M <= 0 || N <= 0 || K <= 0 || !valid_dtype(dtype)) return FTB_ERR_ARG;
  if (K % 64 != 0) return FTB_ERR_ARG;
  if (dtype == FTB_F32 ? (N % 64 != 0) : (N % 128 != 0)) return FTB_ERR_ARG;
  if (!aligned16({A, Bt, out})) return FTB_ERR_ALIGN;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_STORE;
  cl.n_cols = N;
  cl.ld_out = N;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  if (dtype == FTB_F32) {
    cl.act[0] = cl.act[1] = cl.act[2] = static_cast<const float*>(A);
    cl.ld_act[0] = cl.ld_act[1] = cl.ld_act[2] = K;
    cl.w = static_cast<const float*>(Bt);
    cl.ldw = K;
  } else {
    cl.bn = tune.bn ? tune.bn : ((N % 256 == 0) ? 256 : 128);
    if (cl.bn != 128 && cl.bn != 256) return FTB_ERR_ARG;
    cl.pair = tune.use_pair(M);
    rc = make_tmap_2d(&cl.maps[0], A, dtype, M, K, K, 128, 64);
    if (rc) return rc;
    cl.maps[1] = cl.maps[2] = cl.maps[3] = cl.maps[0];
    rc = make_tmap_2d(&cl.mapW, Bt, dtype, N, K, K, cl.w_box_rows(), 64);
    if (rc) return rc;
    cl.mapC = cl.maps[0];
  }
  std::vector<CellItem> items(1, blank_item());
  add_seg(items[0], 0, 0, K, 0);
  items[0].rows = M;
  items[0].out = out;
  return cl.run(items);
}

int ftb_projection_padded_cols(int V) { return V <= 0 ? 0 : ((V + 127) / 128) * 128; }

int ftb_projection_pack(const void* P, void* Pt, int H, int V, int dtype, void* stream) {
  if (!P || !Pt || H <= 0 || V <= 0 || (dtype != FTB_F16 && dtype != FTB_BF16)) return FTB_ERR_ARG;
  if (!aligned16({P, Pt})) return FTB_ERR_ALIGN;
  return pack_projection(P, Pt, H, V, ftb_projection_padded_cols(V), dtype, static_cast<cudaStream_t>(stream));
}

// logits: [T, Vp]; probs: [T, V] without gaps, or the same buffer as logits, with its rows Vp apart.
static int project_softmax(const void* h, const void* Pt, float* logits, float* probs, long long T, int V, int H, int dtype,
                           void* workspace, size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!h || !Pt || !logits || !probs || T <= 0 || T > 0x7fffffffLL || V <= 0 || H <= 0 || H % 64 != 0) return FTB_ERR_ARG;
  if (dtype != FTB_F16 && dtype != FTB_BF16) return FTB_ERR_ARG;
  if (V > 48 * 1024) return FTB_ERR_ARG;  // the softmax runs in place on rows that fit its on-chip row cache
  if (!aligned16({h, Pt, logits, probs})) return FTB_ERR_ALIGN;
  const int Vp = ftb_projection_padded_cols(V);
  if (static_cast<int64_t>(T) * Vp > 0x7fffffffffLL) return FTB_ERR_ARG;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;
  // 1. logits = h . Pt^T, fp32
  CellLauncher cl;
  cl.dtype = dtype;
  cl.epi = EPI_STORE_F32;
  cl.n_cols = Vp;
  cl.ld_out = Vp;
  cl.status = status;
  cl.stream = stream;
  cl.sm_count = current_sm_count();
  cl.bn = (Vp % 256 == 0) ? 256 : 128;
  cl.pair = 0;
  rc = make_tmap_2d(&cl.maps[0], h, dtype, static_cast<uint64_t>(T), H, H, 128, 64);
  if (rc) return rc;
  cl.maps[1] = cl.maps[2] = cl.maps[3] = cl.maps[0];
  rc = make_tmap_2d(&cl.mapW, Pt, dtype, Vp, H, H, cl.w_box_rows(), 64);
  if (rc) return rc;
  cl.mapC = cl.maps[0];
  std::vector<CellItem> items(1, blank_item());
  add_seg(items[0], 0, 0, H, 0);
  items[0].rows = static_cast<int32_t>(T);
  items[0].out = logits;
  rc = cl.run(items);
  if (rc) return rc;
  // 2. softmax over the first V logits of every row, one read and one write per logit
  return online_softmax_rows(logits, probs, static_cast<int>(T), V, Vp, probs == logits ? Vp : V, stream);
}

int ftb_lstm_project_softmax(const void* h, const void* Pt, float* probs, long long T, int V, int H, int dtype,
                             void* workspace, size_t workspace_bytes, void* stream) {
  return project_softmax(h, Pt, probs, probs, T, V, H, dtype, workspace, workspace_bytes, stream);
}

int ftb_lstm_project_softmax_rows(const void* h, const void* Pt, float* logits, float* probs, long long T, int V, int H,
                                  int dtype, void* workspace, size_t workspace_bytes, void* stream) {
  if (probs == logits) return FTB_ERR_ARG;
  return project_softmax(h, Pt, logits, probs, T, V, H, dtype, workspace, workspace_bytes, stream);
}

size_t ftb_project_softmax_scratch_bytes(long long T, int V, int H, int dtype, int unpacked) {
  if (T <= 0 || T > 0x7fffffffLL || V <= 0 || V > 48 * 1024 || H <= 0 || !project_twice_supported(dtype, T, V, H, unpacked != 0)) return 0;
  return project_twice_scratch(T, V);
}

int ftb_project_softmax_fwd(const void* h, const void* P, int unpacked, float* probs, long long ld, long long T, int V, int H,
                            int dtype, void* scratch, size_t scratch_bytes, void* workspace, size_t workspace_bytes,
                            void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!h || !P || !probs || !scratch || T <= 0 || T > 0x7fffffffLL || V <= 0 || H <= 0 || H % 64 != 0) return FTB_ERR_ARG;
  if (dtype != FTB_F16 && dtype != FTB_BF16) return FTB_ERR_ARG;
  if (V > 48 * 1024) return FTB_ERR_ARG;  // what ftb_lstm_project_softmax takes
  const int Vp = ftb_projection_padded_cols(V);
  if (ld != V && ld != Vp) return FTB_ERR_ARG;
  if (!aligned16({h, P, probs, scratch})) return FTB_ERR_ALIGN;
  const size_t need = ftb_project_softmax_scratch_bytes(T, V, H, dtype, unpacked);
  if (need == 0) return FTB_ERR_ARG;
  if (scratch_bytes < need) return FTB_ERR_WORKSPACE;
  int* status = nullptr;
  int rc = begin_call(workspace, workspace_bytes, stream, &status);
  if (rc) return rc;
  return launch_project_twice(dtype, h, P, unpacked != 0, probs, ld, static_cast<int>(T), V, Vp, H, scratch, status, stream);
}

// ------------------------------------------------------------------------------
// Stacked LSTM forward for callers that must not allocate device memory.
//
// Some hosts of this library cannot call cudaMalloc at the point where they need a
// forward pass: a real-time loop that must not enter the allocator, a
// plugin whose host application owns the allocator and hands out nothing but the
// input and output buffers, or a process whose memory pool is already carved up.
// ftb_lstm_stacked_fwd needs a caller-provided workspace for its schedule tables,
// completion counters and status word; this variant keeps that scratch in a
// fixed-size array that is part of the library image instead.
//
// Cost and limits: every GPU that loads the library holds FTB_STATIC_SCRATCH_BYTES
// of device memory for the array until the process exits.  Problems whose
// ftb_lstm_stacked_workspace_bytes(D, L, N, H) exceeds that size are rejected with
// FTB_ERR_SCRATCH_LIMIT.  Only the persistent schedule (16-bit dtypes) is offered.
// All calls on a device share the one array, and it keeps whatever the previous
// call left in it: each call re-zeroes the status word and the counters it uses on
// its stream before launching, so back-to-back calls on one stream are fine, but two
// calls whose kernels can overlap on the GPU (different streams, or different host
// threads) race on the tables and counters and must be serialised by the caller.
//
// The first call on each device resolves the array's device address
// (cudaGetSymbolAddress; the array's name is only a host-side handle, not an
// address a kernel could use) and caches it; make that first call outside any
// stream capture.
#define FTB_STATIC_SCRATCH_BYTES (4u << 20)
static __device__ __align__(256) unsigned char g_static_scratch[FTB_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_scratch_mu;
void* g_static_scratch_ptr[64] = {};
}  // namespace

int ftb_lstm_stacked_fwd_noalloc(const void* x, const void* Wp, const float* bias_p, void* hs, float* c, int D,
                                 int L, int N, int I, int H, int dtype, const int* tuning, void** scratch_out,
                                 void* stream) {
  if (D <= 0 || L <= 0 || N <= 0 || H <= 0) return FTB_ERR_ARG;
  if (dtype != FTB_F16 && dtype != FTB_BF16) return FTB_ERR_ARG;
  if (plan_layout(D * L, stacked_max_tiles_per_cell(N, H)).total > FTB_STATIC_SCRATCH_BYTES) return FTB_ERR_SCRATCH_LIMIT;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FTB_ERR_ARCH;
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_static_scratch_mu);
    if (g_static_scratch_ptr[dev] == nullptr) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) {
        cudaGetLastError();
        return FTB_ERR_DRIVER;
      }
      g_static_scratch_ptr[dev] = p;
    }
    scratch = g_static_scratch_ptr[dev];
  }
  if (scratch_out != nullptr) *scratch_out = scratch;
  int t[FTB_TUNING_INTS] = {0, 0, 0, 0, 0, 0};
  if (tuning != nullptr)
    for (int i = 0; i < FTB_TUNING_INTS; ++i) t[i] = tuning[i];
  // A single-launch schedule: their host side builds nothing on the heap (the one-launch-per-level
  // schedule keeps its cell lists in std::vector).  2 = generic persistent kernel, 3 = static tile
  // ownership; anything else the caller asked for becomes 2.
  if (t[2] != 3) t[2] = 2;
  return ftb_lstm_stacked_fwd(x, Wp, bias_p, hs, c, D, L, N, I, H, dtype, t, scratch, FTB_STATIC_SCRATCH_BYTES,
                              stream);
}

}  // extern "C"
