// Stacked LSTM forward with recurrent weights (and as many others as fit) on chip and hidden states that carry their own
// arrival: the 16-bit path of models whose layer tiles fit on the device (lstm_flow_plan below).
//
// A step of a layer is a chain: recurrent MMAs, gates, hidden state to the layer's other CTAs, next
// step.  With a flag per tile that chain was 5.5 us at H 512 and 64 sequences: store the tile through
// TMA and wait for it (1 us), release a flag that the others poll (1.2 us), load the state through TMA
// (1 us), and only 1 us of MMAs.  Here
//   * the output array is its own flag.  It is filled with 0xFFFF before the launch, a bit pattern no
//     hidden state has (the conversions give 0x7FFF for every NaN).  An epilogue thread stores
//     four units of one sequence as one 8-byte word; the warps of the layer's CTAs read 16-byte
//     chunks of the rows they need and repeat those with a word that still ends in 0xFFFF.  What has
//     arrived goes straight into the MMA's operand tile.  No fence, no flag, no second trip;
//   * weights never move during a sweep over time: a CTA owns 128 packed gate rows (32 units) of one
//     layer, the recurrent K blocks first in tensor memory, the rest of them and the input blocks in
//     the tensor memory left, then in shared memory;
//   * CTAs of neighbouring gate rows run as pairs where that is faster (take_pairs): one MMA over both (.cta_group::2),
//     each with its own weights and accumulator and half the state's rows, so that a state passes L2 half as often.  The
//     state's hand-over is ordered by a fence over this CTA's shared memory alone: mbarrier.arrive.release.cluster would
//     wait for the warp's own stores to the output array too (D8 L100 N64 H512 490 us a call, with the fence 411; single
//     CTAs 510);
//   * the batch is cut into slices of NB columns that never meet (UMMA N = NB), each with its own CTAs.
//     What grows with NB is the state a CTA reads and its gates (20 cycles a column, tanh's 16 a cycle): slices are
//     as narrow as the device has CTAs for;
//   * the warps that have stored a step's state read the whole of it back: the chain is one set of warps
//     with no hand-over but the accumulator's barrier and the operand tile's.  They wait before the
//     first read for as long as it last took the state to arrive: reads that come too early load the L2
//     that the state has to pass through (8.5 us a step without the pause, 4.4 with it: D8 H512 N64, single CTAs);
//   * what does not fit of the input weights passes through a ring of shared memory every step (kStream): the input half
//     is off the chain, and its weights come from L2 while the state is under way.  Against the kernels that keep
//     no weights (csrc/lstm_wmajor.cu and others), us: D4 L73 N14 H896 561 -> 256, D1 L63 N118 H896 573 -> 249, D9 L72 N19 H1024
//     1800 -> 1055, D16 L100 N64 H1024 3820 -> 3420.  Rings of 2 / 3 / 4 blocks: the first 267 / 261 / 256, the third
//     1170 / 1076 / 1055;
//   * the layer below is read through TMA behind a flag per cell (a counter of the tiles stored), which
//     a warp of its own raises: its fences are off the chain, the layers above just run further behind;
//   * the input half of step t + 1 is issued right after the recurrent half of step t.
// A thread reads all gates of its unit for four sequences of every 16 (accumulator fragments, body in lstm_flow.cuh), keeps their
// cell state in fp32 registers for the sweep, and two shuffles make words of four units.
//
// A ragged batch (sorted by decreasing length, rows of a step packed) is the same kernel: the rows of
// step t start at off[t], and columns whose sequence has ended are neither stored nor waited for.
//
// Same arithmetic in the same order as the other 16-bit schedules: bit-identical results.
//
// Roles: warp 0 MMA issuer, warp 1 TMA producer (input tiles, shared-memory weights), warp 2 publisher, warp 3 the ring,
// warps 4.. epilogue and state.  Cooperative launch.  Of a pair the even CTA issues the MMAs.
//
// Program: stacked_lstm() (examples/stacked_rnn/stacked_lstm1.py:66-76, stacked_rnn.py:69-79) in place
// of kaleido/core/device/kernels/lstm/stacked_lstm/region{1,2,3}.h.
#include <algorithm>
#include <cstdlib>

#include "flow_plan.h"
#include "lstm_flow.cuh"

namespace ftb {

namespace {

using namespace flow;

// The output array before the sweep, all 0xFFFF, and the counters, all 0.  The sweep's kernel starts beside this one and
// loads its weights meanwhile: one CTA an SM of 256 threads leaves it room.  Against two memsets before the sweep, us a call:
// D1 L30 N8 H128 49.5 -> 47.5, D4 L16 N45 H256 53 -> 51.5, D15 L92 N50 H128 247 -> 240, D8 L100 N64 H512 (52 MB) 390 -> 388.
__global__ void __launch_bounds__(256) flow_fill_kernel(uint4* hs, int64_t n, int* flags, int n_flags) {
  grid_launch_dependents();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x, first = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const uint32_t ones = 0xFFFFFFFFu;
  for (int64_t i = first; i < n; i += stride) hs[i] = make_uint4(ones, ones, ones, ones);
  for (int64_t i = first; i < n_flags; i += stride) flags[i] = 0;
}

template <typename T, int NB, bool kPair, bool kStream>
__global__ void __launch_bounds__(FlowCfg<NB, kPair>::kThreads, 1)
lstm_flow_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapH,
                 const __grid_constant__ CUtensorMap mapW, const FlowArgs a) {
  const int tile = blockIdx.x % a.n_tiles;
  const int slice = (blockIdx.x / a.n_tiles) % a.S;
  body<T, NB, kPair, kStream>(mapX, mapH, mapW, a, tile, slice, blockIdx.x / (a.n_tiles * a.S), NB);
}

template <typename T, int NB, bool kPair, bool kStream = false>
int launch(const CUtensorMap& mX, const CUtensorMap& mH, const CUtensorMap& mW, const FlowArgs& a, uint32_t smem,
           cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = lstm_flow_kernel<T, NB, kPair, kStream>;
  if (!ensure_dynamic_smem(kfn, kMaxSmem, configured)) return FTB_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min(a.G, a.D) * a.S * a.n_tiles);
  cfg.blockDim = dim3(FlowCfg<NB, kPair>::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[3];
  int na = 0;
  // beside the fill of the output array
  attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[na].val.programmaticStreamSerializationAllowed = 1;
  ++na;
  if (kPair) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = 2;
    attrs[na].val.clusterDim.y = 1;
    attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  // FTB_NO_COOPERATIVE=1 drops the cooperative attribute (profilers that cannot replay cooperative
  // launches); FTB_REFUSE_COOPERATIVE=1 answers as if the driver had refused the launch (tests of the
  // fallback).
  static const bool no_coop = [] {
    const char* e = getenv("FTB_NO_COOPERATIVE");
    return e != nullptr && e[0] == '1';
  }();
  {
    const char* e = getenv("FTB_REFUSE_COOPERATIVE");
    if (e != nullptr && e[0] == '1') return FTB_ERR_LAUNCH;
  }
  if (!no_coop) {
    attrs[na].id = cudaLaunchAttributeCooperative;
    attrs[na].val.cooperative = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  if (cudaLaunchKernelEx(&cfg, kfn, mX, mH, mW, a) != cudaSuccess) {
    cudaGetLastError();
    return FTB_ERR_LAUNCH;
  }
  count_launch();
  return FTB_OK;
}

// Whether the CTAs of a slice run as pairs: half the state for each of them to read, against hand-overs that wait for both.
// What they read weighs when all of them read much of it together (rows: of a step, on average).  Single CTAs / pairs, medians over 11 to 32 of 721
// forms of 400 calls (D 1..16, N 1..256, L 16..128), by the bytes of states that the whole grid reads a step, H <= 512:
//   slices of 16: below 0.8 MB 0.96 to 0.98, 0.9..1.2 MB 1.00, 1.2..1.8 MB 1.01, 1.8..2.3 MB 1.02
//   slices of 32: below 0.6 MB 0.94 to 0.96, 0.8..1 MB 0.96, 1..1.1 MB 0.98, 1.2..1.6 MB 1.00, 1.6..2 MB 1.04, 2..2.6 MB 1.07, 2.7..4.7 MB 1.10
//   slices of 64: below 0.4 MB 0.95, 0.5..0.7 MB 0.97, 0.9..1.5 MB 1.00, 1.5..1.9 MB 0.98, 2..2.6 MB 1.03, 2.7..4.1 MB 1.05, 4.3..7.5 MB 1.14 to 1.24
// (geometric mean of what is taken over the faster of the two: 1.002, 1.003, 1.004; by the best line for these calls 1.002, 1.003, 1.004).
// Above H 512, where a warp of a single CTA takes its rows in two rounds: slices of 16 1.16 to 1.24, of 32 1.31 to 1.33.
// Slices of 128 are always pairs: H 128 1.20, 256 1.18.  What pairs save in shared memory lets wider slices of wider layers
// fit: H 832 on 16 sequences (D7 L28 N15 436 -> 205 us), H 704 on 32, H 640 on 64.
bool take_pairs(int nb, int G, double rows, int H) {
  return nb == 128 || H > 512 || 2e-6 * (H / kUnits) * G * rows * H > (nb == 64 ? 1.1 : 1.4);
}

// Shared memory of a CTA with nb columns.
struct Fit {
  int slots;       // input tiles it leaves room for (0: does not fit)
  int held, ring;  // weight blocks kept there; blocks of the ring that the others pass through (0: all are kept)
  int streamed;
  uint32_t smem;
};
Fit fit(int nb, bool pair, int I, int H) {
  const int kb_h = H / BK, kb_x = std::max(I, H) / BK, copy_kb = 128 / nb, tmem_blocks = (512 - 2 * nb) / 32;
  const int in_smem = std::max(0, kb_h + kb_x - tmem_blocks);
  const uint32_t block = (pair ? nb / 2 : nb) * BK * 2, slot = (kb_x + copy_kb - 1) / copy_kb * copy_kb * block;
  const uint32_t fixed = 1024 + kb_h * block + in_smem * kWBlockBytes;
  if (fixed + slot <= kMaxSmem) {
    // (one for pairs: D8 L100 N64 H512 411 us a call, with two 420; D4 L100 N64 H256 on slices of 64 303 / 306)
    const int slots = std::min<int>(pair ? 1 : kMaxSlots, (kMaxSmem - fixed) / slot);
    return {slots, in_smem, 0, 0, fixed + slots * slot};
  }
  // (not on slices of 128: too little room is left, D14 L86 N113 H576 1293 us, the generic kernel 1202; D4 L64 N256 H512 430, slices of 64
  // 445)
  const uint32_t tiles = 1024 + kb_h * block + slot;
  if (!pair || nb == 128 || tiles >= kMaxSmem) return {};
  const int room = (kMaxSmem - tiles) / kWBlockBytes, n_rec = std::max(0, kb_h - tmem_blocks);
  const int ring = std::min(kMaxRing, room - n_rec);
  if (ring < 2) return {};
  return {1, room - ring, ring, in_smem - (room - ring), tiles + room * kWBlockBytes};
}

}  // namespace

static bool flow_takes(int dtype, int D, int N, int I, int H) {
  return (dtype == FTB_F16 || dtype == FTB_BF16) && N >= 1 && H % 64 == 0 && I % 64 == 0 && (D == 1 || I == H);
}

// Slices of a layer and layers beside each other with slices of nb sequences; false: a layer does not fit on the device.
static bool flow_grid(int D, int N, int H, int sm_count, int nb, FlowPlan* plan) {
  const int tiles = H / kUnits;
  plan->nb = nb;
  plan->S = (N + nb - 1) / nb;
  if (plan->S * tiles > sm_count) return false;
  const int most = std::min(D, sm_count / (plan->S * tiles)), sweeps = (D + most - 1) / most;
  plan->G = (D + sweeps - 1) / sweeps;
  return true;
}

// The kernel with slices, pairs and ring named; false: there is no such form of it.
bool lstm_flow_form(int dtype, int D, int N, int I, int H, int sm_count, int nb, bool pair, bool ring, FlowPlan* plan) {
  if (!flow_takes(dtype, D, N, I, H) || !(nb == 16 || nb == 32 || nb == 64 || (nb == 128 && pair))) return false;
  const Fit f = fit(nb, pair, I, H);
  plan->pair = pair;
  plan->ring = f.ring;
  plan->est_us = 0.0;
  return f.slots >= 1 && (f.ring > 0) == ring && flow_grid(D, N, H, sm_count, nb, plan);
}

// How the kernel would run a problem of T rows; est_us: about what that takes.  stream: input weights may pass through a ring.
bool lstm_flow_plan(int dtype, int D, int L, int N, int64_t T, int I, int H, int sm_count, bool stream, FlowPlan* plan) {
  if (!flow_takes(dtype, D, N, I, H)) return false;
  const int tiles = H / kUnits;
  bool found = false;
  for (int nb = 16; nb <= 128; nb *= 2) {
    FlowPlan p;
    if (!flow_grid(D, N, H, sm_count, nb, &p)) continue;
    const int S = p.S, G = p.G, sweeps = (D + G - 1) / G;
    const bool pair = take_pairs(nb, G, static_cast<double>(T) / L, H);
    const Fit f = fit(nb, pair, I, H);
    if (f.slots < 1 || (f.ring > 0 && !stream)) continue;
    // A step, what every layer adds to the first's start, a sweep's weights, the states' share of L2 and the call itself, fitted
    // to 5277 calls on every form that fits (3 to 7 % in the root mean square; of the forms of a call the one taken is 0.3 % behind
    // the fastest on average, 15 % at most).  A sweep begins when its CTAs are done with the one before and the layer below has begun.
    const double h = H / 512.0, over = std::max(0.0, h - 1.0);
    double step = pair ? (nb == 16   ? 1.24 + 0.42 * h + 0.32 * over
                          : nb == 32 ? 1.37 + 0.43 * h + 0.44 * over
                          : nb == 64 ? 1.84 + 0.76 * h + 0.77 * over
                                     : 2.20 + 1.41 * h + 0.30 * over)
                       : (nb == 16 ? 1.11 + 0.57 * h : nb == 32 ? 1.13 + 0.78 * h : 1.55 + 1.26 * h);
    // A block that passes through the ring costs its turn of the MMA warp, and all of them together their bytes from L2.
    const double mb = 1e-6 * S * tiles * G * f.streamed * kWBlockBytes;
    if (f.ring > 0) step += nb == 16 ? 0.094 * f.streamed + 0.020 * mb : nb == 32 ? 0.082 * f.streamed + 0.020 * mb : 0.078 * f.streamed + 0.018 * mb;
    const double steps = L * step, start = (G - 1) * (step + 2.3);
    const double us = 12.5 + (sweeps - 1) * std::max(steps, start) + steps + start + 4.7 * sweeps + 3.3e-6 * D * T * H;
    if (!found || us < plan->est_us) *plan = {nb, S, G, pair, f.ring, us};
    found = true;
  }
  return found;
}

// x: [T, I]; Wp: [D, 4H, I+H]; hs: [D, T, H]; c: [D, N, H]; off: device [L + 1] or nullptr (T = L * N);
// flags: D * L * S ints (zeroed here).
int launch_lstm_flow(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c, const int* off,
                     int64_t T, int D, int L, int N, int I, int H, const FlowPlan& plan, int* flags, int* status,
                     cudaStream_t stream) {
  FlowArgs a = {};
  const bool pair = plan.pair;
  const Fit f = fit(plan.nb, pair, I, H);
  if (f.slots < 1) return FTB_ERR_ARG;
  const uint32_t smem = f.smem;
  a.n_slots = f.slots;
  a.held = f.held;
  a.ring = f.ring;
  a.D = D; a.L = L; a.N = N; a.I = I; a.H = H; a.G = plan.G; a.S = plan.S;
  a.n_tiles = H / kUnits;
  a.T = T;
  a.off = off;
  a.bias_p = bias_p;
  a.Wp = Wp;
  a.hs = hs;
  a.c_out = c;
  a.c_rows = N;
  a.flag_steps = L;
  a.flags = flags;
  a.status = status;
  const uint32_t nb = plan.nb, held = pair ? nb / 2 : nb, planes = 128 / nb;
  CUtensorMap mX, mH, mW;
  int rc;
  a.by_step = off == nullptr;
  const uint64_t rows = a.by_step ? N : T, steps = a.by_step ? L : 1;
  if ((rc = make_tmap_steps(&mX, x, dtype, steps, rows, I, held, planes))) return rc;
  if ((rc = make_tmap_steps(&mH, hs, dtype, a.by_step ? D * steps : 1, a.by_step ? rows : D * rows, H, held, planes))) return rc;
  if ((rc = make_tmap_gates(&mW, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, I + H))) return rc;
  const int64_t chunks = static_cast<int64_t>(D) * T * H / 8;
  const int n_flags = D * L * a.S;
  flow_fill_kernel<<<static_cast<int>(std::min<int64_t>(current_sm_count(), (std::max<int64_t>(chunks, n_flags) + 255) / 256)), 256, 0, stream>>>(
      static_cast<uint4*>(hs), chunks, flags, n_flags);
  if (cudaGetLastError() != cudaSuccess) return FTB_ERR_LAUNCH;
  count_launch();
#define FTB_FLOW_ARGS mX, mH, mW, a, smem, stream
#define FTB_FLOW_LAUNCH(TT)                                                                                     \
  switch (plan.nb) {                                                                                            \
    case 16:                                                                                                    \
      if (f.ring > 0) return launch<TT, 16, true, true>(FTB_FLOW_ARGS);                                         \
      return pair ? launch<TT, 16, true>(FTB_FLOW_ARGS) : launch<TT, 16, false>(FTB_FLOW_ARGS);                 \
    case 32:                                                                                                    \
      if (f.ring > 0) return launch<TT, 32, true, true>(FTB_FLOW_ARGS);                                         \
      return pair ? launch<TT, 32, true>(FTB_FLOW_ARGS) : launch<TT, 32, false>(FTB_FLOW_ARGS);                 \
    case 64:                                                                                                    \
      if (f.ring > 0) return launch<TT, 64, true, true>(FTB_FLOW_ARGS);                                         \
      return pair ? launch<TT, 64, true>(FTB_FLOW_ARGS) : launch<TT, 64, false>(FTB_FLOW_ARGS);                 \
    default: return launch<TT, 128, true>(FTB_FLOW_ARGS);                                                       \
  }
  if (dtype == FTB_F16) {
    FTB_FLOW_LAUNCH(__half)
  }
  FTB_FLOW_LAUNCH(__nv_bfloat16)
#undef FTB_FLOW_LAUNCH
#undef FTB_FLOW_ARGS
}

}  // namespace ftb
