// Stacked LSTM forward with every weight on chip and hidden states that carry their own arrival:
// the 16-bit path of models whose layer tiles fit on the device (lstm_flow_plan below).
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
//   * the batch is cut into slices of NB columns that never meet (UMMA N = NB), each with its own CTAs.
//     What grows with NB is the state a CTA reads and its gates (20 cycles a column, tanh's 16 a cycle): slices are
//     as narrow as the device has CTAs for;
//   * the warps that have stored a step's state read the whole of it back: the chain is one set of warps
//     with no hand-over but the accumulator's barrier and the operand tile's.  They wait before the
//     first read for as long as it last took the state to arrive: reads that come too early load the L2
//     that the state has to pass through (8.5 us a step without the pause, 4.4 with it: D8 H512 N64);
//   * the layer below is read through TMA behind a flag per cell (a counter of the tiles stored), which
//     a warp of its own raises: its fences are off the chain, the layers above just run further behind;
//   * the input half of step t + 1 is issued right after the recurrent half of step t.
// The epilogue splits the batch columns so that a thread ends up with four consecutive sequences of
// its unit (4 x 4 transposes over the quad that holds the unit's gates), keeps their cell state in
// fp32 registers for the sweep, and two more shuffles make words of four units.
//
// A ragged batch (sorted by decreasing length, rows of a step packed) is the same kernel: the rows of
// step t start at off[t], and columns whose sequence has ended are neither stored nor waited for.
//
// Same arithmetic in the same order as the other 16-bit schedules: bit-identical results.
//
// Roles: warp 0 MMA issuer, warp 1 TMA producer (input tiles, shared-memory weights), warp 2 publisher,
// warps 4.. epilogue and state.  Cooperative launch.
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

template <typename T, int NB>
__global__ void __launch_bounds__(FlowCfg<NB>::kThreads, 1)
lstm_flow_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapH,
                 const __grid_constant__ CUtensorMap mapW, const FlowArgs a) {
  const int tile = blockIdx.x % a.n_tiles;
  const int slice = (blockIdx.x / a.n_tiles) % a.S;
  body<T, NB>(mapX, mapH, mapW, a, tile, slice, blockIdx.x / (a.n_tiles * a.S));
}

template <typename T, int NB>
int launch(const CUtensorMap& mX, const CUtensorMap& mH, const CUtensorMap& mW, const FlowArgs& a, uint32_t smem,
           cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = lstm_flow_kernel<T, NB>;
  if (!ensure_dynamic_smem(kfn, kMaxSmem, configured)) return FTB_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min(a.G, a.D) * a.S * a.n_tiles);
  cfg.blockDim = dim3(FlowCfg<NB>::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[1];
  int na = 0;
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

// Shared memory of a CTA with nb columns: the input tiles it leaves room for (0: does not fit).
int input_slots(int nb, int I, int H, uint32_t* smem) {
  const int kb_h = H / BK, kb_x = std::max(I, H) / BK, copy_kb = 128 / nb;
  const int in_smem = std::max(0, kb_h + kb_x - (512 - 2 * nb) / 32);
  const uint32_t block = nb * BK * 2, slot = (kb_x + copy_kb - 1) / copy_kb * copy_kb * block;
  const uint32_t fixed = 1024 + kb_h * block + in_smem * kWBlockBytes;
  if (fixed >= kMaxSmem) return 0;
  const int slots = std::min<int>(kMaxSlots, (kMaxSmem - fixed) / slot);
  *smem = fixed + slots * slot;
  return slots;
}

}  // namespace

// How the kernel would run a problem; est_us: about what that takes.
bool lstm_flow_plan(int dtype, int D, int L, int N, int I, int H, int sm_count, FlowPlan* plan) {
  if (dtype != FTB_F16 && dtype != FTB_BF16) return false;
  if (N < 1 || H % 64 != 0 || I % 64 != 0 || (D > 1 && I != H)) return false;
  const int tiles = H / kUnits;
  bool found = false;
  for (int nb = 16; nb <= 128; nb *= 2) {
    uint32_t smem = 0;
    if (input_slots(nb, I, H, &smem) < 1) continue;
    const int S = (N + nb - 1) / nb;
    if (S * tiles > sm_count) continue;
    int G = std::min(D, sm_count / (S * tiles));
    const int sweeps = (D + G - 1) / G;
    G = (D + sweeps - 1) / sweeps;
    // Measured steps: 1.8 / 2.0 us at 16 columns and H 256 / 512, 2.2 / 2.6 at 32, 3.0 / 4.3 at 64, more with more CTAs
    // at work; a state of more than eight K blocks is read in two rounds.
    const double busy = static_cast<double>(S * tiles * G) / sm_count;
    const double step = 1.2 + nb / 64.0 + nb * H / 16800.0 + (H > 512 ? 0.5 : 0.0) + 0.3 * busy * nb / 64.0;
    const double us = sweeps * ((L + G - 1) * step + 10.0);
    if (!found || us < plan->est_us) *plan = {nb, S, G, us};
    found = true;
  }
  return found;
}

// x: [T, I]; Wp: [D, 4H, I+H]; hs: [D, T, H]; c: [D, N, H]; off: device [L + 1] or nullptr (T = L * N);
// flags: D * L * S ints (zeroed here).
int launch_lstm_flow(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c, const int* off,
                     int64_t T, int D, int L, int N, int I, int H, const FlowPlan& plan, int* flags, int* status,
                     cudaStream_t stream) {
  FlowArgs a;
  uint32_t smem = 0;
  a.n_slots = input_slots(plan.nb, I, H, &smem);
  if (a.n_slots < 1) return FTB_ERR_ARG;
  a.D = D; a.L = L; a.N = N; a.I = I; a.H = H; a.G = plan.G; a.S = plan.S;
  a.n_tiles = H / kUnits;
  a.T = T;
  a.off = off;
  a.bias_p = bias_p;
  a.Wp = Wp;
  a.hs = hs;
  a.c_out = c;
  a.c_rows = N;
  a.nb_below = plan.nb;
  a.flags = flags;
  a.status = status;
  const uint32_t nb = plan.nb, planes = 128 / plan.nb;
  CUtensorMap mX, mH, mW;
  int rc;
  if ((rc = make_tmap_3d(&mX, x, dtype, 64, T, I / BK, static_cast<uint64_t>(I) * 2, 128, 64, nb, planes))) return rc;
  if ((rc = make_tmap_3d(&mH, hs, dtype, 64, static_cast<uint64_t>(D) * T, H / BK, static_cast<uint64_t>(H) * 2, 128, 64,
                         nb, planes)))
    return rc;
  if ((rc = make_tmap_2d(&mW, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, I + H, I + H, kGateRows, BK))) return rc;
  if (cudaMemsetAsync(hs, 0xFF, static_cast<size_t>(D) * T * H * 2, stream) != cudaSuccess ||
      cudaMemsetAsync(flags, 0, sizeof(int) * static_cast<size_t>(D) * L * a.S, stream) != cudaSuccess)
    return FTB_ERR_LAUNCH;
#define FTB_FLOW_LAUNCH(TT)                                         \
  switch (plan.nb) {                                                \
    case 16: return launch<TT, 16>(mX, mH, mW, a, smem, stream);        \
    case 32: return launch<TT, 32>(mX, mH, mW, a, smem, stream);        \
    case 64: return launch<TT, 64>(mX, mH, mW, a, smem, stream);        \
    default: return launch<TT, 128>(mX, mH, mW, a, smem, stream);       \
  }
  if (dtype == FTB_F16) {
    FTB_FLOW_LAUNCH(__half)
  }
  FTB_FLOW_LAUNCH(__nv_bfloat16)
#undef FTB_FLOW_LAUNCH
}

}  // namespace ftb
