// Grid RNN forward with weights on chip and hidden states that carry their own arrival: the 16-bit path for H up to 256.
//
// A grid row of a batch slice is a chain of B dependent cells; cell (a, b) waits for h_x of the row above and h_y of the column
// before, both of the previous anti-diagonal, so the time is A + B + D - 2 steps of a cell.  The kernel before this one handed h_y
// on through a cluster's shared memory (48 KB a CTA and step at 14 bytes a cycle) and h_x behind a flag (store, fence, release,
// poll, TMA: 3.8 us): 4.1 us a step at H 256 and 64 sequences, for slices of 64 only, and grids with more rows than the device has
// clusters for, or of H 64, went through the generic wavefront at 6 to 11 us a step.  Here, as in csrc/lstm_flow.cu,
//   * the output arrays are their own flags: a cell is 0xFFFF, which no hidden state is, until its states are stored as 8-byte
//     words; the CTAs that need them read until every word has arrived, h_x and h_y alike, straight into the MMA's operand tiles;
//   * the weights of a direction (3H x 128 units a CTA) sit in tensor memory.  Above 128 units the two CTAs of a direction are a
//     pair (.cta_group::2) and each holds half of the sequences' states;
//   * the batch is cut into slices of NB columns, and (layer, row, slice) chains are dealt to the groups of CTAs that the device
//     holds in the order in which they can start (row + layer), so that grids of any size run, of up to 4096 sequences: a group
//     that is done with its chain takes the next one, with other weights where the layer changes;
//   * nobody fills the arrays before the launch.  A warp of every CTA writes 0xFFFF into its own part kAhead columns ahead of the
//     sweep, counts every kFill columns of a chain in (`ready`), and waits there for those that this CTA reads: its chain's others
//     and the chain above.  The epilogue looks at a column when that warp says so (`n_clear`), steps after it did.
// Same arithmetic in the same order as the other 16-bit schedules: bit-identical results.
//
// Roles: warp 0 MMA issuer, warp 1 TMA producer (inputs), warp 2 publisher (a cell's inputs of the layer above), warp 3 fill,
// warps 4.. epilogue and states.  Cooperative launch.  Of a pair the even CTA issues the MMAs.
//
// Program: stacked_grid_rnns() (examples/grid_rnn/grid_rnn.py:42-122) in place of the grid regions
// (benchmarks/rnn/fractaltensor/grid_lstm/regions/region{1..8}.h).
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "flow_plan.h"
#include "lstm_flow.cuh"

namespace ftb {

namespace {

using flow::arrived;
using flow::ld_relaxed_gpu_2x64;
using flow::st_relaxed_gpu64;

constexpr int BK = 64;
constexpr int kTileUnits = 128;
constexpr int kFirstEpi = 4;
constexpr int kSlots = 4;    // input tiles
constexpr int kAhead = 16;   // columns that are filled ahead of the sweep,
constexpr int kFill = 8;     // so many to a count (two counts ahead: who waits for a count can still do the columns of the one before)
constexpr int kMaxPause = 4000;  // cycles
constexpr uint32_t kOneCta = 120 * 1024;  // shared memory of which only one CTA fits on an SM: both would want all of tensor memory

template <int NB, bool kPair>
struct GridCfg {
  static constexpr int kCtas = kPair ? 2 : 1;
  static constexpr int kHeld = NB / kCtas;   // rows of a state that a CTA holds
  static constexpr int kWarps = NB / 4;      // epilogue warps: 32 units x 16 columns each
  static constexpr int kRows = kHeld / kWarps;  // state rows that a warp reads: 2 or 4, and
  static constexpr int kParts = 4 / kRows;      // each by so many groups of eight lanes
  static constexpr int kThreads = 32 * (kFirstEpi + kWarps);
  static constexpr uint32_t kBlockBytes = kHeld * BK * 2;
  // A pause in cycles before the first look, learnt from how many looks it took: looks that come too early load the L2 that the
  // states have to pass.  On slices of 64 it pays (32 x 32, H 256: 64 sequences 203 -> 190 us, 512 933 -> 713), on narrower ones
  // looking at once is faster (32 sequences on slices of 32 128 -> 123 us, 16 on 16 111 -> 101).
  static constexpr bool kPause = NB == 64;
};

struct GridArgs {
  int D, A, B, N, H, S;
  int tiles;            // CTAs of a direction
  int groups;           // chains beside each other
  const void *Wx, *Wy;  // [D, H, 3H], K order state_x, state_y, input
  const float *bx, *by;  // [D, H] or nullptr
  void *hx, *hy;         // [D, A, B, N, H]
  int* ready;            // [D * A * S][counts] CTAs of the chain that have filled these kFill columns
  int counts;            // of a chain
  int* flags;            // [D * A * B * S * 2] tiles of the cell and direction that can be read through TMA (D > 1)
  int* status;
};

struct Chain {
  int d, a, s;
};
// Chain c in the order of row + layer.
__device__ __forceinline__ Chain chain_of(const GridArgs& g, int c) {
  Chain r;
  r.s = c % g.S;
  c /= g.S;
  for (int m = 0;; ++m) {
    const int d0 = max(0, m - g.A + 1), n = min(m, g.D - 1) - d0 + 1;
    if (c < n) {
      r.d = d0 + c;
      r.a = m - r.d;
      return r;
    }
    c -= n;
  }
}
__device__ __forceinline__ int* ready_of(const GridArgs& g, int d, int a, int s, int count) {
  return g.ready + (static_cast<int64_t>(d * g.A + a) * g.S + s) * g.counts + count;
}

template <typename T, int NB, bool kPair>
__global__ void __launch_bounds__(GridCfg<NB, kPair>::kThreads, 1)
grid_flow_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapY,
                 const __grid_constant__ CUtensorMap mapHx, const __grid_constant__ CUtensorMap mapHy, const GridArgs g) {
  using C = GridCfg<NB, kPair>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t in_full[kSlots], in_empty[kSlots];
  __shared__ uint64_t st_full;  // the neighbours' states are in their operand tiles
  __shared__ uint64_t acc_full[2], acc_empty[2];
  __shared__ uint64_t w_full;   // the chain's weights are in place
  __shared__ uint32_t tmem_base_s;
  __shared__ int n_stored;      // epilogue warps that have stored a column, summed over columns
  __shared__ int n_clear;       // columns that this CTA may read, over all chains
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* status = g.status;
  const int kbh = g.H / BK;
  const uint32_t tile_bytes = kbh * C::kBlockBytes;
  uint8_t* s_state = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // of the row above, of the column before
  uint8_t* s_in = s_state + 2 * tile_bytes;

  if (threadIdx.x == 0) {
    prefetch_tmap(&mapX);
    prefetch_tmap(&mapY);
    prefetch_tmap(&mapHx);
    prefetch_tmap(&mapHy);
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&in_full[i], 1);
      mbar_init(&in_empty[i], 1);
    }
    mbar_init(&st_full, C::kCtas * C::kWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], C::kCtas * C::kWarps);
    }
    mbar_init(&w_full, C::kCtas * C::kWarps);
    n_stored = 0;
    n_clear = 0;
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    if constexpr (kPair) {
      tmem_alloc_pair(&tmem_base_s, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&tmem_base_s, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (kPair) cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tmem_w = tmem_base + 2 * NB;

  const int rank = kPair ? static_cast<int>(cluster_ctarank()) : 0;
  const int group = blockIdx.x / (2 * g.tiles), in_group = blockIdx.x - group * 2 * g.tiles;
  const bool ydir = in_group >= g.tiles;
  const int tile = in_group - (ydir ? g.tiles : 0);  // of the direction's units (a pair: its rank)
  const int n_chains = g.D * g.A * g.S;
  auto commit = [](uint64_t* bar) {
    if constexpr (kPair) umma_commit_pair(bar); else umma_commit(bar);
  };
  auto arrive_at_issuer = [](uint64_t* bar) {
    if constexpr (kPair) mbar_arrive_peer(map_to_cta(smem_u32(bar), 0)); else mbar_arrive(bar);
  };
  auto give_up = [&](int code) {
    if (s_abort == 0) {
      s_abort = 1;
      atomicCAS(status, 0, code);
    }
  };

  if (warp == 0 && rank == 0) {
    // -------------------------------------------------------------- MMA issuer
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_f16(C::kCtas * 128, NB, Fmt<T>::kind, 0, 0);
    const uint64_t in_desc = make_sdesc_sw128(smem_u32(s_in), 16, 1024);
    const uint64_t state_desc = make_sdesc_sw128(smem_u32(s_state), 16, 1024);
    constexpr uint32_t kBlockDesc = C::kBlockBytes >> 4;
    auto mma = [](uint32_t d, uint32_t aw, uint64_t bd, uint32_t accumulate) {
      if constexpr (kPair) umma_ts_pair(d, aw, bd, idesc, accumulate); else umma_ts(d, aw, bd, idesc, accumulate);
    };
    // The K blocks of one operand (unrolled: a loop turn costs more than a block's MMAs, csrc/lstm_flow.cuh).
    auto blocks = [&](uint32_t d_tmem, uint32_t aw, uint64_t bd, uint32_t accumulate) {
      if (kbh == 4) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 16; ++i) mma(d_tmem, aw + 8 * i, bd + (i >> 2) * kBlockDesc + 2 * (i & 3), i > 0 ? 1u : accumulate);
        }
        return;
      }
      if (kbh & 2) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 8; ++i) mma(d_tmem, aw + 8 * i, bd + (i >> 2) * kBlockDesc + 2 * (i & 3), i > 0 ? 1u : accumulate);
        }
        aw += 2 * 32;
        bd += 2 * kBlockDesc;
        accumulate = 1;
      }
      if (kbh & 1) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 4; ++i) mma(d_tmem, aw + 8 * i, bd + 2 * i, i > 0 ? 1u : accumulate);
        }
      }
    };
    int slot = 0, k = 0, states = 0, chains = 0;  // k: columns started, states: operand pairs received
    uint32_t phase = 0;
    bool ok = true;
    for (int c = group; c < n_chains && ok; c += g.groups, ++chains) {
      const Chain ch = chain_of(g, c);
      ok = mbar_wait_warp(&w_full, chains & 1, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
      if (!ok) break;
      tc_fence_after();
      for (int b = 0; b < g.B; ++b, ++k) {
        const int acc = k & 1;
        const uint32_t d_tmem = tmem_base + acc * NB;
        ok = mbar_wait_warp(&acc_empty[acc], ((k >> 1) & 1) ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_EPI) &&
             mbar_wait_warp(&in_full[slot], phase, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
        if (!ok) break;
        tc_fence_after();
        blocks(d_tmem, tmem_w + 2 * kbh * 32, in_desc + static_cast<uint64_t>((slot * tile_bytes) >> 4), 0u);
        if (leader) commit(&in_empty[slot]);
        if (++slot == kSlots) {
          slot = 0;
          phase ^= 1u;
        }
        if (ch.a > 0 || b > 0) {
          // (the other CTA's rows are ordered by an acquire of the cluster's scope, as their release is)
          if constexpr (kPair)
            ok = __all_sync(0xffffffffu, mbar_wait_cluster(&st_full, states & 1, &s_abort, status, FTB_ERR_TIMEOUT_DEP));
          else
            ok = mbar_wait_warp(&st_full, states & 1, &s_abort, status, FTB_ERR_TIMEOUT_DEP);
          if (!ok) break;
          if (ch.a > 0) blocks(d_tmem, tmem_w, state_desc, 1u);
          if (b > 0) blocks(d_tmem, tmem_w + kbh * 32, state_desc + static_cast<uint64_t>(tile_bytes >> 4), 1u);
          ++states;
        }
        if (leader) commit(&acc_full[acc]);
      }
    }
  } else if (warp == 1) {
    // ----------------------------------- TMA: inputs, of the call or of the layer below
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int c = group; c < n_chains && ok; c += g.groups) {
      const Chain ch = chain_of(g, c);
      const CUtensorMap* map = ch.d == 0 ? (ydir ? &mapY : &mapX) : (ydir ? &mapHy : &mapHx);
      for (int b = 0; b < g.B && ok; ++b) {
        const int64_t cell = (static_cast<int64_t>(max(ch.d - 1, 0)) * g.A + ch.a) * g.B + b;
        if (ch.d > 0) {
          if (lane == 0) ok = flag_wait_ge(g.flags + (cell * g.S + ch.s) * 2 + ydir, g.tiles, &s_abort, status, FTB_ERR_TIMEOUT_DEP);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          fence_proxy_async_global();  // threads of other CTAs stored what TMA reads
        }
        ok = mbar_wait_warp(&in_empty[slot], phase ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_SLOT);
        if (!ok) break;
        if (lane == 0) {
          // (rows past the batch belong to other cells: their columns of the accumulator are not stored)
          const int row = static_cast<int>(cell * g.N + ch.s * NB + rank * C::kHeld);
          if (rank == 0) mbar_arrive_expect_tx(&in_full[slot], C::kCtas * tile_bytes);
          if constexpr (kPair)
            tma_load_3d_pair(s_in + slot * tile_bytes, map, map_to_cta(smem_u32(&in_full[slot]), 0), 0, row, 0);
          else
            tma_load_3d(s_in + slot * tile_bytes, map, &in_full[slot], 0, row, 0);
        }
        if (++slot == kSlots) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
    if (kPair && ok) ring_drain(in_empty, kSlots, slot, phase, &s_abort, status);
  } else if (warp == 2) {
    // ----------------------------------- publisher: the layer above can read a cell through TMA
    if (lane == 0 && g.D > 1) {
      volatile int* abort_flag = &s_abort;
      volatile int* stored = &n_stored;
      int want = 0;
      bool ok = true;
      for (int c = group; c < n_chains && ok; c += g.groups) {
        const Chain ch = chain_of(g, c);
        for (int b = 0; b < g.B; ++b) {
          want += C::kWarps;
          if (ch.d + 1 == g.D) continue;
          uint64_t t0 = 0;
          for (uint32_t it = 1; *stored < want; ++it) {
            if ((it & 0x3F) != 0) continue;
            if (t0 == 0) t0 = globaltimer_ns();
            if (*abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS) {
              ok = false;
              break;
            }
          }
          if (!ok) {
            give_up(FTB_ERR_TIMEOUT_EPI);
            break;
          }
          __threadfence_block();
          // (The release takes the other warps' stores along; the proxy fence is the reader's, between its acquire and its copy.)
          const int64_t cell = (static_cast<int64_t>(ch.d) * g.A + ch.a) * g.B + b;
          red_release_gpu_add(g.flags + (cell * g.S + ch.s) * 2 + ydir, 1);
        }
      }
    }
  } else if (warp == 3) {
    // ----------------------------------- fill: this CTA's part of the columns ahead of the sweep
    volatile int* abort_flag = &s_abort;
    volatile int* stored = &n_stored;
    const int units = min(kTileUnits, g.H - tile * kTileUnits), lanes = units / 8;  // lanes that fill a row, 16 bytes each
    int total = 0;
    bool ok = true;
    for (int c = group; c < n_chains && ok; c += g.groups) {
      const Chain ch = chain_of(g, c);
      const int rows = min(NB, g.N - ch.s * NB);
      uint16_t* out = static_cast<uint16_t*>(ydir ? g.hy : g.hx) + tile * kTileUnits + (lane % lanes) * 8;
      for (int b = 0; b < g.B; ++b) {
        uint64_t t0 = 0;
        for (uint32_t it = 1; total >= *stored / C::kWarps + kAhead; ++it) {
          if ((it & 0xF) == 0) {
            if (t0 == 0) t0 = globaltimer_ns();
            if (*abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS) {
              ok = false;
              break;
            }
          }
          __nanosleep(200);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) give_up(FTB_ERR_TIMEOUT_EPI);
          break;
        }
        const int64_t row0 = ((static_cast<int64_t>(ch.d) * g.A + ch.a) * g.B + b) * g.N + ch.s * NB;
        for (int n = lane / lanes; n < rows; n += 32 / lanes)
          *reinterpret_cast<uint4*>(out + (row0 + n) * g.H) = make_uint4(~0u, ~0u, ~0u, ~0u);
        __syncwarp();
        ++total;
        if ((b + 1) % kFill != 0 && b + 1 < g.B) continue;
        if (lane == 0) {
          const int count = b / kFill;
          __threadfence();
          red_release_gpu_add(ready_of(g, ch.d, ch.a, ch.s, count), 1);
          // (the row two above for the first look of a chain alone, below)
          for (int up = 0; up <= (count == 0 ? 2 : 1) && up <= ch.a && ok; ++up)
            ok = flag_wait_ge(ready_of(g, ch.d, ch.a - up, ch.s, count), 2 * g.tiles, &s_abort, status, FTB_ERR_TIMEOUT_DEP);
          __threadfence_block();
          if (ok) *const_cast<volatile int*>(&n_clear) = total;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
    }
  } else if (warp >= kFirstEpi) {
    // ------------------------------------------------------- epilogue and states
    const int q = warp & 3, w = warp - kFirstEpi, sub = w >> 2;
    const int r_loc = q * 32 + lane, unit = tile * kTileUnits + r_loc;
    const bool real = unit < g.H;  // (whole warps)
    const bool ub0 = (lane & 1) != 0, ub1 = (lane & 2) != 0;
    // After the exchange below this lane stores four units of sequence n_store of every four.
    const int n_store = sub * 16 + (ub0 ? 2 : 0) + (ub1 ? 1 : 0);
    // What this lane reads of a state: 16 bytes of K blocks `part`, part + kParts of row n_load of those that this CTA holds.
    const int n_load = w * C::kRows + (lane >> 3) % C::kRows, part = (lane >> 3) / C::kRows;
    const uint32_t dst0 = n_load * 128 + (((lane & 7) ^ (n_load & 7)) << 4);
    volatile int* abort_flag = &s_abort;
    volatile int* clear = &n_clear;
    // Columns before `want` can be read: no wait but for a fill that was held up.
    auto cleared = [&](int want) {
      uint64_t t0 = 0;
      bool fine = true;
      for (uint32_t it = 1; *clear < want && fine; ++it) {
        if ((it & 0x3F) != 0) continue;
        if (t0 == 0) t0 = globaltimer_ns();
        if (*abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS) {
          give_up(FTB_ERR_TIMEOUT_EPI);
          fine = false;
        }
      }
      __threadfence_block();
      return __all_sync(0xffffffffu, fine) != 0;
    };
    const T* hx = reinterpret_cast<const T*>(g.hx);
    const T* hy = reinterpret_cast<const T*>(g.hy);
    T* out = reinterpret_cast<T*>(ydir ? g.hy : g.hx);
    const int64_t column = static_cast<int64_t>(g.N) * g.H;
    int k = 0, pause = 300, layer = -1;
    float bias = 0.f;
    bool ok = true;
    for (int c = group; c < n_chains && ok; c += g.groups) {
      const Chain ch = chain_of(g, c);
      if (ch.d != layer) {
        // Weights -> tensor memory (the last column's accumulator is complete, so no MMA reads them): thread r copies row r,
        // two 16-bit values to a column, the warps of a quadrant take K blocks in turn.
        layer = ch.d;
        const uint4* wrow = reinterpret_cast<const uint4*>(static_cast<const T*>(ydir ? g.Wy : g.Wx) +
                                                           (static_cast<size_t>(layer) * g.H + (real ? unit : 0)) * 3 * g.H);
        for (int kb = sub; kb < 3 * kbh; kb += C::kWarps / 4) {
          uint32_t v[32];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 x4 = __ldg(wrow + kb * 8 + i);
            v[4 * i + 0] = x4.x; v[4 * i + 1] = x4.y; v[4 * i + 2] = x4.z; v[4 * i + 3] = x4.w;
          }
          tmem_st32(tmem_w + (static_cast<uint32_t>(q * 32) << 16) + kb * 32, v);
        }
        tmem_st_wait();
        const float* bp = ydir ? g.by : g.bx;
        if (bp != nullptr && real) bias = __ldg(bp + static_cast<size_t>(layer) * g.H + unit);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_at_issuer(&w_full);
      const int n_base = ch.s * NB;
      const bool mine = n_base + rank * C::kHeld + n_load < g.N;
      const int64_t cell0 = (static_cast<int64_t>(ch.d) * g.A + ch.a) * g.B;
      ok = cleared(k + 1);
      // The first state of the row two above says that the one above is about to start: until then this chain looks at one word
      // and not at all of them.
      if (lane == 0) {
        if (ok && ch.a > 1) {
          const T* first = hx + ((cell0 - 2 * g.B) * g.N + n_base) * g.H;
          uint64_t t0 = 0;
          for (uint32_t it = 1; ok; ++it) {
            uint64_t x, y;
            ld_relaxed_gpu_2x64(first, x, y);
            if (arrived(x)) break;
            if ((it & 0x3F) == 0) {
              if (t0 == 0) t0 = globaltimer_ns();
              if (*abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS) {
                give_up(FTB_ERR_TIMEOUT_DEP);
                ok = false;
              }
            }
          }
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      __syncwarp();
      // h_x of the row above (loads 0, 1) and h_y of the column before (2, 3); what this lane stores
      const T* src_x = hx + ((cell0 - g.B) * g.N + n_base + rank * C::kHeld + n_load) * g.H + part * BK + (lane & 7) * 8;
      const T* src_y = hy + ((cell0 - 1) * g.N + n_base + rank * C::kHeld + n_load) * g.H + part * BK + (lane & 7) * 8;
      T* dst = out + (cell0 * g.N + n_base + n_store) * g.H + (unit & ~3);
      uint32_t looks = 0, stores = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (mine && part + (i & 1) * C::kParts < kbh && (i > 1 || ch.a > 0)) looks |= 1u << i;
        if (real && n_base + n_store + 4 * i < g.N) stores |= 1u << i;
      }
      bool counted = true;  // the last column's stores, for the publisher and the fill
      auto count_in = [&] {
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          atomicAdd(&n_stored, 1);
        }
        counted = true;
      };
      for (int b = 0; b < g.B && ok; ++b, ++k, src_x += column, src_y += column, dst += column) {
        if (ch.a > 0 || b > 0) {
          uint64_t x[4], y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i] = y[i] = 0;
          uint32_t missing = b > 0 ? looks : looks & 3u;
          uint64_t t0 = 0;
          uint32_t it = 1;
          for (;; ++it) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (missing & (1u << i)) ld_relaxed_gpu_2x64((i < 2 ? src_x : src_y) + (i & 1) * C::kParts * BK, x[i], y[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (arrived(x[i]) && arrived(y[i])) missing &= ~(1u << i);
            if (__all_sync(0xffffffffu, missing == 0)) break;
            if ((it & 0x3F) == 0) {
              if (t0 == 0) t0 = globaltimer_ns();
              if (__any_sync(0xffffffffu, *abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS)) {
                if (lane == 0) give_up(FTB_ERR_TIMEOUT_DEP);
                ok = false;
                break;
              }
            }
          }
          if (!ok) break;
          if constexpr (C::kPause) {
            // Everything at the first look: try a little earlier next time.  At the second or third: later.  (More looks than
            // that wait for a chain that is behind, whatever the pause.)
            if (it == 1) pause -= pause >> 5;
            else if (it <= 3) pause = min(pause + 100, kMaxPause);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (part + (i & 1) * C::kParts < kbh)
              *reinterpret_cast<ulonglong2*>(s_state + (i >> 1) * tile_bytes + (part + (i & 1) * C::kParts) * C::kBlockBytes + dst0) =
                  make_ulonglong2(x[i], y[i]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if constexpr (kPair) mbar_arrive_peer_smem(map_to_cta(smem_u32(&st_full), 0)); else mbar_arrive(&st_full);
          }
        }
        // While the MMAs run: the last column's stores are counted in, and the next look is cleared.
        if (!counted) count_in();
        if (b + 1 < g.B) ok = cleared(k + 2);
        if (!ok) break;
        const int acc = k & 1;
        ok = mbar_wait_warp(&acc_full[acc], (k >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after();
        uint32_t r[16];
        tmem_ld16(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * NB + sub * 16, r);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at_issuer(&acc_empty[acc]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float h[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) h[j] = tanh_fast(__uint_as_float(r[4 * i + j]) + bias);
          // (unit, 4 sequences) -> (4 units, 1 sequence): trade halves with the units next to this one, twice
          const uint32_t p01 = Fmt<T>::pack2(h[0], h[1]), p23 = Fmt<T>::pack2(h[2], h[3]);
          uint32_t other = __shfl_xor_sync(0xffffffffu, ub0 ? p01 : p23, 1);
          const uint32_t lo = ub0 ? other : p01, hi = ub0 ? p23 : other;  // units u & ~1 and u | 1
          const uint32_t w0 = __byte_perm(lo, hi, 0x5410), w1 = __byte_perm(lo, hi, 0x7632);
          other = __shfl_xor_sync(0xffffffffu, ub1 ? w0 : w1, 2);
          if (stores & (1u << i)) st_relaxed_gpu64(dst + i * 4 * g.H, ub1 ? other : w0, ub1 ? w1 : other);
        }
        counted = false;
        if constexpr (C::kPause) {
          const long long c0 = clock64();
          while (clock64() - c0 < pause) {}
        }
      }
      if (!counted) count_in();
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  // Neither CTA of a pair may leave while the other can still signal its barriers.
  if constexpr (kPair) cluster_sync_all();
  if (warp == 0) {
    if (s_abort) {
      // Give copies and MMAs still in flight time to land before TMEM and shared memory go back.
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    if constexpr (kPair) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, int NB, bool kPair>
int launch(const CUtensorMap* m, const GridArgs& g, uint32_t smem, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = grid_flow_kernel<T, NB, kPair>;
  if (!ensure_dynamic_smem(kfn, flow::kMaxSmem, configured)) return FTB_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.groups * 2 * g.tiles);
  cfg.blockDim = dim3(GridCfg<NB, kPair>::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
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
  if (cudaLaunchKernelEx(&cfg, kfn, m[0], m[1], m[2], m[3], g) != cudaSuccess) {
    cudaGetLastError();
    return FTB_ERR_LAUNCH;
  }
  count_launch();
  return FTB_OK;
}

}  // namespace

constexpr int kGridMaxSlices = 64;
static size_t grid_flow_counters(int D, int A, int B, int64_t S) {
  return static_cast<size_t>(D) * A * S * ((static_cast<size_t>(B) + kFill - 1) / kFill + (D > 1 ? 2 * static_cast<size_t>(B) : 0));
}
// Counters of a call of N sequences on the narrowest slices; N 0: of any batch.
size_t grid_flow_ints(int D, int A, int B, int N) {
  return grid_flow_counters(D, A, B, N == 0 ? kGridMaxSlices : std::min<int64_t>(kGridMaxSlices, (N + INT64_C(15)) / 16));
}

// The kernel with slices of nb sequences; false: there is no such form of it.
bool grid_flow_form(int dtype, int D, int A, int B, int N, int H, int sm_count, int nb, GridFlowPlan* plan) {
  if ((dtype != FTB_F16 && dtype != FTB_BF16) || H < 64 || H > 256 || H % 64 != 0 || N < 1) return false;
  if (!(nb == 16 || nb == 32 || nb == 64)) return false;
  plan->nb = nb;
  plan->S = (N + nb - 1) / nb;
  plan->groups = std::min(static_cast<int64_t>(sm_count / (2 * ((H + 127) / 128))), static_cast<int64_t>(D) * A * plan->S);
  plan->ints = grid_flow_counters(D, A, B, plan->S);
  plan->est_us = 0.0;
  return plan->S <= kGridMaxSlices && plan->groups >= 1;
}

// How the kernel would run a problem with room for max_ints counters; est_us: about what that takes.
bool grid_flow_plan(int dtype, int D, int A, int B, int N, int H, int sm_count, size_t max_ints, GridFlowPlan* plan) {
  bool found = false;
  for (int nb = 16; nb <= 64; nb *= 2) {
    GridFlowPlan p;
    if (!grid_flow_form(dtype, D, A, B, N, H, sm_count, nb, &p) || p.ints > max_ints) continue;
    // Steps until the last chain is done: a chain starts a step behind the one before it in its group (two with other weights), a
    // step after the row above and three after the layer below, and takes B.
    std::vector<double> free_at(p.groups, 0.0), start(static_cast<size_t>(D) * A * p.S, 0.0);
    std::vector<int> layer(p.groups, -1);
    double last = 0.0;
    int c = 0;
    for (int m = 0; m < A + D - 1; ++m)
      for (int d = std::max(0, m - A + 1); d <= std::min(m, D - 1); ++d)
        for (int s = 0; s < p.S; ++s, ++c) {
          const int a = m - d, g = c % p.groups;
          double t = free_at[g] + (layer[g] < 0 ? 0.0 : layer[g] != d ? 2.0 : 1.0);
          if (a > 0) t = std::max(t, start[static_cast<size_t>(d * A + a - 1) * p.S + s] + 1.0);
          if (d > 0) t = std::max(t, start[static_cast<size_t>((d - 1) * A + a) * p.S + s] + 3.0);
          start[static_cast<size_t>(d * A + a) * p.S + s] = t;
          layer[g] = d;
          free_at[g] = t + B;
          last = std::max(last, t + B);
        }
    // A step, fitted to 170 grids (D 1..3, A and B 2..48, N 1..400, H 64..256; 9, 6 and 5 % in the root mean square for the three
    // widths).  Rows and chains beside each other weigh with the bytes that they read.  The width taken is within 0.1 % of the
    // fastest on average (worst 7 %) of 123 grids of 6 to 40 rows and columns and 4 to 64 sequences, and 0.15 to 0.7 times the
    // generic wavefront's time; of 700 grids of 1 to 64 rows and columns and 1 to 4096 sequences within 0.8 % (worst 36 %).
    const double h = H / 256.0, load = h * p.groups / (sm_count / (2 * ((H + 127) / 128))) * std::min(N, nb) / nb;
    const double step = nb == 16 ? 1.05 + 0.37 * h + 0.13 * load : nb == 32 ? 1.13 + 0.38 * h + 0.42 * load : 1.40 + 0.69 * h + 0.73 * load;
    p.est_us = (nb == 16 ? 12.8 : nb == 32 ? 14.4 : 16.7) + last * step;
    if (!found || p.est_us < plan->est_us) *plan = p;
    found = true;
  }
  // Chains of a few columns, many of them one behind the other, spend their time between chains: there the generic wavefront is
  // the faster one, whose tiles large batches fill (us, this / generic: D2 A40 B1 N3613 H256 1024 / 421, D3 A14 B1 N1715 H192 268 /
  // 146, D3 A20 B2 N2798 H192 732 / 538; D3 A32 B15 N1999 H256 4494 / 5245).  Its time by levels and by rounds of tiles, fitted to 184
  // grids of up to 4 columns and 100 sequences or more (11 % in the root mean square); of the 700 it is taken for 20.
  if (found && B <= 4 && static_cast<int64_t>(D) * A * plan->S > 4 * plan->groups) {
    const double h = H / 256.0, rounds = 2.0 * D * A * B * ((N + 127) / 128) / sm_count;
    if (10.8 + (A + B + D - 2) * (5.5 + 1.87 * h) + rounds * (1.45 + 6.37 * h) < plan->est_us) return false;
  }
  return found;
}

// X, Y: [A, B, N, H]; Wpx, Wpy: [D, H, 3H]; hx, hy: [D, A, B, N, H]; counters: plan.ints of them (zeroed here).
int launch_grid_flow(int dtype, const void* X, const void* Y, const void* Wpx, const void* Wpy, const float* bias_x,
                     const float* bias_y, void* hx, void* hy, int D, int A, int B, int N, int H, const GridFlowPlan& plan,
                     int* counters, int* status, cudaStream_t stream) {
  GridArgs g = {};
  g.D = D; g.A = A; g.B = B; g.N = N; g.H = H; g.S = plan.S;
  g.tiles = (H + kTileUnits - 1) / kTileUnits;
  g.groups = plan.groups;
  g.Wx = Wpx; g.Wy = Wpy; g.bx = bias_x; g.by = bias_y; g.hx = hx; g.hy = hy;
  g.ready = counters;
  g.counts = (B + kFill - 1) / kFill;
  g.flags = counters + static_cast<size_t>(D) * A * plan.S * g.counts;
  g.status = status;
  const bool pair = g.tiles == 2;
  const uint32_t held = pair ? plan.nb / 2 : plan.nb, planes = H / BK;
  const uint64_t rows = static_cast<uint64_t>(A) * B * N;
  CUtensorMap m[4];
  const void* base[4] = {X, Y, hx, hy};
  for (int i = 0; i < 4; ++i) {
    const int rc = make_tmap_3d(&m[i], base[i], dtype, 64, i < 2 ? rows : rows * D, planes, static_cast<uint64_t>(H) * 2, 128, 64,
                                held, planes);
    if (rc) return rc;
  }
  const uint32_t smem = std::max(kOneCta, 1024 + (2 + kSlots) * planes * held * BK * 2);
  if (cudaMemsetAsync(counters, 0, sizeof(int) * plan.ints, stream) != cudaSuccess) return FTB_ERR_LAUNCH;
#define FTB_GRID_LAUNCH(TT)                                                                              \
  switch (plan.nb) {                                                                                     \
    case 16: return pair ? launch<TT, 16, true>(m, g, smem, stream) : launch<TT, 16, false>(m, g, smem, stream); \
    case 32: return pair ? launch<TT, 32, true>(m, g, smem, stream) : launch<TT, 32, false>(m, g, smem, stream); \
    default: return pair ? launch<TT, 64, true>(m, g, smem, stream) : launch<TT, 64, false>(m, g, smem, stream); \
  }
  if (dtype == FTB_F16) {
    FTB_GRID_LAUNCH(__half)
  }
  FTB_GRID_LAUNCH(__nv_bfloat16)
#undef FTB_GRID_LAUNCH
}

}  // namespace ftb
