// Device side of the stacked LSTM whose hidden states carry their own arrival: csrc/lstm_flow.cu says how it
// works.  Also a layer of dilation 1 or 2 of the dilated LSTM (csrc/rnn_cluster.cu).
#pragma once

#include "ptx.cuh"
#include "tmap.h"

namespace ftb {

namespace flow {

constexpr int kGateRows = 128;  // packed gate rows of a CTA
constexpr int kUnits = kGateRows / 4;
constexpr int BK = 64;
constexpr uint32_t kWBlockBytes = kGateRows * BK * 2;
constexpr int kFirstEpi = 4;
constexpr int kMaxSlots = 2;     // input tiles [NB x I] in shared memory
constexpr int kMaxRing = 4;      // input weight blocks on their way through shared memory
constexpr int kMaxPause = 4000;  // cycles
constexpr uint32_t kMaxSmem = 226 * 1024;

template <int NB, bool kPair = false>
struct FlowCfg {
  static constexpr int kCtas = kPair ? 2 : 1;              // that share one MMA
  static constexpr int kHeld = NB / kCtas;                 // rows of a state that a CTA holds
  static constexpr int kWarps = NB == 16 ? 4 : (NB == 32 ? 8 : (NB == 48 ? 12 : 16));  // epilogue warps
  static constexpr int kChunks = NB * 4 / kWarps / 16;         // of 16 columns, of a warp
  static constexpr int kRows = kHeld / kWarps;             // state rows a warp reads
  static constexpr int kSpan = kRows < 4 ? kRows : 4;      // of them at a time,
  static constexpr int kParts = 4 / kSpan;                 // each by so many groups of eight lanes
  static constexpr int kThreads = 32 * (kFirstEpi + kWarps);
  static constexpr uint32_t kBlockBytes = kHeld * BK * 2;  // one K block of a state
  static constexpr int kCopyKb = 128 / NB;                 // K blocks of one TMA copy (16 KB, a pair's CTAs 8 KB each)
  static constexpr int kTmemBlocks = (512 - 2 * NB) / 32;  // weight blocks beside the two accumulators
};

struct FlowArgs {
  int D, L, N, I, H, G, S;
  int n_tiles;          // 4H / 128
  int n_slots;          // input tiles
  int held, ring;       // kStream: weight blocks kept in shared memory, blocks of the ring for the others
  int64_t T;            // rows of a layer's output: off[L], or L * N
  const int* off;       // [L + 1] first row of every step (ragged batch), or nullptr: t * N
  const float* bias_p;  // [D, 4H] packed order, or nullptr
  const void* Wp;       // [D, 4H, I+H]
  void* hs;             // [D, T, H], all 0xFFFF before the launch
  float* c_out;         // [D, c_rows, H], the first N of c_rows
  int c_rows;
  int* flags;           // [D][flag_steps][S] tiles of the slice's cell (l, t) that can be read through TMA
  // A layer of the dilated LSTM whose step is `fold` time steps of N1 sequences (N = fold * N1, the last step may be short).
  // fold 0: a step is a time step in every layer.
  int fold, N1;
  int flag_steps;       // cells of a layer in `flags`
  // mapX and mapH are of steps of N rows, so that a slice that is not full reads no rows past the step's; else (a ragged batch, the
  // dilated LSTM) of all rows as one step.  Rows past the step's belong to the next step, which the layer below is storing and
  // polling meanwhile, and what follows closely behind it held it up: D8 L100 H512, 40 sequences on slices of 64, pairs 403 -> 336
  // us, 56 401 -> 358, 64 369 / 370; D18 L151 N33 1269 -> 959.  (A ragged batch by boxes of 8 and 16 rows: 380 -> 477.)
  bool by_step;
  int* status;
};

struct Rows {  // rows of a step: the first one and how many sequences still run
  int64_t first;
  int active;
};
__device__ __forceinline__ Rows rows_of(const FlowArgs& a, int t) {
  if (a.off == nullptr) {
    const int64_t first = static_cast<int64_t>(t) * a.N;
    return {first, t < a.L ? static_cast<int>(min(static_cast<int64_t>(a.N), a.T - first)) : 0};
  }
  if (t >= a.L) return {0, 0};
  const int r0 = __ldg(a.off + t);
  return {r0, __ldg(a.off + t + 1) - r0};
}

__device__ __forceinline__ void st_relaxed_gpu64(void* p, uint32_t lo, uint32_t hi) {
  const uint64_t v = static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void ld_relaxed_gpu_2x64(const void* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
// A word of four hidden states has arrived when its last one is not the fill pattern.
__device__ __forceinline__ bool arrived(uint64_t w) { return (w >> 48) != 0xFFFFu; }

// Whole-warp bounded wait for the counters of a step: how many of the next `n` steps (at most 4) can be read, 0 when the wait
// ran out.  counter(s, f): the f-th counter of step s from now, or nullptr.  Looking at four steps costs no more than at one, and
// a producer that is behind does without the look, and the proxy fence, of the steps that were ready with it: 900 and 1000 cycles.
template <typename F>
__device__ __forceinline__ int wait_steps(int n, int target, F counter, int lane, volatile int* s_abort, int* g_status) {
  const int step = lane >> 3;
  uint64_t t0 = 0;
  for (uint32_t it = 1;; ++it) {
    bool ready = step < n;
    if (ready) {
      const int* p;
      for (int f = lane & 7; (p = counter(step, f)) != nullptr; f += 8) ready = ready && ld_acquire_gpu(p) >= target;
    }
    const uint32_t all = __ballot_sync(0xffffffffu, ready);
    if ((all & 0xffu) == 0xffu) {
      __syncwarp();
      return all == ~0u ? 4 : (all & 0xffffffu) == 0xffffffu ? 3 : (all & 0xffffu) == 0xffffu ? 2 : 1;
    }
    if ((it & 0x3F) == 0) {
      if (t0 == 0) t0 = globaltimer_ns();
      if (__any_sync(0xffffffffu, *s_abort != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS)) {
        if (lane == 0 && *s_abort == 0) {
          *s_abort = 1;
          atomicCAS(g_status, 0, FTB_ERR_TIMEOUT_DEP);
        }
        return 0;
      }
    }
  }
}

// One CTA: packed gate rows `tile` of batch slice `slice`, layers j, j + G, ..  kPair: two CTAs of a cluster, tiles 2 i
// and 2 i + 1, share each MMA; each holds the state rows of its half of the slice.  kStream: the last input weight blocks,
// which do not fit, pass through a ring every step.  The layer below is cut into slices of nb_below sequences, of fold_below time
// steps.
template <typename T, int NB, bool kPair = false, bool kStream = false>
__device__ __forceinline__ void body(const CUtensorMap& mapX, const CUtensorMap& mapH, const CUtensorMap& mapW,
                                     const FlowArgs& a, const int tile, const int slice, const int j, const int nb_below,
                                     const int fold_below = 1) {
  using C = FlowCfg<NB, kPair>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t in_full[kMaxSlots], in_empty[kMaxSlots];
  __shared__ uint64_t st_full;          // the previous step's state is in its operand tile
  __shared__ uint64_t acc_full[2], acc_empty[2];
  __shared__ uint64_t w_tmem, w_smem;   // the sweep's weights are in place
  __shared__ uint64_t ring_full[kStream ? kMaxRing : 1], ring_empty[kStream ? kMaxRing : 1];
  __shared__ uint64_t swept;            // every MMA of the sweep is done
  __shared__ uint32_t tmem_base_s;
  __shared__ int n_stored;              // epilogue warps that have stored a step, summed over steps
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* status = a.status;
  const int kb_h = a.H / BK;
  // Weight blocks in the order tensor memory is filled: recurrent, then input; the rest in shared memory.
  const int rec_t = min(C::kTmemBlocks, kb_h);
  // (an input tile is a whole number of copies)
  const uint32_t slot_bytes = ((max(a.I, a.H) / BK + C::kCopyKb - 1) / C::kCopyKb) * C::kCopyKb * C::kBlockBytes;
  uint8_t* s_state = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* s_in = s_state + kb_h * C::kBlockBytes;
  uint8_t* s_w = s_in + a.n_slots * slot_bytes;
  // Input weight blocks in shared memory, of the kb_x - in_t that tensor memory does not hold.
  auto kept_in = [&](int n) { return kStream ? min(n, a.held - (kb_h - rec_t)) : n; };

  if (threadIdx.x == 0) {
    prefetch_tmap(&mapX);
    prefetch_tmap(&mapH);
    prefetch_tmap(&mapW);
    for (int i = 0; i < kMaxSlots; ++i) {
      mbar_init(&in_full[i], 1);
      mbar_init(&in_empty[i], 1);
    }
    mbar_init(&st_full, C::kCtas * C::kWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], C::kCtas * C::kWarps);
    }
    if constexpr (kStream)
      for (int i = 0; i < kMaxRing; ++i) {
        mbar_init(&ring_full[i], 1);
        mbar_init(&ring_empty[i], 1);
      }
    n_stored = 0;
    mbar_init(&w_tmem, C::kCtas * C::kWarps);
    mbar_init(&w_smem, 1);
    mbar_init(&swept, 1);
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

  const int n_base = slice * NB;
  // Which CTA of the pair this is.  The even one issues the MMAs, and what they wait for is counted on its barriers.
  const int rank = kPair ? static_cast<int>(cluster_ctarank()) : 0;
  const int held_base = n_base + rank * C::kHeld;
  auto commit = [](uint64_t* bar) {
    if constexpr (kPair) umma_commit_pair(bar); else umma_commit(bar);
  };
  auto arrive_at_issuer = [](uint64_t* bar) {
    if constexpr (kPair) mbar_arrive_peer(map_to_cta(smem_u32(bar), 0)); else mbar_arrive(bar);
  };
  const int n_groups = (a.D + a.G - 1) / a.G;
  // Steps this slice takes part in (ragged: until its longest sequence, its first one, ends).
  int steps = a.L;
  if (a.fold > 0 && rows_of(a, a.L - 1).active <= n_base) --steps;
  if (a.off != nullptr) {
    steps = 0;
    for (int hi = a.L; steps < hi;) {
      const int mid = (steps + hi) >> 1;
      if (rows_of(a, mid).active > n_base) steps = mid + 1; else hi = mid;
    }
  }

  if (warp == 0 && rank == 0) {
    // -------------------------------------------------------------- MMA issuer
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_f16(C::kCtas * kGateRows, NB, Fmt<T>::kind, 0, 0);
    auto mma_ts = [](uint32_t d, uint32_t aw, uint64_t bd, uint32_t id, uint32_t accumulate) {
      if constexpr (kPair) umma_ts_pair(d, aw, bd, id, accumulate); else umma_ts(d, aw, bd, id, accumulate);
    };
    auto mma_ss = [](uint32_t d, uint64_t ad, uint64_t bd, uint32_t id, uint32_t accumulate) {
      if constexpr (kPair) umma_ss_pair(d, ad, bd, id, accumulate); else umma_ss(d, ad, bd, id, accumulate);
    };
    const uint64_t in_desc = make_sdesc_sw128(smem_u32(s_in), 16, 1024);
    const uint64_t state_desc = make_sdesc_sw128(smem_u32(s_state), 16, 1024);
    const uint64_t w_desc = make_sdesc_sw128(smem_u32(s_w), 16, 1024);
    constexpr uint32_t kBlockDesc = C::kBlockBytes >> 4;
    // K blocks of a half: weights in tensor memory from column `aw` or in shared memory from `ad`, the
    // other operand from `bd`.  (A wait or a loop turn between K blocks costs more than the four MMAs of
    // one: 250 cycles a block with a barrier each, 113 as a plain loop, 55 unrolled.)
    auto blocks_ts = [&](uint32_t d_tmem, uint32_t aw, uint64_t bd, int n, uint32_t accumulate) {
      for (; n >= 4; n -= 4, aw += 4 * 32, bd += 4 * kBlockDesc, accumulate = 1) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            mma_ts(d_tmem, aw + 8 * i, bd + (i >> 2) * kBlockDesc + 2 * (i & 3), idesc, i > 0 ? 1u : accumulate);
        }
      }
      if (n & 2) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            mma_ts(d_tmem, aw + 8 * i, bd + (i >> 2) * kBlockDesc + 2 * (i & 3), idesc, i > 0 ? 1u : accumulate);
        }
        aw += 2 * 32;
        bd += 2 * kBlockDesc;
        accumulate = 1;
      }
      if (n & 1) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 4; ++i) mma_ts(d_tmem, aw + 8 * i, bd + 2 * i, idesc, i > 0 ? 1u : accumulate);
        }
      }
    };
    auto blocks_ss = [&](uint32_t d_tmem, uint64_t ad, uint64_t bd, int n, uint32_t accumulate) {
      for (; n > 0; --n, ad += kWBlockBytes >> 4, bd += kBlockDesc, accumulate = 1) {
        if (leader) {
#pragma unroll
          for (int i = 0; i < 4; ++i) mma_ss(d_tmem, ad + 2 * i, bd + 2 * i, idesc, i > 0 ? 1u : accumulate);
        }
      }
    };
    int slot = 0, sweep = 0, k = 0, states = 0;  // k: steps started, states: states received
    int rs = 0;
    uint32_t phase = 0, ring_phase = 0;
    bool ok = true;
    for (int g = 0; g < n_groups && ok; ++g) {
      const int l = g * a.G + j;
      if (l >= a.D) continue;
      const int kb_x = l == 0 ? a.I / BK : kb_h;
      const int in_t = min(C::kTmemBlocks - rec_t, kb_x), in_s = kept_in(kb_x - in_t);
      ok = mbar_wait_warp(&w_tmem, sweep & 1, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
      if (ok && (in_s > 0 || rec_t < kb_h))
        ok = mbar_wait_warp(&w_smem, sweep & 1, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
      if (!ok) break;
      tc_fence_after();
      const bool late = leader && a.n_slots == 1, early = leader && a.n_slots > 1;
      for (int t = 0; t < steps; ++t, ++k) {
        const int acc = k & 1;
        const uint32_t d_tmem = tmem_base + acc * NB;
        ok = mbar_wait_warp(&acc_empty[acc], ((k >> 1) & 1) ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_EPI) &&
             mbar_wait_warp(&in_full[slot], phase, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
        if (!ok) break;
        tc_fence_after();
        const uint64_t xd = in_desc + static_cast<uint64_t>((slot * slot_bytes) >> 4);
        blocks_ts(d_tmem, tmem_w + rec_t * 32, xd, in_t, 0u);
        blocks_ss(d_tmem, w_desc + static_cast<uint64_t>(((kb_h - rec_t) * kWBlockBytes) >> 4), xd + in_t * kBlockDesc,
                  in_s, in_t > 0 ? 1u : 0u);
        if constexpr (kStream) {
          const uint64_t ring_desc = w_desc + static_cast<uint64_t>((a.held * kWBlockBytes) >> 4);
          for (int b = in_t + in_s; b < kb_x; ++b) {
            ok = mbar_wait_warp(&ring_full[rs], ring_phase, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
            if (!ok) break;
            tc_fence_after();
            blocks_ss(d_tmem, ring_desc + static_cast<uint64_t>((rs * kWBlockBytes) >> 4), xd + b * kBlockDesc, 1, b > 0 ? 1u : 0u);
            if (leader) commit(&ring_empty[rs]);
            if (++rs == a.ring) {
              rs = 0;
              ring_phase ^= 1u;
            }
          }
          if (!ok) break;
        }
        // Where there is one input tile it goes back behind the recurrent half, not before it: its next copy would otherwise
        // be under way while the warps read the state, through the same L2 and into the same SM (64 KB each at H 512, 64
        // sequences and single CTAs: D8 L100 500 us a call, behind it 460).  With two, the copy made room for is the one after the next: before
        // the half it is 1 % faster at H 256, and so is this order of slot and commits (D1 L100 N16 H256 156 us, with the
        // slot's step behind the half 158.5; inside a branch on the number of slots 8 % behind).
        if (early) commit(&in_empty[slot]);
        if (++slot == a.n_slots) {
          slot = 0;
          phase ^= 1u;
        }
        if (t > 0) {
          // (the other CTA's rows are ordered by an acquire of the cluster's scope, as their release is)
          if constexpr (kPair)
            ok = __all_sync(0xffffffffu, mbar_wait_cluster(&st_full, states & 1, &s_abort, status, FTB_ERR_TIMEOUT_DEP));
          else
            ok = mbar_wait_warp(&st_full, states & 1, &s_abort, status, FTB_ERR_TIMEOUT_DEP);
          if (!ok) break;
          blocks_ts(d_tmem, tmem_w, state_desc, rec_t, 1u);
          blocks_ss(d_tmem, w_desc, state_desc + rec_t * kBlockDesc, kb_h - rec_t, 1u);
          ++states;
        }
        if (leader) commit(&acc_full[acc]);
        if (late) commit(&in_empty[0]);
      }
      if (ok && leader) commit(&swept);
      ++sweep;
    }
  } else if (warp == 1) {
    // ----------------------------------- TMA: shared-memory weights, input tiles
    int slot = 0, sweep = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int g = 0; g < n_groups && ok; ++g) {
      const int l = g * a.G + j;
      if (l >= a.D) continue;
      const int kb_x = l == 0 ? a.I / BK : kb_h;
      const int in_t = min(C::kTmemBlocks - rec_t, kb_x);
      const int n_rec = kb_h - rec_t, n_in = kept_in(kb_x - in_t);
      if (n_rec + n_in > 0) {
        if (sweep > 0) ok = mbar_wait_warp(&swept, (sweep - 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
        if (ok && lane == 0) {
          if (rank == 0) mbar_arrive_expect_tx(&w_smem, C::kCtas * (n_rec + n_in) * kWBlockBytes);
          for (int b = 0; b < n_rec + n_in; ++b) {
            const int x = b < n_rec ? a.I + (rec_t + b) * BK : (in_t + b - n_rec) * BK, w = (l * 4 * a.H + tile * kGateRows) / 32;
            if constexpr (kPair)
              tma_load_4d_pair(s_w + b * kWBlockBytes, &mapW, map_to_cta(smem_u32(&w_smem), 0), x, 0, 0, w);
            else
              tma_load_4d(s_w + b * kWBlockBytes, &mapW, &w_smem, x, 0, 0, w);
          }
        }
      }
      if (sweep == 0) grid_dependency_wait();  // weights need not wait for the fill of the output array and the counters
      ++sweep;
      const int copies = (kb_x + C::kCopyKb - 1) / C::kCopyKb;
      int ready = 0;  // steps of the layer below that can be read
      for (int t = 0; t < steps && ok; ++t) {
        // (the maps' steps: the call's, or all rows as one)
        const int below = l == 0 ? 0 : l - 1;
        const int step = a.by_step ? below * a.L + t : 0;
        const int row = a.by_step ? held_base : static_cast<int>(below * a.T + rows_of(a, t).first + held_base);
        if (l > 0 && t >= ready) {
          // the layer below may be cut differently: its slices that hold this one's rows
          const int* flags = a.flags + static_cast<int64_t>(l - 1) * a.flag_steps * a.S;
          auto counter = [&](int ahead, int f) -> const int* {
            if (a.fold == 0) {
              const int i = n_base / nb_below + f;
              return i > (min(n_base + NB, a.N) - 1) / nb_below ? nullptr : flags + static_cast<int64_t>(t + ahead) * a.S + i;
            }
            const Rows rows = rows_of(a, t + ahead);
            const int64_t per = static_cast<int64_t>(fold_below) * a.N1, end = rows.first + min(n_base + NB, rows.active);
            for (int64_t r = rows.first + n_base; r < end; --f) {
              const int64_t step = r / per;
              const int i = static_cast<int>(r - step * per) / nb_below;
              if (f == 0) return flags + step * a.S + i;
              r = step * per + min((i + 1) * static_cast<int64_t>(nb_below), per);
            }
            return nullptr;
          };
          const int n = wait_steps(min(4, steps - t), a.n_tiles, counter, lane, &s_abort, status);
          ok = n > 0;
          if (!ok) break;
          ready = t + n;
          fence_proxy_async_global();  // threads of other CTAs stored what TMA reads
        }
        ok = mbar_wait_warp(&in_empty[slot], phase ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_SLOT);
        if (!ok) break;
        if (lane == 0) {
          // (K blocks past the last one arrive as zeros and are not multiplied)
          if (rank == 0) mbar_arrive_expect_tx(&in_full[slot], C::kCtas * copies * C::kCopyKb * C::kBlockBytes);
          for (int c = 0; c < copies; ++c) {
            uint8_t* dst = s_in + slot * slot_bytes + c * C::kCopyKb * C::kBlockBytes;
            const CUtensorMap* map = l == 0 ? &mapX : &mapH;
            if constexpr (kPair)
              tma_load_4d_pair(dst, map, map_to_cta(smem_u32(&in_full[slot]), 0), 0, row, c * C::kCopyKb, step);
            else
              tma_load_4d(dst, map, &in_full[slot], 0, row, c * C::kCopyKb, step);
          }
        }
        if (++slot == a.n_slots) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
    // (the input tiles first: with the last sweep's back, `swept` is at most that sweep behind)
    if constexpr (kPair)
      if (ok && ring_drain(in_empty, a.n_slots, slot, phase, &s_abort, status))
        mbar_wait(&swept, (sweep - 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
  } else if (warp == 2) {
    // ----------------------------------- publisher: cell (l, t) can be read through TMA
    volatile int* abort_flag = &s_abort;
    volatile int* stored = &n_stored;
    int want = 0;
    grid_dependency_wait();
    for (int g = 0; g < n_groups && lane == 0; ++g) {
      const int l = g * a.G + j;
      if (l >= a.D) continue;
      for (int t = 0; t < steps; ++t) {
        // (A running count, not a barrier: nothing waits for this warp, which may fall several steps
        // behind, and a parity wait must not.)
        want += C::kWarps;
        if (l + 1 == a.D) continue;
        uint64_t t0 = 0;
        bool ok = true;
        for (uint32_t it = 1; *stored < want; ++it) {
          if ((it & 0x3F) != 0) continue;
          if (t0 == 0) t0 = globaltimer_ns();
          if (*abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS) {
            ok = false;
            break;
          }
        }
        if (!ok) {
          if (*abort_flag == 0) {
            *abort_flag = 1;
            atomicCAS(status, 0, FTB_ERR_TIMEOUT_EPI);
          }
          g = n_groups;
          break;
        }
        __threadfence_block();
        // (The release takes the other warps' stores along; the proxy fence is the reader's, between its acquire and its copy.)
        red_release_gpu_add(a.flags + (static_cast<int64_t>(l) * a.flag_steps + t) * a.S + slice, 1);
      }
    }
  } else if (kStream && warp == 3) {
    // ----------------------------------- TMA: the input weights that are not kept, every step again
    int rs = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int g = 0; g < n_groups && ok; ++g) {
      const int l = g * a.G + j;
      if (l >= a.D) continue;
      const int kb_x = l == 0 ? a.I / BK : kb_h;
      const int in_t = min(C::kTmemBlocks - rec_t, kb_x), first = in_t + kept_in(kb_x - in_t);
      for (int t = 0; t < steps && ok; ++t)
        for (int b = first; b < kb_x; ++b) {
          ok = mbar_wait_warp(&ring_empty[rs], phase ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_SLOT);
          if (!ok) break;
          if (lane == 0) {
            if (rank == 0) mbar_arrive_expect_tx(&ring_full[rs], C::kCtas * kWBlockBytes);
            uint8_t* dst = s_w + (a.held + rs) * kWBlockBytes;
            const int w = (l * 4 * a.H + tile * kGateRows) / 32;
            if constexpr (kPair)
              tma_load_4d_pair(dst, &mapW, map_to_cta(smem_u32(&ring_full[rs]), 0), b * BK, 0, 0, w);
            else
              tma_load_4d(dst, &mapW, &ring_full[rs], b * BK, 0, 0, w);
          }
          if (++rs == a.ring) {
            rs = 0;
            phase ^= 1u;
          }
        }
    }
    if (kPair && ok) ring_drain(ring_empty, a.ring, rs, phase, &s_abort, status);
  } else if (warp >= kFirstEpi && warp < kFirstEpi + C::kWarps) {
    // ------------------------------------------------------- epilogue and state
    const int q = warp & 3, w = warp - kFirstEpi, sub = w >> 2;
    // The gates of a unit sit in tensor memory 8 lanes apart (8 units of gate i, 8 of f, of o, of c in each quadrant), so that
    // fragments of 16 lanes leave a thread with all gates of unit lane / 4 and no exchange between threads is needed (against a
    // 4 x 4 transpose over four lanes for every four columns).
    const int u_quad = q * 8 + (lane >> 2), unit = tile * kUnits + u_quad;
    const bool ub0 = (lane & 4) != 0, ub1 = (lane & 8) != 0;
    // This lane has sequences n_own, n_own + 1, n_own + 8, n_own + 9 of each chunk of 16; after the exchange below it stores four
    // units of n_store.
    const int n_own = sub * C::kChunks * 16 + 2 * (lane & 3);
    const int n_store = n_own + (ub0 ? 8 : 0) + (ub1 ? 1 : 0);
    // What this lane reads of a state: chunk `lane & 7` of K blocks `part`, part + kParts, .. of rows n_load, n_load + 4, ..
    // (counted in the rows that this CTA holds)
    const int n_load = w * C::kRows + (C::kParts == 1 ? lane >> 3 : (lane >> 3) % C::kSpan);
    const int part = C::kParts == 1 ? 0 : (lane >> 3) / C::kSpan;
    volatile int* abort_flag = &s_abort;
    int k = 0, sweep = 0, pause = 300;
    bool ok = true;
    for (int g = 0; g < n_groups && ok; ++g) {
      const int l = g * a.G + j;
      if (l >= a.D) continue;
      if (sweep > 0) ok = mbar_wait_warp(&swept, (sweep - 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
      if (!ok) break;
      ++sweep;
      {
        // Weights -> tensor memory: a thread copies one packed row to its lane, two 16-bit values per 32-bit column
        // (the layout of an A operand there); the warps of a quadrant take K blocks in turn.
        const int kb_x = l == 0 ? a.I / BK : kb_h;
        const int in_t = min(C::kTmemBlocks - rec_t, kb_x);
        const T* wrow = reinterpret_cast<const T*>(a.Wp) +
                        (static_cast<size_t>(l) * 4 * a.H + tile * kGateRows + q * 32 + 4 * (lane & 7) + (lane >> 3)) * (a.I + a.H);
        for (int b = sub; b < rec_t + in_t; b += C::kWarps / 4) {
          const uint4* src = reinterpret_cast<const uint4*>(wrow + (b < rec_t ? a.I + b * BK : (b - rec_t) * BK));
          uint32_t v[32];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 x4 = __ldg(src + i);
            v[4 * i + 0] = x4.x; v[4 * i + 1] = x4.y; v[4 * i + 2] = x4.z; v[4 * i + 3] = x4.w;
          }
          tmem_st32(tmem_w + (static_cast<uint32_t>(q * 32) << 16) + b * 32, v);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at_issuer(&w_tmem);
      }
      if (sweep == 1) grid_dependency_wait();
      float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.bias_p != nullptr)
        bias = __ldg(reinterpret_cast<const float4*>(a.bias_p + static_cast<size_t>(l) * 4 * a.H + tile * kGateRows) + u_quad);
      T* hs_l = reinterpret_cast<T*>(a.hs) + static_cast<size_t>(l) * a.T * a.H;
      float creg[C::kChunks][4];
#pragma unroll
      for (int ch = 0; ch < C::kChunks; ++ch)
#pragma unroll
        for (int i = 0; i < 4; ++i) creg[ch][i] = 0.f;
      Rows now = rows_of(a, 0);
      for (int t = 0; t < steps; ++t, ++k) {
        const int acc = k & 1;
        const Rows next = rows_of(a, t + 1);
        ok = mbar_wait_warp(&acc_full[acc], (k >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after();
        uint32_t r_if[C::kChunks][8], r_oc[C::kChunks][8];
#pragma unroll
        for (int ch = 0; ch < C::kChunks; ++ch) {
          const uint32_t at = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * NB + (sub * C::kChunks + ch) * 16;
          tmem_ld_frag16(at, r_if[ch]);
          tmem_ld_frag16(at + (16u << 16), r_oc[ch]);
        }
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at_issuer(&acc_empty[acc]);
#pragma unroll
        for (int ch = 0; ch < C::kChunks; ++ch) {
          float h[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int at = 4 * (i >> 1) + (i & 1);
            const float gi = __uint_as_float(r_if[ch][at]) + bias.x;
            const float gf = __uint_as_float(r_if[ch][at + 2]) + bias.y;
            const float go = __uint_as_float(r_oc[ch][at]) + bias.z;
            const float gc = __uint_as_float(r_oc[ch][at + 2]) + bias.w;
            const float c_new = sigmoid_fast(gf) * creg[ch][i] + sigmoid_fast(gi) * tanh_fast(gc);
            creg[ch][i] = c_new;
            h[i] = sigmoid_fast(go) * tanh_fast(c_new);
          }
          // (unit, 4 sequences) -> (4 units, 1 sequence): trade halves with the units next to this one, twice
          const uint32_t p01 = Fmt<T>::pack2(h[0], h[1]), p23 = Fmt<T>::pack2(h[2], h[3]);
          uint32_t other = __shfl_xor_sync(0xffffffffu, ub0 ? p01 : p23, 4);
          const uint32_t lo = ub0 ? other : p01, hi = ub0 ? p23 : other;  // units u & ~1 and u | 1
          const uint32_t w0 = __byte_perm(lo, hi, 0x5410), w1 = __byte_perm(lo, hi, 0x7632);
          other = __shfl_xor_sync(0xffffffffu, ub1 ? w0 : w1, 8);
          const int n = n_base + n_store + ch * 16;
          if (n < now.active)
            st_relaxed_gpu64(hs_l + (now.first + n) * a.H + (unit & ~3), ub1 ? other : w0, ub1 ? w1 : other);
        }
        {
          const long long c0 = clock64();
          while (clock64() - c0 < pause) {}
        }
        int rounds = 0;
        // The state of this step, for the next: eight K blocks of four rows in flight at a time.
        const bool more = t + 1 < steps;
#pragma unroll
        for (int rh = 0; rh < C::kRows; rh += C::kSpan) {
          const int n = n_load + rh;
          const bool mine = held_base + n < next.active;
          const T* src = hs_l + (now.first + held_base + n) * a.H + (lane & 7) * 8;
          uint8_t* dst = s_state + n * 128 + (((lane & 7) ^ (n & 7)) << 4);
          for (int kb0 = part; kb0 - part < kb_h && more && ok; kb0 += 8 * C::kParts) {
            uint64_t x[8], y[8];
            uint32_t missing = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              x[i] = y[i] = 0;
              if (mine && kb0 + i * C::kParts < kb_h) missing |= 1u << i;
            }
            uint64_t t0 = 0;
            for (uint32_t it = 1;; ++it) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (missing & (1u << i)) ld_relaxed_gpu_2x64(src + (kb0 + i * C::kParts) * BK, x[i], y[i]);
              if (it == 1 && rh == 0 && kb0 == part) {
                // this warp's part of the step is on its way: count it in for the publisher
                __syncwarp();
                if (lane == 0) {
                  __threadfence_block();
                  atomicAdd(&n_stored, 1);
                }
              }
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (arrived(x[i]) && arrived(y[i])) missing &= ~(1u << i);
              ++rounds;
              if (__all_sync(0xffffffffu, missing == 0)) break;
              if ((it & 0x3F) == 0) {
                if (t0 == 0) t0 = globaltimer_ns();
                if (__any_sync(0xffffffffu, *abort_flag != 0 || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS)) {
                  ok = false;
                  break;
                }
              }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (kb0 + i * C::kParts < kb_h)
                *reinterpret_cast<ulonglong2*>(dst + (kb0 + i * C::kParts) * C::kBlockBytes) = make_ulonglong2(x[i], y[i]);
          }
        }
        if (more) {
          // Everything in the first round: try a little earlier next time; else later.  (Down more slowly on wide slices of pairs,
          // whose repeats load L2 most: D8 L100 N64 H512 384 -> 378 us, D15 L87 N66 H448 861 -> 847; D1 L100 N16 H256, narrow,
          // 164 -> 165.)
          const bool early = rounds > (C::kRows / C::kSpan) * ((kb_h + 8 * C::kParts - 1) / (8 * C::kParts));
          pause = early ? min(pause + 100, kMaxPause) : pause - (pause >> (kPair && NB >= 64 ? 6 : 5));
          if (!ok) {
            if (lane == 0 && *abort_flag == 0) {
              *abort_flag = 1;
              atomicCAS(status, 0, FTB_ERR_TIMEOUT_DEP);
            }
            break;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if constexpr (kPair) mbar_arrive_peer_smem(map_to_cta(smem_u32(&st_full), 0)); else mbar_arrive(&st_full);
          }
        } else {
          __syncwarp();
          if (lane == 0) {
            __threadfence_block();
            atomicAdd(&n_stored, 1);
          }
        }
        if (next.active < now.active) {
          // sequences that end here: their final cell state
#pragma unroll
          for (int ch = 0; ch < C::kChunks; ++ch)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int n = n_base + n_own + ch * 16 + 8 * (i >> 1) + (i & 1);
              if (n < now.active && n >= next.active)
                a.c_out[(static_cast<size_t>(l) * a.c_rows + n) * a.H + unit] = creg[ch][i];
            }
        }
        now = next;
      }
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

}  // namespace flow

}  // namespace ftb
