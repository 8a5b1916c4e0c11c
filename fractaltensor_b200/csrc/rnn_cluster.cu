// A latency-bound recurrence with small hidden size (H <= 256): the dilated stacked LSTM.  (The grid RNN: csrc/grid_flow.cu.)
//
// The program is chains of small cells: 512 dependent steps of [256 x 512].[512 x 1024] in the first layer.  Run as a generic
// wavefront, every dependent level costs a trip through global memory (store, fence, flag, poll, TMA load: 6-9 us) plus a
// re-read of the layer's weights from L2.  Two kernels keep the weights on chip.  rnn_dilated_flow_kernel, the choice nearly
// wherever it fits, has no clusters: layers of dilation 1 and 2 run flow::body (lstm_flow.cuh), whose states are their own flags,
// the others cluster_body with one CTA in place of each of a cluster's.  rnn_cluster_dilated_kernel, for short sequences of a few
// narrow states and for what the other one has too few SMs for, runs cluster_body for all layers, a thread-block cluster per chain of
// dependent steps.  There
//   * the weights never move: a cluster of CL CTAs owns one chain (one layer and batch slice), CTA r of the
//     cluster owns 128 packed weight rows (32 LSTM units x 4 gates) for the whole launch, and that slice of the
//     weights sits in tensor memory as the A operand of every MMA ("recurrent weights resident on chip");
//   * the batch is the N side of the MMA (NB = 128 or 64 columns per slice);
//   * the state a chain hands to its own next step, h(t) of a layer with dilation 1, never leaves the
//     cluster: it goes into the next step's B operand in every CTA of the cluster (distributed shared memory),
//     bytes counted on the receiver's mbarrier.  Each CTA writes its units into a staging tile, a contiguous
//     block of the un-swizzled K-major layout, and copies it with one bulk copy per piece and peer: eight peers'
//     32 KB a step are bound by the bytes, and st.async of 16 at a time takes longer (3.1 us a step instead of 3.0);
//   * everything that crosses chains (the layer below, a layer's own state
//     `dilation` >= 2 steps back) goes through global memory with one release flag per
//     (cell, tile), polled by a whole warp, and TMA loads; those consumers run a few steps behind
//     their producers, so this latency adds to the pipeline's depth, not to every step.  The
//     global flag is published by a warp of its own, off the chain.
// Same arithmetic in the same order as the cell kernels of the generic wavefront (input first,
// then the recurrent state(s)): the results are bit-identical.
//
// Roles: warp 0 producer of the TMA-fed operand blocks, warp 1 MMA issuer (owns TMEM), warp 2
// output store and flag publisher, warp 3 the second producer, warps 4.. epilogue.  tcgen05 cta_group::1; no multicast loads;
// cooperative cluster launch (a chain waits for flags of other clusters).
//
// Programs: dilated_layer()/model() (examples/dilated_rnn/dilated_rnn.py:16-41) in place of
// DilatedLstmRegion1/2 (kaleido/core/device/kernels/lstm/dilated_lstm/region{1,2}.h).
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "lstm_flow.cuh"
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {

namespace {

constexpr int BK = 64;
constexpr int kFirstEpiWarp = 4;
// Epilogue warps: four per TMEM lane quadrant (five MUFU operations per element: latency-bound with fewer).
constexpr int kAllEpiWarps = 16;
constexpr int kCtaThreads = 32 * (kFirstEpiWarp + kAllEpiWarps);
constexpr int kOutUnits = 32;  // hidden units of a CTA
constexpr uint32_t kStageBytes = 16384;

constexpr int kMaxLayers = 16;

#ifdef FTB_TRACE
// Debug builds: globaltimer stamps of CTA rank 0 of every cluster, [cluster][step][16].
__device__ unsigned long long* g_cluster_trace = nullptr;
#define FTB_CL_STAMP(i, s) \
  if (g_cluster_trace != nullptr && rank == 0) g_cluster_trace[(static_cast<size_t>(cid) * n_steps + (i)) * 16 + (s)] = globaltimer_ns()
#else
#define FTB_CL_STAMP(i, s)
#endif
#ifdef FTB_ACCT
// Debug builds: cycles a role of CTA rank 0 spends in each of its waits, summed over the launch and
// written once at the end: [cluster][16].
__device__ unsigned long long* g_cluster_acct = nullptr;
#define ACCT_DECL(n) long long acct_[n] = {}; long long acct_t0_ = 0; (void)acct_t0_
#define ACCT_BEGIN() acct_t0_ = clock64()
#define ACCT_END(k) acct_[k] += clock64() - acct_t0_
#define ACCT_WRITE(k, slot) if (g_cluster_acct != nullptr && rank == 0) g_cluster_acct[static_cast<size_t>(cid) * 16 + (slot)] = acct_[k]
#else
#define ACCT_DECL(n)
#define ACCT_BEGIN()
#define ACCT_END(k)
#define ACCT_WRITE(k, slot)
#endif

struct ClusterArgs {
  int D, L, N, H;  // layers, time steps, batch, hidden size
  int S;           // counters per cell (the most slices of a layer)
  int CL;          // CTAs per cluster
  int max_dil;
  int dil[kMaxLayers];
  int nb[kMaxLayers];                 // batch columns per chain of the layer
  int fold[kMaxLayers];               // time steps of a step of a layer that runs flow::body, 0: it does not
  int first_cluster[kMaxLayers + 1];  // index of the layer's first cluster
  const void* W;      // Wp [D,4H,2H]
  const float* bias;  // bias_p [D,4H] or nullptr
  float* c;           // fp32 [D, max_dil*N, H]
  int* flags;         // [cells][S] counters of CTAs; zero before the launch
  int* status;
};

// One TMA-fed operand segment of a step: all K blocks of activation rows `row`.. of tensor map `map`; flags to wait for first.
// The first is the input half's, the second, where there is one, the recurrent half's.
struct Segment {
  int map, row;
  const int* flags;  // nullptr: an input of the call
  int nflags, target;
};
struct StepPlan {
  int nseg;
  Segment seg[2];
};

// Shared-memory operand descriptor for an un-swizzled K-major tile: core matrices of 8 rows x 16 B
// stored contiguously (128 B); `lbo` = bytes between the two 16-byte K chunks of an MMA's K = 16,
// `sbo` = bytes between consecutive 8-row groups.
__device__ __forceinline__ uint64_t make_sdesc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  return d;
}

// Bulk copy from this CTA's shared memory into a peer's; completion (bytes) counted on the peer's mbarrier.
__device__ __forceinline__ void bulk_copy_to_peer(uint32_t dst_cluster_addr, uint32_t src_addr, uint32_t bytes,
                                                  uint32_t bar_cluster_addr) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   dst_cluster_addr),
               "r"(src_addr), "r"(bytes), "r"(bar_cluster_addr)
               : "memory");
}

// Arrives, once the MMAs issued so far by this thread are done, on the mbarrier at the same
// shared-memory offset in every CTA of the cluster whose bit is set in `mask`.
__device__ __forceinline__ void umma_commit_to(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// What this CTA loads at time step `i` of its chain (layer, slice).  (The state of a layer with dilation 1 comes through shared memory.)
template <int NB>
__device__ __forceinline__ StepPlan plan_step(const ClusterArgs& a, int layer, int slice, int i) {
  StepPlan p;
  p.nseg = 0;
  const int d = a.dil[layer];
  Segment& x = p.seg[p.nseg++];
  if (layer == 0) {
    x.map = 0;
    x.row = i * a.N + slice * NB;
    x.flags = nullptr;
    x.nflags = 0;
  } else {
    x.map = 1;
    x.row = ((layer - 1) * a.L + i) * a.N + slice * NB;
    // One counter per slice of a cell.  The layer below may be cut differently: its slices that hold this
    // one's rows own consecutive counters.
    const int nbp = a.nb[layer - 1], fold = max(a.fold[layer - 1], 1), step = i / fold;
    const int row0 = (i - step * fold) * a.N;
    const int first = (row0 + slice * NB) / nbp;
    x.flags = a.flags + ((layer - 1) * a.L + step) * a.S + first;
    x.nflags = (row0 + min(slice * NB + NB, a.N) - 1) / nbp - first + 1;
    x.target = a.CL;
  }
  if (d > 1 && i >= d) {
    Segment& h = p.seg[p.nseg++];
    h.map = 1;
    h.row = (layer * a.L + i - d) * a.N + slice * NB;
    h.flags = a.flags + (layer * a.L + i - d) * a.S + slice;
    h.nflags = 1;
    h.target = a.CL;
  }
  return p;
}

// mapX, mapH: the inputs and the hidden states (boxes of NB rows x 64 columns, 128-byte swizzle).  mapO: the hidden states
// as 64-byte-swizzled boxes of NB rows x this CTA's units; mapT: the same with the row count of the last, partial batch slice.
// kSplit: the even steps are the first eight epilogue warps', the odd ones the others', so that what a step waits for (accumulator,
// cell state, output tile) is covered by the other half's work.  For even dilations: a cell state then stays one half's.
template <typename T, int NB, bool kSplit>
__device__ __forceinline__ void cluster_body(const CUtensorMap& mapX, const CUtensorMap& mapH, const CUtensorMap& mapO,
                                             const CUtensorMap& mapT, const ClusterArgs& a, const int rank, const int cid,
                                             const int layer, const int slice) {
  constexpr int kEpiWarps = kSplit ? kAllEpiWarps / 2 : kAllEpiWarps;  // of a step
  constexpr int kSub = kEpiWarps / 4;              // of them per TMEM lane quadrant
  constexpr int kBlocksPerStage = 128 / NB;        // [NB x 64] 16-bit blocks per 16 KB stage
  constexpr uint32_t kBlockBytes = NB * BK * 2;
  constexpr int kRing = 4;  // stages of the TMA-fed ring when the chain also uses the self slots
  constexpr uint32_t kOutTileBytes = static_cast<uint32_t>(NB) * kOutUnits * 2;  // row-major [NB][units] staging
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t ring_full[12], ring_empty[12];  // up to 12 ring stages
  __shared__ uint64_t self_full[2];   // the slot holds the whole previous output (bytes counted)
  __shared__ uint64_t self_free[2];   // producers only: every CTA of the cluster has multiplied the slot's contents
  __shared__ uint64_t stg_ready;      // the epilogue warps have written the step's staging tile
  __shared__ int seg_seq;             // operand segments issued into the ring so far (two producer warps)
  __shared__ int out_issued[2];       // epilogue warps that have staged an even / odd step's outputs, summed over steps
  __shared__ int out_stored;          // steps whose output staging tile the publisher has finished reading
  __shared__ uint64_t tfull_bar[2], tempty_bar[2];
  __shared__ uint64_t res_full;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  int* status = a.status;

  const int kbh = a.H / BK;
  const int n_wkb = 2 * kbh;  // K blocks of this CTA's weight tile, all in TMEM
  const int K = n_wkb * BK;
  // Does the chain hand its own output to its next step through the cluster's shared memory?
  const bool self_chain = a.dil[layer] == 1;
  const int self_first_chunk = rank * (kOutUnits / 8);  // of the self operand, 8 units each: this CTA's
  const uint16_t producer_mask = static_cast<uint16_t>((1u << a.CL) - 1u);
  const uint32_t self_slot_bytes = static_cast<uint32_t>(a.H / 8) * NB * 16;  // H units x NB rows, 16-bit
  constexpr uint32_t stage_tile_bytes = static_cast<uint32_t>(kOutUnits / 8) * NB * 16;
  // Shared memory: [self slot 0][self slot 1][staging 0][staging 1][output tile 0][output tile 1][ring ...];
  // chains without a self operand have the output tiles and a longer ring only.
  uint8_t* s_self = smem;
  uint8_t* s_stg = s_self + (self_chain ? 2 * self_slot_bytes : 0);
  uint8_t* s_out = s_stg + (self_chain ? 2 * stage_tile_bytes : 0);  // two row-major output tiles for the TMA stores
  uint8_t* s_ring = s_out + 2 * kOutTileBytes;
  const int n_ring = self_chain ? kRing : 12;
  // ring stages a segment (the H / 64 K blocks of NB rows) takes
  const int seg_stages = (a.H / BK + kBlocksPerStage - 1) / kBlocksPerStage;

  if (threadIdx.x == 0) {
    prefetch_tmap(&mapX);
    prefetch_tmap(&mapH);
    prefetch_tmap(&mapO);
    prefetch_tmap(&mapT);
    for (int i = 0; i < 12; ++i) {
      mbar_init(&ring_full[i], 1);
      mbar_init(&ring_empty[i], 1);
    }
    mbar_init(&self_full[0], 1);
    mbar_init(&self_full[1], 1);
    mbar_init(&self_free[0], a.CL);
    mbar_init(&self_free[1], a.CL);
    mbar_init(&stg_ready, kEpiWarps);
    seg_seq = 0;
    out_issued[0] = out_issued[1] = 0;
    out_stored = 0;
    mbar_init(&tfull_bar[0], 1);
    mbar_init(&tfull_bar[1], 1);
    mbar_init(&tempty_bar[0], kEpiWarps);
    mbar_init(&tempty_bar[1], kEpiWarps);
    mbar_init(&res_full, kAllEpiWarps);
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Peers copy into this CTA's shared memory and arrive on its barriers: nobody starts before all are set up.
  cluster_sync_all();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tmem_w = tmem_base + 2 * NB;  // the weight tile sits behind the two accumulators

  const CUtensorMap* maps[2] = {&mapX, &mapH};
  const int n_steps = a.L;
  const int my_flag_cell0 = layer * a.L;

  if (warp == 0 || warp == 3) {
    // ------------------------------------------ producers of the TMA-fed operand blocks
    // One three-dimensional copy per segment: the NB rows of all its K blocks land in consecutive
    // [NB x 64] tiles of the ring (a segment never wraps: the ring is a whole number of segments long)
    // and complete on the barrier of the segment's first stage; the MMA warp frees a segment through
    // the empty barrier of that same stage.
    // Two warps share the work by segment: warp 0 takes a step's first segment (the input), warp 3
    // its second (the state that arrives through global memory), so one segment's flag wait overlaps
    // the other's ring wait and copy.  Both walk every segment to keep the ring position, and the ring
    // is filled in segment order whichever warp fills it: a warp waits for `seg_seq` to reach its
    // segment's number before it touches the ring (otherwise the warp with the lighter segments could
    // lap the other one and meet a stage's barrier a whole round early, where the parity test cannot
    // tell "not yet filled" from "already drained").
    const int mine = warp == 0 ? 0 : 1;
    int stage = 0, q = 0;
    uint32_t phase = 0;
    bool ok = true;
    volatile int* seq = &seg_seq;
    int ready = 0;  // steps whose segment of this warp can be read
    ACCT_DECL(4);
    for (int i = 0; i < n_steps && ok; ++i) {
      const StepPlan p = plan_step<NB>(a, layer, slice, i);
      for (int s = 0; s < p.nseg && ok; ++s) {
        const Segment& sg = p.seg[s];
        if ((s & 1) == mine) {
          ACCT_BEGIN();
          if (sg.flags != nullptr && i >= ready) {
            // (the layer below may count steps of two time steps: then the next ones' counters lie elsewhere)
            const int* at = sg.flags;
            int count = sg.nflags;
            if (s == 1 || a.fold[layer - 1] < 2) {
              at += (lane >> 3) * a.S;
            } else if (i + (lane >> 3) < n_steps) {
              const StepPlan next = plan_step<NB>(a, layer, slice, i + (lane >> 3));
              at = next.seg[0].flags;
              count = next.seg[0].nflags;
            }
            auto counter = [&](int, int f) -> const int* { return f < count ? at + f : nullptr; };
            const int n = flow::wait_steps(min(4, n_steps - i), sg.target, counter, lane, &s_abort, status);
            if (n == 0) {
              ok = false;
              break;
            }
            ready = i + n;
            // (Producers write their outputs with TMA stores and consumers read them with TMA loads: both
            // sides are in the async proxy, so the flag's release/acquire is all the ordering there is.
            // Threads store the output of flow::body.)
            if (lane == 0 && s == 0 && layer > 0 && a.fold[layer - 1] > 0) fence_proxy_async_global();
          }
          ACCT_END(0);
          bool fine = true;
          if (lane == 0) {
            FTB_CL_STAMP(i, 7 + 2 * s);
            ACCT_BEGIN();
            if (*seq != q) {
              const uint64_t t0 = globaltimer_ns();
              uint32_t it = 0;
              while (*seq != q) {
                if (((++it) & 0xFF) == 0 && (s_abort || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS)) break;
              }
              if (*seq != q) {
                fine = false;
                if (!s_abort) {
                  s_abort = 1;
                  atomicCAS(status, 0, FTB_ERR_TIMEOUT_SLOT);
                }
              }
            }
            ACCT_END(1);
            ACCT_BEGIN();
            if (fine) fine = mbar_wait(&ring_empty[stage], phase ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_SLOT);
            ACCT_END(2);
            ACCT_BEGIN();
            if (fine) {
              mbar_arrive_expect_tx(&ring_full[stage], kbh * kBlockBytes);
              tma_load_3d(s_ring + stage * kStageBytes, maps[sg.map], &ring_full[stage], 0, sg.row, 0);
              *seq = q + 1;
            }
            ACCT_END(3);
            FTB_CL_STAMP(i, 8 + 2 * s);
          }
          ok = __all_sync(0xffffffffu, fine);
        }
        ++q;
        stage += seg_stages;
        if (stage == n_ring) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (lane == 0) {
      ACCT_WRITE(0, mine * 4 + 0);  // flags
      ACCT_WRITE(1, mine * 4 + 1);  // segment order
      ACCT_WRITE(2, mine * 4 + 2);  // ring slots
      ACCT_WRITE(3, mine * 4 + 3);  // issue
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    // (all lanes walk the loop, one issues: mbar_wait_warp in ptx.cuh says why)
    {
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc_f16(128, NB, Fmt<T>::kind, 0, 0);
      const uint64_t ring_desc0 = make_sdesc_sw128(smem_u32(s_ring), 16, 1024);
      // (K chunks of 16 bytes NB * 16 bytes apart; groups of 8 sequences 128)
      const uint64_t self_desc0 = make_sdesc_plain(smem_u32(s_self), NB * 16, 128);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = mbar_wait_warp(&res_full, 0, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
      tc_fence_after();
      ACCT_DECL(6);
#ifdef FTB_ACCT
      const long long acct_loop0 = clock64();
#endif
      // What this thread needs of a step's plan, without the addresses the other roles compute (it is
      // the one thread every MMA of the CTA goes through: its own instructions are the step's floor).
      const int kbh = a.H / BK;
      const int d_layer = a.dil[layer];
      for (int i = 0; i < n_steps && ok; ++i) {
        const int nseg = (d_layer > 1 && i >= d_layer) ? 2 : 1;
        const bool self = d_layer == 1 && i >= 1;
        const int acc = i & 1;
        ACCT_BEGIN();
        ok = mbar_wait_warp(&tempty_bar[acc], ((i >> 1) & 1) ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
        ACCT_END(0);
        if (!ok) break;
        tc_fence_after();
        FTB_CL_STAMP(i, 0);
        const uint32_t d_tmem = tmem_base + acc * NB;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (s >= nseg) break;
          ACCT_BEGIN();
          ok = mbar_wait_warp(&ring_full[stage], phase, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
          ACCT_END(1);
          if (!ok) break;
          FTB_CL_STAMP(i, 12 + s);
          const uint64_t bd0 = ring_desc0 + static_cast<uint64_t>((stage * kStageBytes) >> 4);
          const uint32_t aw = tmem_w + s * kbh * 32;
          ACCT_BEGIN();
          for (int kb = 0; kb < kbh; ++kb) {
            if (leader) {
#pragma unroll
              for (int kk = 0; kk < BK / 16; ++kk)
                umma_ts(d_tmem, aw + kb * 32 + kk * 8, bd0 + static_cast<uint64_t>((kb * kBlockBytes) >> 4) + 2 * kk, idesc,
                        s > 0 || kb > 0 || kk > 0);  // the first MMA of a step overwrites the accumulator
            }
          }
          ACCT_END(4);
          ACCT_BEGIN();
          if (leader) umma_commit(&ring_empty[stage]);  // the whole segment, on its first stage's barrier
          ACCT_END(5);
          stage += seg_stages;
          if (stage == n_ring) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        FTB_CL_STAMP(i, 1);
        if (self) {
          // The cluster's own output of step i-1, copied by its producers into slot (i-1) & 1 of every CTA.
          const int slot = (i - 1) & 1;
          if (leader) mbar_arrive_expect_tx(&self_full[slot], self_slot_bytes);
          ACCT_BEGIN();
          ok = mbar_wait_warp(&self_full[slot], ((i - 1) >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
          ACCT_END(2);
          if (!ok) break;
          FTB_CL_STAMP(i, 2);
          // K = 16 is two 16-byte chunks, NB * 16 bytes apart; the descriptor
          // of MMA j is the slot's plus j * 2 * NB (bytes / 16): nothing is rebuilt per MMA.
          const uint64_t bd = self_desc0 + static_cast<uint64_t>((slot * self_slot_bytes) >> 4);
          const uint32_t aw = tmem_w + kbh * 32;
          for (int kb = 0; kb < kbh; ++kb) {
            if (leader) {
#pragma unroll
              for (int kk = 0; kk < BK / 16; ++kk)
                umma_ts(d_tmem, aw + kb * 32 + kk * 8, bd + static_cast<uint64_t>(kb * 4 + kk) * (2 * NB), idesc, 1u);
            }
          }
          if (leader) umma_commit_to(&self_free[slot], producer_mask);
        }
        if (leader) umma_commit(&tfull_bar[acc]);
        FTB_CL_STAMP(i, 3);
      }
#ifdef FTB_ACCT
      acct_[3] = clock64() - acct_loop0;
#endif
      ACCT_WRITE(0, 8);   // accumulator free
      ACCT_WRITE(1, 9);   // ring data
      ACCT_WRITE(2, 10);  // self operand
      ACCT_WRITE(3, 11);  // whole loop
      ACCT_WRITE(4, 15);  // MMA issue (ring operands)
      if (a.dil[layer] > 1) { ACCT_WRITE(5, 10); }  // commits (the slot of the self operand, unused here)
    }
  } else if (warp == 2) {
    // ------------------------------------------------ output store and flag publisher
    // The epilogue warps count themselves in `out_issued` once their part of a step's output tile is
    // staged in shared memory; this thread writes the tile to global memory with one TMA store, waits
    // for it to complete and releases the step's flag -- all of it off the chain's critical path.
    // (A running count, not an mbarrier: this thread may fall more than one step behind.  One for the even
    // and one for the odd steps: where a step does not need the one before, a warp can stage the next step
    // while another still works on this one, but not the one after that, which waits for `out_stored`.)
    if (lane == 0) {
      volatile int* stored = &out_stored;
      const int n_valid = min(NB, a.N - slice * NB);
      const CUtensorMap* om = n_valid == NB ? &mapO : &mapT;
      const int unit0 = rank * kOutUnits;
      ACCT_DECL(2);
      for (int i = 0; i < n_steps; ++i) {
        volatile int* issued = &out_issued[i & 1];
        const int want = kEpiWarps * ((i >> 1) + 1);
        ACCT_BEGIN();
        if (*issued < want) {
          const uint64_t t0 = globaltimer_ns();
          uint32_t it = 0;
          while (*issued < want) {
            if (((++it) & 0xFF) == 0 && (s_abort || globaltimer_ns() - t0 > FTB_WAIT_TIMEOUT_NS)) break;
          }
          if (*issued < want) {
            if (!s_abort) {
              s_abort = 1;
              atomicCAS(status, 0, FTB_ERR_TIMEOUT_EPI);
            }
            break;
          }
        }
        ACCT_END(0);
        ACCT_BEGIN();
        __threadfence_block();
        const int cell_row = (layer * a.L + i) * a.N + slice * NB;
        tma_store_2d(om, s_out + (i & 1) * kOutTileBytes, unit0, cell_row);
        tma_store_commit();
        tma_store_wait_read<0>();
        *stored = i + 1;  // the tile may be overwritten (two steps from now)
        tma_store_wait<0>();
        red_release_gpu_add(a.flags + (my_flag_cell0 + i) * a.S + slice, 1);
        ACCT_END(1);
        FTB_CL_STAMP(i, 11);
      }
      ACCT_WRITE(0, 13);  // staged outputs
      ACCT_WRITE(1, 14);  // store, wait, flag
    }
  } else if (warp >= kFirstEpiWarp) {
    // ---------------------------------------------------------------- epilogue
    constexpr int kCols = NB / kSub;          // batch columns of a warp
    constexpr int kRound = kCols < 32 ? kCols : 32;  // of them in registers at a time
    static_assert(kCols % 16 == 0 && kCols % kRound == 0, "columns come in fragments of 16");
    const int q = warp & 3, e = warp - kFirstEpiWarp;
    const int half = kSplit ? e >> 3 : 0, sub = kSplit ? (e & 7) >> 2 : e >> 2;
    // Resident weights -> TMEM: a thread copies one packed weight row to its lane, two 16-bit values per 32-bit
    // column (the layout of an A operand in tensor memory); the warps of a quadrant alternate K blocks.  The gates of
    // a unit are put 8 lanes apart, so that fragments of 16 lanes leave a thread with all of them (csrc/lstm_flow.cuh).
    {
      const uint4* wrow =
          reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.W) + (static_cast<size_t>(layer) * 4 * a.H + rank * 128 + q * 32 + 4 * (lane & 7) + (lane >> 3)) * K);
      for (int kb = e >> 2; kb < n_wkb; kb += kAllEpiWarps / 4) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 x4 = __ldg(wrow + kb * 8 + i);
          v[4 * i + 0] = x4.x; v[4 * i + 1] = x4.y; v[4 * i + 2] = x4.z; v[4 * i + 3] = x4.w;
        }
        tmem_st32(tmem_w + (static_cast<uint32_t>(q * 32) << 16) + kb * 32, v);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&res_full);
    }

    const int u_local = q * 8 + (lane >> 2), unit = rank * kOutUnits + u_local;
    const bool ub0 = (lane & 4) != 0, ub1 = (lane & 8) != 0;
    // This thread has batch columns n_own, n_own + 1, n_own + 8, n_own + 9 of every 16; after the exchange below it stores four
    // units of column n_store.
    const int n_own = sub * kCols + 2 * (lane & 3);
    const int n_store = n_own + (ub0 ? 8 : 0) + (ub1 ? 1 : 0);
    auto own = [&](int ci) { return n_own + (ci >> 2) * 16 + ((ci >> 1) & 1) * 8 + (ci & 1); };
    float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.bias != nullptr)
      bias4 = __ldg(reinterpret_cast<const float4*>(a.bias + static_cast<size_t>(layer) * 4 * a.H + rank * 128) + u_local);
    const int dil = a.dil[layer];
    constexpr int kOwn = kCols / 4;  // (unit, batch column) elements per thread
    float creg[kOwn];
#pragma unroll
    for (int i = 0; i < kOwn; ++i) creg[i] = 0.f;
    const int n_valid = min(NB, a.N - slice * NB);  // batch columns of this slice that exist
    // Where this thread's four units of column n sit (a) in the staging tile: 16-byte chunk q of NB rows, then row n, then
    // 8 bytes; (b) in the row-major output tile of 64-byte rows, 16-byte chunks swizzled by the row.
    const uint32_t stg_off = static_cast<uint32_t>(q) * NB * 16 + (lane >> 4) * 8;
    const uint32_t out_off = ((q ^ ((n_store >> 1) & 3)) << 4) + (lane >> 4) * 8;  // (rows 16 apart are swizzled alike)
    volatile int* stored = &out_stored;
    ACCT_DECL(2);

    bool ok = true;
    for (int i = half; i < n_steps && ok; i += kSplit ? 2 : 1) {
      const int acc = i & 1;
      // cell state of a layer with dilation > 1 lives in global memory between the steps that share it
      float* c_rows = nullptr;
      if (dil > 1)
        c_rows = a.c + (static_cast<size_t>(layer) * a.max_dil + (i % dil)) * a.N * a.H + static_cast<size_t>(slice) * NB * a.H + unit;
      if (dil > 1 && i >= dil) {
#pragma unroll
        for (int ci = 0; ci < kOwn; ++ci) creg[ci] = own(ci) < n_valid ? __ldcg(c_rows + static_cast<size_t>(own(ci)) * a.H) : 0.f;
      } else if (dil > 1) {
#pragma unroll
        for (int ci = 0; ci < kOwn; ++ci) creg[ci] = 0.f;
      }
      {
        // every lane waits on the accumulator's barrier (a single sleeping lane per warp and a vote
        // were measured slower: this wait is on the chain of a step)
        bool mine = mbar_wait(&tfull_bar[acc], (i >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
        if (lane == 0) {
          ACCT_BEGIN();
          ACCT_END(0);
          // the output tile of two steps ago must have left shared memory
          if (mine && *stored < i - 1) {
            const uint64_t t0 = globaltimer_ns();
            while (*stored < i - 1 && !s_abort && globaltimer_ns() - t0 < FTB_WAIT_TIMEOUT_NS) __nanosleep(64);
            mine = *stored >= i - 1;
          }
        }
        if (!__all_sync(0xffffffffu, mine)) {
          ok = false;
          break;
        }
      }
      tc_fence_after();
      if (warp == kFirstEpiWarp && lane == 0) { FTB_CL_STAMP(i, 4); }
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * NB + sub * kCols;
      uint8_t* stg = s_stg + (i & 1) * stage_tile_bytes + stg_off;
      uint8_t* outp = s_out + (i & 1) * kOutTileBytes + out_off;
#pragma unroll
      for (int r0 = 0; r0 < kCols; r0 += kRound) {
        uint32_t r_if[kRound / 16][8], r_oc[kRound / 16][8];
#pragma unroll
        for (int ch = 0; ch < kRound / 16; ++ch) {
          tmem_ld_frag16(taddr + r0 + ch * 16, r_if[ch]);
          tmem_ld_frag16(taddr + r0 + ch * 16 + (16u << 16), r_oc[ch]);
        }
        tmem_ld_wait();
        if (r0 + kRound == kCols) {
          // the accumulator is in registers: the MMA issuer may reuse it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty_bar[acc]);
        }
#pragma unroll
        for (int ch = 0; ch < kRound / 16; ++ch) {
          float h[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int at = 4 * (k >> 1) + (k & 1);
            float& c = creg[r0 / 4 + ch * 4 + k];
            const float gi = __uint_as_float(r_if[ch][at]) + bias4.x;
            const float gf = __uint_as_float(r_if[ch][at + 2]) + bias4.y;
            const float go = __uint_as_float(r_oc[ch][at]) + bias4.z;
            const float gc = __uint_as_float(r_oc[ch][at + 2]) + bias4.w;
            const float c_new = sigmoid_fast(gf) * c + sigmoid_fast(gi) * tanh_fast(gc);
            c = c_new;
            h[k] = sigmoid_fast(go) * tanh_fast(c_new);
          }
          // (unit, 4 sequences) -> (4 units, 1 sequence): trade halves with the units next to this one, twice
          const uint32_t p01 = Fmt<T>::pack2(h[0], h[1]), p23 = Fmt<T>::pack2(h[2], h[3]);
          uint32_t other = __shfl_xor_sync(0xffffffffu, ub0 ? p01 : p23, 4);
          const uint32_t lo = ub0 ? other : p01, hi = ub0 ? p23 : other;  // units u & ~1 and u | 1
          const uint32_t w0 = __byte_perm(lo, hi, 0x5410), w1 = __byte_perm(lo, hi, 0x7632);
          other = __shfl_xor_sync(0xffffffffu, ub1 ? w0 : w1, 8);
          const uint2 word = ub1 ? make_uint2(other, w1) : make_uint2(w0, other);
          const int n = n_store + r0 + ch * 16;
          *reinterpret_cast<uint2*>(outp + n * (kOutUnits * 2)) = word;
          if (self_chain) *reinterpret_cast<uint2*>(stg + n * 16) = word;
        }
      }
      if (dil > 1 || i == n_steps - 1) {
        float* c_out = dil > 1 ? c_rows
                               : a.c + static_cast<size_t>(layer) * a.max_dil * a.N * a.H + static_cast<size_t>(slice) * NB * a.H + unit;
#pragma unroll
        for (int ci = 0; ci < kOwn; ++ci)
          if (own(ci) < n_valid) c_out[static_cast<size_t>(own(ci)) * a.H] = creg[ci];
      }
      if (warp == kFirstEpiWarp && lane == 0) { FTB_CL_STAMP(i, 5); }
      fence_proxy_async_smem();  // plain shared-memory stores -> the bulk copies' and the TMA store's reads
      __syncwarp();
      if (warp == kFirstEpiWarp && lane == 0) { FTB_CL_STAMP(i, 14); }
      if (self_chain && i + 1 < n_steps) {
        // Hand the step's output to every CTA of the cluster, once all of them have multiplied what the
        // destination slot held before (two steps ago).
        // Once all epilogue warps have staged their parts, the tile goes to every CTA of the cluster by
        // bulk copies issued side by side by different warps.  (Measured: the SM's copy engine moves
        // about 64 KB in 1.3-2 us however the tile is cut -- 128 copies of 512 B, 32 of 2 KB or 8 of
        // 8 KB -- so the hand-off is bound by the bytes every CTA must receive, not by the slicing.)
        if (lane == 0) mbar_arrive(&stg_ready);
        const uint32_t kPiece = 2048u;
        const int n_pieces = static_cast<int>(stage_tile_bytes / kPiece);
        const int n_copies = n_pieces * a.CL;
        const int per_warp = (n_copies + kEpiWarps - 1) / kEpiWarps;
        const int ci = (warp - kFirstEpiWarp) * per_warp + lane;
        if (lane < per_warp && ci < n_copies) {
          bool go = mbar_wait(&stg_ready, i & 1, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
          if (warp == kFirstEpiWarp && lane == 0) { FTB_CL_STAMP(i, 15); }
          if (go && i >= 2) go = mbar_wait(&self_free[i & 1], ((i - 2) >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
          if (go) {
            const int peer = ci / n_pieces;
            const uint32_t off = static_cast<uint32_t>(ci - peer * n_pieces) * kPiece;
            const uint32_t src = smem_u32(s_stg + (i & 1) * stage_tile_bytes) + off;
            const uint32_t dst = smem_u32(s_self + (i & 1) * self_slot_bytes) +
                                 static_cast<uint32_t>(self_first_chunk) * NB * 16 + off;
            bulk_copy_to_peer(map_to_cta(dst, peer), src, kPiece, map_to_cta(smem_u32(&self_full[i & 1]), peer));
            if (warp == kFirstEpiWarp && lane == 0) { FTB_CL_STAMP(i, 6); }
          }
        }
      }
      // this warp's part of the output tile is staged: count it in for the publisher
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        atomicAdd(&out_issued[i & 1], 1);
      }
    }
    if (warp == kFirstEpiWarp && lane == 0) { ACCT_WRITE(0, 12); }  // accumulator complete
    // The peers' commits for the last two slots, which no step waits for, have to be in before this CTA leaves (ring_drain, ptx.cuh).
    if (self_chain && ok && warp == kFirstEpiWarp && lane == 0)
      for (int i = max(0, n_steps - 3); i <= n_steps - 2 && ok; ++i)
        ok = mbar_wait(&self_free[i & 1], (i >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  // No CTA of the cluster may leave while a peer can still copy into it or signal its barriers.
  cluster_sync_all();
  if (warp == 1) {
    if (s_abort) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Dilated LSTM: a layer's clusters take 64 or 128 sequences each (a.nb[layer]).  A layer whose step
// depends on its own previous step (dilation 1) is a chain of hand-offs inside the cluster, whose
// latency grows with the slice (state bytes every CTA receives, accumulator columns per epilogue
// warp): it runs on slices of 64; the other layers, whose steps are bound by throughput, on 128.
// x128/h128/o128/t128: the input, the hidden states, the output tile and the output tile of the
// batch's last (short) slice as boxes of 128 rows; x64... the same with 64 rows.
template <typename T>
__global__ void __launch_bounds__(kCtaThreads, 1)
rnn_cluster_dilated_kernel(const __grid_constant__ CUtensorMap x128, const __grid_constant__ CUtensorMap h128,
                           const __grid_constant__ CUtensorMap x64, const __grid_constant__ CUtensorMap h64,
                           const __grid_constant__ CUtensorMap o128, const __grid_constant__ CUtensorMap o64,
                           const __grid_constant__ CUtensorMap t128, const __grid_constant__ CUtensorMap t64,
                           const ClusterArgs a) {
  const int cid = blockIdx.x / a.CL;
  int layer = 0;
  while (layer + 1 < a.D && cid >= a.first_cluster[layer + 1]) ++layer;
  const int slice = cid - a.first_cluster[layer];
  const int rank = cluster_ctarank();
  const bool split = a.dil[layer] % 2 == 0;
  if (a.nb[layer] == 64) {
    if (split) cluster_body<T, 64, true>(x64, h64, o64, t64, a, rank, cid, layer, slice);
    else cluster_body<T, 64, false>(x64, h64, o64, t64, a, rank, cid, layer, slice);
  } else {
    if (split) cluster_body<T, 128, true>(x128, h128, o128, t128, a, rank, cid, layer, slice);
    else cluster_body<T, 128, false>(x128, h128, o128, t128, a, rank, cid, layer, slice);
  }
}

// The same program without clusters, where it fits: what the layers with dilation >= 2 exchange goes through
// global memory anyway (at H 256 a step takes 1.5 us on slices of 64, 2.5 on 128, or its part of the trip there and back,
// 4.7 and 5.0 over the dilation: 2.35 on slices of 64 with dilation 2).  A layer with dilation 1 runs as csrc/lstm_flow.cu does, on narrow slices whose state is
// its own flag: 1.6 us a step at H 256 and 32 sequences where a cluster's hand-off of 64 takes 2.6, and no GPC has to
// hold a chain's CTAs (15 clusters of 8 leave 28 SMs idle).  A layer with dilation 2 does so too where its slices fit: as a layer
// of 2 N sequences and half the steps, whose trip there and back it no longer waits for (dilated_flow_widths).
struct DilatedMaps {
  CUtensorMap x64, h64, o64, t64, x128, h128, o128, t128;  // as above
  CUtensorMap nx[2], nh[2], nw;                             // of flow::body, by time steps of a step - 1
};
template <typename T>
__global__ void __launch_bounds__(kCtaThreads, 1)
rnn_dilated_flow_kernel(const __grid_constant__ DilatedMaps m, const __grid_constant__ ClusterArgs a,
                        const __grid_constant__ flow::FlowArgs f1, const __grid_constant__ flow::FlowArgs f2) {
  const int cid = blockIdx.x / a.CL, rank = blockIdx.x - cid * a.CL;
  int layer = 0;
  while (layer + 1 < a.D && cid >= a.first_cluster[layer + 1]) ++layer;
  const int slice = cid - a.first_cluster[layer];
  const int fold = a.fold[layer], nb = a.nb[layer];
  const int nb_below = layer > 0 ? a.nb[layer - 1] : nb, fold_below = layer > 0 ? max(a.fold[layer - 1], 1) : 1;
  if (fold == 1) {
    if (nb == 16) flow::body<T, 16>(m.nx[0], m.nh[0], m.nw, f1, rank, slice, layer, nb_below, fold_below);
    else if (nb == 32) flow::body<T, 32>(m.nx[0], m.nh[0], m.nw, f1, rank, slice, layer, nb_below, fold_below);
    else flow::body<T, 48>(m.nx[0], m.nh[0], m.nw, f1, rank, slice, layer, nb_below, fold_below);
    return;
  }
  if (fold == 2) {
    if (nb == 16) flow::body<T, 16>(m.nx[1], m.nh[1], m.nw, f2, rank, slice, layer, nb_below, fold_below);
    else if (nb == 32) flow::body<T, 32>(m.nx[1], m.nh[1], m.nw, f2, rank, slice, layer, nb_below, fold_below);
    else flow::body<T, 64>(m.nx[1], m.nh[1], m.nw, f2, rank, slice, layer, nb_below, fold_below);
    return;
  }
  const bool split = a.dil[layer] % 2 == 0;
  if (nb == 64) {
    if (split) cluster_body<T, 64, true>(m.x64, m.h64, m.o64, m.t64, a, rank, cid, layer, slice);
    else cluster_body<T, 64, false>(m.x64, m.h64, m.o64, m.t64, a, rank, cid, layer, slice);
  } else {
    if (split) cluster_body<T, 128, true>(m.x128, m.h128, m.o128, m.t128, a, rank, cid, layer, slice);
    else cluster_body<T, 128, false>(m.x128, m.h128, m.o128, m.t128, a, rank, cid, layer, slice);
  }
}

// Tensor map of a row-major [rows, H] activation matrix as the kernel's operand loads see it: three
// dimensions (64 columns of a K block, rows, K blocks), so that one copy brings the NB rows of all
// H / 64 K blocks of a segment into consecutive 128-byte-swizzled [NB x 64] tiles of the ring.
int make_operand_map(CUtensorMap* out, const void* base, int dtype, uint64_t rows, int H, int nb) {
  return make_tmap_3d(out, base, dtype, 64, rows, static_cast<uint64_t>(H / 64), static_cast<uint64_t>(H) * 2, 128, 64,
                      static_cast<uint32_t>(nb), static_cast<uint32_t>(H / 64));
}

template <typename Kernel, typename... Args>
int launch_kernel(Kernel kfn, int cluster, int threads, std::atomic<unsigned long long>& configured, uint32_t max_dynamic,
                  int grid, uint32_t smem_bytes, cudaStream_t stream, const Args&... args) {
  if (smem_bytes > max_dynamic || !ensure_dynamic_smem(kfn, max_dynamic, configured)) return FTB_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
  if (cluster > 1) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = cluster;
    attrs[na].val.clusterDim.y = 1;
    attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  // FTB_NO_COOPERATIVE=1 drops the cooperative attribute (profilers that cannot replay cooperative
  // launches); residency then rests on the grid fitting an otherwise idle device, and the bounded
  // waits turn a violated assumption into a status code.
  static const bool no_coop = [] {
    const char* e = getenv("FTB_NO_COOPERATIVE");
    return e != nullptr && e[0] == '1';
  }();
  // FTB_REFUSE_COOPERATIVE=1 answers as if the driver had refused the launch (host-side failure
  // injection for the tests of the fallback to the generic wavefront).
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
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kfn, args...);
  if (err != cudaSuccess) {
    if (getenv("FTB_VERBOSE") != nullptr) fprintf(stderr, "rnn_cluster launch: %s\n", cudaGetErrorString(err));
    cudaGetLastError();
    return FTB_ERR_LAUNCH;
  }
  count_launch();
  return FTB_OK;
}

constexpr uint32_t smem_for(bool any_self, int H) {
  // worst case over the chains of the launch (slices of 128); must agree with the kernel's carve-up
  constexpr int NB = 128;
  const uint32_t out_tiles = 2u * NB * kOutUnits * 2;
  const uint32_t with_self = 2u * (H / 8) * NB * 16 + 2u * (kOutUnits / 8) * NB * 16 + out_tiles + 4u * kStageBytes;
  const uint32_t without = out_tiles + 12u * kStageBytes;
  return (any_self ? std::max(with_self, without) : without) + 1024;
}
// The largest requests of the two kernels: their static shared memory, the barriers of all their bodies, comes on top (227 KB in
// all; without clusters no state is kept in shared memory, whatever H is).
constexpr uint32_t kClusterSmem = smem_for(true, 256);

template <typename T>
int launch_dilated(const CUtensorMap* m, const ClusterArgs& a, int grid, uint32_t smem_bytes, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  return launch_kernel(rnn_cluster_dilated_kernel<T>, a.CL, kCtaThreads, configured, kClusterSmem, grid, smem_bytes, stream, m[0],
                       m[1], m[2], m[3], m[4], m[5], m[6], m[7], a);
}
template <typename T>
int launch_dilated_flow(const DilatedMaps& m, const ClusterArgs& a, const flow::FlowArgs (&f)[2], int grid, uint32_t smem_bytes,
                        cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  return launch_kernel(rnn_dilated_flow_kernel<T>, 1, kCtaThreads, configured, smem_for(false, 256), grid, smem_bytes, stream, m, a, f[0],
                       f[1]);
}

}  // namespace

// ------------------------------------------------------------------ dilated LSTM
namespace {
// Slice width per layer: 64 for the layers with dilation 1 when the clusters still fit, else 128
// everywhere.  Returns the number of clusters, 0 when even slices of 128 do not fit.
int dilated_slices(const int* dilations, int D, int N, int max_clusters, int* nb) {
  const int s128 = (N + 127) / 128, s64 = (N + 63) / 64;
  auto narrow = [&](int l) { return N <= 64 || (dilations != nullptr && dilations[l] == 1); };
  int mixed = 0;
  for (int l = 0; l < D; ++l) mixed += narrow(l) ? s64 : s128;
  const bool use_mixed = s64 <= 8 && mixed <= max_clusters;
  int total = 0;
  for (int l = 0; l < D; ++l) {
    const bool n64 = use_mixed && narrow(l);
    if (nb != nullptr) nb[l] = n64 ? 64 : 128;
    total += n64 ? s64 : s128;
  }
  return s128 <= 8 && total <= max_clusters ? total : 0;
}

// How a launch without clusters cuts the layers, false: it does not fit or no layer has dilation 1.  Layers of dilation 1 run
// flow::body on slices of 16, 32 or 48 sequences; those of dilation 2 too, on slices of 16, 32 or 64 of 2 N, or like the others as
// cells of slices of 64 or 128 whose states make a trip through global memory.  The slowest layer sets the pace; its time per time
// step is estimated from layers alone and beside others (us, H 128 / 256; 16, 32, 48 and 64 columns 1.5, 1.55, 1.87, 2.1 / 1.6, 1.85,
// 2.15, 2.55 a step of flow::body; cells of 64 and 128 1.15, 1.5 / 1.5, 2.5, a trip 3.6, 4.2 / 4.7, 5.0), the narrowest cut wins a
// tie.  Dilations 1 2 4 and 1 .. 32, us a time step with dilation 2 as cells / as it is taken: H 128, 17 sequences 1.85 / 1.50, 1.80 /
// 1.57; H 256, 33 2.09 / 1.75, 2.16 / 1.81; 128 2.25 / 2.00, 2.32 / 2.18; 256 as cells (2.40; 2.68 as 2 N sequences).
bool dilated_flow_widths(const int* dilations, int D, int N, int H, int CL, int sm_count, int* nb, int* fold) {
  bool one = false, two = false;
  for (int l = 0; l < D; ++l) {
    one = one || dilations[l] == 1;
    two = two || dilations[l] == 2;
  }
  if (!one) return false;
  const double h = H / 128.0 - 1.0;  // -0.5, 0, 1
  // (not below H 128: at H 64 a step of 16 takes 1.3 and one of 32 1.5, and all is latency)
  const double hf = std::max(h, 0.0);
  auto flow_step = [&](int w) { return w == 16 ? 1.5 + 0.1 * hf : w == 32 ? 1.55 + 0.3 * hf : w == 48 ? 1.87 + 0.28 * hf : 2.1 + 0.45 * hf; };
  auto cell = [&](int w, int d) {
    return w == 64 ? std::max(1.15 + 0.35 * h, (3.6 + 1.1 * h) / d) : std::max(1.5 + h, (4.2 + 0.8 * h) / d);
  };
  double best = 0.0;
  for (int wide = 64; wide <= 128; wide *= 2)
    for (int second : {16, 32, 64, 0}) {  // 0: dilation 2 as cells
      if (second > 0 && !two) continue;
      for (int narrow = 16; narrow <= 48; narrow += 16) {
        int ctas = 0;
        double pace = 0.0;
        auto cut = [&](int l, int* f) {
          *f = dilations[l] == 1 ? 1 : dilations[l] == 2 && second > 0 ? 2 : 0;
          return *f == 1 ? narrow : *f == 2 ? second : dilations[l] == 2 ? 64 : wide;
        };
        for (int l = 0; l < D; ++l) {
          int f;
          const int w = cut(l, &f), slices = (std::max(f, 1) * N + w - 1) / w;
          ctas += slices > 64 ? sm_count + 1 : CL * slices;  // (64: counters a cell)
          pace = std::max(pace, f > 0 ? flow_step(w) / f : cell(w, dilations[l]));
        }
        if (ctas > sm_count || (best > 0.0 && pace >= best)) continue;
        best = pace;
        for (int l = 0; l < D; ++l) nb[l] = cut(l, &fold[l]);
      }
    }
  return best > 0.0;
}
// Short sequences of a few narrow states: the arrays that the form without clusters has filled before it starts cost more than its
// shorter steps give back.  us, with clusters / without, H 64: 4 layers, L 8, N 26 34.8 / 41.2; 6 layers, L 12, N 28 46.2 / 51.3, L 22, N 3
// 60.2 / 64.7, L 43, N 29 99.5 / 102.6; L 64 and more 0.92 to 1.0 times without, above 64 sequences 0.73 to 0.94; H 128 0.73 to 0.99, H 256
// 0.62 to 0.98 (400 calls of 8 to 512 steps).
bool dilated_prefers_clusters(int L, int N, int CL) { return CL == 2 && L < 48 && N <= 64; }
// Clusters of `cl` CTAs of the dilated kernel that can be resident at once on the current device (a
// cluster needs its CTAs' SMs inside one GPC, so this is less than SMs / cl: 15 clusters of 8 on a
// 148-SM B200).  0 when the query fails.
int dilated_max_clusters(int dtype, int cl, uint32_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl * 32);
  cfg.blockDim = dim3(kCtaThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  cudaError_t e;
  if (dtype == FTB_F16) {
    static std::atomic<unsigned long long> configured{0};
    if (!ensure_dynamic_smem(rnn_cluster_dilated_kernel<__half>, kClusterSmem, configured)) return 0;
    e = cudaOccupancyMaxActiveClusters(&n, rnn_cluster_dilated_kernel<__half>, &cfg);
  } else {
    static std::atomic<unsigned long long> configured{0};
    if (!ensure_dynamic_smem(rnn_cluster_dilated_kernel<__nv_bfloat16>, kClusterSmem, configured)) return 0;
    e = cudaOccupancyMaxActiveClusters(&n, rnn_cluster_dilated_kernel<__nv_bfloat16>, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}
}  // namespace

bool lstm_dilated_cluster_supported(int dtype, int D, int N, int H, int sm_count) {
  if (dtype != FTB_F16 && dtype != FTB_BF16) return false;
  if (H != 64 && H != 128 && H != 256) return false;  // 4H / 128 = 2, 4 or 8 CTAs per cluster
  if (D < 1 || D > kMaxLayers || N < 1) return false;
  // (coarse: the launcher asks the driver how many clusters fit and falls back if these do not)
  return dilated_slices(nullptr, D, N, sm_count / (4 * H / 128), nullptr) > 0;
}

// one counter per (cell, slice of 16 sequences or more); at most 64 (1024 sequences)
size_t lstm_dilated_cluster_flag_ints(int D, int L) { return static_cast<size_t>(D) * L * 64; }

// x: [L,N,H]; Wp: [D,4H,2H]; hs: [D,L,N,H]; c: [D, max_dil*N, H]; flags: D*L*S ints (zeroed here).  schedule 4: with
// clusters where they fit, 5: without (FTB_ERR_ARG where that does not fit), 0: the faster of the two.
int launch_lstm_dilated_cluster(int dtype, const void* x, const void* Wp, const float* bias_p, void* hs, float* c,
                                const int* dilations, int D, int L, int N, int H, int schedule, int* flags, int* status,
                                int sm_count, cudaStream_t stream) {
  ClusterArgs a = {};
  a.D = D; a.L = L; a.N = N; a.H = H;
  a.CL = 4 * H / 128;
  a.max_dil = 1;
  bool any_self = false;
  for (int l = 0; l < D; ++l) {
    a.dil[l] = dilations[l];
    a.max_dil = std::max(a.max_dil, dilations[l]);
    any_self = any_self || dilations[l] == 1;
  }
  a.W = Wp; a.bias = bias_p; a.c = c; a.flags = flags; a.status = status;
  const uint64_t x_rows = static_cast<uint64_t>(L) * N, h_rows = static_cast<uint64_t>(D) * L * N;
  CUtensorMap m[8];
  int rc;
  const uint32_t cluster_smem = smem_for(any_self, H);
  auto cut_for_clusters = [&] { return dilated_slices(dilations, D, N, dilated_max_clusters(dtype, a.CL, cluster_smem), a.nb); };
  int clusters = schedule == 4 || (schedule == 0 && dilated_prefers_clusters(L, N, a.CL)) ? cut_for_clusters() : 0;
  if (clusters <= 0 && dilated_flow_widths(dilations, D, N, H, a.CL, sm_count, a.nb, a.fold)) {
    int width[2] = {0, 0};  // of the slices of layers that run flow::body, by time steps of a step - 1
    for (int l = 0; l < D; ++l) {
      const int slices = (std::max(a.fold[l], 1) * N + a.nb[l] - 1) / a.nb[l];
      a.S = std::max(a.S, slices);
      a.first_cluster[l + 1] = a.first_cluster[l] + slices;
      if (a.fold[l] > 0) width[a.fold[l] - 1] = a.nb[l];
    }
    DilatedMaps dm;
    for (int wide = 64; wide <= 128; wide *= 2) {
      const int tail = N - ((N + wide - 1) / wide - 1) * wide;
      if ((rc = make_operand_map(wide == 64 ? &dm.x64 : &dm.x128, x, dtype, x_rows, H, wide))) return rc;
      if ((rc = make_operand_map(wide == 64 ? &dm.h64 : &dm.h128, hs, dtype, h_rows, H, wide))) return rc;
      if ((rc = make_tmap_2d_sw64(wide == 64 ? &dm.o64 : &dm.o128, hs, dtype, h_rows, H, H, wide))) return rc;
      if ((rc = make_tmap_2d_sw64(wide == 64 ? &dm.t64 : &dm.t128, hs, dtype, h_rows, H, H, tail))) return rc;
    }
    for (int i = 0; i < 2; ++i) {
      const uint32_t w = width[i] > 0 ? width[i] : width[0], planes = 128 / w;  // of a copy of flow::body
      if ((rc = make_tmap_steps(&dm.nx[i], x, dtype, 1, x_rows, H, w, planes))) return rc;
      if ((rc = make_tmap_steps(&dm.nh[i], hs, dtype, 1, h_rows, H, w, planes))) return rc;
    }
    if ((rc = make_tmap_gates(&dm.nw, Wp, dtype, static_cast<uint64_t>(D) * 4 * H, 2 * H))) return rc;
    flow::FlowArgs f[2] = {};
    for (int i = 0; i < 2; ++i) {
      f[i].fold = i + 1; f[i].N1 = N; f[i].flag_steps = L;
      f[i].D = D; f[i].L = (L + i) / (i + 1); f[i].N = N * (i + 1); f[i].I = H; f[i].H = H; f[i].G = D; f[i].S = a.S;
      f[i].n_tiles = a.CL;
      f[i].n_slots = flow::kMaxSlots;
      f[i].T = static_cast<int64_t>(L) * N;
      f[i].bias_p = bias_p; f[i].Wp = Wp; f[i].hs = hs; f[i].c_out = c; f[i].c_rows = a.max_dil * N; f[i].flags = flags;
      f[i].status = status;
    }
    if (cudaMemsetAsync(flags, 0, sizeof(int) * static_cast<size_t>(D) * L * a.S, stream) != cudaSuccess) return FTB_ERR_LAUNCH;
    const size_t layer_bytes = static_cast<size_t>(L) * N * H * 2;
    for (int l = 0, n; l < D; l += std::max(n, 1)) {  // neighbouring layers in one go
      for (n = 0; l + n < D && a.fold[l + n] > 0;) ++n;
      if (n > 0 && cudaMemsetAsync(static_cast<char*>(hs) + l * layer_bytes, 0xFF, n * layer_bytes, stream) != cudaSuccess)
        return FTB_ERR_LAUNCH;
    }
    const uint32_t smem = smem_for(false, H);
    const int grid = a.first_cluster[D] * a.CL;
    if (dtype == FTB_F16) return launch_dilated_flow<__half>(dm, a, f, grid, smem, stream);
    return launch_dilated_flow<__nv_bfloat16>(dm, a, f, grid, smem, stream);
  }
  if (schedule == 5) return FTB_ERR_ARG;
  if (clusters <= 0) clusters = cut_for_clusters();
  if (clusters <= 0) return FTB_ERR_LAUNCH;  // does not fit on this device: the caller's generic wavefront takes it
  a.S = (N + 63) / 64;
  for (int l = 0; l < D; ++l) a.first_cluster[l + 1] = a.first_cluster[l] + (N + a.nb[l] - 1) / a.nb[l];
  if ((rc = make_operand_map(&m[0], x, dtype, x_rows, H, 128))) return rc;
  if ((rc = make_operand_map(&m[1], hs, dtype, h_rows, H, 128))) return rc;
  if ((rc = make_operand_map(&m[2], x, dtype, x_rows, H, 64))) return rc;
  if ((rc = make_operand_map(&m[3], hs, dtype, h_rows, H, 64))) return rc;
  // output boxes: the slice's (or the last, short slice's) rows x the 32 units of a CTA
  const int tail128 = N - ((N + 127) / 128 - 1) * 128, tail64 = N - ((N + 63) / 64 - 1) * 64;
  if ((rc = make_tmap_2d_sw64(&m[4], hs, dtype, h_rows, H, H, 128))) return rc;
  if ((rc = make_tmap_2d_sw64(&m[5], hs, dtype, h_rows, H, H, 64))) return rc;
  if ((rc = make_tmap_2d_sw64(&m[6], hs, dtype, h_rows, H, H, tail128))) return rc;
  if ((rc = make_tmap_2d_sw64(&m[7], hs, dtype, h_rows, H, H, tail64))) return rc;
  const size_t n_flags = static_cast<size_t>(D) * L * a.S;
  if (cudaMemsetAsync(flags, 0, sizeof(int) * n_flags, stream) != cudaSuccess) return FTB_ERR_LAUNCH;
  const int grid = clusters * a.CL;
  if (dtype == FTB_F16) return launch_dilated<__half>(m, a, grid, cluster_smem, stream);
  return launch_dilated<__nv_bfloat16>(m, a, grid, cluster_smem, stream);
}

}  // namespace ftb

#ifdef FTB_ACCT
extern "C" int ftb_debug_set_cluster_acct(unsigned long long* buf) {
  return cudaMemcpyToSymbol(ftb::g_cluster_acct, &buf, sizeof(buf)) == cudaSuccess ? 0 : 1;
}
#endif
#ifdef FTB_TRACE
extern "C" int ftb_debug_set_cluster_trace(unsigned long long* buf) {
  return cudaMemcpyToSymbol(ftb::g_cluster_trace, &buf, sizeof(buf)) == cudaSuccess ? 0 : 1;
}
#endif

