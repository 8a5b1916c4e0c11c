// Flash attention forward on pairs of CTAs (tcgen05 .cta_group::2), 16-bit inputs, head dimension 128: the recurrence,
// masks and results of flash_attn.cu.
//
// A pair takes 256 query rows of a (batch, head), 128 a CTA, and walks their key/value blocks of 128 keys.  Both products
// are M = 256 MMAs over both SMs: of each K and V tile a CTA loads and holds one half, so that a block costs an SM 32 KB
// from L2 (64 KB a 256-row CTA) and S = Q K^T reads 96 bytes of shared memory a cycle instead of 128, its limit.
// The two slots of flash_attn_kernel are two query tiles; here all of an SM's tensor memory serves ONE tile of 128 rows:
// the accumulator (128 columns), the scores of two blocks (256) and the probabilities of two (128).  Scores are
// dead once they are in registers, so S of block n + 2 is multiplied while block n is in its softmax, and the products of a
// block wait for nothing but its probabilities.
//   warp 0        queries and K tiles (TMA)            warp 3        V tiles
//   warp 1        S = Q K^T (leader CTA)               warp 2        O += P V (leader CTA)
//   warps 4..7    output: O / l -> 16 bits -> the unit's query tile -> TMA store
//   warps 8..11, 12..15   softmax of the even / odd blocks, a row a thread (192 registers: 128 scores stay in them)
// The products have a warp each because tcgen05.fence::after_thread_sync waits for the MMAs that its own warp has issued:
// with one warp for both, every block drained the tensor pipe twice (1560 cycles a block, 1450 with one fence).
// Hand-offs to the leader go by mbarrier.arrive without .release.cluster (they guard tensor memory, which the tcgen05
// fences order): with it the arriving warp stood still for 1400 cycles, 518 us instead of 421 on the first version.
//
// The running maximum of a row passes from group to group (block n needs the reference of block n - 1): a float in shared
// memory and a barrier a warp.  The turn is handed on in the middle of a block's exponentials rather than before them: the
// groups' exponentials then overlap by half and the rest of a block runs beside the other group's (455 -> 437 us).
// What bounds it: the softmax groups, 1500 cycles a block: the special-function unit is busy for 1024 of them, as is the
// tensor pipe; the maximum, the packing and the waits of a group are the rest, beside the other group's exponentials.
// Persistent: 74 pairs take units (256 rows) in turn, a unit's first S behind the last of the one before.  Masked units are
// ordered longest first among as many (batch, head) entries as have 64 MB of K and V, every other round in reverse.
//
// Measured, us, 256-row CTAs / halves / this kernel, one box: full fp16 16 x 16 x 2048 490 / 574 / 438, 1 x 20 x 2048 68 / 63 /
// 45, 1 x 4 x 4096 63 / 37 / 33, 1 x 16 x 256 8.2 / 7.2 / 7.4; causal 16 x 16 x 2048 364 / 448 / 313, 1 x 16 x 2048 37 / 28 / 23.4,
// 1 x 16 x 2560 45 / 41 / 32, 4 x 16 x 512 14.6 / 19 / 16.1; window of 100 2 x 16 x 4096 50 / 57 / 54.
// Built and not kept: scores in three buffers under the probabilities (422 us, on another box: no more than boxes differ by; the
// product of block n then stands between the softmax of n and the scores of n + 3), two threads a row (446: the exchange of half maxima costs what the shorter
// chains give), a polynomial 2^x for a part of the exponentials (a pair costs 26 issue cycles and saves 16 of the
// special-function unit: 455 us at a quarter, 504 at a half), exponentials against the group's own reference, checked afterwards (472).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "../../include/ftb200.h"
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {
namespace {

constexpr int kTileBytes = 128 * 128 * 2;  // 128 query rows of 128 16-bit columns: two halves of 64 columns
constexpr int kHalfBytes = kTileBytes / 2;
constexpr int kSlotBytes = 16384;  // this CTA's half of a K tile (64 keys) or of a V tile (64 columns)
constexpr int kSlotsK = 4, kSlotsV = 4;
constexpr int kThreads = 512;
constexpr float kRescaleThreshold = 8.0f;
// Columns of tensor memory: the accumulator, two blocks of scores, two of probabilities (16-bit pairs).
constexpr uint32_t kScores = 128, kProbs = 384;

// Where a producer of a ring stopped: the slot of its next fill, and the parity of the fills of this pass.
struct RingEnd {
  int at;
  uint32_t phase;
};
struct Control {
  float m_x[2][128];           // [group][row]: the running maximum after the group's latest block
  float2 stats[2][2][128];     // [unit & 1][group][row]: (maximum, row sum) of the group's blocks
  uint64_t q_full[2], q_empty[2];
  uint64_t k_full[kSlotsK], k_empty[kSlotsK], v_full[kSlotsV];
  uint64_t s_full[2], s_free[2], p_full[2];
  uint64_t pv_done[4];
  uint64_t o_full, o_free;
  uint64_t l_full[2];
  uint64_t turn[2][4];         // [group][lane quadrant]
  RingEnd q_end, k_end, v_end;  // where the producers stopped
  uint32_t tmem_base, peer_tmem_base;
  int abort, dead;
};
constexpr uint32_t kTilesBytes = 2 * kTileBytes + (kSlotsK + kSlotsV) * kSlotBytes;
constexpr uint32_t kSmemBytes = 232448;
static_assert(kTilesBytes + sizeof(Control) + 512 <= kSmemBytes, "shared memory budget");

// umma_ts_pair without the rows of one CTA of the pair: off0 / off1 = all ones leave the leader's / the peer's rows as they are.
__device__ __forceinline__ void umma_ts_pair_rows(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                                  uint32_t off0, uint32_t off1, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, {%4, %4, %4, %4, %5, %5, %5, %5}, p;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(off0), "r"(off1), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ uint64_t fma_to_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ void unpair_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// Whether the phase is over, without waiting.
__device__ __forceinline__ bool mbar_test(const uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
template <int N>
__device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

__device__ __forceinline__ uint8_t* sw128_chunk_ptr(uint8_t* tile, int row, int chunk16) {
  return tile + (chunk16 >> 3) * kHalfBytes + row * 128 + (((chunk16 & 7) ^ (row & 7)) << 4);
}

// The walk of one unit: 256 query rows of a (batch, head), 128 a CTA of the pair.
struct Unit {
  int row_base, qpair, blk0, n, first1, last0;
};
struct Shape {
  int S, n_bh, group, left, right;
};
template <bool kMasked>
__device__ __forceinline__ bool unit_of(const Shape& sh, int w, int G, int c, Unit& u) {
  const int pairs = sh.S >> 8;
  const int idx = w * G + ((kMasked && (w & 1)) ? G - 1 - c : c);
  if (idx >= sh.n_bh * pairs) return false;
  int bh = idx / pairs;
  u.qpair = idx - bh * pairs;
  u.blk0 = 0;
  u.n = sh.S >> 7;
  u.first1 = 0;
  u.last0 = u.n - 1;
  if (kMasked) {
    const int per_group = sh.group * pairs;
    const int g = idx / per_group;
    const int r = idx - g * per_group;
    const int gsize = min(sh.group, sh.n_bh - g * sh.group);
    u.qpair = pairs - 1 - r / gsize;
    bh = g * sh.group + r % gsize;
    const int r0 = u.qpair * 256;
    const int lo0 = sh.left >= 0 ? max(0, r0 - sh.left) >> 7 : 0;
    const int lo1 = sh.left >= 0 ? max(0, r0 + 128 - sh.left) >> 7 : 0;
    const int hi0 = min((sh.S >> 7) - 1, (r0 + 127 + sh.right) >> 7);
    const int hi1 = min((sh.S >> 7) - 1, (r0 + 255 + sh.right) >> 7);
    u.blk0 = lo0;
    u.n = hi1 - lo0 + 1;
    u.first1 = lo1 - lo0;
    u.last0 = hi0 - lo0;
  }
  u.row_base = bh * sh.S;
  return true;
}

template <typename T, bool kMasked>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
flash_pair_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                  const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO, Shape sh,
                  float scale_log2, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  // (the segment starts at the same address in both CTAs of a pair: one kernel, one layout)
  if (pad + kTilesBytes + sizeof(Control) > kSmemBytes) {
    grid_dependency_wait();
    if (threadIdx.x == 0) atomicCAS(status, 0, FTB_ERR_ALIGN);
    return;
  }
  uint8_t* smem = smem_raw + pad;
  uint8_t* sQ = smem;                          // two tiles, units in turn
  uint8_t* sK = sQ + 2 * kTileBytes;           // rings
  uint8_t* sV = sK + kSlotsK * kSlotBytes;
  Control& ctl = *reinterpret_cast<Control*>(smem + kTilesBytes);
  volatile int* s_abort = &ctl.abort;
  const int G = gridDim.x >> 1, cid = blockIdx.x >> 1;

  grid_launch_dependents();
  if (threadIdx.x == 0) {
    prefetch_tmap(&mapQ);
    prefetch_tmap(&mapK);
    prefetch_tmap(&mapV);
    prefetch_tmap(&mapO);
    for (int i = 0; i < kSlotsK; ++i) {
      mbar_init(&ctl.k_full[i], 1);
      mbar_init(&ctl.k_empty[i], 1);
    }
    for (int i = 0; i < kSlotsV; ++i) {
      mbar_init(&ctl.v_full[i], 1);
      mbar_init(&ctl.pv_done[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl.s_full[i], 1);
      mbar_init(&ctl.s_free[i], 8);
      mbar_init(&ctl.p_full[i], 8);
      mbar_init(&ctl.l_full[i], 8);
      for (int k = 0; k < 4; ++k) mbar_init(&ctl.turn[i][k], 1);
      mbar_init(&ctl.q_full[i], 1);
      mbar_init(&ctl.q_empty[i], 5);  // the unit's last S, the warps that store its output from there
    }
    mbar_init(&ctl.o_full, 1);
    mbar_init(&ctl.o_free, 8);
    ctl.abort = 0;
    ctl.peer_tmem_base = 0xffffffffu;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc_pair(&ctl.tmem_base, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl.tmem_base;
  if (threadIdx.x == 0 && rank == 1) st_shared_cluster_u32(map_to_cta(smem_u32(&ctl.peer_tmem_base), 0), tmem_base);
  cluster_sync_all();
  grid_dependency_wait();
  if (threadIdx.x == 0) {
    if (rank == 0 && ctl.peer_tmem_base != tmem_base) atomicCAS(status, 0, FTB_ERR_TMEM_LAYOUT);
    ctl.dead = *reinterpret_cast<volatile int*>(status) != 0;
  }
  __syncthreads();
  const bool dead = ctl.dead != 0;

  if (warp < 4) {
    regs_dec<48>();
    const bool leader = elect_one();
    Unit u;
    bool ok = !dead;
    int n = 0;  // blocks so far
    if (warp == 0) {
      // ------------------------------------------------------------ queries and K tiles
      if (leader) {
        int slot = 0, w = 0;
        uint32_t phase = 0;
        for (; ok && unit_of<kMasked>(sh, w, G, cid, u); ++w) {
          const int b = w & 1;
          ok = mbar_wait(&ctl.q_empty[b], ((w >> 1) & 1) ^ 1u, s_abort, status, FTB_ERR_TIMEOUT_SLOT);
          if (!ok) break;
          if (rank == 0) mbar_arrive_expect_tx(&ctl.q_full[b], 2 * kTileBytes);
          const uint32_t q_bar = map_to_cta(smem_u32(&ctl.q_full[b]), 0);
          const int r = u.row_base + u.qpair * 256 + static_cast<int>(rank) * 128;
          tma_load_2d_pair(sQ + b * kTileBytes, &mapQ, q_bar, 0, r);
          tma_load_2d_pair(sQ + b * kTileBytes + kHalfBytes, &mapQ, q_bar, 64, r);
          for (int j = 0; j < u.n; ++j) {
            ok = mbar_wait(&ctl.k_empty[slot], phase ^ 1u, s_abort, status, FTB_ERR_TIMEOUT_SLOT);
            if (!ok) break;
            if (rank == 0) mbar_arrive_expect_tx(&ctl.k_full[slot], 2 * kSlotBytes);
            const uint32_t bar = map_to_cta(smem_u32(&ctl.k_full[slot]), 0);
            uint8_t* dst = sK + slot * kSlotBytes;
            const int k = u.row_base + (u.blk0 + j) * 128 + static_cast<int>(rank) * 64;
            tma_load_2d_pair(dst, &mapK, bar, 0, k);
            tma_load_2d_pair(dst + kSlotBytes / 2, &mapK, bar, 64, k);
            if (++slot == kSlotsK) {
              slot = 0;
              phase ^= 1u;
            }
          }
        }
        ctl.k_end = {slot, phase};
        ctl.q_end = {w & 1, static_cast<uint32_t>(w >> 1) & 1u};
      }
    } else if (warp == 3) {
      // ------------------------------------------------------------ V tiles
      if (leader) {
        for (int w = 0; ok && unit_of<kMasked>(sh, w, G, cid, u); ++w)
          for (int j = 0; j < u.n; ++j, ++n) {
            const int slot = n & 3;
            if (n >= kSlotsV)
              ok = mbar_wait(&ctl.pv_done[slot], ((n - kSlotsV) >> 2) & 1, s_abort, status, FTB_ERR_TIMEOUT_SLOT);
            if (!ok) break;
            if (rank == 0) mbar_arrive_expect_tx(&ctl.v_full[slot], 2 * kSlotBytes);
            tma_load_2d_pair(sV + slot * kSlotBytes, &mapV, map_to_cta(smem_u32(&ctl.v_full[slot]), 0),
                             static_cast<int>(rank) * 64, u.row_base + (u.blk0 + j) * 128);
          }
        ctl.v_end = {n & 3, static_cast<uint32_t>(n >> 2) & 1u};
      }
    } else if (warp == 1 && rank == 0) {
      // ------------------------------------------------------------ S = Q K^T
      constexpr uint32_t idesc = make_idesc_f16(256, 128, Fmt<T>::kind, 0, 0);
      const uint64_t dQ = make_sdesc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t dK = make_sdesc_sw128(smem_u32(sK), 16, 1024);
      int slot = 0;
      uint32_t phase = 0;
      for (int w = 0; ok && unit_of<kMasked>(sh, w, G, cid, u); ++w) {
        const int b = w & 1;
        ok = mbar_wait_warp(&ctl.q_full[b], (w >> 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_TMA);
        const uint64_t dq = dQ + static_cast<uint64_t>((b * kTileBytes) >> 4);
        for (int j = 0; j < u.n && ok; ++j, ++n) {
          ok = mbar_wait_warp(&ctl.k_full[slot], phase, s_abort, status, FTB_ERR_TIMEOUT_TMA);
          if (n >= 2 && ok) {
            ok = mbar_wait_warp(&ctl.s_free[n & 1], ((n - 2) >> 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI);
            tc_fence_after();
          }
          if (!ok) break;
          const uint64_t dk = dK + static_cast<uint64_t>((slot * kSlotBytes) >> 4);
          if (leader) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              umma_ss_pair(tmem_base + kScores + (n & 1) * 128, dq + (((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4),
                           dk + (((k >> 2) * (kSlotBytes / 2) + (k & 3) * 32) >> 4), idesc, k != 0 ? 1u : 0u);
            umma_commit_pair(&ctl.s_full[n & 1]);
            umma_commit_pair(&ctl.k_empty[slot]);
            if (j == u.n - 1) umma_commit_pair(&ctl.q_empty[b]);
          }
          if (++slot == kSlotsK) {
            slot = 0;
            phase ^= 1u;
          }
        }
      }
    } else if (warp == 2 && rank == 0) {
      // ------------------------------------------------------------ O += P V
      constexpr uint32_t idesc = make_idesc_f16(256, 128, Fmt<T>::kind, 0, 1);
      const uint64_t dV = make_sdesc_sw128(smem_u32(sV), kSlotBytes, 1024);
      for (int w = 0; ok && unit_of<kMasked>(sh, w, G, cid, u); ++w) {
        for (int j = 0; j < u.n && ok; ++j, ++n) {
          const int slot = n & 3;
          ok = mbar_wait_warp(&ctl.v_full[slot], (n >> 2) & 1, s_abort, status, FTB_ERR_TIMEOUT_TMA);
          // The unit before has been read.
          if (j == 0 && w > 0 && ok) ok = mbar_wait_warp(&ctl.o_free, (w - 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI);
          ok = ok && mbar_wait_warp(&ctl.p_full[n & 1], (n >> 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI);
          if (!ok) break;
          tc_fence_after();
          const uint64_t dv = dV + static_cast<uint64_t>((slot * kSlotBytes) >> 4);
          const uint32_t a = tmem_base + kProbs + (n & 1) * 64;
          if (leader) {
            if (!kMasked || (j <= u.last0 && j > u.first1) || (j == 0 && u.first1 == 0)) {
#pragma unroll
              for (int k = 0; k < 8; ++k)
                umma_ts_pair(tmem_base, a + k * 8, dv + k * (2048 >> 4), idesc, (j != 0 || k != 0) ? 1u : 0u);
            } else {
              // One CTA's rows see nothing of this block, or begin with it: the rows of each by themselves.
              if (j <= u.last0)
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  umma_ts_pair_rows(tmem_base, a + k * 8, dv + k * (2048 >> 4), idesc, 0u, 0xffffffffu, (j != 0 || k != 0) ? 1u : 0u);
              if (j >= u.first1)
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  umma_ts_pair_rows(tmem_base, a + k * 8, dv + k * (2048 >> 4), idesc, 0xffffffffu, 0u,
                                    (j != u.first1 || k != 0) ? 1u : 0u);
            }
            umma_commit_pair(&ctl.pv_done[slot]);
            if (j == u.n - 1) umma_commit_pair(&ctl.o_full);
          }
        }
      }
    }
  } else if (warp < 8) {
    regs_dec<80>();
    // ---------------------------------------------------------------- output: a row a thread
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t o_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t free_bar = map_to_cta(smem_u32(&ctl.o_free), 0);
    Unit u;
    bool ok = !dead;
    for (int w = 0; ok && unit_of<kMasked>(sh, w, G, cid, u); ++w) {
      ok = __all_sync(0xffffffffu, mbar_wait(&ctl.l_full[w & 1], (w >> 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI));
      if (!ok) break;
      const float2 a = ctl.stats[w & 1][0][row], b = ctl.stats[w & 1][1][row];
      const float m = fmaxf(a.x, b.x);
      const float inv_l = 1.f / (a.y * exp2_fast(a.x - m) + b.y * exp2_fast(b.x - m));
      ok = __all_sync(0xffffffffu, mbar_wait(&ctl.o_full, w & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA));
      if (!ok) break;
      tc_fence_after();
      uint8_t* stage = sQ + (w & 1) * kTileBytes;  // the unit's queries are dead: every S came before the last O
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t o[32];
        tmem_ld32(o_addr + ch * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 x;
          x.x = Fmt<T>::pack2(__uint_as_float(o[8 * c + 0]) * inv_l, __uint_as_float(o[8 * c + 1]) * inv_l);
          x.y = Fmt<T>::pack2(__uint_as_float(o[8 * c + 2]) * inv_l, __uint_as_float(o[8 * c + 3]) * inv_l);
          x.z = Fmt<T>::pack2(__uint_as_float(o[8 * c + 4]) * inv_l, __uint_as_float(o[8 * c + 5]) * inv_l);
          x.w = Fmt<T>::pack2(__uint_as_float(o[8 * c + 6]) * inv_l, __uint_as_float(o[8 * c + 7]) * inv_l);
          *reinterpret_cast<uint4*>(sw128_chunk_ptr(stage, row, ch * 4 + c)) = x;
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive_peer(free_bar);
        const int r = u.row_base + u.qpair * 256 + static_cast<int>(rank) * 128 + q * 32;
        tma_store_2d(&mapO, stage + q * 4096, 0, r);
        tma_store_2d(&mapO, stage + kHalfBytes + q * 4096, 64, r);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&ctl.q_empty[w & 1]);
      }
    }
  } else {
    regs_inc<192>();
    // ---------------------------------------------------------------- softmax: a row a thread, blocks in turn
    const int g = (warp - 8) >> 2, q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t p_bar = map_to_cta(smem_u32(&ctl.p_full[g]), 0), free_bar = map_to_cta(smem_u32(&ctl.s_free[g]), 0);
    const uint32_t s_addr = lane_addr + kScores + g * 128, p_addr = lane_addr + kProbs + g * 64;
    float* my_m = &ctl.m_x[g][row];
    const float* peer_m = &ctl.m_x[g ^ 1][row];
    const uint64_t scale2 = dup_f32x2(scale_log2);
    constexpr int kTurnAt = kMasked ? 47 : 31;  // the pair of exponentials after which the other group's may begin
    Unit u;
    int base = 0;
    bool ok = !dead, s_there = false;
    for (int w = 0; ok && unit_of<kMasked>(sh, w, G, cid, u); ++w) {
      const int my_first = kMasked && rank != 0 ? u.first1 : 0;
      const int my_last = kMasked && rank == 0 ? u.last0 : u.n - 1;
      float m_own = -FLT_MAX, l = 0.f;
      for (int j = (base ^ g) & 1; j < u.n && ok; j += 2) {
        const int n = base + j;
        ok = __all_sync(0xffffffffu, s_there || mbar_wait(&ctl.s_full[g], (n >> 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA));
        if (!ok) break;
        tc_fence_after();
        const bool seen = !kMasked || (j >= my_first && j <= my_last);
        uint32_t s[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + 32 * c, *reinterpret_cast<uint32_t(*)[32]>(s + 32 * c));
        tmem_ld_wait();
        // The scores are in registers: their columns can take the block after next.
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_peer(free_bar);
        if (kMasked) {
          // Query - first key of the block, of this warp's first row.
          const int from = u.qpair * 256 + static_cast<int>(rank) * 128 + q * 32 - (u.blk0 + j) * 128;
          if (sh.left >= 0 && from + 31 > sh.left) {
            const int lo_col = from + lane - sh.left;
#pragma unroll
            for (int i = 0; i < 128; ++i)
              if (i < lo_col) s[i] = 0xff800000u;  // -inf
          }
          if (from + sh.right < 127) {
            const int hi_col = from + lane + sh.right;
#pragma unroll
            for (int i = 0; i < 128; ++i)
              if (i > hi_col) s[i] = 0xff800000u;
          }
        }
        float mx8[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) mx8[i] = fmaxf(__uint_as_float(s[i]), __uint_as_float(s[8 + i]));
#pragma unroll
        for (int i = 16; i < 128; i += 16) {
#pragma unroll
          for (int k = 0; k < 8; ++k) mx8[k] = fmax3(mx8[k], __uint_as_float(s[i + k]), __uint_as_float(s[i + 8 + k]));
        }
        const float mx = fmaxf(fmax3(mx8[0], mx8[1], mx8[2]), fmaxf(fmax3(mx8[3], mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7])));
        const float m_new = fmaxf(mx * scale_log2, -FLT_MAX);
        // The maximum after the block before, from the other group's thread of this row.
        ok = __all_sync(0xffffffffu, n == 0 || mbar_wait(&ctl.turn[g ^ 1][q], ((n - 1) >> 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI));
        if (!ok) break;
        const float m_prev = j > my_first ? *peer_m : m_new;
        const bool need = seen && (m_new - m_prev) > kRescaleThreshold;
        const float m = need ? m_new : m_prev;
        // (The sign of an exponential is 0: it is there so that the turn cannot be handed on before that exponential.)
        const auto publish = [&](float p) {
          *my_m = __uint_as_float(__float_as_uint(m) ^ (__float_as_uint(p) >> 31));
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.turn[g][q]);
        };
        // P's columns: the product of the block before last has read them.  (Looked at here, waited for where they are written.)
        const uint64_t* read = &ctl.pv_done[(n - 2) & 3];
        const uint32_t read_phase = ((n - 2) >> 2) & 1;
        const bool p_there = n < 2 || mbar_test(read, read_phase);
        auto p_free = [&] {
          ok = __all_sync(0xffffffffu, p_there || mbar_wait(const_cast<uint64_t*>(read), read_phase, s_abort, status, FTB_ERR_TIMEOUT_MMA));
          tc_fence_after();
        };
        if (seen) {
          if (__any_sync(0xffffffffu, m != m_own)) {
            l *= exp2_fast(m_own - m);
            m_own = m;
            if (__any_sync(0xffffffffu, need)) {
              // The accumulator is at rest once the block before has been added.
              ok = __all_sync(0xffffffffu, mbar_wait(&ctl.pv_done[(n - 1) & 3], ((n - 1) >> 2) & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA));
              if (!ok) break;
              tc_fence_after();
              const float alpha = need ? exp2_fast(m_prev - m) : 1.f;
#pragma unroll 1
              for (int ch = 0; ch < 8; ++ch) {
                uint32_t o[16];
                tmem_ld16(lane_addr + ch * 16, o);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                tmem_st16(lane_addr + ch * 16, o);
              }
            }
          }
          uint64_t sum[4] = {0, 0, 0, 0};
          const uint64_t neg_m = dup_f32x2(-m);
          // Keys 64 h .. 64 h + 63: 2^(scale s - m) as 16-bit pairs.
          auto half = [&](int h, uint32_t (&pk)[32]) {
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              const int i = 64 * h + 2 * c;
              const uint64_t e = fma_to_f32x2(pair_f32x2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), scale2, neg_m);
              float p0, p1;
              unpair_f32x2(e, p0, p1);
              p0 = exp2_fast(p0);
              p1 = exp2_fast(p1);
              if (32 * h + c == kTurnAt) publish(p0);
              add_f32x2(sum[c & 3], pair_f32x2(p0, p1));
              pk[c] = Fmt<T>::pack2(p0, p1);
            }
          };
          uint32_t pk[32];
          half(0, pk);
          p_free();
          if (!ok) break;
          tmem_st32(p_addr, pk);
          half(1, pk);
          tmem_st32(p_addr + 32, pk);
          s_there = mbar_test(&ctl.s_full[g], ((n + 2) >> 1) & 1);
          add_f32x2(sum[0], sum[1]);
          add_f32x2(sum[2], sum[3]);
          add_f32x2(sum[0], sum[2]);
          float l0, l1;
          unpair_f32x2(sum[0], l0, l1);
          l += l0 + l1;
          tmem_st_wait();
          tc_fence_before();
        } else {
          publish(0.f);
          p_free();
          if (!ok) break;
          s_there = false;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_peer(p_bar);
      }
      if (!ok) break;
      ctl.stats[w & 1][g][row] = make_float2(m_own, l);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.l_full[w & 1]);
      base += u.n;
    }
  }

  tc_fence_before();
  __syncthreads();
  // Every slot of the rings has been given back, a lane each: ring_drain in ptx.cuh says why.  Here and once for the three rings:
  // 4 x 2304 causal 20.8 us without, 21.0 so, 21.2 with a wait for each ring (code that runs once has to come from L2), 21.1 with
  // producers that wait while the softmax is still at work.
  if (warp == 0) {
    static_assert(kSlotsK == 4 && kSlotsV == 4, "lanes 0..3, 4..7, 8 and 9");
    const int i = lane & 3;
    uint64_t* bar = lane < 4 ? ctl.k_empty + i : lane < 8 ? ctl.pv_done + i : ctl.q_empty + i;
    const RingEnd end = lane < 4 ? ctl.k_end : lane < 8 ? ctl.v_end : ctl.q_end;
    if (lane < 10 && *s_abort == 0) mbar_wait(bar, end.phase ^ (i >= end.at ? 1u : 0u), s_abort, status, FTB_ERR_TIMEOUT_SLOT);
    __syncwarp();
  }
  cluster_sync_all();
  if (warp == 1) {
    if (ctl.abort) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

// (batch, head) entries whose units are dealt out together: 64 MB of K and V.
int flash_pair_group(int S) { return static_cast<int>(std::max<long long>(16, (64ll << 20) / (512ll * S))); }

namespace {
template <typename T, bool kMasked>
int launch(const CUtensorMap& mQ, const CUtensorMap& mK, const CUtensorMap& mV, const CUtensorMap& mO, int n_bh,
           int S, int left, int right, float scale_log2, int* status, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = flash_pair_kernel<T, kMasked>;
  if (!ensure_dynamic_smem(kfn, kSmemBytes, configured)) return FTB_ERR_LAUNCH;
  Shape sh = {S, n_bh, flash_pair_group(S), left, right};
  const long long units = static_cast<long long>(n_bh) * (S / 256);
  const int clusters = static_cast<int>(std::min<long long>(units, current_sm_count() / 2));
  const cudaError_t err = launch_dependent(kfn, dim3(2 * clusters), dim3(kThreads), kSmemBytes, stream, mQ, mK, mV, mO, sh,
                                           scale_log2, status);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}
}  // namespace

int flash_pair_launch(const void* q, const void* k, const void* v, void* o, int64_t rows, int n_bh, int S, int dtype,
                      bool masked, int left, int right, float scale_log2, int* status, cudaStream_t stream) {
  CUtensorMap mQ, mK, mV, mO;
  int rc;
  if ((rc = make_tmap_2d(&mQ, q, dtype, rows, 128, 128, 128, 64))) return rc;
  if ((rc = make_tmap_2d(&mK, k, dtype, rows, 128, 128, 64, 64))) return rc;
  if ((rc = make_tmap_2d(&mV, v, dtype, rows, 128, 128, 128, 64))) return rc;
  if ((rc = make_tmap_2d(&mO, o, dtype, rows, 128, 128, 32, 64))) return rc;
  auto go = [&](auto t) {
    using T = decltype(t);
    return masked ? launch<T, true>(mQ, mK, mV, mO, n_bh, S, left, right, scale_log2, status, stream)
                  : launch<T, false>(mQ, mK, mV, mO, n_bh, S, -1, 0, scale_log2, status, stream);
  };
  return dtype == FTB_F16 ? go(__half()) : go(__nv_bfloat16());
}
}  // namespace ftb
