// Flash attention forward with online softmax for 16-bit inputs on sm_100a, head
// dimension 128: unmasked, and (second instantiation) masked to keys i-left..i+right
// of query i, which covers causal attention (no lower limit, right = 0) and one- and
// two-sided sliding windows.  A masked query tile only walks the key/value blocks its
// rows can see; the blocks the window's edges cross are masked element by element.
//
// Follows the recurrence of attn_func (examples/flash_attention/flash_attention.py:14-44):
// per key/value block, scores S = scale * q k^T, running row maximum m and row sum
// l, output rescaled when the maximum moves.  Two algebraic rearrangements that
// leave the result unchanged up to rounding: the division by l is done once at the
// end instead of per block, and the running maximum is only advanced when it
// moves by more than 2^8 (the stale maximum cancels in the final division), so
// the accumulator in TMEM is rarely touched.  The (m, l) merge itself is the one of
// the reference's online softmax (kaleido/core/device/kernels/online_softmax.h:15-112).
//
// One CTA handles 256 query rows of one (batch, head): two 128-row query tiles
// that ping-pong through the tensor pipe (or, where those CTAs would be too few, 128 rows whose keys
// its two slots share: kHalves below).
//   warp 0        TMA producer: Q tiles, ring of K and V tiles
//   warp 1        MMA issuer: S_t = Q_t K^T and O_t += P_t V, accumulators in TMEM
//   warps 2..9    softmax of query tile 0: two threads per query row, one per half
//                 of the 128 keys of a block (warps 2..5 keys 0..63, warps 6..9 keys 64..127)
//   warps 10..17  softmax of query tile 1, same split
// A row's chain per key/value block (S ready -> maximum -> exponentials -> P written) is
// serial and sits between two dependent MMAs, so its length, not the arithmetic, bounds
// the tensor pipe; splitting the row over two threads halves it.  The two threads of a
// row exchange their partial maximum through shared memory (one float each per block) and
// their partial row sums once at the end.
// P never touches shared memory: the softmax threads write it (16-bit pairs) with
// tcgen05.st over the TMEM columns of the S values they have just read, and the PV
// MMA takes its A operand from TMEM.  V is consumed MN-major straight from its
// row-major tile.  Per query tile the tensor pipe sees S(j), [softmax], PV(j),
// S(j+1), ...; the two query tiles are offset so that one is in its softmax while
// the other one's MMAs run.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "../../include/ftb200.h"
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {

// flash_pair.cu
int flash_pair_group(int S);
int flash_pair_launch(const void* q, const void* k, const void* v, void* o, int64_t rows, int n_bh, int S, int dtype,
                      bool masked, int left, int right, float scale_log2, int* status, cudaStream_t stream);

namespace {

constexpr int kHalfBytes = 128 * 128;  // 128 rows x 64 16-bit columns
constexpr int kTileBytes = 2 * kHalfBytes;
constexpr int kKVSlots = 5, kMostSlots = 6;
constexpr int kThreads = 64 + 512;
constexpr float kRescaleThreshold = 8.0f;
constexpr int kCausalGroup = 16;   // (batch, head) entries whose CTAs are ordered longest first together

// Shared memory, all dynamic so that the 1024-byte alignment of the swizzled tiles costs
// no more than the bytes actually skipped: tiles, then the small control block.
struct Control {
  float xchg[2][2][128];  // [query tile][key half][row]: partial row maximum / row sum
  uint64_t q_full;
  uint64_t kv_full[kMostSlots], kv_empty[kMostSlots];
  uint64_t s_full[2], p_full[2], pv_done[2], o_staged[2];
  uint64_t pair_bar[2][4];  // [query tile][TMEM lane quadrant]: the two warps that share 32 rows
  uint32_t tmem_base;
  int abort, dead;
};
constexpr uint32_t kTilesBytes = (2 + kKVSlots) * kTileBytes;  // Q0, Q1 (reused as output staging), KV ring
static_assert(2 + kKVSlots == 1 + kMostSlots, "one query tile leaves room for one K/V tile more");
constexpr uint32_t kSmemBytes = 232448;                        // everything an SM offers one CTA
static_assert(kTilesBytes + sizeof(Control) + 512 <= kSmemBytes, "shared memory budget");

__device__ __forceinline__ void tmem_ld32p(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// 16-byte chunk `chunk16` (0..15) of row `row` in a 128x128 16-bit tile stored as
// two 64-column halves of 128-byte swizzled rows.
__device__ __forceinline__ uint8_t* sw128_chunk_ptr(uint8_t* tile, int row, int chunk16) {
  return tile + (chunk16 >> 3) * kHalfBytes + row * 128 + (((chunk16 & 7) ^ (row & 7)) << 4);
}

#ifdef FTB_TRACE
__device__ unsigned long long g_fa_trace[2][32][8];
#define FA_STAMP(tt, jj, k) if (blockIdx.x == 300 && lane == 0 && q == 0 && h == 0) g_fa_trace[tt][jj][k] = clock64()
#define FA_STAMP_MMA(tt, jj, k) if (blockIdx.x == 300) g_fa_trace[tt][jj][k] = clock64()
#else
#define FA_STAMP(tt, jj, k)
#define FA_STAMP_MMA(tt, jj, k)
#endif

// kHalves: both query slots of a CTA hold the same 128 rows, slot 0 walks the first half of their key/value blocks and
// slot 1 the second, and the two results are put together in shared memory at the end.  A CTA's time is set by its
// slots' chains, not by the tensor pipe, so that half the blocks are half the time; the price is that a K/V tile
// serves one slot and not two.  For calls whose query tiles leave SMs idle (attention_form below).
// The K/V stream of a walk of n0 and n1 blocks (n1 = n0 or n0 - 1): K(0,0), K(1,0), then for j = 0, 1, ..: V(0,j),
// K(0,j+1), V(1,j), K(1,j+1), without the tiles that do not exist.
struct StreamTile {
  int t, j;
  bool is_v;
};
__device__ __forceinline__ StreamTile stream_tile(int n, int n0, int n1) {
  if (n == 0) return {0, 0, false};
  if (n == 1) return n1 > 0 ? StreamTile{1, 0, false} : StreamTile{0, 0, true};
  const int j = (n - 2) >> 2, r = (n - 2) & 3;
  if (n1 == n0 && j == n0 - 1) return {r, j, true};               // nothing follows the last two values
  if (n1 < n0 && j == n0 - 2 && r == 3) return {0, n0 - 1, true};  // slot 1 has ended: slot 0's last values
  return {r >> 1, (r & 1) != 0 ? j + 1 : j, (r & 1) == 0};
}

template <typename T, bool kMasked, bool kHalves>
__global__ void __launch_bounds__(kThreads, 1)
flash_attn_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                  const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO, int S,
                  int n_bh, int group, int left, int right, float scale_log2, int* __restrict__ status) {
  constexpr int kSlots = kHalves ? kMostSlots : kKVSlots;
  constexpr int kRows = kHalves ? 128 : 256;  // query rows of a CTA
  extern __shared__ uint8_t smem_raw[];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  if (pad + kTilesBytes + sizeof(Control) > kSmemBytes) {
    // The dynamic segment starts later than this layout allows for: report, do not run.
    grid_dependency_wait();
    if (threadIdx.x == 0) atomicCAS(status, 0, FTB_ERR_ALIGN);
    return;
  }
  uint8_t* smem = smem_raw + pad;
  uint8_t* sQ = smem;                                 // one or two tiles
  uint8_t* sKV = sQ + (kRows / 128) * kTileBytes;     // ring
  Control& ctl = *reinterpret_cast<Control*>(smem + kTilesBytes);
  volatile int* s_abort = &ctl.abort;

  const int pairs = S / kRows;
  int bh = blockIdx.x / pairs;
  int qpair = blockIdx.x - bh * pairs;
  if (kMasked) {
    // A pair's run length grows with its position, so CTAs are handed out longest first: within
    // a group of `group` (batch, head) entries all last pairs, then all pairs before them, ...
    // The grid's last CTAs are then the shortest, and the group bounds the K/V set in flight.
    const int per_group = group * pairs;
    const int g = blockIdx.x / per_group;
    const int r = blockIdx.x - g * per_group;
    const int gsize = min(group, n_bh - g * group);
    qpair = pairs - 1 - r / gsize;
    bh = g * group + r % gsize;
  }
  const int row_base = bh * S;            // first row of this (batch, head) in the flattened [B*heads*S, d] view
  const int q_row0 = row_base + qpair * kRows;
  // Key/value blocks this CTA walks.  Masked: query i sees keys i-left .. i+right (left < 0: no
  // lower limit; causal attention is left < 0, right = 0).  A query tile walks from the block of the
  // first key its first row sees to the block of the last key its last row sees.  The CTA walks the
  // union, blocks [blk0, blk0 + n_kv); tile 0 takes part in iterations 0..last0 of that walk, tile 1
  // in first1..n_kv-1 (tile 1 starts and ends at most one block after tile 0).
  int blk0 = 0, n_kv = S / 128, first1 = 0, last0 = n_kv - 1;
  if (kMasked && kHalves) {
    const int r0 = qpair * 128;
    blk0 = left >= 0 ? max(0, r0 - left) >> 7 : 0;
    n_kv = min(S / 128 - 1, (r0 + 127 + right) >> 7) - blk0 + 1;
  } else if (kMasked) {
    const int r0 = qpair * 256;
    const int lo0 = left >= 0 ? max(0, r0 - left) >> 7 : 0;
    const int lo1 = left >= 0 ? max(0, r0 + 128 - left) >> 7 : 0;
    const int hi0 = min(S / 128 - 1, (r0 + 127 + right) >> 7);
    const int hi1 = min(S / 128 - 1, (r0 + 255 + right) >> 7);
    blk0 = lo0;
    n_kv = hi1 - lo0 + 1;
    first1 = lo1 - lo0;
    last0 = hi0 - lo0;
  }
  const int n1 = kHalves ? n_kv / 2 : 0, n0 = n_kv - n1;  // halves: blocks of a slot

  grid_launch_dependents();
  if (threadIdx.x == 0) {
    prefetch_tmap(&mapQ);
    prefetch_tmap(&mapK);
    prefetch_tmap(&mapV);
    prefetch_tmap(&mapO);
    mbar_init(&ctl.q_full, 1);
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&ctl.kv_full[i], 1);
      mbar_init(&ctl.kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl.s_full[i], 1);
      mbar_init(&ctl.p_full[i], 8);
      mbar_init(&ctl.pv_done[i], 1);
      mbar_init(&ctl.o_staged[i], kHalves ? 16 : 8);
      for (int k = 0; k < 4; ++k) mbar_init(&ctl.pair_bar[i][k], 2);
    }
    ctl.abort = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  // K0, V0, K1, V1, ... stream (halves: stream_tile): tile n into ring slot n % kSlots.
  auto load_kv = [&](int n) {
    const int slot = n % kSlots;
    uint8_t* dst = sKV + slot * kTileBytes;
    bool is_v = (n & 1) != 0;
    int block = n >> 1;
    if (kHalves) {
      const StreamTile x = stream_tile(n, n0, n1);
      is_v = x.is_v;
      block = x.j + (x.t != 0 ? n0 : 0);
    }
    const CUtensorMap* m = is_v ? &mapV : &mapK;
    const int r = row_base + (blk0 + block) * 128;
    mbar_arrive_expect_tx(&ctl.kv_full[slot], kTileBytes);
    tma_load_2d(dst, m, &ctl.kv_full[slot], 0, r);
    tma_load_2d(dst + kHalfBytes, m, &ctl.kv_full[slot], 64, r);
  };
  const int n_pre = min(kSlots, 2 * n_kv);
  // Everything above touches no global memory: it runs while the kernel before this one in the stream drains.
  grid_dependency_wait();
  if (threadIdx.x == 0) {
    ctl.dead = *reinterpret_cast<volatile int*>(status) != 0;  // an earlier wait ran out: do nothing
    if (!ctl.dead) {
      // Q and the first pass over the (empty) ring are on their way while TMEM is allocated.
      mbar_arrive_expect_tx(&ctl.q_full, (kRows / 128) * kTileBytes);
      for (int t = 0; t < kRows / 128; ++t) {
        tma_load_2d(sQ + t * kTileBytes, &mapQ, &ctl.q_full, 0, q_row0 + t * 128);
        tma_load_2d(sQ + t * kTileBytes + kHalfBytes, &mapQ, &ctl.q_full, 64, q_row0 + t * 128);
      }
      for (int n = 0; n < n_pre; ++n) load_kv(n);
    }
  }
  if (warp == 1) {
    tmem_alloc(&ctl.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl.tmem_base;
  const bool dead = ctl.dead != 0;
  // TMEM columns: S0 [0,128), S1 [128,256), O0 [256,384), O1 [384,512).  P_t (16-bit pairs)
  // overlays S_t: keys 0..63 in columns [0,32), keys 64..127 in columns [64,96), i.e. each
  // half of the row over the S columns its own thread has read.

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0 && !dead) {
      int slot = 0;
      uint32_t phase = 1;  // the first pass was issued above
      for (int n = n_pre; n < 2 * n_kv; ++n) {
        if (!mbar_wait(&ctl.kv_empty[slot], phase ^ 1u, s_abort, status, FTB_ERR_TIMEOUT_SLOT)) break;
        load_kv(n);
        if (++slot == kSlots) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    // (all lanes walk the loop, one issues: mbar_wait_warp in ptx.cuh says why)
    {
      const bool leader = elect_one();
      constexpr uint32_t idesc_qk = make_idesc_f16(128, 128, Fmt<T>::kind, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_f16(128, 128, Fmt<T>::kind, 0, 1);  // V is MN-major
      // This thread's own instructions sit between every softmax hand-off and the MMAs that follow it:
      // operand descriptors are base descriptors plus byte offsets / 16 (nothing is rebuilt per MMA),
      // and the K/V slots' phases are bits of one register.
      const uint64_t dQ = make_sdesc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t dK = make_sdesc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t dV = make_sdesc_sw128(smem_u32(sKV), kHalfBytes, 1024);
      uint32_t full_bits = 0;  // bit s: parity of the next fill of slot s
      bool ok = !dead && mbar_wait_warp(&ctl.q_full, 0, s_abort, status, FTB_ERR_TIMEOUT_TMA);

      // (No tcgen05 fence after these waits: TMA completes the barriers, and the fence would drain the
      // tensor pipe.)
      auto wait_slot = [&](int n) -> bool {  // n-th tile of the K0, V0, K1, V1, ... stream
        const int slot = n % kSlots;
        if (!mbar_wait_warp(&ctl.kv_full[slot], (full_bits >> slot) & 1u, s_abort, status, FTB_ERR_TIMEOUT_TMA)) return false;
        full_bits ^= 1u << slot;
        return true;
      };
      // S_t = Q_t . K^T, K in ring slot `slot`
      auto issue_s = [&](int t, int slot) {
        const uint64_t dq = dQ + static_cast<uint64_t>(kHalves ? 0 : (t * kTileBytes) >> 4);
        const uint64_t dk = dK + static_cast<uint64_t>((slot * kTileBytes) >> 4);
        if (leader) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t off = ((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4;
            umma_ss(tmem_base + t * 128, dq + off, dk + off, idesc_qk, k != 0 ? 1u : 0u);
          }
          umma_commit(&ctl.s_full[t]);
        }
      };
      // O_t += P_t . V: A = P_t from TMEM (16 keys = 8 packed columns per step; the two
      // key halves start 64 columns apart); B = V, MN-major: 16 keys = two 8-row groups
      // (1024 B apart), the two 64-column halves of d are 16 KB apart.
      auto issue_pv = [&](int t, int slot, bool first) {
        const uint64_t dv = dV + static_cast<uint64_t>((slot * kTileBytes) >> 4);
        if (leader) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + (k >> 2) * 64 + (k & 3) * 8, dv + k * (2048 >> 4),
                    idesc_pv, (!first || k != 0) ? 1u : 0u);
          umma_commit(&ctl.pv_done[t]);
        }
      };

      if constexpr (kHalves) {
        int n = 0, slot = 0;  // of the stream; every tile serves one product
        auto next = [&] {
          if (leader) umma_commit(&ctl.kv_empty[slot]);
          ++n;
          if (++slot == kSlots) slot = 0;
        };
        for (int t = 0; t < 2 && ok; ++t)
          if (t == 0 || n1 > 0) {
            ok = wait_slot(n);
            if (ok) {
              issue_s(t, slot);
              next();
            }
          }
        for (int j = 0; j < n0 && ok; ++j)
          for (int t = 0; t < 2 && ok; ++t) {
            const int mine = t == 0 ? n0 : n1;
            if (j >= mine) continue;
            ok = wait_slot(n) && mbar_wait_warp(&ctl.p_full[t], j & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI);
            if (!ok) break;
            tc_fence_after();
            issue_pv(t, slot, j == 0);
            next();
            if (j + 1 < mine) {
              ok = wait_slot(n);
              if (!ok) break;
              issue_s(t, slot);
              next();
            }
          }
        ok = false;
      }
      if (ok) ok = wait_slot(0);
      if (ok) {
        issue_s(0, 0);
        if (first1 == 0) issue_s(1, 0);
        if (leader) umma_commit(&ctl.kv_empty[0]);
      }
      for (int j = 0; j < n_kv && ok; ++j) {
        const bool more = j + 1 < n_kv;
        if (!wait_slot(2 * j + 1)) break;            // V_j
        if (more && !wait_slot(2 * j + 2)) break;    // K_{j+1}
        for (int t = 0; t < 2 && ok; ++t) {
          const int first = t == 0 ? 0 : first1;
          const int last = t == 0 ? last0 : n_kv - 1;
          if (j >= first && j <= last) {
            // P_t(j) is in TMEM (and the softmax is done with S_t(j)).
            if (!mbar_wait_warp(&ctl.p_full[t], (j - first) & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI)) {
              ok = false;
              break;
            }
            tc_fence_after();
            FA_STAMP_MMA(t, j, 5);
            issue_pv(t, (2 * j + 1) % kSlots, j == first);
          }
          // The tensor pipe runs MMAs in issue order: S_t(j+1) overwrites S_t / P_t only after
          // PV_t(j) has read P_t.
          if (more && j + 1 >= first && j + 1 <= last) issue_s(t, (2 * j + 2) % kSlots);
          FA_STAMP_MMA(t, j, 6);
        }
        if (!ok) break;
        if (leader) umma_commit(&ctl.kv_empty[(2 * j + 1) % kSlots]);
        if (leader && more) umma_commit(&ctl.kv_empty[(2 * j + 2) % kSlots]);
      }
    }
  } else {
    // ----------------------------------- softmax: query tile t, key half h, lane quadrant q
    const int t = (warp - 2) >> 3;
    const int h = ((warp - 2) >> 2) & 1;
    const int q = warp & 3;  // TMEM lane quadrant of this warp
    const int row = q * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t s_addr = lane_addr + t * 128 + h * 64;        // this thread's 64 scores; P over the first 32
    const uint32_t o_addr = lane_addr + 256 + t * 128 + h * 64;  // its 64 output columns (rescale, final pass)
    uint8_t* my_stage = sQ + t * kTileBytes;  // output staging: Q_t is dead once the last S MMA is done
    float* my_x = &ctl.xchg[t][h][row];
    const float* peer_x = &ctl.xchg[t][h ^ 1][row];
    uint64_t* pair = &ctl.pair_bar[t][q];
    float m_used = 0.f, l = 0.f;
    const int j_first = kHalves || t == 0 ? 0 : first1;
    const int j_last = kHalves ? (t == 0 ? n0 : n1) - 1 : (t == 0 ? last0 : n_kv - 1);
    const int n_mine = j_last - j_first + 1;
    bool ok = !dead && n_mine > 0;

    for (int j = j_first; j <= j_last && ok; ++j) {
      const int it = j - j_first;  // this tile's block count so far: the phase of its barriers
      if (!__all_sync(0xffffffffu, mbar_wait(&ctl.s_full[t], it & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA))) {
        ok = false;
        break;
      }
      tc_fence_after();
      FA_STAMP(t, j, 0);
      uint32_t s[64];
      tmem_ld32p(s_addr + 0, s + 0);
      tmem_ld32p(s_addr + 32, s + 32);
      tmem_ld_wait();
      FA_STAMP(t, j, 1);
      if (kMasked) {
        // This thread's 64 keys start at key0; its query is `mine`.  Columns below lo_col are before
        // the window, columns above hi_col after it (for causal attention: after the query).
        const int key0 = (blk0 + j + (kHalves && t != 0 ? n0 : 0)) * 128 + h * 64;
        const int mine = qpair * kRows + (kHalves ? 0 : t * 128) + row;
        const int lo_col = left >= 0 ? mine - left - key0 : 0;
        const int hi_col = mine + right - key0;
        if (__any_sync(0xffffffffu, lo_col > 0)) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (i < lo_col) s[i] = 0xff800000u;  // -inf
        }
        if (__any_sync(0xffffffffu, hi_col < 63)) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (i > hi_col) s[i] = 0xff800000u;
        }
      }

      // Maximum of this half of the row: eight independent chains of three-input maxima.
      float mx8[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) mx8[i] = fmaxf(__uint_as_float(s[i]), __uint_as_float(s[8 + i]));
#pragma unroll
      for (int i = 16; i < 64; i += 16) {
#pragma unroll
        for (int k = 0; k < 8; ++k) mx8[k] = fmax3(mx8[k], __uint_as_float(s[i + k]), __uint_as_float(s[i + 8 + k]));
      }
      float mx = fmaxf(fmax3(mx8[0], mx8[1], mx8[2]), fmaxf(fmax3(mx8[3], mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7])));
      // Row maximum = the larger of the two halves.  The slot written here was last read by the
      // other thread before its arrival on p_full of the previous block, which the MMA warp waited
      // for before it issued the S this block started from: no second buffer is needed.
      *my_x = mx;
      __syncwarp();
      if (lane == 0) mbar_arrive(pair);
      if (!__all_sync(0xffffffffu, mbar_wait(pair, it & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI))) {
        ok = false;
        break;
      }
      mx = fmaxf(mx, *peer_x);
      // A row can have no visible key in a block of its tile's walk: the floor keeps 2^(s - m) at 0
      // there instead of inf - inf, and the first real maximum rescales the (zero) accumulator by 0.
      // (Halves: nor need the keys of one half count beside the other's.)  It is the lowest finite number:
      // scores are products of 16-bit numbers, in bf16 of any size, and none that is finite may fall below it.
      const float m_new = kMasked || kHalves ? fmaxf(mx * scale_log2, -FLT_MAX) : mx * scale_log2;
      if (it == 0) {
        m_used = m_new;
      } else {
        // Both threads of a row see the same m_new and m_used, so both take the same branch.
        const bool need = (m_new - m_used) > kRescaleThreshold;
        if (__any_sync(0xffffffffu, need)) {
          // O_t must be at rest: the PV MMA of the previous block has to be done.
          if (!__all_sync(0xffffffffu,
                          mbar_wait(&ctl.pv_done[t], (it - 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const float alpha = need ? exp2_fast(m_used - m_new) : 1.f;
          if (need) m_used = m_new;
          l *= alpha;
#pragma unroll 1
          for (int ch = 0; ch < 4; ++ch) {
            uint32_t o[16];
            tmem_ld16(o_addr + ch * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st16(o_addr + ch * 16, o);
          }
          tmem_st_wait();
        }
      }

      FA_STAMP(t, j, 2);
      // P_t(j) = 2^(scale*S - m) as 16-bit pairs over the first 32 of this thread's 64 S columns
      // (they are in registers now; the MMA that overwrites them next, S_t(j+1), is issued after
      // PV_t(j)); partial row sum for l.  (Packed fp16 exponentials, two per MUFU op, and a cubic
      // 2^x on the FMA pipes for every other element were both measured and are no faster.)
      {
        float sum8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          uint32_t pk[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const float p0 = exp2_fast(fmaf(__uint_as_float(s[32 * part + 2 * c]), scale_log2, -m_used));
            const float p1 = exp2_fast(fmaf(__uint_as_float(s[32 * part + 2 * c + 1]), scale_log2, -m_used));
            sum8[(2 * c) & 7] += p0;
            sum8[(2 * c + 1) & 7] += p1;
            pk[c] = Fmt<T>::pack2(p0, p1);
          }
          tmem_st16(s_addr + 16 * part, pk);
        }
        l += ((sum8[0] + sum8[1]) + (sum8[2] + sum8[3])) + ((sum8[4] + sum8[5]) + (sum8[6] + sum8[7]));
        FA_STAMP(t, j, 4);
        tmem_st_wait();
      }
      FA_STAMP(t, j, 3);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.p_full[t]);
    }

    // Row sum = the two halves' sums (same exchange, one more phase of the pair barrier).
    if (ok) {
      *my_x = l;
      __syncwarp();
      if (lane == 0) mbar_arrive(pair);
      ok = __all_sync(0xffffffffu, mbar_wait(pair, n_mine & 1, s_abort, status, FTB_ERR_TIMEOUT_EPI));
      if (ok) l += *peer_x;
    }
    if constexpr (kHalves) {
      // Both slots' last PV MMAs are done: the accumulators are at rest, and Q and the K/V ring are dead.  (The MMAs
      // run in the order of their issue, so that the other slot's barrier is one phase behind at most.)
      const bool empty = n_mine <= 0;  // one block in all: slot 1 has none
      const int n_other = t == 0 ? n1 : n0;
      bool fine = empty ? !dead : ok;
      if (fine && !empty) fine = mbar_wait(&ctl.pv_done[t], (n_mine - 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA);
      if (fine && n_other > 0)
        fine = mbar_wait(&ctl.pv_done[t ^ 1], (n_other - 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA);
      fine = __all_sync(0xffffffffu, fine);
      tc_fence_after();
      // A thread finishes 32 of its 64 columns, slot 0 the lower and slot 1 the upper ones, and gives the others to the
      // thread of the other slot: [slot][key half][column / 4][row], 512 bytes a warp's access; then (m, l) of the rows.
      float4* give = reinterpret_cast<float4*>(sKV);
      float2* sums = reinterpret_cast<float2*>(sKV + 2 * kTileBytes);
      if (empty) m_used = -FLT_MAX;
      if (fine) {
        uint32_t o[32];
        tmem_ld32(o_addr + (t ^ 1) * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 8; ++c)
          give[((t * 2 + h) * 8 + c) * 128 + row] =
              empty ? make_float4(0.f, 0.f, 0.f, 0.f)
                    : make_float4(__uint_as_float(o[4 * c]), __uint_as_float(o[4 * c + 1]), __uint_as_float(o[4 * c + 2]),
                                  __uint_as_float(o[4 * c + 3]));
        if (h == 0) sums[t * 128 + row] = make_float2(m_used, l);
      }
      asm volatile("bar.sync 1, 512;" ::: "memory");  // (every softmax warp comes here, whatever its waits said)
      if (fine && *s_abort == 0) {
        const float2 other = sums[(t ^ 1) * 128 + row];
        const float m = fmaxf(m_used, other.x), keep = exp2_fast(m_used - m), take = exp2_fast(other.x - m);
        const float inv_l = 1.f / (l * keep + other.y * take);
        uint32_t o[32];
        tmem_ld32(o_addr + t * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float x[8];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float4 p = give[(((t ^ 1) * 2 + h) * 8 + 2 * c + k) * 128 + row];
            const float q4[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
              x[4 * k + i] = (empty ? q4[i] * take : fmaf(__uint_as_float(o[8 * c + 4 * k + i]), keep, q4[i] * take)) * inv_l;
          }
          uint4 u;
          u.x = Fmt<T>::pack2(x[0], x[1]);
          u.y = Fmt<T>::pack2(x[2], x[3]);
          u.z = Fmt<T>::pack2(x[4], x[5]);
          u.w = Fmt<T>::pack2(x[6], x[7]);
          *reinterpret_cast<uint4*>(sw128_chunk_ptr(sQ, row, h * 8 + t * 4 + c)) = u;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.o_staged[0]);
        if (lane == 0 && t == 0 && h == 0 && q == 2 &&
            mbar_wait(&ctl.o_staged[0], 0, s_abort, status, FTB_ERR_TIMEOUT_EPI)) {
          tma_store_2d(&mapO, sQ, 0, q_row0);
          tma_store_2d(&mapO, sQ + kHalfBytes, 64, q_row0);
          tma_store_commit();
          tma_store_wait_read<0>();
        }
      }
      ok = false;
    }
    // Final: O_t / l -> 16-bit -> staging (the Q tile, dead once the last PV is done) -> TMA store.
    if (ok && __all_sync(0xffffffffu,
                         mbar_wait(&ctl.pv_done[t], (n_mine - 1) & 1, s_abort, status, FTB_ERR_TIMEOUT_MMA))) {
      tc_fence_after();
      const float inv_l = 1.f / l;
#pragma unroll 1
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t o[32];
        tmem_ld32(o_addr + ch * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 u;
          u.x = Fmt<T>::pack2(__uint_as_float(o[8 * c + 0]) * inv_l, __uint_as_float(o[8 * c + 1]) * inv_l);
          u.y = Fmt<T>::pack2(__uint_as_float(o[8 * c + 2]) * inv_l, __uint_as_float(o[8 * c + 3]) * inv_l);
          u.z = Fmt<T>::pack2(__uint_as_float(o[8 * c + 4]) * inv_l, __uint_as_float(o[8 * c + 5]) * inv_l);
          u.w = Fmt<T>::pack2(__uint_as_float(o[8 * c + 6]) * inv_l, __uint_as_float(o[8 * c + 7]) * inv_l);
          *reinterpret_cast<uint4*>(sw128_chunk_ptr(my_stage, row, (h * 2 + ch) * 4 + c)) = u;
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.o_staged[t]);
      // One thread per query tile stores it once all eight warps have staged their part.
      if (lane == 0 && h == 0 && q == 2 &&
          mbar_wait(&ctl.o_staged[t], 0, s_abort, status, FTB_ERR_TIMEOUT_EPI)) {
        tma_store_2d(&mapO, my_stage, 0, q_row0 + t * 128);
        tma_store_2d(&mapO, my_stage + kHalfBytes, 64, q_row0 + t * 128);
        tma_store_commit();
        tma_store_wait_read<0>();  // the staging tile has been read; the writes land before the grid ends
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (ctl.abort) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, bool kMasked, bool kHalves>
int launch(const CUtensorMap& mQ, const CUtensorMap& mK, const CUtensorMap& mV, const CUtensorMap& mO, int n_bh,
           int S, int left, int right, float scale_log2, int* status, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = flash_attn_kernel<T, kMasked, kHalves>;
  if (!ensure_dynamic_smem(kfn, kSmemBytes, configured)) return FTB_ERR_LAUNCH;
  const int group = kCausalGroup;
  const cudaError_t err = launch_dependent(kfn, dim3(n_bh * (S / (kHalves ? 128 : 256))), dim3(kThreads), kSmemBytes, stream,
                                           mQ, mK, mV, mO, S, n_bh, group, left, right, scale_log2, status);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

template <typename T>
int launch(bool masked, bool halves, const CUtensorMap& mQ, const CUtensorMap& mK, const CUtensorMap& mV,
           const CUtensorMap& mO, int n_bh, int S, int left, int right, float scale_log2, int* status, cudaStream_t stream) {
  if (masked)
    return halves ? launch<T, true, true>(mQ, mK, mV, mO, n_bh, S, left, right, scale_log2, status, stream)
                  : launch<T, true, false>(mQ, mK, mV, mO, n_bh, S, left, right, scale_log2, status, stream);
  return halves ? launch<T, false, true>(mQ, mK, mV, mO, n_bh, S, -1, 0, scale_log2, status, stream)
                : launch<T, false, false>(mQ, mK, mV, mO, n_bh, S, -1, 0, scale_log2, status, stream);
}

// The form of a call: 1 = CTAs of 256 query rows, 2 = of 128 rows and half of their blocks a slot, 3 = pairs of CTAs (flash_pair.cu),
// by estimates in us.  A tile of query rows takes a fixed time and one for each block that its longer slot walks, and a pair one for
// each block that an edge of a mask crosses.  Where there are more tiles than places for them (SMs, pairs of SMs), equal ones go
// in whole rounds, unequal ones (masks) half a round of CTAs beyond their mean, pairs, which take theirs in a balanced order, a
// quarter.  Of at most two rounds of pairs the largest sum is taken: behind a window all tiles but the first few are equally long (keys
// i-161..i+745, 12 x 2304, 107 tiles: 25.9 us as form 1, 31.3 as pairs; 6 x 4096, i-723..i+1049: 37.4 as form 2, 41.5 as pairs).
// Forms 1 and 2: halves that are estimated less than a tenth faster keep the 256 rows: between 0.9 and 1 of the estimate the
// time is 0.9 to 1.19 of theirs, below it 0.53 to 0.97.  Form 3 against the one of them: its constants are fitted to 150 calls
// over the sizes and masks of 1 to 16 x 4 to 16 heads and 256 to 4096 keys; the estimates of the other two, made for full and
// causal walks, lie a fifth below what short masked walks take, so that pairs are taken up to 1.2 times their estimate.  Of 820 other
// calls none is more than 5 % slower by that than without pairs, and four more than 2 %; all gain 7.5 % (the best form of each would
// gain 8.2; a factor of 1.1 gives 6.6, one call 5 % slower; of 1.3 7.7, 39 slower by up to 17 %).
// Measured, us, forms 1 / 2 / 3 (* taken): full 16 x 256 8.2 / 7.2* / 7.4, 7 x 512 13.0 / 10.4* / 9.5, 99 x 512 30.4 / 34.3 / 19.3*,
// 40 x 1024 39.5 / 40.1 / 26.8*, 16 x 2048 35.9 / 43.0 / 33.2*, 20 x 2048 68 / 63 / 45*, 4 x 4096 63 / 37 / 33*, 256 x 2048 490 / 574 /
// 438*; causal 15 x 256 8.3 / 6.9* / 8.0, 66 x 512 12.8* / 19.7 / 13.9, 36 x 1024 20.4 / 26.7 / 17.4*, 16 x 2048 37 / 28 / 23.4*, 84 x 3328 266 /
// 294 / 225*; window of 65 77 x 768 24.1* / 29.0 / 28.7, of 1307 42 x 3584 110 / 139 / 111*; keys i-751..i+392 42 x 1024 40 / 39 / 29.5*,
// i-49..i+184 54 x 1024 33.8* / - / 38.7.
int attention_form(bool masked, int n_bh, int S, int left, int right, int sm_count) {
  constexpr double kFixed = 4.5, kBlock = 1.9;
  constexpr double kPairCall = 4.6, kPair = 2.25, kPairBlock = 0.83, kPairMasked = 2.7, kPairMaskedBlock = 0.8, kPairEdge = 0.55, kBelow = 1.2;
  double us[3];
  for (int form = 0; form < 3; ++form) {
    const int rows = form == 1 ? 128 : 256, tiles = S / rows;
    const auto time_of = [&](int i) {
      const int r0 = i * rows;
      const bool begins_late = masked && left >= 0 && r0 > left;
      const int lo = begins_late ? (r0 - left) >> 7 : 0;
      const int hi = masked && r0 + rows - 1 < S - right ? (r0 + rows - 1 + right) >> 7 : S / 128 - 1;
      const int blocks = hi - lo + 1;
      return form == 0   ? kFixed + kBlock * blocks
             : form == 1 ? kFixed + kBlock * ((blocks + 1) / 2)
             : masked    ? kPairMasked + kPairMaskedBlock * blocks + kPairEdge * std::min(blocks, begins_late ? 6 : 2)
                         : kPair + kPairBlock * blocks;
    };
    double total = 0, longest = 0, shortest = 1e30;
    for (int i = 0; i < tiles; ++i) {
      const double t = time_of(i);
      total += t;
      longest = std::max(longest, t);
      shortest = std::min(shortest, t);
    }
    const int places = form == 2 ? sm_count / 2 : sm_count;
    const double waves = static_cast<double>(n_bh) * tiles / places;
    if (waves <= 1) {
      us[form] = longest;
    } else if (masked && form == 2 && waves <= 2) {
      const int group = flash_pair_group(S), units = n_bh * tiles;
      const auto unit_time = [&](int u) {  // as the kernel deals them out
        const int g = u / (group * tiles);
        return time_of(tiles - 1 - (u - g * group * tiles) / std::min(group, n_bh - g * group));
      };
      us[form] = longest;
      for (int u = places; u < units; ++u) us[form] = std::max(us[form], unit_time(u) + unit_time(2 * places - 1 - u));
    } else if (masked) {
      us[form] = std::max(form == 2 ? longest + shortest : longest, (waves + (form == 2 ? 0.25 : 0.5)) * total / tiles);
    } else {
      us[form] = std::ceil(waves) * longest;
    }
  }
  const int single = us[1] < 0.9 * us[0] ? 1 : 0;
  return kPairCall + us[2] < kBelow * us[single] ? 3 : single + 1;
}

}  // namespace
}  // namespace ftb

using namespace ftb;

#ifdef FTB_TRACE
extern "C" int ftb_debug_fa_trace(unsigned long long* out) {
  return cudaMemcpyFromSymbol(out, g_fa_trace, sizeof(unsigned long long) * 2 * 32 * 8) == cudaSuccess ? 0 : 1;
}
#endif

namespace {
int flash_attn_entry(const void* q, const void* k, const void* v, void* o, int B, int heads, int S, int d,
                     float scale, int dtype, bool masked, int left, int right, void* workspace,
                     size_t workspace_bytes, void* stream_, int form = 0) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!q || !k || !v || !o || B <= 0 || heads <= 0 || S <= 0) return FTB_ERR_ARG;
  if (dtype != FTB_F16 && dtype != FTB_BF16) return FTB_ERR_ARG;
  if (d != 128 || S % 256 != 0) return FTB_ERR_ARG;
  if (masked && !(scale > 0.f)) return FTB_ERR_ARG;  // masked scores are -inf times the scale
  if (masked && right < 0) return FTB_ERR_ARG;
  if (left >= S) left = -1;  // every earlier key is inside the window
  if (right > S) right = S;
  const int64_t rows = static_cast<int64_t>(B) * heads * S;
  if (rows > 0x7fffffffLL) return FTB_ERR_ARG;
  if (workspace == nullptr || workspace_bytes < ftb_workspace_bytes()) return FTB_ERR_WORKSPACE;
  int rc = check_device_sm100();
  if (rc) return rc;
  // The status word is sticky: the caller zeroes the workspace once; after a device wait ran out
  // every later call on that workspace is a no-op until the caller clears the word.
  int* status = static_cast<int*>(workspace);

  const int units = B * heads;
  const float scale_log2 = scale * 1.4426950408889634f;
  if (form == 0) form = attention_form(masked, units, S, left, right, current_sm_count());
  if (form == 3) return flash_pair_launch(q, k, v, o, rows, units, S, dtype, masked, left, right, scale_log2, status, stream);
  const bool halves = form == 2;
  CUtensorMap mQ, mK, mV, mO;
  if ((rc = make_tmap_2d(&mQ, q, dtype, rows, d, d, 128, 64))) return rc;
  if ((rc = make_tmap_2d(&mK, k, dtype, rows, d, d, 128, 64))) return rc;
  if ((rc = make_tmap_2d(&mV, v, dtype, rows, d, d, 128, 64))) return rc;
  if ((rc = make_tmap_2d(&mO, o, dtype, rows, d, d, 128, 64))) return rc;
  if (dtype == FTB_F16)
    return launch<__half>(masked, halves, mQ, mK, mV, mO, units, S, left, right, scale_log2, status, stream);
  return launch<__nv_bfloat16>(masked, halves, mQ, mK, mV, mO, units, S, left, right, scale_log2, status, stream);
}
}  // namespace

extern "C" int ftb_flash_attn_fwd(const void* q, const void* k, const void* v, void* o, int B, int heads, int S,
                                  int d, float scale, int dtype, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  return flash_attn_entry(q, k, v, o, B, heads, S, d, scale, dtype, false, -1, 0, workspace, workspace_bytes, stream);
}

extern "C" int ftb_flash_attn_causal_fwd(const void* q, const void* k, const void* v, void* o, int B, int heads,
                                         int S, int d, float scale, int dtype, void* workspace,
                                         size_t workspace_bytes, void* stream) {
  return flash_attn_entry(q, k, v, o, B, heads, S, d, scale, dtype, true, -1, 0, workspace, workspace_bytes, stream);
}

extern "C" int ftb_flash_attn_window_fwd(const void* q, const void* k, const void* v, void* o, int B, int heads,
                                         int S, int d, int window, float scale, int dtype, void* workspace,
                                         size_t workspace_bytes, void* stream) {
  if (window <= 0) return FTB_ERR_ARG;
  return flash_attn_entry(q, k, v, o, B, heads, S, d, scale, dtype, true, window - 1, 0, workspace,
                          workspace_bytes, stream);
}

extern "C" int ftb_flash_attn_local_fwd(const void* q, const void* k, const void* v, void* o, int B, int heads,
                                        int S, int d, int left, int right, float scale, int dtype,
                                        void* workspace, size_t workspace_bytes, void* stream) {
  if (left < 0 || right < 0) return FTB_ERR_ARG;
  return flash_attn_entry(q, k, v, o, B, heads, S, d, scale, dtype, true, left, right, workspace, workspace_bytes,
                          stream);
}

extern "C" int ftb_flash_attn_form(int n_bh, int S, int masked, int left, int right, int sm_count) {
  if (n_bh <= 0 || S <= 0 || S % 256 != 0 || sm_count < 2 || (masked && right < 0)) return 0;
  return attention_form(masked != 0, n_bh, S, left < 0 || left >= S ? -1 : left, std::min(right, S), sm_count);
}

extern "C" int ftb_flash_attn_form_fwd(const void* q, const void* k, const void* v, void* o, int B, int heads, int S,
                                       int d, int masked, int left, int right, int form, float scale, int dtype,
                                       void* workspace, size_t workspace_bytes, void* stream) {
  if (form < 0 || form > 3) return FTB_ERR_ARG;
  return flash_attn_entry(q, k, v, o, B, heads, S, d, scale, dtype, masked != 0, left < 0 ? -1 : left, right, workspace,
                          workspace_bytes, stream, form);
}
