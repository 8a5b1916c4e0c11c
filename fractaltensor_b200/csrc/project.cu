// Vocabulary projection with its softmax, probs = softmax(h . P) per row, without the logits in memory: the product is
// computed twice.  The first pass keeps of every row, pair of CTAs and half of its tiles the pair (maximum, sum of e^(x - maximum))
// of the online softmax (online_softmax.cu), the second multiplies again, puts the pairs of its rows together and writes
// e^(max(x - m, -64)) / d, the same number as the row kernel there.
//
// As a product into fp32 logits and a softmax over them, 2240 words x 10000 x 512 cost 33 + 35 us: 90 MB written, read and
// written again, and tiles of 128 x 128 that take 364 MB through L2 (10.4 TB/s, what bounds the product).  Here a pair of CTAs
// (tcgen05 cta_group::2) owns 256 rows, whose operand stays in shared memory for as long as the rows do (128 KB a CTA at
// H 512), and walks tiles of 256 columns, of which each CTA loads one half: 16 KB a K block and CTA, 92 MB a pass.  Two
// accumulators in tensor memory: the epilogue of a tile runs beside the MMAs of the next.
//
// kUnpacked: P itself, [H, V] with V % 8 == 0, as the MN-major operand of the MMA (64 x 64 boxes); else its transpose [Vp, H]
// (ftb_projection_pack), K-major.
//
//   warp 0        TMA producer (both CTAs)      warp 1        MMA issuer (leader)
//   warps 4..11   epilogue, 128 columns of a tile a warp: a row a thread in the first pass; in the second accumulator fragments, of
//                 which a quad has 8 neighbouring numbers of a row, one sector: they go to memory as they are.  (Through shared memory,
//                 by stores of whole rows or by bulk copies, a tile took the MMAs 6100 cycles and not 4400: they read 64
//                 bytes a cycle there.  2240 x 10000 x 512 58.4 -> 52.3 us, 7000 x 12000 x 256 141 -> 117.)
#include <algorithm>
#include <cfloat>

#include "../../include/ftb200.h"
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {
namespace {

constexpr int BK = 64, kTileN = 256;
constexpr int kThreads = 384, kEpiWarps = 8;
constexpr uint32_t kABlock = 128 * BK * 2, kBBlock = 128 * BK * 2;  // one K block of this CTA's rows, of its half of the columns
constexpr int kMaxKBlocks = 10;   // H <= 640: 160 KB of rows, four K blocks of columns beside them
constexpr int kMaxStages = 8;
// Tiles whose sums are added one behind the other before they are added to those before them: with many rows a pair of CTAs has
// all tiles of a row block, and in one running sum the rounding errors of a row's sum were 1.3 (40 tiles) to 2.2 times (192) those
// of tiles that many pairs share; in eights 0.94 to 1.04 times.
constexpr int kSumTiles = 8;
constexpr uint32_t kSmemBudget = 229376;
constexpr float kClamp = -64.f, kLog2e = 1.4426950408889634f;

struct ProjectArgs {
  int T, V, H, kb, stages;
  int n_tiles, tiles;   // column tiles; all tiles
  float2* stats;        // [2 n_tiles][T]: of a row block, two for each pair of CTAs that has tiles of it
  float* probs;
  long long ld;         // of probs
  int n_store;          // columns of probs that are written: V, or all of a padded row; a multiple of 4, as ld
};

// Numbers e^x are sums and shares of 2^(x log2 e - r), r a whole number at or above the largest exponent: what is rescaled when r
// moves, or when sums with different r meet, is multiplied by a power of two.  (A factor e^(m - m') would be a second
// approximate exponential in the sums beside the one in the numbers they divide, whose mean error then no longer cancels: 5 % more error of the result.)
// From 2^23 on a whole number can lie further from the largest exponent than 2^x has range, and beyond 2.36e38 the exponent
// itself is no fp32 number: there the numbers are shares of 2^(x log2 e - r - rest), with what r lacks.  A row with nothing but
// -inf so far has the lowest finite number as its maximum, and sums of 0.
constexpr float kWhole = 8388608.f, kPlain = kWhole - 256.f;
struct Ref {
  float r, rest;
};
__device__ __forceinline__ float exponent_of(float m) { return ceilf(m * kLog2e); }
__device__ __forceinline__ Ref ref_of(float m) {
  const float r = fminf(fmaxf(exponent_of(m), -FLT_MAX), FLT_MAX);
  return {r, fabsf(r) < kWhole ? 0.f : fmaf(m, kLog2e, -r)};
}
__device__ __forceinline__ float pow2_whole(float n) {  // 2^n, n <= 0 and whole; 0 below 2^-126
  return __int_as_float((max(__float2int_rz(n), -127) + 127) << 23);
}
// Whether sums with references of smaller maxima meet this one's by whole powers of two: their rest is 0, or nothing is left of them.
__device__ __forceinline__ bool plain(const Ref& to) { return fabsf(to.r) < kPlain; }
// What a sum with reference `from` is multiplied by where `to`, of a maximum no smaller, takes its place.
__device__ __forceinline__ float rescale(const Ref& from, const Ref& to) {
  return plain(to) ? pow2_whole(from.r - to.r) : exp2_fast((from.r - to.r) + (from.rest - to.rest));
}

template <typename T, bool kStats, bool kUnpacked>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
project_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const ProjectArgs a,
               int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t a_full[kMaxKBlocks], a_empty;
  __shared__ uint64_t b_full[kMaxStages], b_empty[kMaxStages];
  __shared__ uint64_t acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  uint8_t* sA = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sB = sA + a.kb * kABlock;
  if (threadIdx.x == 0) {
    prefetch_tmap(&mapA);
    prefetch_tmap(&mapB);
    for (int i = 0; i < a.kb; ++i) mbar_init(&a_full[i], 1);
    mbar_init(&a_empty, 1);
    for (int i = 0; i < a.stages; ++i) {
      mbar_init(&b_full[i], 1);
      mbar_init(&b_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 2 * kEpiWarps);
    }
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_s, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  cluster_sync_all();
  // The second pass starts while the first drains: it multiplies what the first has read (all of which was there when the first
  // let it start), and only its epilogue waits for the pairs.
  if (kStats) grid_dependency_wait();
  grid_launch_dependents();

  // This pair's share of the tiles, row block by row block.
  const int G = gridDim.x >> 1, c = blockIdx.x >> 1;
  const int first = static_cast<int>(static_cast<long long>(a.tiles) * c / G);
  const int last = static_cast<int>(static_cast<long long>(a.tiles) * (c + 1) / G);
  // The pair that has a tile.
  auto pair_of = [&](int tile) { return static_cast<int>(((static_cast<long long>(tile) + 1) * G - 1) / a.tiles); };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0, blocks = 0, before = -1;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = first; i < last && ok; ++i) {
        const int mb = i / a.n_tiles, nb = i - mb * a.n_tiles;
        const bool fresh = mb != before;
        if (fresh && blocks > 0) ok = mbar_wait(&a_empty, (blocks - 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_SLOT);
        for (int kb = 0; kb < a.kb && ok; ++kb) {
          if (fresh) {
            if (rank == 0) mbar_arrive_expect_tx(&a_full[kb], 2 * kABlock);
            tma_load_2d_pair(sA + kb * kABlock, &mapA, map_to_cta(smem_u32(&a_full[kb]), 0), kb * BK, mb * 256 + static_cast<int>(rank) * 128);
          }
          ok = mbar_wait(&b_empty[stage], phase ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_SLOT);
          if (!ok) break;
          if (rank == 0) mbar_arrive_expect_tx(&b_full[stage], 2 * kBBlock);
          const uint32_t bar = map_to_cta(smem_u32(&b_full[stage]), 0);
          uint8_t* dst = sB + stage * kBBlock;
          const int col = nb * kTileN + static_cast<int>(rank) * 128;
          if (kUnpacked) {
            tma_load_2d_pair(dst, &mapB, bar, col, kb * BK);
            tma_load_2d_pair(dst + kBBlock / 2, &mapB, bar, col + 64, kb * BK);
          } else {
            tma_load_2d_pair(dst, &mapB, bar, kb * BK, col);
          }
          if (++stage == a.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (fresh) {
          before = mb;
          ++blocks;
        }
      }
      if (ok) ring_drain(b_empty, a.stages, stage, phase, &s_abort, status);
    }
  } else if (warp == 1 && rank == 0) {
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_f16(256, kTileN, Fmt<T>::kind, 0, kUnpacked ? 1 : 0);
    const uint64_t dA = make_sdesc_sw128(smem_u32(sA), 16, 1024);
    const uint64_t dB = make_sdesc_sw128(smem_u32(sB), kUnpacked ? kBBlock / 2 : 16, 1024);
    constexpr uint32_t kStepB = kUnpacked ? 2048 >> 4 : 32 >> 4;  // 16 of K: 16 rows of 128 bytes, or 32 bytes of a row
    int stage = 0, blocks = 0, before = -1;
    uint32_t phase = 0;
    bool ok = true;
    for (int i = first; i < last && ok; ++i) {
      const int mb = i / a.n_tiles, k = i - first, acc = k & 1;
      const bool fresh = mb != before;
      if (fresh) {
        before = mb;
        ++blocks;
      }
      ok = mbar_wait_warp(&acc_empty[acc], ((k >> 1) & 1) ^ 1u, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
      if (!ok) break;
      tc_fence_after();
      for (int kb = 0; kb < a.kb; ++kb) {
        if (fresh) ok = mbar_wait_warp(&a_full[kb], (blocks - 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
        ok = ok && mbar_wait_warp(&b_full[stage], phase, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
        if (!ok) break;
        const uint64_t ad = dA + static_cast<uint64_t>((kb * kABlock) >> 4), bd = dB + static_cast<uint64_t>((stage * kBBlock) >> 4);
        if (leader) {
#pragma unroll
          for (int s = 0; s < 4; ++s)
            umma_ss_pair(tmem_base + acc * kTileN, ad + 2 * s, bd + kStepB * s, idesc, (kb | s) != 0 ? 1u : 0u);
          umma_commit_pair(&b_empty[stage]);
        }
        if (++stage == a.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
      if (leader) {
        umma_commit_pair(&acc_full[acc]);
        if (i + 1 < last && (i + 1) / a.n_tiles != mb) umma_commit_pair(&a_empty);  // the next tile has other rows
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3, half = (warp - 4) >> 2;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * 128;
    const uint32_t empty_bar[2] = {map_to_cta(smem_u32(&acc_empty[0]), 0), map_to_cta(smem_u32(&acc_empty[1]), 0)};
    // First pass: the pairs of this thread's row, of up to kSumTiles tiles and of all before them.  Second: of four rows, lane / 4 and
    // 8, 16, 24 further.
    float top = -FLT_MAX, d = 0.f, all_top = -FLT_MAX, all_d = 0.f;
    int summed = 0;
    float inv_d[4], shift[4], rest[4], least[4];
    int before = -1;
    if (!kStats) grid_dependency_wait();
    for (int i = first; i < last; ++i) {
      const int mb = i / a.n_tiles, nb = i - mb * a.n_tiles, k = i - first, acc = k & 1;
      const int row0 = mb * 256 + static_cast<int>(rank) * 128 + q * 32, row = row0 + lane;
      const int col0 = nb * kTileN + half * 128;
      if (mb != before) {
        before = mb;
        if (kStats) {
          top = all_top = -FLT_MAX;
          d = all_d = 0.f;
          summed = 0;
        } else {
          // the pairs of this thread's row
          const int entries = 2 * (pair_of((mb + 1) * a.n_tiles - 1) - pair_of(mb * a.n_tiles) + 1);
          float m = -FLT_MAX, sum = 0.f;
          if (row < a.T) {
            const float2* p = a.stats + row;
            for (int e0 = 0; e0 < entries; e0 += 16) {
              float2 x[16];
#pragma unroll
              for (int e = 0; e < 16; ++e)
                x[e] = e0 + e < entries ? __ldcg(p + static_cast<long long>(e0 + e) * a.T) : make_float2(-FLT_MAX, 0.f);
              float now = m;
#pragma unroll
              for (int e = 0; e < 16; ++e) now = fmaxf(now, x[e].x);
              const float r = exponent_of(now);
              // (sums by halves: additions one behind the other would cost what the exponentials' own error is)
              float s[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) s[e] = x[e].y * pow2_whole(exponent_of(x[e].x) - r);
#pragma unroll
              for (int w = 8; w > 0; w >>= 1)
#pragma unroll
                for (int e = 0; e < w; ++e) s[e] += s[e + w];
              sum = fmaf(sum, pow2_whole(exponent_of(m) - r), s[0]);
              m = now;
            }
            if (!plain(ref_of(m))) {  // (rare: once more, one pair after the other)
              sum = 0.f;
#pragma unroll 1
              for (int e = 0; e < entries; ++e) {
                const float2 one = __ldcg(p + static_cast<long long>(e) * a.T);
                sum = fmaf(one.y, rescale(ref_of(one.x), ref_of(m)), sum);
              }
            }
          }
          const Ref ref = ref_of(m);
          const float inv = 1.f / sum, low = fmaf(m, kLog2e, -ref.r) - ref.rest + kClamp * kLog2e;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int of = 8 * e + (lane >> 2);
            inv_d[e] = __shfl_sync(0xffffffffu, inv, of);
            shift[e] = __shfl_sync(0xffffffffu, -ref.r, of);
            rest[e] = __shfl_sync(0xffffffffu, ref.rest, of);
            least[e] = __shfl_sync(0xffffffffu, low, of);
          }
        }
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (k >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA))) break;
      tc_fence_after();
      float tile_top = -FLT_MAX, tile_d = 0.f;
      Ref from = ref_of(tile_top);
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        const uint32_t at = lane_addr + acc * kTileN + ch * 32;
        const int c0 = col0 + ch * 32;
        auto release = [&] {  // the accumulator is in registers
          tmem_ld_wait();
          if (ch == 3) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_peer(empty_bar[acc]);
          }
        };
        if (kStats) {
          uint32_t r[32];
          tmem_ld32(at, r);
          release();
          if (c0 >= a.V) continue;
          if (c0 + 32 > a.V) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c0 + j >= a.V) r[j] = 0xff800000u;  // -inf: columns of the padding
          }
          float mx[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) mx[j] = fmaxf(__uint_as_float(r[j]), __uint_as_float(r[4 + j]));
#pragma unroll
          for (int j = 8; j < 32; j += 8)
#pragma unroll
            for (int e = 0; e < 4; ++e) mx[e] = fmax3(mx[e], __uint_as_float(r[j + e]), __uint_as_float(r[j + 4 + e]));
          const float now = fmaxf(fmax3(tile_top, mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          const Ref to = ref_of(now);
          float s[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = exp2_fast(fmaf(__uint_as_float(r[j]), kLog2e, -to.r) - to.rest);
#pragma unroll
          for (int j = 8; j < 32; ++j) s[j & 7] += exp2_fast(fmaf(__uint_as_float(r[j]), kLog2e, -to.r) - to.rest);
          tile_d = fmaf(tile_d, rescale(from, to), ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7])));
          from = to;
          tile_top = now;
        } else {
          uint32_t r[2][2][8];  // 16 rows, 16 columns
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int w = 0; w < 2; ++w) tmem_ld_frag16(at + (static_cast<uint32_t>(16 * h) << 16) + 16 * w, r[h][w]);
          release();
          if (c0 >= a.n_store) continue;
          const int c = c0 + 2 * (lane & 3);
          const int c_out = c0 + 2 * (lane & 2) + 8 * (lane & 1);  // first of the four that this lane stores of every 16
          float* out = a.probs + static_cast<long long>(row0 + (lane >> 2)) * a.ld + c_out;
          const bool whole = c0 + 32 <= a.V;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            auto prob = [&](uint32_t x) {
              return exp2_fast(fmaxf(fmaf(__uint_as_float(x), kLog2e, shift[e]) - rest[e], least[e])) * inv_d[e];
            };
            float2 v[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {  // eight columns each
              const uint32_t* x = &r[e >> 1][g >> 1][4 * (g & 1) + 2 * (e & 1)];
              v[g] = make_float2(prob(x[0]), prob(x[1]));
              if (!whole) {
                if (c + 8 * g >= a.V) v[g].x = 0.f;
                if (c + 8 * g + 1 >= a.V) v[g].y = 0.f;
              }
            }
            // Neighbours trade two groups of columns, so that a thread has four numbers of one and a quad 16 of a row: even lanes
            // keep groups 0 and 2, odd ones 1 and 3.
            const bool odd = (lane & 1) != 0;
            float* to = out + static_cast<long long>(8 * e) * a.ld;
#pragma unroll
            for (int g = 0; g < 4; g += 2) {
              const float2 give = odd ? v[g] : v[g + 1], keep = odd ? v[g + 1] : v[g];
              const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, give.x, 1), __shfl_xor_sync(0xffffffffu, give.y, 1));
              if (row0 + 8 * e + (lane >> 2) < a.T && c_out + 8 * g < a.n_store)
                __stcs(reinterpret_cast<float4*>(to + 8 * g),
                       odd ? make_float4(got.x, got.y, keep.x, keep.y) : make_float4(keep.x, keep.y, got.x, got.y));
            }
          }
        }
      }
      if (kStats) {  // (tile by tile: chunk by chunk through all of them adds up more roundings)
        const bool stored = i + 1 == last || (i + 1) / a.n_tiles != mb;
        const float now = fmaxf(top, tile_top);
        const Ref to = ref_of(now);
        d = fmaf(d, rescale(ref_of(top), to), tile_d * rescale(from, to));
        top = now;
        if (++summed == kSumTiles || stored) {
          const float both = fmaxf(all_top, top);
          const Ref to_both = ref_of(both);
          all_d = fmaf(all_d, rescale(ref_of(all_top), to_both), d * rescale(to, to_both));
          all_top = both;
          top = -FLT_MAX;
          d = 0.f;
          summed = 0;
        }
        if (stored && row < a.T)
          __stcg(a.stats + static_cast<long long>(2 * (c - pair_of(mb * a.n_tiles)) + half) * a.T + row, make_float2(all_top, all_d));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    if (s_abort) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <typename T, bool kStats, bool kUnpacked>
int launch(const CUtensorMap& mA, const CUtensorMap& mB, const ProjectArgs& a, uint32_t smem, int* status, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  auto kfn = project_kernel<T, kStats, kUnpacked>;
  if (!ensure_dynamic_smem(kfn, kSmemBudget + 1024, configured)) return FTB_ERR_LAUNCH;
  const int pairs = std::min(a.tiles, current_sm_count() / 2);
  const cudaError_t err = launch_dependent(kfn, dim3(2 * pairs), dim3(kThreads), smem, stream, mA, mB, a, status);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

template <typename T, bool kUnpacked>
int launch_passes(const CUtensorMap& mA, const CUtensorMap& mB, const ProjectArgs& a, uint32_t smem, int* status, cudaStream_t stream) {
  const int rc = launch<T, true, kUnpacked>(mA, mB, a, smem, status, stream);
  return rc ? rc : launch<T, false, kUnpacked>(mA, mB, a, smem, status, stream);
}

}  // namespace

// What the kernel takes, and where it is the faster form: rows that begin on 16 bytes (for others the stores go singly, and
// cost what the logits did), and behind a packed operand only where the logits are many.  us, product and softmax / twice:
// unpacked (packing counted), H 512, V 10000: 40 words 21.3 / 22.8, 300 29.0 / 29.1, 2240 79.2 / 49.5, 5000 169 / 97.2; V 2000: 300 22.6 /
// 20.6, 5000 48.6 / 39.3.  Packed, by millions of probabilities (90 calls of 64 to 20000 words, V 200 to 40000, H 64 to 640; twice as a
// share of product and softmax): up to 4 1.15, 4 to 8 1.07, 8 to 12 0.98, 12 to 16 0.84, 16 to 30 0.80, 30 to 60 0.65, more 0.63.
// V 10004: 1000 words 37.0 / 35.8, 1600 50.5 / 43.4, 2240 71.4 / 52.9, 5000 160 / 110.  The line stays at 16 million, not at 12: this
// kernel's probabilities are 1.04 to 1.15 times as far from 64 bits.  (Rows on 16 bytes and not on 32, V % 8 == 4: runs of 64 bytes
// touch three sectors.  Through whole rows in shared memory the largest were up to 7 % faster, 17732 x 5884 x 512 214 / 229, and all
// others slower, 0.957 of it on average; runs of 128 bytes by another exchange 4 to 15 % slower, but for the largest.)
bool project_twice_supported(int dtype, long long T, int V, int H, bool unpacked) {
  return (dtype == FTB_F16 || dtype == FTB_BF16) && H % BK == 0 && H <= kMaxKBlocks * BK &&
         (unpacked ? V % 8 == 0 : V % 4 == 0 && T * V >= 16000000);
}

size_t project_twice_scratch(long long T, int V) { return static_cast<size_t>(T) * ((V + kTileN - 1) / kTileN) * 2 * sizeof(float2); }

// h [T, H]; P [H, V] (unpacked) or its transpose [Vp, H]; probs: rows `ld` apart, V columns and zeros up to ld.
int launch_project_twice(int dtype, const void* h, const void* P, bool unpacked, float* probs, long long ld, int T, int V,
                         int Vp, int H, void* scratch, int* status, cudaStream_t stream) {
  ProjectArgs a;
  a.T = T; a.V = V; a.H = H; a.kb = H / BK;
  a.n_tiles = (V + kTileN - 1) / kTileN;
  const long long tiles = static_cast<long long>((T + 255) / 256) * a.n_tiles;
  if (tiles > 0x7fffffffLL) return FTB_ERR_ARG;
  a.tiles = static_cast<int>(tiles);
  a.stages = std::min<int>(kMaxStages, (kSmemBudget - a.kb * kABlock) / kBBlock);
  a.stats = static_cast<float2*>(scratch);
  a.probs = probs;
  a.ld = ld;
  a.n_store = static_cast<int>(ld);
  const uint32_t smem = a.kb * kABlock + a.stages * kBBlock + 1024;
  CUtensorMap mA, mB;
  int rc;
  if ((rc = make_tmap_2d(&mA, h, dtype, T, H, H, 128, BK))) return rc;
  if ((rc = unpacked ? make_tmap_2d(&mB, P, dtype, H, V, V, BK, 64) : make_tmap_2d(&mB, P, dtype, Vp, H, H, 128, BK))) return rc;
  if (dtype == FTB_F16)
    return unpacked ? launch_passes<__half, true>(mA, mB, a, smem, status, stream)
                    : launch_passes<__half, false>(mA, mB, a, smem, status, stream);
  return unpacked ? launch_passes<__nv_bfloat16, true>(mA, mB, a, smem, status, stream)
                  : launch_passes<__nv_bfloat16, false>(mA, mB, a, smem, status, stream);
}

}  // namespace ftb
