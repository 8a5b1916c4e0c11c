// Vocabulary projection with its softmax, probs = softmax(h . P) per row, without the logits in memory: the product is
// computed twice.  The first pass keeps of every row and 128 columns the pair (maximum, sum of e^(x - maximum)) of the
// online softmax (online_softmax.cu), the second multiplies again, puts the pairs of its rows together and writes
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
//   warps 4..11   epilogue: a row a thread, 128 columns of a tile a warp
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
constexpr int kMaxKBlocks = 10;   // H <= 640: 160 KB of rows, three K blocks of columns beside them
constexpr int kMaxStages = 8;
constexpr uint32_t kStaging = kEpiWarps * 2048;  // 16 rows x 32 numbers a warp
constexpr uint32_t kSmemBudget = 229376;
constexpr float kClamp = -64.f, kLog2e = 1.4426950408889634f;

struct ProjectArgs {
  int T, V, H, kb, stages;
  int n_tiles, tiles;   // column tiles; all tiles
  float2* stats;        // [2 n_tiles][T]
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
  uint8_t* s_out = sB + a.stages * kBBlock;
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
    uint8_t* s_row = s_out + (warp - 4) * 2048;
    const uint32_t empty_bar[2] = {map_to_cta(smem_u32(&acc_empty[0]), 0), map_to_cta(smem_u32(&acc_empty[1]), 0)};
    float m = 0.f, inv_d = 0.f, shift = 0.f, rest = 0.f, least = 0.f;  // second pass: of this thread's row
    int before = -1;
    if (!kStats) grid_dependency_wait();
    for (int i = first; i < last; ++i) {
      const int mb = i / a.n_tiles, nb = i - mb * a.n_tiles, k = i - first, acc = k & 1;
      const int row0 = mb * 256 + static_cast<int>(rank) * 128 + q * 32, row = row0 + lane;
      const int col0 = nb * kTileN + half * 128;
      if (!kStats && mb != before) {
        before = mb;
        m = -FLT_MAX;
        float d = 0.f;
        if (row < a.T) {
          const float2* p = a.stats + row;
          for (int e0 = 0; e0 < 2 * a.n_tiles; e0 += 16) {
            float2 x[16];
#pragma unroll
            for (int e = 0; e < 16; ++e)
              x[e] = e0 + e < 2 * a.n_tiles ? __ldcg(p + static_cast<long long>(e0 + e) * a.T) : make_float2(-FLT_MAX, 0.f);
            float top = m;
#pragma unroll
            for (int e = 0; e < 16; ++e) top = fmaxf(top, x[e].x);
            const float r = exponent_of(top);
            // (sums by halves: 80 additions one behind the other would cost what the exponentials' own error is)
            float s[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) s[e] = x[e].y * pow2_whole(exponent_of(x[e].x) - r);
#pragma unroll
            for (int w = 8; w > 0; w >>= 1)
#pragma unroll
              for (int e = 0; e < w; ++e) s[e] += s[e + w];
            d = fmaf(d, pow2_whole(exponent_of(m) - r), s[0]);
            m = top;
          }
          if (!plain(ref_of(m))) {  // (rare: once more, one pair after the other)
            d = 0.f;
#pragma unroll 1
            for (int e = 0; e < 2 * a.n_tiles; ++e) {
              const float2 one = __ldcg(p + static_cast<long long>(e) * a.T);
              d = fmaf(one.y, rescale(ref_of(one.x), ref_of(m)), d);
            }
          }
        }
        inv_d = 1.f / d;
        const Ref ref = ref_of(m);
        shift = -ref.r;
        rest = ref.rest;
        least = fmaf(m, kLog2e, shift) - rest + kClamp * kLog2e;
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (k >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA))) break;
      tc_fence_after();
      float top = -FLT_MAX, d = 0.f;
      Ref from = ref_of(top);
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t r[32];
        tmem_ld32(lane_addr + acc * kTileN + ch * 32, r);
        tmem_ld_wait();
        if (ch == 3) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_peer(empty_bar[acc]);
        }
        const int c0 = col0 + ch * 32;
        if (kStats) {
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
          const float now = fmaxf(fmax3(top, mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          const Ref to = ref_of(now);
          float s[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = exp2_fast(fmaf(__uint_as_float(r[j]), kLog2e, -to.r) - to.rest);
#pragma unroll
          for (int j = 8; j < 32; ++j) s[j & 7] += exp2_fast(fmaf(__uint_as_float(r[j]), kLog2e, -to.r) - to.rest);
          d = fmaf(d, rescale(from, to), ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7])));
          from = to;
          top = now;
        } else {
          if (c0 >= a.n_store) continue;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            r[j] = c0 + j < a.V ? __float_as_uint(exp2_fast(fmaxf(fmaf(__uint_as_float(r[j]), kLog2e, shift) - rest, least)) * inv_d) : 0u;
          // A lane has a row of 32 numbers; a store covers whole rows: through shared memory, 16 rows at a time, 16-byte pieces
          // exchanged within a row so that neither side meets a bank twice.
#pragma unroll
          for (int part = 0; part < 32; part += 16) {
            if ((lane & 16) == part) {
#pragma unroll
              for (int g = 0; g < 8; ++g)
                *reinterpret_cast<uint4*>(s_row + (lane & 15) * 128 + ((g ^ (lane & 7)) << 4)) =
                    make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
            }
            __syncwarp();
            const int piece = lane & 7;
#pragma unroll
            for (int g = 0; g < 16; g += 4) {
              const int rr = g + (lane >> 3);
              const float4 v = *reinterpret_cast<const float4*>(s_row + rr * 128 + ((piece ^ (rr & 7)) << 4));
              if (row0 + part + rr < a.T && c0 + 4 * piece < a.n_store)
                __stcs(reinterpret_cast<float4*>(a.probs + (row0 + part + rr) * a.ld + c0 + 4 * piece), v);
            }
            __syncwarp();
          }
        }
      }
      if (kStats && row < a.T) __stcg(a.stats + static_cast<long long>(2 * nb + half) * a.T + row, make_float2(top, d));
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
// unpacked, H 512, V 10000: 40 words 22.5 / 21.0, 300 30.6 / 28.8, 2240 79.9 / 55.1, 5000 170 / 103; V 2000: 300 20.5 / 18.6, 5000 43.1 / 39.0;
// packed: V 2004, 300 words 23.6 / 26.0, 5000 45.1 / 46.2; V 10004, 2240 words 83.3 / 67.7; V 10001, 2240 words 90.3 / 91.5.
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
  a.stages = std::min<int>(kMaxStages, (kSmemBudget - kStaging - a.kb * kABlock) / kBBlock);
  a.stats = static_cast<float2*>(scratch);
  a.probs = probs;
  a.ld = ld;
  a.n_store = static_cast<int>(ld);
  const uint32_t smem = a.kb * kABlock + a.stages * kBBlock + kStaging + 1024;
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
