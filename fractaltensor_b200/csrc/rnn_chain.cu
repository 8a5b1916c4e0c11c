// A tanh recurrence over time as one launch: h_t = tanh(pre_t + h_{t-1} U + b), 16-bit states, H <= 512.
//
// The input half of the cell, pre_t = x_t W, does not depend on the recurrence: it is one matrix
// product over all steps (fp32, csrc/cell_gemm.cu) made beforehand.  What is left is a chain of Ls
// dependent [N x H].[H x H] products, bound by latency alone: as one launch per step it cost 7.4 us a
// step (launch, weights from L2, epilogue, store) for 0.7 us of MMAs.  Here
//   * one thread-block cluster owns 16 sequences for the whole scan; clusters never wait for one
//     another, so any number of them may be resident.  16 is the smallest N of an M = 128 MMA, and
//     an MMA costs the same ~45 cycles at N = 16 as at N = 64: the smallest slice has the shortest
//     epilogue and hand-off;
//   * CTA r of the cluster owns units 128 r .. 128 r + 127; their rows of U^T stay in tensor memory as
//     the A operand (H / 2 columns);
//   * h_t goes from the epilogue's registers straight into the next step's B operand in every CTA
//     of the cluster: a thread holds 8 sequences of one unit, which is one 16-byte row of the
//     MN-major core matrix, and sends it with st.async, its bytes counted on the receiver's mbarrier
//     of that source CTA.  No staging tile, no barrier between the epilogue warps.
// The two state slots need no release: a CTA's step-t output is complete only after it has received
// every peer's step t-1 output, that is after every peer has multiplied what slot t & 1 held before.
// The MMA warp keeps all its lanes in the loop: with one lane alone in it the descriptors were
// divergent values, moved to uniform registers before every MMA (67 cycles an MMA, 2.54 us a step).
// Measured (H 512, 64 sequences, bf16): 1.5 us a step; 50 steps as launches of the cell kernel 370 us,
// here 74 us and 7 us for the product of the input halves.
//
// Program: src_enc_outs = map(scan(cell)) of examples/rnn_attention/rnn_attention.py:40-48, 86-110.
#include "../../include/ftb200.h"
#include "ptx.cuh"
#include "tmap.h"

namespace ftb {
namespace {

constexpr int kNB = 16;                     // sequences of a cluster
constexpr int kMaxCtas = 4;                 // CTAs of a cluster: H / 128, rounded up
constexpr int kEpiWarps = 4 * (kNB / 8);    // a warp: one TMEM lane quadrant, 8 sequences
constexpr int kFirstEpi = 4;                // warp 0 issues the MMAs
constexpr int kThreads = 32 * (kFirstEpi + kEpiWarps);
constexpr uint32_t kAccCols = 32;           // columns between the two accumulators
constexpr uint32_t kCoreK = 128 * (kNB / 8);  // bytes of 8 units x 16 sequences
// More than half of an SM's shared memory, so that no two CTAs share an SM: each takes all of its
// tensor memory, and two clusters holding one SM each of a pair would wait for each other.
constexpr uint32_t kSmemBytes = 120 * 1024;

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
               "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

struct ChainArgs {
  const float* pre;    // [steps, N, H]
  const void* Wp;      // packed rows of ldw elements; the recurrent half starts at element k0
  const float* bias;   // [H] or nullptr
  const void* before;  // [N, H] state before the first step, or nullptr (zeros)
  void* out;           // [steps, N, H]
  int* status;
  int ldw, k0, steps, N, H, CL;
};

template <typename T>
__global__ void __launch_bounds__(kThreads, 1) rnn_chain_kernel(const ChainArgs a) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[2][kMaxCtas];  // slot, source CTA: that source's units of the state have arrived
  __shared__ uint64_t first_full;         // the state before the first step is in slot 1
  __shared__ uint64_t w_full;             // U is in tensor memory
  __shared__ uint64_t acc_full[2];
  __shared__ uint64_t acc_ready[2];       // the step's input half is in the accumulator
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = a.CL > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int slice = blockIdx.x / a.CL;
  uint8_t* slots = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  const uint32_t slot_bytes = static_cast<uint32_t>(a.H / 8) * kCoreK;
  int* status = a.status;
  // Without a state before the first step that step multiplies nothing; accumulators 1 and 0 then begin with
  // steps 1 and 2.  Which use of its accumulator a step is (parity waits):
  const bool from_zero = a.before == nullptr;
  auto use_of = [&](int i) { return from_zero ? ((i - 1 - ((i + 1) & 1)) >> 1) : (i >> 1); };

  if (threadIdx.x == 0) {
    const int unit_warps = min(128, a.H - 128 * rank) / 32 * (kNB / 8);
    for (int s = 0; s < 2; ++s) {
      for (int r = 0; r < kMaxCtas; ++r) mbar_init(&full[s][r], 1);
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_ready[s], unit_warps);
    }
    mbar_init(&first_full, kEpiWarps);
    mbar_init(&w_full, kEpiWarps);
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync_all();  // peers store into this CTA's shared memory: not before its barriers are set up
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tmem_w = tmem_base + 2 * kAccCols;
  grid_launch_dependents();
  grid_dependency_wait();

  if (warp == 0) {
    // All lanes walk the loop, so that addresses and descriptors are warp-uniform values (the MMA takes
    // them from uniform registers); one elected lane issues.
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_f16(128, kNB, Fmt<T>::kind, 0, 1);
    // MN-major, no swizzle: core matrices of 8 units x 8 sequences (128 B), the second 8 sequences
    // 128 B behind the first, the next 8 units kCoreK behind.
    uint64_t bdesc0 = 1ull << 46;
    bdesc0 |= static_cast<uint64_t>((smem_u32(slots) & 0x3FFFFu) >> 4);
    bdesc0 |= static_cast<uint64_t>(kCoreK >> 4) << 16;
    bdesc0 |= static_cast<uint64_t>(128u >> 4) << 32;
    bool ok = mbar_wait_warp(&w_full, 0, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
    tc_fence_after();
    for (int i = from_zero ? 1 : 0; i < a.steps; ++i) {
      const int slot = (i + 1) & 1;  // of the step before
      const uint32_t d_tmem = tmem_base + (i & 1) * kAccCols;
      ok = ok && mbar_wait(&acc_ready[i & 1], use_of(i) & 1, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
      if (i == 0) {
        ok = ok && mbar_wait(&first_full, 0, &s_abort, status, FTB_ERR_TIMEOUT_EPI);
      } else if (lane < a.CL) {
        mbar_arrive_expect_tx(&full[slot][lane], static_cast<uint32_t>(min(128, a.H - 128 * lane)) * kNB * 2);
      }
      // All sources at once, a lane each: a wait and a fence for each of them, in turn, cost 360 cycles a source where the
      // MMAs behind them take 90 (H 512: a step 2690 cycles, so 2350).
      if (i > 0) {
        if (lane < a.CL)
          ok = ok && mbar_wait_cluster(&full[slot][lane], ((i - 1) >> 1) & 1, &s_abort, status, FTB_ERR_TIMEOUT_TMA);
        __syncwarp();
        fence_proxy_async_smem();  // the state was stored by threads, the MMA reads it by the async proxy
      }
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
#pragma unroll
      for (int r = 0; r < kMaxCtas; ++r) {
        if (r >= a.CL) break;
        const uint64_t bd = bdesc0 + static_cast<uint64_t>((slot * slot_bytes + r * 16 * kCoreK) >> 4);
        const uint32_t aw = tmem_w + r * 64;
        if (128 * r + 128 <= a.H) {
          if (leader) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              umma_ts(d_tmem, aw + 8 * j, bd + j * ((2 * kCoreK) >> 4), idesc, 1u);
          }
        } else if (leader) {  // the last CTA of an H that is not a multiple of 128 has 64 units
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_ts(d_tmem, aw + 8 * j, bd + j * ((2 * kCoreK) >> 4), idesc, 1u);
        }
      }
      if (leader) umma_commit(&acc_full[i & 1]);
    }
  } else if (warp >= kFirstEpi) {
    const int q = warp & 3, half = (warp - kFirstEpi) >> 2;
    const int u_loc = q * 32 + lane;
    const int u = rank * 128 + u_loc;
    const bool has_unit = u < a.H;
    const int n0 = slice * kNB + half * 8;
    const int n_mine = min(8, a.N - n0);  // sequences of this thread that exist (may be <= 0)
    {
      // U^T -> tensor memory: one row per lane, two 16-bit values per column; the two warps of a
      // quadrant alternate blocks of 64
      const uint4* wrow = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.Wp) +
                                                         static_cast<size_t>(has_unit ? u : 0) * a.ldw + a.k0);
      for (int kb = half; kb < a.H / 64; kb += kEpiWarps / 4) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 x4 = has_unit ? __ldg(wrow + kb * 8 + i) : make_uint4(0, 0, 0, 0);
          v[4 * i + 0] = x4.x; v[4 * i + 1] = x4.y; v[4 * i + 2] = x4.z; v[4 * i + 3] = x4.w;
        }
        tmem_st32(tmem_w + (static_cast<uint32_t>(q * 32) << 16) + kb * 32, v);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_full);
    }
    if (a.before != nullptr) {
      // the whole state before the first step, in the layout the epilogues send
      const T* h = reinterpret_cast<const T*>(a.before);
      for (int e = threadIdx.x - 32 * kFirstEpi; e < a.H * kNB; e += 32 * kEpiWarps) {
        const int k = e % a.H, n = e / a.H;
        T x = T(0.f);
        if (slice * kNB + n < a.N) x = h[static_cast<size_t>(slice * kNB + n) * a.H + k];
        *reinterpret_cast<T*>(slots + slot_bytes + (k >> 3) * kCoreK + (n >> 3) * 128 + (k & 7) * 16 + (n & 7) * 2) = x;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&first_full);
    }
    const float bias = has_unit && a.bias != nullptr ? __ldg(a.bias + u) : 0.f;
    const size_t step_elems = static_cast<size_t>(a.N) * a.H;
    const float* pre = a.pre + static_cast<size_t>(n0) * a.H + u;
    T* out = reinterpret_cast<T*>(a.out) + static_cast<size_t>(n0) * a.H + u;
    const uint32_t my_chunk = smem_u32(slots) + (u >> 3) * kCoreK + half * 128 + (u & 7) * 16;
    // Where the states go: every CTA of the cluster, its own first (slot 0; slot 1 behind it).
    uint32_t to[kMaxCtas], to_bar[kMaxCtas];
#pragma unroll
    for (int k = 0; k < kMaxCtas; ++k) {
      const int r = rank + k < a.CL ? rank + k : rank + k - a.CL;
      to[k] = to_bar[k] = 0;
      if (k < a.CL) {
        to[k] = map_to_cta(my_chunk, r);
        to_bar[k] = map_to_cta(smem_u32(&full[0][rank]), r);
      }
    }
    float p[8];
    auto load_pre = [&](int i) {
#pragma unroll
      for (int n = 0; n < 8; ++n)
        p[n] = has_unit && n < n_mine ? __ldg(pre + i * step_elems + static_cast<size_t>(n) * a.H) : 0.f;
    };
    // Warps without units (the upper half of the last CTA when H is an odd multiple of 64) are done: nobody waits
    // for anything of theirs, so that nothing would keep acc_full, which is followed by parity, from running two
    // phases ahead of them.  A warp with units is at most one behind: the next MMAs need what it sends.
    const int steps = has_unit ? a.steps : 0;
    const uint32_t my_acc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * 8;
    // The input half of step i, which p holds, into the accumulator that the step's MMAs add to.
    auto begin_acc = [&](int i) {
      tmem_st8(my_acc + (i & 1) * kAccCols, p);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_ready[i & 1]);
    };
    float v[8];
    if (steps > 0) {
      load_pre(0);
      if (from_zero) {
#pragma unroll
        for (int n = 0; n < 8; ++n) v[n] = p[n];
      } else {
        begin_acc(0);
      }
      if (steps > 1) {
        load_pre(1);
        begin_acc(1);
      }
      if (steps > 2) load_pre(2);
    }
    for (int i = 0; i < steps; ++i) {
      if (i > 0 || !from_zero) {
        const bool ok = mbar_wait(&acc_full[i & 1], use_of(i) & 1, &s_abort, status, FTB_ERR_TIMEOUT_MMA);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        uint32_t r[8];
        tmem_ld8(my_acc + (i & 1) * kAccCols, r);
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int n = 0; n < 8; ++n) v[n] = __uint_as_float(r[n]);
      }
      uint32_t h[4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
        h[n] = Fmt<T>::pack2(tanh_fast(v[2 * n] + bias), tanh_fast(v[2 * n + 1] + bias));
      if (i + 1 < steps) {
#pragma unroll
        for (int k = 0; k < kMaxCtas; ++k)
          if (k < a.CL)
            st_async16(to[k] + (i & 1) * slot_bytes, to_bar[k] + (i & 1) * static_cast<uint32_t>(sizeof(full[0])), h);
      }
      if (i + 2 < steps) {
        begin_acc(i + 2);  // (the accumulator just read)
        if (i + 3 < steps) load_pre(i + 3);
      }
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const uint16_t bits = static_cast<uint16_t>(h[n >> 1] >> (16 * (n & 1)));
        if (n < n_mine) *reinterpret_cast<uint16_t*>(out + i * step_elems + static_cast<size_t>(n) * a.H) = bits;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // nobody leaves while a peer may still store into its shared memory
  if (warp == 0) {
    if (s_abort) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T>
int launch(const ChainArgs& a, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  if (!ensure_dynamic_smem(rnn_chain_kernel<T>, kSmemBytes, configured)) return FTB_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((a.N + kNB - 1) / kNB) * a.CL);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = a.CL;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, rnn_chain_kernel<T>, a);
  count_launch();
  if (err != cudaSuccess) cudaGetLastError();
  return err == cudaSuccess ? FTB_OK : FTB_ERR_LAUNCH;
}

}  // namespace

bool rnn_chain_supported(int dtype, int H) {
  return (dtype == FTB_F16 || dtype == FTB_BF16) && H % 64 == 0 && H <= 128 * kMaxCtas;
}

// out[i] = tanh(pre[i] + state U + bias) for i < steps; Wp: [H, ldw], the recurrent half of a row at k0.
int launch_rnn_chain(int dtype, const float* pre, const void* Wp, int ldw, int k0, const float* bias,
                     const void* before, void* out, int steps, int N, int H, int* status, cudaStream_t stream) {
  const ChainArgs a = {pre, Wp, bias, before, out, status, ldw, k0, steps, N, H, (H + 127) / 128};
  return dtype == FTB_F16 ? launch<__half>(a, stream) : launch<__nv_bfloat16>(a, stream);
}

}  // namespace ftb
