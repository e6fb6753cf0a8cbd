// The plain GEMM for few rows:  D[M,N] = A[M,K] * W^T  with M <= 256 (decoded tokens, short chunks), where the time is
// that of streaming W once and of getting started.
//
// Operands are swapped: the 128 rows of a UMMA are 128 rows of W (output columns), its N dimension is the tokens
// (16 .. 256). A tile of the fused kernel would spend 16 KB of shared memory and of copies per K block on a
// 128-row box of A that is mostly padding; here 16 of every 18 KB (16 tokens) are weights, so more of them are in
// flight: the kernel is bound by HBM, and what counts is bytes in flight and no idle SM.
//
// One output tile per cluster of S CTAs, which cut K into S parts. Each CTA leaves its accumulator in its own shared
// memory; after a cluster barrier CTA r sums columns (tokens) r, r + 1, ... of all S, in rank order, through
// distributed shared memory. Nothing is exchanged through global memory: no scratch, no counters, any number of
// launches side by side. Up to 64 tokens a CTA takes half of an SM's shared memory, so that one CTA's prologue and
// reduction overlap another's loads.
#pragma once
#include "gemm_kernel.cuh"

namespace fluxb {

constexpr int kSkinnyThreads = 192;  // warp 0 TMA, warp 1 UMMA + TMEM, warps 2-5 accumulator read-out and output
constexpr int kSkinnyMaxM = 256;
constexpr int kSkinnyMaxSplit = 8;

struct SkinnyParams {
  CUtensorMap tmap_w;  // weights: 128 rows x 128 bytes of K, or [K, N] as 64-column boxes
  CUtensorMap tmap_x;  // tokens: BN rows x 128 bytes of K
  int M, N, num_kb, split;
  int w_kn;     // weight stored [K, N]
  int out_bf16, bias_mode;
  uint16_t* out;
  const uint16_t* bias;
  const float* scale_a;
  const float* scale_b;
  long long ldo, ldbias;
  float alpha;
  unsigned long long timeout_ns;
  int* status;
  unsigned long long* trace;
  int trace_ctas;  // CTAs the timeline has room for: one per SM, of the up to two that this kernel runs there
};

template <int BN>
struct SkinnyLayout {
  static constexpr int kStages = BN == 16 ? 6 : BN == 32 ? 5 : BN == 64 ? 4 : BN == 128 ? 6 : 4;
  static constexpr int kABytes = kBM * kRowBytes;
  static constexpr int kBBytes = BN * kRowBytes;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // the accumulator read-out [BN][128] fp32 reuses the stages
  static_assert(kStages * kStageBytes >= BN * kBM * 4, "the read-out must fit into the stages");
  static constexpr int kBarOffset = kStages * kStageBytes;
  static constexpr int kNumBars = 2 * kStages + 2;  // full / empty per stage, accumulator complete, "UMMAs retired" (abort path)
  static constexpr int kMiscOffset = kBarOffset + kNumBars * 8;
  static constexpr int kTotal = kMiscOffset + 32 + 1024;  // + slack for 1024-byte alignment
  static constexpr uint32_t kTmemCols = BN < 32 ? 32 : BN;
};

// Output columns n, n + 1 of every second token of this CTA's share of the tokens: the sum of the SPLIT parts in rank
// order, then the options. `t` = 0..127; UN tokens' loads are in flight together (one token at a time, each paid the
// latency of distributed shared memory: 128 tokens in four parts took 6 us). A part that gave up leaves garbage
// here; its status word says so.
template <int KIND, int SPLIT, int UN>
__device__ __forceinline__ void skinny_reduce(const SkinnyParams& p, uint32_t smem_base, int n0, int part, int t) {
  const int n = n0 + (t & 63) * 2;
  const int per = (p.M + SPLIT - 1) / SPLIT;
  const int m_end = imin(p.M, (part + 1) * per);
  if (n >= p.N) return;
  uint32_t peer[SPLIT];
#pragma unroll
  for (int s = 0; s < SPLIT; ++s) peer[s] = mapa_u32(smem_base + (t & 63) * 8, s);
  const float sb0 = p.scale_b != nullptr ? p.scale_b[n] : 1.0f, sb1 = p.scale_b != nullptr ? p.scale_b[n + 1] : 1.0f;
  constexpr bool acc_int = KIND == 2;
  const bool has_bias = p.bias_mode != kBiasNone;
  const long long bias_pitch = p.bias_mode == kBiasFull ? p.ldbias : 0;
#pragma unroll 1
  for (int m0 = part * per + (t >> 6); m0 < m_end; m0 += 2 * UN) {
    uint2 v[UN][SPLIT];
    float row_scale[UN];
    uint32_t b2[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int m = m0 + 2 * u < m_end ? m0 + 2 * u : m0;
#pragma unroll
      for (int s = 0; s < SPLIT; ++s) v[u][s] = ld_shared_cluster_v2(peer[s] + static_cast<uint32_t>(m) * (kBM * 4));
      row_scale[u] = p.scale_a != nullptr ? p.alpha * __ldg(p.scale_a + m) : p.alpha;
      b2[u] = has_bias ? __ldg(reinterpret_cast<const uint32_t*>(p.bias + m * bias_pitch + n)) : 0u;
    }
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int m = m0 + 2 * u;
      if (m >= m_end) break;
      float x0, x1;
      if (acc_int) {
        uint32_t i0 = v[u][0].x, i1 = v[u][0].y;
#pragma unroll
        for (int s = 1; s < SPLIT; ++s) {
          i0 += v[u][s].x;
          i1 += v[u][s].y;
        }
        // the reference's order, bit-identical to its golden path (see the fused kernel's epilogue)
        x0 = (row_scale[u] * sb0) * __int2float_rn(static_cast<int>(i0));
        x1 = (row_scale[u] * sb1) * __int2float_rn(static_cast<int>(i1));
        if (has_bias) {
          x0 = p.out_bf16 ? __bfloat162float(__float2bfloat16_rn(x0)) : __half2float(__float2half_rn(x0));
          x1 = p.out_bf16 ? __bfloat162float(__float2bfloat16_rn(x1)) : __half2float(__float2half_rn(x1));
        }
      } else {
        x0 = __uint_as_float(v[u][0].x);
        x1 = __uint_as_float(v[u][0].y);
#pragma unroll
        for (int s = 1; s < SPLIT; ++s) {
          x0 += __uint_as_float(v[u][s].x);
          x1 += __uint_as_float(v[u][s].y);
        }
        x0 = (x0 * row_scale[u]) * sb0;
        x1 = (x1 * row_scale[u]) * sb1;
      }
      if (has_bias) {
        const float2 f = p.out_bf16 ? make_float2(__uint_as_float(b2[u] << 16), __uint_as_float(b2[u] & 0xFFFF0000u))
                                    : __half22float2(*reinterpret_cast<const __half2*>(&b2[u]));
        x0 += f.x;
        x1 += f.y;
      }
      *reinterpret_cast<uint32_t*>(p.out + m * p.ldo + n) = p.out_bf16 ? pack_bf16(x0, x1) : pack_f16(x0, x1);
    }
  }
}

template <int BN, int KIND>
__global__ void __launch_bounds__(kSkinnyThreads)
skinny_gemm_kernel(const __grid_constant__ SkinnyParams p, const uint32_t idesc) {
  using L = SkinnyLayout<BN>;
  constexpr int STAGES = L::kStages;
  constexpr int BKE = kRowBytes / (KIND == 0 ? 2 : 1);  // K elements per stage
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_base + L::kBarOffset;
  const uint32_t bar_done = bar_base + 8u * (2 * STAGES), bar_retired = bar_done + 8u;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + L::kMiscOffset);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOffset + 8);
  const AbortWord ab{s_abort, 0u};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.split;
  const int part = static_cast<int>(cluster_ctarank());
  const int n0 = static_cast<int>(blockIdx.x) / split * kBM;
  const int kb0 = static_cast<int>(static_cast<long long>(part) * p.num_kb / split);
  const int kb1 = static_cast<int>(static_cast<long long>(part + 1) * p.num_kb / split);
  const int nkb = kb1 - kb0;
  unsigned long long* tr = p.trace != nullptr && static_cast<int>(blockIdx.x) < p.trace_ctas ? p.trace + static_cast<size_t>(blockIdx.x) * 8 : nullptr;

  auto load = [&](int i, int stage) {  // K block i of this part
    const uint32_t bar = bar_base + 8u * stage, dst = smem_base + stage * L::kStageBytes;
    const int k = (kb0 + i) * BKE;
    mbar_arrive_expect_tx(bar, L::kStageBytes);
    if (p.w_kn) {
      tma_load_2d(dst, &p.tmap_w, bar, n0, k);
      tma_load_2d(dst + BKE * kRowBytes, &p.tmap_w, bar, n0 + 64, k);
    } else {
      tma_load_2d(dst, &p.tmap_w, bar, k, n0);
    }
    tma_load_2d(dst + L::kABytes, &p.tmap_x, bar, k, 0);
  };

  if (warp == 0 && elect_one()) {
    *s_abort = 0;
    for (int s = 0; s < 2 * STAGES + 2; ++s) mbar_init(bar_base + 8u * s, 1);
    mbar_init_fence();
    if (tr != nullptr) tr[0] = globaltimer_ns();
    // nothing before this line touches global memory; everything after it follows from these loads
    pdl_wait();
    // the first loads need no one else: they fly while tensor memory is allocated and the CTA meets
    for (int i = 0; i < STAGES && i < nkb; ++i) load(i, i);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), L::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    if (elect_one()) {
      pdl_trigger();
      int stage = 0;
      uint32_t phase = 0;
      int i = STAGES;
      for (; i < nkb; ++i) {
        if (!mbar_wait(bar_base + 8u * (STAGES + stage), phase, ab, kStatusTimeoutSmemEmpty, p.timeout_ns)) break;
        load(i, stage);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (*s_abort != 0) {
        // give the copies in flight their time to land (1 ms per stage at most): none may outlive the CTA
        const AbortWord none{nullptr, 0u};
        for (int s = 0; s < STAGES && s < nkb; ++s)
          mbar_wait(bar_base + 8u * s, static_cast<uint32_t>(((i - 1 - s) / STAGES) & 1), none, 0, 1000000ull);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t a_desc0 = p.w_kn ? make_mnmajor_sw128_desc(smem_base, BKE * kRowBytes) : make_kmajor_sw128_desc(smem_base);
      const uint64_t b_desc0 = make_kmajor_sw128_desc(smem_base + L::kABytes);
      const uint32_t a_step = p.w_kn ? 128u : 2u;  // 16 elements of K: 32 bytes of a K-major operand, 16 rows of an MN-major one
      pdl_wait();  // (the budget of the waits below starts when the kernel before this one has ended)
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait(bar_base + 8u * stage, phase, ab, kStatusTimeoutSmemFull, p.timeout_ns)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (tr != nullptr && i == 0) tr[1] = globaltimer_ns();
        const uint64_t off = static_cast<uint32_t>(stage) * (L::kStageBytes >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t a = a_desc0 + off + a_step * k, b = b_desc0 + off + 2u * k;
          const uint32_t accum = (i > 0 || k > 0) ? 1u : 0u;
          if (KIND == 0) umma_f16(tmem_base, a, b, idesc, accum);
          else if (KIND == 2) umma_i8(tmem_base, a, b, idesc, accum);
          else umma_f8(tmem_base, a, b, idesc, accum);
        }
        umma_commit(bar_base + 8u * (STAGES + stage));
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) umma_commit(bar_done);
      if (tr != nullptr) {
        tr[2] = globaltimer_ns();
        tr[7] = 1;
      }
      if (*s_abort != 0) {  // UMMAs in flight still read shared memory and write tensor memory
        umma_commit(bar_retired);
        mbar_wait(bar_retired, 0, AbortWord{nullptr, 0u}, 0, 2000000ull);
      }
    }
  } else {
    // this CTA's accumulator, tokens x 128 output columns, into its shared memory (all loads have landed and all
    // UMMAs have retired by then, so the stages are free)
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    pdl_wait();  // (as above)
    if (__all_sync(0xffffffffu, mbar_wait(bar_done, 0, ab, kStatusTimeoutTmemFull, p.timeout_ns))) {
      tc_fence_after();
      const uint32_t t0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
      if constexpr (BN == 16) {
        uint32_t r[16];
        tmem_ld_32x16(t0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<uint32_t*>(smem + (j * kBM + row) * 4) = r[j];
      } else {
#pragma unroll 1
        for (int c = 0; c < BN / 32 && c * 32 < p.M; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(t0 + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) *reinterpret_cast<uint32_t*>(smem + ((c * 32 + j) * kBM + row) * 4) = r[j];
        }
      }
      tc_fence_before();
    }
  }
  cluster_sync_all();
  if (warp >= 2 && *s_abort == 0) {
    const int t = static_cast<int>(threadIdx.x) - 64;
    if (split == 1) skinny_reduce<KIND, 1, 8>(p, smem_base, n0, part, t);
    else if (split == 2) skinny_reduce<KIND, 2, 8>(p, smem_base, n0, part, t);
    else if (split == 4) skinny_reduce<KIND, 4, 8>(p, smem_base, n0, part, t);
    else skinny_reduce<KIND, 8, 4>(p, smem_base, n0, part, t);
    if (tr != nullptr && t == 0) tr[3] = tr[4] = globaltimer_ns();
  }
  cluster_sync_all();  // no CTA leaves while another still reads its shared memory
  if (*s_abort != 0 && threadIdx.x == 0) {
    *reinterpret_cast<volatile int*>(p.status) = *s_abort;
    __threadfence_system();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::kTmemCols);
  }
}

}  // namespace fluxb
