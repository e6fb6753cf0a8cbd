// The plain GEMM  D[M,N] = A[M,K] * B[N,K]^T (+ scales, bias) with a 16-bit output: the fused kernel's tiles and pipeline
// without its collectives. Short launches are bound by what comes before the first copy and after the last UMMA, and in
// the fused kernel both are long: a block of a few thousand clocks of first-time instruction and constant fetches (the
// roles branch around the collectives' code, parameters are spread over 2.3 KB), tile coordinates by division, and an
// epilogue of four warps. Here the schedule comes from the host with multipliers for its divisions, the scalars share
// two cache lines, and eight warps (two per tensor memory quadrant, alternating 64-column boxes) drain a tile.
// Clocks of 1000 x 3584 x 4096 (fused / here): entry to first copy 5000 / 2000, accumulator complete to end
// 8400 / 5300.
//
// Tiles: one CTA per 128 x BN, or a CTA pair per 256 x BN. BN = 512 is two UMMA column blocks that share A's stages and
// fill tensor memory with one accumulator: a quarter less operand traffic per flop than 256 x 256 (384 instead of 512
// rows of 128 bytes per SM for the same work) against an epilogue that no longer overlaps the next tile's main loop.
#pragma once
#include "gemm_kernel.cuh"

namespace fluxb {

constexpr int kPlainThreads = 320;  // warp 0 TMA, warp 1 UMMA + TMEM, warps 2-9 epilogue

// Division by a number known on the host: q = umulhi(n, mul) >> shr for n < 2^31 (Granlund and Montgomery: with
// p = 31 + ceil(log2 d), mul = ceil(2^p / d) is below 2^32 and exact for 31-bit n).
struct FastDiv {
  uint32_t d, mul, shr;
  void set(uint32_t div) {
    d = div;
    uint32_t l = 0;
    while ((1ull << l) < div) ++l;
    mul = div == 1 ? 0u : static_cast<uint32_t>(((1ull << (31 + l)) + div - 1) / div);
    shr = div == 1 ? 0u : l - 1;
  }
  __host__ __device__ __forceinline__ int quot(int n) const {
#ifdef __CUDA_ARCH__
    return d == 1 ? n : static_cast<int>(__umulhi(static_cast<uint32_t>(n), mul) >> shr);
#else
    return d == 1 ? n : static_cast<int>(((static_cast<uint64_t>(n) * mul) >> 32) >> shr);
#endif
  }
};

struct PlainParams {
  // schedule: worker w takes tiles w, w + workers, ... of `full_waves` waves, then part w % split of tail tile w / split
  int M, N, num_kb;
  int n_tiles, m_tiles, group_m;
  int full_waves, tail_tiles, split;
  FastDiv band_div, gm_div, last_div, split_div;  // group_m * n_tiles, group_m, the last band's height, split
  int b_kn, out_bf16, bias_mode;
  float alpha;
  const float* scale_a;
  const float* scale_b;
  uint16_t* out;
  const uint16_t* bias;
  float* splitk_scratch;  // as in GemmParams, null if nothing is cut; a part's slot is [quadrant][step][piece][lane]
  int* splitk_cnt;
  int* splitk_done;
  unsigned long long* trace;
  int* status;
  unsigned long long timeout_ns;
  CUtensorMap tmap_a, tmap_b, tmap_out;
};

__host__ __device__ __forceinline__ void plain_tile(const PlainParams& p, int t, int& m_idx, int& n_idx) {
  const int band = p.band_div.quot(t);
  const int r = t - band * static_cast<int>(p.band_div.d);
  const FastDiv& h = (band + 1) * p.group_m <= p.m_tiles ? p.gm_div : p.last_div;
  n_idx = h.quot(r);
  m_idx = band * p.group_m + r - n_idx * static_cast<int>(h.d);
}

template <int BN, bool CTA2>
struct PlainLayout {
  static constexpr int kStages = CTA2 ? (BN == 512 ? 4 : BN >= 192 ? 6 : 8) : (BN >= 192 ? 4 : BN == 128 ? 6 : 8);
  static constexpr int kABytes = kBM * kRowBytes;
  static constexpr int kBRows = CTA2 ? BN / 2 : BN;
  static constexpr int kStageBytes = kABytes + kBRows * kRowBytes;
  static constexpr int kEpiOffset = kStages * kStageBytes;  // 4 KB (32 rows x 64 columns) per epilogue warp
  static constexpr int kAccs = BN == 512 ? 1 : 2;
  static constexpr int kNumBars = 2 * kStages + 5;
  static constexpr int kBarOffset = kEpiOffset + 8 * 4096;
  static constexpr int kMiscOffset = kBarOffset + kNumBars * 8;
  static constexpr int kTotal = kMiscOffset + 32 + 1024;
  static constexpr uint32_t kTmemCols = kAccs * BN <= 128 ? 128 : kAccs * BN <= 256 ? 256 : 512;
};

template <int BN, int KIND, bool CTA2>
__global__ void __launch_bounds__(kPlainThreads, 1)
plain_gemm_kernel(const __grid_constant__ PlainParams p, const uint32_t idesc) {
  using L = PlainLayout<BN, CTA2>;
  constexpr int STAGES = L::kStages, ACCS = L::kAccs;
  constexpr int BKE = kRowBytes / (KIND == 0 ? 2 : 1);
  constexpr int TILE_M = CTA2 ? 2 * kBM : kBM;
  constexpr int NB = BN == 512 ? 2 : 1;      // UMMA column blocks
  constexpr int kBlkRows = L::kBRows / NB;   // rows of B of one block in this CTA
  static_assert(L::kTotal <= 232448, "shared memory budget exceeded");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_base + L::kBarOffset;
  auto bar_full = [&](int s) { return bar_base + 8u * s; };
  auto bar_empty = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto bar_tfull = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto bar_tempty = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t bar_retired = bar_base + 8u * (2 * STAGES + 4);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + L::kMiscOffset);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOffset + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = CTA2 ? static_cast<int>(cluster_ctarank()) : 0;
  const bool leader = half == 0;
  const int worker = CTA2 ? static_cast<int>(blockIdx.x) >> 1 : static_cast<int>(blockIdx.x);
  const int workers = CTA2 ? static_cast<int>(gridDim.x) >> 1 : static_cast<int>(gridDim.x);
  const AbortWord ab{s_abort, CTA2 ? mapa_u32(smem_u32(const_cast<int*>(s_abort)), static_cast<uint32_t>(half ^ 1)) : 0u};
  const uint64_t budget = p.timeout_ns;
  unsigned long long* tr = p.trace != nullptr ? p.trace + static_cast<size_t>(blockIdx.x) * 8 : nullptr;

  if (warp == 0 && elect_one()) {
    if (tr != nullptr) {
      tr[0] = globaltimer_ns();
      tr[5] = tr[6] = 0;
    }
    *s_abort = 0;
    for (int s = 0; s < 2 * STAGES; ++s) mbar_init(bar_base + 8u * s, 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_tfull(a), 1);
      mbar_init(bar_tempty(a), CTA2 ? 16 : 8);  // one arrival per epilogue warp (of both CTAs)
    }
    mbar_init(bar_retired, 1);
    mbar_init_fence();
    tma_prefetch_desc(&p.tmap_a);
    tma_prefetch_desc(&p.tmap_b);
  }
  if (warp == 1) {
    if (CTA2) {
      tmem_alloc_2cta(smem_u32(tmem_holder), L::kTmemCols);
      tmem_relinquish_2cta();
    } else {
      tmem_alloc(smem_u32(tmem_holder), L::kTmemCols);
      tmem_relinquish();
    }
  }
  // work item i of this worker: tile and K blocks [kb0, kb1)
  const int split = p.split, full_waves = p.full_waves;
  auto get_item = [&](int i, int& t, int& kb0, int& kb1, int& part) -> bool {
    part = 0;
    kb0 = 0;
    kb1 = p.num_kb;
    t = worker + i * workers;
    if (i < full_waves) return true;
    if (i > full_waves) return false;
    if (split <= 1) return worker < p.tail_tiles;
    const int tt = p.split_div.quot(worker);
    if (tt >= p.tail_tiles) return false;
    part = worker - tt * split;
    t = full_waves * workers + tt;
    kb0 = p.split_div.quot(part * p.num_kb);
    kb1 = p.split_div.quot((part + 1) * p.num_kb);
    return true;
  };
  tc_fence_before();
  if (CTA2) cluster_sync_all(); else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t full0 = CTA2 ? mapa_u32(bar_full(0), 0) : bar_full(0);
      const bool arms = !CTA2 || leader;
      const bool b_kn = p.b_kn != 0;
      int t, kb0, kb1, part;
      for (int wi = 0; ok && get_item(wi, t, kb0, kb1, part); ++wi) {
        int m_idx, n_idx;
        plain_tile(p, t, m_idx, n_idx);
        const int arow = m_idx * TILE_M + half * kBM;
        const int brow = n_idx * BN + half * kBlkRows;
        if (wi == 0) {
          pdl_wait();  // the first touch of global memory; everything else follows from these loads
          pdl_trigger();
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(bar_empty(stage), phase ^ 1u, ab, kStatusTimeoutSmemEmpty, budget)) {
            ok = false;
            break;
          }
          if (arms) mbar_arrive_expect_tx(bar_full(stage), CTA2 ? 2 * L::kStageBytes : L::kStageBytes);
          const uint32_t fb = full0 + 8u * stage;
          const uint32_t sa = smem_base + stage * L::kStageBytes, sb = sa + L::kABytes;
          const int k = kb * BKE;
          auto load = [&](uint32_t dst, const void* map, int x, int y) {
            if (CTA2) tma_load_2d_2cta(dst, map, fb, x, y); else tma_load_2d(dst, map, fb, x, y);
          };
          load(sa, &p.tmap_a, k, arow);
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            if (b_kn) {
#pragma unroll
              for (int j = 0; j < kBlkRows / 64; ++j)
                load(sb + b * (kBlkRows * kRowBytes) + j * (BKE * kRowBytes), &p.tmap_b, brow + b * 256 + j * 64, k);
            } else {
              load(sb + b * (kBlkRows * kRowBytes), &p.tmap_b, k, brow + b * 256);
            }
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (*s_abort != 0 && leader) {
        // every armed stage still has copies in flight or has been filled: wait (1 ms each at most)
        const AbortWord none{nullptr, 0u};
        for (int s2 = 0; s2 < STAGES; ++s2) mbar_wait(bar_full(s2), s2 < stage ? phase : (phase ^ 1u), none, 0, 1000000ull);
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------- UMMA
    if (leader && elect_one()) {
      const bool b_kn = p.b_kn != 0;
      const uint64_t a_desc0 = make_kmajor_sw128_desc(smem_base);
      const uint64_t b_desc0 = b_kn ? make_mnmajor_sw128_desc(smem_base + L::kABytes, BKE * kRowBytes)
                                    : make_kmajor_sw128_desc(smem_base + L::kABytes);
      const uint32_t b_step = b_kn ? 128u : 2u;
      pdl_wait();  // (the budget of the waits below starts when the kernel before this one has ended)
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      int t, kb0, kb1, part;
      for (; ok && get_item(it, t, kb0, kb1, part); ++it) {
        const int acc = ACCS == 2 ? it & 1 : 0;
        const uint32_t acc_phase = (ACCS == 2 ? it >> 1 : it) & 1;
        if (!mbar_wait<CTA2>(bar_tempty(acc), acc_phase ^ 1u, ab, kStatusTimeoutTmemEmpty, budget)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(bar_full(stage), phase, ab, kStatusTimeoutSmemFull, budget)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (tr != nullptr && it == 0 && kb == kb0) tr[1] = globaltimer_ns();
          const uint32_t off = static_cast<uint32_t>(stage) * (L::kStageBytes >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t accum = (kb > kb0 || k > 0) ? 1u : 0u;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              const uint64_t ad = a_desc0 + off + 2u * k;
              const uint64_t bd = b_desc0 + off + static_cast<uint32_t>(b * ((kBlkRows * kRowBytes) >> 4)) + b_step * k;
              const uint32_t d = d_tmem + b * 256;
              if (CTA2) {
                if (KIND == 0) umma_f16_2cta(d, ad, bd, idesc, accum);
                else if (KIND == 2) umma_i8_2cta(d, ad, bd, idesc, accum);
                else umma_f8_2cta(d, ad, bd, idesc, accum);
              } else {
                if (KIND == 0) umma_f16(d, ad, bd, idesc, accum);
                else if (KIND == 2) umma_i8(d, ad, bd, idesc, accum);
                else umma_f8(d, ad, bd, idesc, accum);
              }
            }
          }
          if (CTA2) umma_commit_2cta(bar_empty(stage), 3); else umma_commit(bar_empty(stage));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) {
          if (CTA2) umma_commit_2cta(bar_tfull(acc), 3); else umma_commit(bar_tfull(acc));
        }
      }
      if (tr != nullptr) {
        tr[2] = globaltimer_ns();
        tr[7] = static_cast<unsigned long long>(it);
      }
      if (*s_abort != 0) {  // UMMAs in flight still read shared memory and write tensor memory
        if (CTA2) umma_commit_2cta(bar_retired, 1); else umma_commit(bar_retired);
        mbar_wait(bar_retired, 0, AbortWord{nullptr, 0u}, 0, 2000000ull);
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue
    const int quad = warp & 3, ew = warp - 2, first_box = ew >> 2;
    const uint32_t stage_blk = smem_base + L::kEpiOffset + ew * 4096;
    const uint32_t stage_row = stage_blk + lane * 128;
    const uint32_t tmem_quad = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t tempty0 = CTA2 ? mapa_u32(bar_tempty(0), 0) : bar_tempty(0);
    constexpr bool acc_int = KIND == 2;
    const bool to_bf16 = p.out_bf16 != 0;
    const int bias_mode = p.bias_mode;
    int it = 0;
    int t, kb0, kb1, part;
    for (; get_item(it, t, kb0, kb1, part); ++it) {
      const int acc = ACCS == 2 ? it & 1 : 0;
      const uint32_t acc_phase = (ACCS == 2 ? it >> 1 : it) & 1;
      int m_idx, n_idx;
      plain_tile(p, t, m_idx, n_idx);
      const int row0 = m_idx * TILE_M + half * kBM + quad * 32;  // first row of this warp
      const int row = row0 + lane;
      const int n0 = n_idx * BN;
      // the tile's scales and bias on their way while its main loop runs (a cold 16-byte load per 8 columns cost 2000
      // clocks a box): vectors to L1, rows of a full bias to L2
      if (it == 0) pdl_wait();
      if (p.scale_b != nullptr && lane < BN / 32 && n0 + lane * 32 < p.N) prefetch_l1(p.scale_b + n0 + lane * 32);
      if (p.scale_a != nullptr && row < p.M) prefetch_l1(p.scale_a + row);
      if (bias_mode == kBiasRow && lane < BN / 64 && n0 + lane * 64 < p.N) prefetch_l1(p.bias + n0 + lane * 64);
      if (bias_mode == kBiasFull && row < p.M)
        for (int box = first_box; box < BN / 64 && n0 + box * 64 < p.N; box += 2)
          prefetch_l2(p.bias + static_cast<long long>(row) * p.N + n0 + box * 64);
      if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull(acc), acc_phase, ab, kStatusTimeoutTmemFull, budget, 100))) break;
      tc_fence_after();
      const uint32_t tacc = tmem_quad + static_cast<uint32_t>(acc * BN);
      // Split tail tile: this warp parks the boxes that another part finishes (32-column step c of a slot is 8 x 32
      // 16-byte pieces: every access of the warp is 512 contiguous bytes), waits until the same warp of all parts has,
      // and finishes its own boxes with the others' partial sums added. All of it stays inside this GPU: device scope.
      const bool is_tail = split > 1 && it == full_waves;
      const float* parked = nullptr;
      bool finishes = true;
      if (is_tail) {
        const int tt = t - full_waves * workers;
        const int owners = splitk_owners(split, BN, false);
        float* base = p.splitk_scratch + (static_cast<long long>(tt) * (split - 1) * TILE_M + half * kBM + quad * 32) * BN + lane * 4;
#pragma unroll 1
        for (int box = first_box; box < BN / 64; box += 2) {
          const int oc = splitk_owner_of(2 * box, split, BN, false);
          if (oc == part) continue;
          float* dst = base + static_cast<long long>(part < oc ? part : part - 1) * TILE_M * BN + box * (2 * 8 * 32 * 4);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld_32x32(tacc + box * 64 + h * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 8; ++q)
              *reinterpret_cast<uint4*>(dst + (h * 8 + q) * (32 * 4)) = make_uint4(r[q * 4], r[q * 4 + 1], r[q * 4 + 2], r[q * 4 + 3]);
          }
        }
        __syncwarp();
        int okw = 1;
        if (lane == 0) {
          int* cnt = p.splitk_cnt + (tt * 2 + half) * 8 + ew;
          int* done = p.splitk_done + (tt * 2 + half) * 8 + ew;
          red_add_release_gpu(cnt, 1);
          if (part < owners) okw = flag_wait_eq_gpu(cnt, split, ab, kStatusTimeoutTmemFull, budget) ? 1 : 0;
          // the last part through clears both counters for the next launch
          if (okw && atomicAdd(done, 1) == split - 1) {
            *cnt = 0;
            *done = 0;
          }
        }
        okw = __shfl_sync(0xffffffffu, okw, 0);
        if (!okw) break;
        __syncwarp();
        parked = base;
        finishes = part < owners;
      }
      if (finishes && row0 < p.M) {
        float row_scale = p.alpha;
        if (p.scale_a != nullptr && row < p.M) row_scale *= p.scale_a[row];
        const uint16_t* bias_row = p.bias + (bias_mode == kBiasFull ? static_cast<long long>(row < p.M ? row : row0) * p.N : 0);
#pragma unroll 1
        for (int box = first_box; box < BN / 64; box += 2) {
          const int col0 = n0 + box * 64;
          if (col0 >= p.N) break;
          if (is_tail && splitk_owner_of(2 * box, split, BN, false) != part) continue;
          uint32_t w[32];  // 64 packed outputs
          uint32_t r2[2][32];
          tmem_ld_32x32(tacc + box * 64, r2[0]);
          tmem_ld_32x32(tacc + box * 64 + 32, r2[1]);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t (&r)[32] = r2[h];
            if (is_tail) add_parked(r, parked + (2 * box + h) * (8 * 32 * 4), TILE_M * BN, split - 1, acc_int);
            const int c0 = col0 + h * 32;
            if (p.scale_b != nullptr || acc_int) {
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                float4 s4 = make_float4(1.f, 1.f, 1.f, 1.f);
                if (p.scale_b != nullptr && c0 + q * 4 < p.N) s4 = __ldg(reinterpret_cast<const float4*>(p.scale_b + c0) + q);
                const float s[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  uint32_t& x = r[q * 4 + j];
                  if (acc_int) {
                    // the reference's order, bit-identical to its golden path; a bias joins the already rounded value
                    float v = (row_scale * s[j]) * __int2float_rn(static_cast<int>(x));
                    if (bias_mode != kBiasNone) v = to_bf16 ? __bfloat162float(__float2bfloat16_rn(v)) : __half2float(__float2half_rn(v));
                    x = __float_as_uint(v);
                  } else {
                    x = __float_as_uint((__uint_as_float(x) * row_scale) * s[j]);
                  }
                }
              }
            } else if (row_scale != 1.0f) {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * row_scale);
            }
            if (bias_mode != kBiasNone) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 b = make_uint4(0u, 0u, 0u, 0u);
                if (c0 + q * 8 < p.N) b = __ldg(reinterpret_cast<const uint4*>(bias_row + c0) + q);
                const uint32_t b4[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 f = to_bf16 ? make_float2(__uint_as_float(b4[j] << 16), __uint_as_float(b4[j] & 0xFFFF0000u))
                                           : __half22float2(*reinterpret_cast<const __half2*>(&b4[j]));
                  r[q * 8 + 2 * j] = __float_as_uint(__uint_as_float(r[q * 8 + 2 * j]) + f.x);
                  r[q * 8 + 2 * j + 1] = __float_as_uint(__uint_as_float(r[q * 8 + 2 * j + 1]) + f.y);
                }
              }
            }
#pragma unroll
            for (int q = 0; q < 16; ++q)
              w[h * 16 + q] = to_bf16 ? pack_bf16(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]))
                                      : pack_f16(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]));
          }
          // one 32 x 64 box through shared memory (16-byte pieces XOR-swizzled by row like the map's 128-byte swizzle);
          // the map clips rows and columns past the output's end
          if (elect_one()) bulk_wait_read();
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage_row + ((q ^ (lane & 7)) << 4)),
                         "r"(w[4 * q]), "r"(w[4 * q + 1]), "r"(w[4 * q + 2]), "r"(w[4 * q + 3])
                         : "memory");
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            tma_store_2d(&p.tmap_out, stage_blk, col0, row0);
            bulk_commit();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTA2) mbar_arrive_cluster(tempty0 + 8u * acc); else mbar_arrive(tempty0 + 8u * acc);
      }
    }
    if (elect_one()) bulk_wait_all();  // tiled stores must not outlive the CTA
    if (tr != nullptr && warp == 2 && lane == 0) tr[3] = tr[4] = globaltimer_ns();
  }

  // ------------------------------------------------------------------ teardown
  if (CTA2) cluster_sync_all(); else __syncthreads();
  if (*s_abort != 0 && threadIdx.x == 0) {
    *reinterpret_cast<volatile int*>(p.status) = *s_abort;
    __threadfence_system();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if (CTA2) tmem_dealloc_2cta(tmem_base, L::kTmemCols); else tmem_dealloc(tmem_base, L::kTmemCols);
  }
}

}  // namespace fluxb
