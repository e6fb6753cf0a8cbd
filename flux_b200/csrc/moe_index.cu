// Integer routing work of the MoE ops. Everything here is exact integer
// arithmetic and deterministic (no atomics decide an order).
//
// scatter index (stable): rows are sorted by expert, ties keep (token, k)
// order - the definition of the reference's calc_scatter_index_stable
// (python/flux/testing/moe_utils.py:141-144). The reference's device kernel
// (src/cuda/moe_utils.cu:23-75) orders rows inside an expert with shared
// memory atomics; this one does not.
// gather index: inverse permutation (src/moe_ag_scatter/sort_util.cu:39-92).
#include "internal.h"

namespace fluxb {

constexpr int kIdxThreads = 1024;
constexpr int kIdxWarps = kIdxThreads / 32;
constexpr int kMaxExperts = 1024;
constexpr int kIdxCluster = 8;

// Words of shared memory: per-warp counts [kIdxWarps][pitch] (pitch odd: a column of warps hits every bank), this
// CTA's totals, the totals of all CTAs and those of the lower CTAs per expert.
__host__ __device__ constexpr int idx_pitch(int nexperts) { return nexperts | 1; }
constexpr size_t idx_smem_bytes(int nexperts) {
  return (static_cast<size_t>(kIdxWarps) * idx_pitch(nexperts) + 3 * static_cast<size_t>(nexperts)) * sizeof(int);
}

// One cluster of CTAs (one CTA for few pairs). Every warp owns a contiguous run of the (token, k) pairs, so positions
// inside an expert follow (token, k) order: count the run's pairs per expert, turn the counts into first positions
// (over the warps by shuffles, over the CTAs through distributed shared memory, over the experts by one warp),
// then walk the run again 32 pairs at a time, where the lanes of one expert number themselves with a match. All loads
// are coalesced, and the serial chain is one shared-memory update per 32 pairs of a warp. (One block whose threads
// each walked a slice of their own, with 32 counters per thread, took 36 us for 128 pairs and 58 us for 16384; this
// takes 4.2 and 6.1 us.)
__global__ void __launch_bounds__(kIdxThreads)
scatter_index_kernel(const int* __restrict__ chosen, int total, int nexperts, int* splits,
                     int* scatter_index) {
  extern __shared__ int sh[];
  const int pitch = idx_pitch(nexperts);
  int* cnt = sh;                                  // [kIdxWarps][pitch]
  int* mine = sh + kIdxWarps * pitch;             // [nexperts] this CTA's totals
  int* base = mine + nexperts;                    // [nexperts] totals of all CTAs, then this CTA's first positions
  int* below = base + nexperts;                   // [nexperts] pairs of lower CTAs
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ctas = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);  // the grid is one cluster
  const int per = ((total + ctas * kIdxWarps - 1) / (ctas * kIdxWarps) + 31) & ~31;    // pairs per warp, whole rounds
  const long long lo64 = static_cast<long long>(cta * kIdxWarps + warp) * per;
  const int lo = lo64 < total ? static_cast<int>(lo64) : total;
  const int hi = total - lo < per ? total : lo + per;
  int* wc = cnt + warp * pitch;
  for (int e = lane; e < nexperts; e += 32) wc[e] = 0;
  __syncwarp();
  pdl_wait();
  if (tid == 0) pdl_trigger();
#pragma unroll 4
  for (int i = lo + lane; i < hi; i += 32) {
    const int e = chosen[i];
    if (e >= 0 && e < nexperts) atomicAdd(&wc[e], 1);
  }
  __syncthreads();
  // exclusive prefixes over the warps: warp w takes experts w, w + kIdxWarps, ...; lane l holds warp l's count
  for (int e = warp; e < nexperts; e += kIdxWarps) {
    const int c = cnt[lane * pitch + e];
    int incl = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    cnt[lane * pitch + e] = incl - c;
    if (lane == 31) mine[e] = incl;
  }
  cluster_sync_all();
  // over the CTAs
  for (int e = tid; e < nexperts; e += kIdxThreads) {
    int before = 0, all = 0;
    const uint32_t addr = smem_u32(mine + e);
#pragma unroll
    for (int c = 0; c < kIdxCluster; ++c)
      if (c < ctas) {
        const int v = ld_shared_cluster_u32(mapa_u32(addr, static_cast<uint32_t>(c)));
        if (c < cta) before += v;
        all += v;
      }
    base[e] = all;
    below[e] = before;
    if (cta == 0) splits[e] = all;
  }
  __syncthreads();
  // over the experts
  if (warp == 0) {
    int run = 0;
    for (int e0 = 0; e0 < nexperts; e0 += 32) {
      const int c = e0 + lane < nexperts ? base[e0 + lane] : 0;
      int incl = c;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
      }
      if (e0 + lane < nexperts) base[e0 + lane] = run + incl - c + below[e0 + lane];
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncthreads();
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane;
    const int e = i < hi ? chosen[i] : -1;
    const bool valid = e >= 0 && e < nexperts;
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? e : -1);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int first = 0;
    if (valid) first = wc[e];
    __syncwarp();
    if (valid) {
      scatter_index[i] = base[e] + first + rank;
      if (rank == 0) wc[e] = first + __popc(peers);
    }
    __syncwarp();
  }
  cluster_sync_all();  // no CTA leaves while another still reads its totals
}

__global__ void gather_index_kernel(const int* __restrict__ scatter_index, int total, int topk,
                                    int* gather_index, int* topk_index) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (threadIdx.x == 0) pdl_trigger();
  if (i >= total) return;
  const int row = scatter_index[i];
  if (row < 0 || row >= total) return;
  gather_index[row] = i / topk;
  if (topk_index != nullptr) topk_index[row] = i % topk;
}

}  // namespace fluxb

using namespace fluxb;

extern "C" {

int fluxb_moe_scatter_index(const int* chosen_experts, int ntokens, int topk, int nexperts,
                            int* splits_out, int* scatter_index_out, fluxb_stream_t stream) {
  FLUXB_REQUIRE(chosen_experts != nullptr && splits_out != nullptr && scatter_index_out != nullptr,
                "moe_scatter_index: NULL argument");
  FLUXB_REQUIRE(ntokens >= 0 && topk >= 1, "moe_scatter_index: ntokens=%d topk=%d invalid", ntokens, topk);
  FLUXB_REQUIRE(nexperts >= 1 && nexperts <= kMaxExperts, "moe_scatter_index: nexperts=%d out of [1,%d]",
                nexperts, kMaxExperts);
  const long long total = static_cast<long long>(ntokens) * topk;
  FLUXB_REQUIRE(total < (1ll << 30), "moe_scatter_index: too many routed rows");
  static bool configured[64] = {};
  int dev = 0;
  FLUXB_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {  // up to 140 KB of dynamic shared memory: above the default limit
    FLUXB_CUDA(cudaFuncSetAttribute(scatter_index_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(idx_smem_bytes(kMaxExperts))));
    configured[dev] = true;
  }
  // one CTA while its warps have a round of 32 pairs or two each, else the whole cluster
  const int ctas = total <= 2 * kIdxThreads ? 1 : kIdxCluster;
  return launch_pdl_cluster(scatter_index_kernel, ctas, kIdxThreads, idx_smem_bytes(nexperts), ctas,
                            static_cast<cudaStream_t>(stream), chosen_experts, static_cast<int>(total), nexperts, splits_out, scatter_index_out);
}

int fluxb_moe_gather_index(const int* scatter_index, int ntokens, int topk, int* gather_index_out,
                           int* topk_index_out, fluxb_stream_t stream) {
  FLUXB_REQUIRE(scatter_index != nullptr && gather_index_out != nullptr, "moe_gather_index: NULL argument");
  FLUXB_REQUIRE(ntokens >= 0 && topk >= 1, "moe_gather_index: ntokens=%d topk=%d invalid", ntokens, topk);
  const long long total = static_cast<long long>(ntokens) * topk;
  FLUXB_REQUIRE(total < (1ll << 30), "moe_gather_index: too many routed rows");
  if (total == 0) return FLUXB_OK;
  const int blocks = static_cast<int>((total + 255) / 256);
  return launch_pdl(gather_index_kernel, blocks, 256, static_cast<cudaStream_t>(stream), scatter_index,
                    static_cast<int>(total), topk, gather_index_out, topk_index_out);
}

}  // extern "C"
