// Scores of the top-k path (dg_attn_denoise_topk): S = Q . K^T of every (canvas row, query head) against every key of
// its KV head, in fp32, with the maximum of every 16 consecutive keys beside them (dg_topk.cu selects from both).
//
// CTA pairs (cluster (2, 1, 1), tcgen05 cta_group::2): a pair owns 256 GQA-stacked query rows of one KV head, each CTA
// its own 128 rows, held in shared memory for all of the pair's key tiles.  A tile is 256 keys; each CTA stages half of
// them in slices of 64 head_dim elements through a ring, and the M = 256, N = 256 MMAs fill one of two 256-column
// accumulators while the epilogue warps empty the other.  The (row pair, key tile) units of a launch are cut into
// equal contiguous runs, one per pair, so the last wave is full whatever the key count.
//
// Bound: writing the scores.  4,096 rows x 33,024 keys are 541 MB of fp32 against 61 (head_dim 512) or 31 us (256) of
// MMA work: 143 us in two passes at head_dim 512 (3.8 TB/s of plane, 4.0 TB/s of DRAM traffic, tensor pipe 48 %; smaller
// passes that would stay in L2 lose more to their launches: 372 us for the call with 288 MB, 418 with 144, 462 with 72).  So
// the plane is laid out for the writer: 32 rows of 8 keys are one contiguous KB, which a warp (lane = row) stores with one
// 32-byte access per lane.  A group of 16 keys of a row is then two whole 32-byte sectors, and the selection reads only the
// groups whose maximum can matter, about one in eight.
#include <cuda.h>

#include "dg_attn_sm100_common.cuh"
#include "dg_kernels.h"

namespace dg {

using namespace sm100;

namespace ts {
constexpr uint32_t TM = 128, TN = 256, BK = 64;
constexpr uint32_t THREADS = 320;                 // loader, MMA issuer, eight epilogue warps
constexpr uint32_t ATOM = TM * BK * 2;            // 16 KB: 64 elements of 128 query rows, or of this CTA's 128 keys
__host__ __device__ constexpr uint32_t stages(uint32_t D) { return D == 512 ? 6u : 8u; }
__host__ __device__ constexpr uint32_t smem_bytes(uint32_t D) { return (D / BK + stages(D)) * ATOM + 256 + 1024; }
}  // namespace ts

// A pass of the plane is larger than L2 and one group in eight of it is read, once: marked evict-first it leaves L2 to K,
// which every row pair reads, and to V (33,024 keys, head_dim 512, one run: 368 us for the call without the mark, 357 with it,
// 349 with the selection's reads of the plane marked as well).
__device__ __forceinline__ void st_global_v8(void* dst, const uint32_t* v) {
  asm volatile("st.global.L2::evict_first.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// the larger of three, NaN if any is: a NaN score must reach the selection
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <uint32_t D>
__global__ void __launch_bounds__(ts::THREADS, 1)
dg_topk_scores_kernel(const TopkParams p, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k) {
  using namespace ts;
  constexpr uint32_t ST = stages(D), SL = D / BK;
  enum : uint32_t { B_FULL = 0, B_EMPTY = ST, B_Q = 2 * ST, B_Q_EMPTY = 2 * ST + 1, B_ACC = 2 * ST + 2, B_ACC_EMPTY = 2 * ST + 4,
                    B_COUNT = 2 * ST + 6 };
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t sQ = smem_base, sK = smem_base + SL * ATOM, bar_base = sK + ST * ATOM;
  volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + (SL + ST) * ATOM + B_COUNT * 8);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t xi = cluster_ctarank();               // position inside the pair
  const bool is_leader = xi == 0u;
  auto lead_bar = [&](uint32_t idx) { return dsmem_addr(bar_addr(bar_base, idx), 0u); };
  auto peer_bar = [&](uint32_t idx) { return dsmem_addr(bar_addr(bar_base, idx), 1u); };
  // this pair's run of units; unit = (row pair, key tile), key tiles fastest
  const uint32_t n_kt = p.n_groups / 16u, n_pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
  const uint64_t n_units = uint64_t(p.rp1 - p.rp0) * n_kt;
  const uint32_t u0 = uint32_t(n_units * pair / n_pairs), u1 = uint32_t(n_units * (pair + 1u) / n_pairs);

  if (tid == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(bar_addr(bar_base, B_FULL + s), 1);
      mbar_init(bar_addr(bar_base, B_EMPTY + s), 1);
    }
    mbar_init(bar_addr(bar_base, B_Q), 1);
    mbar_init(bar_addr(bar_base, B_Q_EMPTY), 1);
    for (uint32_t b = 0; b < 2; ++b) {
      mbar_init(bar_addr(bar_base, B_ACC + b), 1);
      mbar_init(bar_addr(bar_base, B_ACC_EMPTY + b), 16);   // eight epilogue warps of each CTA (the leader's copy is used)
    }
    ctl[1] = 0u;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(&ctl[0])), 512);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // the other CTA's barriers exist before anything of ours can signal them
  tc_fence_after();
  const uint32_t tmem = ctl[0];
  volatile uint32_t* abort_flag = &ctl[1];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == 0) {
    // ---------------------------------------------------------------- loader: both CTAs' bytes count on the leader
    if (lane == 0) {
      uint32_t cur = 0xffffffffu, item = 0, it = 0;
      bool ok = true;
      for (uint32_t u = u0; ok && u < u1; ++u) {
        const uint32_t rp = p.rp0 + u / n_kt, kt = u % n_kt;
        const uint32_t kvh = rp / p.rp_per_head;
        if (rp != cur) {
          // the MMAs that read the previous rows are complete
          if (item > 0 && !mbar_wait(bar_addr(bar_base, B_Q_EMPTY), (item - 1u) & 1u, abort_flag)) break;
          cur = rp;
          ++item;
          const uint32_t i0 = ((rp % p.rp_per_head) * 2u + xi) * TM / p.G;   // canvas row of this CTA's first query row
          if (is_leader) mbar_expect_tx(bar_addr(bar_base, B_Q), 2u * SL * ATOM);
          for (uint32_t s = 0; s < SL; ++s)
            tma_load_3d_pair(sQ + s * ATOM, &tm_q, lead_bar(B_Q), int32_t(s * BK), int32_t(kvh * p.G), int32_t(i0));
        }
        for (uint32_t s = 0; s < SL; ++s, ++it) {
          const uint32_t st = it % ST, use = it / ST;
          if (use > 0 && !mbar_wait(bar_addr(bar_base, B_EMPTY + st), (use - 1u) & 1u, abort_flag)) {
            ok = false;
            break;
          }
          if (is_leader) mbar_expect_tx(bar_addr(bar_base, B_FULL + st), 2u * ATOM);
          const int32_t key = int32_t(kt * TN + xi * TM);
          if (D == 512) {      // the cache's map has boxes of 64 keys there, 128 at head_dim 256
            tma_load_3d_pair(sK + st * ATOM, &tm_k, lead_bar(B_FULL + st), int32_t(s * BK), key, int32_t(kvh));
            tma_load_3d_pair(sK + st * ATOM + ATOM / 2, &tm_k, lead_bar(B_FULL + st), int32_t(s * BK), key + 64, int32_t(kvh));
          } else {
            tma_load_3d_pair(sK + st * ATOM, &tm_k, lead_bar(B_FULL + st), int32_t(s * BK), key, int32_t(kvh));
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer of the leader
    if (is_leader) {
      constexpr uint32_t IDESC = umma_idesc_bf16(2 * TM, TN, 0, 0);
      constexpr uint32_t HI = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO 1024, version 1, 128-byte swizzle
      auto mkdesc = [](uint32_t lo, uint32_t hi) { return (uint64_t(hi) << 32) | uint64_t(lo); };
      auto uni = [&](uint32_t idx, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar_addr(bar_base, idx), parity, abort_flag)); };
      uint32_t cur = 0xffffffffu, item = 0, it = 0;
      bool ok = true;
      for (uint32_t u = u0, n = 0; ok && u < u1; ++u, ++n) {
        const uint32_t rp = u / n_kt;
        if (rp != cur) {
          cur = rp;
          if (!uni(B_Q, item & 1u)) break;
          ++item;
        }
        if (n >= 2 && !uni(B_ACC_EMPTY + (n & 1u), ((n >> 1) - 1u) & 1u)) break;
        const uint32_t d_tmem = tmem + (n & 1u) * TN;
        for (uint32_t s = 0; s < SL; ++s, ++it) {
          const uint32_t st = it % ST, use = it / ST;
          if (!uni(B_FULL + st, use & 1u)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t a_lo = (((sQ + s * ATOM) >> 4) & 0x3FFFu) | ((16u >> 4) << 16);
            const uint32_t b_lo = (((sK + st * ATOM) >> 4) & 0x3FFFu) | ((16u >> 4) << 16);
#pragma unroll
            for (uint32_t kk = 0; kk < BK / 16; ++kk)
              umma_ss_pair(d_tmem, mkdesc(a_lo + kk * 2u, HI), mkdesc(b_lo + kk * 2u, HI), IDESC, (s | kk) != 0u);
            umma_commit_pair(lead_bar(B_EMPTY + st));
            umma_commit_pair(peer_bar(B_EMPTY + st));
            if (s + 1 == SL) {
              umma_commit_pair(lead_bar(B_ACC + (n & 1u)));
              umma_commit_pair(peer_bar(B_ACC + (n & 1u)));
              if (u + 1 == u1 || (u + 1) / n_kt != rp) {      // last tile of these rows
                umma_commit_pair(lead_bar(B_Q_EMPTY));
                umma_commit_pair(peer_bar(B_Q_EMPTY));
              }
            }
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue: lane = one query row
    // Two warps per 32 rows, 128 of the tile's keys each, 32 at a time with the next 32 on their way out of tensor memory.
    const uint32_t q4 = warp & 3u, half = warp >= 6u ? 1u : 0u;      // the 32 TMEM lanes this warp may read; which keys
    constexpr uint32_t NC = TN / 64;                                   // blocks of 32 keys per warp
    const uint32_t rows_per_head = p.C * p.G;
    const MaskParams mk = p.mask;
    for (uint32_t u = u0, n = 0; u < u1; ++u, ++n) {
      const uint32_t rp = p.rp0 + u / n_kt, kt = u % n_kt;
      const uint32_t R0 = ((rp % p.rp_per_head) * 2u + xi) * TM + q4 * 32u, R = R0 + lane;
      const uint32_t i_row = R < rows_per_head ? R / p.G : p.C - 1u;
      const RowVis rv = mask_row(mk, i_row);
      const size_t rb = size_t(rp - p.rp0) * 8u + xi * 4u + q4;      // 32-row block of the plane
      const uint32_t g0 = kt * 16u + half * 8u;                        // first group of 16 keys
      float* plane = p.scores + (rb * p.n_groups + g0) * 512u + lane * 8u;
      const uint32_t t_src = tmem + ((q4 * 32u) << 16) + (n & 1u) * TN + half * 128u;
      const bool stored = R0 < rows_per_head;      // warp-uniform: blocks past the last row have no place in the selection
      if (!__all_sync(0xffffffffu, mbar_wait(bar_addr(bar_base, B_ACC + (n & 1u)), (n >> 1) & 1u, abort_flag))) break;
      tc_fence_after();
      uint32_t gm[NC], v[2][32];
      tmem_ld32(t_src, v[0]);
#pragma unroll
      for (uint32_t c = 0; c < NC; ++c) {
        uint32_t(&x)[32] = v[c & 1u];
        tmem_wait_ld();
        if (c + 1 < NC) {
          tmem_ld32(t_src + (c + 1) * 32u, v[(c + 1) & 1u]);
        } else {
          // this warp's part of the accumulator is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(lead_bar(B_ACC_EMPTY + (n & 1u)));
        }
        const uint32_t k0 = g0 * 16u + c * 32u;
        if (!mask_range_full(mk, rv, k0, 32u)) {
          const uint32_t seen = mask_bits16(mk, rv, k0) | (mask_bits16(mk, rv, k0 + 16u) << 16);
#pragma unroll
          for (uint32_t e = 0; e < 32; ++e)
            if (!((seen >> e) & 1u)) x[e] = 0xff800000u;   // -inf
        }
        uint32_t key[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          float m[3];
#pragma unroll
          for (uint32_t e = 0; e < 3; ++e)
            m[e] = max3_nan(__uint_as_float(x[h * 16 + e * 5]), __uint_as_float(x[h * 16 + e * 5 + 1]),
                            max3_nan(__uint_as_float(x[h * 16 + e * 5 + 2]), __uint_as_float(x[h * 16 + e * 5 + 3]),
                                     __uint_as_float(x[h * 16 + e * 5 + 4])));
          const float mx = max3_nan(m[0], m[1], max3_nan(m[2], __uint_as_float(x[h * 16 + 15]), __uint_as_float(x[h * 16 + 15])));
          key[h] = score_order_key(mx) >> 16;
        }
        gm[c] = key[0] | (key[1] << 16);
        if (stored) {
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) st_global_v8(plane + (c * 4u + j) * 256u, &x[j * 8]);
        }
      }
      if (stored) *reinterpret_cast<uint4*>(p.gmax + (rb * 32u + lane) * p.n_groups + g0) = make_uint4(gm[0], gm[1], gm[2], gm[3]);
    }
  }

  if (*abort_flag) {
    if (tid == 0) dev_status_set(p.status, DG_DEV_WAIT_TIMEOUT, KID_SCORES, blockIdx.x, u1 - u0);
    if (warp == 0 && lane == 0) {
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000ll) {}   // ~1 ms: far longer than any tile load in flight
    }
  }
  tc_fence_before();
  __syncthreads();
  // neither CTA frees tensor memory or leaves while the other can still be the target of a pair-wide MMA or commit
  cluster_sync_all();
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

cudaError_t sm100_topk_configure() {
  const cudaError_t e = cudaFuncSetAttribute(dg_topk_scores_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ts::smem_bytes(256)));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(dg_topk_scores_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ts::smem_bytes(512)));
}

cudaError_t launch_topk_scores(const TopkParams& p, const CUtensorMap& tm_q, const CUtensorMap& tm_k, int num_sms, cudaStream_t st) {
  const uint64_t units = uint64_t(p.rp1 - p.rp0) * (p.n_groups / 16u);
  const uint32_t most = num_sms > 1 ? uint32_t(num_sms) / 2u : 74u;
  const uint32_t pairs = units < most ? uint32_t(units) : most;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2u * pairs);
  cfg.blockDim = dim3(ts::THREADS);
  cfg.dynamicSmemBytes = ts::smem_bytes(p.D);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (p.D == 256) return cudaLaunchKernelEx(&cfg, dg_topk_scores_kernel<256>, p, tm_q, tm_k);
  return cudaLaunchKernelEx(&cfg, dg_topk_scores_kernel<512>, p, tm_q, tm_k);
}

}  // namespace dg
