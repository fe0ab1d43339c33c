// Top-k sparse attention of the reference's full layers (DGQ_ATTN_TOPK_DECODE: src/shaders/attn/attention_topk/,
// oracle src/shaders/attn/attention_topk/cpu.rs:39-120), the selection and gathered-PV half.
//
// Per (canvas row, query head): only the k highest-scoring visible keys are kept (ties: lower index first), the
// softmax is renormalised over them and O = sum_j p_j V[idx_j].  dg_topk_scores.cu has written the fp32 scores of all
// keys (masked ones as -inf) and, per group of 16 consecutive keys, the larger half of the order key of its maximum.
// This kernel, one CTA of 256 threads per (row, head),
//   1. finds the k-th largest of the group maxima, to 16 bits, rounded down: at least k keys reach that bound, and every
//      key that does lies in a group whose maximum does.  On scores without structure about 1.03 k groups with
//      1.07 k such keys are left of T / 16 groups (k = T / 128);
//   2. reads those groups only, one in eight, and lists the keys at or above the bound in index order;
//   3. finds the k-th largest of them exactly (radix over the 32-bit order keys) and keeps what lies above it and the
//      lowest indices among what equals it;
//   4. softmax over the kept scores, and the gather of V, a warp per kept key.
// Lists that outgrow shared memory (many equal scores, clustered ones) take the same steps over the groups in memory.
// Bound: the gather (4,096 rows x 258 keys x 1 KB = 1.08 GB out of L2 at head_dim 512): 175 us of 354 for the whole call at
// 33,024 keys, 6.2 TB/s into the SMs.  With bf16 scores, two histograms over all of a row and the exact scores of the kept
// keys computed again from K (another 1.08 GB gathered) the call took 900 us.
#include <cuda.h>

#include "dg_common.cuh"
#include "dg_kernels.h"
#include "sm100_ptx.cuh"

namespace dg {

namespace tk {
constexpr uint32_t THREADS = 256, WARPS = THREADS / 32;
constexpr uint32_t K_CAP = 1024;      // most keys kept per row (the reference's largest slot capacity)
constexpr uint32_t G_CAP = 2048;      // groups listed in shared memory
constexpr uint32_t C_CAP = 256;       // keys listed per warp
}  // namespace tk

// Shared state of the radix steps: bin counts, per-warp sums, and the outcome {bin, keys above it, keys in it}.
struct TopkRadix {
  uint32_t hist[256];
  uint32_t wsum[tk::WARPS];
  uint32_t out[3];
};
// The bin, from the top, in which the running count reaches `need` (1 <= need <= total).  All threads, after a barrier
// that follows the counting; ends with a barrier.
__device__ __forceinline__ void topk_find_bin(TopkRadix& r, uint32_t need) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, bin = 255u - threadIdx.x;
  const uint32_t own = r.hist[bin];
  uint32_t incl = own;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) r.wsum[warp] = incl;
  __syncthreads();
#pragma unroll
  for (uint32_t w = 0; w < tk::WARPS; ++w)
    if (w < warp) incl += r.wsum[w];
  // fewer than `need` in all (scores of -inf or NaN among the visible ones): the last bin, all of it
  if (incl - own < need && (incl >= need || bin == 0u)) {
    r.out[0] = bin;
    r.out[1] = incl - own;
    r.out[2] = own;
  }
  __syncthreads();
}
__device__ __forceinline__ uint32_t warp_excl_sum(uint32_t v, uint32_t lane, uint32_t& total) {
  uint32_t incl = v;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  total = __shfl_sync(0xffffffffu, incl, 31);
  return incl - v;
}

__global__ void __launch_bounds__(tk::THREADS, 5) dg_topk_select_pv_kernel(const TopkParams p) {
  using namespace tk;
  __shared__ TopkRadix rad;
  // listed groups, then the winners in index order with their scores (later probabilities)
  __shared__ __align__(16) uint32_t lists[2 * K_CAP];
  uint32_t* glist = lists;                                        // [G_CAP]
  uint32_t* s_idx = lists;                                        // [K_CAP]
  float* s_sc = reinterpret_cast<float*>(lists + K_CAP);          // [K_CAP]
  static_assert(G_CAP <= 2 * K_CAP, "group list");
  // listed keys and their positions per warp, then the warps' partial output rows
  __shared__ __align__(16) uint32_t cands[2 * WARPS * C_CAP];
  uint32_t(*c_key)[C_CAP] = reinterpret_cast<uint32_t(*)[C_CAP]>(cands);
  uint32_t(*c_idx)[C_CAP] = reinterpret_cast<uint32_t(*)[C_CAP]>(cands + WARPS * C_CAP);
  float(*s_part)[512] = reinterpret_cast<float(*)[512]>(cands);
  static_assert(2 * C_CAP >= 512, "partial rows");
  __shared__ uint32_t c_n[WARPS], w_cnt[WARPS], w_eq[WARPS];
  __shared__ uint32_t sh_bulk;
  __shared__ float red[WARPS];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // blockIdx.x: row of the pass = (row pair, stacked row)
  const uint32_t rp = p.rp0 + blockIdx.x / 256u, R = (rp % p.rp_per_head) * 256u + blockIdx.x % 256u;
  if (R >= p.C * p.G) return;
  const uint32_t kvh = rp / p.rp_per_head, i = R / p.G, h = kvh * p.G + R % p.G;
  const MaskParams mk = p.mask;
  const RowVis rv = mask_row(mk, i);
  const uint32_t T = mk.can_hi;
  const uint32_t n_valid = (mk.pre_hi > rv.lo ? mk.pre_hi - rv.lo : 0u) + (rv.can_hi > rv.can_lo ? rv.can_hi - rv.can_lo : 0u);
  uint32_t k_req = p.k_fixed;
  if (p.k_div != 0u) {
    k_req = n_valid / p.k_div;
    k_req = k_req < p.k_min ? p.k_min : k_req;
    k_req = k_req > p.k_max ? p.k_max : k_req;
  }
  uint32_t k = k_req < n_valid ? k_req : n_valid;
  if (k > K_CAP) k = K_CAP;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __nv_bfloat16* orow = p.out + (size_t(i) * p.Hq + h) * p.D;
  if (k == 0u) {
    for (uint32_t d = tid; d < p.D; d += THREADS) orow[d] = __float2bfloat16(0.f);
    return;
  }
  const uint32_t n_groups = p.n_groups;
  const uint4* gmax = reinterpret_cast<const uint4*>(p.gmax + size_t(blockIdx.x) * n_groups);       // eight groups per load
  // 16 keys of group g of this row: float4 (g * 128 + (q >> 1) * 64 + (q & 1)), q = 0..3
  const uint4* row = reinterpret_cast<const uint4*>(p.scores) + (size_t(blockIdx.x / 32u) * n_groups * 512u + (blockIdx.x % 32u) * 8u) / 4u;
  auto quad = [&](uint32_t g, uint32_t q) { return __ldcs(&row[size_t(g) * 128u + (q >> 1) * 64u + (q & 1u)]); };
  auto okey = [](uint32_t bits) { return score_order_key(__uint_as_float(bits)); };
  const uint32_t n_g8 = n_groups / 8u;

  // ---- 1. bound: the k-th largest group maximum (16 bits of it)
  uint32_t bound16 = 0u;
  if (n_groups > k) {
    uint32_t need = k;
#pragma unroll 1
    for (uint32_t level = 0; level < 2; ++level) {
      rad.hist[tid] = 0u;
      __syncthreads();
      for (uint32_t c = tid; c < n_g8; c += THREADS) {
        const uint4 x = gmax[c];
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (uint32_t w = 0; w < 4; ++w)
#pragma unroll
          for (uint32_t o = 0; o < 2; ++o) {
            const uint32_t key = (xs[w] >> (16 * o)) & 0xffffu;
            if (level == 0) atomicAdd(&rad.hist[key >> 8], 1u);
            else if ((key >> 8) == bound16) atomicAdd(&rad.hist[key & 0xffu], 1u);
          }
      }
      __syncthreads();
      topk_find_bin(rad, need);
      need -= rad.out[1];
      bound16 = (bound16 << 8) | rad.out[0];
      __syncthreads();
    }
  }
  // masked keys are -inf (0x007f...): with fewer groups in sight than k the bound is what lies just above them
  if (bound16 < 0x80u) bound16 = 0x80u;

  // ---- 2. groups that reach the bound, in index order: each warp looks through a contiguous run
  const uint32_t per_w = (n_g8 + WARPS - 1u) / WARPS;
  const uint32_t g8_lo = warp * per_w < n_g8 ? warp * per_w : n_g8, g8_hi = g8_lo + per_w < n_g8 ? g8_lo + per_w : n_g8;
  auto reach = [&](const uint4 x) {      // bit e: group e of the eight reaches the bound
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
    uint32_t m = 0u;
#pragma unroll
    for (uint32_t w = 0; w < 4; ++w) {
      if ((xs[w] & 0xffffu) >= bound16) m |= 1u << (2 * w);
      if ((xs[w] >> 16) >= bound16) m |= 2u << (2 * w);
    }
    return m;
  };
  uint32_t mine = 0u;
  for (uint32_t c = g8_lo + lane; c < g8_hi; c += 32u) mine += __popc(reach(gmax[c]));
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) w_cnt[warp] = mine;
  if (tid == 0) sh_bulk = 0u;
  __syncthreads();
  uint32_t g_off = 0u, n_list = 0u;
#pragma unroll
  for (uint32_t w = 0; w < WARPS; ++w) {
    if (w < warp) g_off += w_cnt[w];
    n_list += w_cnt[w];
  }
  if (n_list <= G_CAP) {
    for (uint32_t c0 = g8_lo; c0 < g8_hi; c0 += 32u) {
      const uint32_t c = c0 + lane;
      uint32_t m = c < g8_hi ? reach(gmax[c]) : 0u, total;
      uint32_t at = g_off + warp_excl_sum(__popc(m), lane, total);
      for (; m != 0u; m &= m - 1u) glist[at++] = c * 8u + (__ffs(m) - 1u);
      g_off += total;
    }
    __syncthreads();
    // ---- keys at or above the bound: four lanes per group, eight groups at a time, in index order
    const uint32_t bound = bound16 << 16;
    const uint32_t l_lo = n_list * warp / WARPS, l_hi = n_list * (warp + 1u) / WARPS;
    uint32_t n = 0u;
#pragma unroll 2
    for (uint32_t l0 = l_lo; l0 < l_hi; l0 += 8u) {
      const uint32_t l = l0 + (lane >> 2), q = lane & 3u;
      uint32_t t0 = 0u, m = 0u, key[4] = {0u, 0u, 0u, 0u};
      if (l < l_hi) {
        const uint32_t g = glist[l];
        const uint4 x = quad(g, q);
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
        t0 = g * 16u + q * 4u;
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
          key[e] = okey(xs[e]);
          if (key[e] >= bound && t0 + e < T) m |= 1u << e;
        }
      }
      uint32_t total;
      uint32_t at = n + warp_excl_sum(__popc(m), lane, total);
      n += total;
      if (n > C_CAP) break;                  // warp-uniform
#pragma unroll
      for (uint32_t e = 0; e < 4; ++e)
        if ((m >> e) & 1u) {
          c_key[warp][at] = key[e];
          c_idx[warp][at] = t0 + e;
          ++at;
        }
    }
    if (lane == 0) {
      c_n[warp] = n;
      if (n > C_CAP) sh_bulk = 1u;
    }
  } else if (tid == 0) {
    sh_bulk = 1u;
  }
  __syncthreads();

  // ---- 3. the k-th largest key, exactly, and the winners in index order
  const bool bulk = sh_bulk != 0u;
  uint32_t n_cand = 0u;
  if (!bulk) {
#pragma unroll
    for (uint32_t w = 0; w < WARPS; ++w) n_cand += c_n[w];
  }
  // keys of the groups that reach the bound, straight from memory: f(t, order key); thread tid takes a contiguous run
  const uint32_t per_t = (n_groups + THREADS - 1u) / THREADS;
  const uint32_t gt_lo = tid * per_t < n_groups ? tid * per_t : n_groups, gt_hi = gt_lo + per_t < n_groups ? gt_lo + per_t : n_groups;
  auto for_bulk = [&](auto f) {
    const uint16_t* g16 = reinterpret_cast<const uint16_t*>(gmax);
    for (uint32_t g = gt_lo; g < gt_hi; ++g) {
      if (g16[g] < bound16) continue;
      for (uint32_t q = 0; q < 4; ++q) {
        const uint4 x = quad(g, q);
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e)
          if (g * 16u + q * 4u + e < T) f(g * 16u + q * 4u + e, okey(xs[e]));
      }
    }
  };
  auto for_listed = [&](auto f) {
    for (uint32_t j = lane; j < c_n[warp]; j += 32u) f(c_idx[warp][j], c_key[warp][j]);
  };
  uint32_t thr = 0u, need = k;              // kept: keys above thr, and the first `need` of those equal to it
  if (bulk || n_cand > k) {
    uint32_t mask = 0u;
#pragma unroll 1
    for (int shift = 24; shift >= 0; shift -= 8) {
      rad.hist[tid] = 0u;
      __syncthreads();
      auto count = [&](uint32_t, uint32_t key) {
        if ((key & mask) == thr) atomicAdd(&rad.hist[(key >> shift) & 0xffu], 1u);
      };
      if (bulk) for_bulk(count);
      else for_listed(count);
      __syncthreads();
      topk_find_bin(rad, need);
      need -= rad.out[1];
      thr |= rad.out[0] << shift;
      mask |= 0xffu << shift;
      const bool done = rad.out[2] == need;   // all of the bin is kept: nothing below matters
      __syncthreads();
      if (done) {
        // every key with this prefix is kept: "above thr - 1"
        need = 0u;
        thr = thr != 0u ? thr - 1u : 0u;
        break;
      }
    }
  }
  uint32_t n_kept;
  if (!bulk) {
    uint32_t gt = 0u, eq = 0u;
    const uint32_t n = c_n[warp];
    for (uint32_t j = lane; j < n; j += 32u) {
      const uint32_t key = c_key[warp][j];
      gt += key > thr ? 1u : 0u;
      eq += key == thr ? 1u : 0u;
    }
    gt = __reduce_add_sync(0xffffffffu, gt);
    eq = __reduce_add_sync(0xffffffffu, eq);
    if (lane == 0) {
      w_cnt[warp] = gt;
      w_eq[warp] = eq;
    }
    __syncthreads();
    uint32_t at = 0u, eq_before = 0u, all_gt = 0u, all_eq = 0u;
#pragma unroll
    for (uint32_t w = 0; w < WARPS; ++w) {
      if (w < warp) {
        at += w_cnt[w];
        eq_before += w_eq[w];
      }
      all_gt += w_cnt[w];
      all_eq += w_eq[w];
    }
    at += eq_before < need ? eq_before : need;
    n_kept = all_gt + (all_eq < need ? all_eq : need);
    for (uint32_t j0 = 0; j0 < n; j0 += 32u) {
      const uint32_t j = j0 + lane;
      const uint32_t key = j < n ? c_key[warp][j] : 0u;
      const bool is_eq = j < n && key == thr;
      const uint32_t eq_mask = __ballot_sync(0xffffffffu, is_eq), below = (1u << lane) - 1u;
      const bool take = (j < n && key > thr) || (is_eq && eq_before + __popc(eq_mask & below) < need);
      const uint32_t take_mask = __ballot_sync(0xffffffffu, take);
      if (take) {
        const uint32_t o = at + __popc(take_mask & below);
        s_idx[o] = c_idx[warp][j];
        s_sc[o] = score_from_key(key);
      }
      at += __popc(take_mask);
      eq_before += __popc(eq_mask);
    }
  } else {
    uint32_t gt = 0u, eq = 0u;
    for_bulk([&](uint32_t, uint32_t key) {
      gt += key > thr ? 1u : 0u;
      eq += key == thr ? 1u : 0u;
    });
    uint32_t gt_w, eq_w;
    const uint32_t gt_x = warp_excl_sum(gt, lane, gt_w), eq_x = warp_excl_sum(eq, lane, eq_w);
    if (lane == 0) {
      w_cnt[warp] = gt_w;
      w_eq[warp] = eq_w;
    }
    __syncthreads();
    uint32_t gt_before = gt_x, eq_before = eq_x, all_gt = 0u, all_eq = 0u;
#pragma unroll
    for (uint32_t w = 0; w < WARPS; ++w) {
      if (w < warp) {
        gt_before += w_cnt[w];
        eq_before += w_eq[w];
      }
      all_gt += w_cnt[w];
      all_eq += w_eq[w];
    }
    n_kept = all_gt + (all_eq < need ? all_eq : need);
    uint32_t at = gt_before + (eq_before < need ? eq_before : need);
    for_bulk([&](uint32_t t, uint32_t key) {
      const bool take = key > thr || (key == thr && eq_before < need);
      if (key == thr) ++eq_before;
      if (take) {
        s_idx[at] = t;
        s_sc[at] = score_from_key(key);
        ++at;
      }
    });
  }
  k = n_kept < k ? n_kept : k;
  __syncthreads();

  // ---- 4. softmax over the winners
  float mx = -INFINITY;
  for (uint32_t j = tid; j < k; j += THREADS) mx = fmaxf(mx, s_sc[j]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (uint32_t w = 1; w < WARPS; ++w) mx = fmaxf(mx, red[w]);
  mx *= p.scale_log2;
  __syncthreads();
  float l = 0.f;
  for (uint32_t j = tid; j < k; j += THREADS) {
    const float pj = fast_exp2(s_sc[j] * p.scale_log2 - mx);
    s_sc[j] = pj;
    l += pj;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if (lane == 0) red[warp] = l;
  __syncthreads();
  l = 0.f;
#pragma unroll
  for (uint32_t w = 0; w < WARPS; ++w) l += red[w];
  const float inv_l = l > 0.f ? 1.0f / l : 0.f;

  // ---- O = sum_j p_j V[idx_j]: a warp takes every eighth kept key, its lanes cover the value row with 16-byte
  // loads (several rows in flight), packed fp32 pairs, and the eight partial rows meet in shared memory
  const __nv_bfloat16* vbase = p.v + size_t(kvh) * p.cap * p.D;
  const uint32_t n_chunk = p.D / 256;            // 16-byte chunks per lane: 1 at head_dim 256, 2 at 512
  uint64_t acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0ull;
  auto add_row = [&](float pj, uint32_t c, const uint4 x) {
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
    const uint64_t p2 = pack_f32x2(pj, pj);
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[c * 4 + e] = fma_f32x2(p2, bf16x2_to_f32x2(xs[e]), acc[c * 4 + e]);
  };
  if (n_chunk == 2u) {
#pragma unroll 4
    for (uint32_t j = warp; j < k; j += WARPS) {
      const uint4* vr = reinterpret_cast<const uint4*>(vbase + size_t(s_idx[j]) * 512u) + lane;
      const uint4 a = vr[0], b = vr[32];
      add_row(s_sc[j], 0, a);
      add_row(s_sc[j], 1, b);
    }
  } else {
#pragma unroll 8
    for (uint32_t j = warp; j < k; j += WARPS)
      add_row(s_sc[j], 0, reinterpret_cast<const uint4*>(vbase + size_t(s_idx[j]) * 256u)[lane]);
  }
#pragma unroll
  for (uint32_t c = 0; c < 2; ++c) {
    if (c >= n_chunk) break;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float a0, a1;
      unpack_f32x2(acc[c * 4 + e], a0, a1);
      s_part[warp][(c * 32u + lane) * 8u + 2 * e] = a0;
      s_part[warp][(c * 32u + lane) * 8u + 2 * e + 1] = a1;
    }
  }
  __syncthreads();
  for (uint32_t d2 = tid; d2 < p.D / 2; d2 += THREADS) {
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (uint32_t w = 0; w < WARPS; ++w) {      // fixed order: same bits every run
      a0 += s_part[w][2 * d2];
      a1 += s_part[w][2 * d2 + 1];
    }
    reinterpret_cast<uint32_t*>(orow)[d2] = pack_bf16x2(a0 * inv_l, a1 * inv_l);
  }
}

cudaError_t launch_topk_select_pv(const TopkParams& p, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.rp1 - p.rp0) * 256u);
  cfg.blockDim = dim3(tk::THREADS);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, dg_topk_select_pv_kernel, p);
}

}  // namespace dg
