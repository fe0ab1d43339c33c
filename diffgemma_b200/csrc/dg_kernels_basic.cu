// Small kernels around the tensor-core attention kernel:
//   * qk_rope_kv / cache append  (per-head RMSNorm + RoPE + KV-cache write + RoPE table)
//   * general attention kernel   (any head_dim <= 512, any mask incl. a decoder bitmap)
//   * local merge of (O, m, l) partials, NCCL-merge helpers, visibility dump
// Reference behaviour restated (paths relative to the reference project):
//   src/shaders/attn/qk_rope_kv/qk_rope_kv.metal:29-149, src/shaders/attn/cpu.rs:67-145 (stage 1)
//   src/shaders/attn/attention/attention.metal:22-133, src/shaders/attn/cpu.rs:148-197 (stage 2)
#include "dg_common.cuh"
#include "dg_append_vec.cuh"
#include "dg_kernels.h"

namespace dg {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ------------------------------------------------------------------------------------------
// qk_rope_kv / append: one warp per (token, head-vector slot).
// slots: [Q heads (if q_in)] [K heads] [V heads] [1 RoPE-table slot (if rope_table)]
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(32) dg_append_kernel(const AppendParams p, const RopeParams rp) {
  __shared__ float xs[kMaxHeadDim];
  // let a dependent kernel (the attention launch that follows on the stream) begin its set-up now;
  // it synchronises on this grid's completion before it reads the cache or the RoPE table
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // when this kernel was itself launched ahead of the end of its predecessor (programmatic dependent
  // launch), everything it reads or writes may still be in use by that kernel: wait for it here
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t tok = blockIdx.x, slot = blockIdx.y, lane = threadIdx.x;
  const uint32_t D = p.D;
  const uint32_t pos = p.pos0 + tok;
  const uint32_t nq = p.q_in ? p.Hq : 0u;
  const float fpos = float(pos);

  if (slot >= nq + 2u * p.Hkv) {  // RoPE table row: (cos, sin) of f32(pos) * inv_freq[i]
    if (p.rope_table == nullptr) return;
    for (uint32_t i = lane; i < rp.rot_half; i += 32) {
      const float a = fpos * rp.inv_freq[i];
      p.rope_table[size_t(tok) * rp.rot_half + i] = make_float2(cosf(a), sinf(a));
    }
    return;
  }
  const bool is_q = slot < nq;
  const bool is_k = !is_q && slot < nq + p.Hkv;
  const uint32_t H = is_q ? p.Hq : p.Hkv;
  const uint32_t h = is_q ? slot : (slot - nq) % p.Hkv;
  const __nv_bfloat16* src = (is_q ? p.q_in : (is_k ? p.k_in : p.v_in)) + (size_t(tok) * H + h) * D;
  __nv_bfloat16* wb = (is_q ? p.q_out : (is_k ? p.k_out : p.v_out));
  if (wb) wb += (size_t(tok) * H + h) * D;
  // ring caches keep position pos in slot pos & ring_mask; positions at or past write_end (the
  // zero-padded tail of a prefill chunk) must not reach the cache, where they would wrap onto live slots
  __nv_bfloat16* cache = (is_q || pos >= p.write_end || pos < p.pos_base)
                             ? nullptr
                             : (is_k ? p.cache_k : p.cache_v) + (size_t(h) * p.cap + ((pos - p.pos_base) & p.ring_mask)) * D;

  // sum of squares in the order of dg_append_table_kernel (a lane takes 8 consecutive elements, then a
  // butterfly), and the rotation through rope_rotate in both, so that the two kernels write the same bits
  float ss = 0.f;
  for (uint32_t c = lane; c < D / 8; c += 32) {
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) {
      const float x = __bfloat162float(src[c * 8 + e]);
      xs[c * 8 + e] = x;
      ss = __fmaf_rn(x, x, ss);
    }
  }
  ss = warp_sum(ss);
  const bool norm = is_q || is_k || p.v_norm;
  const float inv = norm ? 1.0f / sqrtf(ss / float(D) + p.eps) : 1.0f;
  const __nv_bfloat16* w = is_q ? p.qw : (is_k ? p.kw : nullptr);
  if (norm) {
    for (uint32_t d = lane; d < D; d += 32) {
      // the rotated elements of K get their norm inside the rotation (rope_norm_rotate)
      if (is_k && ((d < rp.rot_half) || (d >= rp.pair_off && d < rp.pair_off + rp.rot_half))) continue;
      const float wv = w ? __bfloat162float(w[d]) : 1.0f;
      xs[d] = xs[d] * (inv * wv);
    }
  }
  __syncwarp();
  if (is_q) {
    for (uint32_t i = lane; i < rp.rot_half; i += 32) {
      const float a = fpos * rp.inv_freq[i];
      const float c = cosf(a), s = sinf(a);
      const float x0 = xs[i], x1 = xs[rp.pair_off + i];
      xs[i] = rope_rotate_lo(x0, x1, c, s);
      xs[rp.pair_off + i] = rope_rotate_hi(x0, x1, c, s);
    }
    __syncwarp();
  } else if (is_k) {
    for (uint32_t i = lane; i < rp.rot_half; i += 32) {
      const float a = fpos * rp.inv_freq[i];
      const float c = cosf(a), s = sinf(a);
      const float x0 = xs[i], x1 = xs[rp.pair_off + i];
      const float w0 = w ? __bfloat162float(w[i]) : 1.0f, w1 = w ? __bfloat162float(w[rp.pair_off + i]) : 1.0f;
      xs[i] = rope_norm_rotate(x0, x1, rope_coef_a(w0, c), rope_coef_b(w1, s, true), inv);
      xs[rp.pair_off + i] = rope_norm_rotate(x1, x0, rope_coef_a(w1, c), rope_coef_b(w0, s, false), inv);
    }
    __syncwarp();
  }
  for (uint32_t d = lane; d < D; d += 32) {
    const __nv_bfloat16 y = __float2bfloat16_rn(xs[d]);
    if (wb) wb[d] = y;
    if (cache) cache[d] = y;
  }
}

// Canvas append when the RoPE table of these positions is already in memory (the denoise steps of a
// canvas revisit the same positions): head_dim 256, full split-half rotary, cache writes only.
// One warp per (token, K or V head vector), lane c owns the 16-byte chunk c, the RoPE partner of a
// chunk is chunk c ^ 16 (one shuffle away); eight warps per CTA.  No sincos, no shared memory, 512-byte
// coalesced loads and stores: the kernel is short enough to hide behind the attention kernel's Q
// prologue, which overlaps it through programmatic dependent launch.
__global__ void __launch_bounds__(256) dg_append_table_kernel(const AppendParams p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // see dg_append_kernel
  const uint32_t lane = threadIdx.x & 31u, w = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (w >= p.n * 2u * p.Hkv) return;
  AppendVecArgs a;
  a.k_in = p.k_in;
  a.v_in = p.v_in;
  a.kw = p.kw;
  a.table = p.rope_table_in;
  a.cache_k = p.cache_k;
  a.cache_v = p.cache_v;
  a.cap = p.cap;
  a.pos0 = p.pos0;
  a.Hkv = p.Hkv;
  a.v_norm = p.v_norm;
  a.ring_mask = p.ring_mask;
  a.write_end = p.write_end;
  a.pos_base = p.pos_base;
  a.eps = p.eps;
  append_table_vector(a, w, lane);
}

// ------------------------------------------------------------------------------------------
// The same stage for head_dim 256 and 512 with rotary runs of whole 16-byte chunks: a CTA takes one token, or some of its
// head vectors, computes the token's (cos, sin) pairs once into shared memory, and a warp handles one or two vectors at a
// time, lane c the 16-byte chunks c and c + 32 together with the chunks that hold their rotation partners.
// Bound: latency up to some thousand vectors, memory on long appends.  The kernel above issues a warp per CTA, 2-byte
// accesses and a sincos per (vector, pair): a head_dim-512 step took 5 us longer with it (32k keys 295.8 -> 290.8 us, 150
// keys 23.4 -> 21.9 us).  Order of operations (chunk-wise sums of squares, butterfly, rotation through
// rope_rotate / rope_norm_rotate) as above: both write the same bits.
// ------------------------------------------------------------------------------------------
constexpr uint32_t kRowsMaxWarps = 10, kRowsUnit = 2;

template <uint32_t NS>   // 16-byte chunks of a vector per lane: head_dim 256 -> 1, 512 -> 2
// head_dim 512: 64 registers, so that more CTAs share an SM (16,000 tokens of 2 x 512, four tokens a CTA: 68.7 us with 90, 54.9 so)
__global__ void __launch_bounds__(kRowsMaxWarps * 32, NS == 2 ? 3 : 1) dg_append_rows_kernel(const AppendParams p, const RopeParams rp, uint32_t slots_per_cta) {
  __shared__ __align__(16) float2 cs[kMaxRotHalf];   // read as float4
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // see dg_append_kernel
  constexpr uint32_t D = NS * 256u, U = kRowsUnit;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const uint32_t tok = blockIdx.x, pos = p.pos0 + tok;
  const uint32_t nq = p.q_in ? p.Hq : 0u, slot0 = blockIdx.y * slots_per_cta, slot_end = min(slot0 + slots_per_cta, nq + 2u * p.Hkv);
  const uint32_t rot_chunks = rp.rot_half / 8u, off_chunks = rp.pair_off / 8u;

  // chunk of this lane in slot j, the chunk of its rotation partner (itself when not rotated), its first pair index
  uint32_t chunk[NS], partner[NS], pair0[NS];
  bool rot[NS], low[NS];
#pragma unroll
  for (uint32_t j = 0; j < NS; ++j) {
    const uint32_t c = lane + 32u * j;
    chunk[j] = c;
    low[j] = c < rot_chunks;
    rot[j] = low[j] || (c >= off_chunks && c < off_chunks + rot_chunks);
    partner[j] = !rot[j] ? c : low[j] ? c + off_chunks : c - off_chunks;
    pair0[j] = (low[j] ? c : c - off_chunks) * 8u;
  }
  uint4 x[U][NS], xp[U][NS];
  auto load = [&](uint32_t s0) {
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t slot = s0 + u * n_warps;
      if (slot >= slot_end) break;
      const bool is_q = slot < nq, is_k = !is_q && slot < nq + p.Hkv;
      const uint32_t H = is_q ? p.Hq : p.Hkv, h = is_q ? slot : (slot - nq) % p.Hkv;
      const uint4* src = reinterpret_cast<const uint4*>((is_q ? p.q_in : is_k ? p.k_in : p.v_in) + (size_t(tok) * H + h) * D);
#pragma unroll
      for (uint32_t j = 0; j < NS; ++j) {
        x[u][j] = src[chunk[j]];
        if ((is_q || is_k) && rot[j]) xp[u][j] = src[partner[j]];
      }
    }
  };
  load(slot0 + warp);
  // (cos, sin) of the token's position, while the first vectors are on their way
  for (uint32_t i = threadIdx.x; i < rp.rot_half; i += blockDim.x) {
    const float a = float(pos) * rp.inv_freq[i];
    const float2 v = make_float2(cosf(a), sinf(a));
    cs[i] = v;
    if (p.rope_table && blockIdx.y == 0u) p.rope_table[size_t(tok) * rp.rot_half + i] = v;
  }
  __syncthreads();
  auto lo16 = [](uint32_t w) { return __uint_as_float(w << 16); };
  auto hi16 = [](uint32_t w) { return __uint_as_float(w & 0xffff0000u); };
  for (uint32_t s0 = slot0 + warp; s0 < slot_end; s0 += U * n_warps) {
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t slot = s0 + u * n_warps;
      if (slot >= slot_end) break;                        // warp-uniform
      const bool is_q = slot < nq, is_k = !is_q && slot < nq + p.Hkv;
      const uint32_t H = is_q ? p.Hq : p.Hkv, h = is_q ? slot : (slot - nq) % p.Hkv;
      uint4 y[NS];
      if (is_q || is_k || p.v_norm) {
        float ss = 0.f;
#pragma unroll
        for (uint32_t j = 0; j < NS; ++j) {
          const uint32_t w[4] = {x[u][j].x, x[u][j].y, x[u][j].z, x[u][j].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ss = __fmaf_rn(lo16(w[e]), lo16(w[e]), ss);
            ss = __fmaf_rn(hi16(w[e]), hi16(w[e]), ss);
          }
        }
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / float(D) + p.eps);
        const __nv_bfloat16* wt = is_q ? p.qw : is_k ? p.kw : nullptr;
        const uint4 ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
#pragma unroll
        for (uint32_t j = 0; j < NS; ++j) {
          const uint32_t m[4] = {x[u][j].x, x[u][j].y, x[u][j].z, x[u][j].w};
          const uint4 w4 = wt ? reinterpret_cast<const uint4*>(wt)[chunk[j]] : ones;
          const uint32_t wm[4] = {w4.x, w4.y, w4.z, w4.w};
          float r[8];
          if ((is_q || is_k) && rot[j]) {
            const uint32_t q[4] = {xp[u][j].x, xp[u][j].y, xp[u][j].z, xp[u][j].w};
            const uint4 p4 = wt ? reinterpret_cast<const uint4*>(wt)[partner[j]] : ones;
            const uint32_t wq[4] = {p4.x, p4.y, p4.z, p4.w};
            const float4* tab = reinterpret_cast<const float4*>(cs + pair0[j]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float4 c2 = tab[e];
#pragma unroll
              for (int o = 0; o < 2; ++o) {
                const float c = o ? c2.z : c2.x, s = o ? c2.w : c2.y;
                const float xm = o ? hi16(m[e]) : lo16(m[e]), xq = o ? hi16(q[e]) : lo16(q[e]);
                const float wo = o ? hi16(wm[e]) : lo16(wm[e]), wp = o ? hi16(wq[e]) : lo16(wq[e]);
                if (is_k) {
                  r[2 * e + o] = rope_norm_rotate(xm, xq, rope_coef_a(wo, c), rope_coef_b(wp, s, low[j]), inv);
                } else {
                  const float a = __fmul_rn(xm, __fmul_rn(inv, wo)), b = __fmul_rn(xq, __fmul_rn(inv, wp));
                  r[2 * e + o] = low[j] ? rope_rotate_lo(a, b, c, s) : rope_rotate_hi(b, a, c, s);
                }
              }
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              r[2 * e] = __fmul_rn(lo16(m[e]), __fmul_rn(inv, lo16(wm[e])));
              r[2 * e + 1] = __fmul_rn(hi16(m[e]), __fmul_rn(inv, hi16(wm[e])));
            }
          }
          __nv_bfloat162 b[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) b[e] = __floats2bfloat162_rn(r[2 * e], r[2 * e + 1]);
          y[j] = make_uint4(*reinterpret_cast<uint32_t*>(&b[0]), *reinterpret_cast<uint32_t*>(&b[1]),
                            *reinterpret_cast<uint32_t*>(&b[2]), *reinterpret_cast<uint32_t*>(&b[3]));
        }
      } else {
#pragma unroll
        for (uint32_t j = 0; j < NS; ++j) y[j] = x[u][j];
      }
      __nv_bfloat16* wb = is_q ? p.q_out : is_k ? p.k_out : p.v_out;
      const bool stored = !is_q && pos < p.write_end && pos >= p.pos_base;
      __nv_bfloat16* cache = (is_k ? p.cache_k : p.cache_v) + (size_t(h) * p.cap + ((pos - p.pos_base) & p.ring_mask)) * D;
      __syncwarp();   // the output may be the input: every lane has read its partner's chunk
#pragma unroll
      for (uint32_t j = 0; j < NS; ++j) {
        if (wb) reinterpret_cast<uint4*>(wb + (size_t(tok) * H + h) * D)[chunk[j]] = y[j];
        if (stored) reinterpret_cast<uint4*>(cache)[chunk[j]] = y[j];
      }
    }
    if (s0 + U * n_warps < slot_end) load(s0 + U * n_warps);
  }
}

// tensors off 16-byte boundaries go to the general kernel, which reads element by element
static bool append_aligned(const AppendParams& p) {
  const void* ptrs[] = {p.q_in, p.q_out, p.k_in, p.k_out, p.v_in, p.v_out, p.qw, p.kw};
  for (const void* q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15u) return false;
  return true;
}
static bool append_rows_ok(const AppendParams& p, const RopeParams& rp) {
  return (p.D == 256 || p.D == 512) && rp.rot_half % 8 == 0 && rp.pair_off % 8 == 0 && append_aligned(p);
}

void launch_append(const AppendParams& p, const RopeParams& rp, cudaStream_t st, bool early) {
  if (p.n == 0) return;
  // `early`: the kernel may be scheduled while its predecessor on the stream is still draining (it
  // waits for that kernel's completion before it touches memory), which hides its launch latency
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  if (p.rope_table_in && !p.rope_table && !p.q_in && !p.k_out && !p.v_out && p.D == 256 && rp.rot_half == 128 &&
      rp.pair_off == 128 && append_aligned(p)) {
    const uint32_t warps = p.n * 2u * p.Hkv;
    cfg.gridDim = dim3((warps + 7u) / 8u);
    cfg.blockDim = dim3(256);
    cudaLaunchKernelEx(&cfg, dg_append_table_kernel, p);
    return;
  }
  if (append_rows_ok(p, rp)) {
    // Few vectors: a warp for each, up to eight of a token per CTA, and at least four warps for the token's (cos, sin) pairs;
    // what counts is the latency of one vector.  Many: all of a token's vectors in one CTA, two or more per warp, so that the
    // pairs are computed once and more loads are in flight.  us with a warp per vector / two per warp: 2 KV heads of 256, 256
    // tokens 3.3 / 3.9, 1,000 4.3 / 6.0, 2,000 7.5 / 6.7; 16 of 256, 100 tokens 3.4 / 5.5, 256 6.4 / 5.9; 2 of 512, 17 tokens 3.7 /
    // 4.6, 1,000 6.0 / 8.6, 8,000 29.9 / 27.6; 8 of 512, 256 tokens 7.0 / 7.8, 500 9.4 / 8.4.  (One-warp CTAs of the kernel above:
    // 2 of 512, 17 tokens 3.7, 1,000 7.1, 8,000 35.6.)
    const uint32_t slots = (p.q_in ? p.Hq : 0u) + 2u * p.Hkv;
    const bool few = size_t(p.n) * slots <= (p.D == 256 ? 4096u : 6144u);
    const uint32_t groups = few ? (slots + 7u) / 8u : 1u, spc = (slots + groups - 1u) / groups;
    const uint32_t warps = few ? (spc > 4u ? spc : 4u) : (spc + kRowsUnit - 1u) / kRowsUnit;
    cfg.gridDim = dim3(p.n, (slots + spc - 1u) / spc);
    cfg.blockDim = dim3(32u * (warps < kRowsMaxWarps ? warps : kRowsMaxWarps));
    if (p.D == 256) cudaLaunchKernelEx(&cfg, dg_append_rows_kernel<1>, p, rp, spc);
    else cudaLaunchKernelEx(&cfg, dg_append_rows_kernel<2>, p, rp, spc);
    return;
  }
  const uint32_t slots = (p.q_in ? p.Hq : 0u) + 2u * p.Hkv + (p.rope_table ? 1u : 0u);
  cfg.gridDim = dim3(p.n, slots);
  cfg.blockDim = dim3(32);
  cudaLaunchKernelEx(&cfg, dg_append_kernel, p, rp);
}

// ------------------------------------------------------------------------------------------
// Saved sessions: rows of a token-major [n][Hkv][D] tensor to or from the head-major cache, K and V in one launch
// (blockIdx.y), 16 bytes per access, four in flight per thread.  Bound: memory.  8,192 tokens of 2 x 512 loaded, 2,000
// appended and all read back: 131.3 us with a strided copy per head, tensor and direction, 42.4 us with this and
// dg_append_rows_kernel (84 MB, 12.8 us at copy bandwidth; the rest is launches and the wait of the read).
// ------------------------------------------------------------------------------------------
constexpr uint32_t kCopyChunks = 4;

__global__ void __launch_bounds__(256) dg_kv_copy_kernel(const KvCopyParams p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // see dg_append_kernel
  uint4* flat = reinterpret_cast<uint4*>(blockIdx.y ? p.v : p.k);
  uint4* cache = reinterpret_cast<uint4*>(blockIdx.y ? p.cache_v : p.cache_k);
  const uint32_t first = blockIdx.x * (256u * kCopyChunks) + threadIdx.x;
  uint4 x[kCopyChunks];
  uint4* slot[kCopyChunks];
#pragma unroll
  for (uint32_t j = 0; j < kCopyChunks; ++j) {
    const uint32_t e = first + j * 256u;                   // chunk of the token-major tensor
    if (e >= p.n_chunks) break;
    const uint32_t row = e / p.row_chunks, c = e - row * p.row_chunks, tok = row / p.Hkv, h = row - tok * p.Hkv;
    slot[j] = cache + (size_t(h) * p.cap + ((p.slot0 + tok) & p.ring_mask)) * p.row_chunks + c;
    x[j] = p.to_cache ? flat[e] : *slot[j];
  }
#pragma unroll
  for (uint32_t j = 0; j < kCopyChunks; ++j) {
    const uint32_t e = first + j * 256u;
    if (e >= p.n_chunks) break;
    if (p.to_cache) *slot[j] = x[j];
    else flat[e] = x[j];
  }
}

cudaError_t launch_kv_copy(const KvCopyParams& p, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.n_chunks + 256u * kCopyChunks - 1u) / (256u * kCopyChunks), 2);
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, dg_kv_copy_kernel, p);
}

// ------------------------------------------------------------------------------------------
// General attention: one CTA (4 warps) per (canvas row, q head); keys strided over warps;
// online softmax per warp, merged at the end.  Serves any head_dim <= 512 (multiple of 8),
// partial rotary / proportional pairing, and explicit decoder bitmaps.
// ------------------------------------------------------------------------------------------
constexpr int GEN_WARPS = 4;

__global__ void __launch_bounds__(GEN_WARPS * 32) dg_attn_general_kernel(const AttnParams p) {
  __shared__ float qs[kMaxHeadDim];
  __shared__ float red[GEN_WARPS];
  __shared__ float wm[GEN_WARPS], wl[GEN_WARPS];
  __shared__ float wo[GEN_WARPS][kMaxHeadDim];

  const uint32_t row = blockIdx.x, h = blockIdx.y;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t D = p.D, kvh = h / p.G;

  // ---- Q prologue (norm + weight + RoPE from the table), then round to bf16
  const __nv_bfloat16* qsrc = p.q + (size_t(row) * p.Hq + h) * D;
  float ss = 0.f;
  for (uint32_t d = tid; d < D; d += GEN_WARPS * 32) {
    const float x = __bfloat162float(qsrc[d]);
    qs[d] = x;
    ss += x * x;
  }
  if (!p.q_prenormed) {
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int w = 0; w < GEN_WARPS; ++w) tot += red[w];
    const float inv = 1.0f / sqrtf(tot / float(D) + p.eps);
    for (uint32_t d = tid; d < D; d += GEN_WARPS * 32) {
      const float wv = p.qw ? __bfloat162float(p.qw[d]) : 1.0f;
      qs[d] = qs[d] * (inv * wv);
    }
    __syncthreads();
    for (uint32_t i = tid; i < p.rot_half; i += GEN_WARPS * 32) {
      const float2 cs = p.rope_table[size_t(row) * p.rot_half + i];
      const float x0 = qs[i], x1 = qs[p.pair_off + i];
      qs[i] = x0 * cs.x - x1 * cs.y;
      qs[p.pair_off + i] = x0 * cs.y + x1 * cs.x;
    }
    __syncthreads();
    for (uint32_t d = tid; d < D; d += GEN_WARPS * 32) qs[d] = __bfloat162float(__float2bfloat16_rn(qs[d]));
  }
  __syncthreads();

  // ---- key sweep
  const uint32_t n_chunks = D / 8;  // 16-byte chunks per row
  float acc[2][8];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[j][e] = 0.f;
  float m = -INFINITY, l = 0.f;

  const MaskParams mk = p.mask;
  const RowVis rv = mask_row(mk, row);
  const uint32_t T = mk.kv_len + p.C;
  const __nv_bfloat16* kbase = p.cache_k + size_t(kvh) * p.cap * D;
  const __nv_bfloat16* vbase = p.cache_v + size_t(kvh) * p.cap * D;

  for (int range = 0; range < 2; ++range) {
    uint32_t lo, hi;
    if (p.attend) {
      if (range == 1) break;
      lo = 0;
      hi = T;
    } else if (range == 0) {
      lo = rv.lo;
      hi = mk.pre_hi;
    } else {
      lo = rv.can_lo;
      hi = rv.can_hi;
    }
    for (uint32_t t = lo + warp; t < hi; t += GEN_WARPS) {
      if (p.attend) {
        if (!p.attend[size_t(row) * T + t]) continue;
      }
      const uint32_t ts = (t - p.pos_base) & p.ring_mask;   // cache slot of key position t
      const uint4* kr = reinterpret_cast<const uint4*>(kbase + size_t(ts) * D);
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t c = lane + 32u * j;
        if (c < n_chunks) {
          const uint4 kk = kr[c];
          const uint32_t w[4] = {kk.x, kk.y, kk.z, kk.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            dot += qs[c * 8 + 2 * e] * __uint_as_float(w[e] << 16);
            dot += qs[c * 8 + 2 * e + 1] * __uint_as_float(w[e] & 0xffff0000u);
          }
        }
      }
      dot = warp_sum(dot);
      const float s2 = dot * p.scale_log2;
      const float mn = fmaxf(m, s2);
      const float corr = exp2f(m - mn);  // exp2(-inf) = 0 on the first key
      const float pe = exp2f(s2 - mn);
      l = l * corr + pe;
      m = mn;
      const uint4* vr = reinterpret_cast<const uint4*>(vbase + size_t(ts) * D);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t c = lane + 32u * j;
        if (c < n_chunks) {
          const uint4 vv = vr[c];
          const uint32_t w[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            acc[j][2 * e] = acc[j][2 * e] * corr + pe * __uint_as_float(w[e] << 16);
            acc[j][2 * e + 1] = acc[j][2 * e + 1] * corr + pe * __uint_as_float(w[e] & 0xffff0000u);
          }
        }
      }
    }
  }

  // ---- merge the warps
  if (lane == 0) {
    wm[warp] = m;
    wl[warp] = l;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t c = lane + 32u * j;
    if (c < n_chunks)
#pragma unroll
      for (int e = 0; e < 8; ++e) wo[warp][c * 8 + e] = acc[j][e];
  }
  __syncthreads();
  float mg = -INFINITY;
  for (int w = 0; w < GEN_WARPS; ++w) mg = fmaxf(mg, wm[w]);
  float wgt[GEN_WARPS];
  float lg = 0.f;
  for (int w = 0; w < GEN_WARPS; ++w) {
    wgt[w] = (wm[w] == -INFINITY) ? 0.f : exp2f(wm[w] - mg);
    lg += wgt[w] * wl[w];
  }
  const size_t orow = size_t(row) * p.Hq + h;
  for (uint32_t d = tid; d < D; d += GEN_WARPS * 32) {
    float o = 0.f;
    for (int w = 0; w < GEN_WARPS; ++w) o += wgt[w] * wo[w][d];
    if (p.out) {
      p.out[orow * D + d] = __float2bfloat16_rn(lg > 0.f ? o / lg : 0.f);
    } else {
      p.out_o[orow * D + d] = o;
    }
  }
  if (!p.out && tid == 0) {
    p.out_m[orow] = mg * 0.6931471805599453f;  // log2 units -> natural units
    p.out_l[orow] = lg;
  }
}

// Decoder bitmap uint8 [C][T] -> one bit per key, 128-key tiles [C][n_bits] of uint4, plus for every run of PACK_ROWS
// canvas rows and every tile whether any of the rows sees a key of it.  A CTA packs PACK_ROWS rows of one tile: four
// 32-byte reads per row and tile, all independent.
constexpr uint32_t PACK_ROWS = 32;
__global__ void __launch_bounds__(256) dg_pack_attend_kernel(const uint8_t* __restrict__ attend, uint32_t C, uint32_t T,
                                                             uint4* __restrict__ bits, uint8_t* __restrict__ live) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the kernels ahead may still read the previous call's bits
  const uint32_t j = blockIdx.x, n_bits = gridDim.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  uint32_t any = 0u;
#pragma unroll
  for (uint32_t k = 0; k < PACK_ROWS / 8u; ++k) {
    const uint32_t row = blockIdx.y * PACK_ROWS + k * 8u + warp;
    if (row >= C) continue;   // warp-uniform
    uint32_t w[4];
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
      const uint32_t t = j * 128u + e * 32u + lane;
      w[e] = __ballot_sync(0xffffffffu, t < T && attend[size_t(row) * T + t] != 0);
      any |= w[e];
    }
    if (lane == 0) bits[size_t(row) * n_bits + j] = make_uint4(w[0], w[1], w[2], w[3]);
  }
  any = __syncthreads_or(any != 0u);
  if (threadIdx.x == 0) live[size_t(blockIdx.y) * n_bits + j] = any ? 1 : 0;
}

uint32_t pack_attend_runs(uint32_t C) { return (C + PACK_ROWS - 1u) / PACK_ROWS; }
cudaError_t launch_pack_attend(const uint8_t* attend, uint32_t C, uint32_t T, uint4* bits, uint8_t* live, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((T + 127u) / 128u, pack_attend_runs(C));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, dg_pack_attend_kernel, attend, C, T, bits, live);
}

void launch_attn_general(const AttnParams& p, cudaStream_t st) {
  dg_attn_general_kernel<<<dim3(p.C, p.Hq), GEN_WARPS * 32, 0, st>>>(p);
}

// ------------------------------------------------------------------------------------------
// Local merge of n_parts partials -> bf16.  One warp per row; m in natural-log units.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) dg_merge_local_kernel(uint32_t n_parts, uint32_t rows, uint32_t D,
                                                              const float* __restrict__ o,
                                                              const float* __restrict__ m,
                                                              const float* __restrict__ l,
                                                              __nv_bfloat16* __restrict__ out) {
  const uint32_t row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  float mg = -INFINITY;
  for (uint32_t s = 0; s < n_parts; ++s) mg = fmaxf(mg, m[size_t(s) * rows + row]);
  float lg = 0.f;
  for (uint32_t s = 0; s < n_parts; ++s) {
    const float ms = m[size_t(s) * rows + row];
    lg += (ms == -INFINITY ? 0.f : expf(ms - mg)) * l[size_t(s) * rows + row];
  }
  for (uint32_t d = lane; d < D; d += 32) {
    float acc = 0.f;
    for (uint32_t s = 0; s < n_parts; ++s) {
      const float ms = m[size_t(s) * rows + row];
      const float w = ms == -INFINITY ? 0.f : expf(ms - mg);
      acc += w * o[(size_t(s) * rows + row) * D + d];
    }
    out[size_t(row) * D + d] = __float2bfloat16_rn(lg > 0.f ? acc / lg : 0.f);
  }
}

void launch_merge_local(uint32_t n_parts, uint32_t rows, uint32_t D, const float* o, const float* m,
                        const float* l, __nv_bfloat16* out, cudaStream_t st) {
  dg_merge_local_kernel<<<(rows + 3) / 4, 128, 0, st>>>(n_parts, rows, D, o, m, l, out);
}

// ------------------------------------------------------------------------------------------
// Cross-rank merge helpers.  Payload layout: pay[rows][D+1] = [O row | l]; m separate.
//   pack:     pay = [O | l] * exp(m_local - m_global)   (m_global already all-reduced into mg)
//   finalize: out = pay[:, :D] / pay[:, D]
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) dg_merge_pack_kernel(uint32_t rows, uint32_t D, const float* __restrict__ o,
                                                             const float* __restrict__ m_local,
                                                             const float* __restrict__ m_global,
                                                             const float* __restrict__ l, float* __restrict__ pay) {
  const uint32_t row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float ml = m_local[row], mg = m_global[row];
  const float w = (ml == -INFINITY) ? 0.f : expf(ml - mg);
  for (uint32_t d = lane; d < D; d += 32) pay[size_t(row) * (D + 1) + d] = w * o[size_t(row) * D + d];
  if (lane == 0) pay[size_t(row) * (D + 1) + D] = w * l[row];
}
__global__ void __launch_bounds__(128) dg_merge_finalize_kernel(uint32_t rows, uint32_t D, const float* __restrict__ pay,
                                                                 __nv_bfloat16* __restrict__ out) {
  const uint32_t row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float lg = pay[size_t(row) * (D + 1) + D];
  const float inv = lg > 0.f ? 1.0f / lg : 0.f;
  for (uint32_t d = lane; d < D; d += 32)
    out[size_t(row) * D + d] = __float2bfloat16_rn(pay[size_t(row) * (D + 1) + d] * inv);
}
void launch_merge_pack(uint32_t rows, uint32_t D, const float* o, const float* m_local, const float* m_global,
                       const float* l, float* pay, cudaStream_t st) {
  dg_merge_pack_kernel<<<(rows + 3) / 4, 128, 0, st>>>(rows, D, o, m_local, m_global, l, pay);
}
void launch_merge_finalize(uint32_t rows, uint32_t D, const float* pay, __nv_bfloat16* out, cudaStream_t st) {
  dg_merge_finalize_kernel<<<(rows + 3) / 4, 128, 0, st>>>(rows, D, pay, out);
}

// ------------------------------------------------------------------------------------------
// Visibility dump: the predicate of dg_common.cuh evaluated on the device.
// ------------------------------------------------------------------------------------------
__global__ void dg_visibility_kernel(MaskParams mk, uint32_t C, uint8_t* __restrict__ out) {
  const uint32_t T = mk.kv_len + C;
  const uint32_t row = blockIdx.y;
  const RowVis rv = mask_row(mk, row);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x)
    out[size_t(row) * T + t] = mask_visible_row(mk, rv, t) ? 1 : 0;
}
void launch_visibility(const MaskParams& mk, uint32_t C, uint8_t* out, cudaStream_t st) {
  const uint32_t T = mk.kv_len + C;
  uint32_t gx = (T + 255) / 256;
  if (gx > 1024) gx = 1024;
  dg_visibility_kernel<<<dim3(gx, C), 256, 0, st>>>(mk, C, out);
}

// ------------------------------------------------------------------------------------------
// Self-test of the bounded-wait / device-status path: one thread waits on a flag that nothing
// sets, gives up after `limit_cycles`, and reports DG_DEV_WAIT_TIMEOUT exactly like a kernel whose
// barrier wait ran out.  The context stays usable.
// ------------------------------------------------------------------------------------------
__global__ void dg_selftest_wait_kernel(volatile uint32_t* flag, long long limit_cycles, DevStatus* status) {
  const long long t0 = clock64();
  while (*flag == 0u) {
    if (clock64() - t0 > limit_cycles) {
      dev_status_set(status, DG_DEV_WAIT_TIMEOUT, KID_SELFTEST, blockIdx.x, 0u);
      return;
    }
  }
}
void launch_selftest_wait(uint32_t* flag, long long limit_cycles, DevStatus* status, cudaStream_t st) {
  dg_selftest_wait_kernel<<<1, 1, 0, st>>>(flag, limit_cycles, status);
}

// fill helpers for degenerate launches
__global__ void dg_fill_f32_kernel(float* p, float v, size_t n) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) p[i] = v;
}
void launch_fill_f32(float* p, float v, size_t n, cudaStream_t st) {
  if (n == 0) return;
  size_t g = (n + 255) / 256;
  if (g > 1024) g = 1024;
  dg_fill_f32_kernel<<<unsigned(g), 256, 0, st>>>(p, v, n);
}

}  // namespace dg
