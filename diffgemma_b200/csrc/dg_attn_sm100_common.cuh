// Definitions of the head_dim-256 attention kernel that the host side shares: tile geometry,
// shared-memory map, key-tile schedule, phase stamps.
#pragma once
#include <cuda.h>

#include "dg_common.cuh"
#include "sm100_ptx.cuh"

namespace dg {
namespace sm100 {


constexpr uint32_t BM = 128;            // query rows per CTA
constexpr uint32_t BN = 128;            // keys per tile
constexpr uint32_t HD = 256;            // head_dim
constexpr uint32_t ATOM_BYTES = 128 * 128;        // 128 rows x 128 B (64 bf16): one swizzle-atom column
constexpr uint32_t TILE_BYTES = 4 * ATOM_BYTES;   // 128 rows x 256 bf16
constexpr uint32_t OFF_Q = 0;
constexpr uint32_t OFF_K = TILE_BYTES;
constexpr uint32_t OFF_V = 2 * TILE_BYTES;
constexpr uint32_t OFF_BAR = 3 * TILE_BYTES;
constexpr uint32_t OFF_XCH = OFF_BAR + 256;             // row-group exchange scratch (8 KB)
constexpr uint32_t OFF_LIVE = OFF_XCH + 8192;           // bitmap form: live-tile words
constexpr uint32_t HBUF_LD = 264;                       // halves of a staged row: 256 and 16 bytes (padding, or m, l, 1 / scale)
constexpr uint32_t ROW_BYTES = HBUF_LD * 2;
constexpr uint32_t OFF_STAGE = 72 * 1024;               // partial rows on their way out; what comes in lies at OFF_Q
static_assert(BM * ROW_BYTES <= OFF_STAGE && OFF_STAGE + BM * ROW_BYTES <= OFF_BAR, "exchange buffers");
constexpr uint32_t SMEM_BYTES = OFF_LIVE + 2048 + 1024;   // + alignment slack
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t TM_S = 0;            // two S buffers of 128 columns
constexpr uint32_t TM_O = 256;          // O accumulator, 256 columns
constexpr float RESCALE_THRESHOLD = 8.0f;   // log2 units

struct TileSched {
  uint32_t a0, nA, b0, nB;
};
// Key tiles (absolute index = key / 128) a CTA whose canvas rows are [row_first, row_last] must visit:
// the prefix interval [lo(row_first), pre_hi) and the canvas interval [kv_len, can_hi) - in the causal
// mode only up to row_last's own position -, merged when they touch.  (The lower bounds grow with the
// row, the causal upper bound too, so the first row gives the lowest key and the last row the highest.)
__host__ __device__ inline TileSched tile_sched(const MaskParams& mk, uint32_t row_first, uint32_t row_last) {
  TileSched t{0, 0, 0, 0};
  const uint32_t lo = mask_row_lo(mk, row_first);
  if (mk.pre_hi > lo) {
    t.a0 = lo / BN;
    t.nA = (mk.pre_hi + BN - 1) / BN - t.a0;
  }
  const uint32_t can_hi = mask_can_hi_rows(mk, row_last);
  if (can_hi > mk.kv_len) {
    const uint32_t b0 = mk.kv_len / BN, b1 = (can_hi + BN - 1) / BN;
    if (t.nA > 0 && b0 < t.a0 + t.nA) {
      const uint32_t a1 = (t.a0 + t.nA) > b1 ? (t.a0 + t.nA) : b1;
      t.nA = a1 - t.a0;
    } else {
      t.b0 = b0;
      t.nB = b1 - b0;
    }
  }
  return t;
}

// Key tiles of a launch under a decoder bitmap (p.bits): the 128-key tiles in which any canvas row sees a key, as a
// bit per tile in shared memory, so that padding and windows expressed as a bitmap cost no tile visits.
constexpr uint32_t LIVE_WORDS = 32;                       // up to 1,024 tiles = 131,072 keys; longer ranges visit every tile
__device__ __forceinline__ void build_live_words(const AttnParams& p, uint32_t* live) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, n_warps = blockDim.x >> 5;
  for (uint32_t w = warp; w < LIVE_WORDS; w += n_warps) {
    const uint32_t j = w * 32u + lane;
    uint32_t any = 0u;
    if (j < p.n_bits)
      for (uint32_t c = 0; c < p.n_live_rows; ++c) any |= p.bits_live[size_t(c) * p.n_bits + j];
    const uint32_t word = __ballot_sync(0xffffffffu, any != 0u);
    if (lane == 0) live[w] = word;
  }
}
__device__ __forceinline__ uint32_t count_live_tiles(const AttnParams& p, const uint32_t* live) {
  if (p.n_bits > LIVE_WORDS * 32u) return p.n_bits;
  uint32_t n = 0;
  for (uint32_t w = 0; w * 32u < p.n_bits; ++w) n += __popc(live[w]);
  return n;
}

// Hands out a CTA's key tiles in order, starting with number v of its schedule.  With BITS the schedule is the live
// tiles, else the two intervals of TileSched.
template <bool BITS>
struct TileWalk {
  TileSched ts;
  uint32_t v;
  const uint32_t* live = nullptr;
  uint32_t word = 0, w = 0;
  __device__ __forceinline__ TileWalk(const AttnParams& p, const TileSched& t, const uint32_t* live_words, uint32_t v0) : ts(t), v(v0) {
    if (BITS && p.n_bits <= LIVE_WORDS * 32u) {
      live = live_words;
      word = live[0];
      uint32_t skip = v0;
      while (w + 1u < LIVE_WORDS && skip >= uint32_t(__popc(word))) {
        skip -= __popc(word);
        word = live[++w];
      }
      for (; skip > 0u; --skip) word &= word - 1u;
    }
  }
  __device__ __forceinline__ uint32_t next() {
    if (BITS && live != nullptr) {
      while (word == 0u && w + 1u < LIVE_WORDS) word = live[++w];
      const uint32_t b = word ? __ffs(word) - 1u : 0u;
      word &= word - 1u;
      return w * 32u + b;
    }
    const uint32_t n = v++;
    return n < ts.nA ? ts.a0 + n : ts.b0 + (n - ts.nA);
  }
};

// The same for the 64-key tiles of the head_dim-512 kernels: both halves of every 128-key tile.
struct TileWalk64Bits {
  TileWalk<true> walk;
  uint32_t half, cur = 0;
  __device__ __forceinline__ TileWalk64Bits(const AttnParams& p, const TileSched& t, const uint32_t* live_words, uint32_t v0)
      : walk(p, t, live_words, v0 >> 1), half(v0 & 1u) {
    if (half) cur = walk.next();
  }
  __device__ __forceinline__ uint32_t next() {
    if (half == 0u) cur = walk.next();
    const uint32_t jt = 2u * cur + half;
    half ^= 1u;
    return jt;
  }
};

// ------------------------------------------------------------------------------------------
// A bitmap hides keys whose K and V rows need not hold numbers (padding that was never written).  The general kernel does
// not look at them; here every value row of a visited tile is multiplied by its P, and 0 * inf and 0 * NaN are NaN: a
// row that meets one comes out non-finite in some column, whatever it sees.  So the CTA that stores rows of the output
// notes whether one is not finite, and if any is, a warp computes each of those again over the keys it sees and no others,
// the general kernel's way, which is also what it gives where a visible key is infinite or NaN.  (317 keys, 17 canvas rows:
// 21.5 us without the note, 21.7 with it, 22.8 with a kernel behind this one that looked through the rows.)
// ------------------------------------------------------------------------------------------
// The largest magnitude among the bf16 values seen, as bits, in either half of a word: two instructions a word.
struct Bf16Max {
  uint32_t m = 0u;
  __device__ __forceinline__ void add(const uint4 x) {
    m = __vmaxu2(m, __vmaxu2(__vmaxu2(x.x & 0x7fff7fffu, x.y & 0x7fff7fffu), __vmaxu2(x.z & 0x7fff7fffu, x.w & 0x7fff7fffu)));
  }
  __device__ __forceinline__ bool nonfinite() const { return (m & 0xffffu) >= 0x7f80u || m >= 0x7f800000u; }
};

// Rows [lo, hi) of query tile mt, columns [col0, col0 + 256), all stored by this CTA ahead of a barrier; head_dim 256 NS.
template <uint32_t NS>
__device__ __noinline__ void bitmap_rows_again(const AttnParams& p, uint32_t kvh, uint32_t mt, uint32_t lo, uint32_t hi, uint32_t col0,
                                               volatile uint32_t* abort_flag) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, n_warps = blockDim.x >> 5;
  constexpr uint32_t D = 256u * NS;
  auto warp_sum = [](float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  auto unpack = [](const uint4 x, float* f) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f[2 * e] = __uint_as_float(w[e] << 16);
      f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
    }
  };
  // the canvas rows of the cache may be other CTAs' shares of the in-launch append
  if (p.ap_vectors != 0u && !__all_sync(0xffffffffu, wait_counter_gpu(p.ap_ctl + 1, p.ap_vectors, abort_flag))) {
    if (lane == 0) dev_status_set(p.status, DG_DEV_WAIT_TIMEOUT, KID_SM100, blockIdx.x + gridDim.x * blockIdx.y, p.ap_vectors);
    return;
  }
#pragma unroll 1
  for (uint32_t rl = lo + warp; rl < hi; rl += n_warps) {
    const uint32_t R = mt * BM + rl;
    if (R >= p.C * p.G) return;
    const uint32_t row = R / p.G, h = kvh * p.G + R % p.G;
    uint4* out = reinterpret_cast<uint4*>(p.out + (size_t(row) * p.Hq + h) * D + col0) + lane;
    Bf16Max largest;
    largest.add(*out);
    if (!__any_sync(0xffffffffu, largest.nonfinite())) continue;
    // Q, chunk lane + 32 j: as staged, or normed and rotated here (partners are sixteen lanes apart)
    float q[NS][8];
    const uint4* qs = reinterpret_cast<const uint4*>(p.q + (size_t(row) * p.Hq + h) * D) + lane;
#pragma unroll
    for (uint32_t j = 0; j < NS; ++j) unpack(qs[32u * j], q[j]);
    if (NS == 1 && !p.q_prenormed) {
      float ss = 0.f, w[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += q[0][e] * q[0][e];
      if (p.qw) unpack(reinterpret_cast<const uint4*>(p.qw)[lane], w);
      const float inv = 1.0f / sqrtf(warp_sum(ss) / float(D) + p.eps);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float x = q[0][e] * (inv * w[e]), y = __shfl_xor_sync(0xffffffffu, x, 16);
        const float2 cs = p.rope_table[size_t(row) * 128u + (lane & 15u) * 8u + e];
        q[0][e] = __bfloat162float(__float2bfloat16_rn(lane < 16u ? x * cs.x - y * cs.y : y * cs.y + x * cs.x));
      }
    }
    const uint4* K = reinterpret_cast<const uint4*>(p.cache_k + size_t(kvh) * p.cap * D) + lane;
    const uint4* V = reinterpret_cast<const uint4*>(p.cache_v + size_t(kvh) * p.cap * D + col0) + lane;
    float m = -INFINITY, l = 0.f, acc[8] = {};
#pragma unroll 1
    for (uint32_t t32 = 0; t32 < p.n_bits * 4u; ++t32) {
      uint32_t seen = reinterpret_cast<const uint32_t*>(p.bits + size_t(row) * p.n_bits)[t32];
      for (; seen != 0u; seen &= seen - 1u) {
        const size_t slot = ((t32 * 32u + __ffs(seen) - 1u) - p.pos_base) & p.ring_mask;
        float dot = 0.f, x[8];
#pragma unroll
        for (uint32_t j = 0; j < NS; ++j) {
          unpack(__ldcg(K + slot * (D / 8u) + 32u * j), x);
#pragma unroll
          for (int e = 0; e < 8; ++e) dot += q[j][e] * x[e];
        }
        const float s2 = warp_sum(dot) * p.scale_log2, mn = fmaxf(m, s2), corr = exp2f(m - mn), pe = exp2f(s2 - mn);
        l = l * corr + pe;
        m = mn;
        unpack(__ldcg(V + slot * (D / 8u)), x);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = acc[e] * corr + pe * x[e];
      }
    }
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = pack_bf16x2(l > 0.f ? acc[2 * e] / l : 0.f, l > 0.f ? acc[2 * e + 1] / l : 0.f);
    *out = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ uint32_t bar_addr(uint32_t bar_base, uint32_t idx) { return bar_base + idx * 8u; }

// Phase time stamps (globaltimer, ns) of one CTA, written by thread 0 when a stamp buffer is given:
// 0 start, 1 set-up done, 2 Q prologue done, 3 main loop done, 4 epilogue done, 5 merge done.
// Slots 6-11 hold SM-clock cycles that single threads spent waiting inside the key loop:
// 6 MMA issuer on K tiles, 7 on V tiles, 8 on P (softmax output), 9 its whole loop,
// 10 softmax thread 0 on S (scores), 11 softmax thread 0 on the rescale barrier.
// Slots 12-14 are time stamps inside the tail: 12 the last PV has completed, 13 this CTA's partial rows are staged
// (cluster merge only), 14 the other splits' rows have arrived.  15: this CTA's part of the in-launch append is done.
constexpr uint32_t STAMP_SLOTS = 16;
__device__ __forceinline__ void stamp(const AttnParams& p, uint32_t slot) {
  if (p.stamps != nullptr && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    p.stamps[((size_t(blockIdx.z) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * STAMP_SLOTS + slot] = t;
  }
}
__device__ __forceinline__ void stamp_cycles(const AttnParams& p, uint32_t slot, long long cycles) {
  if (p.stamps != nullptr)
    p.stamps[((size_t(blockIdx.z) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * STAMP_SLOTS + slot] = (unsigned long long)cycles;
}
// runs a wait and, when profiling, adds the cycles it took to acc
template <class F>
__device__ __forceinline__ bool timed_wait(bool prof, long long& acc, F f) {
  if (!prof) return f();
  const long long t = clock64();
  const bool r = f();
  acc += clock64() - t;
  return r;
}


}  // namespace sm100
}  // namespace dg
