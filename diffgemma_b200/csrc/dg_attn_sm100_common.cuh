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
