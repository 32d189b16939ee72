// Pieces shared by the two tcgen05 attention kernels (attn_tc.cu: pairs of query tiles, attn_small.cu:
// single query tiles): output destinations, the packed fp32 softmax arithmetic, the epilogue row store.
#pragma once

#include "tc_common.cuh"

namespace svoo {
namespace tc {

// Optional destination of the output rows on other GPUs: row n of local head bh goes to rank
// n / n_loc, row n % n_loc, head head[bh] of that rank's [n_loc, H, 128] array.  n_loc == 0: the
// rows go to `out` of this GPU.
struct OutPeers {
  bf16* dst[16];
  int n_loc;
  int H;
  int16_t head[128];
};
// O is rescaled only when a row maximum grows by more than 2^8: the running sum keeps the same stale
// maximum, so the final normalisation is exact.
constexpr float kRescaleThreshold = 8.0f;

// Packed fp32 pairs (one instruction for two lanes of data): x = s * scale + neg_m and the
// running pair of row sums.
__device__ __forceinline__ void fma2(float& x0, float& x1, uint32_t a0, uint32_t a1, uint64_t scale2, uint64_t negm2) {
  asm("{\n\t.reg .b64 a, x;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "fma.rn.f32x2 x, a, %4, %5;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}\n"
      : "=f"(x0), "=f"(x1) : "r"(a0), "r"(a1), "l"(scale2), "l"(negm2));
}
__device__ __forceinline__ void add2(uint64_t& acc, float p0, float p1) {
  asm("{\n\t.reg .b64 p;\n\t"
      "mov.b64 p, {%1, %2};\n\t"
      "add.rn.f32x2 %0, %0, p;\n\t}\n"
      : "+l"(acc) : "f"(p0), "f"(p1));
}
__device__ __forceinline__ uint64_t pair2(float v) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float pair_sum(uint64_t acc) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(acc));
  return a + b;
}
// 16 columns: p = exp2(s * scale + neg_m) -> 8 packed bf16 pairs, row sums into `acc`.
__device__ __forceinline__ void exp_pack16(const uint32_t (&r)[16], uint32_t* pk, uint64_t scale2, uint64_t negm2,
                                           uint64_t& acc) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float x0, x1;
    fma2(x0, x1, r[2 * i], r[2 * i + 1], scale2, negm2);
    const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
    add2(acc, p0, p1);
    pk[i] = pack_bf16x2(p0, p1);
  }
}

// CTA index -> (head, tile of the head's list).  The last kHoist tiles of every head's list go first.  Tiles are in
// cluster order and the text blocks come last, so where the whole text is prompt these are the prompt's query tiles,
// which attend to every key (720p HunyuanVideo: 930 key tiles against 160 on average) and would otherwise be started
// last.  A partly used prompt whose unused rows have a tile in the same list keeps its place at the end of the
// head.  After them the heads follow one another, so that the CTAs in flight share a head's K and V in L2, by
// decreasing work, so that the last CTAs are short ones.  counts: (pairs, singles) of every head.
template <int kHoist>
__device__ __forceinline__ bool pick_tile(int id, int BH, int per_head, const int32_t* counts, const int32_t* order, int which,
                                          int& bh, int& t) {
  const int hoist = per_head < kHoist ? per_head : kHoist;
  if (id < BH * hoist) {
    bh = order[id % BH];
    t = counts[2 * bh + which] - 1 - id / BH;
    return t >= 0;
  }
  id -= BH * hoist;
  const int nth = id / (per_head - hoist);
  bh = order[nth];
  t = id - nth * (per_head - hoist);
  return t < counts[2 * bh + which] - hoist;
}

// Run table in shared memory: entry r = (first row, virtual begin) for r < nr, entry nr = (0, L).
// Moves `cur` on to the run that holds virtual row v0 < L (it only ever grows).  Whole warp.
__device__ __forceinline__ void advance_run(const int2* runs_s, int nr, int v0, int lane, int& cur) {
  for (;;) {
    const int n = cur + 1 + lane;
    const int passed = __popc(__ballot_sync(0xffffffffu, n <= nr && runs_s[min(n, nr)].y <= v0));
    cur += passed;
    if (passed < 32) return;
  }
}
// Source row (relative to the head) of virtual row v0 + lane, -1 past the last one.  Whole warp.
__device__ __forceinline__ int gather_source(const int2* runs_s, int nr, int L, int v0, int lane, int& cur) {
  if (v0 >= L) return -1;
  advance_run(runs_s, nr, v0, lane, cur);
  const int n = cur + 1 + lane;                          // bit d: a run begins at row v0 + d (runs are not empty)
  const int d = n <= nr ? runs_s[n].y - v0 : 32;
  const unsigned begins = __reduce_or_sync(0xffffffffu, d < 32 ? 1u << d : 0u);
  const int r = cur + __popc(begins & (0xffffffffu >> (31 - lane)));
  return v0 + lane < L ? runs_s[r].x + (v0 + lane - runs_s[r].y) : -1;
}
// Copies the 32 rows `src` (lane r: source row of tile row row0 + r, -1: zeros) into a tile of two
// 64-column halves of `half_bytes` each, 128-byte swizzle.  Lane l copies chunk l % 16 of every other row;
// `dst` and `src_base` already include that chunk's half and column.
__device__ __forceinline__ void gather_rows32(uint32_t dst, const bf16* src_base, int src, int row0, int lane) {
  const int chunk = lane & 15;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = 2 * i + (lane >> 4), row = row0 + r;
    const int s = __shfl_sync(0xffffffffu, src, r);
    cp_async16(dst + row * 128 + (((chunk & 7) ^ (row & 7)) << 4), src_base + (int64_t)max(s, 0) * kHeadDim, s >= 0);
  }
}

// Row `dst` of head bh in the output: this GPU's tensor or the owning rank's sequence shard.
__device__ __forceinline__ bf16* out_row(const OutPeers& peers, bf16* out, int bh, int S, int dst) {
  if (peers.n_loc == 0) return out + ((int64_t)bh * S + dst) * kHeadDim;
  const int p = dst / peers.n_loc;
  return peers.dst[p] + ((int64_t)(dst - p * peers.n_loc) * peers.H + peers.head[bh]) * kHeadDim;
}

}  // namespace tc
}  // namespace svoo
