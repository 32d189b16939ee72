// Block-sparse attention for query tiles that stand alone (at most 128 rows: small query clusters and the
// tails of larger ones), tcgen05 + TMEM.
//
// attn_tc.cu owns pairs of query tiles: one CTA per SM, two softmax warpgroups that hide each other's
// latency, K and V by TMA boxes.  A single tile in that kernel leaves half of the CTA idle and pays for
// every wait.  Here a CTA owns one query tile and walks 64-key steps with 102 KB of shared memory (106 KB
// in the EAR form) and 256 TMEM columns, so that TWO CTAs share an SM and cover each other's waits, start and end.
//
//   warps 0-3   softmax: thread r owns row r; S -> registers, row max, exp2, row sum, P packed to bf16
//               over the S columns it came from
//   warp 4      MMA issuer: S = Q K^T into one of two S buffers, O += P V with P read from TMEM
//   warps 5-6   K loaders, warps 7-8 V loaders: cp.async row gathers into two-stage rings
//
// The rows of K and V are gathered with cp.async, not TMA: with 256 / 1024 clusters a run of selected
// rows is a handful of rows long and a 128-key tile takes about 35 TMA boxes per tensor, which at 113
// cycles a box is the whole time (hunyuan-shaped layer, 24 heads x 8,505 tokens: 4.5 us per tile against
// 1.9 us when the same number of selected rows is contiguous).  A gather costs the same for any run.
//
// The softmax takes its maximum over 128 keys (two steps), as the pair kernel does, and adds in the same order, so that
// a row comes out the same bit for bit in either kernel.  A maximum per 64-key step would be simpler, but the key that is
// the maximum has P = 1, which bf16 holds exactly, and is found in the first step less often: 0.5 % more error
// against 64 bits at 4 heads x 960 tokens.
#include "attn_common.cuh"

namespace svoo {
namespace tc {

constexpr int kSmBN = 64;                              // keys per step
constexpr int kSmQBytes = 128 * kRowBytes;             // 32 KB: two halves of 128 rows x 64 columns
constexpr int kSmQHalf = 128 * 128;
constexpr int kSmTile = kSmBN * kRowBytes;             // 16 KB: two halves of 64 rows x 64 columns
constexpr int kSmHalf = kSmBN * 128;
constexpr int kSmTiles = kSmQBytes + 4 * kSmTile;      // Q | K0 K1 | V0 V1
constexpr int kSmThreads = 9 * 32;
constexpr int kSmMmaWarp = 4, kSmKWarp = 5, kSmVWarp = 7;
template <bool kEar>
struct SmallSmem {
  static constexpr int kMaxRuns = SVOO_MAX_ATTN_CLUSTERS / 2 + (kEar ? 4 : 2);      // see AttnSmem in attn_tc.cu
  static constexpr int kRunTableBytes = (kMaxRuns * 8 + 255) / 256 * 256;
  static constexpr int kBiasFloats = kEar ? SVOO_MAX_ATTN_CLUSTERS + kSmBN + 6 : 0;
  static constexpr int kBiasBytes = (kBiasFloats * 4 + 255) / 256 * 256;
  static constexpr int kBytes = kSmTiles + 256 + kRunTableBytes + kBiasBytes + 1024;
};
static_assert(2 * (SmallSmem<true>::kBytes + 1024) <= 228 * 1024, "two CTAs share an SM");

// PV_DONE has one barrier per step parity because the softmax does not wait for every PV: when it has S of
// step j, the PV of step j - 2 is known to be complete (S of step j was issued after it).
enum SmBar { SM_Q_FULL = 0, SM_K_FULL = 1, SM_K_EMPTY = 3, SM_V_FULL = 5, SM_V_EMPTY = 7, SM_S_FULL = 9, SM_P_READY = 11,
             SM_PV_DONE = 13, SM_NUM_BARS = 15 };
// TMEM columns: two S buffers (P of a step overwrites the first half of its S buffer), then O.
constexpr uint32_t kSmColO = 128;

template <bool kEar>
__global__ void __launch_bounds__(kSmThreads, 2) sparse_attn_small_kernel(
    const __grid_constant__ CUtensorMap q_map, const __grid_constant__ OutPeers peers, const bf16* __restrict__ k,
    const bf16* __restrict__ v, bf16* __restrict__ out, const int32_t* __restrict__ out_row_idx,
    const int4* __restrict__ qtiles, const int32_t* __restrict__ nqtiles,
    const int32_t* __restrict__ head_order, const int2* __restrict__ runs,
    const int32_t* __restrict__ nruns, int BH, int S, int QC, int max_tiles, int max_runs, float scale_log2,
    int32_t* __restrict__ status, float* __restrict__ lse, const uint8_t* __restrict__ map,
    const int32_t* __restrict__ k_offsets, int KC) {
  constexpr int kMaxRunsSmem = SmallSmem<kEar>::kMaxRuns;
  extern __shared__ unsigned char smem_raw[];
  // The kernel may start while the pair kernel before it drains (it reads nothing that one writes); its
  // last CTA waits for that grid, so that this kernel's completion covers both.
  const bool last_cta = blockIdx.x == gridDim.x - 1;
  int bh, t;
  if (!pick_tile<2>((int)blockIdx.x, BH, QC, nqtiles, head_order, 1, bh, t)) {
    if (last_cta) pdl_wait();
    return;
  }
  const int4 tile = qtiles[(int64_t)bh * max_tiles + (max_tiles - QC) + t];
  const int qi = tile.x, row0 = tile.y, row1 = tile.z;
  const int nr = min(nruns[(int64_t)bh * QC + qi], kMaxRunsSmem - 1);
  const int2* rl = runs + ((int64_t)bh * QC + qi) * max_runs;
  const bool m64 = row1 - row0 <= 64;                    // M = 64 MMAs: row i in TMEM lane (i % 16) + 32 (i / 16)

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_s = base, k_s = base + kSmQBytes, v_s = k_s + 2 * kSmTile;
  const uint32_t bars = base + kSmTiles;
  unsigned char* gen_base = smem_raw + (base - smem_u32(smem_raw));
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen_base + kSmTiles + SM_NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_base + kSmTiles + SM_NUM_BARS * 8 + 8);
  int2* runs_s = reinterpret_cast<int2*>(gen_base + kSmTiles + 256);
  float* bias_s = reinterpret_cast<float*>(gen_base + kSmTiles + 256 + SmallSmem<kEar>::kRunTableBytes);
  auto bar = [&](int i) { return bars + 8u * i; };

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  if (tid == 0) {
    for (int i = 0; i < SM_NUM_BARS; ++i) {
      int count = 1;
      if (i == SM_P_READY || i == SM_P_READY + 1) count = 4;                              // one per softmax warp
      if (i == SM_K_FULL || i == SM_K_FULL + 1 || i == SM_V_FULL || i == SM_V_FULL + 1) count = 2;   // one per loader warp
      mbar_init(bar(i), count);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(bar(SM_Q_FULL), kSmQBytes);           // rows past the tile are other clusters' rows or zeros: never stored
    for (int h = 0; h < 2; ++h) tma_load_2d(q_s + h * kSmQHalf, &q_map, h * 64, bh * S + row0, bar(SM_Q_FULL));
  }
  for (int i = tid; i <= nr; i += kSmThreads) runs_s[i] = rl[i];
  if (warp == kSmMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int L = runs_s[nr].y;                            // selected key rows in total
  const int T = (L + kSmBN - 1) / kSmBN;
  int l_tok = L, bias0 = L;                              // centroid keys and their bias: as in attn_tc.cu
  if (kEar) {
    l_tok = nr > 0 ? runs_s[nr - 1].y : L;
    bias0 = l_tok / kSmBN * kSmBN;
    const int32_t* ko = k_offsets + (int64_t)bh * (KC + 1);
    const uint8_t* mrow = map + ((int64_t)bh * QC + qi) * KC;
    for (int x = bias0 + tid; x < L; x += kSmThreads) {
      float b = 0.f;
      if (x >= l_tok) {
        const int j = min(x - l_tok, KC - 1);
        b = mrow[j] ? -INFINITY : __log2f((float)(ko[j + 1] - ko[j]) + 1e-6f) / scale_log2;
      }
      bias_s[x - bias0] = b;
    }
    __syncthreads();
  }

  if (warp >= kSmKWarp) {
    // ---------------------------------------------------------------- K / V loaders
    // Warp `half` of the pair gathers rows [32 half, 32 half + 32) of every step: lane r looks up the
    // source row of tile row r, then 16 lanes copy each row.  The copies of step j are waited for, made
    // visible to the tensor core and reported after those of step j + 1 are issued, or at once when the
    // ring has no free stage (the tensor core may be waiting for exactly these).
    const bool is_v = warp >= kSmVWarp;
    const int half = (warp - kSmKWarp) & 1, chunk = lane & 15;
    const bf16* src_base = (is_v ? v : k) + (int64_t)bh * S * kHeadDim + chunk * 8;
    const uint32_t stage0 = (is_v ? v_s : k_s) + (chunk >> 3) * kSmHalf;
    const int full = is_v ? SM_V_FULL : SM_K_FULL, empty = is_v ? SM_V_EMPTY : SM_K_EMPTY;
    auto report = [&](int stage) {
      fence_async_proxy();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(full + stage));
    };
    int cur = 0;
    bool pending = false;
    for (int j = 0; j < T; ++j) {
      const int st = j & 1;
      const uint32_t par = ((j >> 1) & 1) ^ 1;
      const int src = gather_source(runs_s, nr, L, j * kSmBN + half * 32, lane, cur);
      if (!__all_sync(0xffffffffu, mbar_test_wait(bar(empty + st), par))) {
        if (pending) {
          cp_async_wait<0>();
          report(st ^ 1);
          pending = false;
        }
        if (!__all_sync(0xffffffffu, mbar_wait(bar(empty + st), par, abort_flag))) break;
      }
      gather_rows32(stage0 + st * kSmTile, src_base, src, half * 32, lane);
      cp_async_commit();
      if (pending) {
        cp_async_wait<1>();
        report(st ^ 1);
      }
      pending = true;
    }
    cp_async_wait<0>();
    if (pending) report((T - 1) & 1);
  } else if (warp == kSmMmaWarp) {
    // ---------------------------------------------------------------- MMA issuer
    // QK of step j + 2 overwrites the S buffer that holds P of step j, so it is issued when the PV that reads
    // that P has completed: the order of two MMAs is only promised for one accumulator and shape.  The
    // softmax is at work on step j + 1 meanwhile, and the other CTA of the SM on its own steps.
    if (lane == 0 && T > 0) {
      constexpr uint32_t kDescHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
      const uint32_t q_lo = ((q_s & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t k_lo = ((k_s & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t v_lo = ((v_s & 0x3FFFFu) >> 4) | ((uint32_t)(kSmHalf >> 4) << 16);
      const uint32_t idesc_qk = idesc_bf16(m64 ? 64 : 128, kSmBN, false);
      const uint32_t idesc_pv = idesc_bf16(m64 ? 64 : 128, kHeadDim, true);
      auto qk = [&](int j) -> bool {
        const int st = j & 1;
        if (!mbar_wait(bar(SM_K_FULL + st), (j >> 1) & 1, abort_flag)) return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_ss_lo(tmem + st * kSmBN, q_lo + (((ks >> 2) * kSmQHalf + (ks & 3) * 32) >> 4),
                     k_lo + ((st * kSmTile + (ks >> 2) * kSmHalf + (ks & 3) * 32) >> 4), kDescHi, idesc_qk, ks > 0);
        tc_commit(bar(SM_S_FULL + st));
        tc_commit(bar(SM_K_EMPTY + st));
        return true;
      };
      bool ok = mbar_wait(bar(SM_Q_FULL), 0, abort_flag) && qk(0);
      if (ok && T > 1) ok = qk(1);
      for (int j = 0; ok && j < T; ++j) {
        const int st = j & 1;
        ok = mbar_wait(bar(SM_V_FULL + st), (j >> 1) & 1, abort_flag) &&
             mbar_wait(bar(SM_P_READY + st), (j >> 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_ts_lo(tmem + kSmColO, tmem + st * kSmBN + ks * 8, v_lo + ((st * kSmTile + ks * 2048) >> 4), kDescHi, idesc_pv,
                     (j > 0 || ks > 0) ? 1u : 0u);
        tc_commit(bar(SM_V_EMPTY + st));
        tc_commit(bar(SM_PV_DONE + st));
        if (j + 2 < T) ok = mbar_wait(bar(SM_PV_DONE + st), (j >> 1) & 1, abort_flag) && qk(j + 2);
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax + epilogue
    const int r_local = m64 ? warp * 16 + (lane & 15) : tid;     // row of the query tile served by this TMEM lane
    const bool lane_has_row = !m64 || lane < 16;
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    const uint32_t o_t = tmem + lane_addr + kSmColO;
    float m_used = -INFINITY, l_sum = 0.f;
    bool ok = true;
    const uint64_t scale2 = pair2(scale_log2);
    const int bias_step = l_tok / kSmBN;                          // first step with centroid keys (EAR)
    // f(c, scores [16 c, 16 c + 16) of step j) for the four quarters of a step in order, bias and end of the list applied;
    // a quarter is read while the one before it is worked on.
    auto quarters = [&](int j, auto f) {
      const uint32_t s_t = tmem + lane_addr + (j & 1) * kSmBN;
      const bool biased = kEar && j >= bias_step;
      uint32_t sc[2][16];
      tmem_ld16_nowait(s_t, sc[0]);
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t(&x)[16] = sc[c & 1];
        if (c < 3) tmem_ld16_nowait(s_t + 16 * (c + 1), sc[(c + 1) & 1]);
        if (biased) {
          const uint32_t bj = base + kSmTiles + 256 + SmallSmem<kEar>::kRunTableBytes + 4u * ((j - bias_step) * kSmBN + c * 16);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float b0, b1;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(b0), "=f"(b1) : "r"(bj + 4 * i));
            x[i] = __float_as_uint(__uint_as_float(x[i]) + b0);
            x[i + 1] = __float_as_uint(__uint_as_float(x[i + 1]) + b1);
          }
        }
        const int valid = L - j * kSmBN - c * 16;
        if (valid < 16) {                                         // last step only: columns past the last key
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i >= valid) x[i] = 0xff800000u;
        }
        f(c, x);
        tmem_wait_ld();
      }
    };
    auto max16 = [](const uint32_t (&x)[16], float& m0, float& m1) {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        m0 = fmaxf(m0, fmaxf(__uint_as_float(x[i]), __uint_as_float(x[i + 1])));
        m1 = fmaxf(m1, fmaxf(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])));
      }
    };
    // 128 keys: both steps' maxima decide on the maximum before any of their P goes to the tensor core.  It rarely
    // changes after the first 128 keys, so the first step's P is computed on the old one while the second step's S is
    // still being formed, kept in registers, and computed again if the maximum did change.  Whether the first step changes
    // it is looked at only where its P add up to more than 250: one above 2^8 would.
    for (int j0 = 0; j0 < T; j0 += 2) {
      const uint32_t par = (j0 >> 1) & 1;
      const int n = min(T - j0, 2);
      uint32_t pk[32];
      uint64_t acc = 0;                                           // two fp32 zeros
      float m0 = -INFINITY, m1 = -INFINITY;
      ok = __all_sync(0xffffffffu, mbar_wait(bar(SM_S_FULL), par, abort_flag));
      if (!ok) break;
      tc_fence_after();
      bool have_p = j0 > 0;
      int u0 = 0;                                                 // steps [u0, n) are searched for their maximum
      if (have_p) {
        quarters(j0, [&](int c, const uint32_t (&x)[16]) { exp_pack16(x, &pk[c * 8], scale2, pair2(-m_used), acc); });
        u0 = __any_sync(0xffffffffu, lane_has_row && !(pair_sum(acc) <= 250.f)) ? 0 : 1;
      }
#pragma unroll 1
      for (int u = u0; u < n; ++u) {
        if (u == 1) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar(SM_S_FULL + 1), par, abort_flag));
          if (!ok) break;
          tc_fence_after();
        }
        quarters(j0 + u, [&](int, const uint32_t (&x)[16]) { max16(x, m0, m1); });
      }
      if (!ok) break;
      const float m_tile = fmaxf(m0, m1) * scale_log2;            // the scale is positive
      if (j0 == 0) {
        m_used = kEar ? fmaxf(m_tile, -1e30f) : m_tile;           // EAR: first steps of masked centroids only
      } else {
        const bool need = lane_has_row && m_tile > m_used + kRescaleThreshold;
        if (__any_sync(0xffffffffu, need)) {                      // rare: rescale O once the previous PV is complete
          ok = __all_sync(0xffffffffu, mbar_wait(bar(SM_PV_DONE + 1), par ^ 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
          const float alpha = need ? fast_exp2(m_used - m_tile) : 1.0f;
#pragma unroll 1
          for (int ch = 0; ch < 16; ++ch) {
            uint32_t x[8];
            tmem_ld8(o_t + ch * 8, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * alpha);
            tmem_st8(o_t + ch * 8, x);
          }
          l_sum *= alpha;
          if (need) m_used = m_tile;
          have_p = false;
        }
      }
      const uint64_t negm2 = pair2(-m_used);
      auto hand_over = [&](int u) {                               // P over the S it came from
        tmem_st16(tmem + lane_addr + u * kSmBN, *reinterpret_cast<const uint32_t(*)[16]>(&pk[0]));
        tmem_st16(tmem + lane_addr + u * kSmBN + 16, *reinterpret_cast<const uint32_t(*)[16]>(&pk[16]));
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(SM_P_READY + u));
      };
      if (have_p)
        hand_over(0);
      else
        acc = 0;
#pragma unroll 1
      for (int u = have_p ? 1 : 0; u < n; ++u) {
        quarters(j0 + u, [&](int c, const uint32_t (&x)[16]) { exp_pack16(x, &pk[c * 8], scale2, negm2, acc); });
        hand_over(u);
      }
      l_sum += pair_sum(acc);
    }
    // epilogue: O / l -> bf16 rows
    const int4 mine = __ldg(qtiles + (int64_t)bh * max_tiles + (max_tiles - QC) + t);     // again: registers are short above
    const int row = mine.y + r_local;
    const bool store = lane_has_row && row < mine.z;
    int dst = row;
    if (store && out_row_idx) dst = out_row_idx[(int64_t)bh * S + row];
    dst = store ? min(max(dst, 0), S - 1) : 0;
    bf16* orow = out_row(peers, out, bh, S, dst);
    // log2 of the softmax denominator, sum_j 2^(s_j * scale * log2 e); -inf for a row without keys
    if (lse && store && (T == 0 || ok))
      lse[(int64_t)bh * S + dst] = (T == 0 || !(l_sum > 0.f)) ? -INFINITY : m_used + __log2f(l_sum);
    if (T == 0) {
      if (store) {
#pragma unroll
        for (int ch = 0; ch < 16; ++ch) reinterpret_cast<uint4*>(orow)[ch] = make_uint4(0, 0, 0, 0);
      }
    } else if (ok && __all_sync(0xffffffffu, mbar_wait(bar(SM_PV_DONE + ((T - 1) & 1)), ((T - 1) >> 1) & 1, abort_flag))) {
      tc_fence_after();
      const float inv = l_sum > 0.f ? 1.0f / l_sum : 0.f;
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t ra[32];
        tmem_ld32(o_t + ch * 32, ra);
        if (store) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 val;
            val.x = pack_bf16x2(__uint_as_float(ra[8 * g + 0]) * inv, __uint_as_float(ra[8 * g + 1]) * inv);
            val.y = pack_bf16x2(__uint_as_float(ra[8 * g + 2]) * inv, __uint_as_float(ra[8 * g + 3]) * inv);
            val.z = pack_bf16x2(__uint_as_float(ra[8 * g + 4]) * inv, __uint_as_float(ra[8 * g + 5]) * inv);
            val.w = pack_bf16x2(__uint_as_float(ra[8 * g + 6]) * inv, __uint_as_float(ra[8 * g + 7]) * inv);
            reinterpret_cast<uint4*>(orow)[ch * 4 + g] = val;
          }
        }
      }
    }
  }
  // ------------------------------------------------------------------ teardown
  // Q was requested before the number of keys was known; without keys nobody has waited for it.
  if (tid == 0) mbar_drain(bar(SM_Q_FULL), 0);
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag) atomicExch(status, 1);
  if (warp == kSmMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
  }
  if (last_cta) pdl_wait();
}

}  // namespace tc

// after_pairs: the pair kernel of the same call was launched just before on this stream, as an ordinary launch behind
// the lists.  This one then starts beside it and needs no wait for the lists: they were complete before the pair
// kernel began, and it begins after that.  Only the last CTA waits, for the pair kernel's end.
cudaError_t launch_sparse_attn_small(const CUtensorMap& q_map, const tc::OutPeers& peers, const void* k, const void* v,
                                     void* out, const int32_t* out_row_idx, const int4* qtiles, const int32_t* nqtiles,
                                     const int32_t* head_order, const int2* runs, const int32_t* nruns, int32_t* status, int64_t BH, int64_t S,
                                     int64_t QC, int64_t KC, int max_runs, float scale_log2, float* lse, cudaStream_t st,
                                     const uint8_t* ear_map, const int32_t* ear_k_offsets, bool after_pairs) {
  const bool ear = ear_map != nullptr;
  auto* kernel = ear ? &tc::sparse_attn_small_kernel<true> : &tc::sparse_attn_small_kernel<false>;
  const int smem = ear ? tc::SmallSmem<true>::kBytes : tc::SmallSmem<false>::kBytes;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)(BH * QC));
  count_launches(1);
  if (!after_pairs) {
    kernel<<<grid, tc::kSmThreads, smem, st>>>(q_map, peers, (const bf16*)k, (const bf16*)v, (bf16*)out, out_row_idx, qtiles,
                                              nqtiles, head_order, runs, nruns, (int)BH, (int)S, (int)QC, max_qtiles(S, QC), max_runs,
                                              scale_log2, status, lse, ear_map, ear_k_offsets, (int)KC);
    return cudaGetLastError();
  }
  return launch_pdl(kernel, grid, dim3(tc::kSmThreads), (size_t)smem, st, q_map, peers, (const bf16*)k, (const bf16*)v,
                    (bf16*)out, out_row_idx, qtiles, nqtiles, head_order, runs, nruns, (int)BH, (int)S, (int)QC, max_qtiles(S, QC), max_runs,
                    scale_log2, status, lse, ear_map, ear_k_offsets, (int)KC);
}

}  // namespace svoo
