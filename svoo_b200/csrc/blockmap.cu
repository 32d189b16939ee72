// Cluster-block map (which key clusters each query cluster attends), and the two small
// index builders the attention kernel consumes: merged key-row runs per query cluster and
// the list of 128-row query tiles.
//
// The map follows identify_dynamic_map (svoo/co_clustering.py:556-633) for bf16
// centroids.  Its arithmetic is fixed to IEEE fp32 add/mul/div in a fixed order (no
// fma, sequential sums), so the result is reproducible bit for bit:
//   score  = sum_d q_d*k_d (d ascending, fp32) -> bf16 -> / fp32(sqrt(D)) -> bf16
//   prob   = size_j * exp(score - max) / max(sum_j, 1e-12)  (sum j ascending) -> bf16
//   order  = descending prob, ties by lower cluster index
//   cumsum = running fp32 sum of sorted probs, each prefix rounded to bf16, vs bf16(top_p)
#include "map_common.cuh"

namespace svoo {

// One CTA = 8 consecutive query clusters of one head, one warp each; kM = key clusters per lane (KC <= 32 kM).
//   * Scores, all 8 warps together: a thread multiplies one or two key centroids with the 8 query centroids; every
//     (query, key) sum runs over d in ascending order, two query clusters to an instruction (f32x2).
//   * The rest is per query cluster and runs in the 8 warps side by side: exp, the sequential sum (lane 0,
//     the next shared-memory reads in flight), the probabilities as keys in registers.
//   * Which clusters stay is a question of how many when the limits or the first probability decide
//     (cap <= floor, or top_p below the largest probability): then the n-th largest key is found bit by bit
//     (26 counts) and nothing is sorted.  Otherwise the keys are sorted and their prefix sums formed up to
//     the first one above top_p.
// 24 heads x 256 x 1024 clusters: 257 us with one query cluster to an instruction, a bitonic sort in every
// case and unpipelined sums (of which scores 94, sort 42, sums 62).
constexpr int kMapRows = 8;
// Key clusters per pass of the score phase.
__host__ __device__ constexpr int map_rows_pass(int M) { return 32 * M < 512 ? 32 * M : 512; }
inline size_t map_smem_bytes(int M) {
  const size_t keys = (size_t)kMapRows * 32 * M * 4, stages = 2 * (size_t)map_rows_pass(M) * 64;
  return (size_t)kMapRows * kHeadDim * 4 + keys + (keys > stages ? keys : stages);              // at most 100 KB
}

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t both(float v) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ void unpair(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }

// x[0] + x[1] + ... + x[n - 1] in that order; x is 16-byte aligned and readable up to a multiple of 16 past n.
__device__ __forceinline__ float ordered_sum(const float* x, int n) {
  const float4* p = reinterpret_cast<const float4*>(x);
  float tot = 0.f;
  float4 a[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = p[i];
  int j = 0;
  for (; j + 16 <= n; j += 16) {
    float4 nxt[4];
    const int q = j + 16 < n ? (j + 16) / 4 : 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) nxt[i] = p[q + i];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      tot = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(tot, a[i].x), a[i].y), a[i].z), a[i].w);
      a[i] = nxt[i];
    }
  }
  for (; j < n; ++j) tot = __fadd_rn(tot, x[j]);
  return tot;
}

template <int kM>
__global__ void __launch_bounds__(256, 2) block_map_kernel(const bf16* __restrict__ qc, const bf16* __restrict__ kc,
                                                        const int32_t* __restrict__ ksizes, uint8_t* __restrict__ map,
                                                        int QC, int KC, float sqrt_d, float top_p,
                                                        const __grid_constant__ HeadLimits lim) {
  constexpr int kPad = 32 * kM, kRowsPass = map_rows_pass(kM), kJ = kRowsPass > 256 ? 2 : 1;
  extern __shared__ __align__(16) unsigned char map_sm[];
  float* q_s = reinterpret_cast<float*>(map_sm);                       // [128][8]
  float* val = q_s + kMapRows * kHeadDim;                              // [8][kPad]: scores, then weighted exps
  uint32_t* key = reinterpret_cast<uint32_t*>(val + kMapRows * kPad);  // two stages of key centroids, then [8][kPad] sorted keys
  const int i0 = blockIdx.x * kMapRows, bh = blockIdx.y, tid = threadIdx.x;
  const int lane = tid % 32, warp = tid / 32;
  if (top_p >= 1.0f) {
    for (int r = 0; r < kMapRows && i0 + r < QC; ++r)
      for (int j = tid; j < KC; j += 256) map[((int64_t)bh * QC + i0 + r) * KC + j] = 1;
    return;
  }
  for (int t = tid; t < kMapRows * kHeadDim; t += 256) {
    const int r = t / kHeadDim, d = t % kHeadDim;
    q_s[d * kMapRows + r] = i0 + r < QC ? __bfloat162float(qc[((int64_t)bh * QC + i0 + r) * kHeadDim + d]) : 0.f;
  }
  __syncthreads();

  // The key centroids pass through shared memory 32 dims of 512 rows at a time (64-byte rows, chunks
  // XOR-swizzled by the row pair so that 8 lanes read 8 different bank groups), double buffered: read row by row
  // from global memory, a warp's 16-byte loads touch 32 rows each and their latency was the score phase's time.
  const uint32_t kbuf = smem_u32(key);
  const int passes = (KC + kRowsPass - 1) / kRowsPass, stages = passes * 4;
  auto load = [&](int s) {
    const int base = s / 4 * kRowsPass, dim0 = s % 4 * 32;
    const uint32_t dst = kbuf + (s & 1) * kRowsPass * 64;
    for (int t = tid; t < kRowsPass * 4; t += 256) {
      const int r = t >> 2, ch = t & 3;
      cp_async16(dst + r * 64 + ((ch ^ ((r >> 1) & 3)) << 4),
                 kc + ((int64_t)bh * KC + min(base + r, KC - 1)) * kHeadDim + dim0 + ch * 8, base + r < KC);
    }
    cp_async_commit();
  };
  load(0);
  uint64_t acc[kJ][4];                                                 // [row of this thread][pair of query clusters]
  for (int s = 0; s < stages; ++s) {
    if (s + 1 < stages) {
      load(s + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (s % 4 == 0) {
#pragma unroll
      for (int x = 0; x < kJ; ++x)
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[x][p] = 0;                     // two fp32 zeros
    }
    const unsigned char* kb = reinterpret_cast<const unsigned char*>(key) + (s & 1) * kRowsPass * 64;
    if (tid < kRowsPass) {
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint4 kv[kJ];
#pragma unroll
        for (int x = 0; x < kJ; ++x) {
          const int r = tid + 256 * x;
          kv[x] = *reinterpret_cast<const uint4*>(kb + r * 64 + ((ch ^ ((r >> 1) & 3)) << 4));
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const ulonglong2* qd = reinterpret_cast<const ulonglong2*>(q_s + (s % 4 * 32 + ch * 8 + e) * kMapRows);
          const ulonglong2 qa = qd[0], qb = qd[1];
          const uint64_t q2[4] = {qa.x, qa.y, qb.x, qb.y};
#pragma unroll
          for (int x = 0; x < kJ; ++x) {
            // bf16 -> fp32: the low half of the word shifted up, or the high half masked
            const uint32_t w = reinterpret_cast<const uint32_t*>(&kv[x])[e / 2];
            const uint64_t k2 = both(__uint_as_float((e & 1) ? (w & 0xFFFF0000u) : (w << 16)));
#pragma unroll
            for (int p = 0; p < 4; ++p) acc[x][p] = add2(acc[x][p], mul2(q2[p], k2));
          }
        }
      }
      if (s % 4 == 3) {
#pragma unroll
        for (int x = 0; x < kJ; ++x) {
          const int j = s / 4 * kRowsPass + tid + 256 * x;
          if (j < KC) {
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              float lo, hi;
              unpair(acc[x][p], lo, hi);
              val[(2 * p) * kPad + j] = bf16_round(__fdiv_rn(bf16_round(lo), sqrt_d));
              val[(2 * p + 1) * kPad + j] = bf16_round(__fdiv_rn(bf16_round(hi), sqrt_d));
            }
          }
        }
      }
    }
    __syncthreads();                                                   // the next load overwrites this stage's buffer
  }

  // ---- from here on: warp w works on query cluster i0 + w
  const int i = i0 + warp;
  if (i >= QC) return;
  float* vw = val + warp * kPad;
  uint32_t* kw = key + warp * kPad;
  float mx = -INFINITY;
#pragma unroll
  for (int m = 0; m < kM; ++m)
    if (lane + 32 * m < KC) mx = fmaxf(mx, vw[lane + 32 * m]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
  for (int m = 0; m < kM; ++m) {
    const int j = lane + 32 * m;
    float e = 0.f;
    if (j < KC) e = __fmul_rn((float)ksizes[(int64_t)bh * KC + j], exp_f32_fixed(__fsub_rn(vw[j], mx)));
    vw[j] = e;
  }
  __syncwarp();
  float tot = 0.f;
  if (lane == 0) tot = fmaxf(ordered_sum(vw, KC), 1e-12f);             // j ascending
  tot = __shfl_sync(0xffffffffu, tot, 0);
  // key of cluster j: (bf16 probability << 16) | (0xFFFF - j); descending keys = descending probability, ties by
  // lower index
  uint32_t v[kM], top = 0;
#pragma unroll
  for (int m = 0; m < kM; ++m) {
    const int j = lane + 32 * m;
    v[m] = 0;
    if (j < KC) {
      const bf16 pb = __float2bfloat16_rn(__fdiv_rn(vw[j], tot));
      v[m] = ((uint32_t)__bfloat16_as_ushort(pb) << 16) | (uint32_t)(0xFFFF - j);
    }
    top = max(top, v[m]);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  // Position r of the descending order stays iff r < cap and (r < floor or r <= cut), cut = the first position
  // whose bf16 prefix sum is above top_p (prefix sums do not decrease).
  const float p_b = bf16_round(top_p);
  const int preserve = max(lim.preserve[bh], 0), cap = max(min(lim.cap[bh], KC), 0);
  uint8_t* out = map + ((int64_t)bh * QC + i) * KC;
  int n = cap;                                          // kept positions
  uint32_t thr = 0;
  if (cap > preserve && __uint_as_float(top & 0xFFFF0000u) > p_b) n = min(cap, max(preserve, 1));    // cut = 0
  if (cap <= preserve || __uint_as_float(top & 0xFFFF0000u) > p_b) {
    if (n > 0 && n < KC) {                              // thr = the n-th largest key (keys are distinct)
#pragma unroll 1
      for (int bit = 31; bit >= 0; --bit) {
        if (bit == 15) {                                // 0xFFFF - j with j < 1024: bits 10 to 15 are set in every key
          thr |= 0xFC00u;
          bit = 9;
        }
        const uint32_t cand = thr | (1u << bit);
        int cnt = 0;
#pragma unroll
        for (int m = 0; m < kM; ++m) cnt += v[m] >= cand;
        if ((int)__reduce_add_sync(0xffffffffu, (unsigned)cnt) >= n) thr = cand;
      }
    }
  } else {
    uint32_t sorted[kM];
#pragma unroll
    for (int m = 0; m < kM; ++m) sorted[m] = v[m];
    warp_sort_desc<kM>(sorted, lane);
#pragma unroll
    for (int m = 0; m < kM; ++m) kw[lane + 32 * m] = sorted[m];
    __syncwarp();
    int cut = cap;                                      // past the cap nothing stays
    if (lane == 0) {                                    // r ascending, eight per step
      float run = 0.f;
      for (int r = 0; r < cap && cut == cap; r += 8) {
        const uint4 a = *reinterpret_cast<const uint4*>(kw + r), b = *reinterpret_cast<const uint4*>(kw + r + 4);
        const uint32_t k8[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float pre[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          run = __fadd_rn(run, __uint_as_float(k8[u] & 0xFFFF0000u));
          pre[u] = run;
        }
#pragma unroll
        for (int u = 7; u >= 0; --u)
          if (bf16_round(pre[u]) > p_b) cut = min(r + u, cap);
      }
    }
    cut = __shfl_sync(0xffffffffu, cut, 0);
    n = min(cap, max(preserve, cut + 1));
    if (n > 0 && n < KC) thr = kw[n - 1];
  }
#pragma unroll
  for (int m = 0; m < kM; ++m) {
    const int j = lane + 32 * m;
    if (j < KC) out[j] = n > 0 && v[m] >= thr ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------------------------
// The two index lists of the attention kernels, in one launch: blocks [0, BH) write the query tiles of
// one head each, the blocks after them the key-row runs of eight query clusters of a head each.
// ---------------------------------------------------------------------------------------------
// Query tiles of every non-empty query cluster, in cluster order; thread i owns clusters
// [kPer i, kPer (i + 1)).  Tiles of kRows rows; with kSplit (kRows = 256) a remainder of up to 128 rows goes
// to a list of its own (the last QC entries of the head's tiles, for attn_small.cu).
constexpr int kListThreads = 256;
template <int kRows, bool kSplit>
__device__ void build_qtiles(const int32_t* __restrict__ off, int4* __restrict__ out, int32_t* __restrict__ counts, int QC,
                             int max_tiles) {
  constexpr int kPer = (SVOO_MAX_ATTN_CLUSTERS + kListThreads - 1) / kListThreads;
  __shared__ unsigned long long warp_tot[kListThreads / 32];
  const int i = threadIdx.x, lane = i % 32, warp = i / 32;
  int b[kPer + 1];
#pragma unroll
  for (int u = 0; u <= kPer; ++u) b[u] = off[min(kPer * i + u, QC)];
  auto single = [](int rows) { return (int)(kSplit && rows > 0 && (rows - 1) % kRows < kAttnBM); };
  unsigned long long n = 0;                              // (whole tiles, single tiles) of this thread's clusters
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int rows = b[u + 1] - b[u], s1 = single(rows);
    n += (unsigned long long)((rows + kRows - 1) / kRows - s1) | (unsigned long long)s1 << 32;
  }
  unsigned long long incl = n;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const unsigned long long o = __shfl_up_sync(0xffffffffu, incl, s);
    if (lane >= s) incl += o;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  unsigned long long before = incl - n, total = 0;
#pragma unroll
  for (int w = 0; w < kListThreads / 32; ++w) {
    if (w < warp) before += warp_tot[w];
    total += warp_tot[w];
  }
  int pos = (int)(before & 0xffffffffu), spos = max_tiles - QC + (int)(before >> 32);
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int rows = b[u + 1] - b[u], s1 = single(rows), nt = (rows + kRows - 1) / kRows - s1;
    int r = b[u];
    for (int t = 0; t < nt; ++t, ++pos, r += kRows)
      if (pos < max_tiles) out[pos] = make_int4(kPer * i + u, r, min(r + kRows, b[u + 1]), 0);
    if (s1) {
      if (spos < max_tiles) out[spos] = make_int4(kPer * i + u, r, b[u + 1], 0);
      ++spos;
    }
  }
  if (i == 0) {
    counts[0] = min((int)(total & 0xffffffffu), max_tiles);
    counts[1] = min((int)(total >> 32), QC);
  }
}

// One warp per (head, query cluster): maximal stretches of consecutive selected, non-empty
// key clusters become runs of the cluster-ordered K/V.  Run r is stored as
// (first_row, virtual_begin): virtual_begin is the number of selected key rows before it, so
// the concatenation of all runs is addressed by one "virtual" row index; entry [nruns] is a
// sentinel (0, total selected rows).
// kEar: the K/V tensors are the cluster-ordered rows of all heads followed by the centroid rows of all
// heads ([BH*S + BH*KC, 128]), and the list ends with ONE more run, the KC centroid rows of the head
// (the attention kernels mask the centroids of the selected clusters).
// The block's rows belong to one head, whose offsets (and a bit per non-empty cluster) are staged in shared
// memory.  Lane l of a row's warp reads its own 32 map bytes, keeps them as a 32-bit mask and walks the runs
// of that mask twice: their rows are summed, a scan over the lanes gives the first run and virtual row, and
// they are written.  The instruction count is what this costs: about 450 per row; with a vote for every 32
// clusters and 64-bit masks 2,300 (24 heads x 258 rows x 1,026 clusters: 36 us), with a scan for every 32
// clusters 43 us.
constexpr int kListRows = kListThreads / 32;
template <bool kEar>
__device__ void build_runs(const uint8_t* __restrict__ map, const int32_t* __restrict__ k_offsets, int2* __restrict__ runs,
                           int32_t* __restrict__ nruns, int32_t* __restrict__ head_work, int bh, int i0, int BH, int S, int QC,
                           int KC, int max_runs) {
  constexpr int kMask = 1024;                                          // clusters in the lanes' masks; the rest: lane 31
  __shared__ int32_t off_s[SVOO_MAX_ATTN_CLUSTERS + 1];
  __shared__ uint32_t filled[kMask / 32];
  const int32_t* off = k_offsets + (int64_t)bh * (KC + 1);
  for (int j = threadIdx.x; j <= KC; j += kListThreads) off_s[j] = off[j];
  const int r = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t row = (int64_t)bh * QC + min(i0 + r, QC - 1);
  const uint8_t* m = map + row * KC;
  // bytes [32 lane, 32 lane + 32) of the row
  const int j0 = lane * 32;
  uint32_t w[9];
  const int skew = map_words(w, m + j0, max(min(KC - j0, 32), 0), map, map + (int64_t)BH * QC * KC, MapLoad());
  __syncthreads();
  for (int t = r; t < kMask / 32; t += kListRows) {
    const int j = t * 32 + lane;
    const unsigned word = __ballot_sync(0xffffffffu, j < KC && off_s[min(j + 1, KC)] > off_s[min(j, KC)]);
    if (lane == 0) filled[t] = word;
  }
  __syncthreads();
  if (i0 + r >= QC) return;
  uint32_t sel = 0;                                                    // bit b: cluster j0 + b, selected and not empty
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t x = __funnelshift_r(w[i], w[i + 1], 8 * skew);
    uint32_t nz = ((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu | x) & 0x80808080u;       // top bit of every byte that is not zero
    nz = (nz >> 7) * 0x10204080u >> 28;                                      // the four of them side by side
    sel |= nz << (4 * i);
  }
  sel &= filled[lane];
  int2* out = runs + row * max_runs;
  const int limit = max_runs - (kEar ? 2 : 1);
  // [b, e) = the first run of `rest`; what is left of it
  auto next_run = [](uint32_t& rest, int& b, int& e) {
    b = __ffs(rest) - 1;
    const uint32_t gap = ~(rest >> b);
    e = gap ? b + __ffs(gap) - 1 : 32;
    rest = e >= 32 ? 0u : rest >> e << e;
  };
  int n = 0, sum = 0;
  for (uint32_t rest = sel; rest;) {
    int b, e;
    next_run(rest, b, e);
    sum += off_s[j0 + e] - off_s[j0 + b];
    ++n;
  }
  // the lane's first run may continue the one of the lane before
  const uint32_t before = __shfl_up_sync(0xffffffffu, sel >> 31, 1);
  const bool joined = lane > 0 && before && (sel & 1);
  n -= joined;
  int n_incl = n, s_incl = sum;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, n_incl, s), b = __shfl_up_sync(0xffffffffu, s_incl, s);
    if (lane >= s) { n_incl += a; s_incl += b; }
  }
  int pos = n_incl - n - joined, vbeg = s_incl - sum;
  bool skip = joined;
  for (uint32_t rest = sel; rest;) {
    int b, e;
    next_run(rest, b, e);
    if (!skip && pos < limit) out[pos] = make_int2(off_s[j0 + b], vbeg);
    skip = false;
    ++pos;
    vbeg += off_s[j0 + e] - off_s[j0 + b];
  }
  if (lane == 31) {
    int k = n_incl, rows_sel = s_incl;
    bool in_run = sel >> 31;
    for (int j = kMask; j < KC; ++j) {                                 // the text blocks of a 1024-cluster layer
      const int size = m[j] != 0 ? off_s[j + 1] - off_s[j] : 0;
      if (size > 0 && !in_run) {
        if (k < limit) out[k] = make_int2(off_s[j], rows_sel);
        ++k;
      }
      in_run = size > 0;
      rows_sel += size;
    }
    k = min(k, limit);
    if (kEar) {
      out[k++] = make_int2((BH - bh) * S + bh * KC, rows_sel);         // the head's centroid rows
      rows_sel += KC;
    }
    out[k] = make_int2(0, rows_sel);
    nruns[row] = k;
    atomicAdd(&head_work[bh], (rows_sel + 127) / 128);
  }
}

template <int kRows, bool kSplit, bool kEar>
__global__ void __launch_bounds__(kListThreads) attn_lists_kernel(
    const int32_t* __restrict__ q_offsets, int4* __restrict__ qtiles, int32_t* __restrict__ nqtiles, int max_tiles,
    const uint8_t* __restrict__ map, const int32_t* __restrict__ k_offsets, int2* __restrict__ runs,
    int32_t* __restrict__ nruns, int32_t* __restrict__ sched, int32_t* __restrict__ head_order, int BH, int S, int QC, int KC,
    int max_runs, bool ordered) {
  if ((int)blockIdx.x < BH) {
    const int bh = blockIdx.x;
    build_qtiles<kRows, kSplit>(q_offsets + (int64_t)bh * (QC + 1), qtiles + (int64_t)bh * max_tiles, nqtiles + 2 * bh, QC, max_tiles);
  } else {
    const int per_head = (QC + kListRows - 1) / kListRows, b = blockIdx.x - BH;
    build_runs<kEar>(map, k_offsets, runs, nruns, sched + 1, b / per_head, b % per_head * kListRows, BH, S, QC, KC, max_runs);
  }
  if (!ordered) {
    if ((int)blockIdx.x < BH && threadIdx.x == 0) head_order[blockIdx.x] = blockIdx.x;
    return;
  }
  // The last block to finish orders the heads by their selected key tiles (summed over query clusters).
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(sched, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  constexpr int kMaxOrdered = 1024;                      // with more heads any order ends evenly
  __shared__ int work[kMaxOrdered];
  for (int h = threadIdx.x; h < min(BH, kMaxOrdered); h += kListThreads) work[h] = __ldcg(sched + 1 + h);
  __syncthreads();
  for (int h = threadIdx.x; h < BH; h += kListThreads) {
    int rank = h;
    if (BH <= kMaxOrdered) {
      const int mine = work[h];
      rank = 0;
      for (int g = 0; g < BH; ++g) rank += work[g] > mine || (work[g] == mine && g < h);
    }
    head_order[rank] = h;
  }
}

cudaError_t launch_block_map(const void* qc, const void* kc, const int32_t* ksizes, uint8_t* map, int64_t BH,
                             int64_t QC, int64_t KC, float top_p, const int32_t* preserve_host,
                             const int32_t* cap_host, cudaStream_t st) {
  HeadLimits lim;
  for (int h = 0; h < SVOO_MAX_HEADS; ++h) {
    lim.preserve[h] = h < BH ? preserve_host[h] : 0;
    lim.cap[h] = h < BH ? cap_host[h] : (int32_t)KC;
  }
  // key clusters per lane: the next power of two
  int M = 1;
  while (32 * M < KC) M <<= 1;
  auto* kernel = M == 1   ? &block_map_kernel<1>
                 : M == 2 ? &block_map_kernel<2>
                 : M == 4 ? &block_map_kernel<4>
                 : M == 8 ? &block_map_kernel<8>
                 : M == 16 ? &block_map_kernel<16>
                           : &block_map_kernel<32>;
  const size_t smem = map_smem_bytes(M);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)map_smem_bytes(32));
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)ceil_div64(QC, kMapRows), (unsigned)BH);
  kernel<<<grid, 256, smem, st>>>((const bf16*)qc, (const bf16*)kc, ksizes, map, (int)QC, (int)KC,
                                  (float)sqrt((double)kHeadDim), top_p, lim);
  count_launches(1);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Text tokens of a joint-attention layer (svoo/models/hunyuan10/attention.py:999-1019): the
// `text` rows that follow the N clustered video rows of every head become two more blocks,
// "prompt" (the first `prompt` text rows) and "unused prompt" (the rest).
//   map  [BH, QC, KC]   -> [BH, QC+2, KC+2]: prompt queries see every video and prompt key, every
//                          query but the unused prompt sees the prompt keys, the unused prompt sees itself
//   offsets [BH, K+1]   -> [BH, K+3]  (block sizes `prompt`, `text - prompt` appended)
//   sorted_idx [BH, N]  -> [BH, N+text]  (identity on the text rows)
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) append_text_blocks_kernel(
    const uint8_t* __restrict__ map, const int32_t* __restrict__ q_off, const int32_t* __restrict__ k_off,
    const int32_t* __restrict__ q_idx, const int32_t* __restrict__ k_idx, uint8_t* __restrict__ map_out,
    int32_t* __restrict__ q_off_out, int32_t* __restrict__ k_off_out, int32_t* __restrict__ q_idx_out,
    int32_t* __restrict__ k_idx_out, int N, int QC, int KC, int text, int prompt) {
  const int bh = blockIdx.y;
  const int S = N + text, QC2 = QC + 2, KC2 = KC + 2;
  const int stride = gridDim.x * 256;
  for (int t = blockIdx.x * 256 + threadIdx.x; t < QC2 * KC2; t += stride) {
    const int i = t / KC2, j = t - i * KC2;
    uint8_t v;
    if (i < QC) v = j < KC ? (uint8_t)(map[((int64_t)bh * QC + i) * KC + j] != 0) : (uint8_t)(j == KC);
    else if (i == QC) v = (uint8_t)(j <= KC);
    else v = (uint8_t)(j == KC + 1);
    map_out[(int64_t)bh * QC2 * KC2 + t] = v;
  }
  for (int t = blockIdx.x * 256 + threadIdx.x; t < S; t += stride) {
    q_idx_out[(int64_t)bh * S + t] = t < N ? q_idx[(int64_t)bh * N + t] : t;
    k_idx_out[(int64_t)bh * S + t] = t < N ? k_idx[(int64_t)bh * N + t] : t;
  }
  for (int t = blockIdx.x * 256 + threadIdx.x; t <= QC2; t += stride)
    q_off_out[(int64_t)bh * (QC2 + 1) + t] = t <= QC ? q_off[(int64_t)bh * (QC + 1) + t] : (t == QC + 1 ? N + prompt : S);
  for (int t = blockIdx.x * 256 + threadIdx.x; t <= KC2; t += stride)
    k_off_out[(int64_t)bh * (KC2 + 1) + t] = t <= KC ? k_off[(int64_t)bh * (KC + 1) + t] : (t == KC + 1 ? N + prompt : S);
}

cudaError_t launch_append_text_blocks(const uint8_t* map, const int32_t* q_off, const int32_t* k_off, const int32_t* q_idx,
                                      const int32_t* k_idx, uint8_t* map_out, int32_t* q_off_out, int32_t* k_off_out,
                                      int32_t* q_idx_out, int32_t* k_idx_out, int64_t BH, int64_t N, int64_t QC, int64_t KC,
                                      int64_t text, int64_t prompt, cudaStream_t st) {
  const int64_t work = (QC + 2) * (KC + 2) > N + text ? (QC + 2) * (KC + 2) : N + text;
  int64_t blocks = ceil_div64(work, 256 * 4);
  blocks = blocks < 1 ? 1 : (blocks > 1024 ? 1024 : blocks);
  append_text_blocks_kernel<<<dim3((unsigned)blocks, (unsigned)BH), 256, 0, st>>>(
      map, q_off, k_off, q_idx, k_idx, map_out, q_off_out, k_off_out, q_idx_out, k_idx_out, (int)N, (int)QC, (int)KC,
      (int)text, (int)prompt);
  count_launches(1);
  return cudaGetLastError();
}

// The heads are ordered by work above 256 query clusters in all: below that the call is small, or has a few heads of
// many tokens, whose tiles then run in the order of the heads.
// tile_rows: 128 (mma.sync kernel) or 256; split: single tiles in their own list.  ear: with the head's
// centroid run (256-row tiles only).
cudaError_t launch_attn_lists(const int32_t* q_offsets, int4* qtiles, int32_t* nqtiles, const uint8_t* map,
                              const int32_t* k_offsets, int2* runs, int32_t* nruns, int32_t* sched, int32_t* head_order, int64_t BH,
                              int64_t S, int64_t QC, int64_t KC, int max_runs, int tile_rows, bool split, bool ear, cudaStream_t st) {
  auto* kernel = tile_rows == 128 ? &attn_lists_kernel<128, false, false>
                 : ear ? (split ? &attn_lists_kernel<256, true, true> : &attn_lists_kernel<256, false, true>)
                       : (split ? &attn_lists_kernel<256, true, false> : &attn_lists_kernel<256, false, false>);
  const int64_t blocks = BH + BH * ceil_div64(QC, kListRows);
  kernel<<<(unsigned)blocks, kListThreads, 0, st>>>(q_offsets, qtiles, nqtiles, max_qtiles(S, QC), map, k_offsets, runs, nruns,
                                                   sched, head_order, (int)BH, (int)S, (int)QC, (int)KC, max_runs, BH * QC > 256);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace svoo
