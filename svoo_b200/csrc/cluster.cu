// QK co-clustering kernels: profile prologue (builds the W operand of the assignment GEMM,
// which lives in assign_tc.cu), stable counting sort of labels, deterministic centroid update.
//
// Algebra used by the assignment.  The reference (svoo/co_clustering.py:2148-2255)
// computes, for token x and own-centroid j,
//     score_j = sum_k ((x . c_k) / norm(x)) * Phat[j,k],   label = first argmax_j score_j
// with c_k the profile-forming centroids and Phat the row-normalised centroid-centroid
// profile.  norm(x) > 0 does not depend on j and the double sum is linear in x, so
//     label = first argmax_j  x . W_j,     W_j = sum_k Phat[j,k] c_k      (W is [J,128])
// One GEMM [N,128] x [128,J] per side and iteration replaces the two chained GEMMs and
// the separate norm pass.  W is carried as a bf16 pair (hi, lo = bf16(W - hi)) so the
// products keep ~16 mantissa bits, more than the TF32 operands of the reference.
#include <atomic>

#include "common.cuh"

namespace svoo {

// ---------------------------------------------------------------------------------------
// centroids[bh,c,:] = x[bh, idx[bh,c], :]     (svoo/co_clustering.py:2417-2421)
// ---------------------------------------------------------------------------------------
__global__ void gather_rows_kernel(const bf16* __restrict__ x, const int32_t* __restrict__ idx,
                                   bf16* __restrict__ out, int N, int K, int64_t x_head_rows) {
  pdl_trigger();
  pdl_wait();
  const int bh = blockIdx.y;
  const int c = blockIdx.x * (blockDim.x / 16) + threadIdx.x / 16;
  if (c >= K) return;
  const int lane = threadIdx.x % 16;
  int src = idx[(int64_t)bh * K + c];
  src = min(max(src, 0), N - 1);
  const uint4* s = reinterpret_cast<const uint4*>(x + (bh * x_head_rows + src) * kHeadDim);
  uint4* d = reinterpret_cast<uint4*>(out + ((int64_t)bh * K + c) * kHeadDim);
  d[lane] = s[lane];
}

// ---------------------------------------------------------------------------------------
// Prologue: P = bf16(own . form^T), Phat = P / sqrt(sum P^2 + 1e-8) (fp32),
//           W = Phat . form (fp32) -> (hi, lo) bf16.     One CTA = 16 rows j of one head.
// Both products run on mma.sync (m16n8k16, fp32 accumulation): the problem is a few MFLOP
// per head and latency-bound, so the point is the short dependency chain, not throughput.
// `form` is streamed twice through a double-buffered shared-memory ring of 64-row chunks
// (cp.async).  Phat (fp32) enters the second product as three bf16 terms hi + mid + lo,
// which carries 24 mantissa bits, so W matches an fp32 product to rounding.
// (svoo/co_clustering.py:2427-2428 and svoo/kernels/triton/l2norm.py:36-41)
// ---------------------------------------------------------------------------------------
constexpr int kProR = 16;            // own rows per CTA
constexpr int kProC = 64;            // form rows per chunk

__host__ __device__ inline int pro_kround(int K) { return (K + kProC - 1) / kProC * kProC; }
__host__ __device__ inline int pro_p_stride(int K) { return pro_kround(K) + 4; }       // floats
__host__ __device__ inline int pro_hat_stride(int K) { return pro_kround(K) + 8; }     // bf16: 16 bytes past a multiple of 128
inline size_t pro_smem_bytes(int K) {
  return (size_t)kProR * kRowBytes + 2 * (size_t)kProC * kRowBytes + (size_t)kProR * pro_p_stride(K) * 4 +
         3 * (size_t)kProR * pro_hat_stride(K) * 2;
}

__global__ void __launch_bounds__(256) profile_prologue_kernel(
    const bf16* __restrict__ own, const bf16* __restrict__ form, bf16* __restrict__ w_hi,
    bf16* __restrict__ w_lo, int J, int K, int Jpad) {
  extern __shared__ __align__(128) unsigned char pro_sm[];
  pdl_trigger();
  pdl_wait();                                           // the centroids come from the previous kernel
  const int bh = blockIdx.y, j0 = blockIdx.x * kProR;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (j0 >= J) {                                        // padding rows of W: zeros
    const int d = tid & 127, rg = tid >> 7;
    for (int r = rg * 8; r < rg * 8 + 8; ++r)
      if (j0 + r < Jpad) {
        w_hi[((int64_t)bh * Jpad + j0 + r) * kHeadDim + d] = __float2bfloat16_rn(0.f);
        w_lo[((int64_t)bh * Jpad + j0 + r) * kHeadDim + d] = __float2bfloat16_rn(0.f);
      }
    return;
  }
  const int pstride = pro_p_stride(K), hstride = pro_hat_stride(K);
  unsigned char* own_p = pro_sm;                                    // [16][128] bf16, swizzled
  unsigned char* form_p = own_p + kProR * kRowBytes;                // 2 x [64][128] bf16, swizzled
  float* p_s = reinterpret_cast<float*>(form_p + 2 * kProC * kRowBytes);       // [16][pstride]
  bf16* hat = reinterpret_cast<bf16*>(p_s + kProR * pstride);                  // 3 x [16][hstride]
  const uint32_t own_s = smem_u32(own_p), form_s = smem_u32(form_p), hat_s = smem_u32(hat);
  const bf16* form_b = form + (int64_t)bh * K * kHeadDim;
  const int nch = (K + kProC - 1) / kProC;

  auto load_chunk = [&](int c, int buf) {               // rows past K arrive as zeros
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
      const int i = tid + pass * 256, row = i >> 4, ch = i & 15;
      const int k = c * kProC + row;
      cp_async16(form_s + buf * (kProC * kRowBytes) + swz(row, ch),
                 form_b + (int64_t)min(k, K - 1) * kHeadDim + ch * 8, k < K);
    }
  };
  {
    const int row = tid >> 4, ch = tid & 15;
    const int j = j0 + row;
    cp_async16(own_s + swz(row, ch), own + ((int64_t)bh * J + min(j, J - 1)) * kHeadDim + ch * 8, j < J);
  }
  load_chunk(0, 0);
  cp_async_commit();

  // ---- sweep 1: P[16][K]; warps 0..3 take 16 form rows of the chunk each
  uint32_t qa[8][4];
  for (int c = 0; c < nch; ++c) {
    if (c + 1 < nch) load_chunk(c + 1, (c + 1) & 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (warp < 4) {
      if (c == 0) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          ldmatrix_x4(qa[ks], own_s + swz((lane % 8) + ((lane / 8) % 2) * 8, ks * 2 + lane / 16));
      }
      const uint32_t f = form_s + (c & 1) * (kProC * kRowBytes);
      float acc[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t b[4];
        ldmatrix_x4(b, f + swz(warp * 16 + (lane % 8) + (lane / 16) * 8, ks * 2 + ((lane / 8) % 2)));
        mma_bf16(acc[0], qa[ks], b[0], b[1]);
        mma_bf16(acc[1], qa[ks], b[2], b[3]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {                   // torch.matmul of bf16 tensors returns bf16
          const int row = lane / 4 + (e >> 1) * 8;
          const int k = c * kProC + warp * 16 + nt * 8 + 2 * (lane % 4) + (e & 1);
          p_s[row * pstride + k] = bf16_round(acc[nt][e]);
        }
    }
    __syncthreads();
  }
  load_chunk(0, 0);                                     // first chunk of sweep 2, in flight during the norms
  cp_async_commit();

  // ---- row norms (16 threads per row, fixed order), Phat = P / norm split into three bf16 terms
  {
    const int row = tid >> 4, sub = tid & 15;
    const int kr = pro_kround(K);
    float ss = 0.f;
    for (int k = sub; k < kr; k += 16) { const float x = p_s[row * pstride + k]; ss = fmaf(x, x, ss); }
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float nr = sqrtf(ss + 1e-8f);
    for (int k = sub; k < kr; k += 16) {
      const float x = p_s[row * pstride + k] / nr;
      const bf16 h = __float2bfloat16_rn(x);
      const float r1 = x - __bfloat162float(h);
      const bf16 m = __float2bfloat16_rn(r1);
      const bf16 l = __float2bfloat16_rn(r1 - __bfloat162float(m));
      hat[(0 * kProR + row) * hstride + k] = h;
      hat[(1 * kProR + row) * hstride + k] = m;
      hat[(2 * kProR + row) * hstride + k] = l;
    }
  }

  // ---- sweep 2: W[16][128] = sum_k Phat[r][k] form[k][d]; warp w owns dims 16w .. 16w+15
  float wacc[3][2][4];
#pragma unroll
  for (int t = 0; t < 3; ++t)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) wacc[t][i][e] = 0.f;
  for (int c = 0; c < nch; ++c) {
    if (c + 1 < nch) load_chunk(c + 1, (c + 1) & 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const uint32_t f = form_s + (c & 1) * (kProC * kRowBytes);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t b[4];
      ldmatrix_x4_trans(b, f + swz(kk * 16 + (lane % 8) + ((lane / 8) % 2) * 8, warp * 2 + lane / 16));
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        uint32_t a[4];
        const int arow = (lane % 8) + ((lane / 8) % 2) * 8;
        const int acol = c * kProC + kk * 16 + (lane / 16) * 8;
        ldmatrix_x4(a, hat_s + (uint32_t)(((t * kProR + arow) * hstride + acol) * 2));
        mma_bf16(wacc[t][0], a, b[0], b[1]);
        mma_bf16(wacc[t][1], a, b[2], b[3]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int j = j0 + lane / 4 + half * 8;
      if (j < Jpad) {
        float v0 = wacc[0][nt][half * 2] + (wacc[1][nt][half * 2] + wacc[2][nt][half * 2]);
        float v1 = wacc[0][nt][half * 2 + 1] + (wacc[1][nt][half * 2 + 1] + wacc[2][nt][half * 2 + 1]);
        if (j >= J) v0 = v1 = 0.f;
        const bf16 h0 = __float2bfloat16_rn(v0), h1 = __float2bfloat16_rn(v1);
        const bf16 l0 = __float2bfloat16_rn(v0 - __bfloat162float(h0)), l1 = __float2bfloat16_rn(v1 - __bfloat162float(h1));
        const int64_t o = ((int64_t)bh * Jpad + j) * kHeadDim + warp * 16 + nt * 8 + 2 * (lane % 4);
        __nv_bfloat162 hv, lv;
        hv.x = h0; hv.y = h1; lv.x = l0; lv.y = l1;
        *reinterpret_cast<__nv_bfloat162*>(w_hi + o) = hv;
        *reinterpret_cast<__nv_bfloat162*>(w_lo + o) = lv;
      }
    }
}

// ---------------------------------------------------------------------------------------
// Stable counting sort of the labels of a head, in one launch: a cluster of up to 16 CTAs per head.
// Every warp owns a contiguous range of tokens and counts its labels in a histogram of its own.  The CTAs exchange their
// totals through distributed shared memory, every CTA scans the head's totals, and a second walk over the
// same tokens writes them to their places.
// kGroups > 0: the labels are first reduced from the assignment kernel's per-column-group winners
// (lower group wins ties) and written out on the way.
//
// As separate histogram, scan and scatter kernels this was three of the seven launches of a clustering
// phase, each of them a chain of dependent loads.  Labels alone, before -> now: 12 x 32,760 tokens, 100 / 1024 clusters
// 14.2 -> 9.7 / 16.9 -> 13.3 us, 40 x 75,600, 100 / 500 clusters 34.9 -> 28.2 / 43.2 -> 32.6, 24 x 118,800, 500 clusters
// 44.9 -> 35.7, 1 x 4,096 tokens, 100 clusters 9.5 -> 5.5.  What is left is shared-memory work (an atomic per token in the first walk, two
// accesses in the second) and the scattered stores.  One head has 16 CTAs at most: with one million tokens a head and fewer
// than five heads the three kernels were faster (1 x 1,000,000, 100 clusters: 39 against 67 us).
// ---------------------------------------------------------------------------------------
constexpr int kSortWarps = 16;
constexpr int kSortThreads = 32 * kSortWarps;
// Up to this many labels every CTA of the cluster reads the totals of all (one barrier less on the way); above, that is most
// of the time once an SM holds several CTAs (16 CTAs: 64 KB of remote reads each at 1024 labels) and each does a share
// for all.  Direct / shared: 12 x 75,600 tokens, 100 labels 18.2 / 19.1 us, 500 labels 22.7 / 21.2, 1024 labels 32.9 / 22.9.
constexpr int kSortDirect = 256;
static_assert(kSortDirect <= kSortThreads, "one label per thread");
inline size_t sort_smem_bytes(int64_t K) { return (size_t)(kSortWarps + 2) * K * 4; }          // 72 KB at 1024 clusters

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ int ld_cluster(uint32_t addr, uint32_t rank) {
  int v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.s32 %0, [a];\n\t}\n"
               : "=r"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}

__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t rank, int v) {
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.s32 [a], %2;\n\t}\n"
               ::"r"(addr), "r"(rank), "r"(v) : "memory");
}

// Lanes whose label equals this lane's; `bits` = width of a label.  A vote per bit: __match_any_sync takes time for every
// different value among the lanes, and with it the second walk was most of the kernel.
__device__ __forceinline__ unsigned same_label(int label, bool ok, int bits) {
  unsigned grp = __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int b = 0; b < 10; ++b) {                         // labels are below SVOO_MAX_CLUSTERS = 2^10
    if (b < bits) {
      const bool one = (label >> b) & 1;
      const unsigned v = __ballot_sync(0xffffffffu, one);
      grp &= one ? v : ~v;
    }
  }
  return grp;
}

template <int kGroups>
__global__ void __launch_bounds__(kSortThreads, kSortCtasPerSm) sort_labels_kernel(
    const int2* __restrict__ partial, int32_t* labels, int32_t* __restrict__ sorted_idx, int32_t* __restrict__ offsets, int BH,
    int N, int K) {
  extern __shared__ int sort_sm[];
  int* wh = sort_sm;                                     // [16][K] counts, then positions, per warp
  int* tot = wh + kSortWarps * K;                        // [K] this CTA's totals, then the head's
  int* add = tot + K;                                    // [K] tokens of the CTAs before this one, then first positions
  __shared__ int warp_tot[kSortWarps];
  pdl_trigger();
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int rank = (int)cluster_rank(), ctas = (int)cluster_size();
  const int bh = blockIdx.x / ctas;
  for (int i = tid; i < kSortWarps * K; i += kSortThreads) wh[i] = 0;
  // ranges are whole groups of 32 tokens
  const int per_cta = (int)ceil_div64(ceil_div64(N, ctas), 32) * 32;
  const int c0 = min(rank * per_cta, N), c1 = min(c0 + per_cta, N);
  const int per_warp = ceil_div(ceil_div(c1 - c0, kSortWarps), 32) * 32;
  const int w0 = min(c0 + warp * per_warp, c1), w1 = min(w0 + per_warp, c1);
  int* mine = wh + warp * K;
  int32_t* lb = labels + (int64_t)bh * N;
  __syncthreads();
  pdl_wait();

  // ---- walk 1: labels and the warp's counts; the loads of kU steps are in flight together
  constexpr int kU = kGroups > 2 ? (kGroups > 4 ? 1 : 2) : 4;
  for (int s = w0; s < w1; s += 32 * kU) {
    int l[kU];
    if constexpr (kGroups == 0) {
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int n = s + u * 32 + lane;
        l[u] = n < w1 ? lb[n] : -1;
      }
    } else {
      int2 c[kU][kGroups];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int n = min(s + u * 32 + lane, w1 - 1);
#pragma unroll
        for (int g = 0; g < kGroups; ++g) c[u][g] = partial[((int64_t)g * BH + bh) * N + n];
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int n = s + u * 32 + lane;
        int2 best = c[u][0];
#pragma unroll
        for (int g = 1; g < kGroups; ++g)
          if (__int_as_float(c[u][g].x) > __int_as_float(best.x)) best = c[u][g];
        l[u] = n < w1 ? best.y : -1;
        if (n < w1) lb[n] = best.y;
      }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (l[u] >= 0 && l[u] < K) atomicAdd(&mine[l[u]], 1);
    }
  }
  __syncthreads();
  for (int k = tid; k < K; k += kSortThreads) {
    int run = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const int t = wh[w * K + k];
      wh[w * K + k] = run;
      run += t;
    }
    tot[k] = run;
  }
  __syncwarp();                                          // the lanes left the loop at different counts; the barrier is .aligned
  cluster_arrive();
  cluster_wait();

  // ---- tokens of the head and of the CTAs before this one, per label
  constexpr int kPer = (SVOO_MAX_CLUSTERS + kSortThreads - 1) / kSortThreads;
  const int per = ceil_div(K, kSortThreads);             // labels per thread
  int all[kPer] = {}, before[kPer] = {}, sum = 0;
  if (K <= kSortDirect) {                                // every CTA reads everybody's totals
    if (tid < K)
      for (int r0 = 0; r0 < ctas; r0 += 8) {             // eight remote reads in flight
        int v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = r0 + r < ctas ? ld_cluster(smem_u32(tot + tid), r0 + r) : 0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          if (r0 + r < rank) before[0] += v[r];
          all[0] += v[r];
        }
      }
    __syncwarp();
    cluster_arrive();                                    // this CTA has read the others' totals (waited for at the end)
  } else {                                               // every CTA does its share of the labels for all of them
    const int share = ceil_div(K, ctas), k1 = min((rank + 1) * share, K);
    for (int k = rank * share + tid; k < k1; k += kSortThreads) {
      int run = 0;
      for (int r0 = 0; r0 < ctas; r0 += 8) {
        int v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = r0 + r < ctas ? ld_cluster(smem_u32(tot + k), r0 + r) : 0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          if (r0 + r < ctas) st_cluster(smem_u32(add + k), r0 + r, run);
          run += v[r];
        }
      }
      for (int r = 0; r < ctas; ++r) st_cluster(smem_u32(tot + k), r, run);
    }
    __syncwarp();
    cluster_arrive();                                    // nothing remote after this barrier
    cluster_wait();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int k = tid * per + u;
      if (u < per && k < K) {
        all[u] = tot[k];
        before[u] = add[k];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) sum += all[u];

  // ---- exclusive scan over the labels
  int incl = sum;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, s);
    if (lane >= s) incl += o;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  int excl = incl - sum, total = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    if (w < warp) excl += warp_tot[w];
    total += warp_tot[w];
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = tid * per + u;
    if (u < per && k < K) {
      add[k] = excl + before[u];
      if (rank == 0) offsets[(int64_t)bh * (K + 1) + k] = excl;
    }
    excl += all[u];
  }
  if (rank == 0 && tid == 0) offsets[(int64_t)bh * (K + 1) + K] = total;
  __syncthreads();

  // ---- walk 2: the warp's tokens to their places, in order
  int32_t* out = sorted_idx + (int64_t)bh * N;
  const int bits = 32 - __clz(K - 1);
  for (int s = w0; s < w1; s += 32 * 4) {
    int l[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int n = s + u * 32 + lane;
      l[u] = n < w1 ? lb[n] : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool ok = l[u] >= 0 && l[u] < K;
      const unsigned grp = same_label(l[u], ok, bits);
      const int pos_in_grp = __popc(grp & ((1u << lane) - 1u));
      int base = 0;
      if (ok) base = mine[l[u]];
      __syncwarp();
      if (ok && pos_in_grp == 0) mine[l[u]] = base + __popc(grp);
      __syncwarp();
      if (ok) {
        const int pos = add[l[u]] + base + pos_in_grp;
        if (pos < N) out[pos] = s + u * 32 + lane;
      }
    }
  }
  if (K <= kSortDirect) {
    __syncwarp();
    cluster_wait();
  }
}

// ---------------------------------------------------------------------------------------
// Centroid update: fixed-order fp32 sums over the sorted order, then mean / keep-old.
// ---------------------------------------------------------------------------------------
constexpr int kSlabMin = 256;

// Rows [s0, s1) of slab z when a cluster is cut into `nslabs` pieces of at least kSlabMin rows.
__device__ __forceinline__ void slab_range(int begin, int end, int z, int nslabs, int& s0, int& s1) {
  const int size = end - begin;
  int per = (size + nslabs - 1) / nslabs;
  per = per < kSlabMin ? kSlabMin : per;
  s0 = begin + z * per;
  s1 = s0 + per < end ? s0 + per : end;
}

__global__ void __launch_bounds__(256) centroid_partial_kernel(const bf16* __restrict__ x,
                                                               const int32_t* __restrict__ sorted_idx,
                                                               const int32_t* __restrict__ offsets,
                                                               float* __restrict__ partial, int N, int K, int nslabs,
                                                               int64_t x_head_rows) {
  __shared__ float red[16][kHeadDim + 4];
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x, z = blockIdx.y, bh = blockIdx.z;
  const int begin = offsets[(int64_t)bh * (K + 1) + c], end = offsets[(int64_t)bh * (K + 1) + c + 1];
  int s0, s1;
  slab_range(begin, end, z, nslabs, s0, s1);
  if (s0 >= s1) return;
  const int grp = threadIdx.x / 16, lane = threadIdx.x % 16;
  const int32_t* idx = sorted_idx + (int64_t)bh * N;
  const bf16* xb = x + bh * x_head_rows * kHeadDim;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  // a thread adds rows s0 + grp + 16 k, k = 0, 1, 2, ... in that order; eight gathers are in flight
  for (int s = s0 + grp; s < s1; s += 128) {
    int row[8];
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int ss = s + u * 16;
      row[u] = ss < s1 ? idx[ss] : -1;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (row[u] >= 0) {
        v[u] = __ldg(reinterpret_cast<const uint4*>(xb + (int64_t)row[u] * kHeadDim) + lane);
      } else {
        v[u] = make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[u]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[2 * i] += __low2float(h[i]);
        acc[2 * i + 1] += __high2float(h[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[grp][lane * 8 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < kHeadDim) {
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < 16; ++g) s += red[g][threadIdx.x];
    partial[(((int64_t)bh * K + c) * kCentroidSlabs + z) * kHeadDim + threadIdx.x] = s;
  }
}

// Four clusters per CTA (one per group of 128 threads): a CTA per cluster would be 20,000 CTAs of
// a few hundred bytes of work each at 40 heads x 500 clusters.
constexpr int kFinalizePerCta = 4;
__global__ void __launch_bounds__(128 * kFinalizePerCta) centroid_finalize_kernel(
    const float* __restrict__ partial, const int32_t* __restrict__ offsets, const bf16* __restrict__ old_c,
    bf16* __restrict__ new_c, int32_t* __restrict__ sizes, int K, int nslabs) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * kFinalizePerCta + threadIdx.x / 128, bh = blockIdx.y, d = threadIdx.x % 128;
  if (c >= K) return;
  const int begin = offsets[(int64_t)bh * (K + 1) + c], end = offsets[(int64_t)bh * (K + 1) + c + 1];
  const int cnt = end - begin;
  const int64_t o = ((int64_t)bh * K + c) * kHeadDim + d;
  float s = 0.f;
  for (int z = 0; z < nslabs; ++z) {
    int s0, s1;
    slab_range(begin, end, z, nslabs, s0, s1);
    if (s0 < s1) s += partial[(((int64_t)bh * K + c) * kCentroidSlabs + z) * kHeadDim + d];
  }
  const bf16 keep = old_c[o];
  new_c[o] = cnt > 0 ? __float2bfloat16_rn(s / (float)cnt) : keep;
  if (d == 0 && sizes) sizes[(int64_t)bh * K + c] = cnt;
}

// sizes [BH,K] -> offsets [BH,K+1]; thread k owns entries 2k and 2k + 1 (K <= 2048)
__global__ void __launch_bounds__(1024) offsets_from_sizes_kernel(const int32_t* __restrict__ sizes,
                                                                  int32_t* __restrict__ offsets, int K) {
  __shared__ int warp_tot[32];
  const int bh = blockIdx.x, k = threadIdx.x, lane = k % 32, warp = k / 32;
  const int v0 = 2 * k < K ? sizes[(int64_t)bh * K + 2 * k] : 0;
  const int v1 = 2 * k + 1 < K ? sizes[(int64_t)bh * K + 2 * k + 1] : 0;
  const int v = v0 + v1;
  int incl = v;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, s);
    if (lane >= s) incl += o;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int t = warp_tot[lane];
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, t, s);
      if (lane >= s) t += o;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  const int excl = incl - v + (warp ? warp_tot[warp - 1] : 0);
  int32_t* out = offsets + (int64_t)bh * (K + 1);
  if (2 * k < K) out[2 * k] = excl;
  if (2 * k + 1 < K) out[2 * k + 1] = excl + v0;
  if (2 * k == K - 1) out[K] = excl + v0;
  if (2 * k + 1 == K - 1) out[K] = excl + v;
}

// ---------------------------------------------------------------------------------------
// Host launchers (called from api.cu)
// ---------------------------------------------------------------------------------------
// x_head_rows >= N: rows from one head of x to the next.
cudaError_t launch_gather_rows(const void* x, int64_t x_head_rows, const int32_t* idx, void* out, int64_t BH, int64_t N,
                               int64_t K, cudaStream_t st) {
  dim3 grid((unsigned)ceil_div64(K, 16), (unsigned)BH);
  count_launches(1);
  return launch_pdl(gather_rows_kernel, grid, dim3(256), 0, st, (const bf16*)x, idx, (bf16*)out, (int)N, (int)K, x_head_rows);
}

cudaError_t launch_prologue(const void* own, const void* form, void* w_hi, void* w_lo, int64_t BH, int64_t J,
                            int64_t K, cudaStream_t st) {
  const int Jpad = pad_clusters(J);
  const size_t smem = pro_smem_bytes((int)K);
  cudaError_t e = cudaFuncSetAttribute(profile_prologue_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)(Jpad / kProR), (unsigned)BH);
  count_launches(1);
  return launch_pdl(profile_prologue_kernel, grid, dim3(256), smem, st, (const bf16*)own, (const bf16*)form, (bf16*)w_hi,
                    (bf16*)w_lo, (int)J, (int)K, Jpad);
}

// Whether the device can place a cluster of `ctas` CTAs of the sort with the shared memory of the most clusters: sizes
// above 8 are not portable, and a partition of a GPU has fewer SMs to a GPC.  Asked once per device, kernel form
// and size; the answer is the device's.
using SortKernel = void (*)(const int2*, int32_t*, int32_t*, int32_t*, int, int, int);
static bool sort_cluster_fits(SortKernel kernel, int form, int dev, int ctas) {
  constexpr int kDevices = 64;
  static std::atomic<signed char> known[kDevices][5][5];                     // [log2 ctas]: 0 not asked, 1 yes, -1 no
  std::atomic<signed char>* cell = dev < kDevices ? &known[dev][form][31 - __builtin_clz(ctas)] : nullptr;
  const signed char before = cell ? cell->load(std::memory_order_relaxed) : 0;
  if (before) return before > 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kSortThreads);
  cfg.dynamicSmemBytes = sort_smem_bytes(SVOO_MAX_CLUSTERS);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (cell) cell->store(n >= 1 ? 1 : -1, std::memory_order_relaxed);
  return n >= 1;
}

// groups > 0: `labels` are first reduced from that many column groups of `partial` (see assign_tc.cu).
cudaError_t launch_sort_labels(const int2* partial, int groups, int32_t* labels, int64_t BH, int64_t N, int64_t K,
                               int32_t* sorted_idx, int32_t* offsets, cudaStream_t st) {
  SortKernel kernel = nullptr;
  switch (groups) {                                      // two per 256 (at most 128 clusters: 128) W rows
    case 0: kernel = sort_labels_kernel<0>; break;
    case 2: kernel = sort_labels_kernel<2>; break;
    case 4: kernel = sort_labels_kernel<4>; break;
    case 6: kernel = sort_labels_kernel<6>; break;
    case 8: kernel = sort_labels_kernel<8>; break;
    default: return cudaErrorInvalidValue;
  }
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_smem_bytes(SVOO_MAX_CLUSTERS));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int ctas = sort_cluster_ctas(BH, N, K, sms, [&](int n) { return sort_cluster_fits(kernel, groups / 2, dev, n); });
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(BH * ctas));
  cfg.blockDim = dim3(kSortThreads);
  cfg.dynamicSmemBytes = sort_smem_bytes(K);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)ctas;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  count_launches(1);
  return cudaLaunchKernelEx(&cfg, kernel, partial, labels, sorted_idx, offsets, (int)BH, (int)N, (int)K);
}

cudaError_t launch_centroid_update(const void* x, int64_t x_head_rows, const int32_t* sorted_idx, const int32_t* offsets,
                                   const void* old_c, void* new_c, int32_t* sizes, float* partial, int64_t BH,
                                   int64_t N, int64_t K, cudaStream_t st) {
  // slabs per cluster: enough for clusters of four times the mean size to keep the 256-row minimum,
  // at most kCentroidSlabs; larger clusters just get longer slabs (most launched CTAs of a finer
  // split would find their slab empty)
  int nslabs = (int)ceil_div64(4 * ceil_div64(N, K), kSlabMin);
  nslabs = nslabs < 1 ? 1 : (nslabs > kCentroidSlabs ? kCentroidSlabs : nslabs);
  dim3 grid((unsigned)K, (unsigned)nslabs, (unsigned)BH);
  cudaError_t e = launch_pdl(centroid_partial_kernel, grid, dim3(256), 0, st, (const bf16*)x, sorted_idx, offsets, partial,
                             (int)N, (int)K, nslabs, x_head_rows);
  if (e != cudaSuccess) return e;
  dim3 grid2((unsigned)ceil_div64(K, kFinalizePerCta), (unsigned)BH);
  count_launches(2);
  return launch_pdl(centroid_finalize_kernel, grid2, dim3(128 * kFinalizePerCta), 0, st, (const float*)partial, offsets, (const bf16*)old_c,
                    (bf16*)new_c, sizes, (int)K, nslabs);
}

cudaError_t launch_offsets_from_sizes(const int32_t* sizes, int32_t* offsets, int64_t BH, int64_t K, cudaStream_t st) {
  offsets_from_sizes_kernel<<<(unsigned)BH, 1024, 0, st>>>(sizes, offsets, (int)K);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace svoo

// ---------------------------------------------------------------------------------------
// svoo_b200_sort_labels_static: the label sort for callers that cannot hand over a workspace (device memory
// carved up once at start-up, a plug-in without an allocator, a loop that must not meet the implicit
// synchronisation of an allocation).  The sort keeps its counts in shared memory, so it needs no scratch at
// all; the size limit of the entry point (it once had a fixed scratch array) is part of its interface.
// ---------------------------------------------------------------------------------------
extern "C" int svoo_b200_sort_labels_static(const int32_t* labels, int64_t BH, int64_t N, int64_t K,
                                            int32_t* sorted_idx, int32_t* offsets, void* stream) {
  using namespace svoo;
  constexpr int64_t kMaxCounts = 1 << 20, kCountChunk = 2048;
  if (!labels || !sorted_idx || !offsets) return SVOO_ERR_NULL;
  if (BH < 1 || BH > 65535 || N < 1 || N > (1 << 24) || K < 1 || BH * N > (int64_t)INT32_MAX) return SVOO_ERR_SHAPE;
  if (K > SVOO_MAX_CLUSTERS) return SVOO_ERR_CLUSTERS;
  if (BH * ceil_div64(N, kCountChunk) * K > kMaxCounts) return SVOO_ERR_STATIC_SCRATCH;
  cudaError_t e = launch_sort_labels(nullptr, 0, const_cast<int32_t*>(labels), BH, N, K, sorted_idx, offsets, (cudaStream_t)stream);
  return e == cudaSuccess ? SVOO_OK : (int)e;
}
