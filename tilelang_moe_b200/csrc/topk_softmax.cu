// Fused top-k + softmax router kernels for sm_100a.
//
// Four kernels behind one entry point:
//   * topk_group_kernel  4-32 lanes per row, the row in their registers, a threshold from part maxima, then a ranking of
//                        the few logits not below it; N <= 1024, k <= 8, aligned rows, M >= 2048 or N > 256.
//   * topk_lane_kernel   the same with one lane per row, staged through shared memory; N <= 32.
//   * topk_warp_kernel   one warp per row, the row lives in registers; k rounds of
//                        warp-wide arg-max by redux; N <= 1024, k <= 64.
//   * topk_radix_kernel  a thread-block cluster per row; each CTA keeps its share of
//                        the row in registers, the cluster runs a radix select on
//                        order-preserving keys with histograms combined over
//                        distributed shared memory until few enough are left, every
//                        CTA sorts its part (bitonic, 64-bit key|index) and places
//                        it by binary search in the other CTAs' parts.
// All read every logit once from HBM.
//
// Ordering contract: descending by value, equal values lowest index first,
// -0.0 == +0.0, NaN above every number.
#include "common.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace moe {

// ------------------------------------------------------------------------------------
// warp-per-row kernel
// ------------------------------------------------------------------------------------
template <int ELTS, int VEC>
__device__ __forceinline__ uint32_t warp_col(int i, int lane) {
  if (VEC == 4) return (uint32_t)((i >> 2) * 128 + lane * 4 + (i & 3));
  return (uint32_t)(i * 32 + lane);
}

template <int ELTS, int VEC>
__global__ void __launch_bounds__(128)
topk_warp_kernel(const float* __restrict__ logits, int64_t M, int N, int64_t ld, int k, int mode,
                 float* __restrict__ scores, int64_t* __restrict__ idx64, int32_t* __restrict__ idx32) {
  pdl_trigger();
  const unsigned FULL = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * 4;
  for (int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); row < M; row += nwarps) {
    const float* p = logits + row * ld;
    uint32_t key[ELTS];
    if (VEC == 4) {
#pragma unroll
      for (int c = 0; c < ELTS / 4; ++c) {
        const int col0 = c * 128 + lane * 4;
        if (col0 < N) {  // N % 4 == 0 on this path: the whole vector is in range
          const float4 v = __ldg(reinterpret_cast<const float4*>(p + col0));
          key[c * 4 + 0] = float_to_key(v.x);
          key[c * 4 + 1] = float_to_key(v.y);
          key[c * 4 + 2] = float_to_key(v.z);
          key[c * 4 + 3] = float_to_key(v.w);
        } else {
          key[c * 4 + 0] = key[c * 4 + 1] = key[c * 4 + 2] = key[c * 4 + 3] = 0u;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < ELTS; ++i) {
        const int col = i * 32 + lane;
        key[i] = col < N ? float_to_key(__ldg(p + col)) : 0u;
      }
    }

    // lane-local best (strict > keeps the lowest column among equals: columns grow with i)
    uint32_t bk = 0u, bc = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < ELTS; ++i) {
      if (key[i] > bk) { bk = key[i]; bc = warp_col<ELTS, VEC>(i, lane); }
    }
    const uint32_t maxkey = __reduce_max_sync(FULL, bk);
    const float vmax = key_to_float(maxkey);

    float rowsum = 0.f;
    if (mode != MOE_TOPK_MODE_B) {
#pragma unroll
      for (int i = 0; i < ELTS; ++i)
        if (key[i] != 0u) rowsum += expf(key_to_float(key[i]) - vmax);
      rowsum = warp_sum(rowsum);
    }

    uint32_t selk0 = 0u, selk1 = 0u, selc0 = 0u, selc1 = 0u;
    for (int r = 0; r < k; ++r) {
      const uint32_t m = __reduce_max_sync(FULL, bk);
      const uint32_t c = __reduce_min_sync(FULL, (bk == m) ? bc : 0xFFFFFFFFu);
      if (lane == (r & 31)) {
        if (r < 32) { selk0 = m; selc0 = c; } else { selk1 = m; selc1 = c; }
      }
      if (bk == m && bc == c) {  // the owning lane retires the winner and rescans its registers
        bk = 0u; bc = 0xFFFFFFFFu;
#pragma unroll
        for (int i = 0; i < ELTS; ++i) {
          if (warp_col<ELTS, VEC>(i, lane) == c) key[i] = 0u;
          if (key[i] > bk) { bk = key[i]; bc = warp_col<ELTS, VEC>(i, lane); }
        }
      }
    }

    const bool v0 = lane < k, v1 = lane + 32 < k;
    float e0 = v0 ? expf(key_to_float(selk0) - vmax) : 0.f;
    float e1 = v1 ? expf(key_to_float(selk1) - vmax) : 0.f;
    float s0, s1;
    if (mode == MOE_TOPK_MODE_B) {
      const float denom = warp_sum(e0 + e1);
      s0 = e0 / denom; s1 = e1 / denom;
    } else {
      s0 = e0 / rowsum; s1 = e1 / rowsum;
      if (mode == MOE_TOPK_MODE_A_RENORM) {
        const float s = warp_sum(s0 + s1);
        s0 = s0 / s; s1 = s1 / s;
      }
    }
    const int64_t o = row * (int64_t)k;
    if (v0) {
      scores[o + lane] = s0;
      if (idx64) idx64[o + lane] = (int64_t)selc0;
      if (idx32) idx32[o + lane] = (int32_t)selc0;
    }
    if (v1) {
      scores[o + lane + 32] = s1;
      if (idx64) idx64[o + lane + 32] = (int64_t)selc1;
      if (idx32) idx32[o + lane + 32] = (int32_t)selc1;
    }
  }
}

template <int ELTS, int VEC>
static int launch_warp(const float* logits, int64_t M, int N, int64_t ld, int k, int mode, float* scores,
                       int64_t* idx64, int32_t* idx32, int sm_count, cudaStream_t st) {
  int64_t blocks = ceil_div64(M, 4);
  const int64_t cap = (int64_t)sm_count * 16;
  if (blocks > cap) blocks = cap;
  topk_warp_kernel<ELTS, VEC><<<(unsigned)blocks, 128, 0, st>>>(logits, M, N, ld, k, mode, scores, idx64, idx32);
  MOE_CHECK_LAUNCH("topk_warp_kernel");
  return MOE_OK;
}


// ------------------------------------------------------------------------------------
// lane-group kernel for small k (k <= 8, N <= 1024, N % 4 == 0, 16-byte aligned rows)
//
// L = 4 .. 32 neighbouring lanes share a row, EPT = 8 .. 32 logits per lane, straight from global memory into registers
// with 16-byte loads (the only pass over the logits).  A row is never ordered as a whole:
//   1. every lane takes the maxima of four parts of its logits, strided over the row; the group merges them over shuffles
//      (sorted lists, the upper half kept) into V, the K-th largest of the 4 * L part maxima - a lower bound of the K-th largest logit;
//   2. the logits not below V, seven or eight of them as a rule, are collected in shared memory as 64-bit key | column
//      entries (equal keys: lowest column first);
//   3. each lane ranks its share of them against all of them; the entries of rank < k are the result, in order.
// NaNs do not enter V (max and min ignore them) and are never below it, so they are collected and rank first by key.
// A warp with more than CAP entries in one of its rows takes the logits equal to V in column order, as many as those above V
// leave of K; where the logits above V alone are too many (rows sorted by expert), every lane keeps a sorted list.
//
// What bounds it: instruction issue at N = 128, HBM from N = 512 on.  Few rows: the chain of one warp.  Measured (us,
// thread-per-row tiles with a list of K per thread before -> now): 1048576 x 128, k = 6: 169 -> 138 (HBM 93);
// 131072 x 256, k = 8: 65.7 -> 34.3; 131072 x 1024, k = 8: 291 -> 115 (HBM 84); 16384 x 256: 11.7 -> 6.8; 2048 x 256:
// 8.8 -> 3.4.  With a few lanes per row 32 warps per SM fit beside each other; the tiles had 12.  Equal logits: 131072 x
// 128, k = 6 all equal 25.0 -> 20.8, rounded to integers 29.0 -> 23.6; rounded, k = 8: 32768 x 128 13.2 -> 11.2, 131072 x 64
// 33.0 -> 20.9.  Slower than the tiles and the warp kernel: rounded to integers, k = 2, 32768 x 36 4.8 -> 6.2, x 100 6.1 -> 6.8 (a
// dozen entries to rank for two places), and 64 x 300, k = 8 3.9 -> 4.5.
// ------------------------------------------------------------------------------------
constexpr int GROUP_WARPS = 8;

__device__ __forceinline__ void ce_desc(float& a, float& b) {
  const float hi = fmaxf(a, b), lo = fminf(a, b);
  a = hi; b = lo;
}
// s is bitonic: sorts it descending
template <int P>
__device__ __forceinline__ void bitonic_merge_desc(float (&s)[P]) {
#pragma unroll
  for (int st = P / 2; st > 0; st >>= 1)
#pragma unroll
    for (int i = 0; i < P; ++i)
      if ((i & st) == 0) ce_desc(s[i], s[i | st]);
}

template <int K, int L, int EPT>
__global__ void __launch_bounds__(GROUP_WARPS * 32, EPT == 32 ? 4 : 5)
topk_group_kernel(const float* __restrict__ logits, int64_t M, int N, int64_t ld, int k, int mode,
                  float* __restrict__ scores, int64_t* __restrict__ idx64, int32_t* __restrict__ idx32) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int RPW = 32 / L;                       // rows per warp
  constexpr int CAP = L == 32 ? 32 : 16;            // entries a row may collect
  constexpr int HELD = CAP / L;                     // entries a lane ranks
  constexpr int P = K > 4 ? 8 : (K > 2 ? 4 : 2);    // length of the merged lists of maxima
  __shared__ uint64_t cand_s[GROUP_WARPS][RPW][CAP + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & (L - 1), rw = lane / L;
  const int64_t row0 = ((int64_t)blockIdx.x * GROUP_WARPS + warp) * RPW;
  pdl_trigger();
  if (row0 >= M) return;                            // whole warps only: no block barrier below
  const int64_t row = row0 + rw;
  const bool live = row < M;
  const float* p = logits + (live ? row : M - 1) * ld;
  uint64_t* cand = cand_s[warp][rw];
  const float NEG_INF = __int_as_float((int)0xFF800000);

  // logits 4i .. 4i+3 of this lane are columns 4 * (i * L + sub) ...: a group reads 16 * L consecutive bytes at a time
  float x[EPT];
  uint32_t valid = 0u;
#pragma unroll
  for (int i = 0; i < EPT / 4; ++i) {
    const int col = 4 * (i * L + sub);
    if (col < N) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p + col));
      x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
      valid |= 0xFu << (4 * i);
    } else {
      x[4 * i] = x[4 * i + 1] = x[4 * i + 2] = x[4 * i + 3] = NEG_INF;
    }
  }

  // ---- 1. V.  Part q of a lane holds the q-th logits of all its vectors: parts are equally long for every N, and a masked
  //      run of columns takes as much from each
  float g[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float m = NEG_INF;
#pragma unroll
    for (int i = 0; i < EPT / 4; ++i) m = fmaxf(m, x[4 * i + q]);
    g[q] = m;
  }
  ce_desc(g[0], g[1]); ce_desc(g[2], g[3]); ce_desc(g[0], g[2]); ce_desc(g[1], g[3]); ce_desc(g[1], g[2]);
  float s[P];
  if (P == 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { s[i] = g[i]; s[P - 1 - i] = __shfl_xor_sync(FULL, g[i], 1); }
    bitonic_merge_desc<P>(s);
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) s[i] = g[i];
  }
#pragma unroll
  for (int d = P == 8 ? 2 : 1; d < L / 2; d <<= 1) {
    float o[P];
#pragma unroll
    for (int i = 0; i < P; ++i) o[i] = __shfl_xor_sync(FULL, s[i], d);
#pragma unroll
    for (int i = 0; i < P; ++i) s[i] = fmaxf(s[i], o[P - 1 - i]);
    bitonic_merge_desc<P>(s);
  }
  float V;
  {   // K-th largest of two descending lists: the best split into i entries of one and K - i of the other
    float o[K];
#pragma unroll
    for (int i = 0; i < K; ++i) o[i] = __shfl_xor_sync(FULL, s[i], L / 2);
    V = fmaxf(s[K - 1], o[K - 1]);
#pragma unroll
    for (int i = 1; i < K; ++i) V = fmaxf(V, fminf(s[i - 1], o[K - i - 1]));
  }

  // ---- 2. collect
  uint32_t mask = 0u;
#pragma unroll
  for (int b = 0; b < EPT; ++b) mask |= !(x[b] < V) ? (1u << b) : 0u;
  mask &= valid;
  int mine_n = __popc(mask);
  int inc = mine_n;
#pragma unroll
  for (int d = 1; d < L; d <<= 1) {
    const int v = __shfl_up_sync(FULL, inc, d, L);
    if (sub >= d) inc += v;
  }
  int c = __shfl_sync(FULL, inc, L - 1, L);
  int cmax = __reduce_max_sync(FULL, c);
  if (cmax > CAP) {
    // many logits equal to V: collect those above it and, where these are fewer than K, the first of the equal ones, one
    // column at a time
    uint32_t eq = 0u;
#pragma unroll
    for (int b = 0; b < EPT; ++b) eq |= x[b] == V ? (1u << b) : 0u;
    eq &= mask;
    mask &= ~eq;
    mine_n = __popc(mask);
    inc = mine_n;
#pragma unroll
    for (int d = 1; d < L; d <<= 1) {
      const int v = __shfl_up_sync(FULL, inc, d, L);
      if (sub >= d) inc += v;
    }
    c = __shfl_sync(FULL, inc, L - 1, L);
    cmax = __reduce_max_sync(FULL, c);
    if (cmax <= CAP) {
      const uint64_t vkey = (uint64_t)float_to_key(V) << 32;
      for (int r = 0; r < K; ++r) {                 // a bound known to the compiler: with K - c the kernel was 1 % slower on every row
        const int b = __ffs(eq) - 1;
        const uint32_t col = eq ? (uint32_t)(4 * ((b >> 2) * L + sub) + (b & 3)) : 0xFFFFFFFFu;
        uint32_t first = col;
#pragma unroll
        for (int d = 1; d < L; d <<= 1) first = min(first, __shfl_xor_sync(FULL, first, d));
        if (first != 0xFFFFFFFFu && c < K) {
          if (col == first) {
            cand[c] = vkey | (uint64_t)(0xFFFFFFFFu - col);
            eq &= eq - 1;
          }
          ++c;
        }
      }
      cmax = __reduce_max_sync(FULL, c);
    } else {
      cmax = CAP + 1;
    }
  }
  if (cmax <= CAP) {
    int slot = inc - mine_n;
    while (mask) {                                  // the value comes from L1 again: registers have no dynamic index
      const int b = __ffs(mask) - 1;
      mask &= mask - 1;
      const int col = 4 * ((b >> 2) * L + sub) + (b & 3);
      cand[slot++] = ((uint64_t)float_to_key(__ldg(p + col)) << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)col);
    }
    __syncwarp();
    // ---- 3. rank
    uint64_t mine[HELD];
    int rank[HELD];
#pragma unroll
    for (int h = 0; h < HELD; ++h) {
      const int q = h * L + sub;
      mine[h] = q < c ? cand[q] : 0ull;
      rank[h] = 0;
    }
    for (int j = 0; j < cmax; ++j) {
      const uint64_t v = j < c ? cand[j] : 0ull;
#pragma unroll
      for (int h = 0; h < HELD; ++h)
        if (h == 0 || h * L < cmax) rank[h] += v > mine[h] ? 1 : 0;
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < HELD; ++h)
      if (h * L + sub < c && rank[h] < k) cand[rank[h]] = mine[h];
  } else {
    // every lane keeps a sorted list of its K largest (columns ascend within a lane, so equal keys keep the lowest
    // column first), then k rounds of arg-max over the heads of the group's lists
    int kv[K], ki[K];
#pragma unroll
    for (int j = 0; j < K; ++j) { kv[j] = (int)0x80000000; ki[j] = 0; }
#pragma unroll 1                                    // rolled, values from L1: unrolled it would cost the whole kernel registers
    for (int i = 0; i < EPT / 4; ++i) {
      const int col = 4 * (i * L + sub);
      if (col < N) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p + col));
        const int c0 = float_to_ikey(v.x), c1 = float_to_ikey(v.y), c2 = float_to_ikey(v.z), c3 = float_to_ikey(v.w);
        if (c0 > kv[K - 1]) list_insert<K>(kv, ki, c0, col);
        if (c1 > kv[K - 1]) list_insert<K>(kv, ki, c1, col + 1);
        if (c2 > kv[K - 1]) list_insert<K>(kv, ki, c2, col + 2);
        if (c3 > kv[K - 1]) list_insert<K>(kv, ki, c3, col + 3);
      }
    }
    for (int r = 0; r < k; ++r) {
      const uint64_t head = ((uint64_t)((uint32_t)kv[0] ^ 0x80000000u) << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)ki[0]);
      uint64_t top = head;
#pragma unroll
      for (int d = 1; d < L; d <<= 1) {
        const uint64_t o = __shfl_xor_sync(FULL, top, d);
        top = o > top ? o : top;
      }
      if (head == top && kv[0] != (int)0x80000000) {   // entries differ in their columns: one lane
        cand[r] = top;
#pragma unroll
        for (int j = 0; j + 1 < K; ++j) { kv[j] = kv[j + 1]; ki[j] = ki[j + 1]; }
        kv[K - 1] = (int)0x80000000;
      }
    }
  }
  __syncwarp();

  // ---- softmax over the k selected (mode B) or against the whole row (modes A)
  const float vmax = key_to_float((uint32_t)(cand[0] >> 32));
  constexpr int RL = (K + L - 1) / L;
  float e[RL];
  uint32_t ec[RL];
  float denom = 0.f;
#pragma unroll
  for (int t = 0; t < RL; ++t) {
    const int r = t * L + sub;
    e[t] = 0.f; ec[t] = 0u;
    if (r < k) {
      const uint64_t ent = cand[r];
      e[t] = expf(key_to_float((uint32_t)(ent >> 32)) - vmax);
      ec[t] = 0xFFFFFFFFu - (uint32_t)ent;
    }
    denom += e[t];
  }
  if (mode != MOE_TOPK_MODE_B) {
    denom = 0.f;
#pragma unroll
    for (int i = 0; i < EPT / 4; ++i)
      denom += (expf(x[4 * i] - vmax) + expf(x[4 * i + 1] - vmax)) + (expf(x[4 * i + 2] - vmax) + expf(x[4 * i + 3] - vmax));
  }
#pragma unroll
  for (int d = 1; d < L; d <<= 1) denom += __shfl_xor_sync(FULL, denom, d);
  float renorm = 0.f;
#pragma unroll
  for (int t = 0; t < RL; ++t) { e[t] = e[t] / denom; renorm += e[t]; }
  if (mode == MOE_TOPK_MODE_A_RENORM) {
#pragma unroll
    for (int d = 1; d < L; d <<= 1) renorm += __shfl_xor_sync(FULL, renorm, d);
#pragma unroll
    for (int t = 0; t < RL; ++t) e[t] = e[t] / renorm;
  }
  if (!live) return;
  const int64_t o = row * (int64_t)k;
#pragma unroll
  for (int t = 0; t < RL; ++t) {
    const int r = t * L + sub;
    if (r < k) {
      scores[o + r] = e[t];
      if (idx64) idx64[o + r] = (int64_t)ec[t];
      if (idx32) idx32[o + r] = (int32_t)ec[t];
    }
  }
}

template <int K, int L, int EPT>
static int launch_group(const float* logits, int64_t M, int N, int64_t ld, int k, int mode, float* scores,
                        int64_t* idx64, int32_t* idx32, cudaStream_t st) {
  const int64_t blocks = ceil_div64(M, GROUP_WARPS * (32 / L));     // M * 8 fits an int: so does this
  topk_group_kernel<K, L, EPT><<<(unsigned)blocks, GROUP_WARPS * 32, 0, st>>>(logits, M, N, ld, k, mode, scores, idx64, idx32);
  MOE_CHECK_LAUNCH("topk_group_kernel");
  return MOE_OK;
}

// ------------------------------------------------------------------------------------
// lane-per-row kernel: many rows of at most 32 logits, small k (k <= 8, N % 4 == 0, 16-byte aligned rows)
//
// With so few logits a row is one lane's work: a warp stages 32 rows in its own part of shared memory with 16-byte
// cp.async (coalesced, the only read of the logits), every lane takes V, the K-th largest of the maxima of 16 pairs of
// neighbouring logits (two sorted lists of eight) - a lower bound of the K-th largest logit - and passes the logits not
// below V (NaNs are not; they do not enter V either) in column order through a sorted list of K entries.  Scores and
// indices leave through shared memory as contiguous runs of the warp's 32 rows.
//
// What bounds it: the stores and the lists.  Measured (us, thread-per-row tiles before -> now): 1048576 x 16, k = 2:
// 58.8 -> 26.7; 1048576 x 8: 54.7 -> 24.8; 16384 x 16: 3.7 -> 2.6; all logits equal, 32768 x 32, k = 2: 4.3 -> 4.9.  (The same form for 128 logits: 132 us for 1048576 rows
// against 140 with four lanes per row, but twice its time on tied logits, and 6.7 against 4.9 us for 16384 rows: not built.)
// ------------------------------------------------------------------------------------
constexpr int LANE_WARPS = 4;
constexpr int LANE_NMAX = 32;

__device__ __forceinline__ void sort8_desc(float (&a)[16], int o) {   // 19 exchanges
  ce_desc(a[o + 0], a[o + 2]); ce_desc(a[o + 1], a[o + 3]); ce_desc(a[o + 4], a[o + 6]); ce_desc(a[o + 5], a[o + 7]);
  ce_desc(a[o + 0], a[o + 4]); ce_desc(a[o + 1], a[o + 5]); ce_desc(a[o + 2], a[o + 6]); ce_desc(a[o + 3], a[o + 7]);
  ce_desc(a[o + 0], a[o + 1]); ce_desc(a[o + 2], a[o + 3]); ce_desc(a[o + 4], a[o + 5]); ce_desc(a[o + 6], a[o + 7]);
  ce_desc(a[o + 2], a[o + 4]); ce_desc(a[o + 3], a[o + 5]);
  ce_desc(a[o + 1], a[o + 4]); ce_desc(a[o + 3], a[o + 6]);
  ce_desc(a[o + 1], a[o + 2]); ce_desc(a[o + 3], a[o + 4]); ce_desc(a[o + 5], a[o + 6]);
}

template <int K>
__global__ void __launch_bounds__(LANE_WARPS * 32)
topk_lane_kernel(const float* __restrict__ logits, int64_t M, int N, int64_t ld, int k, int mode,
                 float* __restrict__ scores, int64_t* __restrict__ idx64, int32_t* __restrict__ idx32) {
  constexpr int NV = LANE_NMAX / 4;
  pdl_trigger();
  __shared__ __align__(16) float lane_s[LANE_WARPS][32 * (LANE_NMAX + 4)];   // rows; later 32 x k scores and columns
  static_assert(32 * 8 * 2 <= 32 * (LANE_NMAX + 4), "the output of 32 rows fits where their logits were");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pitch = N + 4;                           // floats: rows stay 16-byte aligned and spread over the banks
  float* buf = lane_s[warp];
  const float* mine = buf + lane * pitch;
  const int nv = N >> 2;
  const int rpi = 32 / nv, lr = lane / nv, lc = lane - lr * nv;   // staging: rows per instruction, this lane's row and vector
  const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(buf) + (uint32_t)(lr * pitch + lc * 4) * 4u;
  const float NEG_INF = __int_as_float((int)0xFF800000);
  const int64_t n_tiles = (M + 31) / 32;

  for (int64_t tile = (int64_t)blockIdx.x * LANE_WARPS + warp; tile < n_tiles; tile += (int64_t)gridDim.x * LANE_WARPS) {
    const int64_t row0 = tile * 32;
    const int rows = (int)(M - row0 < 32 ? M - row0 : 32);
    __syncwarp();                                    // the previous tile's output has left the buffer
    if (lr < rpi) {
      const float* src = logits + (row0 + lr) * ld + lc * 4;
      uint32_t dst = dst0;
      for (int r = lr; r < rows; r += rpi) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        src += rpi * ld;
        dst += (uint32_t)(rpi * pitch) * 4u;
      }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncwarp();

    float x[LANE_NMAX], g[16];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float4 f = make_float4(NEG_INF, NEG_INF, NEG_INF, NEG_INF);
      if (v < nv) f = *reinterpret_cast<const float4*>(mine + v * 4);
      x[4 * v] = f.x; x[4 * v + 1] = f.y; x[4 * v + 2] = f.z; x[4 * v + 3] = f.w;
      g[2 * v] = fmaxf(NEG_INF, fmaxf(f.x, f.y));
      g[2 * v + 1] = fmaxf(NEG_INF, fmaxf(f.z, f.w));
    }
    sort8_desc(g, 0);
    sort8_desc(g, 8);
    float V = fmaxf(g[K - 1], g[8 + K - 1]);
#pragma unroll
    for (int i = 1; i < K; ++i) V = fmaxf(V, fminf(g[i - 1], g[8 + K - i - 1]));

    uint32_t m = 0u;
#pragma unroll
    for (int b = 0; b < LANE_NMAX; ++b) m |= !(x[b] < V) ? (1u << b) : 0u;
    m &= N < 32 ? (1u << N) - 1u : 0xFFFFFFFFu;
    if (lane >= rows) m = 0u;                        // lanes past the last row worked on whatever the buffer held

    int kv[K], ki[K];                                // equal keys: the earlier column stays ahead
#pragma unroll
    for (int j = 0; j < K; ++j) { kv[j] = (int)0x80000000; ki[j] = 0; }
    while (m) {
      const int col = __ffs(m) - 1;
      m &= m - 1u;
      list_insert<K>(kv, ki, float_to_ikey(mine[col]), col);
    }

    // softmax over the k selected (mode B) or against the whole row (modes A)
    const float vmax = ikey_to_float(kv[0]);
    float e[K];
    float denom = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      e[j] = j < k ? expf(ikey_to_float(kv[j]) - vmax) : 0.f;
      denom += e[j];
    }
    if (mode != MOE_TOPK_MODE_B) {                   // columns past N hold -inf: they add nothing
      denom = 0.f;
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (v < nv)
          denom += (expf(x[4 * v] - vmax) + expf(x[4 * v + 1] - vmax)) + (expf(x[4 * v + 2] - vmax) + expf(x[4 * v + 3] - vmax));
    }
    float renorm = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) { e[j] = e[j] / denom; renorm += e[j]; }
    if (mode == MOE_TOPK_MODE_A_RENORM) {
#pragma unroll
      for (int j = 0; j < K; ++j) e[j] = e[j] / renorm;
    }

    __syncwarp();                                    // every lane is done with its logits
    int* col_s = reinterpret_cast<int*>(buf) + 32 * k;
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (j < k) { buf[lane * k + j] = e[j]; col_s[lane * k + j] = ki[j]; }
    __syncwarp();
    const int64_t o = row0 * (int64_t)k;
    for (int i = lane; i < rows * k; i += 32) {
      scores[o + i] = buf[i];
      const int c = col_s[i];
      if (idx64) idx64[o + i] = (int64_t)c;
      if (idx32) idx32[o + i] = (int32_t)c;
    }
  }
}

template <int K>
static int launch_lane(const float* logits, int64_t M, int N, int64_t ld, int k, int mode, float* scores,
                       int64_t* idx64, int32_t* idx32, int sm_count, cudaStream_t st) {
  int64_t blocks = ceil_div64(M, 32 * LANE_WARPS);
  if (blocks > (int64_t)sm_count * 8) blocks = (int64_t)sm_count * 8;
  topk_lane_kernel<K><<<(unsigned)blocks, LANE_WARPS * 32, 0, st>>>(logits, M, N, ld, k, mode, scores, idx64, idx32);
  MOE_CHECK_LAUNCH("topk_lane_kernel");
  return MOE_OK;
}

// ------------------------------------------------------------------------------------
// cluster radix-select kernel
// ------------------------------------------------------------------------------------
constexpr int RT = 512;             // threads per CTA
constexpr int RWARPS = RT / 32;
constexpr int RBINS = 2048;         // histogram bins (11-bit digit)
constexpr int RBPT = RBINS / RT;    // bins owned by one thread in the scan (4)
constexpr int RCTRL_BYTES = 288;
constexpr int RCHUNKS = 512;        // 128-byte chunks of a row that one CTA holds (RMAX_SLICE / 32; one per thread in their scan)
constexpr int RMAX_SLICE = 16384;   // keys one CTA holds (32 per thread)
constexpr int RMAX_KPAD = 4096;

struct RadixCtrl {
  uint32_t warp_tot[RWARPS];
  double warp_d[RWARPS];
  uint32_t sel_bin;
  uint32_t k_rem;
  uint32_t bin_count;   // entries of the selected bin in the whole row
  uint32_t blk_maxkey;
  uint32_t loc_count;   // collected entries of this CTA
  double blk_sum;       // this CTA's share of the full-row denominator (modes A)
  double sel_sum;       // ... of a sum over the k selected
  uint2 cand[3];        // this CTA's candidates in passes 1, 2 and 3: smallest key, complement of the largest
};
static_assert(sizeof(RadixCtrl) <= RCTRL_BYTES && RCTRL_BYTES % 16 == 0, "control block too large");
static_assert(RMAX_SLICE / 32 <= RCHUNKS && RCHUNKS <= RT, "a thread per chunk");

__device__ __forceinline__ uint64_t pack_entry(uint32_t key, uint32_t col) {
  return ((uint64_t)key << 32) | (uint64_t)(0xFFFFFFFFu - col);
}

// Sum of one value per thread over the CTA in a fixed order; result valid in every thread.
// Softmax denominators over thousands of terms are accumulated in fp64 so that the only
// rounding left in a score is that of expf and of the final division.
__device__ __forceinline__ double block_sum_ordered(double v, RadixCtrl* ctrl, int lane, int wid) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  __syncthreads();
  if (lane == 0) ctrl->warp_d[wid] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < RWARPS; ++w) t += ctrl->warp_d[w];
  return t;
}

// Descending bitonic sort of RT*EPT 64-bit entries held EPT per thread (entry g = tid*EPT + e).
// Exchanges at distance < EPT stay in registers, distance < 32*EPT go through warp shuffles, and only the
// few long-distance stages of the last merges use shared memory with a block barrier.
template <int EPT>
__device__ __forceinline__ void block_sort_desc(uint64_t* sbuf, int tid) {
  constexpr int NSORT = RT * EPT;
  uint64_t v[EPT];
#pragma unroll
  for (int e = 0; e < EPT; ++e) v[e] = sbuf[tid * EPT + e];
  for (int size = 2; size <= NSORT; size <<= 1) {
    int stride = size >> 1;
    // long distance: through shared memory
    for (; stride >= 32 * EPT; stride >>= 1) {
      __syncthreads();
#pragma unroll
      for (int e = 0; e < EPT; ++e) sbuf[tid * EPT + e] = v[e];
      __syncthreads();
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const int g = tid * EPT + e;
        const uint64_t o = sbuf[g ^ stride];
        const bool keep_max = ((g & stride) == 0) == ((g & size) == 0);
        v[e] = keep_max ? (v[e] > o ? v[e] : o) : (v[e] < o ? v[e] : o);
      }
    }
    // inside a warp: shuffles
    for (; stride >= EPT; stride >>= 1) {
      const int lx = stride / EPT;
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const int g = tid * EPT + e;
        const uint64_t o = __shfl_xor_sync(0xFFFFFFFFu, v[e], lx);
        const bool keep_max = ((g & stride) == 0) == ((g & size) == 0);
        v[e] = keep_max ? (v[e] > o ? v[e] : o) : (v[e] < o ? v[e] : o);
      }
    }
    // inside a thread: registers (compile-time distances)
#pragma unroll
    for (int st = EPT / 2; st > 0; st >>= 1) {
      if (st <= (size >> 1)) {
#pragma unroll
        for (int e = 0; e < EPT; ++e) {
          if ((e & st) == 0) {
            const int g = tid * EPT + e;
            const bool desc = (g & size) == 0;
            const uint64_t a = v[e], b = v[e | st];
            const bool swap = (a < b) == desc;
            v[e] = swap ? b : a;
            v[e | st] = swap ? a : b;
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < EPT; ++e) sbuf[tid * EPT + e] = v[e];
  __syncthreads();
}

// entries of the descending list a[0 .. n) that are greater than x
__device__ __forceinline__ uint32_t count_above(const uint64_t* a, uint32_t n, uint64_t x) {
  uint32_t lo = 0u, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] > x) lo = mid + 1u; else hi = mid;
  }
  return lo;
}

// One cluster of C CTAs per row.  The row's 128-byte chunks go round the CTAs (a row in sorted order is spread evenly), each
// keeps its share as keys in registers, KPT per thread.
//   1. radix select on the key, 11 / 11 / 10 bits: histograms of all CTAs are added over distributed shared memory.  It stops
//      as soon as the entries not below the selected bin are few enough to be sorted outright (totcap), after one digit as a
//      rule.  Where the bin holds one value only (masked, constant or quantised rows; after three digits in any case), as many
//      of its entries as are needed are taken in column order: the CTAs exchange their counts per chunk at the same barrier.
//   2. every CTA collects those of its share and sorts them;
//   3. it copies the other CTAs' sorted entries; an entry's place in the row's order is its place in its own list plus, by
//      binary search, the entries of the other lists ahead of it.  Places below k are written out.
// What bounds it: latency (barriers, shared-memory atomics, the sort's chain of exchanges).
// Measured (us, gathering the k selected into the leading CTA and sorting them there after all three digits -> this):
// 64 x 32768, k = 2048: 43.7 -> 30.9; one such row 30.6 -> 19.3; 4096 x 4096, k = 64: 178 -> 138; 256 x 32768, k = 2048: 99.8 -> 88.5;
// 16 x 65536, k = 1024: 34.7 -> 26.4; 64 x 32768, k = 32: 19.8 -> 17.1.  Rows of equal logits (with two more digits, of the
// column, in place of the counts per chunk: in brackets): 64 x 32768, k = 32 20.2 -> 21.3 [26.8], k = 2048 45.4 -> 28.0 [32.9];
// 4096 x 2048, k = 8 138 -> 132 [201].  The counts cost registers: rows above 65536 that need all three digits and hold no
// ties, 32 x 131072, k = 64 35.8 -> 39.5 [35.7].
template <int KPT>
__global__ void __launch_bounds__(RT, 2)
topk_radix_kernel(const float* __restrict__ logits, int64_t M, int N, int64_t ld, int k, int totcap, int lcap, int mode,
                  int vec_ok, float* __restrict__ scores, int64_t* __restrict__ idx64,
                  int32_t* __restrict__ idx32, int32_t* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  const unsigned FULL = 0xFFFFFFFFu;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned C = cluster.num_blocks();
  const unsigned crank = cluster.block_rank();
  const int64_t row = blockIdx.x / C;

  RadixCtrl* ctrl = reinterpret_cast<RadixCtrl*>(smem_raw);
  uint32_t* hist = reinterpret_cast<uint32_t*>(smem_raw + RCTRL_BYTES);
  uint32_t* chunk_n = hist + 2 * RBINS;      // candidates per chunk of this CTA, read by the others
  uint32_t* chunk_at = chunk_n + RCHUNKS;    // candidates of the row in the chunks before each of them
  uint64_t* lbuf = reinterpret_cast<uint64_t*>(chunk_at + RCHUNKS);                       // [lcap] this CTA's entries
  uint64_t* others = lbuf + lcap;                                                         // [totcap] the other CTAs'

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) { ctrl->blk_maxkey = 0u; ctrl->blk_sum = 0.0; ctrl->sel_bin = 0u; ctrl->k_rem = 0u; ctrl->bin_count = 0u; }
  if (tid < 3) ctrl->cand[tid] = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
  for (int i = tid; i < 2 * RBINS; i += RT) hist[i] = 0u;

  // ---- this CTA's share as keys (the only read of the logits); 0 where there is none (no float has that key)
  const float* p = logits + row * ld;
  auto col_of = [&](int j) {                          // column of key j of this thread
    const int v = (j >> 2) * RT + tid;                // vector of four in the CTA's share, eight to a chunk
    return (((v >> 3) * (int)C + (int)crank) << 5) + ((v & 7) << 2) + (j & 3);
  };
  uint32_t key[KPT];
#pragma unroll
  for (int q = 0; q < KPT / 4; ++q) {
    const int i = col_of(4 * q);
    if (vec_ok) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      const bool in = i < N;                          // N % 4 == 0 on this path
      if (in) v = __ldg(reinterpret_cast<const float4*>(p + i));
      key[4 * q] = in ? float_to_key(v.x) : 0u;
      key[4 * q + 1] = in ? float_to_key(v.y) : 0u;
      key[4 * q + 2] = in ? float_to_key(v.z) : 0u;
      key[4 * q + 3] = in ? float_to_key(v.w) : 0u;
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) key[4 * q + c] = i + c < N ? float_to_key(__ldg(p + i + c)) : 0u;
    }
  }
  __syncthreads();  // control block and histograms initialised
  if (mode != MOE_TOPK_MODE_B) {
    uint32_t lmax = 0u;
#pragma unroll
    for (int j = 0; j < KPT; ++j) lmax = max(lmax, key[j]);
    lmax = __reduce_max_sync(FULL, lmax);
    if (lane == 0) atomicMax(&ctrl->blk_maxkey, lmax);
  }

  // ---- 1. radix select: `prefix` is the lowest key of the bin that holds the k-th largest entry (after three digits its key)
  uint32_t prefix = 0u, pmask = 0u, k_rem = (uint32_t)k;
  uint32_t m = 0u;                                    // keys that are taken
  double rowsum = 0.0;
  bool tied = false;
  auto count = [&](int w, uint32_t value) {         // this thread's keys of that value in vectors 4w .. 4w + 3, a byte each
    uint32_t n = 0u;
#pragma unroll
    for (int j = 16 * w; j < 16 * w + 16 && j < KPT; ++j) n += key[j] == value ? 1u << (8 * ((j >> 2) & 3)) : 0u;
    return n;
  };
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = pass == 0 ? 21 : (pass == 1 ? 10 : 0);
    const uint32_t dmask = pass == 2 ? 1023u : 2047u;
    uint32_t* h = hist + (pass & 1) * RBINS;
    if (pass == 2) {  // this buffer again: every remote read of it ended before the last pass's cluster barrier
      for (int i = tid; i < RBINS; i += RT) h[i] = 0u;
      __syncthreads();
    }
    uint32_t lo = 0xFFFFFFFFu, hi = 0u;               // smallest and largest candidate of this warp, then of the row
    if (pass == 0) {
#pragma unroll
      for (int j = 0; j < KPT; ++j)
        if (key[j] != 0u) atomicAdd(&h[key[j] >> 21], 1u);
    } else {
#pragma unroll
      for (int j = 0; j < KPT; ++j) {
        if (key[j] != 0u && (key[j] & pmask) == prefix) {
          if (pass < 3) atomicAdd(&h[(key[j] >> shift) & dmask], 1u);
          lo = min(lo, key[j]);
          hi = max(hi, key[j]);
        }
      }
    }
    if (pass > 0) {
      lo = __reduce_min_sync(FULL, lo);
      hi = __reduce_max_sync(FULL, hi);
      if (lane == 0 && hi != 0u) { atomicMin(&ctrl->cand[pass - 1].x, lo); atomicMin(&ctrl->cand[pass - 1].y, ~hi); }
      if (lo >= hi) {                                 // one value, or none: else the counts are of no use
#pragma unroll
        for (int w = 0; w < (KPT + 15) / 16; ++w) {   // over the eight lanes of a chunk
          uint32_t v = hi != 0u ? count(w, lo) : 0u;
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(FULL, v, o);
          if ((lane & 7) < 4 && 4 * w + (lane & 7) < KPT / 4)
            chunk_n[(4 * w + (lane & 7)) * (RT / 8) + (tid >> 3)] = (v >> (8 * (lane & 7))) & 0xFFu;
        }
      }
    }
    cluster.sync();

    uint2 cand = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
    if (pass > 0 && (unsigned)lane < C) cand = cluster.map_shared_rank(ctrl, lane)->cand[pass - 1];
    uint32_t g[RBPT];
#pragma unroll
    for (int j = 0; j < RBPT; ++j) g[j] = 0u;
#pragma unroll
    for (unsigned c = 0; c < 8; ++c) {   // all remote loads are issued before the first is consumed
      if (c < C) {
        const uint32_t* rh = cluster.map_shared_rank(h, c);
        const uint4 v = *reinterpret_cast<const uint4*>(rh + tid * RBPT);
        g[0] += v.x; g[1] += v.y; g[2] += v.z; g[3] += v.w;
      }
    }
    if (pass > 0) {
      lo = __reduce_min_sync(FULL, cand.x);
      hi = ~__reduce_min_sync(FULL, cand.y);
      if (lo == hi) { prefix = lo; tied = true; break; }   // the same in every CTA of the cluster
    }
    const uint32_t tsum = g[0] + g[1] + g[2] + g[3];
    uint32_t inc = tsum;  // suffix-inclusive sum over lanes >= lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t n = __shfl_down_sync(FULL, inc, o);
      if (lane + o < 32) inc += n;
    }
    if (lane == 0) ctrl->warp_tot[wid] = inc;
    __syncthreads();
    uint32_t S = inc - tsum;
    for (int w = wid + 1; w < RWARPS; ++w) S += ctrl->warp_tot[w];
#pragma unroll
    for (int j = RBPT - 1; j >= 0; --j) {
      if (S < k_rem && k_rem <= S + g[j]) {
        ctrl->sel_bin = (uint32_t)(tid * RBPT + j);
        ctrl->k_rem = k_rem - S;
        ctrl->bin_count = g[j];
      }
      S += g[j];
    }
    __syncthreads();
    const uint32_t bin = ctrl->sel_bin;
    k_rem = ctrl->k_rem;
    const uint32_t total_ge = (uint32_t)k - k_rem + ctrl->bin_count;
    prefix |= bin << shift;
    pmask |= dmask << shift;

    if (pass == 0 && mode != MOE_TOPK_MODE_B) {
      // full-row softmax denominator: cluster max, then this CTA's share of sum exp(v - max)
      uint32_t gmax = 0u;
      for (unsigned c = 0; c < C; ++c) gmax = max(gmax, cluster.map_shared_rank(ctrl, c)->blk_maxkey);
      const float vmax = key_to_float(gmax);
      double part = 0.0;
#pragma unroll
      for (int j = 0; j < KPT; ++j)
        if (key[j] != 0u) part += (double)expf(key_to_float(key[j]) - vmax);
      part = block_sum_ordered(part, ctrl, lane, wid);
      if (tid == 0) ctrl->blk_sum = part;  // published by the next cluster barrier
    }
    if (total_ge <= (uint32_t)totcap) break;          // the same in every CTA of the cluster; pass 3 never gets here
    __syncthreads();                                  // every thread has read the selection before the next pass replaces it
  }

  if (tied) {                                         // k_rem of the entries equal to prefix
    // thread t: chunk t of every CTA.  Row order is chunk by chunk, and within a chunk number the CTAs in turn
    uint32_t all = 0u, ahead = 0u;
    if (tid < KPT * 16) {
#pragma unroll
      for (unsigned c = 0; c < 8; ++c) {
        if (c < C) {
          const uint32_t v = cluster.map_shared_rank(chunk_n, c)[tid];
          all += v;
          if (c < crank) ahead += v;
        }
      }
    }
    uint32_t inc = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) ctrl->warp_tot[wid] = inc;
    __syncthreads();
    uint32_t before = ahead + inc - all;
#pragma unroll
    for (int w = 0; w < RWARPS; ++w) before += w < wid ? ctrl->warp_tot[w] : 0u;
    chunk_at[tid] = before;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < (KPT + 15) / 16; ++w) {
      const uint32_t own = count(w, prefix);
      uint32_t lower = own;                       // candidates of the chunk's lanes up to this one: at most 32, a byte each
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, lower, o, 8);
        if ((lane & 7) >= o) lower += v;
      }
      lower -= own;
#pragma unroll
      for (int q = 4 * w; q < KPT / 4 && q < 4 * w + 4; ++q) {
        uint32_t r = chunk_at[q * (RT / 8) + (tid >> 3)] + ((lower >> (8 * (q & 3))) & 0xFFu);
#pragma unroll
        for (int j = 4 * q; j < 4 * q + 4; ++j)
          if (key[j] == prefix) { m |= r < k_rem ? (1u << j) : 0u; ++r; }
      }
    }
  }

  // ---- 2. collect
#pragma unroll
  for (int j = 0; j < KPT; ++j) m |= (key[j] != 0u && (tied ? key[j] > prefix : key[j] >= prefix)) ? (1u << j) : 0u;
  uint32_t total = 0u;
  {
    const uint32_t n = (uint32_t)__popc(m);
    uint32_t inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += v;
    }
    __syncthreads();
    if (lane == 31) ctrl->warp_tot[wid] = inc;
    __syncthreads();
    uint32_t slot = inc - n;
#pragma unroll
    for (int w = 0; w < RWARPS; ++w) {
      const uint32_t t = ctrl->warp_tot[w];
      if (w < wid) slot += t;
      total += t;
    }
#pragma unroll
    for (int j = 0; j < KPT; ++j)
      if ((m >> j) & 1u) lbuf[slot++] = pack_entry(key[j], (uint32_t)col_of(j));
  }
  // ---- sort, descending; unused places are 0 and sink to the end.  From 129 entries on in registers and shuffles,
  //      below that the plain shared-memory network
  int size = 2;
  while (size < (int)total) size <<= 1;
  if (size > 128 && size < RT) size = RT;
  for (int i = (int)total + tid; i < size; i += RT) lbuf[i] = 0ull;
  if (tid == 0) ctrl->loc_count = total;
  __syncthreads();
  if (size >= RT) {   // block-uniform
    if (size == RT) block_sort_desc<1>(lbuf, tid);
    else if (size == 2 * RT) block_sort_desc<2>(lbuf, tid);
    else if (size == 4 * RT) block_sort_desc<4>(lbuf, tid);
    else block_sort_desc<8>(lbuf, tid);
  } else {
    for (int sz = 2; sz <= size; sz <<= 1) {
      for (int stride = sz >> 1; stride > 0; stride >>= 1) {
        for (int t = tid; t < (size >> 1); t += RT) {
          const int i = 2 * t - (t & (stride - 1));
          const int j = i + stride;
          const bool desc = (i & sz) == 0;
          const uint64_t a = lbuf[i], b = lbuf[j];
          if ((a < b) == desc) { lbuf[i] = b; lbuf[j] = a; }
        }
        __syncthreads();
      }
    }
  }

  // ---- 3. the other CTAs' entries, and every entry's place in the row
  uint32_t cnt[8], all = total;
  float vmax = key_to_float((uint32_t)(lbuf[0] >> 32));
  rowsum = ctrl->blk_sum;
  if (C > 1) {
    cluster.sync();                                   // sorted lists, counts and denominators of all CTAs are there
    uint32_t at = 0u, top = 0u;
    all = 0u;
    rowsum = 0.0;
#pragma unroll
    for (unsigned c = 0; c < 8; ++c) {
      cnt[c] = 0u;
      if (c < C) {
        const RadixCtrl* rc = cluster.map_shared_rank(ctrl, c);
        const uint32_t n = rc->loc_count;
        rowsum += rc->blk_sum;
        const uint64_t* rl = cluster.map_shared_rank(lbuf, c);
        if (n > 0u) top = max(top, (uint32_t)(rl[0] >> 32));
        all += n;
        if (c != crank) {
          for (uint32_t i = tid; i < n; i += RT) others[at + i] = rl[i];
          cnt[c] = n;
          at += n;
        }
      }
    }
    vmax = key_to_float(top);
    __syncthreads();
  }
  if (tid == 0 && crank == 0 && all < (uint32_t)k && status) {
    status[0] = ST_INTERNAL; status[1] = (int32_t)all; status[2] = (int32_t)row;
  }
  auto place = [&](uint32_t i, uint64_t ent) {        // entry i of this CTA's list
    uint32_t r = i, at = 0u;
    if (C > 1) {
#pragma unroll
      for (unsigned c = 0; c < 8; ++c)
        if (c < C) { r += count_above(others + at, cnt[c], ent); at += cnt[c]; }
    }
    return r;
  };
  constexpr int EMAX = 8;                             // RMAX_KPAD / RT entries per thread at most
  uint32_t rank[EMAX];
  double part = 0.0;
#pragma unroll
  for (int e = 0; e < EMAX; ++e) {
    const uint32_t i = (uint32_t)(e * RT + tid);
    rank[e] = 0xFFFFFFFFu;
    if (i < total) {
      const uint64_t ent = lbuf[i];
      rank[e] = place(i, ent);
      if (mode == MOE_TOPK_MODE_B && rank[e] < (uint32_t)k) part += (double)expf(key_to_float((uint32_t)(ent >> 32)) - vmax);
    }
  }
  float denom = (float)rowsum;
  if (mode == MOE_TOPK_MODE_A_RENORM) {
#pragma unroll
    for (int e = 0; e < EMAX; ++e)
      if (rank[e] < (uint32_t)k)
        part += (double)(expf(key_to_float((uint32_t)(lbuf[e * RT + tid] >> 32)) - vmax) / denom);
  }
  float renorm = 1.f;
  if (mode != MOE_TOPK_MODE_A) {                      // a sum over the k selected, added up over the cluster
    double sum = block_sum_ordered(part, ctrl, lane, wid);
    if (C > 1) {
      if (tid == 0) ctrl->sel_sum = sum;
      cluster.sync();
      sum = 0.0;
      for (unsigned c = 0; c < C; ++c) sum += cluster.map_shared_rank(ctrl, c)->sel_sum;
    }
    if (mode == MOE_TOPK_MODE_B) denom = (float)sum; else renorm = (float)sum;
  }
  const int64_t o = row * (int64_t)k;
#pragma unroll
  for (int e = 0; e < EMAX; ++e) {
    if (rank[e] < (uint32_t)k) {
      const uint64_t ent = lbuf[e * RT + tid];
      float s = expf(key_to_float((uint32_t)(ent >> 32)) - vmax) / denom;
      if (mode == MOE_TOPK_MODE_A_RENORM) s = s / renorm;
      const uint32_t col = 0xFFFFFFFFu - (uint32_t)(ent & 0xFFFFFFFFull);
      scores[o + rank[e]] = s;
      if (idx64) idx64[o + rank[e]] = (int64_t)col;
      if (idx32) idx32[o + rank[e]] = (int32_t)col;
    }
  }
  if (C > 1) cluster.sync();                          // nobody leaves while its shared memory is still read
}

static int next_pow2(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}

static int launch_radix(const float* logits, int64_t M, int N, int64_t ld, int k, int mode, float* scores,
                        int64_t* idx64, int32_t* idx32, int32_t* status, const DeviceInfo& dev, cudaStream_t st) {
  // cluster size: a share must fit 32 keys per thread; beyond that split rows until the grid covers the SMs
  const int chunks = (N + 31) / 32;
  int C = 1;
  while (C < 8 && ((chunks + C - 1) / C * 32 > RMAX_SLICE || (M * C < dev.sm_count && N / (2 * C) >= 2048))) C <<= 1;
  const int slice = (chunks + C - 1) / C * 32;
  if (slice > RMAX_SLICE) return fail(MOE_ERR_UNSUPPORTED, "topk_softmax: N=%d exceeds %d", N, 8 * RMAX_SLICE);
  int kpad = next_pow2(k);
  if (kpad < 2) kpad = 2;
  if (kpad > RMAX_KPAD) return fail(MOE_ERR_UNSUPPORTED, "topk_softmax: k=%d exceeds %d", k, RMAX_KPAD);
  // Entries a row may hand to the sort.  One CTA: what a sort of k entries (or of RT) takes anyway.  More CTAs: three
  // quarters of the length their shares of k, with a quarter on top, round up to.
  int totcap = kpad > RT ? kpad : RT;
  if (C > 1) {
    const int share = 3 * C * next_pow2((k + k / 4) / C + 1) / 4;
    if (share > totcap) totcap = share;
    if (totcap > RMAX_KPAD) totcap = RMAX_KPAD;
  }
  const int lcap = next_pow2(totcap);
  const size_t smem = (size_t)RCTRL_BYTES + 2 * RBINS * 4 + 2 * RCHUNKS * 4 + (size_t)lcap * 8 + (C > 1 ? (size_t)totcap * 8 : 0);
  const int vec_ok = (N % 4 == 0) && (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(logits) & 15) == 0);
  auto kernel = slice <= 8 * RT ? topk_radix_kernel<8> : (slice <= 16 * RT ? topk_radix_kernel<16> : topk_radix_kernel<32>);
  MOE_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(M * C), 1, 1);
  cfg.blockDim = dim3(RT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MOE_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, logits, M, N, ld, k, totcap, lcap, mode, vec_ok, scores,
                                    idx64, idx32, status));
  return MOE_OK;
}

}  // namespace moe

extern "C" int moe_topk_softmax(const float* logits, int64_t M, int64_t N, int64_t ld, int k, int mode, float* scores,
                                int64_t* indices, int32_t* indices32, int32_t* status, void* stream) {
  using namespace moe;
  if (!logits || !scores || (!indices && !indices32)) return fail(MOE_ERR_ARG, "topk_softmax: null pointer");
  if (M < 0 || N < 1 || k < 1 || k > N || ld < N) return fail(MOE_ERR_ARG, "topk_softmax: bad shape M=%lld N=%lld k=%d ld=%lld", (long long)M, (long long)N, k, (long long)ld);
  if (mode < 0 || mode > 2) return fail(MOE_ERR_ARG, "topk_softmax: unknown mode %d", mode);
  if (N > 8 * (int64_t)RMAX_SLICE) return fail(MOE_ERR_UNSUPPORTED, "topk_softmax: N=%lld exceeds %d", (long long)N, 8 * RMAX_SLICE);
  if (M * 8 > 0x7FFFFFFFll) return fail(MOE_ERR_UNSUPPORTED, "topk_softmax: M too large");
  if (M == 0) return MOE_OK;
  DeviceInfo dev;
  int rc = current_device_info(&dev);
  if (rc) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int n = (int)N;
  const bool vec_rows = (n % 4 == 0) && (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(logits) & 15) == 0);
  // Measured (us): 320 rows of 128, k = 6: a warp per row 2.5, lane groups 3.5; of 256, k = 8: 3.2, 3.3; of 512: 4.0, 3.3;
  // of 1024: 5.8, 3.4.  2048 rows of 16: a lane per row 2.5, lane groups 2.5; 8192: 2.6, 2.6; 32768: 2.9, 3.8; rows of 64
  // (a lane per row is built for 32 at most): 32768 4.3, 4.5.
  // k = 7, 8 of 65 to 128: four lanes have 16 parts, of which the 8th leaves some rows with more than 16 entries; eight lanes
  // have 32 (2048 rows 3.1 against 6.3, 32768 9.2 against 13.0, 131072 27.5 against 28.9, 1048576 190 against 178).
  if (n <= 1024 && k <= 8 && n >= 8 && vec_rows && (M >= 2048 || n > 256)) {
    if (n <= LANE_NMAX) {
#define MOE_LANE_CASE(K_) return launch_lane<K_>(logits, M, n, ld, k, mode, scores, indices, indices32, dev.sm_count, st)
      if (k <= 2) MOE_LANE_CASE(2);
      if (k <= 4) MOE_LANE_CASE(4);
      if (k <= 6) MOE_LANE_CASE(6);
      MOE_LANE_CASE(8);
#undef MOE_LANE_CASE
    }
#define MOE_GROUP_CASE(K_, L_, E_) return launch_group<K_, L_, E_>(logits, M, n, ld, k, mode, scores, indices, indices32, st)
#define MOE_GROUP_K(K_)                          \
  {                                              \
    if (n <= 64) MOE_GROUP_CASE(K_, 4, 16);      \
    if (n <= 128 && K_ == 8 && M <= 262144) MOE_GROUP_CASE(K_, 8, 16); \
    if (n <= 128) MOE_GROUP_CASE(K_, 4, 32);     \
    if (n <= 256) MOE_GROUP_CASE(K_, 8, 32);     \
    if (n <= 512) MOE_GROUP_CASE(K_, 16, 32);    \
    MOE_GROUP_CASE(K_, 32, 32);                  \
  }
    if (k <= 2) MOE_GROUP_K(2)
    if (k <= 4) MOE_GROUP_K(4)
    if (k <= 6) MOE_GROUP_K(6)
    MOE_GROUP_K(8)
#undef MOE_GROUP_K
#undef MOE_GROUP_CASE
  }
  if (n <= 1024 && k <= 64) {
    const bool vec = vec_rows;
#define MOE_WARP_CASE(E_, V_) return launch_warp<E_, V_>(logits, M, n, ld, k, mode, scores, indices, indices32, dev.sm_count, st)
    if (n <= 32) MOE_WARP_CASE(1, 1);
    if (n <= 64) MOE_WARP_CASE(2, 1);
    if (n <= 128) { if (vec) MOE_WARP_CASE(4, 4); MOE_WARP_CASE(4, 1); }
    if (n <= 256) { if (vec) MOE_WARP_CASE(8, 4); MOE_WARP_CASE(8, 1); }
    if (n <= 512) { if (vec) MOE_WARP_CASE(16, 4); MOE_WARP_CASE(16, 1); }
    if (vec) MOE_WARP_CASE(32, 4);
    MOE_WARP_CASE(32, 1);
#undef MOE_WARP_CASE
  }
  return launch_radix(logits, M, n, ld, k, mode, scores, indices, indices32, status, dev, st);
}
