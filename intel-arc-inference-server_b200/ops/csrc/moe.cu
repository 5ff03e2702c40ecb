// Mixture-of-experts glue kernels: routing, expert-major sorting with a device-side block table,
// gather, and the weighted combine.
//
//   moe_route     scores of all experts (softmax or sigmoid) -> optional choice of expert groups -> top-k (ties to the
//                 lower id) -> weights (renormalised over the chosen, or the scores)
//   moe_count     per-expert histogram + the rank of every (token, slot) inside its expert
//   moe_plan      prefix over experts padded to 128-row blocks -> block table for the grouped GEMM
//   moe_scatter   (token, slot) -> sorted row; gather of the activation rows in sorted order
//   moe_combine   out = resid + sum_slot w * y[row(token, slot)] + sigmoid(gate) * shared   (fixed slot order)
//
// Same division of labour as the reference's pf_moe_sort_mw.cl / pf_moe.cl / moe.cl (moe_route):
// the host never reads a count; the tile table is padded and the grouped GEMM reads the block
// count on the device.  The rank inside an expert comes from an atomic counter, so the ORDER of
// rows inside an expert varies from run to run, but every row is computed independently of its
// neighbours and the combine adds a token's slots in slot order, so the output bits do not.
#include "common.cuh"

using namespace b2;

namespace {

// ---------------------------------------------------------------- route: one warp per token
// How logits become a choice of experts and their weights.
struct RouteRule {
  int sigmoid;   // 0: softmax over all experts, 1: a sigmoid per expert
  int groups;    // > 1: experts form this many equal groups of neighbours; only the `keep` groups with the largest sums
  int keep;      //      of their two best scores stay eligible
  int renorm;    // 1: weights divided by their sum over the chosen experts, 0: the scores themselves
};

// logits fp32 [T][ld], the first E columns are the experts (E <= 512).  topk_idx int32 [T][k], topk_w fp32 [T][k].
// One row's routing by a whole warp: scores of E logits, top-k by repeated arg-max (ties to the lower id).
// `stride` >= k entries per row in topk_idx / topk_w.  PLAIN: the rule is softmax, no groups, renormalised (the code of the
// other rules costs the decode step's router 1.5 us a layer when it is compiled in).
template <bool PLAIN>
__device__ __forceinline__ void route_row(const float* __restrict__ lrow, int E, int k, const RouteRule rule,
                                          int* __restrict__ idx_out, float* __restrict__ w_out, int lane) {
  constexpr int PER = 16;  // experts per lane (E <= 512)
  float v[PER];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    v[i] = e < E ? __ldcg(lrow + e) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
  mx = warp_max(mx);
  float total = 0.f;   // softmax normaliser, only needed when the weights are not renormalised
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    if (!PLAIN && 32 * i >= E) { v[i] = -1.f; continue; }
    // softmax: unnormalised probabilities; -1 marks "taken / absent", -1/2 a score that is NaN: it is taken after all others (a
    // row's ids index weights and tables, so they are E's whatever the logits) and makes the row's weights NaN
    const bool in = (lane + 32 * i) < E;
    if (!PLAIN && rule.sigmoid) v[i] = in ? 1.f / (1.f + expf(-v[i])) : -1.f;
    else v[i] = in ? __expf(v[i] - mx) : -1.f;
    if (!PLAIN) total += in ? v[i] : 0.f;
    v[i] = fmaxf(v[i], in ? -0.5f : -1.f);
  }
  if (!PLAIN && rule.groups > 1) {
    const int size = E / rule.groups;
    float mine = -INFINITY;      // lane g keeps the score of group g (groups <= 32)
    for (int g = 0; g < rule.groups; ++g) {
      float a = -1.f, b = -1.f;  // two best of the group among this lane's experts
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        if (32 * i >= E) break;
        const int e = lane + 32 * i;
        if (e >= g * size && e < (g + 1) * size) {
          if (v[i] > a) { b = a; a = v[i]; }
          else b = fmaxf(b, v[i]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, a, o), ob = __shfl_xor_sync(0xffffffffu, b, o);
        b = fmaxf(fminf(a, oa), fmaxf(b, ob));
        a = fmaxf(a, oa);
      }
      const float score = a + fmaxf(b, 0.f);    // a group of one expert has no second score
      if (lane == g) mine = score;
    }
    unsigned kept = 0;
    for (int r = 0; r < rule.keep; ++r) {
      float bv = (kept >> lane) & 1u ? -INFINITY : mine;
      int bi = lane;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      kept |= 1u << bi;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (32 * i >= E) break;
      const int e = lane + 32 * i;
      if (e < E && !((kept >> (e / size)) & 1u)) v[i] = -1.f;
    }
  }
  float wsum = 0.f;
  float myw = 0.f;
  int myid = 0;
  for (int r = 0; r < k; ++r) {
    // arg-max over the remaining experts; ties resolve to the lower id
    float bv = -1.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (!PLAIN && 32 * i >= E) break;
      const int e = lane + 32 * i;
      if (v[i] > bv) { bv = v[i]; bi = e; }  // e ascends with i inside a lane: the first maximum is the lowest id
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((bi & 31) == lane) v[bi >> 5] = -1.f;
    if (bv < 0.f) bv = __int_as_float(0x7fc00000);
    wsum += bv;
    if (lane == r) { myw = bv; myid = bi; }
  }
  float norm = wsum;                                // renormalised: the softmax normaliser cancels
  if (!PLAIN && !rule.renorm) norm = rule.sigmoid ? 1.f : warp_sum(total);
  if (lane < k) {
    idx_out[lane] = myid;
    w_out[lane] = myw / norm;
  }
}

template <bool PLAIN>
__global__ void __launch_bounds__(256) moe_route_kernel(const float* __restrict__ logits, int ld, int T, int E, int k,
                                                        const RouteRule rule, int* __restrict__ topk_idx,
                                                        float* __restrict__ topk_w, int shared) {
  pdl_wait();
  pdl_launch_dependents();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T) return;
  const size_t at = (size_t)warp * (k + shared);
  route_row<PLAIN>(logits + (size_t)warp * ld, E, k, rule, topk_idx + at, topk_w + at, lane);
  for (int i = lane; i < shared; i += 32) {
    topk_idx[at + k + i] = E + i;
    topk_w[at + k + i] = 1.f;
  }
}

// ---------------------------------------------------------------- decode rows: router logits + routing in one launch
// logits[m][r] = x[m] . W[r] for the R router rows (E experts, then the shared expert's gate row when there is one):
// sixteen router rows a CTA, eight token rows per pass over the weights, on mma.sync, k spread over the warps (fp32 products of a
// warp per router row were bound by issue: 257 x 2048, the launch for 1 / 8 / 48 rows 6.2 / 10.6 / 13.3 us, now 6.9 / 7.9 / 8.0).  The CTA that finishes last (a ticket) then
// routes every token row.  With `shared_slot` each row gets one more slot: expert id E (the shared expert, see the
// batched GEMV's alt weights) with weight sigmoid(gate logit), or 1 without a gate row; with shared_slot n > 1 (no gate
// row) n more slots, ids E .. E + n - 1 with weight 1: runs of a shared expert's hidden columns.
struct RouterRowsParams {
  const __nv_bfloat16* w;   // [R][H]
  const __nv_bfloat16* x;   // [M][H]
  float* logits;            // [M][ld]
  int M, R, H, ld, E, k;
  int shared_slot, has_gate;
  RouteRule rule;
  int* topk_idx;            // [M][k + shared_slot]
  float* topk_w;
  int* ticket;              // zeroed words, left zero: one, or (gridDim.y > 1) one per slice of token rows and one for all
  int* groups;              // table of (row, slot) pairs by expert (gemv_w4.cu: ExpertGroups), or nullptr
};

// The pairs of M rows x `stride` slots, ordered by expert, in groups of up to eight of one expert.  256 threads; the order of the
// pairs inside an expert comes from an atomic counter (a pair's result does not depend on its neighbours).
constexpr int kGroupIds = 544;      // expert ids: 512 routed and up to 32 runs of a shared expert
__device__ void group_pairs(const int* topk_idx, int pairs, int* groups, int* s_count, int* s_first) {
  const int tid = threadIdx.x;
  for (int i = tid; i < kGroupIds; i += 256) s_count[i] = 0;
  __syncthreads();
  for (int i = tid; i < pairs; i += 256) atomicAdd(&s_count[__ldcg(topk_idx + i)], 1);
  __syncthreads();
  // groups before an expert's: three experts a thread, prefixes over the warp, the warps in turn
  __shared__ int s_warp[8];
  int n[3], mine = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    n[i] = 3 * tid + i < kGroupIds ? (s_count[3 * tid + i] + 7) >> 3 : 0;
    mine += n[i];
  }
  int x = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, x, o);
    if ((tid & 31) >= o) x += v;
  }
  if ((tid & 31) == 31) s_warp[tid >> 5] = x;
  __syncthreads();
  int first = x - mine;
  for (int i = 0; i < (tid >> 5); ++i) first += s_warp[i];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (3 * tid + i < kGroupIds) s_first[3 * tid + i] = first;
    first += n[i];
  }
  if (tid == 255) groups[0] = first;
  __syncthreads();
  for (int e = tid; e < kGroupIds; e += 256) {
    const int c = s_count[e];
    for (int j = 0; 8 * j < c; ++j) {
      groups[16 + (s_first[e] + j) * 10] = e;
      groups[16 + (s_first[e] + j) * 10 + 1] = min(8, c - 8 * j);
    }
  }
  __syncthreads();
  for (int i = tid; i < kGroupIds; i += 256) s_count[i] = 0;
  __syncthreads();
  for (int i = tid; i < pairs; i += 256) {
    const int e = __ldcg(topk_idx + i), r = atomicAdd(&s_count[e], 1);
    groups[16 + (s_first[e] + (r >> 3)) * 10 + 2 + (r & 7)] = i;
  }
}

// Groups of eight router rows a CTA.  With one the launch alone is faster up to 16 rows (8 rows 7.3 us where it is 7.9), but its 33 CTAs are in the way of the experts' CTAs
// that start behind it: 4 requests, 16 layers 1165 us where it is 1090.
constexpr int kRouterTiles = 2;

template <bool PLAIN>
__global__ void __launch_bounds__(256) moe_router_rows_kernel(const RouterRowsParams p) {
  __shared__ int s_last, s_count[kGroupIds], s_first[kGroupIds];
  pdl_wait();
  pdl_launch_dependents();
  constexpr int RT = kRouterTiles, RR = 8 * RT;      // router rows of the CTA
  __shared__ float s_red[8][8][RR + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = blockIdx.x * RR;
  // token rows of this CTA: all of them, or the slice of eight that blockIdx.y names
  const int m_lo = gridDim.y > 1 ? blockIdx.y * 8 : 0, m_hi = gridDim.y > 1 ? min(p.M, m_lo + 8) : p.M;
  for (int m0 = m_lo; m0 < m_hi; m0 += 8) {
    // A lane's 16 bytes of a row are eight k of a 32-k chunk: two MMAs take them as they are, since both operands have them in the same order.
    // Chunks go round the warps; eight of a warp's are in flight together.  Token rows are the MMA's rows (the upper eight are zero).  A tensor core cuts off
    // where it adds, so every MMA starts from zero and their results are added as a tree in fp32: errors of 7.5e-8 of the logits at 2048, as fp32 FMAs made (one chain
    // of MMAs a warp: 2.4e-7, and 4.7e-7 at 4096).
    float c[RT][2] = {};
    const auto piece = [&](const __nv_bfloat16* base, int row, int rows, int k) {
      return row < rows && k < p.H ? __ldg(reinterpret_cast<const uint4*>(base + (size_t)row * p.H + k)) : make_uint4(0, 0, 0, 0);
    };
    for (int k0 = warp * 32 + t * 8; k0 - t * 8 < p.H; k0 += 8 * 8 * 32) {
      uint4 w[RT][8], x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = k0 + i * 8 * 32;
#pragma unroll
        for (int r = 0; r < RT; ++r) w[r][i] = piece(p.w, r0 + 8 * r + g, p.R, k);
        x[i] = piece(p.x, m0 + g, m_hi, k);
      }
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        float d[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
          mma_bf16_16816(lo, x[i].x, 0u, x[i].y, 0u, w[r][i].x, w[r][i].y);
          mma_bf16_16816(hi, x[i].z, 0u, x[i].w, 0u, w[r][i].z, w[r][i].w);
          d[i][0] = lo[0] + hi[0];
          d[i][1] = lo[1] + hi[1];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) c[r][j] += ((d[0][j] + d[1][j]) + (d[2][j] + d[3][j])) + ((d[4][j] + d[5][j]) + (d[6][j] + d[7][j]));
      }
    }
    if (m0 > m_lo) __syncthreads();
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      s_red[warp][g][8 * r + 2 * t] = c[r][0];
      s_red[warp][g][8 * r + 2 * t + 1] = c[r][1];
    }
    __syncthreads();
    const int row = threadIdx.x % RR, m = m0 + threadIdx.x / RR;
    if (threadIdx.x < 8 * RR && r0 + row < p.R && m < m_hi) {
      float w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = s_red[i][threadIdx.x / RR][row];
      p.logits[(size_t)m * p.ld + r0 + row] = ((w[0] + w[1]) + (w[2] + w[3])) + ((w[4] + w[5]) + (w[6] + w[7]));
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int t = atomicAdd(p.ticket + blockIdx.y, 1);
    s_last = t == (int)gridDim.x - 1;
    if (s_last) p.ticket[blockIdx.y] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int stride = p.k + p.shared_slot;
  for (int m = m_lo + warp; m < m_hi; m += 8) {
    const float* lrow = p.logits + (size_t)m * p.ld;
    route_row<PLAIN>(lrow, p.E, p.k, p.rule, p.topk_idx + (size_t)m * stride, p.topk_w + (size_t)m * stride, lane);
    for (int i = lane; i < p.shared_slot; i += 32) {
      p.topk_idx[(size_t)m * stride + p.k + i] = p.E + i;
      p.topk_w[(size_t)m * stride + p.k + i] = p.has_gate ? 1.f / (1.f + __expf(-__ldcg(lrow + p.E))) : 1.f;
    }
  }
  if (!p.groups) return;
  // every slice has routed its rows: the CTA that sees that last makes the table
  __threadfence();
  __syncthreads();
  if (gridDim.y > 1) {
    if (threadIdx.x == 0) {
      const int t = atomicAdd(p.ticket + gridDim.y, 1);
      s_last = t == (int)gridDim.y - 1;
      if (s_last) p.ticket[gridDim.y] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
  }
  group_pairs(p.topk_idx, p.M * stride, p.groups, s_count, s_first);
}

// ---------------------------------------------------------------- count + rank
__global__ void moe_count_kernel(const int* __restrict__ topk_idx, int n, int* __restrict__ counts,
                                 int* __restrict__ rank) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) rank[i] = atomicAdd(&counts[topk_idx[i]], 1);
}

// ---------------------------------------------------------------- plan: one CTA, E <= 1024
// expert_base[e] = first sorted row of expert e (a multiple of 128); block table of 128-row blocks.
__global__ void __launch_bounds__(1024) moe_plan_kernel(const int* __restrict__ counts, int E, int max_blk,
                                                        int* __restrict__ expert_base, int* __restrict__ blk_expert,
                                                        int* __restrict__ blk_row0, int* __restrict__ blk_rows,
                                                        int* __restrict__ n_blk, int* __restrict__ total_rows) {
  __shared__ int s_blocks[1024];
  __shared__ int s_scan[1024];
  const int e = threadIdx.x;
  const int c = e < E ? counts[e] : 0;
  const int nb = (c + 127) >> 7;
  s_blocks[e] = nb;
  s_scan[e] = nb;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {  // inclusive scan (Hillis-Steele)
    const int v = e >= o ? s_scan[e - o] : 0;
    __syncthreads();
    s_scan[e] += v;
    __syncthreads();
  }
  const int first = s_scan[e] - nb;  // exclusive
  if (e < E) {
    expert_base[e] = first * 128;
    for (int j = 0; j < nb && first + j < max_blk; ++j) {
      blk_expert[first + j] = e;
      blk_row0[first + j] = (first + j) * 128;
      blk_rows[first + j] = min(128, c - j * 128);
    }
  }
  if (e == 1023) {
    *n_blk = min(s_scan[1023], max_blk);
    *total_rows = s_scan[1023] * 128;
  }
}

// ---------------------------------------------------------------- scatter + gather
// One CTA per token: writes the inverse map of its slots and copies its activation row to their sorted positions, each piece read
// once (a CTA per slot: 2048 rows of 2048, eight slots, 26 -> 14 us; the bytes take 11.5).
constexpr int kScatterSlots = 32;
__global__ void __launch_bounds__(256) moe_scatter_kernel(const int* __restrict__ topk_idx, const int* __restrict__ rank,
                                                          const int* __restrict__ expert_base, int k,
                                                          const __nv_bfloat16* __restrict__ x, int H,
                                                          int* __restrict__ row_of, __nv_bfloat16* __restrict__ xs) {
  __shared__ int s_pos[kScatterSlots];
  const int token = blockIdx.x;
  for (int s0 = 0; s0 < k; s0 += kScatterSlots) {
    const int ns = min(kScatterSlots, k - s0);
    if (s0) __syncthreads();
    if ((int)threadIdx.x < ns) {
      const int i = token * k + s0 + threadIdx.x;
      row_of[i] = s_pos[threadIdx.x] = expert_base[topk_idx[i]] + rank[i];
    }
    __syncthreads();
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)token * H);
    for (int j = threadIdx.x; j < H / 8; j += blockDim.x) {
      const uint4 v = src[j];
      for (int s = 0; s < ns; ++s) reinterpret_cast<uint4*>(xs + (size_t)s_pos[s] * H)[j] = v;
    }
  }
}

// ---------------------------------------------------------------- combine (prefill): one CTA per token
// out[token] = resid[token] + sum_slot w[slot] * y[row_of[token][slot]] + sigmoid(gate_logit[token]) * shared[token], added in that order.
// V: columns a thread takes at a time, 8 where rows begin on 16 bytes; up to eight slots' pieces are in flight together (one after another, two
// columns a thread: 2048 rows of 2048, eight slots, 46 -> 25 us; the bytes take 14).
template <int V>
__global__ void __launch_bounds__(256) moe_combine_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ row_of,
                                                          const float* __restrict__ topk_w, int k, int H,
                                                          const __nv_bfloat16* __restrict__ shared_y,
                                                          const float* __restrict__ gate_logit, int gate_ld,
                                                          const __nv_bfloat16* resid,
                                                          __nv_bfloat16* out) {
  constexpr int W = V / 2;       // words
  struct __align__(4 * W) Piece { uint32_t w[W]; };
  const auto at = [](const __nv_bfloat16* p, size_t row, int H, int j) { return *reinterpret_cast<const Piece*>(p + row * H + (size_t)j * V); };
  const int token = blockIdx.x;
  float g = 0.f;
  if (shared_y) g = gate_logit ? 1.f / (1.f + __expf(-gate_logit[(size_t)token * gate_ld])) : 1.f;
  for (int j = threadIdx.x; j < H / V; j += blockDim.x) {
    float acc[V];
    const auto add = [&](float w, const Piece& v) {
#pragma unroll
      for (int i = 0; i < W; ++i) {
        acc[2 * i] = fmaf(w, bf16_lo(v.w[i]), acc[2 * i]);
        acc[2 * i + 1] = fmaf(w, bf16_hi(v.w[i]), acc[2 * i + 1]);
      }
    };
    const Piece r = at(resid, token, H, j);
    Piece sh = {};
    if (shared_y) sh = at(shared_y, token, H, j);
#pragma unroll
    for (int i = 0; i < W; ++i) { acc[2 * i] = bf16_lo(r.w[i]); acc[2 * i + 1] = bf16_hi(r.w[i]); }
    for (int s0 = 0; s0 < k; s0 += 8) {
      Piece v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s0 + u < k) v[u] = at(y, row_of[token * k + s0 + u], H, j);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s0 + u < k) add(topk_w[token * k + s0 + u], v[u]);
    }
    if (shared_y) add(g, sh);
    Piece o;
#pragma unroll
    for (int i = 0; i < W; ++i) o.w[i] = pack_bf16(acc[2 * i], acc[2 * i + 1]);
    *reinterpret_cast<Piece*>(out + (size_t)token * H + (size_t)j * V) = o;
  }
}

// ---------------------------------------------------------------- combine (decode rows): a thread per (row, column)
// Folds the split-K slices of the batched expert GEMVs: part is [batch = M * k (+ M shared)][S][H] fp32,
// written as out[0][m][H] fp32 (one slice) for the next residual fold.  Grid (M, H / 256): a thread's k * S loads
// are independent, so the kernel is one memory latency long (one CTA per row looping over the columns took 75 us
// for a 2048-wide row).
__global__ void __launch_bounds__(256) moe_combine_rows_kernel(const float* __restrict__ part, int S, int M, int k, int H,
                                                               const float* __restrict__ topk_w,
                                                               const float* __restrict__ shared_part, int S_sh,
                                                               const float* __restrict__ gate_logit, int gate_ld,
                                                               float* __restrict__ out, __nv_bfloat16* fold_resid,
                                                               float* __restrict__ fold_ssq) {
  __shared__ float s_ss[8];
  pdl_wait();
  pdl_launch_dependents();
  const int m = blockIdx.x;
  float g = 0.f;
  if (shared_part) g = gate_logit ? 1.f / (1.f + __expf(-gate_logit[(size_t)m * gate_ld])) : 1.f;
  const int j = blockIdx.y * blockDim.x + threadIdx.x;
  float acc = 0.f;
  if (j < H) {
    // every load of the row's slots goes out before the first is used (up to 12 slots x 4 slices a pass)
    for (int s0 = 0; s0 < k; s0 += 12) {
      float v[12][4], w[12];
#pragma unroll
      for (int u = 0; u < 12; ++u) {
        const int s = s0 + u;
        w[u] = s < k ? topk_w[m * k + s] : 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          v[u][q] = (s < k && q < S) ? part[((size_t)(m * k + s) * S + q) * H + j] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 12; ++u) {
        float t = v[u][0];
#pragma unroll
        for (int q = 1; q < 4; ++q) t += v[u][q];      // slices in order; absent ones add 0
        acc = fmaf(w[u], t, acc);
      }
    }
    if (S > 4) {   // more slices than a pass holds: the rest, slot by slot
      for (int s = 0; s < k; ++s) {
        float t = 0.f;
        for (int q = 4; q < S; ++q) t += part[((size_t)(m * k + s) * S + q) * H + j];
        acc = fmaf(topk_w[m * k + s], t, acc);
      }
    }
    if (shared_part) {
      const float* p = shared_part + (size_t)m * H + j;  // shared expert: [S_sh][M][H]
      float v = 0.f;
      for (int q = 0; q < S_sh; ++q) v += p[(size_t)q * M * H];
      acc = fmaf(g, v, acc);
    }
  }
  if (!fold_resid) {
    if (j < H) out[(size_t)m * H + j] = acc;
    return;
  }
  // Fold form: the row's residual stream takes the sum in place (bf16) and every 128-column block's sum of squares
  // of the ROUNDED values is left for the next layer's fused RMSNorm -- the arithmetic and the order of the four
  // 32-column partial sums are those of the GEMV's fold epilogue.
  float rf = 0.f;
  if (j < H) {
    const __nv_bfloat16 rb = __float2bfloat16(__bfloat162float(fold_resid[(size_t)m * H + j]) + acc);
    fold_resid[(size_t)m * H + j] = rb;
    rf = __bfloat162float(rb);
  }
  const float ss = warp_sum(rf * rf);
  if ((threadIdx.x & 31) == 0) s_ss[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x < 2) {
    const int nb = blockIdx.y * 2 + threadIdx.x;
    if (nb * 128 < H) {
      const float* q = s_ss + 4 * threadIdx.x;
      fold_ssq[(size_t)m * ((H + 127) / 128) + nb] = ((q[0] + q[1]) + q[2]) + q[3];
    }
  }
}

}  // namespace

static bool route_plain(const RouteRule& r) { return !r.sigmoid && r.groups <= 1 && r.renorm; }

static bool route_ok(int E, int k, const RouteRule& r) {
  if (E < 1 || E > 512 || k > 32 || k < 1) return false;
  if (r.groups <= 1) return k <= E;
  return r.groups <= 32 && E % r.groups == 0 && r.keep >= 1 && r.keep <= r.groups && k <= r.keep * (E / r.groups);
}

// shared: more slots per row, ids E .. with weight 1
extern "C" int b2_moe_route(const float* logits, int ld, int T, int E, int k, int sigmoid, int groups, int keep, int renorm,
                            int* topk_idx, float* topk_w, int shared, void* stream) {
  const RouteRule rule{sigmoid, groups, keep, renorm};
  if (!route_ok(E, k, rule) || shared < 0) return -1;
  const int blocks = (T * 32 + 255) / 256;
  return b2_launch(route_plain(rule) ? moe_route_kernel<true> : moe_route_kernel<false>, dim3(blocks), dim3(256), 0, (cudaStream_t)stream, true, logits, ld, T, E, k,
                   rule, topk_idx, topk_w, shared);
}

extern "C" int b2_moe_router_rows(const void* w, const void* x, float* logits, int M, int R, int H, int ld, int E, int k,
                                  int shared_slot, int has_gate, int sigmoid, int groups, int keep, int renorm,
                                  int* topk_idx, float* topk_w, int* ticket, int n_tickets, int* table, void* stream) {
  const RouteRule rule{sigmoid, groups, keep, renorm};
  if (!route_ok(E, k, rule) || H % 8 || M < 1 || R < E + (has_gate ? 1 : 0) || ld < R || shared_slot < 0 || (has_gate && shared_slot > 1))
    return -1;
  RouterRowsParams p{(const __nv_bfloat16*)w, (const __nv_bfloat16*)x, logits, M, R, H, ld, E, k, shared_slot, has_gate,
                     rule, topk_idx, topk_w, ticket, table};
  if (table && E + shared_slot > kGroupIds) return -1;
  // Slices of eight token rows have CTAs of their own, which also route them (a router of 257 rows is 17 CTAs: 48 token rows
  // behind one another took 58 us of a layer's step).  Callers with a single ticket word keep one slice.
  const int slices = (M + 7) / 8 < n_tickets ? (M + 7) / 8 : 1;
  return b2_launch(route_plain(rule) ? moe_router_rows_kernel<true> : moe_router_rows_kernel<false>, dim3((R + 8 * kRouterTiles - 1) / (8 * kRouterTiles), slices), dim3(256), 0,
                   (cudaStream_t)stream, true, p);
}

// counts must hold E zeros on entry (the caller clears it on the stream).
extern "C" int b2_moe_sort(const int* topk_idx, int T, int k, int E, int max_blk, int* counts, int* rank,
                           int* expert_base, int* blk_expert, int* blk_row0, int* blk_rows, int* n_blk,
                           int* total_rows, void* stream) {
  if (E > 1024) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  const int n = T * k;
  moe_count_kernel<<<(n + 255) / 256, 256, 0, st>>>(topk_idx, n, counts, rank);
  moe_plan_kernel<<<1, 1024, 0, st>>>(counts, E, max_blk, expert_base, blk_expert, blk_row0, blk_rows, n_blk, total_rows);
  return (int)cudaGetLastError();
}

// histogram + rank only (the expert-parallel plan needs every rank's counts before it can lay rows out)
extern "C" int b2_moe_count(const int* topk_idx, int n, int* counts, int* rank, void* stream) {
  moe_count_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(topk_idx, n, counts, rank);
  return (int)cudaGetLastError();
}

extern "C" int b2_moe_scatter(const int* topk_idx, const int* rank, const int* expert_base, int T, int k, const void* x,
                              int H, int* row_of, void* xs, void* stream) {
  if (H % 8) return -1;
  moe_scatter_kernel<<<T, 256, 0, (cudaStream_t)stream>>>(topk_idx, rank, expert_base, k, (const __nv_bfloat16*)x, H,
                                                                row_of, (__nv_bfloat16*)xs);
  return (int)cudaGetLastError();
}

extern "C" int b2_moe_combine(const void* y, const int* row_of, const float* topk_w, int T, int k, int H,
                              const void* shared_y, const float* gate_logit, int gate_ld, const void* resid, void* out,
                              void* stream) {
  if (H % 2) return -1;
  const bool wide = H % 8 == 0 && (((uintptr_t)y | (uintptr_t)shared_y | (uintptr_t)resid | (uintptr_t)out) & 15) == 0;
  const auto kernel = wide ? moe_combine_kernel<8> : moe_combine_kernel<2>;
  kernel<<<T, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)y, row_of, topk_w, k, H,
                                                           (const __nv_bfloat16*)shared_y, gate_logit, gate_ld,
                                                           (const __nv_bfloat16*)resid, (__nv_bfloat16*)out);
  return (int)cudaGetLastError();
}

extern "C" int b2_moe_combine_rows(const float* part, int S, int M, int k, int H, const float* topk_w,
                                   const float* shared_part, int S_sh, const float* gate_logit, int gate_ld, float* out,
                                   void* fold_resid, float* fold_ssq, void* stream) {
  if (fold_resid && (!fold_ssq || H % 128)) return -1;
  return b2_launch(moe_combine_rows_kernel, dim3(M, (H + 255) / 256), dim3(256), 0, (cudaStream_t)stream, true, part, S, M,
                   k, H, topk_w, shared_part, S_sh, gate_logit, gate_ld, out, (__nv_bfloat16*)fold_resid, fold_ssq);
}

B2_DEFINE_STATUS(moe)
