// KV splits of decode attention for a step whose rows are several requests', by their lengths.
//
// A count that looks at the number of rows alone gives one long context among short ones as few CTAs as each of those, and rows of one
// request, which one CTA serves, as many as if each had its own.  16 layers, 8 KV heads, that rule / this one: step of 7
// requests at 300 positions and one at 30000 2.82 / 2.05 ms, 63 at 100 and one at 60000 14.5 / 4.89, 60 rows of one request at 1000
// and four requests at 4000 4.83 / 4.51, 64 requests at 150 to 300 4.36 / 4.24.
//
// The longest group of rows gets k splits, the others as many as make their pieces no longer.  Of all k the one is taken that
// makes the estimated time least: the longest piece, or the waves of CTAs (two on each of 148 SMs) times the mean piece, where a CTA's
// start, first copies and partials cost about as much as kFixedPages.  It ranks what was measured: 24 requests at 1000 to 2000
// positions with 1, 2, 3, 4 splits each 57, 51, 46, 51 us, 8 at 2000 to 4000 with 1, 2, 4, 8, 10 73, 42, 39, 41, 47.
// One CTA of at least 64 threads, thread i standing for row i and for k = i + 1.  As a launch of its own of 1024 threads, which tried all k at
// once, it took 8 us of every step; as one more CTA of the embedding's launch it adds 1 (2 to 8 rows) to 4 (40 rows).
#pragma once
#include "common.cuh"

namespace b2 {

struct AttnPlanParams {
  const int* ctrl;
  int M, rmax, n_kv, nsplit, entries, window;
  int* plan;       // [64] splits of every row, [entries] first row | split << 8 | splits << 16 of a CTA column, -1: none
};

constexpr int kPlanFixedPages = 8, kPlanSlots = 296;

struct AttnPlanShared {      // the caller's: beside an embedding it takes the place of a row's values, whose width may need all there is
  int req[64], pos[64], pages[64], n[64], piece[64];
  unsigned best[2], start[2];
  int top[2], sum[2];
};

__device__ __forceinline__ void attn_plan(const AttnPlanParams& p, AttnPlanShared& sh) {
  constexpr int kReq = 16, kPos = 80;      // words of the control block
  auto &s_req = sh.req, &s_pos = sh.pos, &s_pages = sh.pages, &s_n = sh.n, &s_piece = sh.piece;
  auto &s_best = sh.best, &s_start = sh.start;
  auto &s_top = sh.top, &s_sum = sh.sum;
  const int i = threadIdx.x;
  if (i < 64) {
    s_req[i] = i < p.M ? __ldcg(p.ctrl + kReq + i) : -1;
    s_pos[i] = i < p.M ? __ldcg(p.ctrl + kPos + i) : 0;
  }
  for (int e = i; e < p.entries; e += blockDim.x) p.plan[64 + e] = -1;
  __syncthreads();
  if (i >= 64) return;
  const auto sync = [] { asm volatile("bar.sync 1, 64;" ::: "memory"); };
  // groups: up to rmax consecutive rows of a request, led by the first
  int pages = 0, rows = 0;
  const unsigned start = __ballot_sync(0xffffffffu, i == 0 || s_req[i] != s_req[i - 1]);
  if ((i & 31) == 0) s_start[i >> 5] = start;
  sync();
  if (i < p.M) {
    const int first = 63 - __clzll((s_start[0] | (unsigned long long)s_start[1] << 32) & (~0ull >> (63 - i)));
    if ((i - first) % p.rmax == 0) {
      int ctx = 0;
      for (; rows < p.rmax && i + rows < p.M && s_req[i + rows] == s_req[i]; ++rows) ctx = max(ctx, s_pos[i + rows] + 1);
      pages = max(1, ((ctx + 15) >> 4) - (p.window > 0 ? max(0, s_pos[i] + 1 - p.window) >> 4 : 0));
    }
  }
  s_pages[i] = pages;
  const int top = __reduce_max_sync(0xffffffffu, pages), sum = __reduce_add_sync(0xffffffffu, pages);
  if ((i & 31) == 0) s_top[i >> 5] = top, s_sum[i >> 5] = sum;
  sync();
  const int longest = max(s_top[0], s_top[1]), total = s_sum[0] + s_sum[1];
  const auto ceil_div = [](int a, int b) { return (a + b - 1) / b; };
  unsigned best = ~0u;
  if (i < min(p.nsplit, longest)) {
    const int span = ceil_div(longest, i + 1);
    const float inv = 1.f / (float)span;
    int n = 0;
    for (int j0 = 0; j0 < p.M; j0 += 8)
#pragma unroll
      for (int j = j0; j < j0 + 8; ++j) {   // ceil(pages / span): a quotient that is off by one at most, put right
        const int a = s_pages[j], q = (int)((float)a * inv), r = a - q * span;
        n += q + (r > 0) + (r > span);
      }
    if (n <= p.entries) best = (unsigned)max(kPlanFixedPages + span, ceil_div(n * p.n_kv, kPlanSlots) * (kPlanFixedPages + ceil_div(total, n))) << 7 | (i + 1);
  }
  best = __reduce_min_sync(0xffffffffu, best);
  if ((i & 31) == 0) s_best[i >> 5] = best;
  sync();
  const int span = ceil_div(longest, (int)(min(s_best[0], s_best[1]) & 127u)), n = ceil_div(pages, span);
  const int piece = n ? ceil_div(pages, n) : 0;
  s_n[i] = n;
  s_piece[i] = piece;
  sync();
  for (int r = 0; r < rows; ++r) p.plan[i + r] = n;
  int at = 0;                               // longest pieces first
  for (int j0 = 0; j0 < p.M; j0 += 8)
#pragma unroll
    for (int j = j0; j < j0 + 8; ++j) at += s_piece[j] > piece || (s_piece[j] == piece && j < i) ? s_n[j] : 0;
  for (int s = 0; s < n; ++s) p.plan[64 + at + s] = i | s << 8 | n << 16;
}

inline bool attn_plan_params(AttnPlanParams& p, const int* ctrl, int M, int n_q, int n_kv, int nsplit, int window, int* plan, int entries) {
  if (M < 1 || M > 64 || n_kv < 1 || n_q % n_kv != 0 || n_q / n_kv > 16 || nsplit < 1 || nsplit > 64 || entries < M || entries > 65535 || !plan) return false;
  const int gqa = n_q / n_kv;
  p = {ctrl, M, 64 / gqa < 8 ? 64 / gqa : 8, n_kv, nsplit, entries, window > 0 ? window : 0, plan};
  return true;
}

}  // namespace b2
