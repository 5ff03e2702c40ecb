// W4A16 linears of decode steps with several rows (9 to 64) on tcgen05: weights in tensor memory, activations in shared memory.
//
//   out[s][m][n] = sum over the k range of split s of  x[m][k] * (q[n][k] - 8) * scale[n][k/64]
//
// The integer GEMV (gemv_w4.cu) reads the weights once for any number of rows, but mma.sync pays for every eight of them: from
// 9 rows up it is bound by that, not by the weight stream.  Here one tcgen05.mma takes 128 weight rows against all
// token rows.  A 64-k group of weights becomes the A operand as the small numbers (q - 8) / 64, exact in bf16, written
// straight into TENSOR MEMORY from registers: a W4B block's 16-byte vectors hold (row g, row g + 8) x four lanes, which is the
// fragment of tcgen05.st 16x128b, so nothing is transposed and no expanded tile crosses shared memory (a
// shared-memory A tile costs 128 cycles to store and 128 to read per block, the block's HBM time is 180).  B is the token rows in
// bf16 as they are -- in the k order in which the nibbles fall out, an order both operands share -- and a group's products are
// summed in its own fp32 accumulator, which the workers scale by the rows' fp16 scales and add up in registers: half a packed
// FMA per row, token and group, no conversion, no quantised activation, no zero-point term.
//
// One persistent CTA per SM.  A stage of the ring is a pair of n-blocks (one where there are few) x two groups and the groups' token rows, which both share:
//   warps 0-15    workers, one per TMEM quarter and block: expand a block's quarter, then add up a quarter of the token rows of all four blocks of the
//                 stage before, whose products were made in the meantime;
//   warps 16-17   issue an n-block's MMAs each;   warp 18  bulk copies.
// Two sets of weights are in tensor memory; up to 32 token rows two sets of accumulators fit beside them, and one hand-over a stage is all that
// the roles wait for.  From 33 on there is one, handed back n-block by n-block (all at once: 64 rows 38.2 us where it is 35.7).
// What bounds it is issue, the logic pipe first, beside a memory floor of 20 us with 136 pairs on 148 SMs: every instruction that the loops do not
// hold counts, and their code has to fit the instruction caches (bounded waits inlined in them cost 14 of 48 us).
// A row's bits do not depend on the other rows of the step; they are not those of the integer GEMV, whose activations are 15-bit integers.
// 34816 x 5120 / 5120 x 17408, us: 9 - 16 rows 23.3 / 12.9 (integer GEMV 31.2 / 17.0), 17 - 32 rows 26.0 / 15.0, 33 - 48 rows 31.0 / 17.7, 64 rows
// 34.5 / 19.6; with expanding and adding warps of two pipelines, as first built, 46.8 / 25.3, 59.4 / 32.3 and 65.9 / 36.2.  Measured and dropped: two CTAs of
// eight workers per SM (24.5 / 28.8 / 33.2 / 40.3 for the four row counts: twice the splits, and 64 rows have no registers).
#include "common.cuh"

using namespace b2;

namespace {

constexpr int kBlockBytes = 4352;
constexpr int kWorkers = 16, kThreads = 32 * (kWorkers + 3);      // workers, two MMA warps, one copy warp
constexpr int kMaxSplits = 16;

struct RowsParams {
  const uint8_t* w;    // [nb][KG][4352]
  const uint8_t* x;    // [KG][T][128]: stage_rows_kernel
  float* out;          // [S][M][N]
  int M, N, KG, S, gps, nb;
  int stages;          // of a CTA that are copied (tests: the others' waits run out), or more than there are
  int* fold_tickets;                    // [nb] zeroed counters, or nullptr: no fold
  const __nv_bfloat16* fold_resid_in;   // [M][N]
  __nv_bfloat16* fold_resid_out;
  float* fold_ssq;                      // [M][nb]
};

template <int T>
struct Cfg {
  static constexpr int XT = T * 128;                         // a group's token rows
  static constexpr int STAGE = 4 * kBlockBytes + 2 * XT;     // two n-blocks x two groups, and the groups' rows
  static constexpr int NS = (225 * 1024 / STAGE) < 8 ? 225 * 1024 / STAGE : 8;
  static constexpr bool TWO = T <= 32;                       // two sets of accumulators fit beside the two sets of weights
  static constexpr int DS = T <= 32 ? T : 64;                // columns from one block's accumulator to the next
  static constexpr int TW = T / 4;                           // token rows that a worker adds up
  static constexpr int OFF_BAR = NS * STAGE, BARS = (2 * NS + 8) * 8 + 16;
  static constexpr int SMEM = 1024 + OFF_BAR + BARS;
};

__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// A wait of a whole warp.  The first look is all that the hot loops hold: it costs 70 cycles where the bounded loop behind it, inlined, costs twice that
// even if the phase is over, and the loops' code has to stay small.  After a failed wait (``failed``, a word of the CTA) nobody waits for another role any
// more: no copy is issued, workers and MMAs finish on what is there, so that the tickets are counted, and what is under way is waited for before the CTA ends.
// (MMA warps that looked at the result of their waits cost 3 % at 16 rows.)
__device__ __noinline__ void wait_long(uint32_t bar, uint32_t parity, uint32_t failed, unsigned int code) {
  uint32_t f;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(f) : "r"(failed) : "memory");
  if (!f && !mbar_wait(bar, parity, code)) asm volatile("st.shared.u32 [%0], %1;" ::"r"(failed), "r"(1) : "memory");
  __syncwarp();
}
__device__ __forceinline__ void wait_all(uint32_t bar, uint32_t parity, uint32_t failed, unsigned int code) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  if (!__all_sync(0xffffffffu, ok != 0)) wait_long(bar, parity, failed, code);
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* r) {
  if constexpr (N == 4) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
  } else if constexpr (N == 8) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
  } else if constexpr (N == 12) {
    tmem_ld<8>(taddr, r);
    tmem_ld<4>(taddr + 8, r + 8);
  } else {
    static_assert(N == 16);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
  }
}
// 16 lanes x 32 columns: register 2 i + h of lane 4 g + t is lane g + 8 h, column 4 i + t
#define B2_TMEM_ST_16X128_8(taddr, r)                                                                                 \
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::   \
                   "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), \
               "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)                     \
               : "memory")

// Eight nibbles of a word -> (q - 8) / 64 as four pairs of bf16, exactly.  Up to 255 the bits of a bf16 are an integer times 2^-133, denormal or not: a nibble
// is a number where it lies (bits 0-3: q, bits 4-7: 16 q), and one fused multiply-add moves it to q / 64 - 1 / 8.  Five logic instructions a word, whose
// pipe (two cycles a warp instruction) bounds the expansion; with a shift for every nibble there are seven.
__device__ __forceinline__ void nibbles_bf16(uint32_t w, uint32_t& n0, uint32_t& n1, uint32_t& n2, uint32_t& n3) {
  const uint32_t u = w >> 8, a[4] = {w & 0x000F000Fu, w & 0x00F000F0u, u & 0x000F000Fu, u & 0x00F000F0u};
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(n0) : "r"(a[0]), "r"(0x7f007f00u), "r"(0xbe00be00u));      // 2^127
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(n1) : "r"(a[1]), "r"(0x7d007d00u), "r"(0xbe00be00u));      // 2^123
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(n2) : "r"(a[2]), "r"(0x7f007f00u), "r"(0xbe00be00u));
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(n3) : "r"(a[3]), "r"(0x7d007d00u), "r"(0xbe00be00u));
}
constexpr float kWeightScale = 64.f;
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}

// ONE: an item is a single n-block, the second of each pair is not there
template <int T, bool ONE>
__global__ void __launch_bounds__(kThreads, 1) gemm_rows_kernel(const RowsParams p) {
  using C = Cfg<T>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = smem0 + C::OFF_BAR, full0 = bars, empty0 = full0 + 8 * C::NS;
  const uint32_t afull0 = empty0 + 8 * C::NS;                           // [stage parity]
  const uint32_t done0 = afull0 + 16, free0 = done0 + 16;               // two sets of accumulators: done of [stage parity]; one: done and free of [n-block]
  const uint32_t last0 = free0 + 16;                                    // all products of [n-block] are made
  const uint32_t misc = last0 + 16, failed = misc + 8;                  // TMEM address, "last" flag; a wait ran out
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pairs = ONE ? p.nb : (p.nb + 1) >> 1, items = pairs * p.S;

  if (tid == 0) {
    for (int i = 0; i < C::NS; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, 2);     // both MMA warps' products have read the token rows; they were issued behind the workers' reading of weights and scales
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(afull0 + 8 * i, kWorkers);
      mbar_init(done0 + 8 * i, C::TWO ? 2 : 1);
      mbar_init(free0 + 8 * i, kWorkers);
      mbar_init(last0 + 8 * i, 1);
    }
    mbar_fence_init();
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(failed), "r"(0) : "memory");
  }
  if (warp == kWorkers) {
    tmem_alloc(misc, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(misc));
  const auto first_of = [&](int item) { return item % p.S * p.gps; };
  const auto groups_of = [&](int item) { const int g = first_of(item); return min(p.KG, g + p.gps) - g; };
  const auto two_of = [&](int item) { return !ONE && 2 * (item / p.S) + 1 < p.nb; };       // the last of an odd number of n-blocks is alone

  if (warp == kWorkers + 2) {
    // ---------------------------------------------------------------- copies
    if (lane == 0) {
      struct Cursor { int item, left; bool two; const uint8_t *w, *x; };      // groups left of the item; the stage's blocks of the first n-block, its rows
      const auto at = [&](int item) {
        const int pair = item / p.S, g = (item - pair * p.S) * p.gps;
        return Cursor{item, min(p.KG, g + p.gps) - g, !ONE && 2 * pair + 1 < p.nb, p.w + ((size_t)(ONE ? pair : 2 * pair) * p.KG + g) * kBlockBytes, p.x + (size_t)g * C::XT};
      };
      const auto step = [&](Cursor& c) {
        c.w += 2 * kBlockBytes;
        c.x += 2 * C::XT;
        if ((c.left -= 2) <= 0) c = at(c.item + gridDim.x);
      };
      const size_t next_block = (size_t)p.KG * kBlockBytes;
      const auto weights = [&](const Cursor& c, int slot) {
        const uint32_t ng = min(c.left, 2), bar = full0 + 8 * slot, dst = smem0 + slot * C::STAGE + 2 * C::XT;
        mbar_expect_tx(bar, ng * ((c.two ? 2 : 1) * kBlockBytes + C::XT));
        bulk_g2s(dst, c.w, ng * kBlockBytes, bar);
        if (c.two) bulk_g2s(dst + 2 * kBlockBytes, c.w + next_block, ng * kBlockBytes, bar);
      };
      const auto rows = [&](const Cursor& c, int slot) { bulk_g2s(smem0 + slot * C::STAGE, c.x, min(c.left, 2) * C::XT, full0 + 8 * slot); };
      Cursor cw = at(blockIdx.x), cx = cw;
      int n = 0;
      for (; n < C::NS && n < p.stages && cw.item < items; ++n, step(cw)) weights(cw, n);      // they depend on nothing: asked for before the previous kernel is done
      pdl_wait();
      for (int i = 0; i < n; ++i, step(cx)) rows(cx, i);
      int slot = 0, round = 1;
      for (int left = p.stages - n; left > 0 && cw.item < items; --left, step(cw)) {
        uint32_t stop = !mbar_wait(empty0 + 8 * slot, (round - 1) & 1, ERR_GEMM_EMPTY_WAIT);
        if (!stop) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(stop) : "r"(failed) : "memory");      // (a stage may then be "empty" that is still on its way)
        if (stop) break;
        weights(cw, slot);
        rows(cw, slot);
        if (++slot == C::NS) { slot = 0; ++round; }
      }
      // every slot's last copies arrive (bounded) before the CTA ends, whether anybody else has waited for them or not
      for (int i = 0; i < n; ++i) mbar_wait(full0 + 8 * i, (i < slot ? round : round - 1) & 1, ERR_GEMM_FULL_WAIT);
    }
  } else if (warp >= kWorkers) {
    // ---------------------------------------------------------------- MMAs of one n-block of the pair
    const int h = warp - kWorkers;
    constexpr uint32_t idesc = make_idesc(1, 1, 128, T);
    const uint64_t xdesc = make_desc_sw128(smem0);
    const uint32_t xd_lo = (uint32_t)xdesc, xd_hi = (uint32_t)(xdesc >> 32), a0 = tmem + h * 64, d0 = tmem + 256 + h * 2 * C::DS;
    int slot = 0, phase = 0, n = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const bool live = h == 0 || two_of(item);
#pragma unroll 1
      for (int left = groups_of(item); left > 0; left -= 2, ++n) {
        const uint32_t par = n & 1;
        wait_all(full0 + 8 * slot, phase, failed, ERR_GEMM_FULL_WAIT);
        wait_all(afull0 + 8 * par, (n >> 1) & 1, failed, ERR_GEMM_TMEM_FULL_WAIT);
        if (!C::TWO && n > 0) wait_all(free0 + 8 * h, (n - 1) & 1, failed, ERR_GEMM_TMEM_EMPTY_WAIT);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t xlo = xd_lo + slot * (C::STAGE >> 4), a = a0 + par * 128, d = d0 + (C::TWO ? par * 128 : 0);
          if (live) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              if (left <= j) break;
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f16_ts_w(d + j * C::DS, a + j * 32 + 8 * k, xlo + j * (C::XT >> 4) + 2 * k, xd_hi, idesc, k != 0);    // 16 k = 32 bytes a step
            }
          }
          tc_commit(empty0 + 8 * slot);
          tc_commit(done0 + 8 * (C::TWO ? par : h));
        }
        __syncwarp();
        if (++slot == C::NS) { slot = 0; phase ^= 1; }
      }
    }
    // what was issued is done (bounded) before tensor memory is given back
    if (elect_one()) tc_commit(last0 + 8 * h);
    __syncwarp();
    if (lane == 0) mbar_wait(last0 + 8 * h, 0, ERR_GEMM_TMEM_FULL_WAIT);
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- expand a stage, add up the one before
    const int q = warp & 3, sub = warp >> 2;                   // quarter of the rows; block to expand and token rows to add up
    const int row = 32 * q + lane;
    const uint32_t lanes = (uint32_t)(32 * q) << 16;
    const uint32_t v_off = 2 * C::XT + sub * kBlockBytes + 2 * q * 512 + lane * 16;
    const uint32_t sc_off = 2 * C::XT + 4096 + ((row >> 4) * 16 + 2 * (row & 7) + ((row >> 3) & 1)) * 2;
    pdl_wait();
    pdl_launch_dependents();
    uint64_t acc[2][C::TW / 2];
    uint32_t st = smem0, full = full0, phase = 0;                                     // the ring
    uint32_t a = tmem + sub * 32 + lanes, afull = afull0;                             // weights' columns; alternate
    uint32_t d = tmem + 256 + sub * C::TW + lanes, done = done0, done_phase = 0;      // products' columns
    struct Scales { __half2 h[2]; };                                                  // the row's, two groups of each n-block
    const auto none = [] {};
    // between: done while the expanded weights are on their way into tensor memory
    const auto expand = [&](auto&& between) -> Scales {
      wait_all(full, phase, failed, ERR_GEMM_FULL_WAIT);
      uint4 v[2];
      unsigned short sc[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[e].x), "=r"(v[e].y), "=r"(v[e].z), "=r"(v[e].w) : "r"(st + v_off + e * 512));
#pragma unroll
      for (int b = 0; b < 4; ++b) asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sc[b]) : "r"(st + sc_off + b * kBlockBytes));
      // these columns were read by the MMAs of two stages ago, whose products this warp has waited for
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t w[4] = {v[e].x, v[e].y, v[e].z, v[e].w};
        uint32_t r[16];
        // column 4 i + t, i = 4 (32-k step) + 2 (low or high byte of a pair) + (nibble): k = 32 ks + 16 hi + 4 t + o + 2 e
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) nibbles_bf16(w[2 * ks + hf], r[8 * ks + hf], r[8 * ks + 2 + hf], r[8 * ks + 4 + hf], r[8 * ks + 6 + hf]);
        B2_TMEM_ST_16X128_8(a + ((uint32_t)(16 * e) << 16), r);
      }
      between();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(afull);
      st += C::STAGE;
      full += 8;
      if (full == empty0) { st = smem0; full = full0; phase ^= 1; }
      a ^= 128;
      afull ^= 8;
      Scales o;
#pragma unroll
      for (int e = 0; e < 2; ++e) o.h[e] = __halves2half2(__ushort_as_half(sc[2 * e]), __ushort_as_half(sc[2 * e + 1]));
      return o;
    };
    // One set of accumulators: an n-block's is handed back as soon as it is in registers, and its next products are made while the other n-block's are
    // added up and a stage is expanded.  groups: of the stage (1: its second one is not there); two: the pair has its second n-block.
    const auto fold = [&](const Scales& sc, int b, const uint32_t* v) {
      const float2 f = __half22float2(sc.h[b >> 1]);
      const float w = b & 1 ? f.y : f.x;
      const uint64_t w2 = pack2(__float_as_uint(w), __float_as_uint(w));
#pragma unroll
      for (int i = 0; i < C::TW; i += 2)
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[b >> 1][i / 2]) : "l"(pack2(v[i], v[i + 1])), "l"(w2));
    };
    const auto add = [&](const Scales& sc, int groups, bool two) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        wait_all(done0 + 8 * h, done_phase, failed, ERR_GEMM_TMEM_FULL_WAIT);
        tc_fence_after();
        uint32_t v[2][C::TW];
#pragma unroll
        for (int j = 0; j < 2; ++j) tmem_ld<C::TW>(d + (2 * h + j) * C::DS, v[j]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(free0 + 8 * h);
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (!(j && groups == 1) && !(h && !two)) fold(sc, 2 * h + j, v[j]);      // else the block is not there
      }
      done_phase ^= 1;
    };
    // Two sets: load() asks for a stage's products, sum() adds them up
    uint32_t v2[4][C::TWO ? C::TW : 1];
    const auto load = [&] {
      wait_all(done, done_phase, failed, ERR_GEMM_TMEM_FULL_WAIT);
      tc_fence_after();
      if constexpr (C::TWO) {
#pragma unroll
        for (int b = 0; b < 4; ++b) tmem_ld<C::TW>(d + b * C::DS, v2[b]);
      }
      d ^= 128;
      done_phase ^= done != done0;
      done ^= 8;
    };
    const auto sum = [&](const Scales& sc, int groups, bool two) {
      tmem_ld_wait();
      if constexpr (C::TWO) {
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (!((b & 1) && groups == 1) && !((b >> 1) && !two)) fold(sc, b, v2[b]);
      }
    };
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int pair = item / p.S, split = item - pair * p.S;
      const bool two = two_of(item);
#pragma unroll
      for (int i = 0; i < C::TW / 2; ++i) acc[0][i] = acc[1][i] = 0;
      Scales scales = expand(none);
      int left = groups_of(item);
      if (C::TWO) {
        // up to 16 token rows the products of the stage before are on their way while a stage is expanded and the one before them is added up (24.7 -> 23.1 us;
        // with 32 they are made in time: 26.6 / 27.4)
        if (T > 16) {
#pragma unroll 1
          for (; left > 2; left -= 2) {
            const Scales next = expand(none);
            load();
            sum(scales, 2, two);
            scales = next;
          }
        } else if (left > 2) {
          Scales next = expand(none);
#pragma unroll 1
          for (left -= 2; left > 2; left -= 2) {
            load();
            const Scales after = expand([&] { sum(scales, 2, two); });
            scales = next;
            next = after;
          }
          load();
          sum(scales, 2, two);
          scales = next;
        }
        load();
        sum(scales, left, two);
      } else {
#pragma unroll 1
        for (; left > 2; left -= 2) {
          const Scales next = expand(none);
          add(scales, 2, two);
          scales = next;
        }
        add(scales, left, two);
      }
      // ---- the item's sums
#pragma unroll
      for (int h = 0; h < (ONE ? 1 : 2); ++h) {
        const int col = ((ONE ? pair : 2 * pair) + h) * 128 + row;
        float* o = p.out + ((size_t)split * p.M + sub * C::TW) * p.N + col;
#pragma unroll
        for (int i = 0; i < C::TW; ++i)
          if (sub * C::TW + i < p.M && col < p.N) o[(size_t)i * p.N] = kWeightScale * __uint_as_float((uint32_t)(acc[h][i / 2] >> (32 * (i & 1))));
      }
      if (p.fold_tickets == nullptr) continue;
      // ---- the last split of a pair adds the slices in split order to the residual rows and leaves the sums of squares of each
      // n-block's 128 columns.
      __threadfence();
      workers_sync();
      if (tid == 0) {
        const int last = atomicAdd(&p.fold_tickets[ONE ? pair : 2 * pair], 1) == p.S - 1;
        if (last) p.fold_tickets[ONE ? pair : 2 * pair] = 0;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(misc + 4), "r"(last) : "memory");
      }
      workers_sync();
      int last;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(last) : "r"(misc + 4));
      if (!last) continue;
      __threadfence();
      const int blocks = two ? 2 : 1;
      for (int t = warp; t < p.M * blocks; t += kWorkers) {       // a warp per row and n-block, four columns per lane, the slices' loads in flight together
        const int m = t / blocks, nblk = (ONE ? pair : 2 * pair) + t % blocks, fn = nblk * 128 + lane * 4;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (p.N % 4 == 0 && fn + 4 <= p.N) {
          const uint2 r = *reinterpret_cast<const uint2*>(p.fold_resid_in + (size_t)m * p.N + fn);
          f[0] = bf16_lo(r.x); f[1] = bf16_hi(r.x); f[2] = bf16_lo(r.y); f[3] = bf16_hi(r.y);
#pragma unroll 1
          for (int s0 = 0; s0 < p.S; s0 += 8) {
            float4 u[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
              u[e] = s0 + e < p.S ? __ldcg(reinterpret_cast<const float4*>(p.out + ((size_t)(s0 + e) * p.M + m) * p.N + fn)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 8; ++e) { f[0] += u[e].x; f[1] += u[e].y; f[2] += u[e].z; f[3] += u[e].w; }
          }
          const uint2 o2 = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
          *reinterpret_cast<uint2*>(p.fold_resid_out + (size_t)m * p.N + fn) = o2;
          f[0] = bf16_lo(o2.x); f[1] = bf16_hi(o2.x); f[2] = bf16_lo(o2.y); f[3] = bf16_hi(o2.y);
        } else {
          for (int i = 0; i < 4 && fn + i < p.N; ++i) {
            f[i] = __bfloat162float(p.fold_resid_in[(size_t)m * p.N + fn + i]);
            for (int sp = 0; sp < p.S; ++sp) f[i] += __ldcg(p.out + ((size_t)sp * p.M + m) * p.N + fn + i);
            const __nv_bfloat16 rb = __float2bfloat16(f[i]);
            p.fold_resid_out[(size_t)m * p.N + fn + i] = rb;
            f[i] = __bfloat162float(rb);
          }
        }
        const float ss = warp_sum((f[0] * f[0] + f[1] * f[1]) + (f[2] * f[2] + f[3] * f[3]));
        if (lane == 0) p.fold_ssq[(size_t)m * p.nb + nblk] = ss;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kWorkers) tmem_dealloc(tmem, 512);
}

template <int T, bool ONE>
int launch_items(const RowsParams& p, int items, cudaStream_t stream) {
  using C = Cfg<T>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<T, ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  return b2_launch(gemm_rows_kernel<T, ONE>, dim3(items), dim3(kThreads), C::SMEM, stream, true, p);
}
// While every n-block and split has an SM of its own, a CTA takes one n-block: half the stage, and a fold of half the columns, whose slices a lone SM reads at
// 64 bytes a cycle.  us with fold, pairs / one, 17 / 32 / 64 rows: 2048 x 2048 in eight splits 9.2 / 7.3, 11.1 / 7.6, 17.0 / 11.0, 512 x 1408 in six 8.4 / 6.7,
// 10.2 / 6.9, 15.7 / 10.3; without one 2816 x 512 3.1 / 2.8, 3.3 / 2.8, 4.4 / 3.5.  (The bits are the same: a block's sums do not know its neighbour.)
template <int T>
int launch_rows(const RowsParams& p, cudaStream_t stream) {
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!sms[dev & 63]) {
    int n = 0;
    const cudaError_t e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    sms[dev & 63] = n;
  }
  if (p.nb * p.S <= sms[dev & 63]) return launch_items<T, true>(p, p.nb * p.S, stream);
  const int items = (p.nb + 1) / 2 * p.S;
  return launch_items<T, false>(p, items < sms[dev & 63] ? items : sms[dev & 63], stream);
}

}  // namespace

// ``x``: b2_stage_rows of the same M and K, whose rows are padded to 16, 32, 48 or 64 (decode steps come here from 9 rows on).  S <= 16 splits of whole fours of groups, none of them empty.
// stages: of every CTA that are copied, for tests of what waits that run out leave behind (0: all).
extern "C" int b2_gemm_w4_rows(const void* w4b, const void* x, float* out, int M, int N, int K, int S, int* fold_tickets,
                               const void* fold_resid_in, void* fold_resid_out, float* fold_ssq, int stages, void* stream) {
  if (M < 1 || M > 64 || N < 1 || K < 64 || K % 64 != 0 || S < 1 || S > kMaxSplits) return -1;
  if ((((uintptr_t)w4b | (uintptr_t)x | (uintptr_t)out) & 15) || (((uintptr_t)fold_resid_in | (uintptr_t)fold_resid_out) & 7)) return -4;
  RowsParams p;
  p.w = (const uint8_t*)w4b; p.x = (const uint8_t*)x; p.out = out;
  p.M = M; p.N = N; p.KG = K / 64; p.S = S; p.nb = (N + 127) / 128;
  p.gps = ((p.KG + S - 1) / S + 3) / 4 * 4;
  if (p.gps * (S - 1) >= p.KG) return -2;                      // every split has groups
  p.stages = stages > 0 ? stages : 1 << 30;
  p.fold_tickets = fold_tickets; p.fold_resid_in = (const __nv_bfloat16*)fold_resid_in;
  p.fold_resid_out = (__nv_bfloat16*)fold_resid_out; p.fold_ssq = fold_ssq;
  cudaStream_t st = (cudaStream_t)stream;
  if (M <= 16) return launch_rows<16>(p, st);
  if (M <= 32) return launch_rows<32>(p, st);
  if (M <= 48) return launch_rows<48>(p, st);
  return launch_rows<64>(p, st);
}

B2_DEFINE_STATUS(gemmrows)
