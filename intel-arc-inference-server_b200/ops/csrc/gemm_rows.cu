// W4A16 linears of decode steps with many rows (up to 64) on tcgen05: weights in tensor memory, activations in shared memory.
//
//   out[s][m][n] = sum over the k range of split s of  x[m][k] * (q[n][k] - 8) * scale[n][k/64]
//
// The integer GEMV (gemv_w4.cu) reads the weights once for any number of rows, but mma.sync pays for every eight of them: from
// 9 rows up it is bound by that, not by the weight stream.  Here one tcgen05.mma takes 128 weight rows against all
// token rows.  A 64-k group of weights becomes the A operand as the small integers q - 8, exact in bf16, written
// straight into TENSOR MEMORY from registers: a W4B block's 16-byte vectors hold (row g, row g + 8) x four lanes, which is the
// fragment of tcgen05.st 16x128b, so nothing is transposed and no expanded tile crosses shared memory (a
// shared-memory A tile costs 128 cycles to store and 128 to read per block, the block's HBM time is 180).  B is the token rows in
// bf16 as they are -- in the k order in which the nibbles fall out, an order both operands share -- and a group's products are
// summed in its own fp32 accumulator, which the workers scale by the rows' fp16 scales and add up in registers: one
// FMA per row, token and group, no conversion, no quantised activation, no zero-point term.
//
// One persistent CTA per SM, 20 warps.  A ring stage is four consecutive blocks; even and odd blocks go through two pipelines of
// the same roles, which meet nowhere but at barriers, so that expanding, multiplying and adding up different blocks overlap:
//   warps 0-7    expand: four warps (one per TMEM quarter) a pipeline, its two blocks of a stage at a time; A buffers for two stages;
//   warps 8-15   add up: wait for a block's products, scale, add; two accumulators a pipeline (2 x (4 x 32 + 2 x 64) TMEM columns);
//   warp 16      bulk copies of weights, 17 KB a stage;   warp 17  bulk copies of the token rows, 4 T x 128 bytes a stage;
//   warps 18-19  issue a pipeline's MMAs each (a lone thread retires an instruction every ten cycles or so).
// At the end of an item (128 output rows x one k split) the pipelines' sums meet in shared memory, even blocks first, while the
// other roles are ahead in the next item.  A row's bits do
// not depend on the other rows of the step; they are not those of the integer GEMV, whose activations are 15-bit integers.
// 34816 x 5120 / 5120 x 17408, us (integer GEMV in brackets): 17 - 32 rows 47 / 26 (88 / 46), 33 - 48 rows 61 / 34 (132 / 70), 64 rows
// 65 / 36 (156 / 82).  The bytes would take 14 / 7: a stage takes 2100 to 3300 cycles in which no role is busy more than half the
// time; they wait for one another's products.  (One role per warp set with a barrier per block, as first built: 57, 68 and 84 us.
// One lane polling for its warp: 4 to 9 % slower.  One MMA in place of four: no change.)
#include "common.cuh"

using namespace b2;

namespace {

constexpr int kBlockBytes = 4352;
constexpr int kStageBlocks = 4, kThreads = 640;
constexpr int kMaxSplits = 16;

struct RowsParams {
  const uint8_t* w;    // [nb][KG][4352]
  const uint8_t* x;    // [KG][T][128]: stage_rows_kernel
  float* out;          // [S][M][N]
  int M, N, KG, S, gps, nb;
  int* fold_tickets;                    // [nb] zeroed counters, or nullptr: no fold
  const __nv_bfloat16* fold_resid_in;   // [M][N]
  __nv_bfloat16* fold_resid_out;
  float* fold_ssq;                      // [M][nb]
};

template <int T>
struct Cfg {
  static constexpr int XB = kStageBlocks * T * 128, WB = kStageBlocks * kBlockBytes;      // a stage's token rows and weights
  static constexpr int RED = T * 512;                                       // half the token rows of each pipeline's sums
  static constexpr int NX = T <= 32 ? 6 : T <= 48 ? 4 : 3, NW = T <= 32 ? 6 : 5;
  static constexpr int OFF_RAW = NX * XB, OFF_RED = OFF_RAW + NW * WB, OFF_BAR = OFF_RED + RED;
  static constexpr int BARS = (2 * NW + 2 * NX + 16) * 8 + 16;
  static constexpr int SMEM = 1024 + OFF_BAR + BARS;
};

__device__ __forceinline__ void adders_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

#define B2_TMEM_LD_16(taddr, r)                                                                                       \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" \
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),  \
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])                    \
               : "r"(taddr)                                                                                           \
               : "memory")
// 16 lanes x 32 columns: register 2 i + h of lane 4 g + t is lane g + 8 h, column 4 i + t
#define B2_TMEM_ST_16X128_8(taddr, r)                                                                                 \
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::   \
                   "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), \
               "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)                     \
               : "memory")

// two nibbles (bits 0-3 and 16-19) -> q - 8 as a pair of bf16: 0x4300 | q is 128 + q, and the difference is exact
__device__ __forceinline__ uint32_t nibbles_bf16(uint32_t w, int shift) {
  const uint32_t x = ((w >> shift) & 0x000F000Fu) | 0x43004300u;
  uint32_t y;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(y) : "r"(x), "r"(0x43084308u));
  return y;
}

template <int T>
__global__ void __launch_bounds__(kThreads, 1) gemm_rows_kernel(const RowsParams p) {
  using C = Cfg<T>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t xs0 = smem0, raw0 = smem0 + C::OFF_RAW, red0 = smem0 + C::OFF_RED, bars = smem0 + C::OFF_BAR;
  const uint32_t wfull0 = bars, wempty0 = wfull0 + 8 * C::NW, xfull0 = wempty0 + 8 * C::NW, xempty0 = xfull0 + 8 * C::NX;
  const uint32_t afull0 = xempty0 + 8 * C::NX, afree0 = afull0 + 32;           // [pipeline][stage parity]
  const uint32_t dfull0 = afree0 + 32, dempty0 = dfull0 + 32;                  // [pipeline][block of the stage]
  const uint32_t misc = dempty0 + 32;                                          // TMEM address, "last" flag
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int items = p.nb * p.S;

  if (tid == 0) {
    for (int i = 0; i < C::NW; ++i) {
      mbar_init(wfull0 + 8 * i, 1);
      mbar_init(wempty0 + 8 * i, 16);            // expanding warps have read their vectors, adding warps their scales
    }
    for (int i = 0; i < C::NX; ++i) {
      mbar_init(xfull0 + 8 * i, 1);
      mbar_init(xempty0 + 8 * i, 2);             // both pipelines' MMAs have read the token rows
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(afull0 + 8 * i, 4);
      mbar_init(afree0 + 8 * i, 1);
      mbar_init(dfull0 + 8 * i, 1);
      mbar_init(dempty0 + 8 * i, 4);
    }
    mbar_fence_init();
  }
  if (warp == 17) {
    tmem_alloc(misc, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(misc));
  const auto groups_of = [&](int item) { const int s = item % p.S; return min(p.KG, (s + 1) * p.gps) - s * p.gps; };

  if (warp >= 18) {
    // ---------------------------------------------------------------- MMAs of pipeline warp - 18
    if (lane == 0) {
      const int pipe = warp - 18;
      constexpr uint32_t idesc = make_idesc(1, 1, 128, T);
      const uint64_t xdesc = make_desc_sw128(xs0 + pipe * T * 128);
      const uint32_t xd_lo = (uint32_t)xdesc, xd_hi = (uint32_t)(xdesc >> 32), a0 = tmem + pipe * 256, d0 = a0 + 128;
      const uint32_t af = afull0 + 16 * pipe, fr = afree0 + 16 * pipe, df = dfull0 + 16 * pipe, de = dempty0 + 16 * pipe;
      int xs = 0, xp = 0, n = 0, used[2] = {0, 0};       // n: stages before
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        for (int left = groups_of(item) - pipe; left > -pipe && ok; left -= kStageBlocks, ++n) {      // blocks of the stage from this one on
          const uint32_t par = n & 1;
          ok = mbar_wait(xfull0 + 8 * xs, xp, ERR_GEMM_FULL_WAIT) && mbar_wait(af + 8 * par, (n >> 1) & 1, ERR_GEMM_TMEM_FULL_WAIT);
          if (!ok) break;
          const uint32_t xlo = xd_lo + xs * (C::XB >> 4), a = a0 + par * 64;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (left <= 2 * j) break;
            if (used[j] > 0) {
              ok = mbar_wait(de + 8 * j, (used[j] - 1) & 1, ERR_GEMM_TMEM_EMPTY_WAIT);
              if (!ok) break;
              tc_fence_after();
            }
            ++used[j];
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_f16_ts_w(d0 + j * 64, a + j * 32 + 8 * k, xlo + j * (2 * T * 128 >> 4) + 2 * k, xd_hi, idesc, k != 0);    // 16 k = 32 bytes a step
            tc_commit(df + 8 * j);
          }
          if (left > 0) tc_commit(fr + 8 * par);
          else mbar_arrive(fr + 8 * par);
          if (++xs == C::NX) { xs = 0; xp ^= 1; }
        }
      }
    }
  } else if (warp >= 16) {
    // ---------------------------------------------------------------- copies
    if (lane == 0) {
      const bool wt = warp == 16;
      const int n = wt ? C::NW : C::NX, unit = wt ? kBlockBytes : T * 128;
      const uint32_t full0 = wt ? wfull0 : xfull0, empty0 = wt ? wempty0 : xempty0, dst0 = wt ? raw0 : xs0;
      const uint32_t stage = kStageBlocks * unit;
      if (!wt) pdl_wait();       // the weights depend on nothing: their first stages are asked for before the previous kernel is done
      int slot = 0, round = 0;   // stage of the ring, times it was filled before
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int nblk = item / p.S, g0 = (item - nblk * p.S) * p.gps;
        int left = min(p.KG, g0 + p.gps) - g0;
        const uint8_t* src = wt ? p.w + ((size_t)nblk * p.KG + g0) * kBlockBytes : p.x + (size_t)g0 * (T * 128);
        for (; left > 0; left -= kStageBlocks, src += stage) {
          if (round > 0) ok = mbar_wait(empty0 + 8 * slot, (round - 1) & 1, ERR_GEMM_EMPTY_WAIT);
          if (!ok) break;
          const uint32_t bytes = min(left, kStageBlocks) * unit, bar = full0 + 8 * slot;
          mbar_expect_tx(bar, bytes);
          bulk_g2s(dst0 + slot * stage, src, bytes, bar);
          if (++slot == n) { slot = 0; ++round; }
        }
      }
      if (!ok)   // wait (bounded) for the copies that were issued and possibly never consumed: those of the last round
        for (int i = 0; i < n; ++i) {
          const int r = i < slot ? round : round - 1;
          if (r >= 0) mbar_wait(full0 + 8 * i, r & 1, ERR_GEMM_FULL_WAIT);
        }
    }
  } else if (warp < 8) {
    // ---------------------------------------------------------------- expand
    const int pipe = warp >> 2, q = warp & 3;
    const uint32_t a0 = tmem + pipe * 256 + ((uint32_t)(32 * q) << 16), af = afull0 + 16 * pipe, fr = afree0 + 16 * pipe;
    const uint32_t v_off = pipe * kBlockBytes + 2 * q * 512 + lane * 16;
    int ws = 0, wp = 0, n = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      for (int left = groups_of(item) - pipe; left > -pipe; left -= kStageBlocks, ++n) {
        ok = __all_sync(0xffffffffu, mbar_wait(wfull0 + 8 * ws, wp, ERR_GEMM_FULL_WAIT));
        if (!ok) break;
        const uint32_t st = raw0 + ws * C::WB + v_off, par = n & 1;
        uint4 v[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (left > 2 * j)
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[j][h].x), "=r"(v[j][h].y), "=r"(v[j][h].z), "=r"(v[j][h].w) : "r"(st + j * 2 * kBlockBytes + h * 512));
        __syncwarp();
        if (lane == 0) mbar_arrive(wempty0 + 8 * ws);
        if (++ws == C::NW) { ws = 0; wp ^= 1; }
        if (n >= 2) ok = __all_sync(0xffffffffu, mbar_wait(fr + 8 * par, ((n >> 1) - 1) & 1, ERR_GEMM_TMEM_EMPTY_WAIT));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (left <= 2 * j) break;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t w[4] = {v[j][h].x, v[j][h].y, v[j][h].z, v[j][h].w};
            uint32_t r[16];
            // column 4 i + t, i = 4 (32-k step) + 2 (low or high byte of a pair) + (nibble): k = 32 ks + 16 hi + 4 t + o + 2 e
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) r[2 * i + hf] = nibbles_bf16(w[2 * (i >> 2) + hf], 8 * ((i >> 1) & 1) + 4 * (i & 1));
            B2_TMEM_ST_16X128_8(a0 + par * 64 + j * 32 + ((uint32_t)(16 * h) << 16), r);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(af + 8 * par);
      }
    }
  } else {
    // ---------------------------------------------------------------- add up
    const int pipe = (warp - 8) >> 2, q = warp & 3;
    const uint32_t d0 = tmem + pipe * 256 + 128 + ((uint32_t)(32 * q) << 16), df = dfull0 + 16 * pipe, de = dempty0 + 16 * pipe;
    const int row = 32 * q + lane, at = tid - 256;
    const uint32_t sc_off = pipe * kBlockBytes + 4096 + ((row >> 4) * 16 + 2 * (row & 7) + ((row >> 3) & 1)) * 2;
    pdl_wait();
    pdl_launch_dependents();
    int ws = 0, wp = 0, xs = 0, xp = 0, used[2] = {0, 0};
    bool ok = true;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int nblk = item / p.S, split = item - nblk * p.S;
      float acc[T];
#pragma unroll
      for (int i = 0; i < T; ++i) acc[i] = 0.f;
      for (int left = groups_of(item) - pipe; left > -pipe; left -= kStageBlocks) {
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(wfull0 + 8 * ws, wp, ERR_GEMM_FULL_WAIT));
        float scale[2] = {0.f, 0.f};
        if (ok) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            unsigned short h = 0;
            if (left > 2 * j) asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(raw0 + ws * C::WB + j * 2 * kBlockBytes + sc_off));
            scale[j] = __half2float(__ushort_as_half(h));
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(wempty0 + 8 * ws);
        }
        if (++ws == C::NW) { ws = 0; wp ^= 1; }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (left <= 2 * j) break;
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(df + 8 * j, used[j] & 1, ERR_GEMM_TMEM_FULL_WAIT));
          ++used[j];
          if (!ok) continue;
          tc_fence_after();
#pragma unroll
          for (int c0 = 0; c0 < T; c0 += 16) {
            uint32_t d[16];
            B2_TMEM_LD_16(d0 + j * 64 + c0, d);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[c0 + i] = fmaf(scale[j], __uint_as_float(d[i]), acc[c0 + i]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(de + 8 * j);
        }
        // the stage's token rows have been read by this pipeline's MMAs (which its products say; without one, the copy has to have
        // landed before the stage may be handed back)
        if (ok && q == 0) {
          if (left <= 0) ok = __all_sync(0xffffffffu, mbar_wait(xfull0 + 8 * xs, xp, ERR_GEMM_FULL_WAIT));
          if (ok && lane == 0) mbar_arrive(xempty0 + 8 * xs);
        }
        if (++xs == C::NX) { xs = 0; xp ^= 1; }
      }
      // ---- the pipelines' sums: each takes half of the token rows from the other, even blocks first
      constexpr int H = T / 2;
      const uint32_t col = red0 + (uint32_t)row * 4;
      const int n = nblk * 128 + row;
      adders_sync();              // what was in the buffers before has been read
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const float give = pipe ? acc[i] : acc[H + i];
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(col + (pipe * H + i) * 512), "f"(give) : "memory");
      }
      adders_sync();
      float* o = p.out + ((size_t)split * p.M + pipe * H) * p.N + n;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        float other;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(other) : "r"(col + ((pipe ^ 1) * H + i) * 512));
        const float mine = pipe ? acc[H + i] : acc[i];
        if (pipe * H + i < p.M && n < p.N) o[(size_t)i * p.N] = pipe ? other + mine : mine + other;
      }
      if (p.fold_tickets == nullptr) continue;
      // ---- the last split of an n-block adds the slices in split order to the residual rows and leaves the sums of squares of
      // its 128 columns.
      __threadfence();
      adders_sync();
      if (at == 0) {
        const int last = atomicAdd(&p.fold_tickets[nblk], 1) == p.S - 1;
        if (last) p.fold_tickets[nblk] = 0;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(misc + 4), "r"(last) : "memory");
      }
      adders_sync();
      int last;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(last) : "r"(misc + 4));
      if (!last) continue;
      __threadfence();
      const int fn = nblk * 128 + lane * 4;       // a warp per row, four columns per lane, the slices' loads in flight together
      for (int m = warp - 8; m < p.M; m += 8) {
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (p.N % 4 == 0 && fn + 4 <= p.N) {
          const uint2 r = *reinterpret_cast<const uint2*>(p.fold_resid_in + (size_t)m * p.N + fn);
          f[0] = bf16_lo(r.x); f[1] = bf16_hi(r.x); f[2] = bf16_lo(r.y); f[3] = bf16_hi(r.y);
#pragma unroll 1
          for (int s0 = 0; s0 < p.S; s0 += 8) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              v[u] = s0 + u < p.S ? __ldcg(reinterpret_cast<const float4*>(p.out + ((size_t)(s0 + u) * p.M + m) * p.N + fn)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; ++u) { f[0] += v[u].x; f[1] += v[u].y; f[2] += v[u].z; f[3] += v[u].w; }
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
  if (warp == 17) tmem_dealloc(tmem, 512);
}

template <int T>
int launch_rows(const RowsParams& p, cudaStream_t stream) {
  using C = Cfg<T>;
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!sms[dev & 63]) {
    int n = 0;
    cudaError_t e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return (int)e;
    sms[dev & 63] = n;
  }
  const int items = p.nb * p.S, grid = items < sms[dev & 63] ? items : sms[dev & 63];
  return b2_launch(gemm_rows_kernel<T>, dim3(grid), dim3(kThreads), C::SMEM, stream, true, p);
}

}  // namespace

// ``x``: b2_stage_rows of the same M and K, whose rows are padded to 32, 48 or 64 (decode steps come here from 17 rows on).  S <= 16 splits of whole fours of groups, none of them empty.
extern "C" int b2_gemm_w4_rows(const void* w4b, const void* x, float* out, int M, int N, int K, int S, int* fold_tickets,
                               const void* fold_resid_in, void* fold_resid_out, float* fold_ssq, void* stream) {
  if (M < 1 || M > 64 || N < 1 || K < 64 || K % 64 != 0 || S < 1 || S > kMaxSplits) return -1;
  if ((((uintptr_t)w4b | (uintptr_t)x | (uintptr_t)out) & 15) || (((uintptr_t)fold_resid_in | (uintptr_t)fold_resid_out) & 7)) return -4;
  RowsParams p;
  p.w = (const uint8_t*)w4b; p.x = (const uint8_t*)x; p.out = out;
  p.M = M; p.N = N; p.KG = K / 64; p.S = S; p.nb = (N + 127) / 128;
  p.gps = ((p.KG + S - 1) / S + kStageBlocks - 1) / kStageBlocks * kStageBlocks;    // whole stages
  if (p.gps * (S - 1) >= p.KG) return -2;                      // every split has groups
  p.fold_tickets = fold_tickets; p.fold_resid_in = (const __nv_bfloat16*)fold_resid_in;
  p.fold_resid_out = (__nv_bfloat16*)fold_resid_out; p.fold_ssq = fold_ssq;
  cudaStream_t st = (cudaStream_t)stream;
  if (M <= 32) return launch_rows<32>(p, st);
  if (M <= 48) return launch_rows<48>(p, st);
  return launch_rows<64>(p, st);
}

B2_DEFINE_STATUS(gemmrows)
