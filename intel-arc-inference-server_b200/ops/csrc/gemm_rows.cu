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
// One persistent CTA per SM, 18 warps.  A stage is four consecutive blocks, one for each set of workers:
//   warps 0-15  four sets of four warps (a warp per TMEM quarter): load the block's vectors, expand, store A; when the group's products
//               are there, scale and add.  A set expands its next block while the MMAs of this one run (two A buffers, one
//               accumulator: 4 x (2 x 32 + 64) = 512 TMEM columns), then meets at a named barrier and its first lane issues
//               the next MMAs: issuing for four sets by one thread cost 1200 cycles a block (a lone thread retires an instruction
//               every ten cycles), four threads do it side by side;
//   warp 16     bulk copies of weights, 17 KB a stage;   warp 17  bulk copies of the token rows, 4 T x 128 bytes a stage.
// At the end of an item (128 output rows x one k split) the sets' sums meet in shared memory in a fixed order.  A row's bits do
// not depend on the other rows of the step; they are not those of the integer GEMV, whose activations are 15-bit integers.
// 34816 x 5120 / 5120 x 17408, us (integer GEMV in brackets): 17 - 32 rows 57 / 32 (88 / 46), 33 - 48 rows 68 / 38 (133 / 70), 64 rows
// 84 / 50 (156 / 82); a step of 40 requests through 16 layers of the 27B shape 5.90 -> 4.43 ms.  The bytes would take 14 / 7: a stage
// takes 2200 cycles, of which a set spends 580 expanding, 620 on its first lane's issue and 470 waiting for the products.
#include "common.cuh"

using namespace b2;

namespace {

constexpr int kBlockBytes = 4352;
constexpr int kSets = 4, kWorkers = kSets * 128, kThreads = kWorkers + 64;
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
  static constexpr int XB = kSets * T * 128, WB = kSets * kBlockBytes;      // a stage's token rows and weights
  static constexpr int RED = 2 * (kSets - 1) * (T / 4) * 512;               // twice the sets' sums of a quarter of the token rows
  static constexpr int NX = T <= 16 ? 9 : T <= 32 ? 6 : T <= 48 ? 4 : 3, NW = T <= 16 ? 7 : T <= 32 ? 6 : T <= 48 ? 5 : 4;
  static constexpr int OFF_RAW = NX * XB, OFF_RED = OFF_RAW + NW * WB, OFF_BAR = OFF_RED + RED;
  static constexpr int BARS = (2 * NW + 2 * NX + kSets) * 8 + 16;
  static constexpr int SMEM = 1024 + OFF_BAR + (BARS + 15) / 16 * 16 + 64 * 16;
};

__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void set_sync(int set) { asm volatile("bar.sync %0, 128;" ::"r"(2 + set) : "memory"); }

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
  const uint32_t dfull0 = xempty0 + 8 * C::NX, misc = dfull0 + 8 * kSets;      // misc: TMEM address, "last" flag
  const uint32_t ss0 = bars + (C::BARS + 15) / 16 * 16;                        // [64][4] sums of squares of the fold
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int items = p.nb * p.S;

  if (tid == 0) {
    for (int i = 0; i < C::NW; ++i) {
      mbar_init(wfull0 + 8 * i, 1);
      mbar_init(wempty0 + 8 * i, 4 * kSets);     // every worker warp has read its block
    }
    for (int i = 0; i < C::NX; ++i) {
      mbar_init(xfull0 + 8 * i, 1);
      mbar_init(xempty0 + 8 * i, kSets);         // every set's MMAs have read the token rows
    }
    for (int i = 0; i < kSets; ++i) mbar_init(dfull0 + 8 * i, 1);
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

  if (warp >= 16) {
    // ---------------------------------------------------------------- copies
    if (lane == 0) {
      const bool wt = warp == 16;
      const int n = wt ? C::NW : C::NX, unit = wt ? kBlockBytes : T * 128;
      const uint32_t full0 = wt ? wfull0 : xfull0, empty0 = wt ? wempty0 : xempty0, dst0 = wt ? raw0 : xs0;
      const uint32_t stage = kSets * unit;
      if (!wt) pdl_wait();       // the weights depend on nothing: their first stages are asked for before the previous kernel is done
      int slot = 0, round = 0;   // stage of the ring, times it was filled before
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int nblk = item / p.S, g0 = (item - nblk * p.S) * p.gps;
        int left = min(p.KG, g0 + p.gps) - g0;
        const uint8_t* src = wt ? p.w + ((size_t)nblk * p.KG + g0) * kBlockBytes : p.x + (size_t)g0 * (T * 128);
        for (; left > 0; left -= kSets, src += stage) {
          if (round > 0) ok = mbar_wait(empty0 + 8 * slot, (round - 1) & 1, ERR_GEMM_EMPTY_WAIT);
          if (!ok) break;
          const uint32_t bytes = min(left, kSets) * unit, bar = full0 + 8 * slot;
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
  } else {
    // ---------------------------------------------------------------- workers
    const int set = warp >> 2, q = warp & 3;
    const uint32_t my_tmem = tmem + set * 128 + ((uint32_t)(32 * q) << 16), dfull = dfull0 + 8 * set;
    const int row = 32 * q + lane;
    const uint32_t v_off = set * kBlockBytes + 2 * q * 512 + lane * 16;
    const uint32_t sc_off = set * kBlockBytes + 4096 + ((row >> 4) * 16 + 2 * (row & 7) + ((row >> 3) & 1)) * 2;
    constexpr uint32_t idesc = make_idesc(1, 1, 128, T);
    const uint64_t xdesc = make_desc_sw128(xs0 + set * T * 128);
    const uint32_t xd_lo = (uint32_t)xdesc, xd_hi = (uint32_t)(xdesc >> 32);
    pdl_wait();
    pdl_launch_dependents();
    int ws = 0, wp = 0, xs = 0, xp = 0;     // ring stages and their parities
    int done = 0, read = 0;                 // blocks of this set expanded, accumulators read
    bool ok = true;
    float next_scale = 0.f;
    // this set's block of the next weight stage into its A buffer; `has`: there is one
    const auto expand = [&](bool has) {
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(wfull0 + 8 * ws, wp, ERR_GEMM_FULL_WAIT));
      const uint32_t st = raw0 + ws * C::WB, empty = wempty0 + 8 * ws;
      if (++ws == C::NW) { ws = 0; wp ^= 1; }
      if (!ok) return;
      if (!has) {
        if (lane == 0) mbar_arrive(empty);
        return;
      }
      uint4 v[2];
#pragma unroll
      for (int j = 0; j < 2; ++j)
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[j].x), "=r"(v[j].y), "=r"(v[j].z), "=r"(v[j].w) : "r"(st + v_off + j * 512));
      unsigned short h;
      asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(st + sc_off));
      next_scale = __half2float(__ushort_as_half(h));
      __syncwarp();
      if (lane == 0) mbar_arrive(empty);
      const uint32_t a = my_tmem + (done & 1) * 32;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        uint32_t r[16];
        // column 4 i + t, i = 4 (32-k step) + 2 (low or high byte of a pair) + (nibble): k = 32 ks + 16 hi + 4 t + o + 2 e
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) r[2 * i + hf] = nibbles_bf16(w[2 * (i >> 2) + hf], 8 * ((i >> 1) & 1) + 4 * (i & 1));
        B2_TMEM_ST_16X128_8(a + ((uint32_t)(16 * j) << 16), r);
      }
      tmem_st_wait();
      ++done;
    };
    // the MMAs of the block that was expanded last, by the set's first lane once all four warps have stored it
    const auto multiply = [&](bool has) {
      tc_fence_before();
      set_sync(set);
      if (q == 0) {
        if (ok && lane == 0) {
          tc_fence_after();
          const bool got = mbar_wait(xfull0 + 8 * xs, xp, ERR_GEMM_FULL_WAIT);
          if (got && has) {
            const uint32_t am = tmem + set * 128 + ((done - 1) & 1) * 32, dm = tmem + set * 128 + 64, lo = xd_lo + xs * (C::XB >> 4);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_f16_ts_w(dm, am + 8 * k, lo + 2 * k, xd_hi, idesc, k != 0);    // 16 k = 32 bytes a step
            tc_commit(dfull);
          } else if (got) {
            mbar_arrive(xempty0 + 8 * xs);
          }
        }
        __syncwarp();
      }
      if (++xs == C::NX) { xs = 0; xp ^= 1; }
    };
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int nblk = item / p.S, split = item - nblk * p.S;
      const int ng = min(p.KG, (split + 1) * p.gps) - split * p.gps, ns = (ng + kSets - 1) / kSets;
      const auto has = [&](int k) { return k * kSets + set < ng; };
      float acc[T];
#pragma unroll
      for (int i = 0; i < T; ++i) acc[i] = 0.f;
      expand(has(0));
      multiply(has(0));
      for (int k = 0; k < ns; ++k) {
        const float scale = next_scale;
        if (k + 1 < ns) expand(has(k + 1));
        if (has(k)) {
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(dfull, read & 1, ERR_GEMM_TMEM_FULL_WAIT));
          if (ok && q == 0 && lane == 0) mbar_arrive(xempty0 + 8 * (xs == 0 ? C::NX - 1 : xs - 1));    // the MMAs have read the token rows
          ++read;
          if (ok) {
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < T; c0 += 16) {
              uint32_t d[16];
              B2_TMEM_LD_16(my_tmem + 64 + c0, d);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) acc[c0 + i] = fmaf(scale, __uint_as_float(d[i]), acc[c0 + i]);
            }
          }
        }
        if (k + 1 < ns) multiply(has(k + 1));
      }
      // ---- the sets' sums, a quarter of the token rows at a time: set h takes quarter h from the others' buffers, in set order
      constexpr int Q = T / 4;
      const uint32_t col = red0 + (uint32_t)row * 4;
      const int n = nblk * 128 + row;
#pragma unroll
      for (int h = 0; h < kSets; ++h) {
        const uint32_t buf = col + (h & 1) * ((kSets - 1) * Q * 512);      // two rounds' buffers in turn
        if (set != h) {
#pragma unroll
          for (int i = 0; i < Q; ++i) asm volatile("st.shared.f32 [%0], %1;" ::"r"(buf + ((set < h ? set : set - 1) * Q + i) * 512), "f"(acc[h * Q + i]) : "memory");
        }
        workers_sync();
        if (set == h) {
          float* o = p.out + ((size_t)split * p.M + h * Q) * p.N + n;
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < kSets; ++j) {
              float v = acc[h * Q + i];
              if (j != h) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(buf + ((j < h ? j : j - 1) * Q + i) * 512));
              sum = j ? sum + v : v;
            }
            if (h * Q + i < p.M && n < p.N) o[(size_t)i * p.N] = sum;
          }
        }
      }
      if (p.fold_tickets == nullptr) continue;
      // ---- the last split of an n-block adds the slices in split order to the residual rows and leaves the sums of squares of
      // its 128 columns (the arithmetic and order of the integer GEMV's fold).  Four rows are in flight per thread.
      __threadfence();
      workers_sync();
      if (tid == 0) {
        const int last = atomicAdd(&p.fold_tickets[nblk], 1) == p.S - 1;
        if (last) p.fold_tickets[nblk] = 0;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(misc + 4), "r"(last) : "memory");
      }
      workers_sync();
      int last;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(last) : "r"(misc + 4));
      if (!last) continue;
      __threadfence();
      const int c = tid & 127, rsub = tid >> 7, fn = nblk * 128 + c;     // four rows of 128 columns at a time
      for (int m0 = rsub; m0 < p.M; m0 += 16) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (m0 + 4 * u < p.M && fn < p.N) v[u] = __bfloat162float(p.fold_resid_in[(size_t)(m0 + 4 * u) * p.N + fn]);
#pragma unroll 4
        for (int sp = 0; sp < p.S; ++sp)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (m0 + 4 * u < p.M && fn < p.N) v[u] += __ldcg(p.out + ((size_t)sp * p.M + m0 + 4 * u) * p.N + fn);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int m = m0 + 4 * u;
          if (m >= p.M) break;
          const __nv_bfloat16 rb = __float2bfloat16(v[u]);
          if (fn < p.N) p.fold_resid_out[(size_t)m * p.N + fn] = rb;
          const float rf = fn < p.N ? __bfloat162float(rb) : 0.f;
          const float ss = warp_sum(rf * rf);
          if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(ss0 + (m * 4 + (c >> 5)) * 4), "f"(ss) : "memory");
        }
      }
      workers_sync();
      if (tid < p.M) {
        float4 q4;
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(q4.x), "=f"(q4.y), "=f"(q4.z), "=f"(q4.w) : "r"(ss0 + tid * 16));
        p.fold_ssq[(size_t)tid * p.nb + nblk] = ((q4.x + q4.y) + q4.z) + q4.w;
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

// ``x``: b2_stage_rows of the same M and K.  S <= 16 splits of whole fours of groups, none of them empty.
extern "C" int b2_gemm_w4_rows(const void* w4b, const void* x, float* out, int M, int N, int K, int S, int* fold_tickets,
                               const void* fold_resid_in, void* fold_resid_out, float* fold_ssq, void* stream) {
  if (M < 1 || M > 64 || N < 1 || K < 64 || K % 64 != 0 || S < 1 || S > kMaxSplits) return -1;
  if (((uintptr_t)w4b | (uintptr_t)x) & 15) return -4;
  RowsParams p;
  p.w = (const uint8_t*)w4b; p.x = (const uint8_t*)x; p.out = out;
  p.M = M; p.N = N; p.KG = K / 64; p.S = S; p.nb = (N + 127) / 128;
  p.gps = ((p.KG + S - 1) / S + kSets - 1) / kSets * kSets;    // whole stages
  if (p.gps * (S - 1) >= p.KG) return -2;                      // every split has groups
  p.fold_tickets = fold_tickets; p.fold_resid_in = (const __nv_bfloat16*)fold_resid_in;
  p.fold_resid_out = (__nv_bfloat16*)fold_resid_out; p.fold_ssq = fold_ssq;
  cudaStream_t st = (cudaStream_t)stream;
  if (M <= 16) return launch_rows<16>(p, st);
  if (M <= 32) return launch_rows<32>(p, st);
  if (M <= 48) return launch_rows<48>(p, st);
  return launch_rows<64>(p, st);
}

B2_DEFINE_STATUS(gemmrows)
