// Prefill GEMMs on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a only.
//
//   C[M][N] = A[M][K] * B[N][K]^T        A, B K-major (row-major activations, row-major weights)
//
//   * bf16 x bf16 -> fp32 (kind::f16)            prefill linears on dequantised weights
//   * int8 x int8 -> int32 (kind::i8)            the int8 prompt pass: per-token activation scales and
//                                                per-row weight scales applied in the epilogue
//   * grouped form (MoE): the M dimension is a device-side table of expert row blocks, B is a
//     3-D tensor [E][N][K]; tile counts are read on the device so the host never syncs
//
// They replace the reference's pf_gemm / pf_gemm_small (src/kernels/prefill/pf_gemm.cl), its int8
// GEMM (pf_int8.cl: pf_gemm_i8) and the grouped expert GEMM (pf_moe_gemm.cl).
//
// Structure: one persistent CTA per SM, 192 threads, warp-specialised.
//   warp 0   TMA producer: cp.async.bulk.tensor 2-D/3-D tiles (128-byte swizzle) into a smem ring
//   warp 1   MMA issuer: one elected lane issues tcgen05.mma (M = 128, N = BN, K = 16 / 32) and
//            commits stage-free and accumulator-full mbarriers; owns the TMEM allocation
//   warps 2-5 epilogue: tcgen05.ld of the accumulator (two TMEM buffers, so the epilogue of tile i
//            overlaps the main loop of tile i + 1), scale / SiLU*up / residual add, global stores
// Tiles are walked M-fastest so CTAs that run together share one weight tile in L2.
//
// W4 form (template parameter W4): B is never materialised in global memory.  The producer fetches the W4B blocks of
// a stage (4352 bytes per 128 rows x 64 k: nibbles + fp16 group scales) with bulk copies; sixteen more warps expand them
// to bf16 -- bf16_rne((q - 8) * scale), the same rounding as the dequantising pass -- straight into the stage's
// B tile in the 128-byte-swizzled K-major layout the MMA descriptors expect, fence the generic stores against the
// async proxy and complete the stage's barrier.  The weights cross HBM as int4 (a quarter of the bf16 bytes), once per row of
// tiles; chunks of several rows of tiles expand a weight once with dequant_w4b_kernel instead, into a workspace of the largest matrix, and
// experts of a whole tile of rows and more read such copies.  The role of the reference's direct-int4 GEMMs
// (src/kernels/prefill/pf_gemm_q4.cl, src/kernels/prefill/pf_moe_q4gemm.cl:1-40).  The blocks have a ring of their own,
// filled by a warp of its own, and so have the tiles of A: tied to the tiles of B, every trip from HBM was part of the loop.
// 2048 rows over 256 experts (64 rows each), gate||up 1024 x 2048 / down 2048 x 512, us: 186 / 102 -> 145 / 87 with A apart, tiles of eight blocks together, no rows fetched beyond
// a block's last, and groups of expanding warps on alternate k blocks.
#include "common.cuh"
#include "wire.cuh"

#include <map>
#include <mutex>
#include <tuple>

using namespace b2;

namespace {

constexpr int BM = 128;
constexpr int BKB = 128;  // bytes of K per stage row (64 bf16 or 128 int8)
constexpr int kThreads = 192;
constexpr int kGroupRun = 8;    // grouped form: blocks whose tiles run together
constexpr int kGroupBox = 32;   // grouped form: rows of a copy of A; a block's rows beyond its last such box are not fetched, four boxes are one copy (map_part: the
                                // boxes; in four copies 8 x 256 rows of 4096 x 14336 took 231 us, in one 218)

enum Epi : int { EPI_BF16 = 0, EPI_F32 = 1, EPI_SILU_MUL = 2, EPI_RESID_ADD = 3, EPI_RS_PUSH = 4, EPI_EP_RETURN = 5, EPI_GLU = 6, EPI_RELU2 = 7 };

struct GemmParams {
  int M, N, K;       // K in elements
  int ldc;           // leading dimension of C (elements)
  void* C;
  const __nv_bfloat16* resid;  // EPI_RESID_ADD: [M][ldc]
  const float* a_scale;        // int8: per row of A
  const float* b_scale;        // int8: per row of B ([E][N] in the grouped form)
  int epi;
  // grouped form
  const int* blk_expert;  // [n_blk]
  const int* blk_row0;    // [n_blk] first row of the block in A / C
  const int* blk_rows;    // [n_blk] valid rows (<= 128)
  const int* n_blk;       // device scalar
  int max_blk;
  // ---- tensor-parallel forms (see wire.cuh for the protocol)
  // EPI_RS_PUSH (row-parallel GEMM -> reduce-scatter): the bf16 tile of m-tile mt is stored into the
  // landing buffer of the rank that owns those rows, [source rank][rows_cap][N], and the owner's counter
  // [source rank][m-tile of the owner] gets one increment per epilogue warp and n-tile.
  const unsigned long long* rs_table;  // [2][kMaxRanks]: landing, counters of every rank
  int rs_rank, rs_world;
  int rs_tpr;       // m-tiles per owner (rows_cap = 128 rs_tpr)
  int mt_rot;       // m-tile walk starts here, so ranks do not all push to one owner at a time
  // all-gather -> GEMM: the producer waits until m-tile mt of A (pushed into this GPU's memory by the
  // owners of those rows) has ag_expect arrivals
  const int* ag_cnt;
  int ag_expect;
  // ---- expert-parallel forms (grouped mode)
  // dispatch -> grouped GEMM: block i of the expert-sorted rows is loaded once blk_wait[i] (arrivals counted
  // by the source ranks' dispatch kernels) has reached the block's row count.
  const int* blk_wait;
  // EPI_EP_RETURN (grouped GEMM -> combine): row r of the sorted buffer belongs to slot (row_src[r] & 0xffffff)
  // of source rank (row_src[r] >> 24); its bf16 result row is stored into that rank's return buffer
  // ret_table[rank][slot][N] over NVLink, where the source adds its tokens' slots in slot order.
  const int* row_src;
  const unsigned long long* ret_table;
  // ---- W4 form: B as W4B blocks [expert][ceil(N / 128)][K / 64][4352 bytes]
  const uint8_t* w4;
  long long w4_expert_bytes;
  Glu glu;           // EPI_GLU: SiLU(gate) * up with other constants
  // ---- pair form: the tiles of the last, partly filled wave cut along K into `split` parts each
  int split;         // 0 or 1: not
  float* part;       // [tile of that wave][part][CTA][chunk of 32 columns][warp][8][lane] float4
  int* part_tickets; // [tile of that wave][CTA][warp][half of the columns], zeroed, left zero
};

constexpr int kW4Block = 4352;     // one W4B block: 128 rows x 64 k of nibbles (4096 B) + 128 fp16 scales
constexpr int kDequantWarps = 16;  // W4 form: warps that expand the blocks into the B tile

// The expanding warps are four groups on alternate k blocks: a k block's chain (wait, load, expand, store, fence, hand over) is longer than its share of any
// pipe, and with all warps on every k block it was the loop (256 experts of 64 rows, 1024 x 2048, us: one group 175, two 164, four 157).
constexpr int kDequantGroups = 4, kGroupWarps = kDequantWarps / kDequantGroups;

template <int BN, bool W4 = false>
struct Cfg {
  static constexpr int A_BYTES = BM * BKB;
  static constexpr int B_BYTES = BN * BKB;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int RAW = W4 ? (BN / 128) * kW4Block : 0;   // a k block's W4B blocks
  static constexpr int STAGES = W4 ? ((BN == 256) ? 4 : 5) : ((BN == 256) ? 4 : 6);
  static constexpr int ASTAGES = W4 ? ((BN == 256) ? 3 : 6) : 0;   // W4: tiles of A, a ring of their own too
  static constexpr int RAWS = W4 ? ((BN == 256) ? 4 : 10) : 0; // k blocks of the ring of W4B blocks
  static_assert(!W4 || (STAGES >= kDequantGroups && RAWS >= kDequantGroups));   // else a group could meet a barrier two phases behind: the parity lies
  static constexpr int PUSH_STAGE = W4 ? 0 : 4 * 32 * 144;  // per epilogue warp: 32 rows x (128 B + 16 B pad) for coalesced peer stores
  static constexpr int BARS = 512;
  static constexpr int TILES = W4 ? STAGES * B_BYTES + ASTAGES * A_BYTES : STAGES * STAGE;
  static constexpr int SMEM = TILES + 1024 /*align*/ + BARS + PUSH_STAGE + RAWS * RAW;
  static constexpr int TMEM_COLS = 2 * BN;  // two accumulators
  static constexpr int THREADS = kThreads + (W4 ? (kDequantWarps + 1) * 32 : 0);
};

// 32 accumulators of one row, columns n0 .. n0 + 31, through the epilogue into C
__device__ __forceinline__ void store_chunk(const GemmParams& p, const uint32_t (&v)[32], int grow, int n0) {
  float f[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
  if (p.epi == EPI_SILU_MUL || p.epi == EPI_GLU) {
    // columns alternate 16 gate, 16 up: 16 outputs per 32 accumulator columns
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)grow * p.ldc + (n0 >> 1);
    uint32_t o[8];
    if (p.epi == EPI_GLU && p.glu.bias) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(p.glu.bias + n0) + j);
        f[4 * j] += b.x; f[4 * j + 1] += b.y; f[4 * j + 2] += b.z; f[4 * j + 3] += b.w;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      o[j] = p.epi == EPI_GLU ? pack_bf16(glu(p.glu, f[2 * j], f[16 + 2 * j]), glu(p.glu, f[2 * j + 1], f[17 + 2 * j]))
                              : pack_bf16(silu(f[2 * j]) * f[16 + 2 * j], silu(f[2 * j + 1]) * f[17 + 2 * j]);
    *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint4*>(dst + 8) = make_uint4(o[4], o[5], o[6], o[7]);
  } else if (p.epi == EPI_F32) {
    float* dst = reinterpret_cast<float*>(p.C) + (size_t)grow * p.ldc + n0;
    if (n0 + 32 <= p.N) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float4*>(dst + 4 * j) = make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
    } else {
      for (int j = 0; j < 32 && n0 + j < p.N; ++j) dst[j] = f[j];
    }
  } else {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)grow * p.ldc + n0;
    if (p.epi == EPI_RESID_ADD) {
      const __nv_bfloat16* rs = p.resid + (size_t)grow * p.ldc + n0;
      if (n0 + 32 <= p.N) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 rv = *reinterpret_cast<const uint4*>(rs + 8 * j);
          const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            f[8 * j + 2 * q] += bf16_lo(rw[q]);
            f[8 * j + 2 * q + 1] += bf16_hi(rw[q]);
          }
        }
      } else {
        for (int j = 0; j < 32 && n0 + j < p.N; ++j) f[j] += __bfloat162float(rs[j]);
      }
    }
    if (p.epi == EPI_RELU2) {
#pragma unroll
      for (int j = 0; j < 32; ++j) f[j] = relu2(f[j]);
    }
    if (n0 + 32 <= p.N) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(dst + 8 * j) =
            make_uint4(pack_bf16(f[8 * j], f[8 * j + 1]), pack_bf16(f[8 * j + 2], f[8 * j + 3]),
                       pack_bf16(f[8 * j + 4], f[8 * j + 5]), pack_bf16(f[8 * j + 6], f[8 * j + 7]));
    } else {
      for (int j = 0; j < 32 && n0 + j < p.N; ++j) dst[j] = __float2bfloat16(f[j]);
    }
  }
}

// A weight's scale, times 64, as two bf16 of five significant bits whose sum it is (an fp16 has eleven: the rest behind the first five is
// at most half a unit of them, so five bits or a power of two), each in both halves of a word.  One that is not finite stays as it is: the carry of
// the rounding would make a NaN zero.
__device__ __forceinline__ void split_scale(float s, uint32_t& hi, uint32_t& lo) {
  s *= 64.f;
  const bool finite = fabsf(s) < __int_as_float(0x7f800000);
  const uint32_t h = finite ? (__float_as_uint(s) + 0x00040000u) & 0xFFF80000u : __float_as_uint(s);
  hi = __byte_perm(h, 0, 0x3232);
  lo = __byte_perm(__float_as_uint(finite ? s - __uint_as_float(h) : 0.f), 0, 0x3232);
}

// Vector `u` of a stage's W4B blocks (256 vectors a block) -> sixteen 8-byte pieces of the bf16 B tile.  A vector holds rows g and
// g + 8 of a 16-row tile, 64 k: low nibbles are k 4t..4t+3 of a 32-k step, high nibbles k + 16 (the operand order of the decode
// GEMV); row r lies at r * 128 bytes, 16-byte chunk (k / 8) XOR (r mod 8) -- the 128-byte swizzle.
// Two bytes of a word go into the halves of a register, where each nibble already is a bf16 (up to 255 the bits are an integer times
// 2^-133, denormal or not); a fused multiply-add makes it (q - 8) / 64, and with the scale in two exact parts v s_lo is exact and
// v s_hi + v s_lo is rounded once: bf16_rne((q - 8) * scale), packed all the way.
__device__ __forceinline__ void expand_w4(int u, uint32_t raw, uint32_t sb) {
  const int b = u >> 8, v = u & 255, j = v >> 5, l = v & 31, g = l >> 2, tq = l & 3;
  uint4 wv;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(wv.x), "=r"(wv.y), "=r"(wv.z), "=r"(wv.w)
               : "r"(raw + b * kW4Block + v * 16));
  uint32_t sc2;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc2) : "r"(raw + b * kW4Block + 4096 + (j * 16 + 2 * g) * 2));
  const __half2 sh = *reinterpret_cast<const __half2*>(&sc2);
  uint32_t s1[2], s2[2];
  split_scale(__low2float(sh), s1[0], s2[0]);
  split_scale(__high2float(sh), s1[1], s2[1]);
  // A store instruction of 16 lanes covers four rows, 32 bytes each; in the order of the k they would meet in two of the row's four
  // 32-byte banks groups.  A lane starts with another 32-k step and nibble, by its row: all four are used.
  const int turn = (g >> 1) ^ (g & 3);
  const uint32_t wa[4] = {turn & 2 ? wv.z : wv.x, turn & 2 ? wv.w : wv.y, turn & 2 ? wv.x : wv.z, turn & 2 ? wv.y : wv.w};
  const uint32_t mask0 = turn & 1 ? 0x00F000F0u : 0x000F000Fu, mul0 = turn & 1 ? 0x7d007d00u : 0x7f007f00u;      // 2^123 or 2^127
  const uint32_t dst0 = sb + (b * 128 + j * 16 + g) * 128 + (((tq >> 1) ^ g ^ (2 * turn)) << 4) + (tq & 1) * 8;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint32_t w01 = __byte_perm(wa[c], 0, 0x4140), w23 = __byte_perm(wa[c], 0, 0x4342);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint32_t mask = e ? mask0 ^ 0x00FF00FFu : mask0, mul = e ? mul0 ^ 0x02000200u : mul0;
      uint32_t p[2] = {w01 & mask, w23 & mask};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t t;
        asm("fma.rn.bf16x2 %0, %0, %1, %2;" : "+r"(p[i]) : "r"(mul), "r"(0xbe00be00u));      // -1/8
        asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(t) : "r"(p[i]), "r"(s2[c & 1]));
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(p[i]) : "r"(p[i]), "r"(s1[c & 1]), "r"(t));
      }
      const uint32_t dst = (dst0 ^ (uint32_t)((4 * (c >> 1) + 2 * e) << 4)) + (c & 1) * 1024;
      asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst), "r"(p[0]), "r"(p[1]) : "memory");
    }
  }
}

template <int BN, bool I8, bool W4 = false>
__global__ void __launch_bounds__(Cfg<BN, W4>::THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_part,
               const GemmParams p) {
  using C = Cfg<BN, W4>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::TILES);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + C::STAGES);
  const uint32_t tfull0 = smem_u32(bars + 2 * C::STAGES), tempty0 = smem_u32(bars + 2 * C::STAGES + 2);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::STAGES + 4);
  const uint32_t rawfull0 = smem_u32(bars + 2 * C::STAGES + 6), rawempty0 = rawfull0 + 8 * C::RAWS;   // W4 form: ring of W4B blocks
  const uint32_t afull0 = rawempty0 + 8 * C::RAWS, aempty0 = afull0 + 8 * C::ASTAGES;                                         // and of tiles of A
  const uint32_t smem_base = smem_u32(smem), a_base = smem_base + C::STAGES * C::B_BYTES;
  const uint32_t push_base = smem_base + C::TILES + C::BARS;
  const uint32_t raw_base = push_base + C::PUSH_STAGE;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool grouped = p.blk_expert != nullptr;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int tiles_m = grouped ? min(*p.n_blk, p.max_blk) : (p.M + BM - 1) / BM;
  const int n_tiles = tiles_m * tiles_n;
  // Dense: tiles that run together share weights.  Grouped: the columns of eight blocks of rows run together, which share both the rows and, where an expert has
  // several blocks, its weights.  With all blocks innermost, 256 blocks of 4 KB rows (134 MB with their padding) came from HBM again for every column of tiles;
  // with the columns of one block innermost, so did the weights of an expert of 1024 rows for every block.  us, all blocks / columns of one / of eight, bf16:
  // 256 experts x 64 rows, 1024 x 2048 251 / 179 / 181; 8 x 1024, 28672 x 4096 1575 / 1926 / 1397; 1 x 8192, 16384 x 8192 1655 / 2035 / 1566 (four blocks
  // 1767, sixteen 1647, both before whole blocks were one copy).
  const auto at_of = [&](int t, int& mt, int& nt) {
    if (grouped) {
      const int run = t / (kGroupRun * tiles_n), first = run * kGroupRun, n = min(kGroupRun, tiles_m - first), i = t - first * tiles_n;
      mt = first + i % n;
      nt = i / n;
    } else {
      mt = (t % tiles_m + p.mt_rot) % tiles_m;
      nt = t / tiles_m;
    }
  };
  const int KB = (p.K * (I8 ? 1 : 2) + BKB - 1) / BKB;  // k blocks

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(full0 + 8 * i, W4 ? kGroupWarps : 1);
      mbar_init(empty0 + 8 * i, 1);
    }
    for (int i = 0; i < C::ASTAGES; ++i) {
      mbar_init(afull0 + 8 * i, 1);
      mbar_init(aempty0 + 8 * i, 1);
    }
    for (int i = 0; i < C::RAWS; ++i) {
      mbar_init(rawfull0 + 8 * i, 1);
      mbar_init(rawempty0 + 8 * i, kGroupWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tfull0 + 8 * i, 1);
      mbar_init(tempty0 + 8 * i, 4);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tmap(&map_a);
      prefetch_tmap(&map_b);
      if (grouped) prefetch_tmap(&map_part);
      int it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        int mt, nt;
        at_of(t, mt, nt);
        int row0 = mt * BM, expert = 0, boxes = BM / kGroupBox;
        if (grouped) {
          row0 = p.blk_row0[mt];
          expert = p.blk_expert[mt];
          boxes = (min(BM, max(1, p.blk_rows[mt])) + kGroupBox - 1) / kGroupBox;
        }
        if (p.ag_cnt) {
          // rows of this m-tile arrive from their owner rank: bounded wait on the tile's counter in this
          // GPU's own memory, then order the generic-proxy acquire before the async-proxy (TMA) reads
          ok = wire_wait(p.ag_cnt + mt, p.ag_expect, (unsigned)(0x20000000u | mt));
          if (!ok) break;
          asm volatile("fence.proxy.async;" ::: "memory");
        }
        if (p.blk_wait) {
          ok = wire_wait(p.blk_wait + mt, p.blk_rows[mt], (unsigned)(0x28000000u | mt));
          if (!ok) break;
          asm volatile("fence.proxy.async;" ::: "memory");
        }
        // W4: A alone; the last warp copies the weights' blocks, other warps expand them
        constexpr int S = W4 ? C::ASTAGES : C::STAGES;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S;
          const uint32_t full = (W4 ? afull0 : full0) + 8 * s;
          if (it >= S) ok = mbar_wait_lone((W4 ? aempty0 : empty0) + 8 * s, ((it / S) - 1) & 1, ERR_GEMM_EMPTY_WAIT);
          if (!ok) break;
          const uint32_t sa = W4 ? a_base + s * C::A_BYTES : smem_base + s * C::STAGE, sb = sa + C::A_BYTES;
          const int kx = kb * (I8 ? BKB : BKB / 2);
          mbar_expect_tx(full, (W4 ? 0 : C::B_BYTES) + boxes * kGroupBox * BKB);
          if (boxes == BM / kGroupBox) tma_load_2d(sa, &map_a, kx, row0, full);
          else
            for (int i = 0; i < boxes; ++i) tma_load_2d(sa + i * kGroupBox * BKB, &map_part, kx, row0 + i * kGroupBox, full);
          if (!W4) {
            if (grouped) tma_load_3d(sb, &map_b, kx, nt * BN, expert, full);
            else tma_load_2d(sb, &map_b, kx, nt * BN, full);
          }
        }
      }
      if (!ok) {  // drain what was issued and may never be consumed
        constexpr int S = W4 ? C::ASTAGES : C::STAGES;
        for (int i = max(0, it - S); i < it; ++i) mbar_wait((W4 ? afull0 : full0) + 8 * (i % S), (i / S) & 1, ERR_GEMM_FULL_WAIT);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = I8 ? make_idesc(2, 1, BM, BN) : make_idesc(1, 1, BM, BN);
      int it = 0, lt = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++lt) {
        const int a = lt & 1;
        if (lt >= 2) ok = mbar_wait_lone(tempty0 + 8 * a, ((lt >> 1) - 1) & 1, ERR_GEMM_TMEM_EMPTY_WAIT);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + a * BN;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % C::STAGES;
          constexpr int AS = W4 ? C::ASTAGES : 1;
          const int as = it % AS;
          ok = mbar_wait_lone(full0 + 8 * s, (it / C::STAGES) & 1, ERR_GEMM_FULL_WAIT) &&
               (!W4 || mbar_wait_lone(afull0 + 8 * as, (it / AS) & 1, ERR_GEMM_FULL_WAIT));
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = W4 ? a_base + as * C::A_BYTES : smem_base + s * C::STAGE, sb = W4 ? smem_base + s * C::B_BYTES : sa + C::A_BYTES;
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // 4 x 32 bytes of K per stage
            const uint64_t da = make_desc_sw128(sa + k * 32), db = make_desc_sw128(sb + k * 32);
            if (I8) umma_i8(d_tmem, da, db, idesc, (kb | k) != 0);
            else umma_f16(d_tmem, da, db, idesc, (kb | k) != 0);
          }
          if (W4) tc_commit(aempty0 + 8 * as);
          tc_commit(empty0 + 8 * s);  // stage is free once these MMAs have read it
        }
        if (ok) tc_commit(tfull0 + 8 * a);
      }
    }
  } else if (W4 && warp == 6 + kDequantWarps) {
    // ------------------------------------------------------------ W4 blocks: a ring of their own, several k blocks ahead of the tiles
    if (lane == 0) {
      int slot = 0, round = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        int mt, nt;
        at_of(t, mt, nt);
        const int expert = grouped ? p.blk_expert[mt] : 0;
        const int nb0 = nt * (BN / 128), nblk = min(BN / 128, (p.N + 127) / 128 - nb0);
        const uint8_t* src = p.w4 + (size_t)expert * p.w4_expert_bytes + (size_t)nb0 * KB * kW4Block;
        for (int kb = 0; kb < KB; ++kb, src += kW4Block) {
          if (round > 0) ok = mbar_wait_lone(rawempty0 + 8 * slot, (round - 1) & 1, ERR_GEMM_EMPTY_WAIT);
          if (!ok) break;
          mbar_expect_tx(rawfull0 + 8 * slot, (uint32_t)nblk * kW4Block);
          for (int b = 0; b < nblk; ++b)
            bulk_g2s(raw_base + slot * C::RAW + b * kW4Block, src + (size_t)b * KB * kW4Block, kW4Block, rawfull0 + 8 * slot);
          if (++slot == C::RAWS) { slot = 0; ++round; }
        }
      }
      if (!ok)   // wait (bounded) for the copies that were issued and possibly never consumed
        for (int i = 0; i < C::RAWS; ++i) {
          const int r = i < slot ? round : round - 1;
          if (r >= 0) mbar_wait(rawfull0 + 8 * i, r & 1, ERR_GEMM_FULL_WAIT);
        }
    }
  } else if (W4 && warp >= 6) {
    // ------------------------------------------------------------ W4 expansion (warps 6 .. 6 + kDequantWarps - 1)
    const int grp = (warp - 6) / kGroupWarps, dt = threadIdx.x - 6 * 32 - grp * kGroupWarps * 32;
    int it = 0, slot = 0, par = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
      int mt, nt;
      at_of(t, mt, nt);
      const int nb_total = (p.N + 127) / 128, nb0 = nt * (BN / 128);
      const int nblk = min(BN / 128, nb_total - nb0);
      for (int kb = 0; kb < KB; ++kb, ++it) {
        if (it % kDequantGroups != grp) {      // the other groups'
          if (++slot == C::RAWS) { slot = 0; par ^= 1; }
          continue;
        }
        const int s = it % C::STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(rawfull0 + 8 * slot, par, ERR_GEMM_FULL_WAIT));
        // the tile's last products are done
        if (ok && it >= C::STAGES) ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ((it / C::STAGES) - 1) & 1, ERR_GEMM_EMPTY_WAIT));
        if (!ok) break;
        const uint32_t sb = smem_base + s * C::B_BYTES, raw = raw_base + slot * C::RAW;
        for (int u = dt; u < nblk * 256; u += kGroupWarps * 32) expand_w4(u, raw, sb);
        fence_proxy_async_smem();   // the MMA reads the tile through the async proxy
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(full0 + 8 * s);
          mbar_arrive(rawempty0 + 8 * slot);
        }
        if (++slot == C::RAWS) { slot = 0; par ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    const int quarter = warp & 3;  // TMEM lane quarter this warp may read
    int lt = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++lt) {
      const int a = lt & 1;
      int mt, nt;
      at_of(t, mt, nt);
      int row0 = mt * BM, rows = min(BM, p.M - row0), expert = 0;
      if (grouped) {
        row0 = p.blk_row0[mt];
        rows = p.blk_rows[mt];
        expert = p.blk_expert[mt];
      }
      ok = mbar_wait(tfull0 + 8 * a, (lt >> 1) & 1, ERR_GEMM_TMEM_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      const int r = quarter * 32 + lane;  // row inside the tile
      const int grow = row0 + r;
      const bool row_ok = r < rows;
      float asc = 1.f;
      if (I8 && row_ok) asc = p.a_scale[grow];
      const float* bsc = I8 ? p.b_scale + (size_t)expert * p.N : nullptr;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t v[32];
        const uint32_t taddr = tmem_base + a * BN + c * 32 + ((uint32_t)(quarter * 32) << 16);
        B2_TMEM_LD_32(taddr, v);
        tmem_ld_wait();
        const int n0 = nt * BN + c * 32;
        if (I8) {  // integer accumulators -> scaled floats, once, for every epilogue form
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint((float)(int)v[j] * asc * bsc[min(n0 + j, p.N - 1)]);
        }
        if (p.epi == EPI_RS_PUSH || p.epi == EPI_EP_RETURN) {
          // bf16 row piece -> this warp's staging tile; every second chunk the warp copies 32 rows x 128 B
          // to the owner's landing buffer as whole 128-byte lines (coalesced stores cross NVLink far better
          // than one row per thread)
          const uint32_t stg = push_base + (uint32_t)quarter * (32 * 144);
          const uint32_t mine = stg + lane * 144 + (c & 1) * 64;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(mine + 16 * j),
                         "r"(pack_bf16(__uint_as_float(v[8 * j]), __uint_as_float(v[8 * j + 1]))),
                         "r"(pack_bf16(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]))),
                         "r"(pack_bf16(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]))),
                         "r"(pack_bf16(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7])))
                         : "memory");
          if ((c & 1) && p.epi == EPI_EP_RETURN) {
            __syncwarp();
            if (n0 - 32 < p.N) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int rw = i * 4 + (lane >> 3), piece = lane & 7;
                uint4 q;
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                             : "r"(stg + rw * 144 + piece * 16));
                if (quarter * 32 + rw < rows) {
                  const int meta = p.row_src[row0 + quarter * 32 + rw];
                  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.ret_table[meta >> 24]) +
                                       (size_t)(meta & 0xffffff) * p.N + (n0 - 32) + piece * 8;
                  *reinterpret_cast<uint4*>(dst) = q;
                }
              }
            }
            __syncwarp();
          } else if (c & 1) {
            __syncwarp();
            const int owner = mt / p.rs_tpr, mtl = mt - owner * p.rs_tpr;
            __nv_bfloat16* land = reinterpret_cast<__nv_bfloat16*>(p.rs_table[owner]) +
                                  ((size_t)p.rs_rank * p.rs_tpr * BM + (size_t)mtl * BM + quarter * 32) * p.N + (n0 - 32);
            if (n0 - 32 < p.N) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int rw = i * 4 + (lane >> 3), piece = lane & 7;
                uint4 q;
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                             : "r"(stg + rw * 144 + piece * 16));
                if (quarter * 32 + rw < rows) *reinterpret_cast<uint4*>(land + (size_t)rw * p.N + piece * 8) = q;
              }
            }
            __syncwarp();
          }
        } else if (row_ok && n0 < p.N) {
          store_chunk(p, v, grow, n0);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty0 + 8 * a);
      if (p.epi == EPI_RS_PUSH) {
        // this warp's part of the tile is on its way: make it visible system-wide, then count one arrival
        // at the owner (4 epilogue warps x tiles_n arrivals complete an m-tile of one source rank)
        __syncwarp();   // the warp's stores are ordered before lane 0's fence and release
        if (lane == 0) {
          const int owner = mt / p.rs_tpr, mtl = mt - owner * p.rs_tpr;
          int* cnt = reinterpret_cast<int*>(p.rs_table[kMaxRanks + owner]) + p.rs_rank * p.rs_tpr + mtl;
          __threadfence_system();
          asm volatile("red.release.sys.global.add.s32 [%0], 1;" ::"l"(cnt) : "memory");
        }
      }
    }
  }

  // ---- teardown: every thread arrives here on every path, then the owner frees the TMEM
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// ------------------------------------------------------------------ two SMs on one tile (cta_group::2)
// A cluster of two CTAs computes 256 x 256 tiles: each holds 128 rows of A and 128 of the 256 rows of B in its shared memory and
// 128 rows of the accumulator in its tensor memory; the even CTA issues the MMAs for both.  Per k block a CTA then fetches,
// stores and reads 16 KB of B instead of 32: six stages fit instead of four, and the tensor core's operand reads fall from 96 to
// 64 bytes a cycle.  bf16 GEMMs that are not grouped, with the local epilogues; the loads carry no multicast.
// 4096 rows x 34816 x 5120: 986 -> 908 us (1.61 PFLOP/s); x 5120 x 17408: 573 -> 504; 900 rows x 34816 x 5120: 272 -> 247.
//
// A last wave of a few tiles leaves most pairs idle for a whole tile's time (5120 columns at 900 rows: 80 tiles on 74 pairs).  Its tiles are cut along K, a
// part per pair: a warp leaves its fp32 sums of half the columns in a workspace, and whichever part comes last for them adds the parts in order and goes
// through the epilogue; every second part begins with the other half.  us without / with: 5120 x 17408,
// 130 rows 128 / 68, 900 260 / 161, 4096 506 / 474; 5120 x 5120, 900 rows 58 / 49; 7168 x 5120, 2048 rows 118 / 110.  (Counted for each 32 columns, the fences took
// what was gained: 5120 x 5120, 900 rows 58 / 55.)
struct PairCfg {
  static constexpr int BN = 256, HALF = 128 * BKB, STAGE = 2 * HALF, STAGES = 6, BARS = 256;
  static constexpr int SMEM = STAGES * STAGE + 1024 + BARS;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank0(uint32_t addr) {     // the even CTA's copy of a shared-memory word
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// mbar_wait for a barrier on which threads of the other CTA arrive
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, unsigned int code) {
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i) {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(bar), "r"(parity), "r"(kSuspendHintNs)
          : "memory");
      if (ok) return true;
    }
    if (clock64() - t0 > kWaitCycles) {
      record_error(code, (blockIdx.x << 8) | (threadIdx.x >> 5));
      return false;
    }
  }
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(map), "r"(cluster_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {     // arrives on this barrier of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
  using C = PairCfg;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = smem + C::STAGES * C::STAGE;
  const uint32_t full0 = bars, empty0 = full0 + 8 * C::STAGES, tfull0 = empty0 + 8 * C::STAGES, tempty0 = tfull0 + 16, slot = tempty0 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_rank();
  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM), tiles_n = (p.N + C::BN - 1) / C::BN, n_tiles = tiles_m * tiles_n;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, KB = p.K * 2 / BKB;
  // work of this pair: whole tiles pair, pair + pairs, ..., then (split) a part of a tile of the last wave
  const int whole = p.split > 1 ? n_tiles / pairs * pairs : n_tiles;
  struct Work { int t, kb0, kb1, part; };      // part < 0: a whole tile
  const auto work = [&](int i, Work& w) -> bool {
    w.t = pair + i * pairs;
    w.kb0 = 0; w.kb1 = KB; w.part = -1;
    if (w.t < whole) return true;
    if (p.split <= 1 || i != whole / pairs || pair >= (n_tiles - whole) * p.split) return false;
    w.t = whole + pair / p.split;
    w.part = pair % p.split;
    w.kb0 = w.part * KB / p.split;
    w.kb1 = (w.part + 1) * KB / p.split;
    return true;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(full0 + 8 * i, 1);           // used in the even CTA: both CTAs' bytes
      mbar_init(empty0 + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tfull0 + 8 * i, 1);
      mbar_init(tempty0 + 8 * i, 8);         // used in the even CTA: both CTAs' epilogue warps
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // both CTAs' barriers are there before anything arrives on them
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(slot));

  if (warp == 0) {
    // ------------------------------------------------------------ copies: this CTA's halves of A and B
    if (lane == 0) {
      prefetch_tmap(&map_a);
      prefetch_tmap(&map_b);
      int it = 0;
      bool ok = true;
      Work w;
      for (int i = 0; ok && work(i, w); ++i) {
        const int row0 = (w.t % tiles_m) * 2 * BM + rank * BM, n0 = (w.t / tiles_m) * C::BN + rank * (C::BN / 2);
        for (int kb = w.kb0; kb < w.kb1; ++kb, ++it) {
          const int s = it % C::STAGES;
          if (it >= C::STAGES) ok = mbar_wait_lone(empty0 + 8 * s, ((it / C::STAGES) - 1) & 1, ERR_GEMM_EMPTY_WAIT);
          if (!ok) break;
          const uint32_t sa = smem + s * C::STAGE, bar = map_rank0(full0 + 8 * s);
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * C::STAGE);
          tma_load_2d_pair(sa, &map_a, kb * (BKB / 2), row0, bar);
          tma_load_2d_pair(sa + C::HALF, &map_b, kb * (BKB / 2), n0, bar);
        }
      }
      // After a wait that ran out, the even CTA waits (bounded) for the bytes both have asked for; the odd one meets it at the
      // cluster barrier below.
      if (!ok && rank == 0)
        for (int i = max(0, it - C::STAGES); i < it; ++i) mbar_wait(full0 + 8 * (i % C::STAGES), (i / C::STAGES) & 1, ERR_GEMM_FULL_WAIT);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMAs, even CTA only
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = make_idesc(1, 1, 2 * BM, C::BN);
      int it = 0, lt = 0;
      bool ok = true;
      Work w;
      for (; ok && work(lt, w); ++lt) {
        const int a = lt & 1;
        if (lt >= 2) ok = mbar_wait_cluster(tempty0 + 8 * a, ((lt >> 1) - 1) & 1, ERR_GEMM_TMEM_EMPTY_WAIT);
        if (!ok) break;
        tc_fence_after();
        for (int kb = w.kb0; kb < w.kb1; ++kb, ++it) {
          const int s = it % C::STAGES;
          ok = mbar_wait_cluster(full0 + 8 * s, (it / C::STAGES) & 1, ERR_GEMM_FULL_WAIT);
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = make_desc_sw128(smem + s * C::STAGE), db = make_desc_sw128(smem + s * C::STAGE + C::HALF);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_pair(tmem + a * C::BN, da + 2 * k, db + 2 * k, idesc, ((kb - w.kb0) | k) != 0);
          tc_commit_pair(empty0 + 8 * s);
        }
        if (ok) tc_commit_pair(tfull0 + 8 * a);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5): this CTA's 128 rows
    const int quarter = warp & 3;
    int lt = 0;
    bool ok = true;
    Work w;
    for (; work(lt, w); ++lt) {
      const int a = lt & 1, nt = w.t / tiles_m;
      const int grow = (w.t % tiles_m) * 2 * BM + rank * BM + quarter * 32 + lane;
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * a, (lt >> 1) & 1, ERR_GEMM_TMEM_FULL_WAIT));
      if (!ok && w.part < 0) continue;      // (a part is counted even if nothing arrived: the tickets go back to zero)
      tc_fence_after();
      const auto sums = [&](int c, uint32_t (&v)[32]) {
        B2_TMEM_LD_32(tmem + a * C::BN + c * 32 + ((uint32_t)(quarter * 32) << 16), v);
        tmem_ld_wait();
      };
      if (w.part < 0) {
#pragma unroll 1
        for (int c = 0; c < C::BN / 32; ++c) {
          uint32_t v[32];
          sums(c, v);
          const int n0 = nt * C::BN + c * 32;
          if (grow < p.M && n0 < p.N) store_chunk(p, v, grow, n0);
        }
      } else {
        const int tail = w.t - whole;
        constexpr int kHalf = C::BN / 64;                          // chunks of a half of the columns, which are counted together
        constexpr size_t kPart = 2 * (C::BN / 32) * 4 * 256;       // float4 of a part of both CTAs
        float4* mine = reinterpret_cast<float4*>(p.part) + (((size_t)tail * p.split * 2 + rank) * (C::BN / 32) * 4 + quarter) * 256 + lane;
        for (int hh = 0; hh < 2; ++hh) {
          const int half = (hh + w.part) & 1;
#pragma unroll 1
          for (int c = half * kHalf; c < (half + 1) * kHalf; ++c) {
            uint32_t v[32];
            sums(c, v);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              __stcg(mine + w.part * kPart + c * 1024 + 32 * j, make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
          }
          __threadfence();
          __syncwarp();
          int last = 0;
          if (lane == 0) {
            int* tk = p.part_tickets + ((tail * 2 + rank) * 4 + quarter) * 2 + half;
            last = atomicAdd(tk, 1) == p.split - 1;
            if (last) *tk = 0;
          }
          if (!__shfl_sync(0xffffffffu, last, 0)) continue;
          __threadfence();
#pragma unroll 1
          for (int c = half * kHalf; c < (half + 1) * kHalf; ++c) {
            float f[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = 0.f;
#pragma unroll 1
            for (int q0 = 0; q0 < p.split; q0 += 4) {
              float4 x[4][8];
#pragma unroll
              for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int j = 0; j < 8; ++j) x[q][j] = q0 + q < p.split ? __ldcg(mine + (q0 + q) * kPart + c * 1024 + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int j = 0; j < 8; ++j) { f[4 * j] += x[q][j].x; f[4 * j + 1] += x[q][j].y; f[4 * j + 2] += x[q][j].z; f[4 * j + 3] += x[q][j].w; }
            }
            uint32_t v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(f[j]);
            const int n0 = nt * C::BN + c * 32;
            if (grow < p.M && n0 < p.N) store_chunk(p, v, grow, n0);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_rank0(tempty0 + 8 * a));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // nothing of the other CTA is on its way here any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// ------------------------------------------------------------------ W4B -> bf16 [N][K] (two-pass prefill path)
// grid (ceil(K / 256), N / 128), 256 threads: a thread (tile j = warp, lane) expands its 16 bytes of four consecutive blocks, all
// loaded at once.  The four lanes of a quad hold 32 contiguous bytes of a row, so they store whole sectors from registers;
// through a shared-memory tile, one block per CTA, the pass ran at 4.6 TB/s.
// 34816 x 5120: 98 -> 83 us (451 MB, 5.5 TB/s).  PAIRS: 4-byte stores, for an output that is aligned to no more.
template <bool PAIRS>
__global__ void __launch_bounds__(256) dequant_w4b_kernel(const uint8_t* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                                          int N, int K) {
  constexpr int U = 4;
  const int kg0 = blockIdx.x * U, nb = blockIdx.y, KG = K / 64;
  const uint8_t* blk = w + ((size_t)nb * KG + kg0) * 4352;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint4 wv[U];
  uint32_t sc[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (kg0 + u >= KG) break;
    wv[u] = __ldg(reinterpret_cast<const uint4*>(blk + (size_t)u * 4352 + warp * 512 + lane * 16));
    sc[u] = __ldg(reinterpret_cast<const uint32_t*>(blk + (size_t)u * 4352 + 4096) + warp * 8 + g);   // scales are stored as (g, g + 8) pairs
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (kg0 + u >= KG) break;
    const __half2 sh = *reinterpret_cast<const __half2*>(&sc[u]);
    const uint32_t wa[4] = {wv[u].x, wv[u].y, wv[u].z, wv[u].w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int n = nb * 128 + warp * 16 + g + 8 * (c & 1);
      const float s = (c & 1) ? __high2float(sh) : __low2float(sh);
      if (n >= N) continue;
      __nv_bfloat16* row = out + (size_t)n * K + (kg0 + u) * 64 + 32 * (c >> 1) + 4 * t;
#pragma unroll
      for (int e = 0; e < 2; ++e) {  // e = 0: low nibbles (k = 4t + b of the 32-k step), 1: high nibbles (+ 16)
        const uint32_t x = (wa[c] >> (4 * e)) & 0x0F0F0F0Fu;
        float f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = (float)((int)((x >> (8 * i)) & 0xFF) - 8) * s;
        const uint32_t lo = pack_bf16(f[0], f[1]), hi = pack_bf16(f[2], f[3]);
        if (PAIRS) {
          reinterpret_cast<uint32_t*>(row + 16 * e)[0] = lo;
          reinterpret_cast<uint32_t*>(row + 16 * e)[1] = hi;
        } else {
          *reinterpret_cast<uint2*>(row + 16 * e) = make_uint2(lo, hi);
        }
      }
    }
  }
}

// ------------------------------------------------------------------ per-token int8 activation quant
// one CTA per row: scale = max|x| / 127
__global__ void __launch_bounds__(256) quant_rows_i8_kernel(const __nv_bfloat16* __restrict__ x, int8_t* __restrict__ q,
                                                            float* __restrict__ scale, int K) {
  __shared__ float red[8];
  const int m = blockIdx.x;
  const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(x + (size_t)m * K);
  float amax = 0.f;
  for (int i = threadIdx.x; i < K / 2; i += 256) {
    const float2 v = __bfloat1622float2(xp[i]);
    amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, red[i]);
  const float sc = amax > 0.f ? amax / 127.f : 1.f, inv = 1.f / sc;
  for (int i = threadIdx.x; i < K / 2; i += 256) {
    const float2 v = __bfloat1622float2(xp[i]);
    char2 o;
    o.x = (signed char)__float2int_rn(v.x * inv);
    o.y = (signed char)__float2int_rn(v.y * inv);
    reinterpret_cast<char2*>(q + (size_t)m * K)[i] = o;
  }
  if (threadIdx.x == 0) scale[m] = sc;
}

// ------------------------------------------------------------------ host side: tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// rows x cols (cols contiguous) matrix (batch 0), or a stack of `batch` of them; box = box_rows x 128 bytes
int make_map(CUtensorMap* map, const void* ptr, bool i8, uint64_t rows, uint64_t cols, uint64_t batch,
             uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -100;
  const uint64_t esz = i8 ? 1 : 2;
  cuuint64_t dims[3] = {cols, rows, batch ? batch : 1};
  cuuint64_t strides[2] = {cols * esz, rows * cols * esz};
  cuuint32_t box[3] = {(cuuint32_t)(BKB / esz), box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const int rank = batch ? 3 : 2;
  CUresult r = fn(map, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank,
                  const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -101 - (int)r;
}

int sm_count() {
  static int n[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!n[dev & 63]) cudaDeviceGetAttribute(&n[dev & 63], cudaDevAttrMultiProcessorCount, dev);
  return n[dev & 63];
}

template <int BN, bool I8>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& part, const GemmParams& p, int n_tiles_max, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<BN, I8>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  const int grid = min(n_tiles_max, sm_count());
  gemm_tc_kernel<BN, I8><<<grid, kThreads, Cfg<BN>::SMEM, st>>>(ma, mb, part, p);
  return (int)cudaGetLastError();
}

template <int BN>
int launch_w4(const CUtensorMap& ma, const CUtensorMap& part, const GemmParams& p, int n_tiles_max, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<BN, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Cfg<BN, true>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  const int grid = min(n_tiles_max, sm_count());
  gemm_tc_kernel<BN, false, true><<<grid, Cfg<BN, true>::THREADS, Cfg<BN, true>::SMEM, st>>>(ma, ma, part, p);
  return (int)cudaGetLastError();
}

int launch_pair(const CUtensorMap& ma, const CUtensorMap& mb, const GemmParams& p, cudaStream_t st) {
  using C = PairCfg;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + C::BN - 1) / C::BN), pairs = min(tiles, sm_count() / 2);
  gemm_pair_kernel<<<p.split > 1 ? sm_count() / 2 * 2 : 2 * pairs, kThreads, C::SMEM, st>>>(ma, mb, p);
  return (int)cudaGetLastError();
}

// Parts along K of the pair form's last wave of tiles: the longest part, and what leaving, counting and adding parts costs (in k blocks of a tile, the unit
// of tile_of), against the whole tile; parts of 8 k blocks and more.  Behind more than six whole waves a last one is too little of the product to gain by
// (34816 x 5120 at 900 rows, seven: 244 / 245 us; 3000 rows, 22: 676 / 682).
int parts_of(int tiles, int kb) {
  const int pairs = sm_count() / 2, rest = tiles % pairs;
  int best = 1, cost = kb;
  for (int s = 2; s <= 8 && rest > 0 && rest * s <= pairs && kb >= 8 * s && tiles / pairs <= 6; ++s) {
    const int c = (kb + s - 1) / s + 24 + 2 * s;
    if (c < cost) { cost = c; best = s; }
  }
  return best;
}

// Tile of a bf16 product that is not grouped: -256 the pair form, or 256 / 128 columns on one SM.  Waves of tiles times what a
// wave takes (K = 5120, weights beyond L2): 256 x 256 on two SMs 30 us, 128 x 256 on one 33, 128 x 128 22; the narrow tile only
// where it fits in one wave.  130 x 5120 x 17408: 110 / 78 us wide / narrow, 300 x 34816 x 5120: 128 / 116 pair / wide,
// 512 x 5120 x 17408: 93 / 126, 4096 x 34816 x 5120: 908 / 986.  parts: a workspace for cutting the last wave of pairs is there.
// cost: the estimate, in k blocks of a 256 x 256 tile, 0.375 us each and a launch, cut or not (256 rows, estimate / us: 16480 x 5120 80 / 38, 22016 x 4096 111 / 57;
// cut 2048 x 6144 52 / 22, 5120 x 5120 57 / 24, 4096 x 11008 75 / 32, 5120 x 17408 121 / 48).
int tile_of(int M, int N, int K, bool parts, int* cost = nullptr) {
  const int sms = sm_count(), mt = (M + BM - 1) / BM, mp = (M + 2 * BM - 1) / (2 * BM), kb = K / 64;
  const int wide = (N >= 256 && (N % 256 == 0 || N > 2048)) ? 256 : 128;
  const auto waves = [](int tiles, int at_once) { return (tiles + at_once - 1) / at_once; };
  const int n256 = (N + 255) / 256, n128 = (N + 127) / 128, s = parts ? parts_of(mp * n256, kb) : 1;
  const int pair = s > 1 ? mp * n256 / (sms / 2) * kb + (kb + s - 1) / s + 24 + 2 * s : waves(mp * n256, sms / 2) * kb;
  const int one = waves(mt * n256, sms) * kb * 11 / 10, narrow = kb * 11 / 15;
  const bool fits = mt * n128 <= sms && (N < 256 || narrow < min(pair, one));
  if (cost) *cost = fits ? narrow : min(pair, one);
  if (N < 256) return wide;
  if (fits) return 128;
  return pair <= one ? -256 : wide;
}

}  // namespace

// C = A * W^T with W read as int4: a [M][K] bf16, w4b the W4B blocks [E][ceil(N / 128)][K / 64][4352] (E = 1 unless the
// blk_* tables of the grouped form are given).  Epilogues 0..3 as b2_gemm_tc.
extern "C" int b2_gemm_w4(const void* a, const void* w4b, void* c, int M, int N, int K, int ldc, int epi, const void* resid,
                          const int* blk_expert, const int* blk_row0, const int* blk_rows, const int* n_blk, int max_blk,
                          int n_experts, int bn, void* stream) {
  if (K % 64 != 0 || M < 1 || N % 8 != 0 || epi < EPI_BF16 || epi > EPI_RESID_ADD) return -1;
  if (epi == EPI_SILU_MUL && N % 32 != 0) return -2;
  if (((uintptr_t)w4b) & 15) return -3;
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.C = c; p.resid = (const __nv_bfloat16*)resid; p.epi = epi;
  p.blk_expert = blk_expert; p.blk_row0 = blk_row0; p.blk_rows = blk_rows; p.n_blk = n_blk; p.max_blk = max_blk;
  p.rs_world = 1; p.rs_tpr = 1;
  p.w4 = (const uint8_t*)w4b;
  p.w4_expert_bytes = (long long)((N + 127) / 128) * (K / 64) * kW4Block;
  if (bn != 128 && bn != 256) {
    bn = (N >= 256 && (N % 256 == 0 || N > 2048)) ? 256 : 128;
    // narrow tiles while they fit in one wave (100 x 7168 x 5120: 57 / 46 us wide / narrow, x 5120 x 17408 166 / 137)
    if (!blk_expert && (M + BM - 1) / BM * ((N + 127) / 128) <= sm_count()) bn = 128;
  }
  CUtensorMap ma, part;
  int rc = make_map(&ma, a, false, (uint64_t)M, (uint64_t)K, 0, BM);
  if (!rc) rc = make_map(&part, a, false, (uint64_t)M, (uint64_t)K, 0, kGroupBox);
  if (rc) return rc;
  const int tiles_m = blk_expert ? max_blk : (M + BM - 1) / BM;
  const int n_tiles = tiles_m * ((N + bn - 1) / bn);
  (void)n_experts;
  cudaStream_t st = (cudaStream_t)stream;
  return bn == 256 ? launch_w4<256>(ma, part, p, n_tiles, st) : launch_w4<128>(ma, part, p, n_tiles, st);
}

// C = A * B^T.  a: [M][K], b: [N][K] (or [E][N][K] when blk_* are given), both bf16 (i8 = 0) or int8 (i8 = 1).
static int gemm_tc_impl(const void* a, const void* b, void* c, int M, int N, int K, int ldc, int i8, int epi,
                        const void* resid, const float* a_scale, const float* b_scale, const int* blk_expert,
                        const int* blk_row0, const int* blk_rows, const int* n_blk, int max_blk, int n_experts,
                        int bn, const void* rs_table, int rs_rank, int rs_world, int rs_tpr, const int* ag_cnt,
                        int ag_expect, const int* blk_wait, const int* row_src, const void* ret_table, void* stream,
                        const Glu& glu = Glu{}, float* part = nullptr, long long part_floats = 0, int* part_tickets = nullptr, int n_tickets = 0) {
  if (K % (i8 ? 128 : 64) != 0 || M < 1 || N % 8 != 0) return -1;
  if ((epi == EPI_SILU_MUL || epi == EPI_GLU) && N % 32 != 0) return -2;
  if (epi == EPI_RS_PUSH && (!rs_table || rs_world < 1 || rs_world > kMaxRanks || rs_rank < 0 || rs_rank >= rs_world ||
                             rs_tpr < 1 || N % 64 != 0 || blk_expert || (M + BM - 1) / BM > rs_tpr * rs_world))
    return -3;
  GemmParams p;
  p.rs_table = (const unsigned long long*)rs_table; p.rs_rank = rs_rank; p.rs_world = rs_world; p.rs_tpr = rs_tpr;
  p.ag_cnt = ag_cnt; p.ag_expect = ag_expect;
  p.blk_wait = blk_wait; p.row_src = row_src; p.ret_table = (const unsigned long long*)ret_table;
  if (epi == EPI_EP_RETURN && (!row_src || !ret_table || !blk_expert || N % 64 != 0)) return -4;
  p.mt_rot = (epi == EPI_RS_PUSH) ? (rs_rank * rs_tpr) % ((M + BM - 1) / BM) : 0;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.C = c; p.resid = (const __nv_bfloat16*)resid;
  p.a_scale = a_scale; p.b_scale = b_scale; p.epi = epi; p.glu = glu;
  p.split = 0; p.part = part; p.part_tickets = part_tickets;
  p.blk_expert = blk_expert; p.blk_row0 = blk_row0; p.blk_rows = blk_rows; p.n_blk = n_blk; p.max_blk = max_blk;
  const bool local = !i8 && !blk_expert && !ag_cnt && epi != EPI_RS_PUSH && epi != EPI_EP_RETURN;
  bool pair = local && bn == -256;
  if (!pair && bn != 128 && bn != 256) {
    bn = local ? tile_of(M, N, K, part != nullptr) : (N >= 256 && (N % 256 == 0 || N > 2048)) ? 256 : 128;
    // few rows: narrower tiles while they still fit in one wave
    if (!local && !blk_expert && ((M + BM - 1) / BM) * ((N + 127) / 128) <= sm_count()) bn = 128;
    pair = bn == -256;
  }
  if (pair) {
    bn = 128;       // B arrives in two halves
    const int tiles = (M + 2 * BM - 1) / (2 * BM) * ((N + 255) / 256), rest = tiles % (sm_count() / 2);
    if (part) p.split = parts_of(tiles, K / 64);
    if (p.split > 1 && ((long long)rest * p.split * 65536 > part_floats || rest * 16 > n_tickets || ((uintptr_t)part & 15))) return -8;
  }
  CUtensorMap ma, mb, mp;
  int rc = make_map(&ma, a, i8 != 0, (uint64_t)M, (uint64_t)K, 0, BM);
  if (rc) return rc;
  mp = ma;
  if (blk_expert) rc = make_map(&mp, a, i8 != 0, (uint64_t)M, (uint64_t)K, 0, kGroupBox);
  if (rc) return rc;
  rc = make_map(&mb, b, i8 != 0, (uint64_t)N, (uint64_t)K, blk_expert ? (uint64_t)n_experts : 0, (uint32_t)bn);
  if (rc) return rc;
  const int tiles_m = blk_expert ? max_blk : (M + BM - 1) / BM;
  const int n_tiles = tiles_m * ((N + bn - 1) / bn);
  cudaStream_t st = (cudaStream_t)stream;
  if (pair) return launch_pair(ma, mb, p, st);
  if (bn == 256) return i8 ? launch<256, true>(ma, mb, mp, p, n_tiles, st) : launch<256, false>(ma, mb, mp, p, n_tiles, st);
  return i8 ? launch<128, true>(ma, mb, mp, p, n_tiles, st) : launch<128, false>(ma, mb, mp, p, n_tiles, st);
}

extern "C" int b2_gemm_tc(const void* a, const void* b, void* c, int M, int N, int K, int ldc, int i8, int epi,
                          const void* resid, const float* a_scale, const float* b_scale, const int* blk_expert,
                          const int* blk_row0, const int* blk_rows, const int* n_blk, int max_blk, int n_experts,
                          int bn, void* stream) {
  return gemm_tc_impl(a, b, c, M, N, K, ldc, i8, epi, resid, a_scale, b_scale, blk_expert, blk_row0, blk_rows, n_blk,
                      max_blk, n_experts, bn, nullptr, 0, 1, 1, nullptr, 0, nullptr, nullptr, nullptr, stream);
}

// 1: a product of M rows with an int4 weight is estimated to be faster from the blocks (b2_gemm_w4) than from an expanded copy that has to be made first
// (b2_dequant_w4b and b2_gemm_tc_parts).  us: 6 and 0.456 (128 x 128 tiles) or 0.6 (128 x 256) for a k block and wave; against 0.43 for a million weights expanded,
// the product's tiles, or 0.31 for a million bf16 weights read where that is more, and 6.  Blocks / copy, device time, weights from HBM:
//   100 rows  3072 x 2048 20.2 / 17.9, 2048 x 4096 34.4 / 26.4, 9216 x 2048 20.9 / 23.0, 5120 x 5120 43.6 / 39.3, 7168 x 5120 42.8 / 44.4, 8192 x 5120 42.5 / 45.0,
//             16480 x 5120 42.4 / 73.3, 34816 x 5120 57 / 148, 4096 x 11008 83 / 48, 5120 x 17408 129 / 89
//   160 rows  12288 x 2048 27.8 / 30.6, 7168 x 5120 42.8 / 44.8, 16480 x 5120 52 / 77, 22016 x 4096 84 / 95, 34816 x 5120 99 / 150, 5120 x 17408 128 / 89
// Weights of up to four million stay where the rows put them, from the blocks up to one row of tiles: the forms differ by a microsecond (1024 x 1024, 100 rows
// 12.7 / 11.8, but 14.7 / 17.8 as issued from the host, 160 rows 12.7 / 11.9).
extern "C" int b2_gemm_w4_blocks(int M, int N, int K) {
  const int mt = (M + BM - 1) / BM, kb = K / 64, sms = sm_count();
  const bool narrow = mt * ((N + 127) / 128) <= sms;
  const double blocks = narrow ? 0.456 * kb : 0.6 * kb * ((mt * ((N + 255) / 256) + sms - 1) / sms);
  int cost = 0;
  tile_of(M, N, K, true, &cost);
  const double millions = 1e-6 * N * K, tiles = 0.375 * cost, read = 0.31 * millions;
  return millions <= 4.2 ? mt == 1 : blocks <= 0.43 * millions + (tiles > read ? tiles : read);
}

// bf16 C = A * B^T with a workspace for cutting the last wave of tiles along K: b2_gemm_parts() floats and tickets, the latter zeroed once.  One product at a
// time per workspace.
extern "C" void b2_gemm_parts(long long* floats, int* tickets) {
  *floats = (long long)(sm_count() / 2) * 65536;
  *tickets = sm_count() / 2 * 16;
}
// 1: a product of this shape uses one
extern "C" int b2_gemm_in_parts(int M, int N, int K) {
  return tile_of(M, N, K, true) == -256 && parts_of((M + 2 * BM - 1) / (2 * BM) * ((N + 255) / 256), K / 64) > 1;
}
extern "C" int b2_gemm_tc_parts(const void* a, const void* b, void* c, int M, int N, int K, int ldc, int epi, const void* resid, int bn, float* part,
                                long long part_floats, int* part_tickets, int n_tickets, void* stream) {
  if (!part || !part_tickets || (epi != EPI_BF16 && epi != EPI_F32 && epi != EPI_SILU_MUL && epi != EPI_RESID_ADD && epi != EPI_RELU2)) return -1;
  return gemm_tc_impl(a, b, c, M, N, K, ldc, 0, epi, resid, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 1, bn, nullptr, 0, 1, 1, nullptr, 0, nullptr,
                      nullptr, nullptr, stream, Glu{}, part, part_floats, part_tickets, n_tickets);
}

// bf16 C [M][N / 2] = gated product of the interleave16 columns of A * B^T (common.cuh, Glu)
extern "C" int b2_gemm_tc_glu(const void* a, const void* b, void* c, int M, int N, int K, int ldc, float limit, float alpha,
                              float shift, int gelu, const float* bias, void* stream) {
  return gemm_tc_impl(a, b, c, M, N, K, ldc, 0, EPI_GLU, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 1, 0,
                      nullptr, 0, 1, 1, nullptr, 0, nullptr, nullptr, nullptr, stream, Glu{limit, alpha, shift, gelu, bias});
}

// Tensor-parallel forms of the same kernel.  epi = 4 (row-parallel GEMM -> reduce-scatter): c is unused, the
// bf16 tiles go to the row owners' landing buffers of rs_table (rs_tpr m-tiles per owner) and arrivals are
// counted at the owners.  ag_cnt (all-gather -> GEMM): the rows of a arrive from their owners in this GPU's
// memory; m-tile i is loaded once ag_cnt[i] has reached ag_expect.
extern "C" int b2_gemm_tc_tp(const void* a, const void* b, void* c, int M, int N, int K, int ldc, int i8, int epi,
                             const void* resid, const float* a_scale, const float* b_scale, int bn,
                             const void* rs_table, int rs_rank, int rs_world, int rs_tpr, const int* ag_cnt,
                             int ag_expect, void* stream) {
  return gemm_tc_impl(a, b, c, M, N, K, ldc, i8, epi, resid, a_scale, b_scale, nullptr, nullptr, nullptr, nullptr, 0, 1,
                      bn, rs_table, rs_rank, rs_world, rs_tpr, ag_cnt, ag_expect, nullptr, nullptr, nullptr, stream);
}

// Expert-parallel forms of the grouped GEMM.  blk_wait: the rows of a block arrive from the source ranks'
// dispatch kernels; block i is loaded once blk_wait[i] >= blk_rows[i].  epi = 5: every result row is stored
// into the return buffer of the rank its token came from (row_src, ret_table).
extern "C" int b2_gemm_tc_ep(const void* a, const void* b, void* c, int M, int N, int K, int ldc, int epi,
                             const int* blk_expert, const int* blk_row0, const int* blk_rows, const int* n_blk,
                             int max_blk, int n_experts, int bn, const int* blk_wait, const int* row_src,
                             const void* ret_table, void* stream) {
  return gemm_tc_impl(a, b, c, M, N, K, ldc, 0, epi, nullptr, nullptr, nullptr, blk_expert, blk_row0, blk_rows, n_blk,
                      max_blk, n_experts, bn, nullptr, 0, 1, 1, nullptr, 0, blk_wait, row_src, ret_table, stream);
}

extern "C" int b2_dequant_w4b(const void* w4b, void* out_bf16, int N, int K, void* stream) {
  if (K % 64) return -1;
  if (((uintptr_t)w4b & 15) || ((uintptr_t)out_bf16 & 3)) return -3;
  dim3 grid((K / 64 + 3) / 4, (N + 127) / 128);
  const auto kernel = ((uintptr_t)out_bf16 & 7) ? dequant_w4b_kernel<true> : dequant_w4b_kernel<false>;
  kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint8_t*)w4b, (__nv_bfloat16*)out_bf16, N, K);
  return (int)cudaGetLastError();
}

extern "C" int b2_quant_rows_i8(const void* x, void* q, float* scale, int M, int K, void* stream) {
  if (K % 2) return -1;
  quant_rows_i8_kernel<<<M, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, (int8_t*)q, scale, K);
  return (int)cudaGetLastError();
}

B2_DEFINE_STATUS(gemm)
