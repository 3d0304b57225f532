// Prefill product (M > 32 activation rows) on the 5th-generation tensor cores: tcgen05.mma with
// the accumulator in tensor memory (TMEM).
//
// Bound: tensor cores (2 M N K flops). Replaces the reference's tiled quantised matmul
// (fusor-ml/tile-ir-kernels/src/kernels/qmatmul.rs:237-349) for large M, where the small-batch
// kernels would re-read W once per 32 rows.
//
// This file packs the activations, chooses how a product runs, and holds the kernel of single CTAs, which is left for
// few rows of wide matrices; most products run on CTA pairs (qgemm_pair.cu). In the kernel here a CTA computes a tile of
// 256 weight rows by 128 activation rows of Y^T = W . X^T; the fp32 accumulators (two halves of 128 lanes x 128 columns)
// live in TMEM. The roles are coupled only by mbarriers, there is no CTA-wide barrier in the main loop:
//  * weight loader (one thread): W stays quantised in HBM; the raw tile-groups of the CTA's
//    16 row-tiles for one K group come by 1-D TMA bulk copies, two K groups in flight.
//  * conversion warps (16, one per row-tile): dequantise to fp16 in registers (byte -> 1024 +
//    byte by a byte permute, exact subtraction, one fused multiply-add with block scale and
//    offset) and store into the A operand stage in the canonical K-major core-matrix layout of
//    the MMA (8 rows x 16 bytes per core matrix, no swizzle); a proxy fence, then one arrive per
//    warp on the stage's "A full" barrier.
//  * activation loader (one thread): X is converted once per call to fp16 rows scaled by a power
//    of two and stored tile by tile in the same operand layout, so a B stage is one contiguous
//    bulk copy.
//  * MMA issuer (one thread): waits for "A full" and "B full", issues 8 tcgen05.mma (M = 128,
//    N = 128, K = 16, kind::f16, fp32 accumulate) per 64-wide K block; tcgen05.commit on the
//    stage's "free" barrier hands the stage back to both producers (2..4 stages, as many as fit
//    beside the raw buffers).
//  * Epilogue: tcgen05.ld brings the accumulator out of TMEM (each warp its 32 lanes), rows are
//    scaled back and written, with the residual adds or SwiGLU (gate and up rows are the two
//    halves of one CTA, so both values of an output sit in the same TMEM lane).
// Every wait is bounded (2^22 polls): on a time-out the status word and a give-up flag in shared
// memory are set, the other roles leave at their next poll, loaders and issuer wait (with a limit) for
// their copies and MMAs in flight, and the CTA releases its TMEM columns and exits.
// FB200_TCGEN05=0 switches the kernel off (32-row kernel in chunks);
// FB200_TC_TILE forces a tile shape (tests, tuning).
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "half_weights.cuh"
#include "qgemm_pair.cuh"
#include "tcgen05.cuh"

int fb200_ensure(fb200_device* dev, void** buf, size_t* cur, size_t bytes);

namespace {

constexpr int BN = 128;  // weight rows per MMA (M of the MMA)
constexpr int NH = 2;    // such halves in a CTA tile
constexpr int BM = 128;  // activation rows per CTA tile (N of the MMA), and of a packed activation tile
constexpr int BK = 64;   // K elements per operand stage (four K = 16 MMAs)
constexpr int A_SBO = (BK / 8) * 128 + 64;        // A operand: bytes between 8-row groups, padded by half a
                                                  // core matrix so that rows g and g + 8 fall into different banks
constexpr int A_HALF = (BN / 8) * A_SBO;          // one 128-row half of an A stage
constexpr int CORE_LBO = 128;                     // bytes between core matrices adjacent in K
constexpr int CORE_SBO = (BK / 8) * 128;          // B operand: bytes between 8-row groups
constexpr int MAX_STAGES = 4;
constexpr int TAIL_BYTES = 256;                   // barriers, TMEM slot, give-up flag
constexpr int SMEM_BUDGET = 227 * 1024;
constexpr int A_BYTES = NH * A_HALF, B_BYTES = BM * BK * 2, STAGE = A_BYTES + B_BYTES;  // operands of a stage
constexpr int TMEM_COLS = NH * BM;            // fp32 accumulator columns
constexpr int DQ_WARPS = 8 * NH;              // one warp per 16-row tile
constexpr int THREADS = (DQ_WARPS + 3) * 32;  // + weight loader, activation loader, MMA issuer
// instruction descriptor: fp32 accumulator, fp16 A and B, both K-major, N = BM, M = BN
constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(BM >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);

struct TcArgs {
  const uint8_t* w;      // tiled weights
  const __half* xh;      // fp16 activations, [Mp / BM][K / 64] tiles already in the operand layout
  const float* xscale;   // [Mp] power-of-two scale of each row
  float* y;              // [M, N]
  const float* r1;       // optional residuals [M, N], or one bias row [N] when r1_stride is 0
  const float* r2;
  int r1_stride;
  int M, N, K;
  int ngroups, ntiles, type, tgb, group_elems;
  int stages, raw_stride;  // operand stages that fit beside the raw buffers; bytes per raw tile-group slot
  int pair_tiles;          // SwiGLU: half 0 = gate rows, half 1 = up rows pair_tiles row-tiles further;
                           // y[M, N / 2] = silu(gate) * up. 0 = plain product
  int* status;
};

__device__ __forceinline__ uint32_t lds4(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint4 lds16(const uint8_t* p) { return *reinterpret_cast<const uint4*>(p); }

// Row-tile `tile` of one K group: the four registers of 32-element chunk c for lane (g, t) --
// bytes of rows g / g + 8, elements 4t.. and 16 + 4t.. -- dequantised and stored into operand
// stage `abuf` at rows 16 * wrow + g (+ 8), K offset 32 * cib (chunk inside the 64-wide block).
struct RowScales {
  float sc[2][2], mn[2][2];  // Q4_K: [row half][sub-block t + 4 i]
  uint4 q6[2];               // Q6_K: scale bytes of rows g, g + 8
  float d[2];                // Q6_K: super-block scale
};

__device__ __forceinline__ void store_chunk(uint8_t* abuf, int wrow, int g, int t, int cib, uint2 lo_g, uint2 lo_g8,
                                            uint2 hi_g, uint2 hi_g8) {
  // In one store instruction the lanes with t < 2 write row g and the others row g + 8 (then the
  // other way round): with the padded row-group stride the 16 lanes of a half-warp cover all 32
  // banks once, where "every lane its row g" would put K chunks t / 2 = 0 and 1 on the same banks.
  const bool odd = (t & 2) != 0;
  uint8_t* base = abuf + (2 * wrow) * A_SBO + g * 16 + (t & 1) * 8 + (4 * cib + (t >> 1)) * CORE_LBO;
  uint8_t* p1 = base + (odd ? A_SBO : 0);
  uint8_t* p2 = base + (odd ? 0 : A_SBO);
  *reinterpret_cast<uint2*>(p1) = odd ? lo_g8 : lo_g;
  *reinterpret_cast<uint2*>(p2) = odd ? lo_g : lo_g8;
  *reinterpret_cast<uint2*>(p1 + 2 * CORE_LBO) = odd ? hi_g8 : hi_g;
  *reinterpret_cast<uint2*>(p2 + 2 * CORE_LBO) = odd ? hi_g : hi_g8;
}

template <int type>
__device__ __forceinline__ void prepare_scales(const uint8_t* tg, int g, int t, RowScales& S) {
  if (type == FB200_Q4_K) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 hd = lds16(tg + 2048 + (g + 8 * h) * 16);
      const float d = fb::half_bits_to_float((uint16_t)(hd.x & 0xFFFF));
      const float dmin = fb::half_bits_to_float((uint16_t)(hd.x >> 16));
      const uint32_t s0 = hd.y, s1 = hd.z, s2 = hd.w;
      const uint32_t scB = (s2 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u);
      const uint32_t mnB = ((s2 >> 4) & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u);
      const int sh = 8 * t;
      S.sc[h][0] = d * (float)((s0 >> sh) & 0x3F);
      S.mn[h][0] = dmin * (float)((s1 >> sh) & 0x3F);
      S.sc[h][1] = d * (float)((scB >> sh) & 0xFF);
      S.mn[h][1] = dmin * (float)((mnB >> sh) & 0xFF);
    }
  } else if (type == FB200_Q6_K) {
    S.q6[0] = lds16(tg + 3072 + g * 16);
    S.q6[1] = lds16(tg + 3072 + (g + 8) * 16);
    S.d[0] = fb::half_bits_to_float(*reinterpret_cast<const uint16_t*>(tg + 3328 + g * 2));
    S.d[1] = fb::half_bits_to_float(*reinterpret_cast<const uint16_t*>(tg + 3328 + (g + 8) * 2));
  }
}

// chunk c of the tile-group (32 elements: c < 4 for Q4_0 / Q8_0, c < 8 for the K-quants)
template <int type>
__device__ __forceinline__ void dequant_chunk(const uint8_t* tg, int c, int lane, const RowScales& S,
                                              uint8_t* abuf, int wrow, int cib) {
  const int g = lane >> 2, t = lane & 3;
  const __half2 zero2 = __float2half2_rn(0.f);
  if (type == FB200_Q4_K) {
    const int pair = c >> 1, hi = c & 1, ch = pair >> 1, ps = pair & 1;
    const int off = g * 32 + ps * 16 + 4 * t;
    const uint32_t sh4 = hi ? 4u : 0u;
    const uint32_t w00 = (lds4(tg + ((ch * 2 + 0) * 2 + 0) * 256 + off) >> sh4) & 0x0F0F0F0Fu;  // row g, lo
    const uint32_t w01 = (lds4(tg + ((ch * 2 + 0) * 2 + 1) * 256 + off) >> sh4) & 0x0F0F0F0Fu;  // row g, hi
    const uint32_t w10 = (lds4(tg + ((ch * 2 + 1) * 2 + 0) * 256 + off) >> sh4) & 0x0F0F0F0Fu;  // row g + 8
    const uint32_t w11 = (lds4(tg + ((ch * 2 + 1) * 2 + 1) * 256 + off) >> sh4) & 0x0F0F0F0Fu;
    const int src = (lane & ~3) | (c & 3);
    const __half2 s_g = __float2half2_rn(__shfl_sync(0xFFFFFFFFu, ((c >> 2) ? S.sc[0][1] : S.sc[0][0]), src));
    const __half2 s_g8 = __float2half2_rn(__shfl_sync(0xFFFFFFFFu, ((c >> 2) ? S.sc[1][1] : S.sc[1][0]), src));
    const __half2 o_g = __float2half2_rn(-__shfl_sync(0xFFFFFFFFu, ((c >> 2) ? S.mn[0][1] : S.mn[0][0]), src));
    const __half2 o_g8 = __float2half2_rn(-__shfl_sync(0xFFFFFFFFu, ((c >> 2) ? S.mn[1][1] : S.mn[1][0]), src));
    const __half2 ctr = __float2half2_rn(1024.0f);
    store_chunk(abuf, wrow, g, t, cib, deq4(w00, ctr, s_g, o_g), deq4(w10, ctr, s_g8, o_g8), deq4(w01, ctr, s_g, o_g),
                deq4(w11, ctr, s_g8, o_g8));
  } else if (type == FB200_Q6_K) {
    const int c2 = c >> 2, q = c & 3;
    uint2 out[2][2];  // [u][row half]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int cu = c2 * 2 + u, grp = 8 * c2 + 2 * q + u;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t wl = lds4(tg + (cu * 2 + h) * 256 + g * 32 + (q & 1) * 16 + 4 * t);
        const uint32_t wh = lds4(tg + 2048 + (cu * 2 + h) * 128 + g * 16 + 4 * t);
        const uint32_t hb = q == 0 ? (wh << 4) : q == 1 ? (wh << 2) : q == 2 ? wh : (wh >> 2);
        const uint32_t bytes = (((q >> 1) ? (wl >> 4) : wl) & 0x0F0F0F0Fu) | (hb & 0x30303030u);
        const uint32_t scw = grp >> 2 == 0 ? S.q6[h].x : grp >> 2 == 1 ? S.q6[h].y : grp >> 2 == 2 ? S.q6[h].z : S.q6[h].w;
        const float s = S.d[h] * (float)(int)(int8_t)((scw >> (8 * (grp & 3))) & 0xFF);
        out[u][h] = deq4(bytes, __float2half2_rn(1056.0f), __float2half2_rn(s), zero2);  // (q - 32) d scale
      }
    }
    store_chunk(abuf, wrow, g, t, cib, out[0][0], out[0][1], out[1][0], out[1][1]);
  } else {
    const int dofs = type == FB200_Q4_0 ? 1024 : 2048;
    const __half2 d_g = __half2half2(__ushort_as_half(*reinterpret_cast<const uint16_t*>(tg + dofs + (g * 4 + c) * 2)));
    const __half2 d_g8 = __half2half2(__ushort_as_half(*reinterpret_cast<const uint16_t*>(tg + dofs + ((g + 8) * 4 + c) * 2)));
    if (type == FB200_Q4_0) {
      const uint32_t w0 = lds4(tg + g * 64 + c * 16 + 4 * t);
      const uint32_t w1 = lds4(tg + 512 + g * 64 + c * 16 + 4 * t);
      const __half2 ctr = __float2half2_rn(1032.0f);  // (q - 8) d
      store_chunk(abuf, wrow, g, t, cib, deq4(w0 & 0x0F0F0F0Fu, ctr, d_g, zero2), deq4(w1 & 0x0F0F0F0Fu, ctr, d_g8, zero2),
                  deq4((w0 >> 4) & 0x0F0F0F0Fu, ctr, d_g, zero2), deq4((w1 >> 4) & 0x0F0F0F0Fu, ctr, d_g8, zero2));
    } else {
      const int off = g * 64 + c * 16 + 4 * t;
      const __half2 ctr = __float2half2_rn(1152.0f);  // signed byte b as (b ^ 0x80) - 128
      store_chunk(abuf, wrow, g, t, cib, deq4(lds4(tg + off) ^ 0x80808080u, ctr, d_g, zero2),
                  deq4(lds4(tg + 1024 + off) ^ 0x80808080u, ctr, d_g8, zero2),
                  deq4(lds4(tg + 512 + off) ^ 0x80808080u, ctr, d_g, zero2),
                  deq4(lds4(tg + 1536 + off) ^ 0x80808080u, ctr, d_g8, zero2));
    }
  }
}

template <int TYPE>
__global__ void __launch_bounds__(THREADS, 1)
qgemm_tc_kernel(const TcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int raw_bytes = DQ_WARPS * a.raw_stride;
  uint8_t* opnd = smem;                                   // [stage][A halves | B]
  uint8_t* raw = smem + a.stages * STAGE;              // [2][DQ_WARPS tile-groups]
  uint64_t* bars = reinterpret_cast<uint64_t*>(raw + 2 * raw_bytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * (a.pair_tiles ? BN : BN * NH), m0 = blockIdx.y * BM;
  const uint32_t bar_raw_full = smem_u32(bars), bar_raw_free = smem_u32(bars + 2), bar_a_full = smem_u32(bars + 4),
                 bar_b_full = smem_u32(bars + 4 + MAX_STAGES), bar_free = smem_u32(bars + 4 + 2 * MAX_STAGES),
                 bar_done = smem_u32(bars + 4 + 3 * MAX_STAGES), bar_end = bar_done + 8;  // bar_end: of a CTA that gave up

  if (tid == 0) {
    *dead = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_raw_full + 8 * i, 1);
      mbar_init(bar_raw_free + 8 * i, DQ_WARPS);
    }
    for (int i = 0; i < MAX_STAGES; ++i) {
      mbar_init(bar_a_full + 8 * i, DQ_WARPS);
      mbar_init(bar_b_full + 8 * i, 1);
      mbar_init(bar_free + 8 * i, 1);
    }
    mbar_init(bar_done, 1);
    mbar_init(bar_end, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot;

  const int tile0 = n0 / 16;
  // row-tile converted by warp i, and whether the matrix has it
  auto tile_of = [&](int i) { return a.pair_tiles ? tile0 + (i & 7) + (i >> 3) * a.pair_tiles : tile0 + i; };
  auto has_tile = [&](int i) { return a.pair_tiles ? tile0 + (i & 7) < a.pair_tiles : tile0 + i < a.ntiles; };
  constexpr int blocks_per_group = (TYPE == FB200_Q4_K || TYPE == FB200_Q6_K ? 256 : 128) / BK;
  const int ngr = a.ngroups, nblocks = ngr * blocks_per_group;

  int issued = 0;  // requests of a loader
  if (warp < DQ_WARPS) {
    // ---- conversion: warp w turns row-tile w of each K block into fp16 operand rows
    const bool mine = has_tile(warp);
    uint8_t* const a_rows = opnd + (warp >> 3) * A_HALF;
    int s = 0, round = 0;
    for (int kg = 0; kg < ngr; ++kg) {
      const int rb = kg & 1;
      // (the warp leaves together: its lanes meet in the shuffles of the conversion)
      if (!w_wait(bar_raw_full + 8 * rb, (uint32_t)((kg >> 1) & 1), dead, a.status)) break;
      const uint8_t* tg = raw + rb * raw_bytes + warp * a.raw_stride;
      RowScales S;
      if (mine) prepare_scales<TYPE>(tg, lane >> 2, lane & 3, S);
#pragma unroll
      for (int b = 0; b < blocks_per_group; ++b) {
        // the stage is free once the MMAs of its previous use have read it (or a role gave up, and nothing of this is stored)
        if (round > 0) x_wait(bar_free + 8 * s, (uint32_t)((round - 1) & 1), dead, a.status);
        uint8_t* abuf = a_rows + s * STAGE;
        if (mine) {
          dequant_chunk<TYPE>(tg, 2 * b, lane, S, abuf, warp & 7, 0);
          dequant_chunk<TYPE>(tg, 2 * b + 1, lane, S, abuf, warp & 7, 1);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> tensor-core reads
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_a_full + 8 * s);
        if (++s == a.stages) { s = 0; ++round; }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_raw_free + 8 * rb);
    }
  } else if (warp == DQ_WARPS) {
    // ---- weight loader: raw tile-groups of one K group, two groups in flight
    if (lane == 0) {
      int ntile_here = 0;
      for (int i = 0; i < DQ_WARPS; ++i) ntile_here += has_tile(i) ? 1 : 0;
      for (int kg = 0; kg < ngr; ++kg, ++issued) {
        const int rb = kg & 1;
        if (kg >= 2 && !x_wait(bar_raw_free + 8 * rb, (uint32_t)(((kg >> 1) - 1) & 1), dead, a.status)) break;
        mbar_expect_tx(bar_raw_full + 8 * rb, (uint32_t)(ntile_here * a.tgb));
        for (int i = 0; i < DQ_WARPS; ++i)
          if (has_tile(i))
            bulk_g2s(smem_u32(raw + rb * raw_bytes + i * a.raw_stride),
                     a.w + ((size_t)tile_of(i) * a.ngroups + kg) * a.tgb, (uint32_t)a.tgb, bar_raw_full + 8 * rb);
      }
    }
  } else if (warp == DQ_WARPS + 1) {
    // ---- activation loader: one bulk copy per K block (the tile is stored in operand layout)
    if (lane == 0) {
      const __half* src = a.xh + (size_t)blockIdx.y * nblocks * (BM * BK);
      int s = 0, round = 0;
      for (int blk = 0; blk < nblocks; ++blk, ++issued) {
        if (round > 0 && !x_wait(bar_free + 8 * s, (uint32_t)((round - 1) & 1), dead, a.status)) break;
        mbar_expect_tx(bar_b_full + 8 * s, (uint32_t)B_BYTES);
        bulk_g2s(smem_u32(opnd + s * STAGE + A_BYTES), src + (size_t)blk * (BM * BK), (uint32_t)B_BYTES,
                 bar_b_full + 8 * s);
        if (++s == a.stages) { s = 0; ++round; }
      }
    }
  } else {
    // ---- MMA issuer: eight instructions per K block; the commit frees the stage
    if (lane == 0) {
      int s = 0, round = 0;
      bool alive = true;
      for (int blk = 0; blk < nblocks; ++blk) {
        alive = x_wait(bar_a_full + 8 * s, (uint32_t)(round & 1), dead, a.status) &&
                x_wait(bar_b_full + 8 * s, (uint32_t)(round & 1), dead, a.status);
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = smem_u32(opnd + s * STAGE), sb = sa + A_BYTES;
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks)
            x_mma(tmem_d + (uint32_t)(h * BM), x_desc(sa + h * A_HALF + ks * 2 * CORE_LBO, CORE_LBO, A_SBO),
                   x_desc(sb + ks * 2 * CORE_LBO, CORE_LBO, CORE_SBO), IDESC, (blk | ks) ? 1u : 0u);
        x_commit(bar_free + 8 * s);
        if (++s == a.stages) { s = 0; ++round; }
      }
      if (alive) x_commit(bar_done);
    }
  }

  // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 (weight rows) of one half and one
  // half of that half's columns
  const bool stores = warp < DQ_WARPS && __all_sync(0xFFFFFFFFu, x_wait(bar_done, 0u, dead, a.status) && !*dead);
  if (a.pair_tiles) {
    // SwiGLU: the gate and the up value of an output sit in the same TMEM lane, BM columns apart
    if (stores) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int n = n0 + 32 * (warp & 3) + lane, n_out = a.pair_tiles * 16;
      const int cbase = (BM / 4) * (warp >> 2);
#pragma unroll
      for (int i = 0; i < BM / 64; ++i) {
        uint32_t g[16], u[16];
        const uint32_t taddr = tmem_d + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(cbase + 16 * i);
        x_ld16(taddr, g);
        x_ld16(taddr + BM, u);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int m = m0 + cbase + 16 * i + j;
          if (m < a.M && n < n_out) {
            // silu(gate) * up, fusor-ml/fusor/src/composite/activations.rs:47-64: x / (1 + exp(-x))
            const float sc = a.xscale[m], gate = __uint_as_float(g[j]) * sc;
            a.y[(size_t)m * n_out + n] = (gate / (1.0f + expf(-gate))) * (__uint_as_float(u[j]) * sc);
          }
        }
      }
    }
  } else if (stores) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int part = warp >> 2, h = part >> 1;
    const int n = n0 + h * BN + 32 * (warp & 3) + lane;
    const int cbase = (BM / 2) * (part & 1);
#pragma unroll
    for (int i = 0; i < BM / 64; ++i) {
      uint32_t v[32];
      const uint32_t taddr = tmem_d + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(h * BM + cbase + 32 * i);
      x_ld32(taddr, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int m = m0 + cbase + 32 * i + j;
        if (m < a.M && n < a.N) {
          const size_t idx = (size_t)m * a.N + n;
          float out = __uint_as_float(v[j]) * a.xscale[m];
          if (a.r1) out += a.r1[(size_t)m * a.r1_stride + n];
          if (a.r2) out += a.r2[idx];
          a.y[idx] = out;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*dead) {  // a role gave up: copies and MMAs in flight are waited for, with a limit, before shared and tensor memory are free
    if (lane == 0 && warp == DQ_WARPS) {
      for (int i = max(0, issued - 2); i < issued; ++i) x_drain(bar_raw_full + 8 * (i & 1), (uint32_t)((i >> 1) & 1));
    } else if (lane == 0 && warp == DQ_WARPS + 1) {
      for (int i = max(0, issued - a.stages); i < issued; ++i) x_drain(bar_b_full + 8 * (i % a.stages), (uint32_t)((i / a.stages) & 1));
    } else if (lane == 0 && warp == DQ_WARPS + 2) {
      x_commit(bar_end);
      x_drain(bar_end, 0);
    }
    __syncthreads();
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "n"(TMEM_COLS) : "memory");
}

// x[M, K] f32 -> fp16 scaled by a power of two per row into (-64, 64), stored as [Mp / 128][K / 64]
// tiles of 128 rows x 64 values in the operand layout of the MMA (8 rows x 16 bytes per core
// matrix, core matrices adjacent in K 128 bytes apart, 8-row groups 1024 bytes apart), so that a
// tile is one contiguous bulk copy; rows >= M are zero. With NORM the rows are (x + res) / rms * w (RMSNorm; res may be null).
// Bound: latency of one read of the rows, HBM for many of them. A CTA takes ROWS rows and every thread all its values at once into
// registers (CHUNKS times 8 values; what is behind 14336 of a row is read again), so that the maximum, or sum of squares and
// maximum, cost no second pass; adjacent threads take the same place of the rows and write whole sectors.
// With two rows and the registers of 14336 values for every width one CTA fit an SM, and many narrow rows took longer than in two
// passes (times with a product of 64 columns behind it, two passes / that / now): 16384 rows of 512 values 32 / 91 / 26 us, of 1024
// 48 / 112 / 38, of 2048 69 / 124 / 61, of 4096 142 / 153 / 94; 512 rows of 4096 37 / 24 / 22.
constexpr int PACK_THREADS = 512, PACK_CHUNKS = 7;
template <int N> using PackInt = std::integral_constant<int, N>;
template <bool NORM, int ROWS, int CHUNKS>
__global__ void __launch_bounds__(PACK_THREADS, NORM ? (CHUNKS <= 2 ? 2 : 0) : CHUNKS == 1 ? 4 : CHUNKS == PACK_CHUNKS ? 1 : 0)
pack_rows16_kernel(const float* __restrict__ x, const float* __restrict__ res, const float* __restrict__ w, float eps, int M, int K,
                   __half* __restrict__ xh, float* __restrict__ xscale) {
  constexpr int STEP = PACK_THREADS / ROWS;
  __shared__ float part[2][PACK_THREADS / 32][ROWS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid % ROWS, c0 = tid / ROWS;
  const int m0 = blockIdx.x * ROWS, m = m0 + r, chunks = K / 8;
  pdl_launch_dependents_small();
  const bool in = m < M;
  const float4* xr = reinterpret_cast<const float4*>(x + (size_t)(in ? m : 0) * K);
  const float4* rr = NORM && res ? reinterpret_cast<const float4*>(res + (size_t)(in ? m : 0) * K) : nullptr;
  auto load = [&](int c, float4 (&v)[2]) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      v[e] = in && c < chunks ? __ldg(xr + 2 * c + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (NORM && rr && in && c < chunks) {
        const float4 q = __ldg(rr + 2 * c + e);
        v[e] = make_float4(v[e].x + q.x, v[e].y + q.y, v[e].z + q.z, v[e].w + q.w);
      }
    }
  };
  // over the threads of the own row: 32 / ROWS lanes of every warp
  auto block = [&](float v, int slot, bool sum) {
#pragma unroll
    for (int o = 16; o >= ROWS; o >>= 1) {
      const float other = __shfl_xor_sync(0xFFFFFFFFu, v, o);
      v = sum ? v + other : fmaxf(v, other);
    }
    if (lane < ROWS) part[slot][warp][lane] = v;
    __syncthreads();
    v = part[slot][0][r];
#pragma unroll
    for (int i = 1; i < PACK_THREADS / 32; ++i) v = sum ? v + part[slot][i][r] : fmaxf(v, part[slot][i][r]);
    return v;
  };
  float4 held[CHUNKS][2];
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) load(c0 + i * STEP, held[i]);
  float rms = 1.f;
  if (NORM) {
    auto squares = [](const float4 (&v)[2], float acc) {
#pragma unroll
      for (int e = 0; e < 2; ++e) acc = fmaf(v[e].x, v[e].x, fmaf(v[e].y, v[e].y, fmaf(v[e].z, v[e].z, fmaf(v[e].w, v[e].w, acc))));
      return acc;
    };
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) ss = squares(held[i], ss);
    for (int c = c0 + CHUNKS * STEP; c < chunks; c += STEP) {
      float4 v[2];
      load(c, v);
      ss = squares(v, ss);
    }
    rms = sqrtf(block(ss, 0, true) / (float)K + eps);
  }
  // a chunk as it is packed
  auto finish = [&](int c, float4 (&v)[2]) {
    if (!NORM || c >= chunks) return;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(w) + 2 * c + e);
      v[e] = make_float4((v[e].x / rms) * q.x, (v[e].y / rms) * q.y, (v[e].z / rms) * q.z, (v[e].w / rms) * q.w);
    }
  };
  auto biggest = [](const float4 (&v)[2], float acc) {
#pragma unroll
    for (int e = 0; e < 2; ++e) acc = fmaxf(fmaxf(acc, fmaxf(fabsf(v[e].x), fabsf(v[e].y))), fmaxf(fabsf(v[e].z), fabsf(v[e].w)));
    return acc;
  };
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    finish(c0 + i * STEP, held[i]);
    amax = biggest(held[i], amax);
  }
  for (int c = c0 + CHUNKS * STEP; c < chunks; c += STEP) {
    float4 v[2];
    load(c, v);
    finish(c, v);
    amax = biggest(v, amax);
  }
  amax = block(amax, 1, false);
  int ex = 0;
  if (amax > 0.f && amax < 3.0e38f) frexpf(amax, &ex);
  const float inv = ldexpf(64.0f, -ex);
  if (tid < ROWS) xscale[m] = ldexpf(1.0f, ex - 6);
  uint8_t* tile_row = reinterpret_cast<uint8_t*>(xh) + (size_t)(m0 / BM) * (K / BK) * ((size_t)BM * BK * 2) +
                      ((m0 % BM) >> 3) * CORE_SBO + (m & 7) * 16;
  auto store = [&](int c, const float4 (&v)[2]) {
    if (c >= chunks) return;
    *reinterpret_cast<uint4*>(tile_row + (size_t)(c >> 3) * ((size_t)BM * BK * 2) + (c & 7) * CORE_LBO) =
        make_uint4(h2u(__floats2half2_rn(v[0].x * inv, v[0].y * inv)), h2u(__floats2half2_rn(v[0].z * inv, v[0].w * inv)),
                   h2u(__floats2half2_rn(v[1].x * inv, v[1].y * inv)), h2u(__floats2half2_rn(v[1].z * inv, v[1].w * inv)));
  };
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) store(c0 + i * STEP, held[i]);
  for (int c = c0 + CHUNKS * STEP; c < chunks; c += STEP) {
    float4 v[2];
    load(c, v);
    finish(c, v);
    store(c, v);
  }
}

template <int TYPE>
int launch_tc_type(fb200_device* dev, const TcArgs& a, unsigned grid_n, unsigned grid_m, int smem) {
  static bool configured[64] = {false};
  if (!configured[dev->ordinal & 63]) {
    FB_CUDA(dev, cudaFuncSetAttribute(qgemm_tc_kernel<TYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BUDGET));
    configured[dev->ordinal & 63] = true;
  }
  return fb200_launch(dev, qgemm_tc_kernel<TYPE>, dim3(grid_n, grid_m), dim3(THREADS), (size_t)smem, false, a);
}

int launch_tc(fb200_device* dev, const TcArgs& a, unsigned grid_n, unsigned grid_m, int smem) {
  switch (a.type) {
    case FB200_Q4_0: return launch_tc_type<FB200_Q4_0>(dev, a, grid_n, grid_m, smem);
    case FB200_Q8_0: return launch_tc_type<FB200_Q8_0>(dev, a, grid_n, grid_m, smem);
    case FB200_Q4_K: return launch_tc_type<FB200_Q4_K>(dev, a, grid_n, grid_m, smem);
    case FB200_Q6_K: return launch_tc_type<FB200_Q6_K>(dev, a, grid_n, grid_m, smem);
  }
  return 1;
}

// How one product runs: on CTA pairs (qgemm_pair.cu, tiles of 256 activation rows by nw = 128 or 256 weight rows), or on
// single CTAs (nw = 0; 256 weight rows by 128 activation rows, `stages` operand stages); split = K ranges side by side.
struct TcShape { int nw = 0, stages = 0, split = 1; size_t ctas = 0; double ns = 0; };

// Cost model in ns, a fit to 40..2048 rows of Llama-8B-shaped matrices: time of one tile per 256 values of K, and beside its K
// loop. At 512 rows 28672 x 4096 Q4_K with SwiGLU takes 118 / 121 us on pairs (nw = 256 / 128) and 224 us on single CTAs,
// 4096 x 14336 Q6_K 124 / 87 / 235 us. Single CTAs win where the pairs need one round more: up to 128 rows of many weight rows
// (100 rows of 28672 x 4096: 63.6 us, pairs 70.1).
double tile_ns(const fb200_qmatrix* w, const TcShape& sh) {
  const double k256 = (double)w->k / 256.0 / sh.split;
  return sh.nw == 256 ? k256 * 1700.0 + 2500.0 : sh.nw ? k256 * 1050.0 + 1500.0 : k256 * 3300.0;
}

// Fills in what follows from nw / split; false when the shape does not fit.
bool tc_shape(const fb200_device* dev, const fb200_qmatrix* w, const TileGeom& geo, size_t m, int swiglu, TcShape* sh) {
  const size_t n_rows = swiglu ? w->n / 2 : w->n;  // weight rows along the grid
  size_t rows, tiles_m, slots;
  if (sh->nw) {
    rows = (size_t)(swiglu ? sh->nw / 2 : sh->nw);
    tiles_m = (m + 255) / 256;
    slots = (size_t)dev->sm_count / 2;
  } else {
    const int raw_stride = (geo.tg_bytes + 127) & ~127, stage = NH * A_HALF + BM * BK * 2;
    sh->stages = std::min(MAX_STAGES, (SMEM_BUDGET - TAIL_BYTES - 2 * 8 * NH * raw_stride) / stage);
    if (sh->stages < 2) return false;
    rows = (size_t)(swiglu ? BN : BN * NH);
    tiles_m = (m + BM - 1) / BM;
    slots = (size_t)dev->sm_count;
  }
  sh->ctas = ((n_rows + rows - 1) / rows) * tiles_m * sh->split;
  sh->ns = 9000.0 + (double)((sh->ctas + slots - 1) / slots) * tile_ns(w, *sh);  // packing, launches, filling the pipeline
  if (sh->split > 1) {  // the ranges' partial products and the adding kernel
    const double out_bytes = (double)m * (double)w->n * 4.0;
    sh->ns += sh->split * out_bytes / 3000.0 + 2000.0 + (sh->split + 1) * out_bytes / 7000.0;
  }
  return true;
}

// FB200_TC_TILE="BM,NH" or "BM,NH,SPLIT": "256,2" / "256,1" pairs with 256 / 128 weight rows, "128,2" single CTAs, in SPLIT ranges
// of K (1 if not given). A combination that there is not, or that the product cannot take, leaves the choice to the model.
struct TcForce { int nw = -1, split = 1; };  // nw < 0: nothing is forced
TcForce tc_force() {
  TcForce f;
  int bm = 0, nh = 0;
  const char* cfg = getenv("FB200_TC_TILE");
  if (!cfg || sscanf(cfg, "%d,%d,%d", &bm, &nh, &f.split) < 2) return f;
  if (bm == 256 && (nh == 1 || nh == 2)) f.nw = 128 * nh;
  else if (bm == BM && nh == NH) f.nw = 0;
  return f;
}

bool tc_covers(const fb200_qmatrix* w, const float* x, size_t m, TileGeom* geo) {
  static const bool enabled = !(getenv("FB200_TCGEN05") && getenv("FB200_TCGEN05")[0] == '0');
  if (!enabled || !w->tiled || !tile_geom(w->type, geo)) return false;
  const size_t kp = (size_t)w->ngroups * geo->group_elems;
  if (kp != w->k || m > (1u << 20)) return false;  // K is a whole number of K groups
  return (reinterpret_cast<uintptr_t>(x) & 15) == 0;
}

// y = p[0] + p[1] + .. (+ r1 + r2): the partial products of a split-K launch, added in split order.
__global__ void __launch_bounds__(256)
splitk_add_kernel(const float4* __restrict__ parts, int nsplit, size_t n4, int ncols4, const float* __restrict__ r1,
                  int r1_stride, const float* __restrict__ r2, float4* __restrict__ y) {
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  float4 acc = __ldg(parts + i);
  for (int s = 1; s < nsplit; ++s) {
    const float4 v = __ldg(parts + (size_t)s * n4 + i);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  if (r1) {
    const size_t m = i / (size_t)ncols4, c = i - m * (size_t)ncols4;
    const float4 v = __ldg(reinterpret_cast<const float4*>(r1 + m * (size_t)r1_stride) + c);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  if (r2) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(r2) + i);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  y[i] = acc;
}

// Launches the product of packed rows (xh, xscale: pack_rows16_kernel with 128-row tiles) on dev->stream.
// With sh.split > 1 every K range writes its partial product into the handle's split-K scratch (tc_parts) and a second kernel
// adds them (+ residuals). `early`: the packing kernel is the last work on the stream, and the product may start beside it.
int tc_launch(fb200_device* dev, const fb200_qmatrix* w, const TileGeom& geo, const TcShape& sh, const __half* xh,
              const float* xscale, size_t m, float* y, bool r1_is_bias, const float* r1, const float* r2, int swiglu, bool early) {
  const int halves = (int)((m + 127) / 128), split = sh.split;
  const size_t n_rows = swiglu ? w->n / 2 : w->n;
  int rc;
  if (sh.nw) {
    PairArgs a = {};
    a.w = w->data; a.xh = xh; a.xscale = xscale; a.y = y; a.r1 = r1; a.r2 = r2; a.r1_stride = r1_is_bias ? 0 : (int)w->n;
    a.M = (int)m; a.N = (int)w->n; a.ngroups = w->ngroups; a.ntiles = w->ntiles; a.pair_tiles = swiglu ? w->ntiles / 2 : 0;
    const int rows = swiglu ? sh.nw / 2 : sh.nw;
    a.m_tiles = (halves + 1) / 2; a.n_tiles = (int)((n_rows + rows - 1) / rows);
    a.kg_per = (w->ngroups + split - 1) / split;
    a.splits = (w->ngroups + a.kg_per - 1) / a.kg_per;  // every range holds at least one K group
    a.x_halves = halves; a.status = dev->status;
    if (split > 1) {
      a.y = reinterpret_cast<float*>(dev->splitk);
      a.r1 = a.r2 = nullptr;
    }
    a.vec = n_rows % 2 == 0 && ((reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.r1) | reinterpret_cast<uintptr_t>(a.r2)) & 7) == 0;
    rc = fb200_qgemm_pair(dev, sh.nw, w->type, a, early);
    if (rc || split == 1) return rc;
    const size_t n4 = m * w->n / 4;
    splitk_add_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, dev->stream>>>(
        reinterpret_cast<const float4*>(a.y), a.splits, n4, (int)(w->n / 4), r1, r1_is_bias ? 0 : (int)w->n, r2,
        reinterpret_cast<float4*>(y));
    FB_LAUNCH_CHECK(dev);
    return FB200_OK;
  }
  const int raw_stride = (geo.tg_bytes + 127) & ~127;
  TcArgs a;
  a.w = w->data; a.xh = xh; a.xscale = xscale; a.y = y; a.r1 = r1; a.r2 = r2;
  a.r1_stride = r1_is_bias ? 0 : (int)w->n;
  a.M = (int)m; a.N = (int)w->n; a.K = (int)w->k;
  a.ngroups = w->ngroups; a.ntiles = w->ntiles; a.type = (int)w->type; a.tgb = geo.tg_bytes;
  a.group_elems = geo.group_elems; a.status = dev->status;
  a.stages = sh.stages; a.raw_stride = raw_stride;
  a.pair_tiles = swiglu ? w->ntiles / 2 : 0;
  const int smem = sh.stages * (NH * A_HALF + BM * BK * 2) + 2 * 8 * NH * raw_stride + TAIL_BYTES;
  const size_t rows_per_cta = swiglu ? BN : BN * NH;
  const unsigned gn = (unsigned)((n_rows + rows_per_cta - 1) / rows_per_cta), gm = (unsigned)halves;
  return launch_tc(dev, a, gn, gm, smem);
}

// Scratch of packed rows: fp16 tiles of 128 rows, then the row scales
int tc_reserve(fb200_device* dev, size_t m, size_t k) {
  const size_t mp = (m + 127) / 128 * 128;
  return fb200_ensure(dev, &dev->xpack, &dev->xpack_bytes, mp * k * 2 + mp * sizeof(float));
}

// Scratch of a split's partial products. A budget or a card without room for them is not an error: the product then runs unsplit.
bool tc_parts(fb200_device* dev, const fb200_qmatrix* w, size_t m, int split) {
  if (fb200_ensure(dev, &dev->splitk, &dev->splitk_bytes, (size_t)split * m * w->n * sizeof(float)) == FB200_OK) return true;
  cudaGetLastError();  // a refused allocation is not the next launch's error
  return false;
}

// x (under `norm`, if given) -> fp16 tiles and row scales in the handle's scratch
int tc_pack(fb200_device* dev, const float* x, size_t m, size_t k, const fb200_row_norm* norm, const __half** xh, const float** xscale) {
  const int mp = (int)((m + 127) / 128) * 128;
  const size_t xbytes = (size_t)mp * k * 2;
  int rc = tc_reserve(dev, m, k);
  if (rc) return rc;
  __half* h = reinterpret_cast<__half*>(dev->xpack);
  float* s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(dev->xpack) + xbytes);
  auto launch = [&](auto plain_rows, auto chunks) {
    constexpr int R = decltype(plain_rows)::value, C = decltype(chunks)::value;
    if (norm) pack_rows16_kernel<true, 2, C><<<mp / 2, PACK_THREADS, 0, dev->stream>>>(x, norm->res, norm->w, norm->eps, (int)m, (int)k, h, s);
    else pack_rows16_kernel<false, R, C><<<mp / R, PACK_THREADS, 0, dev->stream>>>(x, nullptr, nullptr, 0.f, (int)m, (int)k, h, s);
  };
  // as many registers as a thread of this width has values, several narrow rows to a CTA
  if (k <= 512) launch(PackInt<8>(), PackInt<1>());
  else if (k <= 1024) launch(PackInt<4>(), PackInt<1>());
  else if (k <= 2048) launch(PackInt<2>(), PackInt<1>());
  else if (k <= 4096) launch(PackInt<2>(), PackInt<2>());
  else if (k <= 8192) launch(PackInt<2>(), PackInt<4>());
  else launch(PackInt<2>(), PackInt<PACK_CHUNKS>());
  FB_LAUNCH_CHECK(dev);
  *xh = h;
  *xscale = s;
  return FB200_OK;
}

// 16-byte loads of the norm's weights and residual
bool norm_covers(const fb200_row_norm* norm) {
  return !norm || ((reinterpret_cast<uintptr_t>(norm->w) | reinterpret_cast<uintptr_t>(norm->res)) & 15) == 0;
}

}  // namespace

bool fb200_qgemm_covers(const fb200_qmatrix* w, const float* x, size_t m, const fb200_row_norm* norm) {
  TileGeom geo;
  return tc_covers(w, x, m, &geo) && norm_covers(norm);
}

// y[M, N] = x[M, K] . W^T (+ r1 + r2) for M > 32; with `swiglu`, W stacks gate rows over up rows
// and y[M, N / 2] = silu(gate) * up. Returns 1 when the shape is not covered (the
// caller falls back to the small-batch kernel in chunks of 32 rows).
int fb200_qgemm(fb200_device* dev, const fb200_qmatrix* w, const float* x, size_t m, float* y, bool r1_is_bias, const float* r1,
                const float* r2, int swiglu, const fb200_row_norm* norm) {
  TileGeom geo;
  if (!tc_covers(w, x, m, &geo) || !norm_covers(norm)) return 1;
  // A split of K (plain and residual epilogues, 16-byte aligned outputs, at least 2048 values of K per range) fills the
  // SMs where there are few tiles; it has to promise a tenth less, and runs only where the scratch for its partial products fits.
  static const bool no_split = getenv("FB200_TC_SPLITK") && getenv("FB200_TC_SPLITK")[0] == '0';
  const bool may_split = !no_split && !swiglu && w->n % 4 == 0 &&
                         ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(r1) | reinterpret_cast<uintptr_t>(r2)) & 15) == 0;
  TcShape best, whole;  // whole: the best without a split
  const TcForce force = tc_force();
  for (int split = 1; split <= (may_split ? 4 : 1); split *= 2) {
    if (split > 1 && (w->k / split < 2048 || w->ngroups < 2 * split)) break;
    bool done = false;
    for (int nw = 256; nw >= (split > 1 ? 128 : 0) && !done; nw -= 128) {
      TcShape sh;
      sh.nw = nw; sh.split = split;
      if (!tc_shape(dev, w, geo, m, swiglu, &sh)) continue;
      done = nw == force.nw && split == force.split;
      if (done || !best.ctas || sh.ns < (split > 1 ? 0.9 : 1.0) * best.ns) best = sh;
    }
    if (split == 1) whole = best;
    if (done) break;
  }
  if (!best.ctas) return 1;
  int rc = tc_reserve(dev, m, w->k);  // what the product needs comes before what it can do without
  if (rc) return rc;
  if (best.split > 1 && !tc_parts(dev, w, m, best.split)) best = whole;
  const __half* xh;
  const float* xscale;
  rc = tc_pack(dev, x, m, w->k, norm, &xh, &xscale);
  return rc ? rc : tc_launch(dev, w, geo, best, xh, xscale, m, y, r1_is_bias, r1, r2, swiglu, true);
}

// Up to three products of the same rows (the q, k and v projections of a prompt pass):
// ys[i][M, N_i] = x[M, K] . W_i^T. One of them alone leaves most SMs idle (a 1024-row matrix at
// 512 rows is 16..32 CTA tiles, each walking the whole K), so the rows are packed once and the
// products run side by side: the first on the handle's stream, the others on side streams forked
// behind the packing kernel and joined again before the call returns to the stream. Returns 1 when
// the shapes are not covered (the caller issues the products one after the other).
int fb200_qgemm_group(fb200_device* dev, const fb200_qmatrix* const* ws, float* const* ys, int n, const float* x, size_t m,
                      const fb200_row_norm* norm) {
  static const bool off = getenv("FB200_TC_GROUP") && getenv("FB200_TC_GROUP")[0] == '0';
  if (off || n < 2 || n > 3 || m <= 32 || getenv("FB200_TC_TILE") || !norm_covers(norm)) return 1;
  TileGeom geo[3];
  for (int i = 0; i < n; ++i)
    if (!ws[i] || !tc_covers(ws[i], x, m, &geo[i]) || ws[i]->k != ws[0]->k) return 1;
  // one kind of tile for all; cost = rounds of all CTAs together x the time of the slowest tile
  TcShape best[3];
  double best_ns = 0;
  for (int nw = 256; nw >= 128; nw -= 128) {
    TcShape sh[3];
    double slowest = 0;
    size_t ctas = 0;
    bool ok = true;
    for (int i = 0; i < n && ok; ++i) {
      sh[i].nw = nw;
      ok = tc_shape(dev, ws[i], geo[i], m, 0, &sh[i]);
      ctas += sh[i].ctas;
      slowest = std::max(slowest, tile_ns(ws[i], sh[i]));
    }
    const size_t slots = (size_t)dev->sm_count / 2;
    const double ns = (double)((ctas + slots - 1) / slots) * slowest;
    if (ok && (best_ns == 0 || ns < best_ns)) { best_ns = ns; for (int i = 0; i < n; ++i) best[i] = sh[i]; }
  }
  if (best_ns == 0) return 1;
  for (int i = 0; i < n - 1; ++i) {
    if (!dev->side_stream[i]) FB_CUDA(dev, cudaStreamCreateWithFlags(&dev->side_stream[i], cudaStreamNonBlocking));
    if (!dev->join_ev[i]) FB_CUDA(dev, cudaEventCreateWithFlags(&dev->join_ev[i], cudaEventDisableTiming));
  }
  if (!dev->fork_ev) FB_CUDA(dev, cudaEventCreateWithFlags(&dev->fork_ev, cudaEventDisableTiming));
  const __half* xh;
  const float* xscale;
  int rc = tc_pack(dev, x, m, ws[0]->k, norm, &xh, &xscale);
  if (rc) return rc;
  FB_CUDA(dev, cudaEventRecord(dev->fork_ev, dev->stream));
  cudaStream_t main_stream = dev->stream;
  // the largest product stays on the handle's stream
  int first = 0;
  for (int i = 1; i < n; ++i) if (best[i].ctas > best[first].ctas) first = i;
  int side = 0;
  for (int i = 0; i < n && !rc; ++i) {
    if (i == first) continue;
    cudaStream_t st = dev->side_stream[side];
    FB_CUDA(dev, cudaStreamWaitEvent(st, dev->fork_ev, 0));
    dev->stream = st;  // the launch helpers take the handle's stream
    rc = tc_launch(dev, ws[i], geo[i], best[i], xh, xscale, m, ys[i], false, nullptr, nullptr, 0, false);  // (its stream's last work is a wait for an event, not the packing kernel)
    dev->stream = main_stream;
    if (!rc) {
      FB_CUDA(dev, cudaEventRecord(dev->join_ev[side], st));
      ++side;
    }
  }
  if (!rc) rc = tc_launch(dev, ws[first], geo[first], best[first], xh, xscale, m, ys[first], false, nullptr, nullptr, 0, false);
  // join whatever was forked, also after a failed launch: the stream must not run ahead of its side streams
  for (int j = 0; j < side; ++j) FB_CUDA(dev, cudaStreamWaitEvent(main_stream, dev->join_ev[j], 0));
  return rc;
}
