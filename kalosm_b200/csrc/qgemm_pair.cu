// Prefill product on CTA pairs: Y = X . W^T with X in the M role (256 rows per pair) and the dequantised weights in
// the N role, tcgen05.mma.cta_group::2 with the accumulators in tensor memory.
//
// Bound: tensor cores (2 M N K flops). The single-CTA kernel (qgemm.cu) holds W in the M role: a CTA converts 256
// weight rows for 128 activation rows (once 256), its raw buffers leave few operand stages, and every MMA waits for the round
// trip of one of them. Here a CTA of the pair converts half of the weight rows, and the pair's MMA reads both halves: a tile of
// 256 x 256 costs a CTA half of the conversion and half of the operand reads of W, and the raw bytes go from global memory
// straight into the registers of the lane that converts them, so three stages of 128 values of K fit (four with 128 weight rows).
//
// The grid is persistent: a pair walks over tiles (activation tiles fastest, so that the pairs that run together share
// their weight rows in L2), with two accumulators per CTA: the epilogue of a tile runs beside the MMAs of the next.
//  * conversion (16 warps): a unit is 16 weight rows x 128 values of K, a warp's part of one stage. A lane owns one row and 16
//    consecutive values of a 32-value block; it loads its bytes one unit ahead, dequantises (byte -> 1024 + byte by a
//    byte permute, exact subtraction, one fused multiply-add with block scale and offset), and writes 16-byte core-matrix
//    rows; eight lanes write 128 consecutive bytes.
//  * activation loader (one thread): one bulk copy of 32 KB per stage, packed rows in the operand layout.
//  * issuer (one warp): in the even CTA eight MMAs (M = 256, N = NW, K = 16) per stage; in the odd CTA it passes "stage
//    full" on to the even one. tcgen05.commit frees the stage in both CTAs.
//  * epilogue (4 warps): tcgen05.ld, row scale, residuals or SwiGLU (gate and up values of an output sit in one lane,
//    NW / 2 columns apart), whole 32-byte sectors per row.
// Every wait is bounded (2^22 polls); a role that gives up sets the status word and a flag that makes the roles of its
// CTA leave (those of the other CTA follow by their own limits); copies and MMAs in flight are waited for, with a limit, and the
// cluster barrier before the release of the TMEM columns keeps either CTA alive while the other may still reach it.
#include <algorithm>

#include "half_weights.cuh"
#include "qgemm_pair.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int PAIR_M = 256, PAIR_BK = 64;        // an operand block is 64 values of K wide; a stage holds two (one unit)
constexpr int PAIR_CONV_WARPS = 16, PAIR_EPI_WARPS = 4;
constexpr int PAIR_THREADS = (PAIR_CONV_WARPS + PAIR_EPI_WARPS + 2) * 32;
constexpr int PAIR_A_BLOCK = 128 * PAIR_BK * 2, PAIR_A_BYTES = 2 * PAIR_A_BLOCK;  // activation rows of one CTA: block, stage
constexpr int PAIR_MAX_STAGES = 4;
constexpr int PAIR_TAIL = 512;

template <int NW>
struct Pair {
  static constexpr int TILES = NW / 32;                  // 16-row tiles that one CTA converts
  static constexpr int SETS = PAIR_CONV_WARPS / TILES;   // units in conversion at a time
  static constexpr int B_BLOCK = NW / 2 * PAIR_BK * 2;
  static constexpr int STAGE = PAIR_A_BYTES + 2 * B_BLOCK;
  static constexpr int STAGES = NW == 256 ? 3 : 4;
  static constexpr int COLS = 2 * NW;                    // two accumulators
  static constexpr int SMEM = STAGES * STAGE + PAIR_TAIL;
  // instruction descriptor: fp32 accumulator, fp16 A and B, both K-major, N = NW, M = 256 over the pair
  static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NW >> 3) << 17) | ((uint32_t)(PAIR_M >> 4) << 24);
};

__device__ __forceinline__ uint4 p_ldg(const uint8_t* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint2 p_ldg8(const uint8_t* p) { return __ldg(reinterpret_cast<const uint2*>(p)); }

__device__ __forceinline__ void p_store8(uint8_t* dst, uint32_t w0, uint32_t w1, __half2 centre, __half2 scale, __half2 offset) {
  const uint2 a = deq4(w0, centre, scale, offset), b = deq4(w1, centre, scale, offset);
  *reinterpret_cast<uint4*>(dst) = make_uint4(a.x, a.y, b.x, b.y);
}

// What a lane holds of one unit: row g + 8 h of a 16-row tile, piece i (lane = g + 8 h + 16 i).
//  Q4_K: the 16 bytes of values 16 i .. of two block pairs (low nibbles: block 2 p, high: 2 p + 1), row header
//  Q6_K: low nibbles of two blocks and the two-bit planes of values 16 i .., half of the row's scales, d
//  Q8_0: values 16 i .. of four blocks, four scales;  Q4_0: blocks i and 2 + i whole, four scales
template <int TYPE> struct Raw;
template <> struct Raw<FB200_Q4_K> { uint4 q[2], head; int odd; };
template <> struct Raw<FB200_Q6_K> { uint4 q[2], hi; uint2 sc; uint16_t d; };
template <> struct Raw<FB200_Q8_0> { uint4 q[4]; uint2 sc; };
template <> struct Raw<FB200_Q4_0> { uint4 q[2]; uint2 sc; };

// unit u of a row-tile whose tile-groups start at `tile`
template <int TYPE>
__device__ __forceinline__ void load_unit(Raw<TYPE>& r, const uint8_t* tile, int u, int g, int h, int i) {
  if constexpr (TYPE == FB200_Q4_K) {
    const uint8_t* tg = tile + (size_t)(u >> 1) * 2304;
    const uint8_t* p = tg + (((u & 1) * 2 + h) * 2 + i) * 256 + g * 32;
    r.q[0] = p_ldg(p);
    r.q[1] = p_ldg(p + 16);
    r.head = p_ldg(tg + 2048 + (g + 8 * h) * 16);
    r.odd = u & 1;
  } else if constexpr (TYPE == FB200_Q6_K) {
    const uint8_t* tg = tile + (size_t)(u >> 1) * 3360;
    const int part = ((u & 1) * 2 + i) * 2 + h;
    r.q[0] = p_ldg(tg + part * 256 + g * 32);
    r.q[1] = p_ldg(tg + part * 256 + g * 32 + 16);
    r.hi = p_ldg(tg + 2048 + part * 128 + g * 16);
    r.sc = p_ldg8(tg + 3072 + (g + 8 * h) * 16 + 8 * (u & 1));
    r.d = __ldg(reinterpret_cast<const uint16_t*>(tg + 3328 + (g + 8 * h) * 2));
  } else if constexpr (TYPE == FB200_Q8_0) {
    const uint8_t* tg = tile + (size_t)u * 2176;
    const uint8_t* p = tg + (h * 2 + i) * 512 + g * 64;
#pragma unroll
    for (int c = 0; c < 4; ++c) r.q[c] = p_ldg(p + 16 * c);
    r.sc = p_ldg8(tg + 2048 + (g + 8 * h) * 8);
  } else {
    const uint8_t* tg = tile + (size_t)u * 1152;
    const uint8_t* p = tg + h * 512 + g * 64 + i * 16;
    r.q[0] = p_ldg(p);
    r.q[1] = p_ldg(p + 32);
    r.sc = p_ldg8(tg + 1024 + (g + 8 * h) * 8);
  }
}

// block b (64 values of K) of the unit -> operand rows; `dst` is row g + 8 h of the tile at K = 0 of the block
template <int TYPE>
__device__ __forceinline__ void convert_block(const Raw<TYPE>& r, int b, int i, uint8_t* dst) {
  const __half2 zero2 = __float2half2_rn(0.f);
  if constexpr (TYPE == FB200_Q4_K) {
    const float d = fb::half_bits_to_float((uint16_t)(r.head.x & 0xFFFF)), dmin = fb::half_bits_to_float((uint16_t)(r.head.x >> 16));
    const uint32_t s0 = r.head.y, s1 = r.head.z, s2 = r.head.w;
    uint32_t sc = r.odd ? (s2 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u) : s0 & 0x3F3F3F3Fu;
    uint32_t mn = r.odd ? ((s2 >> 4) & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u) : s1 & 0x3F3F3F3Fu;
    sc >>= 16 * b;
    mn >>= 16 * b;
    const __half2 ctr = __float2half2_rn(1024.0f);
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const __half2 s = __float2half2_rn(d * (float)((sc >> (8 * hi)) & 0xFF));
      const __half2 o = __float2half2_rn(-(dmin * (float)((mn >> (8 * hi)) & 0xFF)));
      const uint4 q = r.q[b];
      uint8_t* p = dst + (hi * 4 + i * 2) * 128;
      p_store8(p, (q.x >> (4 * hi)) & 0x0F0F0F0Fu, (q.y >> (4 * hi)) & 0x0F0F0F0Fu, ctr, s, o);
      p_store8(p + 128, (q.z >> (4 * hi)) & 0x0F0F0F0Fu, (q.w >> (4 * hi)) & 0x0F0F0F0Fu, ctr, s, o);
    }
  } else if constexpr (TYPE == FB200_Q6_K) {
    const float d = fb::half_bits_to_float(r.d);
    const __half2 ctr = __float2half2_rn(1056.0f);  // (q - 32) d scale
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // 32-value block 2 b + c of the unit: nibble b of plane c, bits 4 b + 2 c of the two-bit plane
      const int q = 2 * b + c, grp = 2 * q + i;
      const uint32_t scw = q < 2 ? r.sc.x : r.sc.y;
      const __half2 s = __float2half2_rn(d * (float)(int)(int8_t)((scw >> (8 * (grp & 3))) & 0xFF));
      const uint4 lo = r.q[c];
      uint32_t w[4] = {lo.x, lo.y, lo.z, lo.w};
      const uint32_t hv[4] = {r.hi.x, r.hi.y, r.hi.z, r.hi.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t hb = q == 0 ? hv[j] << 4 : q == 1 ? hv[j] << 2 : q == 2 ? hv[j] : hv[j] >> 2;
        w[j] = ((w[j] >> (4 * b)) & 0x0F0F0F0Fu) | (hb & 0x30303030u);
      }
      uint8_t* p = dst + (c * 4 + i * 2) * 128;
      p_store8(p, w[0], w[1], ctr, s, zero2);
      p_store8(p + 128, w[2], w[3], ctr, s, zero2);
    }
  } else if constexpr (TYPE == FB200_Q8_0) {
    const __half2 ctr = __float2half2_rn(1152.0f);  // signed byte b as (b ^ 0x80) - 128
    const uint32_t scw = b ? r.sc.y : r.sc.x;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const __half2 s = __half2half2(__ushort_as_half((uint16_t)(scw >> (16 * c))));
      const uint4 q = r.q[2 * b + c];
      uint8_t* p = dst + (c * 4 + i * 2) * 128;
      p_store8(p, q.x ^ 0x80808080u, q.y ^ 0x80808080u, ctr, s, zero2);
      p_store8(p + 128, q.z ^ 0x80808080u, q.w ^ 0x80808080u, ctr, s, zero2);
    }
  } else {
    const __half2 ctr = __float2half2_rn(1032.0f);  // (q - 8) d
    const uint32_t scw = b ? r.sc.y : r.sc.x;
    const __half2 s = __half2half2(__ushort_as_half((uint16_t)(scw >> (16 * i))));
    const uint4 q = r.q[b];
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      uint8_t* p = dst + (i * 4 + hi * 2) * 128;
      p_store8(p, (q.x >> (4 * hi)) & 0x0F0F0F0Fu, (q.y >> (4 * hi)) & 0x0F0F0F0Fu, ctr, s, zero2);
      p_store8(p + 128, (q.z >> (4 * hi)) & 0x0F0F0F0Fu, (q.w >> (4 * hi)) & 0x0F0F0F0Fu, ctr, s, zero2);
    }
  }
}

// One tile of work: activation tile, weight tile, K range.
struct Item { int mt, nt, kg0, units; };
__device__ __forceinline__ Item item_of(const PairArgs& a, int item, int units_per_group) {
  const int per_z = a.m_tiles * a.n_tiles, z = item / per_z, rest = item - z * per_z;
  Item t;
  t.nt = rest / a.m_tiles;
  t.mt = rest - t.nt * a.m_tiles;
  t.kg0 = z * a.kg_per;
  t.units = min(a.kg_per, a.ngroups - t.kg0) * units_per_group;
  return t;
}

template <int NW, int TYPE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
qgemm_pair_kernel(const PairArgs a) {
  using P = Pair<NW>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P::STAGES * P::STAGE);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * PAIR_MAX_STAGES + 5);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank(), pair = (int)blockIdx.x >> 1, npairs = (int)gridDim.x >> 1;
  const uint32_t full = smem_u32(bars), stage_free = full + 8 * PAIR_MAX_STAGES, acc_full = stage_free + 8 * PAIR_MAX_STAGES,
                 acc_free = acc_full + 16, drained = acc_free + 16;
  constexpr int UPG = TYPE == FB200_Q4_K || TYPE == FB200_Q6_K ? 2 : 1;  // units per K group
  constexpr int TGB = TYPE == FB200_Q4_K ? 2304 : TYPE == FB200_Q6_K ? 3360 : TYPE == FB200_Q8_0 ? 2176 : 1152;
  const int items = a.m_tiles * a.n_tiles * a.splits;

  if (tid == 0) {
    *dead = 0;
    for (int i = 0; i < P::STAGES; ++i) {
      // the activations, the converted row-tiles, and in the even CTA the word that the odd one has both
      mbar_init(full + 8 * i, 1 + P::TILES + (rank == 0 ? 1 : 0));
      mbar_init(stage_free + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_free + 8 * i, 2 * PAIR_EPI_WARPS);
    }
    mbar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) pair_tmem_alloc(smem_u32(tmem_slot), P::COLS);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp < PAIR_CONV_WARPS) {
    // ---- conversion: row-tile warp % TILES of this CTA's half, every SETS-th unit
    const int tl = warp % P::TILES, set = warp / P::TILES;
    const int g = lane & 7, h = (lane >> 3) & 1, i = lane >> 4;
    uint8_t* const rows = smem + PAIR_A_BYTES + (2 * tl + h) * 1024 + g * 16;
    int item = pair, u = set, units = 0;
    const uint8_t* src = nullptr;  // null: the matrix has no such rows
    auto enter = [&]() {
      const Item t = item_of(a, item, UPG);
      units = t.units;
      const int local = t.nt * (a.pair_tiles ? P::TILES : 2 * P::TILES) + (a.pair_tiles ? 0 : rank * P::TILES) + tl;
      const int tile = local + (a.pair_tiles ? rank * a.pair_tiles : 0);
      src = local < (a.pair_tiles ? a.pair_tiles : a.ntiles) ? a.w + ((size_t)tile * a.ngroups + t.kg0) * TGB : nullptr;
    };
    auto settle = [&]() {  // u may lie behind the end of its tile
      while (item < items && u >= units) {
        u -= units;
        item += npairs;
        if (item < items) enter();
      }
    };
    if (item < items) enter();
    settle();
    Raw<TYPE> cur = {}, next = {};
    bool have = item < items, mine = have && src, alive = true;
    if (mine) load_unit<TYPE>(cur, src, u, g, h, i);
    for (int n = set; have && alive; n += P::SETS) {
      u += P::SETS;
      settle();
      const bool have_next = item < items, mine_next = have_next && src;
      if (mine_next) load_unit<TYPE>(next, src, u, g, h, i);
      const int s = n % P::STAGES, round = n / P::STAGES;
      if (round > 0 && !(alive = w_wait(stage_free + 8 * s, (uint32_t)((round - 1) & 1), dead, a.status))) break;
      if (mine) {
#pragma unroll
        for (int b = 0; b < 2; ++b) convert_block<TYPE>(cur, b, i, rows + s * P::STAGE + b * P::B_BLOCK);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> tensor-core reads
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * s);
      cur = next;
      have = have_next;
      mine = mine_next;
    }
  } else if (warp < PAIR_CONV_WARPS + PAIR_EPI_WARPS) {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. of this CTA's 128 activation rows
    const int quad = warp & 3;
    int n = 0;
    pdl_wait();
    for (int item = pair; item < items; item += npairs, ++n) {
      const int buf = n & 1;
      if (!w_wait(acc_full + 8 * buf, (uint32_t)((n >> 1) & 1), dead, a.status)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const Item t = item_of(a, item, UPG);
      const int m_first = t.mt * PAIR_M + rank * 128 + quad * 32;
      const int n_out = a.pair_tiles ? a.pair_tiles * 16 : a.N;
      const int c_first = t.nt * (a.pair_tiles ? NW / 2 : NW);
      float* const y = a.y + (size_t)(t.kg0 / a.kg_per) * a.M * a.N;
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        const int mrow = m_first + 16 * hh + (lane >> 2);  // and eight rows further
        if (m_first + 16 * hh >= a.M) break;
        const float xs[2] = {mrow < a.M ? __ldg(a.xscale + mrow) : 0.f, mrow + 8 < a.M ? __ldg(a.xscale + mrow + 8) : 0.f};
        const uint32_t tl = tmem + ((uint32_t)(32 * quad + 16 * hh) << 16) + (uint32_t)(buf * NW);
        auto put = [&](int e2, int col, float v0, float v1) {  // columns col, col + 1 of row mrow + 8 e2
          const int m = mrow + 8 * e2;
          if (m >= a.M) return;
          const size_t idx = (size_t)m * n_out + col;
          if (a.vec && col + 1 < n_out) {
            *reinterpret_cast<float2*>(y + idx) = make_float2(v0, v1);
          } else {
            if (col < n_out) y[idx] = v0;
            if (col + 1 < n_out) y[idx + 1] = v1;
          }
        };
        if (a.pair_tiles) {
#pragma unroll 1
          for (int c0 = 0; c0 < NW / 2 && c_first + c0 < n_out; c0 += 32) {
            uint32_t gv[16], uv[16];
            __syncwarp();
            x_ld16x256_32(tl + (uint32_t)c0, gv);
            x_ld16x256_32(tl + (uint32_t)(NW / 2 + c0), uv);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int e2 = j & 1, at = 4 * (j >> 1) + 2 * e2;
              float o[2];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                // silu(gate) * up, fusor-ml/fusor/src/composite/activations.rs:47-64: x / (1 + exp(-x))
                const float gate = __uint_as_float(gv[at + e]) * xs[e2];
                o[e] = (gate / (1.0f + expf(-gate))) * (__uint_as_float(uv[at + e]) * xs[e2]);
              }
              put(e2, c_first + c0 + 8 * (j >> 1) + 2 * (lane & 3), o[0], o[1]);
            }
          }
        } else {
#pragma unroll 1
          for (int c0 = 0; c0 < NW && c_first + c0 < n_out; c0 += 32) {
            uint32_t v[16];
            __syncwarp();
            x_ld16x256_32(tl + (uint32_t)c0, v);
            float o[16];
            const int col0 = c_first + c0 + 2 * (lane & 3);
            if (a.vec && c_first + c0 + 32 <= n_out) {
              // all residual loads of the chunk in flight at once, the accumulator's beside them; rows behind M read row M - 1
              const size_t m[2] = {(size_t)min(mrow, a.M - 1), (size_t)min(mrow + 8, a.M - 1)};
              float2 r[2][8];
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                const float* p = k ? a.r2 : a.r1;
                const size_t stride = k ? (size_t)a.N : (size_t)a.r1_stride;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  r[k][j] = p ? *reinterpret_cast<const float2*>(p + m[j & 1] * stride + col0 + 8 * (j >> 1)) : make_float2(0.f, 0.f);
              }
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int at = 4 * (j >> 1) + 2 * (j & 1);
                o[at] = __uint_as_float(v[at]) * xs[j & 1];
                o[at + 1] = __uint_as_float(v[at + 1]) * xs[j & 1];
                if (a.r1) { o[at] += r[0][j].x; o[at + 1] += r[0][j].y; }
                if (a.r2) { o[at] += r[1][j].x; o[at + 1] += r[1][j].y; }
              }
            } else {
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const int m = mrow + 8 * ((j >> 1) & 1), col = col0 + 8 * (j >> 2) + (j & 1);
                o[j] = __uint_as_float(v[j]) * xs[(j >> 1) & 1];
                if (m >= a.M || col >= n_out) continue;
                if (a.r1) o[j] += a.r1[(size_t)m * a.r1_stride + col];
                if (a.r2) o[j] += a.r2[(size_t)m * a.N + col];
              }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int at = 4 * (j >> 1) + 2 * (j & 1);
              put(j & 1, c_first + c0 + 8 * (j >> 1) + 2 * (lane & 3), o[at], o[at + 1]);
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) cluster_arrive(acc_free + 8 * buf, 0);
    }
  } else if (warp == PAIR_CONV_WARPS + PAIR_EPI_WARPS) {
    // ---- activation loader: this CTA's 128 rows of the tile, one bulk copy per stage. Only this role and the epilogue wait for
    // the packing kernel in front: the first stages' weights are loaded and converted beside it
    if (lane == 0) {
      pdl_wait();
      int n = 0;
      bool alive = true;
      for (int item = pair; item < items && alive; item += npairs) {
        const Item t = item_of(a, item, UPG);
        // a last tile whose second half lies behind the packed rows reads the last rows again: its results are not stored
        const int half = min(2 * t.mt + rank, a.x_halves - 1);
        const uint8_t* src = reinterpret_cast<const uint8_t*>(a.xh) + ((size_t)half * a.ngroups + t.kg0) * UPG * PAIR_A_BYTES;
        for (int u = 0; u < t.units; ++u, ++n) {
          const int s = n % P::STAGES, round = n / P::STAGES;
          if (round > 0 && !(alive = x_wait(stage_free + 8 * s, (uint32_t)((round - 1) & 1), dead, a.status))) break;
          mbar_expect_tx(full + 8 * s, PAIR_A_BYTES);
          bulk_g2s(smem_u32(smem + s * P::STAGE), src + (size_t)u * PAIR_A_BYTES, PAIR_A_BYTES, full + 8 * s);
        }
      }
      if (*dead)
        for (int i = max(0, n - P::STAGES); i < n; ++i) x_drain(full + 8 * (i % P::STAGES), (uint32_t)((i / P::STAGES) & 1));
    }
  } else {
    // ---- MMA issuer of the pair (even CTA), or the messenger of its "stage full" (odd CTA). The next stage's barrier is
    // polled before this one's MMAs are issued: a wait that finds its phase done still takes some 200 cycles, and with
    // three of them in front of four MMAs the issuer bounded the kernel (1150 cycles per stage, of 512 for the MMAs)
    int s = 0, n = 0;
    uint32_t parity = 0, ready = 0;
    bool alive = true;
    const uint64_t adesc0 = x_desc(smem_u32(smem), 128, 1024), bdesc0 = x_desc(smem_u32(smem) + PAIR_A_BYTES, 128, 1024);
    for (int item = pair; item < items && alive; item += npairs, ++n) {
      const int units = item_of(a, item, UPG).units, buf = n & 1;
      if (rank == 0 && n >= 2) {
        alive = w_wait(acc_free + 8 * buf, (uint32_t)(((n >> 1) - 1) & 1), dead, a.status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      for (int u = 0; u < units && alive; ++u) {
        if (!__all_sync(0xFFFFFFFFu, ready) && !(alive = w_wait(full + 8 * s, parity, dead, a.status))) break;
        const int now = s;
        if (++s == P::STAGES) { s = 0; parity ^= 1u; }
        ready = x_poll(full + 8 * s, parity);
        if (rank == 1) {
          if (lane == 0) cluster_arrive(full + 8 * now, 0);
          __syncwarp();
          continue;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int b = 0; b < 2; ++b)
          pair_mma4<16>(tmem + (uint32_t)(buf * NW), adesc0 + (uint64_t)((now * P::STAGE + b * PAIR_A_BLOCK) >> 4),
                    bdesc0 + (uint64_t)((now * P::STAGE + b * P::B_BLOCK) >> 4), P::IDESC, (u | b) ? 1u : 0u);
        pair_commit(stage_free + 8 * now);
      }
      if (rank == 0 && alive) pair_commit(acc_full + 8 * buf);
    }
    if (rank == 0) pair_commit(drained);
    x_drain(drained, 0);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0) pair_tmem_free(tmem, P::COLS);
}

template <int NW, int TYPE>
int launch_pair(fb200_device* dev, const PairArgs& a, bool early) {
  using P = Pair<NW>;
  static bool configured[64] = {false};
  if (!configured[dev->ordinal & 63]) {
    FB_CUDA(dev, cudaFuncSetAttribute(qgemm_pair_kernel<NW, TYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::SMEM));
    configured[dev->ordinal & 63] = true;
  }
  const int items = a.m_tiles * a.n_tiles * a.splits, pairs = std::min(items, dev->sm_count / 2);
  return fb200_launch(dev, qgemm_pair_kernel<NW, TYPE>, dim3((unsigned)(2 * pairs)), dim3(PAIR_THREADS), (size_t)P::SMEM, early, a);
}

}  // namespace

int fb200_qgemm_pair(fb200_device* dev, int nw, uint32_t type, const PairArgs& a, bool early) {
  const bool wide = nw == 256;
  switch (type) {
    case FB200_Q4_0: return wide ? launch_pair<256, FB200_Q4_0>(dev, a, early) : launch_pair<128, FB200_Q4_0>(dev, a, early);
    case FB200_Q8_0: return wide ? launch_pair<256, FB200_Q8_0>(dev, a, early) : launch_pair<128, FB200_Q8_0>(dev, a, early);
    case FB200_Q4_K: return wide ? launch_pair<256, FB200_Q4_K>(dev, a, early) : launch_pair<128, FB200_Q4_K>(dev, a, early);
    case FB200_Q6_K: return wide ? launch_pair<256, FB200_Q6_K>(dev, a, early) : launch_pair<128, FB200_Q6_K>(dev, a, early);
  }
  return 1;
}
