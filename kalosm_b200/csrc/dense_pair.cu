// Products of many activation rows with BF16 weights on CTA pairs: tcgen05.mma.cta_group::2, 256 activation rows by NW weight rows
// per pair, persistent, two accumulators per CTA.
//
// Bound: tensor cores (2 M N K flops). A single CTA with a tile of 256 x 256 left the tensor cores idle during its epilogue and had
// half as many operand stages for the same tile (8192 rows of 14336 x 2048: 486 us, 343 here); a pair writes one tile while it
// multiplies the next. The activations are in the M role, so that gate and up rows of an output (halves of the weight tile, one
// per CTA) meet in one TMEM lane, NW / 2 columns apart.
//  * copy requester (one thread per CTA): a stage is 64 values of K: boxes of 64 columns by 128 activation rows and by NW / 2
//    weight rows, by tensor TMA with 128-byte swizzle; rows and columns outside the matrices arrive as zeros. The copies of both CTAs
//    are counted on the even CTA's barrier (a message from the odd CTA would lengthen every refill);
//  * issuer (one warp of the even CTA): four MMAs (M = 256, N = NW, K = 16) per stage;
//  * epilogue (8 warps): tcgen05.ld, then f32 or bf16 rows (factor, bias, residual, softcap), gelu rows or SwiGLU.
// Every wait is bounded (2^22 polls), as in qgemm_pair.cu.
#include "dense.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int DP_EPI_WARPS = 8, DP_THREADS = (DP_EPI_WARPS + 2) * 32;
constexpr int DP_A_BYTES = 128 * 64 * 2, DP_MAX_STAGES = 8, DP_TAIL = 512;

template <int NW>
struct DPair {
  static constexpr int STAGE = DP_A_BYTES + NW / 2 * 64 * 2, STAGES = NW == 256 ? 6 : 8, COLS = 2 * NW;
  static constexpr int SMEM = STAGES * STAGE + DP_TAIL + 1024;
  // instruction descriptor: fp32 accumulator, bf16 A and B, both K-major, N = NW, M = 256 over the pair
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NW >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
};

struct DPairArgs {
  float* y;
  __nv_bfloat16* yb;
  const float* add;
  const float* bias;
  __nv_bfloat16* z;
  size_t ldy, ldadd, ldz;
  int m, kblocks, row0, n_plain, gate0, up0, ff, gelu, ff_col, plain_tiles, n_tiles, m_tiles;
  int vec_y, vec_z;  // pairs of columns of y (and of add), and of z, are aligned
  float alpha, softcap;
  int* status;
};

__device__ __forceinline__ void dp_put(float* p, uint32_t v) { *p = __uint_as_float(v); }
__device__ __forceinline__ void dp_put(__nv_bfloat16* p, uint32_t v) { *p = __float2bfloat16(__uint_as_float(v)); }
__device__ __forceinline__ void dp_put2(float* p, uint32_t v0, uint32_t v1) { *reinterpret_cast<uint2*>(p) = make_uint2(v0, v1); }
__device__ __forceinline__ void dp_put2(__nv_bfloat16* p, uint32_t v0, uint32_t v1) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(__uint_as_float(v0), __uint_as_float(v1));
}
// A chunk of 16 rows x 32 columns as x_ld16x256_32 lays it out: columns col, col + 1, col + 8, .. of rows m (p0) and m + 8 (p1).
template <typename T>
__device__ __forceinline__ void dp_store(T* p0, T* p1, const uint32_t (&v)[16], bool whole, int m, int m_end, int col, int n_out, int vec) {
  if (whole) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      dp_put2(p0 + 8 * i, v[4 * i], v[4 * i + 1]);
      dp_put2(p1 + 8 * i, v[4 * i + 2], v[4 * i + 3]);
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int at = 4 * (j >> 1) + 2 * (j & 1), c = col + 8 * (j >> 1);
    T* p = (j & 1 ? p1 : p0) + 8 * (j >> 1);
    if (m + 8 * (j & 1) >= m_end || c >= n_out) continue;
    if (vec && c + 1 < n_out) {
      dp_put2(p, v[at], v[at + 1]);
    } else {
      dp_put(p, v[at]);
      if (c + 1 < n_out) dp_put(p + 1, v[at + 1]);
    }
  }
}

template <int NW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(DP_THREADS, 1)
dense_pair_kernel(const DPairArgs a, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap) {
  using P = DPair<NW>;
  extern __shared__ uint8_t sm_raw[];
  // the same offset in both CTAs: their dynamic shared memory starts at the same address
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + P::STAGES * P::STAGE);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * DP_MAX_STAGES + 5);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank(), pair = (int)blockIdx.x >> 1, npairs = (int)gridDim.x >> 1;
  const uint32_t full = smem_u32(bars), stage_free = full + 8 * DP_MAX_STAGES, acc_full = stage_free + 8 * DP_MAX_STAGES,
                 acc_free = acc_full + 16, drained = acc_free + 16;
  const int items = a.m_tiles * a.n_tiles;

  if (tid == 0) {
    *dead = 0;
    for (int i = 0; i < P::STAGES; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(stage_free + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_free + 8 * i, 2 * DP_EPI_WARPS);
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

  // activation tiles fastest: the pairs that run together share their weight rows in L2
  auto split = [&](int item, int& mt, int& nt, bool& ffn, bool& gated) {
    nt = item / a.m_tiles;
    mt = item - nt * a.m_tiles;
    ffn = nt >= a.plain_tiles;
    gated = ffn && !a.gelu;
    if (ffn) nt -= a.plain_tiles;
  };

  if (warp < DP_EPI_WARPS) {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. of this CTA's 128 activation rows, one half of the columns
    const int quad = warp & 3, ch = warp >> 2;
    int n = 0;
    pdl_wait();
    for (int item = pair; item < items; item += npairs, ++n) {
      const int buf = n & 1;
      if (!w_wait(acc_full + 8 * buf, (uint32_t)((n >> 1) & 1), dead, a.status)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      int mt, nt;
      bool ffn, gated;
      split(item, mt, nt, ffn, gated);
      const int m_first = mt * 256 + rank * 128 + quad * 32;
      const int width = gated ? NW / 2 : NW, n_out = ffn ? a.ff : a.n_plain, c_end = (ch + 1) * (width / 2);
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        if (m_first + 16 * hh >= a.m) break;
        const int mrow = m_first + 16 * hh + (lane >> 2);  // and eight rows further
        const uint32_t tl = tmem + ((uint32_t)(32 * quad + 16 * hh) << 16) + (uint32_t)(buf * NW);
        const size_t rows[2] = {(size_t)min(mrow, a.m - 1), (size_t)min(mrow + 8, a.m - 1)};
        const bool all_rows = m_first + 16 * hh + 16 <= a.m;
#pragma unroll 1
        for (int c0 = ch * (width / 2); c0 < c_end && nt * width + c0 < n_out; c0 += 32) {
          const int col0 = nt * width + c0 + 2 * (lane & 3);  // and 8, 16, 24 columns further
          // Nothing in the chunk has to be left out: straight code with one address per row. (With the checks below on every
          // pair a chunk took 2500 cycles and the epilogue of a 2048-wide K was longer than its MMAs.)
          const bool whole = all_rows && nt * width + c0 + 32 <= n_out && (ffn ? a.vec_z : a.vec_y);
          uint32_t v[16];
          __syncwarp();
          x_ld16x256_32(tl + (uint32_t)c0, v);
          if (ffn) {
            uint32_t u[16];
            if (gated) x_ld16x256_32(tl + (uint32_t)(NW / 2 + c0), u);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (gated) {
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const float g = __uint_as_float(v[i]);
                v[i] = __float_as_uint(g / (1.0f + __expf(-g)) * __uint_as_float(u[i]));
              }
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(fb_gelu_tanh_fast(__uint_as_float(v[i])));
            }
            dp_store<__nv_bfloat16>(a.z + rows[0] * a.ldz + col0, a.z + rows[1] * a.ldz + col0, v, whole, mrow, a.m, col0, n_out, a.vec_z);
            continue;
          }
          float2 r[8];
          if (a.add) {  // in flight beside the accumulator's load
            const float *p0 = a.add + rows[0] * a.ldadd + col0, *p1 = a.add + rows[1] * a.ldadd + col0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float* p = (j & 1 ? p1 : p0) + 8 * (j >> 1);
              if (whole) r[j] = *reinterpret_cast<const float2*>(p);
              else r[j] = make_float2(col0 + 8 * (j >> 1) < n_out ? p[0] : 0.f, col0 + 8 * (j >> 1) + 1 < n_out ? p[1] : 0.f);
            }
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (a.bias) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int col = col0 + 8 * (i >> 2) + (i & 1);
              v[i] = __float_as_uint(fmaf(a.alpha, __uint_as_float(v[i]), col < n_out ? a.bias[col] : 0.f));
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(fmaf(a.alpha, __uint_as_float(v[i]), 0.f));
          }
          if (a.softcap > 0.f) {  // of a product without a residual
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(a.softcap * tanhf(__uint_as_float(v[i]) / a.softcap));
          }
          if (a.yb) {
            dp_store<__nv_bfloat16>(a.yb + rows[0] * a.ldy + col0, a.yb + rows[1] * a.ldy + col0, v, whole, mrow, a.m, col0, n_out, a.vec_y);
            continue;
          }
          if (a.add) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int at = 4 * (j >> 1) + 2 * (j & 1);
              v[at] = __float_as_uint(__uint_as_float(v[at]) + r[j].x);
              v[at + 1] = __float_as_uint(__uint_as_float(v[at + 1]) + r[j].y);
            }
          }
          dp_store<float>(a.y + rows[0] * a.ldy + col0, a.y + rows[1] * a.ldy + col0, v, whole, mrow, a.m, col0, n_out, a.vec_y);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) cluster_arrive(acc_free + 8 * buf, 0);
    }
  } else if (warp == DP_EPI_WARPS) {
    // ---- copy requester
    if (lane == 0) {
      pdl_wait();
      int k = 0;
      bool alive = true;
      for (int item = pair; item < items && alive; item += npairs) {
        int mt, nt;
        bool ffn, gated;
        split(item, mt, nt, ffn, gated);
        const int xr = mt * 256 + rank * 128, xc = ffn ? a.ff_col : 0;
        const int wr = gated ? (rank ? a.up0 : a.gate0) + nt * (NW / 2) : (ffn ? a.up0 : a.row0) + nt * NW + rank * (NW / 2);
        for (int kb = 0; kb < a.kblocks; ++kb, ++k) {
          const int s = k % P::STAGES, round = k / P::STAGES;
          if (round > 0 && !(alive = x_wait(stage_free + 8 * s, (uint32_t)((round - 1) & 1), dead, a.status))) break;
          const uint32_t dst = smem_u32(sm + s * P::STAGE), bar = cluster_addr(full + 8 * s, 0);
          if (rank == 0) mbar_expect_tx(full + 8 * s, 2 * P::STAGE);
          pair_tma_box2(dst, &xmap, xc + kb * 64, xr, bar);
          pair_tma_box2(dst + DP_A_BYTES, &wmap, kb * 64, wr, bar);
        }
      }
      if (*dead) {
        // the even CTA waits for the copies that its barriers count; the odd one has no barrier of its own that counts
        // them and lets the limit of a wait run out instead, which takes far longer than a copy
        if (rank) x_drain(full, 0);
        else
          for (int i = max(0, k - P::STAGES); i < k; ++i) x_drain(full + 8 * (i % P::STAGES), (uint32_t)((i / P::STAGES) & 1));
      }
    }
  } else {
    // ---- MMA issuer; the next stage's barrier is polled before this one's MMAs are issued
    int s = 0, n = 0;
    uint32_t parity = 0, ready = 0;
    bool alive = rank == 0;
    const uint64_t adesc0 = x_desc_rows(smem_u32(sm)), bdesc0 = x_desc_rows(smem_u32(sm) + DP_A_BYTES);
    for (int item = pair; item < items && alive; item += npairs, ++n) {
      const int buf = n & 1;
      if (n >= 2) {
        alive = w_wait(acc_free + 8 * buf, (uint32_t)(((n >> 1) - 1) & 1), dead, a.status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      for (int kb = 0; kb < a.kblocks && alive; ++kb) {
        if (!__all_sync(0xFFFFFFFFu, ready) && !(alive = w_wait(full + 8 * s, parity, dead, a.status))) break;
        const int now = s;
        if (++s == P::STAGES) { s = 0; parity ^= 1u; }
        ready = x_poll(full + 8 * s, parity);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t at = (uint64_t)((now * P::STAGE) >> 4);
        pair_mma4<2>(tmem + (uint32_t)(buf * NW), adesc0 + at, bdesc0 + at, P::IDESC, kb ? 1u : 0u);
        pair_commit(stage_free + 8 * now);
      }
      if (alive) pair_commit(acc_full + 8 * buf);
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

template <int NW>
int launch_pair(fb200_device* dev, const fb200_dense_job& j, DPairArgs a) {
  using P = DPair<NW>;
  CUtensorMap wmap, xmap;
  if (!fb200_make_map_2d(&wmap, j.w->data, 1, j.w->k, j.w->n, j.w->k * 2, NW / 2) ||
      !fb200_make_map_2d(&xmap, j.x, 1, (uint64_t)(j.ff_off + j.kx), (uint64_t)j.m, j.ldx * 2, 128))
    return fb200_fail(dev, FB200_ERR_CUDA, "dense product: tensor map refused (w %llu x %llu, x %d x %d stride %zu)",
                      (unsigned long long)j.w->n, (unsigned long long)j.w->k, j.m, j.kx, j.ldx);
  a.plain_tiles = (j.n_plain + NW - 1) / NW;
  const int ff_rows = a.gelu ? NW : NW / 2;
  a.n_tiles = a.plain_tiles + (j.ff + ff_rows - 1) / ff_rows;
  a.m_tiles = (j.m + 255) / 256;
  const int items = a.n_tiles * a.m_tiles, pairs = items < dev->sm_count / 2 ? items : dev->sm_count / 2;
  if (items == 0) return FB200_OK;
  static bool configured[64] = {false};
  if (!configured[dev->ordinal & 63]) {
    FB_CUDA(dev, cudaFuncSetAttribute(dense_pair_kernel<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::SMEM));
    configured[dev->ordinal & 63] = true;
  }
  return fb200_launch(dev, dense_pair_kernel<NW>, dim3((unsigned)(2 * pairs)), dim3(DP_THREADS), (size_t)P::SMEM, true, a, wmap, xmap);
}

}  // namespace

int fb200_dense_gemm_pair(fb200_device* dev, const fb200_dense_job& j, int nw) {
  DPairArgs a = {};
  if (j.y_bf16) a.yb = (__nv_bfloat16*)j.y;
  else a.y = (float*)j.y;
  a.add = j.add; a.bias = j.bias; a.z = (__nv_bfloat16*)j.z; a.ldy = j.ldy; a.ldadd = j.ldadd; a.ldz = j.ldz;
  a.m = j.m; a.kblocks = (j.kx + 63) / 64; a.row0 = j.row0; a.n_plain = j.n_plain; a.gate0 = j.gate0; a.up0 = j.up0; a.ff = j.ff;
  a.gelu = j.act == FB200_FFN_GELU; a.ff_col = (int)j.ff_off; a.alpha = j.alpha; a.softcap = j.softcap; a.status = dev->status;
  const uintptr_t pair_bytes = j.y_bf16 ? 4 : 8;
  a.vec_y = j.ldy % 2 == 0 && (uintptr_t)j.y % pair_bytes == 0 && (!j.add || (j.ldadd % 2 == 0 && (uintptr_t)j.add % 8 == 0));
  a.vec_z = j.ldz % 2 == 0 && (uintptr_t)j.z % 4 == 0;
  return nw == 256 ? launch_pair<256>(dev, j, a) : launch_pair<128>(dev, j, a);
}
