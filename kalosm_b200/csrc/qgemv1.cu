// Decode GEMV: y[N] = W[N, K] . x[K] for ONE activation row, the shape of batch-1 decoding.
//
// Bound: HBM (algorithmic bytes = the raw GGUF bytes of W). Structure:
//  * persistent CTAs (SM count x CTAs per SM) walk the 16-row tiles of W; the warps of a CTA
//    split a tile's K groups; partial sums meet in shared memory in a fixed order;
//  * every warp owns a ring of shared-memory stages filled by 1-D TMA bulk copies
//    (cp.async.bulk + mbarrier complete_tx), one contiguous tile-group per stage, so tens of KB
//    per SM are in flight without holding registers; the first copies are issued before
//    griddepcontrol.wait, i.e. under programmatic dependent launch the weights stream in
//    while the kernel that produces x is still running;
//  * one launch may carry up to three matrices that share the activation row (the q, k and v
//    projections), of different quant types;
//  * the prologue turns x into int8 MMA B operands in shared memory once per CTA: optional
//    residual add and RMSNorm (so the norm needs no kernel of its own), a power-of-two scale
//    per 16 elements, then FOUR 7-bit limbs per element, the bit fields of q = rint(x/scale * 2^27)
//    (x/scale = (l0 + u1/2^7 + u2/2^14 + u3/2^21) / 64 to 2^-28, l0 signed, u 0..127), plus the
//    per-16 sums the offsets of Q4_K/Q4_0/Q6_K need;
//  * quants stay in the byte domain: one logic op turns four packed nibbles into four u8
//    operands of mma.sync.m16n8k32 (u8 x s8 -> s32, exact), so the ALU pipe that limits an
//    fp16 expansion is nearly idle;
//  * "scale group per lane": in every MMA lane t of a quad feeds eight elements of scale group
//    t (for rows g and g+8), and the B operand carries the limbs of group t' only in columns
//    2t', 2t'+1. The accumulator of lane t then holds exactly its own group's integer dot
//    products, so each lane decodes and applies ONE scale per chain of MMAs and no data is
//    exchanged between lanes until the final sum;
//  * integer dot products are exact; they are scaled and accumulated in fp32.
//
// Replaces the reference's qgemv kernels (fusor-ml/tile-ir-kernels/src/kernels/qgemv.rs:356-678,
// qgemv_q6k.rs:84-385), their SwiGLU and residual epilogues
// (fusor-ml/core/src/quantized/matmul/mod.rs:435-439, 666-722) and the fused RMSNorm cluster
// (fusor-ml/core/src/composite/rms_norm_fused.rs:10-54) in front of a projection.
#include "packed_act.cuh"
#include "qgemv1_groups.cuh"

namespace {

struct Gemv1Args {
  const uint8_t* w;     // tiled weight bytes
  float* y;             // [n_out]
  int tg;               // bytes per tile-group
  int n_out;
  const float* x;       // [K]
  const float* xres;    // optional [K]: v = x + xres
  const float* norm_w;  // optional [K]: activation = v / sqrt(mean(v^2) + eps) * norm_w
  float eps;
  int K, Kp;            // logical and padded (ngroups * group_elems) inner size
  const float* r1;
  const float* r2;
  int ngroups, nunits, pair_tile_offset, stages, stride;
  int* status;
};

// TYPE: ggml type of the matrix. EPI: 0 none, 1 residual(s), 2 SwiGLU pair. W = warps per CTA,
// MINB = CTAs per SM.
template <int TYPE, int EPI, int W, int MINB>
__global__ void __launch_bounds__(W * 32, MINB)
qgemv1_kernel(const Gemv1Args a) {
  constexpr int NP = EPI == 2 ? 2 : 1;
  constexpr int THREADS = W * 32;
  extern __shared__ __align__(128) uint8_t smem[];
  const int S = a.stages;
  uint8_t* zeros = smem;  // written before the prologue's barrier
  for (int i = threadIdx.x; i < ZERO_BYTES / 16; i += THREADS) reinterpret_cast<uint4*>(zeros)[i] = make_uint4(0u, 0u, 0u, 0u);
  uint8_t* ring = smem + ZERO_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + W * S * a.stride);
  uint8_t* xl = ring + W * S * a.stride + W * S * 8;  // limbs (4 B / element)
  float* xsc = reinterpret_cast<float*>(xl + (size_t)a.Kp * 4);  // per-16 scale of the limbs
  float* xss = xsc + a.Kp / 16;    // per-16 sum of the activations
  float* red = xss + a.Kp / 16;    // [NP][W][16]
  float* tmp = red + NP * W * 16;  // [2 W] block reductions

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Lane L = make_lane(lane);
  uint8_t* my_ring = ring + warp * S * a.stride;
  const uint32_t my_bar = smem_u32(bars + warp * S);

  pdl_launch_dependents();
  if (lane == 0) {
    for (int s = 0; s < S; ++s) mbar_init(my_bar + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();

  // this warp's items in issue order: for each unit of the CTA, for each pass (gate / up), the
  // K groups warp, warp + W, ...
  const int gw = a.ngroups > warp ? (a.ngroups - warp + W - 1) / W : 0;
  const int my_units = a.nunits > (int)blockIdx.x ? (a.nunits - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const int n_items = my_units * NP * gw;
  int is_unit = blockIdx.x, is_p = 0, is_kk = 0, issued = 0;  // issue-side cursor (lane 0)
  auto issue_next = [&](int st) {
    const uint8_t* src = a.w + ((size_t)(is_unit + is_p * a.pair_tile_offset) * a.ngroups + (warp + W * is_kk)) * a.tg;
    mbar_expect_tx(my_bar + 8 * st, a.tg);
    bulk_g2s(smem_u32(my_ring + st * a.stride), src, a.tg, my_bar + 8 * st);
    ++issued;
    if (++is_kk == gw) {
      is_kk = 0;
      if (++is_p == NP) { is_p = 0; is_unit += gridDim.x; }
    }
  };
  if (lane == 0) {
    const int pre = n_items < S ? n_items : S;
    for (int i = 0; i < pre; ++i) issue_next(i);
  }
  // only weights were touched so far; x comes from the kernel before this one
  pdl_wait();

  // ---- activation prologue ------------------------------------------------------------------
  // One trip: every thread turns blocks of 8 elements into limbs as they arrive, under the power of two of their 16 elements
  // (q = rint(v / scale 2^27); l0 = q >> 21 signed, u1, u2, u3 = the next three 7-bit fields), and adds up the squares; 1 / rms
  // goes to the outputs. One scale for the whole row took a second pass behind a block reduction. Together with the operand
  // loads of qgemv1_groups.cuh, before -> now, back to back on weights that are not in L2: 6144 x 4096 Q4_K 9.4 -> 7.5 us,
  // 4096 x 4096 Q4_0 8.2 -> 7.6 and Q8_0 9.3 -> 7.9, 28672 x 4096 Q4_K with SwiGLU 22.5 -> 20.4, 4096 x 14336 Q6_K 19.9 -> 17.3,
  // 128256 x 4096 Q6_K 80.5 -> 75.8 (5.7 TB/s) and Q4_K 62.9 -> 54.5 (5.4 TB/s).
  {
    const bool vec = !((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.xres) | reinterpret_cast<uintptr_t>(a.norm_w)) & 15);
    float ss = 0.f;
    auto get = [&](const float* p, int k, float (&v)[8]) {
      if (vec && k + 8 <= a.K) {
        const float4 u = *reinterpret_cast<const float4*>(p + k), w = *reinterpret_cast<const float4*>(p + k + 4);
        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w; v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = k + i < a.K ? p[k + i] : 0.f;
      }
    };
    const int nblk = a.Kp >> 3;
    for (int b0 = 0; b0 < nblk; b0 += THREADS) {
      const int kb = b0 + (int)threadIdx.x;
      const bool in = kb < nblk;  // (blocks come in pairs of lanes)
      float v[8], w[8], amax = 0.f;
      if (kb * 8 < a.Kp) {
        get(a.x, kb * 8, v);
        if (a.norm_w) get(a.norm_w, kb * 8, w);
        if (a.xres) {
          float r[8];
          get(a.xres, kb * 8, r);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] += r[i];
        }
      }
      if (in) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (a.norm_w) {
            ss = fmaf(v[i], v[i], ss);
            v[i] *= w[i];
          }
          amax = fmaxf(amax, fabsf(v[i]));
        }
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
      int ex = 0;
      if (amax > 0.f && amax < 3.0e38f) frexpf(amax, &ex);  // amax = f * 2^ex, f in [0.5, 1)
      ex = max(ex, -110);                                   // 2^(6 - ex) and 2^(ex - 13) stay in range
      const float inv64 = ldexpf(64.0f, -ex);               // v * inv64 in (-64, 64)
      const float out_scale = ldexpf(1.0f, ex - 13);        // 2^ex / (64 * 128)
      uint32_t sum = 0;  // of the q, as int: 16 of them stay below 2^31 (floats in their place: 2.15e-7 of error at 4096 x 4096 Q4_0, not 1.7e-7)
      if (in) {
        uint32_t r[8], wl[2][4];  // [half of the block][limb 3, 2, 1, 0] four elements per word
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int q = __float2int_rn((v[i] * inv64) * 2097152.0f);
          sum += (uint32_t)q;
          // fields at bits 0, 7, 14, 21 -> bytes 0..3 (byte 3 = bits 21..28 = l0 as s8)
          r[i] = ((uint32_t)q & 0x7Fu) | (((uint32_t)q << 1) & 0x7F00u) | (((uint32_t)q << 2) & 0x7F0000u) |
                 (((uint32_t)q << 3) & 0xFF000000u);
        }
#pragma unroll
        for (int hb = 0; hb < 2; ++hb) {
          // 4 x 4 byte transpose: word j = byte j of the four elements
          const uint32_t t01l = __byte_perm(r[4 * hb], r[4 * hb + 1], 0x5140), t23l = __byte_perm(r[4 * hb + 2], r[4 * hb + 3], 0x5140);
          const uint32_t t01h = __byte_perm(r[4 * hb], r[4 * hb + 1], 0x7362), t23h = __byte_perm(r[4 * hb + 2], r[4 * hb + 3], 0x7362);
          wl[hb][0] = __byte_perm(t01l, t23l, 0x5410);  // u3
          wl[hb][1] = __byte_perm(t01l, t23l, 0x7632);  // u2
          wl[hb][2] = __byte_perm(t01h, t23h, 0x5410);  // u1
          wl[hb][3] = __byte_perm(t01h, t23h, 0x7632);  // l0
        }
        uint4* dst = reinterpret_cast<uint4*>(xl + (size_t)limb_block(kb) * 32);
        dst[0] = make_uint4(wl[0][3], wl[1][3], wl[0][1], wl[1][1]);  // limb 0, limb 2
        dst[1] = make_uint4(wl[0][2], wl[1][2], wl[0][0], wl[1][0]);  // limb 1, limb 3
      }
      // per-16 sums in the units of the integer dot products (128 * sum(v) = sum(q) / 2^14)
      sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
      if (in && (threadIdx.x & 1) == 0) {
        xsc[kb >> 1] = out_scale;
        xss[kb >> 1] = (float)(int)sum * (1.0f / 16384.0f) * out_scale;
      }
    }
    if (a.norm_w) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
      if (lane == 0) tmp[warp] = ss;
    }
    __syncthreads();
    if (threadIdx.x < 16) {  // the half warp that forms the outputs
      float fs = 1.f;
      if (a.norm_w) {
        ss = 0.f;
        for (int i = 0; i < W; ++i) ss += tmp[i];
        // rms_norm_fused_cpu_impl, fusor-ml/fusor/src/composite/normalization.rs:404-461
        const float rms = sqrtf(ss / (float)a.K + a.eps);
        fs = rms == 0.f ? 0.f : 1.0f / rms;  // a row of zeros without an eps stays zero
      }
      __syncwarp(0xFFFFu);
      if (threadIdx.x == 0) tmp[0] = fs;
      __syncwarp(0xFFFFu);
    }
  }

  int item = 0, st = 0;
  uint32_t phase = 0;
  FeedB B(L);
  constexpr int BLOCKS16 = (TYPE == FB200_Q4_K || TYPE == FB200_Q6_K) ? 16 : 8;  // 16-element blocks per K group
  for (int j = 0; j < my_units; ++j) {
    const int tile = (int)blockIdx.x + j * (int)gridDim.x;
    if (j > 0) __syncthreads();  // the previous unit's reduction has read `red`
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float acc_g = 0.f, acc_g8 = 0.f;
      GroupPtrs G = group_ptrs(L, xl, zeros, xsc, xss, warp, BLOCKS16);
      for (int kk = 0; kk < gw; ++kk, ++item) {
        mbar_wait(my_bar + 8 * st, phase, a.status);
        const uint8_t* tg = my_ring + st * a.stride;
        group1_any(TYPE, B, G, tg, L, acc_g, acc_g8);
        // Every lane has read the stage (its loads precede this barrier in program order and
        // shared loads complete long before a refill from global memory can land).
        __syncwarp();
        if (lane == 0 && issued < n_items) issue_next(st);
        if (++st == S) { st = 0; phase ^= 1u; }
        group_ptrs_next(G, BLOCKS16 * W);  // K group warp + W * (kk + 1)
      }
      // lane t accumulated the scale groups it owns: sum over the quad
      acc_g += __shfl_xor_sync(0xFFFFFFFFu, acc_g, 1);
      acc_g += __shfl_xor_sync(0xFFFFFFFFu, acc_g, 2);
      acc_g8 += __shfl_xor_sync(0xFFFFFFFFu, acc_g8, 1);
      acc_g8 += __shfl_xor_sync(0xFFFFFFFFu, acc_g8, 2);
      if (L.t == 0) {
        red[(p * W + warp) * 16 + L.g] = acc_g;
        red[(p * W + warp) * 16 + L.g + 8] = acc_g8;
      }
    }
    __syncthreads();
    if (threadIdx.x < 16) {
      const int r = threadIdx.x;
      const int n = tile * 16 + r;
      float v[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float s = 0.f;
        for (int w = 0; w < W; ++w) s += red[(p * W + w) * 16 + r];
        v[p] = s * tmp[0];
      }
      if (n < a.n_out) {
        float out;
        if (EPI == 2) {
          // silu(gate) * up, fusor-ml/fusor/src/composite/activations.rs:47-64
          const float gate = v[0];
          out = (gate / (1.0f + expf(-gate))) * v[NP - 1];
        } else if (EPI == 1) {
          out = v[0] + a.r1[n];
          if (a.r2) out += a.r2[n];
        } else {
          out = v[0];
        }
        a.y[n] = out;
      }
    }
  }
}

constexpr int SMEM_LIMIT = 227 * 1024;

template <int EPI, int W>
size_t gemv1_smem(int stages, int stride, int kp) {
  constexpr int NP = EPI == 2 ? 2 : 1;
  return (size_t)ZERO_BYTES + (size_t)W * stages * stride + (size_t)W * stages * 8 + (size_t)kp * 4 + (size_t)kp / 16 * 4 +
         (size_t)kp / 16 * 4 + (size_t)NP * W * 16 * 4 + (size_t)2 * W * 4 + 64;
}

template <int TYPE, int EPI, int W, int MINB>
int launch_w(fb200_device* dev, Gemv1Args& a) {
  auto kern = qgemv1_kernel<TYPE, EPI, W, MINB>;
  static bool configured[64] = {false};
  if (!configured[dev->ordinal & 63]) {
    FB_CUDA(dev, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
    configured[dev->ordinal & 63] = true;
  }
  int grid = dev->sm_count * MINB;
  if (grid > a.nunits) grid = a.nunits;
  // same number of units for every CTA where the unit count allows it
  const int rounds = (a.nunits + grid - 1) / grid;
  grid = (a.nunits + rounds - 1) / rounds;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(W * 32);
  cfg.dynamicSmemBytes = gemv1_smem<EPI, W>(a.stages, a.stride, a.Kp);
  cfg.stream = dev->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dev->pdl ? 1 : 0;
  FB_CUDA(dev, cudaLaunchKernelEx(&cfg, kern, a));
  dev->launches++;
  return FB200_OK;
}

// Shared memory per SM is split between the activation limbs (4 B per element of K, one copy
// per CTA, built by every CTA in its prologue) and the weight rings. More, smaller CTAs give
// deeper rings per warp and more independent tiles in flight; larger K forces fewer CTAs.
template <int TYPE, int EPI>
int launch_cfg(fb200_device* dev, Gemv1Args& a) {
  const int per_sm = SMEM_LIMIT - 2048;
  auto fits = [&](size_t need, int ctas) { return (need + 1024) * ctas <= (size_t)per_sm; };
  for (int s = 3; s >= 2; --s)
    if (fits(gemv1_smem<EPI, 8>(s, a.stride, a.Kp), 4)) { a.stages = s; return launch_w<TYPE, EPI, 8, 4>(dev, a); }
  for (int s = 3; s >= 2; --s)
    if (fits(gemv1_smem<EPI, 8>(s, a.stride, a.Kp), 3)) { a.stages = s; return launch_w<TYPE, EPI, 8, 3>(dev, a); }
  for (int s = 3; s >= 2; --s)
    if (fits(gemv1_smem<EPI, 16>(s, a.stride, a.Kp), 2)) { a.stages = s; return launch_w<TYPE, EPI, 16, 2>(dev, a); }
  for (int s = 2; s >= 1; --s)
    // (the zeros come out of the 2 KB that are left free: no row length is refused for them)
    if (fits(gemv1_smem<EPI, 32>(s, a.stride, a.Kp) - ZERO_BYTES, 1)) { a.stages = s; return launch_w<TYPE, EPI, 32, 1>(dev, a); }
  return fb200_fail(dev, FB200_ERR_CAPACITY, "qgemv1: K = %d does not fit in shared memory", a.K);
}

template <int TYPE>
int launch_typed(fb200_device* dev, Gemv1Args& a, int epi) {
  if (epi == FB200_EPI_SWIGLU) return launch_cfg<TYPE, 2>(dev, a);
  if (epi == FB200_EPI_RESIDUAL) return launch_cfg<TYPE, 1>(dev, a);
  return launch_cfg<TYPE, 0>(dev, a);
}

}  // namespace

// Largest K the single-row kernel takes (activation limbs live in shared memory).
bool fb200_qgemv1_fits(const fb200_qmatrix* w) {
  TileGeom geo;
  if (!tile_geom(w->type, &geo)) return false;
  const uint64_t kp = (uint64_t)w->ngroups * geo.group_elems;
  return kp * 4 + kp / 4 + 16 * 3456 + 8192 <= (uint64_t)SMEM_LIMIT - 2048;
}

// y[n] = epilogue(W . act(x)) for one activation row; act = optional residual add + RMSNorm
// (norm_w != null).
int fb200_qgemv1(fb200_device* dev, const fb200_qmatrix* w, const float* x, const float* xres,
                 const float* norm_w, float eps, float* y, int epi, const float* r1,
                 const float* r2) {
  TileGeom geo;
  if (!w->tiled || !tile_geom(w->type, &geo))
    return fb200_fail(dev, FB200_ERR_UNSUPPORTED_DTYPE, "qgemv1: type %u has no tiled storage", w->type);
  Gemv1Args a = {};
  a.w = w->data; a.y = y; a.tg = geo.tg_bytes; a.n_out = (int)w->n;
  a.nunits = w->ntiles;
  a.stride = (geo.tg_bytes + 127) / 128 * 128;
  a.x = x; a.xres = xres; a.norm_w = norm_w; a.eps = eps;
  a.K = (int)w->k; a.Kp = w->ngroups * geo.group_elems;
  a.r1 = r1; a.r2 = r2;
  a.ngroups = w->ngroups; a.pair_tile_offset = 0;
  a.stages = 2; a.status = dev->status;
  if (epi == FB200_EPI_SWIGLU) {
    a.nunits = w->ntiles / 2;
    a.n_out = (int)(w->n / 2);
    a.pair_tile_offset = w->ntiles / 2;
  }
  switch (w->type) {
    case FB200_Q4_K: return launch_typed<FB200_Q4_K>(dev, a, epi);
    case FB200_Q6_K: return launch_typed<FB200_Q6_K>(dev, a, epi);
    case FB200_Q8_0: return launch_typed<FB200_Q8_0>(dev, a, epi);
    default: return launch_typed<FB200_Q4_0>(dev, a, epi);
  }
}
