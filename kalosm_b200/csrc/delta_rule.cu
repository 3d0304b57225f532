// Gated delta rule: short convolution, unit q / k, the recurrence and its gated, normalised read-out.
//
//   S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//
// per head, with S [d, v] in 32-bit floats. The columns of S are independent, so a column (or a few) is
// what a group of lanes owns for the whole sequence: it stays in registers, k and q come from shared memory.
// Both sums over d are formed in one pass from the state BEFORE the token,
//   S^T k -> g (S^T k),   o = g (S^T q) + u (k . q),
// and in a prompt eight tokens share a pass: with a_i = S^T k_i, c_i = S^T q_i from the state before the eight,
// G_i = g_0 .. g_i and w_j = (g_(j+1) .. g_i) u_j,
//   u_i = beta_i (v_i - G_i a_i - sum_(j<i) (k_j . k_i) w_j),   o_i = G_i c_i + sum_(j<=i) (k_j . q_i) w_j,
//   S <- G_7 S + sum_j k_j w_j,
// the same recurrence with one reduction over the lanes per eight tokens. Everything is f32 (on tensor cores as three bf16 values).
//
//  * delta_step_kernel: one new token per sequence. One CTA per (head, sequence): convolution, unit vectors,
//    decay, state update, read-out, RMSNorm and gate. Bound: HBM on the state (read and written once).
//  * prompts: delta_prep_kernel (convolution, SiLU, unit vectors, decay and write strength), then delta_pairs_kernel (products of
//    eight tokens' k and q) and delta_scan_kernel (the recurrence; bound: latency of the pass, a warp per scheduler), or, for long
//    prompts, delta_chunk_kernel and delta_chunk_scan_kernel (the same over chunks of 32 tokens, on tensor cores), delta_out_kernel
//    (RMSNorm, gate) and conv_ring_kernel (the convolution's memory).
#include "mixers.cuh"
#include "qgemv_common.cuh"
#include "state_columns.cuh"

#include <cstdlib>

namespace {

constexpr float UNIT_EPS = 1e-6f;  // inside the root of the unit vectors

__device__ __forceinline__ float dr_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }
__device__ __forceinline__ float dr_decay(float a_log, float a, float dt) { return expf(-expf(a_log) * dr_softplus(a + dt)); }
// input of convolution channel c at position pos + t of sequence b (t < 0: earlier than this pass)
__device__ __forceinline__ float conv_in(const fb200_delta_args& a, int b, int c, int t, int pos) {
  if (t >= 0) return a.y[((size_t)b * a.s + t) * a.ldy + c];
  const int p = pos + t;
  if (p < 0) return 0.f;
  return a.ring[((size_t)b * a.taps + p % a.taps) * a.channels + c];
}
__device__ __forceinline__ float conv_silu(const fb200_delta_args& a, int b, int c, int t, int pos) {
  float acc = 0.f;
  for (int j = 0; j < a.taps; ++j) acc = fmaf(a.conv_w[(size_t)j * a.channels + c], conv_in(a, b, c, t - (a.taps - 1) + j, pos), acc);
  return dr_silu(acc);
}

// what the cached inputs contribute to the convolution of channel c at position pos
__device__ __forceinline__ float conv_past(const fb200_delta_args& a, int b, int c, int pos) {
  float acc = 0.f;
#pragma unroll 4
  for (int j = 0; j < a.taps - 1; ++j) {
    const int p = pos - (a.taps - 1) + j;
    if (p >= 0) acc = fmaf(a.conv_w[(size_t)j * a.channels + c], a.ring[((size_t)b * a.taps + p % a.taps) * a.channels + c], acc);
  }
  return acc;
}

// sums of S k and S q over this lane's elements
template <int EPT, int LPC>
__device__ __forceinline__ void column_dots(const float2 (&s)[EPT / 2], const float* ks, const float* qs, int p, float& dk, float& dq) {
  float2 k0 = make_float2(0.f, 0.f), k1 = k0, q0 = k0, q1 = k0;
#pragma unroll
  for (int i = 0; i < EPT / 4; ++i) {
    const float4 k = *reinterpret_cast<const float4*>(ks + 4 * (i * LPC + p));
    const float4 q = *reinterpret_cast<const float4*>(qs + 4 * (i * LPC + p));
    k0 = fma2(s[2 * i], make_float2(k.x, k.y), k0);
    k1 = fma2(s[2 * i + 1], make_float2(k.z, k.w), k1);
    q0 = fma2(s[2 * i], make_float2(q.x, q.y), q0);
    q1 = fma2(s[2 * i + 1], make_float2(q.z, q.w), q1);
  }
  dk = (k0.x + k0.y) + (k1.x + k1.y);
  dq = (q0.x + q0.y) + (q1.x + q1.y);
#pragma unroll
  for (int o = LPC / 2; o > 0; o >>= 1) {
    dk += __shfl_xor_sync(0xFFFFFFFFu, dk, o);
    dq += __shfl_xor_sync(0xFFFFFFFFu, dq, o);
  }
}
// S <- g S + k u
template <int EPT, int LPC>
__device__ __forceinline__ void column_update(float2 (&s)[EPT / 2], const float* ks, int p, float g, float u) {
  const float2 g2 = make_float2(g, g), u2 = make_float2(u, u);
#pragma unroll
  for (int i = 0; i < EPT / 4; ++i) {
    const float4 k = *reinterpret_cast<const float4*>(ks + 4 * (i * LPC + p));
    s[2 * i] = fma2(make_float2(k.x, k.y), u2, mul2(s[2 * i], g2));
    s[2 * i + 1] = fma2(make_float2(k.z, k.w), u2, mul2(s[2 * i + 1], g2));
  }
}

// ---- one new token -------------------------------------------------------------------------------------
constexpr int ST_MAX_THREADS = 512;

template <int EPT, int LPC>
__global__ void __launch_bounds__(ST_MAX_THREADS) delta_step_kernel(const fb200_delta_args a) {
  extern __shared__ __align__(16) float dsm[];  // k, q [dp] (silu of the convolution), read-out [v]
  __shared__ float red[3 * 16], gbs[2];
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  float *ks = dsm, *qs = dsm + a.dp, *os = dsm + 2 * a.dp;
  const int group = a.h / a.hk, hk = h / group;
  const int pos = *a.pos_dev;
  const int p = tid % LPC, cols = nt / LPC, c0 = tid / LPC;
  float* st = a.state + ((size_t)b * a.h + h) * (size_t)a.v * a.dp;
  // the state was written by an earlier step: its loads do not wait for this step's projections
  float2 s[EPT / 2];
  const bool has0 = c0 < a.v && pos > 0;
  if (has0) load_column<EPT, LPC>(st + (size_t)c0 * a.dp, p, s);
  // so were the convolution's older inputs: threads take q [dp] | k [dp], and a lane per column its v channel
  auto qk_channel = [&](int i) { return i < a.dp ? (i < a.d ? hk * a.d + i : -1) : (i - a.dp < a.d ? (a.hk + hk) * a.d + i - a.dp : -1); };
  const int ch0 = tid < 2 * a.dp ? qk_channel(tid) : -1;
  const float past0 = ch0 >= 0 ? conv_past(a, b, ch0, pos) : 0.f, w0 = ch0 >= 0 ? a.conv_w[(size_t)(a.taps - 1) * a.channels + ch0] : 0.f;
  float vpast = 0.f, vw = 0.f;
  if (p == 0 && c0 < a.v) {
    vpast = conv_past(a, b, a.off_v + h * a.v + c0, pos);
    vw = a.conv_w[(size_t)(a.taps - 1) * a.channels + a.off_v + h * a.v + c0];
  }
  pdl_wait();
  pdl_launch_dependents();
  const float* yr = a.y + (size_t)b * a.ldy;
  float v0 = 0.f;
  if (p == 0 && c0 < a.v) v0 = dr_silu(fmaf(vw, yr[a.off_v + h * a.v + c0], vpast));
  v0 = __shfl_sync(0xFFFFFFFFu, v0, lane & ~(LPC - 1));
  for (int i = tid; i < 2 * a.dp; i += nt) {
    const int ch = i == tid ? ch0 : qk_channel(i);
    float x = 0.f;
    if (ch >= 0) x = i == tid ? dr_silu(fmaf(w0, yr[ch], past0)) : conv_silu(a, b, ch, 0, pos);
    (i < a.dp ? qs : ks - a.dp)[i] = x;
  }
  __syncthreads();
  float skk = 0.f, sqq = 0.f, skq = 0.f;
  for (int i = tid; i < a.dp; i += nt) {
    const float k = ks[i], q = qs[i];
    skk = fmaf(k, k, skk);
    sqq = fmaf(q, q, sqq);
    skq = fmaf(k, q, skq);
  }
  skk = warp_sum(skk);
  sqq = warp_sum(sqq);
  skq = warp_sum(skq);
  if (lane == 0) { red[warp] = skk; red[16 + warp] = sqq; red[32 + warp] = skq; }
  if (tid == 0) {
    gbs[0] = dr_decay(a.a_log[h], yr[a.off_a + h], a.dt_bias[h]);
    gbs[1] = dr_sigmoid(yr[a.off_b + h]);
  }
  __syncthreads();
  skk = sqq = skq = 0.f;
  for (int i = 0; i < nw; ++i) { skk += red[i]; sqq += red[16 + i]; skq += red[32 + i]; }
  const float ik = 1.0f / sqrtf(skk + UNIT_EPS), iq = (1.0f / sqrtf(sqq + UNIT_EPS)) / sqrtf((float)a.d);
  const float g = gbs[0], beta = gbs[1], kq = skq * ik * iq;
  float ss = 0.f;
  const int rounds = (a.v + cols - 1) / cols;
  for (int it = 0; it < rounds; ++it) {
    const int c = c0 + it * cols;
    const bool in = c < a.v;
    if (!(it == 0 && has0)) {
      if (in && pos > 0) {
        load_column<EPT, LPC>(st + (size_t)c * a.dp, p, s);
      } else {
#pragma unroll
        for (int i = 0; i < EPT / 2; ++i) s[i] = make_float2(0.f, 0.f);
      }
    }
    const float v = it == 0 ? v0 : in ? conv_silu(a, b, a.off_v + h * a.v + c, 0, pos) : 0.f;
    float dk, dq;
    column_dots<EPT, LPC>(s, ks, qs, p, dk, dq);
    const float u = beta * (v - g * (dk * ik));
    const float o = fmaf(g, dq * iq, u * kq);
    if (in) {
      if (a.commit) {
        column_update<EPT, LPC>(s, ks, p, g, u * ik);
        store_column<EPT, LPC>(st + (size_t)c * a.dp, p, s);
      }
      if (p == 0) {
        os[c] = o;
        ss = fmaf(o, o, ss);
      }
    }
  }
  ss = warp_sum(ss);
  __syncthreads();
  if (lane == 0) red[warp] = ss;
  // this token's convolution inputs, into the slot that no convolution of this step reads
  float* ring = a.ring + ((size_t)b * a.taps + pos % a.taps) * a.channels;
  if (h % group == 0)
    for (int i = tid; i < a.d; i += nt) {
      ring[hk * a.d + i] = yr[hk * a.d + i];
      ring[(a.hk + hk) * a.d + i] = yr[(a.hk + hk) * a.d + i];
    }
  for (int i = tid; i < a.v; i += nt) ring[a.off_v + h * a.v + i] = yr[a.off_v + h * a.v + i];
  __syncthreads();
  ss = 0.f;
  for (int i = 0; i < nw; ++i) ss += red[i];
  const float rms = sqrtf(ss / (float)a.v + a.eps);
  for (int i = tid; i < a.v; i += nt) {
    const float val = (os[i] / rms) * a.out_norm[i] * dr_silu(yr[a.off_g + h * a.v + i]);
    const size_t zi = (size_t)b * a.ldz + h * a.v + i;
    if (a.z_bf16) reinterpret_cast<__nv_bfloat16*>(a.z)[zi] = __float2bfloat16(val);
    else reinterpret_cast<float*>(a.z)[zi] = val;
  }
}

// ---- prompts ---------------------------------------------------------------------------------------------
// Tokens per pass of the recurrence: 8192 tokens of 16 heads of 128 take 1.22 ms, 1.36 with four (heads of 64, 256 and 512 gain alike)
constexpr int CH = 8;
constexpr int PREP_TOK = 4;  // tokens per warp of the preparation
constexpr int PREP_WARPS = 4, PREP_VCH = 128;
constexpr int KK = CH * (CH - 1) / 2, PAIRS = CH * CH;  // k_j . k_i (j < i), then k_j . q_i (j <= i), i-major

// convolution + SiLU of channel c for the PREP_TOK tokens from t0 (zeros from token s on); inputs before this pass come
// from the ring. Addresses are selected, not branched on, so that a channel's loads go out together.
__device__ __forceinline__ void conv_chunk(const fb200_delta_args& a, int b, int c, int t0, int pos, float (&out)[PREP_TOK]) {
#pragma unroll
  for (int i = 0; i < PREP_TOK; ++i) out[i] = 0.f;
  for (int j0 = 0; j0 < a.taps; j0 += 4) {  // four taps at a time meet seven inputs
    float w[4], x[PREP_TOK + 3];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = j0 + j < a.taps ? a.conv_w[(size_t)(j0 + j) * a.channels + c] : 0.f;
#pragma unroll
    for (int r = 0; r < PREP_TOK + 3; ++r) {
      const int t = t0 - (a.taps - 1) + j0 + r, p = pos + t;
      const bool valid = j0 + r < a.taps + PREP_TOK - 1 && t < a.s && p >= 0;
      const float* src = t >= 0 ? a.y + ((size_t)b * a.s + t) * a.ldy + c : a.ring + ((size_t)b * a.taps + (valid ? p % a.taps : 0)) * a.channels + c;
      x[r] = valid ? *src : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j0 + j < a.taps) {  // (what a tap too many would meet are later tokens, which may not be numbers)
#pragma unroll
        for (int i = 0; i < PREP_TOK; ++i) out[i] = fmaf(w[j], x[i + j], out[i]);
      }
  }
#pragma unroll
  for (int i = 0; i < PREP_TOK; ++i) out[i] = t0 + i < a.s ? dr_silu(out[i]) : 0.f;
}

// Sums v[0..31] over the lanes of a warp; lane l returns the total of v[l].
__device__ __forceinline__ float warp_sum32(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
    }
  }
  return v[0];
}

// A warp per (unit, PREP_TOK tokens): units 0 .. hk are the q and k vectors of a q/k head, then blocks of 128 v channels, then
// the decays and write strengths of all heads. NE = channels of a q/k head per lane.
template <int NE>
__global__ void __launch_bounds__(PREP_WARPS * 32) delta_prep_kernel(const fb200_delta_args a) {
  const int lane = threadIdx.x & 31, b = blockIdx.z, t0 = blockIdx.x * PREP_TOK, n = min(PREP_TOK, a.s - t0);
  const int hv = a.h * a.v, vblocks = (hv + PREP_VCH - 1) / PREP_VCH;
  int unit = blockIdx.y * PREP_WARPS + (threadIdx.x >> 5);
  pdl_launch_dependents_small();  // delta_pairs_kernel's launch is over when this one's work is
  const int pos = *a.pos_dev;
  if (unit < a.hk) {
    float q[NE][PREP_TOK], k[NE][PREP_TOK], sum[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) sum[i] = 0.f;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int c = lane + 32 * e;
#pragma unroll
      for (int i = 0; i < PREP_TOK; ++i) q[e][i] = k[e][i] = 0.f;
      if (c < a.d) {
        conv_chunk(a, b, unit * a.d + c, t0, pos, q[e]);
        conv_chunk(a, b, (a.hk + unit) * a.d + c, t0, pos, k[e]);
      }
#pragma unroll
      for (int i = 0; i < PREP_TOK; ++i) {
        sum[i] = fmaf(k[e][i], k[e][i], sum[i]);
        sum[4 + i] = fmaf(q[e][i], q[e][i], sum[4 + i]);
      }
    }
    const float total = warp_sum32(sum);
    const float inv = (1.0f / sqrtf(total + UNIT_EPS)) * (lane >= 4 ? 1.0f / sqrtf((float)a.d) : 1.0f);  // lanes 0..3: k, 4..7: q
#pragma unroll
    for (int i = 0; i < PREP_TOK; ++i) {
      const float ik = __shfl_sync(0xFFFFFFFFu, inv, i), iq = __shfl_sync(0xFFFFFFFFu, inv, 4 + i);
      if (i >= n) continue;
      const size_t row = ((size_t)b * a.s + t0 + i) * a.hk + unit;
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const int c = lane + 32 * e;
        if (c < a.dp) {
          a.qn[row * a.dp + c] = q[e][i] * iq;
          a.kn[row * a.dp + c] = k[e][i] * ik;
        }
      }
    }
    return;
  }
  unit -= a.hk;
  if (unit < vblocks) {
    float v[PREP_VCH / 32][PREP_TOK];
#pragma unroll
    for (int e = 0; e < PREP_VCH / 32; ++e) {
      const int c = unit * PREP_VCH + lane + 32 * e;
      if (c < hv) conv_chunk(a, b, a.off_v + c, t0, pos, v[e]);
    }
#pragma unroll
    for (int e = 0; e < PREP_VCH / 32; ++e) {
      const int c = unit * PREP_VCH + lane + 32 * e;
#pragma unroll
      for (int i = 0; i < PREP_TOK; ++i)
        if (c < hv && i < n) a.vn[((size_t)b * a.s + t0 + i) * hv + c] = v[e][i];
    }
    return;
  }
  if (unit > vblocks) return;
  for (int i = lane; i < n * a.h; i += 32) {
    const int t = t0 + i / a.h, h = i % a.h;
    const size_t row = (size_t)b * a.s + t;
    const float* yr = a.y + row * a.ldy;
    a.gb[(row * a.h + h) * 2] = dr_decay(a.a_log[h], yr[a.off_a + h], a.dt_bias[h]);
    a.gb[(row * a.h + h) * 2 + 1] = dr_sigmoid(yr[a.off_b + h]);
  }
}

// The same with four consecutive channels a lane and eight tokens a warp, for sizes and strides that are multiples of four: 16-byte
// loads, eleven rows of y for eight tokens (seven for four above), 16-byte stores. NE: 128-channel blocks of a q/k head. Bound: HBM and
// its latency. 8192 tokens of 8 + 8 + 16 heads of 128: 129 us (167 above).
constexpr int PREP4_TOK = 8;
__device__ __forceinline__ void conv_chunk4(const fb200_delta_args& a, int b, int c, int t0, int pos, float4 (&out)[PREP4_TOK]) {
#pragma unroll
  for (int i = 0; i < PREP4_TOK; ++i) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = 0; j0 < a.taps; j0 += 4) {
    float4 w[4], x[PREP4_TOK + 3];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = j0 + j < a.taps ? *reinterpret_cast<const float4*>(a.conv_w + (size_t)(j0 + j) * a.channels + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < PREP4_TOK + 3; ++r) {
      const int t = t0 - (a.taps - 1) + j0 + r, p = pos + t;
      const bool valid = j0 + r < a.taps + PREP4_TOK - 1 && t < a.s && p >= 0;
      const float* src = t >= 0 ? a.y + ((size_t)b * a.s + t) * a.ldy + c : a.ring + ((size_t)b * a.taps + (valid ? p % a.taps : 0)) * a.channels + c;
      x[r] = valid ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j0 + j < a.taps) {
#pragma unroll
        for (int i = 0; i < PREP4_TOK; ++i) {
          out[i].x = fmaf(w[j].x, x[i + j].x, out[i].x);
          out[i].y = fmaf(w[j].y, x[i + j].y, out[i].y);
          out[i].z = fmaf(w[j].z, x[i + j].z, out[i].z);
          out[i].w = fmaf(w[j].w, x[i + j].w, out[i].w);
        }
      }
  }
#pragma unroll
  for (int i = 0; i < PREP4_TOK; ++i) {
    const bool in = t0 + i < a.s;
    out[i] = in ? make_float4(dr_silu(out[i].x), dr_silu(out[i].y), dr_silu(out[i].z), dr_silu(out[i].w)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

template <int NE>
__global__ void __launch_bounds__(PREP_WARPS * 32) delta_prep4_kernel(const fb200_delta_args a) {
  const int lane = threadIdx.x & 31, b = blockIdx.z, t0 = blockIdx.x * PREP4_TOK, n = min(PREP4_TOK, a.s - t0);
  const int hv = a.h * a.v, vblocks = (hv + PREP_VCH - 1) / PREP_VCH;
  int unit = blockIdx.y * PREP_WARPS + (threadIdx.x >> 5);
  pdl_launch_dependents_small();
  const int pos = *a.pos_dev;
  if (unit < a.hk) {
    float4 q[NE][PREP4_TOK], k[NE][PREP4_TOK];
    float sum[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) sum[i] = 0.f;
    auto dot = [](float4 x) { return fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w))); };
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int c = 4 * lane + 128 * e;
      if (c < a.d) {
        conv_chunk4(a, b, unit * a.d + c, t0, pos, q[e]);
        conv_chunk4(a, b, (a.hk + unit) * a.d + c, t0, pos, k[e]);
      } else {
#pragma unroll
        for (int i = 0; i < PREP4_TOK; ++i) q[e][i] = k[e][i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < PREP4_TOK; ++i) {
        sum[i] += dot(k[e][i]);
        sum[PREP4_TOK + i] += dot(q[e][i]);
      }
    }
    const float total = warp_sum32(sum);
    const float inv = (1.0f / sqrtf(total + UNIT_EPS)) * (lane >= PREP4_TOK ? 1.0f / sqrtf((float)a.d) : 1.0f);  // lanes 0..7: k, 8..15: q
#pragma unroll
    for (int i = 0; i < PREP4_TOK; ++i) {
      const float ik = __shfl_sync(0xFFFFFFFFu, inv, i), iq = __shfl_sync(0xFFFFFFFFu, inv, PREP4_TOK + i);
      if (i >= n) continue;
      const size_t row = ((size_t)b * a.s + t0 + i) * a.hk + unit;
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const int c = 4 * lane + 128 * e;
        if (c < a.dp) {
          *reinterpret_cast<float4*>(a.qn + row * a.dp + c) = make_float4(q[e][i].x * iq, q[e][i].y * iq, q[e][i].z * iq, q[e][i].w * iq);
          *reinterpret_cast<float4*>(a.kn + row * a.dp + c) = make_float4(k[e][i].x * ik, k[e][i].y * ik, k[e][i].z * ik, k[e][i].w * ik);
        }
      }
    }
    return;
  }
  unit -= a.hk;
  if (unit < vblocks) {
    const int c = unit * PREP_VCH + 4 * lane;
    if (c >= hv) return;
    float4 v[PREP4_TOK];
    conv_chunk4(a, b, a.off_v + c, t0, pos, v);
#pragma unroll
    for (int i = 0; i < PREP4_TOK; ++i)
      if (i < n) *reinterpret_cast<float4*>(a.vn + ((size_t)b * a.s + t0 + i) * hv + c) = v[i];
    return;
  }
  if (unit > vblocks) return;
  for (int i = lane; i < n * a.h; i += 32) {
    const int t = t0 + i / a.h, h = i % a.h;
    const size_t row = (size_t)b * a.s + t;
    const float* yr = a.y + row * a.ldy;
    a.gb[(row * a.h + h) * 2] = dr_decay(a.a_log[h], yr[a.off_a + h], a.dt_bias[h]);
    a.gb[(row * a.h + h) * 2 + 1] = dr_sigmoid(yr[a.off_b + h]);
  }
}

// A warp per (CH tokens, q/k head): k_j . k_i (j < i) and k_j . q_i (j <= i) of the unit vectors; tokens behind the last are zero.
__global__ void __launch_bounds__(PREP_WARPS * 32) delta_pairs_kernel(const fb200_delta_args a) {
  const int lane = threadIdx.x & 31, b = blockIdx.z, t0 = blockIdx.x * CH, hk = blockIdx.y * PREP_WARPS + (threadIdx.x >> 5);
  if (hk >= a.hk) return;
  pdl_wait();
  float sum[2][32];
#pragma unroll
  for (int i = 0; i < 32; ++i) sum[0][i] = sum[1][i] = 0.f;
  for (int c = 4 * lane; c < a.dp; c += 128) {
    float4 k[CH], q[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const size_t at = (((size_t)b * a.s + min(t0 + i, a.s - 1)) * a.hk + hk) * a.dp + c;
      const bool in = t0 + i < a.s;
      k[i] = in ? *reinterpret_cast<const float4*>(a.kn + at) : make_float4(0.f, 0.f, 0.f, 0.f);
      q[i] = in ? *reinterpret_cast<const float4*>(a.qn + at) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    auto dot = [](float4 x, float4 y, float acc) { return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, acc)))); };
#pragma unroll
    for (int i = 0; i < CH; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const int kq = KK + i * (i + 1) / 2 + j;
        sum[kq >> 5][kq & 31] = dot(k[j], q[i], sum[kq >> 5][kq & 31]);
        if (j < i) {
          const int kk = i * (i - 1) / 2 + j;
          sum[kk >> 5][kk & 31] = dot(k[j], k[i], sum[kk >> 5][kk & 31]);
        }
      }
  }
  float* out = a.kq + (((size_t)b * gridDim.x + blockIdx.x) * a.hk + hk) * PAIRS;
  out[lane] = warp_sum32(sum[0]);
  out[32 + lane] = warp_sum32(sum[1]);
}

constexpr int SC_WARPS = 4, CPT = 4;  // columns per group of lanes

// A group of LPC lanes owns CPT columns of S: k and q read from shared memory serve all of them, and the sums are
// reduced so that lane p ends up with those of column p % 4, so one pass over the eight tokens does all columns.
// TOK tokens make a shared-memory stage (a multiple of CH).
template <int EPT, int LPC, int TOK>
__global__ void __launch_bounds__(SC_WARPS * 32) delta_scan_kernel(const fb200_delta_args a) {
  constexpr int DP = EPT * LPC, GROUPS = SC_WARPS * 32 / LPC, COLS = GROUPS * CPT, THREADS = SC_WARPS * 32, NC = TOK / CH;
  // floats of a stage: k, q [TOK][DP], v [COLS][TOK], pairs [NC][PAIRS], g [TOK], beta [TOK]
  constexpr int OV = 2 * TOK * DP, OP = OV + COLS * TOK, OG = OP + NC * PAIRS, STAGE = OG + 2 * TOK;
  constexpr bool KEEP = EPT <= 8;  // k of the eight tokens stays in registers for the update
  extern __shared__ __align__(16) float dsm[];
  const int tid = threadIdx.x, lane = tid & 31, h = blockIdx.y, b = blockIdx.z, group = a.h / a.hk, hk = h / group, hv = a.h * a.v;
  const int p = tid % LPC, cl = tid / LPC, c = blockIdx.x * COLS + cl;  // columns c, c + GROUPS, ..
  const int pos = *a.pos_dev, nchunks = (a.s + CH - 1) / CH;
  const size_t row0 = (size_t)b * a.s;
  auto cp4 = [](const float* dst, const float* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
  auto cp16 = [](const float* dst, const float* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
  auto fetch = [&](int t0, int stage) {
    float* sb = dsm + stage * STAGE;
    const int n = min(TOK, a.s - t0);
    for (int i = tid; i < TOK * (DP / 4); i += THREADS) {
      const int t = i / (DP / 4), e = (i % (DP / 4)) * 4;
      if (t < n) {
        const size_t src = ((row0 + t0 + t) * a.hk + hk) * (size_t)DP + e;
        cp16(sb + t * DP + e, a.kn + src);
        cp16(sb + (TOK + t) * DP + e, a.qn + src);
      } else {  // beyond the last token: k = q = v = 0, g = 1, beta = 0 change nothing
        *reinterpret_cast<float4*>(sb + t * DP + e) = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(sb + (TOK + t) * DP + e) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    for (int i = tid; i < TOK * COLS; i += THREADS) {
      const int t = i / COLS, cc = i % COLS, col = blockIdx.x * COLS + cc;
      if (t < n && col < a.v) cp4(sb + OV + cc * TOK + t, a.vn + (row0 + t0 + t) * hv + h * a.v + col);
      else sb[OV + cc * TOK + t] = 0.f;
    }
    for (int i = tid; i < NC * (PAIRS / 4); i += THREADS) {
      const int ch = t0 / CH + i / (PAIRS / 4), e = (i % (PAIRS / 4)) * 4;
      if (ch < nchunks) cp16(sb + OP + (i / (PAIRS / 4)) * PAIRS + e, a.kq + (((size_t)b * nchunks + ch) * a.hk + hk) * PAIRS + e);
      else *reinterpret_cast<float4*>(sb + OP + (i / (PAIRS / 4)) * PAIRS + e) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int i = tid; i < 2 * TOK; i += THREADS) {
      const int t = i % TOK, f = i / TOK;
      if (t < n) cp4(sb + OG + i, a.gb + ((row0 + t0 + t) * a.h + h) * 2 + f);
      else sb[OG + i] = f ? 0.f : 1.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, 0);
  float2 s[CPT][EPT / 2];
  float* state = a.state + ((size_t)b * a.h + h) * (size_t)a.v * a.dp;
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc) {
    if (c + cc * GROUPS < a.v && pos > 0) {
      load_column<EPT, LPC>(state + (size_t)(c + cc * GROUPS) * a.dp, p, s[cc]);
    } else {
#pragma unroll
      for (int i = 0; i < EPT / 2; ++i) s[cc][i] = make_float2(0.f, 0.f);
    }
  }
  const int stages = (a.s + TOK - 1) / TOK;
  for (int st = 0; st < stages; ++st) {
    if (st + 1 < stages) {
      fetch((st + 1) * TOK, (st + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* sb = dsm + (st & 1) * STAGE;
#pragma unroll 1
    for (int ch = 0; ch < NC; ++ch) {
      const int t0 = st * TOK + ch * CH;
      if (t0 >= a.s) break;
      const float *kb = sb + ch * CH * DP, *qb = sb + (TOK + ch * CH) * DP;
      // ---- a_i = S^T k_i, c_i = S^T q_i over this lane's elements
      float2 kf[KEEP ? CH : 1][EPT / 2];
      float val[CPT][2 * CH];
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        float2 ka[CPT], qa[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) ka[cc] = qa[cc] = make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < EPT / 4; ++e) {
          const float4 k = *reinterpret_cast<const float4*>(kb + i * DP + 4 * (e * LPC + p));
          const float4 q = *reinterpret_cast<const float4*>(qb + i * DP + 4 * (e * LPC + p));
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) {
            ka[cc] = fma2(s[cc][2 * e], make_float2(k.x, k.y), ka[cc]);
            qa[cc] = fma2(s[cc][2 * e], make_float2(q.x, q.y), qa[cc]);
            ka[cc] = fma2(s[cc][2 * e + 1], make_float2(k.z, k.w), ka[cc]);
            qa[cc] = fma2(s[cc][2 * e + 1], make_float2(q.z, q.w), qa[cc]);
          }
          if (KEEP) {
            kf[KEEP ? i : 0][2 * e] = make_float2(k.x, k.y);
            kf[KEEP ? i : 0][2 * e + 1] = make_float2(k.z, k.w);
          }
        }
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          val[cc][i] = ka[cc].x + ka[cc].y;
          val[cc][CH + i] = qa[cc].x + qa[cc].y;
        }
      }
      // ---- totals over the LPC lanes: two halving steps leave lane p with column p % 4, the rest adds up its lanes
#pragma unroll
      for (int x = 0; x < 2 * CH; ++x) {
        const bool odd = lane & 1, high = lane & 2;
        const float s01 = odd ? val[0][x] : val[1][x], k01 = odd ? val[1][x] : val[0][x];
        const float s23 = odd ? val[2][x] : val[3][x], k23 = odd ? val[3][x] : val[2][x];
        const float c01 = k01 + __shfl_xor_sync(0xFFFFFFFFu, s01, 1), c23 = k23 + __shfl_xor_sync(0xFFFFFFFFu, s23, 1);
        float t = (high ? c23 : c01) + __shfl_xor_sync(0xFFFFFFFFu, high ? c01 : c23, 2);
#pragma unroll
        for (int o = 4; o < LPC; o <<= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
        val[0][x] = t;
      }
      // ---- the eight tokens in order
      const int mycol = cl + (p & 3) * GROUPS;
      float gi[CH], bi[CH], vi[CH];
#pragma unroll
      for (int i = 0; i < CH; i += 4) {
        const float4 g4 = *reinterpret_cast<const float4*>(sb + OG + ch * CH + i), b4 = *reinterpret_cast<const float4*>(sb + OG + TOK + ch * CH + i);
        const float4 v4 = *reinterpret_cast<const float4*>(sb + OV + mycol * TOK + ch * CH + i);
        gi[i] = g4.x; gi[i + 1] = g4.y; gi[i + 2] = g4.z; gi[i + 3] = g4.w;
        bi[i] = b4.x; bi[i + 1] = b4.y; bi[i + 2] = b4.z; bi[i + 3] = b4.w;
        vi[i] = v4.x; vi[i + 1] = v4.y; vi[i + 2] = v4.z; vi[i + 3] = v4.w;
      }
      const float* pr = sb + OP + ch * PAIRS;
      float u[CH], out[CH], G = 1.f;
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        G *= gi[i];
        float uk[2] = {G * val[0][i], 0.f}, o[2] = {G * val[0][CH + i], 0.f};  // two chains each
#pragma unroll
        for (int j = 0; j < i; ++j) {
          u[j] *= gi[i];
          uk[j & 1] = fmaf(pr[i * (i - 1) / 2 + j], u[j], uk[j & 1]);
          o[j & 1] = fmaf(pr[KK + i * (i + 1) / 2 + j], u[j], o[j & 1]);
        }
        u[i] = bi[i] * (vi[i] - (uk[0] + uk[1]));
        out[i] = fmaf(pr[KK + i * (i + 1) / 2 + i], u[i], o[0] + o[1]);
      }
      const float2 G2 = make_float2(G, G);
      // every four lanes (one per column) store some of the tokens
      constexpr int QUADS = LPC / 4 < CH ? LPC / 4 : CH, EACH = CH / QUADS;
      if (blockIdx.x * COLS + mycol < a.v) {
        const int quad = p >> 2;
        float* dst = a.o + (row0 + t0 + quad * EACH) * hv + h * a.v + blockIdx.x * COLS + mycol;
#pragma unroll
        for (int e = 0; e < EACH; ++e) {
          float pick[QUADS];  // token quad * EACH + e, by selects (an index would put the array into local memory)
#pragma unroll
          for (int i = 0; i < QUADS; ++i) pick[i] = out[i * EACH + e];
#pragma unroll
          for (int o = QUADS / 2; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < o; ++i) pick[i] = quad & o ? pick[i + o] : pick[i];
          if (quad < QUADS && t0 + quad * EACH + e < a.s) dst[(size_t)e * hv] = pick[0];
        }
      }
      float w[CPT][CH];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
        for (int i = 0; i < CH; ++i) w[cc][i] = __shfl_sync(0xFFFFFFFFu, u[i], (lane & ~3) | cc);
      // ---- S <- G S + sum_j k_j w_j
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
        for (int e = 0; e < EPT / 2; ++e) s[cc][e] = mul2(s[cc][e], G2);
#pragma unroll
      for (int i = 0; i < CH; ++i) {
#pragma unroll
        for (int e = 0; e < EPT / 4; ++e) {
          float2 k0, k1;
          if (KEEP) {
            k0 = kf[KEEP ? i : 0][2 * e];
            k1 = kf[KEEP ? i : 0][2 * e + 1];
          } else {
            const float4 k = *reinterpret_cast<const float4*>(kb + i * DP + 4 * (e * LPC + p));
            k0 = make_float2(k.x, k.y);
            k1 = make_float2(k.z, k.w);
          }
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) {
            const float2 w2 = make_float2(w[cc][i], w[cc][i]);
            s[cc][2 * e] = fma2(k0, w2, s[cc][2 * e]);
            s[cc][2 * e + 1] = fma2(k1, w2, s[cc][2 * e + 1]);
          }
        }
      }
    }
    __syncthreads();  // the stage is free before the one after next lands in it
  }
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc)
    if (c + cc * GROUPS < a.v) store_column<EPT, LPC>(state + (size_t)(c + cc * GROUPS) * a.dp, p, s[cc]);
}

// ---- prompts in chunks of 32 tokens ------------------------------------------------------------------------
// With r_ij = g_(j+1) .. g_i, A_ij = beta_i (k_i . k_j) r_ij (j < i), P_ij = (q_i . k_j) r_ij (j <= i) and S the state before a
// chunk, the recurrence above reads
//   (1 + A) u = beta (v - G K S),   o = G Q S + P u,   S <- G_last S + K^T (r_last u),
// so u = U - W S and o = O + Z S with W = (1 + A)^-1 beta G K, U = (1 + A)^-1 beta v, Z = G Q - P W, O = P U: all that does not
// need the state is formed for all chunks side by side (delta_chunk_kernel), and what is left in order is three products with the
// state per chunk (delta_chunk_scan_kernel). Every decay is a product of decays, never a quotient, and unit k with beta below one
// keep 1 + A well conditioned: its inverse has entries of at most one.
//
// Contractions run on mma.sync with both operands as three bf16 values each, which hold all 24 bits; of the nine products the three
// below 2^-23 of the whole are left out (2^-26 of it in the mean, less than the rounding of a 32-bit sum). Two tf32 values, three products, take the
// same tensor time (four layers of 16 heads of 128, 2048 tokens: 1122 us, now 1141), but they drop bits, and their rounding made
// zero of a NaN. One layer with f32 products around it against 64 bits, 24 prompts of 200 .. 2400 tokens: 4.159e-7 (two tf32 4.198e-7,
// passes of eight 4.151e-7), with decays near one 8.494e-7 (8.524e-7, 8.453e-7).
constexpr int CT = 32;        // tokens of a chunk
constexpr int CDEC = CT + 4;  // decays of a chunk: r_last of every token, then the product of all
constexpr int CK_THREADS = 128, CS_THREADS = 288, CS_STAGES = 3, SCOLS = 16;

__device__ __forceinline__ float4 lds_v4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float2 lds_v2(const float* p) { return *reinterpret_cast<const float2*>(p); }
// Two neighbouring elements as three bf16 each (x in the lower half): 8 bits by a cut, 8 of the rest rounded, and what is left, which
// fits 8 bits: together all 24. A NaN stays one in `hi` (or, by its last bits, in `mid`), an infinite value brings a NaN in `mid`
struct Parts { uint32_t hi, mid, lo; };
__device__ __forceinline__ Parts split_pair(float x, float y) {
  Parts s;
  s.hi = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
  x -= __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
  y -= __uint_as_float(__float_as_uint(y) & 0xFFFF0000u);
  const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
  s.mid = *reinterpret_cast<const uint32_t*>(&m);
  x -= __uint_as_float(s.mid << 16);
  y -= __uint_as_float(s.mid & 0xFFFF0000u);
  s.lo = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
  return s;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Operand A of m16n8k16 from two accumulator tiles [16][8], side by side along K
struct PartsA { uint32_t hi[4], mid[4], lo[4]; };
__device__ __forceinline__ PartsA split_a(const float (&p)[4], const float (&q)[4]) {
  const Parts x0 = split_pair(p[0], p[1]), x1 = split_pair(p[2], p[3]), x2 = split_pair(q[0], q[1]), x3 = split_pair(q[2], q[3]);
  return {{x0.hi, x1.hi, x2.hi, x3.hi}, {x0.mid, x1.mid, x2.mid, x3.mid}, {x0.lo, x1.lo, x2.lo, x3.lo}};
}
// c += a b; the small products apart, the large ones added with rounding (an accumulator of the tensor cores is cut off)
__device__ __forceinline__ void mma_split(float (&c)[4], float (&small)[4], const PartsA& a, const Parts& b0, const Parts& b1) {
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  mma_bf16(small, a.lo, b0.hi, b1.hi);
  mma_bf16(small, a.hi, b0.lo, b1.lo);
  mma_bf16(d, a.hi, b0.hi, b1.hi);
  mma_bf16(small, a.mid, b0.mid, b1.mid);
  mma_bf16(small, a.mid, b0.hi, b1.hi);
  mma_bf16(small, a.hi, b0.mid, b1.mid);
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += d[i];
}
__device__ __forceinline__ bool not_finite(float4 v) { return fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, v.w * 0.f))) != 0.f; }
// v: [eight tokens][token 2 t, 2 t + 1; column g, g + 8]. Where a column has values that are not finite, the tokens from the first on become
// zeros and `cut` goes down to it; whether any lane's column has
__device__ __forceinline__ bool zero_from_bad(float (&v)[4][4], int (&cut)[2], int t) {
  bool any = false;
#pragma unroll
  for (int k = 0; k < 4; ++k) any |= not_finite(make_float4(v[k][0], v[k][1], v[k][2], v[k][3]));
  if (!__any_sync(0xFFFFFFFFu, any)) return false;
  auto token = [&](int k, int i) { return 8 * k + 2 * t + (i & 1); };
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (v[k][i] * 0.f != 0.f) cut[i >> 1] = min(cut[i >> 1], token(k, i));
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    cut[j] = min(cut[j], __shfl_xor_sync(0xFFFFFFFFu, cut[j], 1));
    cut[j] = min(cut[j], __shfl_xor_sync(0xFFFFFFFFu, cut[j], 2));
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (token(k, i) >= cut[i >> 1]) v[k][i] = 0.f;
  return true;
}
// A CTA per (chunk, head): the lower tiles of K K^T and Q K^T; the inverse of 1 + A, whose diagonal blocks of 16 are solved by columns, a
// lane each, and joined by -T22 A21 T11; then 16 columns of [K | V] at a time per warp, transposed: W^T = (beta G K)^T T^T, whose
// accumulators are the operand of (P W)^T = W^T P^T as they are. Writes W and Z (16-byte piece c of row i at c ^ 2 (i & 3)), U in place
// of v, O, and the decays. Zeros that the products meet above the diagonals of T and P keep no value out that is not finite, so tokens from the
// first such k, decay or strength on (values: per column) take part as zeros, and their rows are written as NaN: the rows in front of
// them stay what they are without them. Bound: mma.sync (1728 products of 8.2 cycles a CTA). With a thread per column and the substitution unrolled
// (no products on tensor cores) 8192 tokens of 16 heads took 225 us a layer, most of it fetching that code.
template <int DP>
__global__ void __launch_bounds__(CK_THREADS, 4) delta_chunk_kernel(const fb200_delta_args a) {
  constexpr int LD = DP + 4, LA = CT + 4;
  extern __shared__ __align__(16) float dsm[];
  float *ks = dsm, *qs = dsm + CT * LD;
  __shared__ __align__(16) float A[CT][LA], P[CT][LA], T[CT][LA], M[16][20], gs[CT], bs[CT], Gs[CT];
  __shared__ int bad[CK_THREADS / 32];  // first token whose k, decay or strength is not finite, as the warps see it
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int t0 = blockIdx.x * CT, h = blockIdx.y, b = blockIdx.z, hk = h / (a.h / a.hk), hv = a.h * a.v;
  const int n = min(CT, a.s - t0);
  const size_t row0 = (size_t)b * a.s + t0, chunk = ((size_t)b * a.h + h) * gridDim.x + blockIdx.x;
  pdl_wait();
  int first = CT;
#pragma unroll 4
  for (int i = tid; i < CT * (DP / 4); i += CK_THREADS) {
    const int tk = i / (DP / 4), e = (i % (DP / 4)) * 4;
    const size_t src = ((row0 + min(tk, n - 1)) * a.hk + hk) * (size_t)DP + e;
    const float4 k = *reinterpret_cast<const float4*>(a.kn + src), q = *reinterpret_cast<const float4*>(a.qn + src);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(ks + tk * LD + e) = tk < n ? k : z;
    *reinterpret_cast<float4*>(qs + tk * LD + e) = tk < n ? q : z;
    if (not_finite(k) && tk < n) first = min(first, tk);
  }
  if (tid < CT) {  // tokens behind the last one: decay 1, strength 0
    const float2 gb = *reinterpret_cast<const float2*>(a.gb + ((row0 + min(tid, n - 1)) * a.h + h) * 2);
    gs[tid] = tid < n ? gb.x : 1.f;
    bs[tid] = tid < n ? gb.y : 0.f;
    if (not_finite(make_float4(gb.x, gb.y, 0.f, 0.f)) && tid < n) first = min(first, tid);
  }
  first = __reduce_min_sync(0xFFFFFFFFu, first);
  if (lane == 0) bad[warp] = first;
  __syncthreads();
  first = min(min(bad[0], bad[1]), min(bad[2], bad[3]));
  if (first < CT) {
    for (int i = tid; i < (CT - first) * DP; i += CK_THREADS) ks[(first + i / DP) * LD + i % DP] = 0.f;
    if (tid >= first && tid < CT) {
      gs[tid] = 1.f;
      bs[tid] = 0.f;
    }
    __syncthreads();
  }
  if (warp == 0) {  // decays from token `lane` on, and from the chunk's start; T holds r_ij until the products are there
    float r = 1.f, G = 1.f;
#pragma unroll 8
    for (int i = 0; i < CT; ++i) {
      const float gi = gs[i];
      r = i > lane ? r * gi : 1.f;
      G *= i <= lane ? gi : 1.f;
      T[i][lane] = r;
    }
    Gs[lane] = G;
    float* dec = a.dec + chunk * CDEC;
    dec[lane] = r;
    if (lane == CT - 1) dec[CT] = G;
  }
  // tiles of 16 rows i by 8 rows j with i >= j: (0, 0), (0, 1), (1, 0) .. (1, 3) of K K^T, then of Q K^T; three a warp
  {
    float c[3][4], cs[3][4];
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) c[x][i] = cs[x][i] = 0.f;
    const float* rows = (warp & 2 ? qs : ks);
    // warps 0, 2: (0, 0), (0, 1), (1, 0); warps 1, 3: (1, 1), (1, 2), (1, 3)
    const int m01 = warp & 1 ? 16 : 0, n0 = warp & 1 ? 8 : 0, n1 = warp & 1 ? 16 : 8, n2 = warp & 1 ? 24 : 0;
#pragma unroll 1
    for (int e = 2 * t; e < DP; e += 16) {
      auto rows_a = [&](const float* r) {
        const float2 x0 = lds_v2(r + e), x1 = lds_v2(r + 8 * LD + e), y0 = lds_v2(r + e + 8), y1 = lds_v2(r + 8 * LD + e + 8);
        return split_a({x0.x, x0.y, x1.x, x1.y}, {y0.x, y0.y, y1.x, y1.y});
      };
      auto rows_b = [&](int n, int half) {
        const float2 x = lds_v2(ks + (n + g) * LD + e + 8 * half);
        return split_pair(x.x, x.y);
      };
      const PartsA f = rows_a(rows + (m01 + g) * LD);
      const Parts b0 = rows_b(n0, 0), b1 = rows_b(n0, 1);
      mma_split(c[0], cs[0], f, b0, b1);
      mma_split(c[1], cs[1], f, rows_b(n1, 0), rows_b(n1, 1));
      if (warp & 1) mma_split(c[2], cs[2], f, rows_b(n2, 0), rows_b(n2, 1));
      else mma_split(c[2], cs[2], rows_a(rows + (16 + g) * LD), b0, b1);
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = (x == 2 ? 16 : m01) + g + 8 * (i >> 1), col = (x == 0 ? n0 : x == 1 ? n1 : n2) + 2 * t + (i & 1);
        const float v = (c[x][i] + cs[x][i]) * T[row][col];
        if (warp & 2) P[row][col] = col <= row ? v : 0.f;
        else A[row][col] = col < row ? bs[row] * v : 0.f;
      }
  }
  __syncthreads();
  if (warp == 0) {  // T = (1 + A)^-1
    const int o = lane & 16, j = lane & 15;  // block and column
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s0 = i == j ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
      for (int l = 0; l < i; l += 4) {
        const float4 v = lds_v4(&A[o + i][o + l]);
        s0 = fmaf(-v.x, x[l], s0);
        if (l + 1 < i) s1 = fmaf(-v.y, x[l + 1], s1);
        if (l + 2 < i) s0 = fmaf(-v.z, x[l + 2], s0);
        if (l + 3 < i) s1 = fmaf(-v.w, x[l + 3], s1);
      }
      x[i] = s0 + s1;
      T[o + i][o + j] = x[i];
      if (o == 0) T[i][16 + j] = 0.f;
    }
    __syncwarp();
    const int i = lane & 15, c8 = lane >> 4 << 3;
#pragma unroll
    for (int step = 0; step < 2; ++step) {  // M = A21 T11, then T21 = -T22 M
      float m[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) m[e] = 0.f;
#pragma unroll 4
      for (int l = 0; l < 16; ++l) {
        const float w = step ? -T[16 + i][16 + l] : A[16 + i][l];
        const float4 u = lds_v4(step ? &M[l][c8] : &T[l][c8]), v = lds_v4(step ? &M[l][c8 + 4] : &T[l][c8 + 4]);
        m[0] = fmaf(w, u.x, m[0]); m[1] = fmaf(w, u.y, m[1]); m[2] = fmaf(w, u.z, m[2]); m[3] = fmaf(w, u.w, m[3]);
        m[4] = fmaf(w, v.x, m[4]); m[5] = fmaf(w, v.y, m[5]); m[6] = fmaf(w, v.z, m[6]); m[7] = fmaf(w, v.w, m[7]);
      }
      float* d = step ? &T[16 + i][c8] : &M[i][c8];
      *reinterpret_cast<float4*>(d) = make_float4(m[0], m[1], m[2], m[3]);
      *reinterpret_cast<float4*>(d + 4) = make_float4(m[4], m[5], m[6], m[7]);
      __syncwarp();
    }
  }
  __syncthreads();
  float* wq = a.wq + chunk * (size_t)(2 * CT * DP);
  for (int c0 = 16 * warp; c0 < DP + a.v; c0 += 64) {
    const bool key = c0 < DP;
    const int col = c0 - DP + g;
    const size_t at = row0 * hv + h * a.v + col;
    float d1[4][4], e1[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) d1[x][i] = e1[x][i] = 0.f;
    float in[4][4];  // [eight tokens][token 2 t, 2 t + 1; column g, g + 8]
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tk = 8 * k + 2 * t + (i & 1);
        if (key) in[k][i] = ks[tk * LD + c0 + g + 8 * (i >> 1)];
        else in[k][i] = tk < n && col + 8 * (i >> 1) < a.v ? a.vn[at + (size_t)tk * hv + 8 * (i >> 1)] : 0.f;
      }
    int cut[2] = {first, first};  // tokens of column g and g + 8 from which on rows are NaN
    bool cuts = first < CT;
    cuts |= zero_from_bad(in, cut, t);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tk = 8 * k + 2 * t + (i & 1);
        in[k][i] *= bs[tk] * (key ? Gs[tk] : 1.f);
      }
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
      const PartsA x = split_a(in[k], in[k + 1]);
#pragma unroll
      for (int r = k; r < 4; ++r) {
        const float2 y0 = lds_v2(&T[8 * r + g][8 * k + 2 * t]), y1 = lds_v2(&T[8 * r + g][8 * k + 8 + 2 * t]);
        mma_split(d1[r], e1[r], x, split_pair(y0.x, y0.y), split_pair(y1.x, y1.y));
      }
    }
    float d2[4][4], e2[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        d1[x][i] += e1[x][i];
        d2[x][i] = e2[x][i] = 0.f;
      }
    cuts |= zero_from_bad(d1, cut, t);
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
      const PartsA x = split_a(d1[k], d1[k + 1]);
#pragma unroll
      for (int r = k; r < 4; ++r) {
        const float2 y0 = lds_v2(&P[8 * r + g][8 * k + 2 * t]), y1 = lds_v2(&P[8 * r + g][8 * k + 8 + 2 * t]);
        mma_split(d2[r], e2[r], x, split_pair(y0.x, y0.y), split_pair(y1.x, y1.y));
      }
    }
    if (cuts)
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (8 * r + 2 * t + (i & 1) >= cut[i >> 1]) d1[r][i] = d2[r][i] = __uint_as_float(0x7FC00000u);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tk = 8 * r + 2 * t + (i & 1), c = c0 + g + 8 * (i >> 1);
        const float pw = d2[r][i] + e2[r][i];
        if (key) {
          float* w = wq + tk * DP + (((c >> 2) ^ ((tk & 3) << 1)) << 2) + (c & 3);
          w[0] = d1[r][i];
          w[CT * DP] = fmaf(Gs[tk], qs[tk * LD + c], -pw);
        } else if (tk < n && c < DP + a.v) {
          const size_t to = at + (size_t)tk * hv + 8 * (i >> 1);
          a.vn[to] = d1[r][i];
          a.o[to] = pw;
        }
      }
  }
}

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// A CTA per (16 columns of S, head). Warps 0 .. 3 carry the recurrence: each holds a quarter of d of S^T [16][d] as accumulator tiles,
// which are the A operands of S^T W^T as they are; the quarters' sums meet in shared memory, become w = r_last (U - W S), again an A
// operand, and S^T <- G S^T + w^T K. Warps 4 .. 7 follow with the read-out O + Z S from a copy of S, a chunk behind at most. Warp 8
// fetches the matrices two chunks ahead (what 128 CTAs have in flight a chunk ahead is too little for HBM). The update is summed
// from zero and added to S in one rounding, so S drifts no more than with 32-bit sums. Bound: issue (144 products of 8.2 cycles and
// 1500 other instructions per chunk and scheduler) and the chain of a chunk: 3500 cycles. 8192 tokens of 16 heads of 128: 0.51 ms and 0.19
// ms of preparation (with two tf32 values 0.49 and 0.18; delta_scan_kernel: 1.22 ms and 0.03).
template <int DP>
__global__ void __launch_bounds__(CS_THREADS, 1) delta_chunk_scan_kernel(const fb200_delta_args a) {
  constexpr int KS = DP / 4, KT = KS / 8, MAT = CT * DP, KLD = DP + 4;  // a warp's part of d, in tiles of 8; floats of a matrix, of a row of K
  extern __shared__ __align__(16) float dsm[];  // STAGES x (W, K); STAGES x Z; two copies of S [4][KT][32 lanes] float4
  __shared__ uint64_t full[2][CS_STAGES], empty[2][CS_STAGES];
  __shared__ __align__(16) float4 part[2][4][4][32];  // [half][warp][tile of 8 rows][lane]
  __shared__ uint2 ws[3][4][32];                      // w: hi, mid, lo; tile of 8 rows; a pair of column g, a pair of column g + 8
  const int tid = threadIdx.x & 127, lane = tid & 31, warp = tid >> 5, half = threadIdx.x >> 7, g = lane >> 2, t = lane & 3;
  const int h = blockIdx.y, b = blockIdx.z, hk = h / (a.h / a.hk), hv = a.h * a.v, c0 = blockIdx.x * SCOLS, nch = (a.s + CT - 1) / CT;
  const size_t row0 = (size_t)b * a.s, chunk0 = ((size_t)b * a.h + h) * nch;
  const int STAGE = half ? MAT : MAT + CT * KLD;
  float* stages = dsm + (half ? CS_STAGES * (MAT + CT * KLD) : 0);
  float4* copies = reinterpret_cast<float4*>(dsm + CS_STAGES * (2 * MAT + CT * KLD));
  constexpr int COPY = 4 * KT * 32;
  const int FULL = 3, EMPTY = 5;  // barriers of the copies (1, 2: the halves' own)
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * CS_STAGES; ++i) {
      mbar_init(smem_u32(&full[i / CS_STAGES][i % CS_STAGES]), 1);
      mbar_init(smem_u32(&empty[i / CS_STAGES][i % CS_STAGES]), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  if (threadIdx.x >= 256) {  // the last warp fetches: a matrix in one copy, a row of K per lane (rows behind the last token are zero)
    for (int ch = 0; ch < nch; ++ch) {
      const int st = ch % CS_STAGES;
      const uint32_t round = (uint32_t)(ch / CS_STAGES);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float* dst = dsm + (x ? CS_STAGES * (MAT + CT * KLD) + st * MAT : st * (MAT + CT * KLD));
        const uint32_t bar = smem_u32(&full[x][st]);
        const int rows = x ? 0 : min(CT, a.s - ch * CT);
        if (round > 0) mbar_wait(smem_u32(&empty[x][st]), (round - 1) & 1, a.status);
        if (!x && lane >= rows)
          for (int e = 0; e < DP; e += 4) *reinterpret_cast<float4*>(dst + MAT + lane * KLD + e) = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        if (lane == 0) {
          mbar_expect_tx(bar, (uint32_t)(MAT + rows * DP) * 4);
          bulk_g2s(smem_u32(dst), a.wq + ((chunk0 + ch) * 2 + x) * (size_t)MAT, MAT * 4, bar);
        }
        __syncwarp();
        if (lane < rows) bulk_g2s(smem_u32(dst + MAT + lane * KLD), a.kn + ((row0 + ch * CT + lane) * a.hk + hk) * (size_t)DP, DP * 4, bar);
      }
    }
    return;
  }
  auto release = [&](int ch) {  // this warp is through with its half's stage
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[half][ch % CS_STAGES])) : "memory");
  };
  // what the sums of a chunk are added to (rows 8 warp + 2 t + i % 2, columns c0 + g + 8 (i / 2)), and its decays
  struct Ahead { float base[4], rl[2], G; };
  auto look = [&](int ch, Ahead& n) {
    const float* add = half ? a.o : a.vn;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tk = ch * CT + 8 * warp + 2 * t + (i & 1), col = c0 + g + 8 * (i >> 1);
      n.base[i] = tk < a.s && col < a.v ? add[(row0 + tk) * hv + h * a.v + col] : 0.f;
    }
    if (half || ch >= nch) return;
    const float* dec = a.dec + (chunk0 + ch) * CDEC;
    n.rl[0] = dec[8 * warp + 2 * t];
    n.rl[1] = dec[8 * warp + 2 * t + 1];
    n.G = dec[CT];
  };
  Ahead next = {};
  look(0, next);
  const int pos = *a.pos_dev;
  float* state = a.state + ((size_t)b * a.h + h) * (size_t)a.v * DP;
  // entry i of tile x: column c0 + g + 8 (i / 2), element warp KS + 8 x + 2 t + i % 2
  float s[KT][4];
  if (!half) {
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const int col = c0 + g + 4 * i;
        const float2 v = col < a.v && pos > 0 ? *reinterpret_cast<const float2*>(state + (size_t)col * DP + warp * KS + 8 * x + 2 * t) : make_float2(0.f, 0.f);
        s[x][i] = v.x;
        s[x][i + 1] = v.y;
      }
  }
  for (int ch = 0; ch < nch; ++ch) {
    if (half) bar_sync(2, 128);  // the sums of the chunk before have been read
    const float* st = stages + ch % CS_STAGES * STAGE;
    float4* copy = copies + (ch & 1) * COPY + warp * KT * 32 + lane;
    const Ahead now = next;
    look(ch + 1, next);
    if (half) {
      bar_sync(FULL + (ch & 1), 256);
#pragma unroll
      for (int x = 0; x < KT; ++x) {
        const float4 v = copy[x * 32];
        s[x][0] = v.x; s[x][1] = v.y; s[x][2] = v.z; s[x][3] = v.w;
      }
      if (ch + 2 < nch) bar_arrive(EMPTY + (ch & 1), 256);
    } else {
      if (ch >= 2) bar_sync(EMPTY + (ch & 1), 256);
#pragma unroll
      for (int x = 0; x < KT; ++x) copy[x * 32] = make_float4(s[x][0], s[x][1], s[x][2], s[x][3]);
      bar_arrive(FULL + (ch & 1), 256);
    }
    mbar_wait(smem_u32(&full[half][ch % CS_STAGES]), (uint32_t)(ch / CS_STAGES) & 1, a.status);
    // ---- this warp's part of S^T (W or Z)^T: 16 columns by four tiles of 8 rows
    float c[4][4], cs[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) c[j][i] = cs[j][i] = 0.f;
#pragma unroll
    for (int x = 0; x < KT; x += 2) {
      const PartsA f = split_a(s[x], s[x + 1]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        auto part_b = [&](int tile) {
          const int piece = (warp * KS + 8 * tile) / 4 + (t >> 1);
          const float2 v = lds_v2(st + (8 * j + g) * DP + ((piece ^ ((g & 3) << 1)) << 2) + 2 * (t & 1));
          return split_pair(v.x, v.y);
        };
        mma_split(c[j], cs[j], f, part_b(x), part_b(x + 1));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) part[half][warp][j][lane] = make_float4(c[j][0] + cs[j][0], c[j][1] + cs[j][1], c[j][2] + cs[j][2], c[j][3] + cs[j][3]);
    bar_sync(1 + half, 128);
    float sum[4];
    {
      const float4 p0 = part[half][0][warp][lane], p1 = part[half][1][warp][lane], p2 = part[half][2][warp][lane], p3 = part[half][3][warp][lane];
      sum[0] = (p0.x + p1.x) + (p2.x + p3.x);
      sum[1] = (p0.y + p1.y) + (p2.y + p3.y);
      sum[2] = (p0.z + p1.z) + (p2.z + p3.z);
      sum[3] = (p0.w + p1.w) + (p2.w + p3.w);
    }
    if (half) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tk = ch * CT + 8 * warp + 2 * t + (i & 1), col = c0 + g + 8 * (i >> 1);
        if (tk < a.s && col < a.v) a.o[(row0 + tk) * hv + h * a.v + col] = now.base[i] + sum[i];
      }
      release(ch);
      continue;
    }
    {
      float w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = ch * CT + 8 * warp + 2 * t + (i & 1) < a.s ? now.rl[i & 1] * (now.base[i] - sum[i]) : 0.f;
      const Parts p0 = split_pair(w[0], w[1]), p1 = split_pair(w[2], w[3]);
      ws[0][warp][lane] = make_uint2(p0.hi, p1.hi);
      ws[1][warp][lane] = make_uint2(p0.mid, p1.mid);
      ws[2][warp][lane] = make_uint2(p0.lo, p1.lo);
    }
    bar_sync(1, 128);
    // ---- S^T <- G S^T + w^T K
    const float* kb = st + MAT;
    float up[KT][4], us[KT][4];
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) up[x][i] = us[x][i] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {  // tokens 8 j ..
      const uint2 h0 = ws[0][j][lane], h1 = ws[0][j + 1][lane], m0 = ws[1][j][lane], m1 = ws[1][j + 1][lane], l0 = ws[2][j][lane], l1 = ws[2][j + 1][lane];
      const PartsA f = {{h0.x, h0.y, h1.x, h1.y}, {m0.x, m0.y, m1.x, m1.y}, {l0.x, l0.y, l1.x, l1.y}};
#pragma unroll
      for (int x = 0; x < KT; ++x) {
        const float* p = kb + (8 * j + 2 * t) * KLD + warp * KS + 8 * x + g;
        mma_split(up[x], us[x], f, split_pair(p[0], p[KLD]), split_pair(p[8 * KLD], p[9 * KLD]));
      }
    }
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[x][i] = fmaf(now.G, s[x][i], up[x][i] + us[x][i]);
    release(ch);
  }
  if (!half) {
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const int col = c0 + g + 4 * i;
        if (col < a.v) *reinterpret_cast<float2*>(state + (size_t)col * DP + warp * KS + 8 * x + 2 * t) = make_float2(s[x][i], s[x][i + 1]);
      }
  }
}

// A warp per (row, head): RMSNorm over v, the plain weight, the SiLU gate.
__global__ void __launch_bounds__(256) delta_out_kernel(const fb200_delta_args a) {
  const int lane = threadIdx.x & 31;
  const size_t id = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (id >= (size_t)a.b * a.s * a.h) return;
  const size_t row = id / a.h;
  const int h = (int)(id % a.h);
  const float* o = a.o + id * a.v;
  const float* g = a.y + row * a.ldy + a.off_g + h * a.v;
  float ss = 0.f;
  for (int i = lane; i < a.v; i += 32) ss = fmaf(o[i], o[i], ss);
  const float rms = sqrtf(warp_sum(ss) / (float)a.v + a.eps);
  for (int i = lane; i < a.v; i += 32) {
    const float val = (o[i] / rms) * a.out_norm[i] * dr_silu(g[i]);
    const size_t zi = row * a.ldz + h * a.v + i;
    if (a.z_bf16) reinterpret_cast<__nv_bfloat16*>(a.z)[zi] = __float2bfloat16(val);
    else reinterpret_cast<float*>(a.z)[zi] = val;
  }
}

// The same with 16-byte pieces, all of a row's loads before the first use: NV x 128 values. 8192 rows of 16 x 128: 43 us (66 above).
template <int NV>
__global__ void __launch_bounds__(256) delta_out4_kernel(const fb200_delta_args a) {
  const int lane = threadIdx.x & 31;
  const size_t id = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (id >= (size_t)a.b * a.s * a.h) return;
  const size_t row = id / a.h;
  const int h = (int)(id % a.h);
  const float* o = a.o + id * a.v;
  const float* g = a.y + row * a.ldy + a.off_g + h * a.v;
  float4 x[NV], y[NV], w[NV];
#pragma unroll
  for (int e = 0; e < NV; ++e) {
    const int c = 128 * e + 4 * lane;
    const bool in = c < a.v;
    x[e] = in ? *reinterpret_cast<const float4*>(o + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    y[e] = in ? *reinterpret_cast<const float4*>(g + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    w[e] = in ? *reinterpret_cast<const float4*>(a.out_norm + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < NV; ++e) ss += fmaf(x[e].x, x[e].x, fmaf(x[e].y, x[e].y, fmaf(x[e].z, x[e].z, x[e].w * x[e].w)));
  const float rms = sqrtf(warp_sum(ss) / (float)a.v + a.eps);
#pragma unroll
  for (int e = 0; e < NV; ++e) {
    const int c = 128 * e + 4 * lane;
    if (c >= a.v) continue;
    const float4 r = make_float4((x[e].x / rms) * w[e].x * dr_silu(y[e].x), (x[e].y / rms) * w[e].y * dr_silu(y[e].y),
                                 (x[e].z / rms) * w[e].z * dr_silu(y[e].z), (x[e].w / rms) * w[e].w * dr_silu(y[e].w));
    const size_t zi = row * a.ldz + h * a.v + c;
    if (a.z_bf16) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(r.x, r.y), hi = __floats2bfloat162_rn(r.z, r.w);
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.z) + zi) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    } else {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.z) + zi) = r;
    }
  }
}

// The last min(s, taps) inputs of every sequence into their slots (after every convolution of the pass has run).
__global__ void conv_ring_kernel(const fb200_delta_args a) {
  const int n = min(a.s, a.taps), pos = *a.pos_dev;
  const size_t total = (size_t)a.b * n * a.channels;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % a.channels), t = a.s - 1 - (int)(i / a.channels % n), b = (int)(i / a.channels / n);
    a.ring[((size_t)b * a.taps + (pos + t) % a.taps) * a.channels + c] = a.y[((size_t)b * a.s + t) * a.ldy + c];
  }
}

template <int EPT, int LPC>
int launch_step(fb200_device* dev, const fb200_delta_args& a) {
  int threads = (a.v * LPC + 31) / 32 * 32;
  threads = threads > ST_MAX_THREADS ? ST_MAX_THREADS : threads < 64 ? 64 : threads;
  const size_t smem = (size_t)(2 * a.dp + a.v) * 4;
  return fb200_launch(dev, delta_step_kernel<EPT, LPC>, dim3((unsigned)a.h, (unsigned)a.b), dim3((unsigned)threads), smem, true, a);
}

template <int EPT, int LPC, int TOK>
int launch_scan(fb200_device* dev, const fb200_delta_args& a) {
  constexpr int DP = EPT * LPC, COLS = SC_WARPS * 32 / LPC * CPT;
  constexpr size_t smem = (size_t)2 * (2 * TOK * DP + COLS * TOK + TOK / CH * PAIRS + 2 * TOK) * 4;
  static bool configured[64] = {false};
  if (!configured[dev->ordinal & 63]) {
    FB_CUDA(dev, cudaFuncSetAttribute(delta_scan_kernel<EPT, LPC, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev->ordinal & 63] = true;
  }
  delta_scan_kernel<EPT, LPC, TOK><<<dim3((unsigned)((a.v + COLS - 1) / COLS), (unsigned)a.h, (unsigned)a.b), SC_WARPS * 32, smem, dev->stream>>>(a);
  FB_LAUNCH_CHECK(dev);
  return FB200_OK;
}

template <int DP>
int launch_chunks(fb200_device* dev, const fb200_delta_args& a) {
  const unsigned nch = (unsigned)((a.s + CT - 1) / CT);
  constexpr int ck_smem = 2 * CT * (DP + 4) * 4, cs_smem = (CS_STAGES * CT * (3 * DP + 4) + 2 * SCOLS * DP) * 4;
  static bool configured[64] = {false};
  if (!configured[dev->ordinal & 63]) {
    FB_CUDA(dev, cudaFuncSetAttribute(delta_chunk_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ck_smem));
    FB_CUDA(dev, cudaFuncSetAttribute(delta_chunk_scan_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, cs_smem));
    configured[dev->ordinal & 63] = true;
  }
  if (int rc = fb200_launch(dev, delta_chunk_kernel<DP>, dim3(nch, (unsigned)a.h, (unsigned)a.b), dim3(CK_THREADS), ck_smem, true, a)) return rc;
  return fb200_launch(dev, delta_chunk_scan_kernel<DP>, dim3((unsigned)((a.v + SCOLS - 1) / SCOLS), (unsigned)a.h, (unsigned)a.b),
                      dim3(CS_THREADS), cs_smem, true, a);
}

template <int NE>
int launch_prep(fb200_device* dev, const fb200_delta_args& a) {
  const int units = a.hk + (a.h * a.v + PREP_VCH - 1) / PREP_VCH + 1;
  const bool by4 = !((a.d | a.v | a.off_v | (int)(a.ldy & 3)) & 3) &&
                   !((reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.conv_w) | reinterpret_cast<uintptr_t>(a.ring)) & 15);
  auto launch = [&](auto kernel, int tok) {
    kernel<<<dim3((unsigned)((a.s + tok - 1) / tok), (unsigned)((units + PREP_WARPS - 1) / PREP_WARPS), (unsigned)a.b), PREP_WARPS * 32, 0, dev->stream>>>(a);
  };
  bool pieces = false;
  if constexpr (NE <= 8) {  // (heads of 512 need more registers than there are)
    if ((pieces = by4)) launch(delta_prep4_kernel<(NE + 3) / 4>, PREP4_TOK);
  }
  if (!pieces) launch(delta_prep_kernel<NE>, PREP_TOK);
  FB_LAUNCH_CHECK(dev);
  return FB200_OK;
}

}  // namespace

// Chunks of 32 tokens or passes of eight. A chunk's preparation has a longer chain than a few passes, and the scan over chunks takes 16 columns
// a CTA and one CTA per SM, where the passes take 32 columns and two CTAs share an SM. Four layers, b = 1, passes / chunks in us:
//   heads of 128, v 128         192 tokens    256          512          2048
//    8  ( 64 CTAs of 148 SMs)   356 /  349   402 /  386   554 /  453   1540 /  914
//   16  (128)                   391 /  398   418 /  413   605 /  518   1686 / 1141
//   24  (192)                               498 /  518   733 /  681   2208 / 1821
//   32  (256)                   481 /  525   542 /  557   802 /  751   2376 / 2092
//   40  (320)                               681 /  665  1060 /  965   3310 / 2729
//   54  (432)                               760 /  751  1166 / 1080   3528 / 3071
//   64  (512)                   707 /  777   816 /  872  1243 / 1309   3706 / 3840
//   heads of 64, v 64           192           256          512          1024          4096
//   16  ( 64)                   349 /  324   392 /  332   563 /  406
//   32  (128)                   391 /  359   432 /  375   622 /  470
//   38  (152)                                            648 /  628   1049 /  995   3452 / 3069
//   48  (192)                                            672 /  674   1096 / 1053   3634 / 3352
//   64  (256)                   449 /  466   532 /  532   761 /  791   1230 / 1243   3951 / 3841
// (384 tokens of 20, 32, 36, 40 and 54 heads of 128: 610 / 581, 683 / 675, 698 / 683, 872 / 804, 962 / 936.)
// What counts is columns, not heads: 8 heads of four sequences or of four times the columns lie where 32 heads do (16 heads of 128, four sequences:
// 512 tokens 1130 / 1201, as 64 heads). Heads of more than 128 do not fit: three stages of their matrices take 290 KB.
// Models in float32 keep the passes of eight, whose error is the smaller one (by 0.2 %, see above): there a chunk rounds W, U and Z
// between its products. FB200_DELTA_CHUNKS=1 takes chunks wherever the head size allows, 0 never.
bool fb200_delta_in_chunks(const fb200_device* dev, int dp, int h, int v, int b, int s, bool bf16) {
  if (s == 1 || (dp != 64 && dp != 128)) return false;
  if (const char* e = getenv("FB200_DELTA_CHUNKS")) return e[0] == '1';
  const long ctas = (long)b * h * ((v + SCOLS - 1) / SCOLS), sms = dev->sm_count;
  if (!bf16) return false;
  if (dp == 64) return ctas <= sms ? s >= 192 : 2 * ctas <= 3 * sms && s >= 512;
  return 2 * ctas <= sms ? s >= 192 : ctas <= sms ? s >= 256 : ctas <= 3 * sms && s >= 384;
}
size_t fb200_delta_wq_floats(int b, int s, int h, int dp) { return (size_t)b * h * ((s + CT - 1) / CT) * 2 * CT * dp; }
size_t fb200_delta_dec_floats(int b, int s, int h) { return (size_t)b * h * ((s + CT - 1) / CT) * CDEC; }

int fb200_delta_dp(int d) {
  for (int dp : {32, 64, 128, 256, 512})
    if (d <= dp) return dp;
  return 0;
}

int fb200_delta_step(fb200_device* dev, const fb200_delta_args& a) {
  switch (a.dp) {
    case 32: return launch_step<8, 4>(dev, a);
    case 64: return launch_step<16, 4>(dev, a);
    case 128: return launch_step<32, 4>(dev, a);
    case 256: return launch_step<32, 8>(dev, a);
    case 512: return launch_step<32, 16>(dev, a);
    default: return fb200_fail(dev, FB200_ERR_INVALID_SHAPE, "delta rule: head size %d", a.d);
  }
}

int fb200_delta_prompt(fb200_device* dev, const fb200_delta_args& a) {
  int rc;
  switch (a.dp) {
    case 32: rc = launch_prep<1>(dev, a); break;
    case 64: rc = launch_prep<2>(dev, a); break;
    case 128: rc = launch_prep<4>(dev, a); break;
    case 256: rc = launch_prep<8>(dev, a); break;
    case 512: rc = launch_prep<16>(dev, a); break;
    default: return fb200_fail(dev, FB200_ERR_INVALID_SHAPE, "delta rule: head size %d", a.d);
  }
  if (rc) return rc;
  if (a.wq && fb200_delta_in_chunks(dev, a.dp, a.h, a.v, a.b, a.s, a.z_bf16)) {
    rc = a.dp == 64 ? launch_chunks<64>(dev, a) : launch_chunks<128>(dev, a);
  } else {
    rc = fb200_launch(dev, delta_pairs_kernel, dim3((unsigned)((a.s + CH - 1) / CH), (unsigned)((a.hk + PREP_WARPS - 1) / PREP_WARPS), (unsigned)a.b),
                      dim3(PREP_WARPS * 32), 0, true, a);
    if (rc) return rc;
    switch (a.dp) {
      case 32: rc = launch_scan<4, 8, 16>(dev, a); break;
      case 64: rc = launch_scan<4, 16, 16>(dev, a); break;
      case 128:
        // 16 lanes per column group do less per token (fewer shuffles); 32 lanes make more CTAs where there are few heads
        if ((a.v + 15) / 16 * a.h * a.b <= dev->sm_count) rc = launch_scan<4, 32, 16>(dev, a);
        else rc = launch_scan<8, 16, 16>(dev, a);
        break;
      case 256: rc = launch_scan<8, 32, 16>(dev, a); break;
      default: rc = launch_scan<16, 32, 8>(dev, a); break;
    }
  }
  if (rc) return rc;
  const size_t warps = (size_t)a.b * a.s * a.h;
  const bool by4 = !((a.v | a.off_g | (int)((a.ldy | a.ldz) & 3)) & 3) && a.v <= 512 &&
                   !((reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.z) | reinterpret_cast<uintptr_t>(a.out_norm)) & 15);
  const unsigned blocks = (unsigned)((warps + 7) / 8);
  if (by4 && a.v <= 128) delta_out4_kernel<1><<<blocks, 256, 0, dev->stream>>>(a);
  else if (by4) delta_out4_kernel<4><<<blocks, 256, 0, dev->stream>>>(a);
  else delta_out_kernel<<<blocks, 256, 0, dev->stream>>>(a);
  FB_LAUNCH_CHECK(dev);
  conv_ring_kernel<<<(unsigned)(a.channels / 256 + 1), 256, 0, dev->stream>>>(a);
  FB_LAUNCH_CHECK(dev);
  return FB200_OK;
}
