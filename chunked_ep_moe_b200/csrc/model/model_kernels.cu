// Bandwidth-bound pieces of the decoder around the MoE layers, each as one kernel instead of a chain of framework
// elementwise kernels: residual add + RMSNorm (forward and backward), rotary embedding of q and k straight out of the
// fused qkv projection (forward and backward), and the cross-entropy of bf16 logits (forward and backward).
// The reference ships no model code (its host model lived in an external MaxText branch); these serve the trainer of
// `models/deepseek_tiny.py`.
#include "model_kernels.cuh"

#include <cuda_bf16.h>

#include <cfloat>
#include <type_traits>

#include "../common/umma.cuh"

namespace cem {

namespace {

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t bf_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int kNormThreads = 256;  // 8 warps, one row per warp at a time
constexpr int kMaxNormUnits = 8;   // 16-byte units per lane: rows of up to 8 * 32 * 8 = 2048 columns

// The norm kernels are instantiated per number of 16-byte units a lane holds of a row (UNITS): sized for 2048 columns, the
// 1024-column norms of the decoder paid for twice the registers and ran with 8 warps per SM. All of a row's loads go out
// before the first value is used. 8192 rows of 1024 columns: forward 18 -> 10.5 us,
// backward 37 -> 13.4 us, its column sums 11.6 -> 4.6 us (67 MB take 10.2 us at the measured copy rate).

__device__ __forceinline__ void unpack8(const int4& v, float (&f)[8]) {
  const uint32_t w[4] = {(uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) { f[2 * e] = bf_lo(w[e]); f[2 * e + 1] = bf_hi(w[e]); }
}

// s = x + delta (rounded to bf16, as the unfused residual add stores it); y = s * rsqrt(mean(s^2) + eps) * w.
template <int UNITS>
__global__ void __launch_bounds__(kNormThreads, UNITS <= 4 ? 3 : 1)
add_rms_norm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* delta, const __nv_bfloat16* w,
                        __nv_bfloat16* s_out, __nv_bfloat16* y, float* rstd_out, int rows, int cols, float eps) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = cols >> 3;
  const int4 zero = make_int4(0, 0, 0, 0);
  for (int row = blockIdx.x * (kNormThreads / 32) + warp; row < rows; row += gridDim.x * (kNormThreads / 32)) {
    const int4* xr = reinterpret_cast<const int4*>(x + static_cast<size_t>(row) * cols);
    const int4* dr = reinterpret_cast<const int4*>(delta + static_cast<size_t>(row) * cols);
    int4 a[UNITS], b[UNITS];
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
      const int u = lane + 32 * i;
      a[i] = u < units ? xr[u] : zero;
      b[i] = delta != nullptr && u < units ? dr[u] : zero;
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
      float av[8], bv[8];
      unpack8(a[i], av);
      unpack8(b[i], bv);
      uint32_t so[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        so[e] = bf_pack(av[2 * e] + bv[2 * e], av[2 * e + 1] + bv[2 * e + 1]);
        const float lo = bf_lo(so[e]), hi = bf_hi(so[e]);
        ss += lo * lo + hi * hi;
      }
      a[i] = make_int4(so[0], so[1], so[2], so[3]);
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / cols + eps);
    if (lane == 0) rstd_out[row] = rstd;
    const int4* wr = reinterpret_cast<const int4*>(w);
    int4* sr = reinterpret_cast<int4*>(s_out + static_cast<size_t>(row) * cols);
    int4* yr = reinterpret_cast<int4*>(y + static_cast<size_t>(row) * cols);
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
      const int u = lane + 32 * i;
      if (u < units) {
        float v[8], wv[8];
        unpack8(a[i], v);
        unpack8(wr[u], wv);
        uint32_t yo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) yo[e] = bf_pack(v[2 * e] * rstd * wv[2 * e], v[2 * e + 1] * rstd * wv[2 * e + 1]);
        if (delta) sr[u] = a[i];
        yr[u] = make_int4(yo[0], yo[1], yo[2], yo[3]);
      }
    }
  }
}

// ds = ds_in + rstd * (dy * w) - s * rstd^3 / D * sum(dy * w * s);  dw partial = sum over this block's rows of
// dy * s * rstd, one fp32 row per block (summed afterwards in fixed order).
template <int UNITS>
__global__ void __launch_bounds__(kNormThreads, UNITS <= 4 ? 2 : 1)
add_rms_norm_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* ds_in, const __nv_bfloat16* s,
                        const __nv_bfloat16* w, const float* rstd_in, __nv_bfloat16* ds_out, float* dw_partial,
                        int rows, int cols) {
  extern __shared__ float s_dw[];  // [8 warps][cols]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = cols >> 3;
  const int4 zero = make_int4(0, 0, 0, 0);
  float dw_acc[UNITS][8];
  const int4* wr = reinterpret_cast<const int4*>(w);
#pragma unroll
  for (int i = 0; i < UNITS; ++i) {
#pragma unroll
    for (int e = 0; e < 8; ++e) dw_acc[i][e] = 0.0f;
  }
  for (int row = blockIdx.x * (kNormThreads / 32) + warp; row < rows; row += gridDim.x * (kNormThreads / 32)) {
    const int4* gr = reinterpret_cast<const int4*>(dy + static_cast<size_t>(row) * cols);
    const int4* sr = reinterpret_cast<const int4*>(s + static_cast<size_t>(row) * cols);
    const int4* ir = reinterpret_cast<const int4*>(ds_in + static_cast<size_t>(row) * cols);
    const float rstd = rstd_in[row];
    int4 gq[UNITS], sq[UNITS], iq[UNITS];
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
      const int u = lane + 32 * i;
      gq[i] = u < units ? gr[u] : zero;
      sq[i] = u < units ? sr[u] : zero;
      iq[i] = ds_in != nullptr && u < units ? ir[u] : zero;
    }
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
      float g[8], sv[8], wv[8];
      unpack8(gq[i], g);
      unpack8(sq[i], sv);
      const int u = lane + 32 * i;
      unpack8(u < units ? wr[u] : zero, wv);  // (from L1: kept in registers they would spill)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        dw_acc[i][2 * e] += g[2 * e] * sv[2 * e] * rstd;
        dw_acc[i][2 * e + 1] += g[2 * e + 1] * sv[2 * e + 1] * rstd;
        dot += g[2 * e] * wv[2 * e] * sv[2 * e] + g[2 * e + 1] * wv[2 * e + 1] * sv[2 * e + 1];
      }
    }
    dot = warp_sum(dot);
    const float coef = dot * rstd * rstd * rstd / cols;
    int4* outr = reinterpret_cast<int4*>(ds_out + static_cast<size_t>(row) * cols);
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
      const int u = lane + 32 * i;
      if (u < units) {
        float g[8], sv[8], wv[8], in[8];
        unpack8(gq[i], g);
        unpack8(sq[i], sv);
        unpack8(wr[u], wv);
        unpack8(iq[i], in);
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          o[e] = bf_pack(in[2 * e] + g[2 * e] * wv[2 * e] * rstd - sv[2 * e] * coef,
                         in[2 * e + 1] + g[2 * e + 1] * wv[2 * e + 1] * rstd - sv[2 * e + 1] * coef);
        outr[u] = make_int4(o[0], o[1], o[2], o[3]);
      }
    }
  }
  // Block-level sum of the eight warps' weight-gradient rows, then one row of partials per block.
#pragma unroll
  for (int i = 0; i < UNITS; ++i) {
    const int u = lane + 32 * i;
    if (u < units)
#pragma unroll
      for (int e = 0; e < 8; ++e) s_dw[warp * cols + u * 8 + e] = dw_acc[i][e];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float t = 0.0f;
#pragma unroll
    for (int wi = 0; wi < kNormThreads / 32; ++wi) t += s_dw[wi * cols + c];
    dw_partial[static_cast<size_t>(blockIdx.x) * cols + c] = t;
  }
}

// dW = column sums of the blocks' partials, fp32 in fixed order, rounded once. Eight warps take every eighth row of 32
// columns each.
__global__ void __launch_bounds__(256) norm_dw_kernel(const float* partial, int blocks, int cols, __nv_bfloat16* dw) {
  __shared__ float sums[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  float t = 0.0f;
  if (c < cols) {
#pragma unroll 8
    for (int r = warp; r < blocks; r += 8) t += partial[static_cast<size_t>(r) * cols + c];
  }
  sums[warp][lane] = t;
  __syncthreads();
  if (warp == 0 && c < cols) {
    for (int i = 1; i < 8; ++i) t += sums[i][lane];
    dw[c] = __float2bfloat16_rn(t);
  }
}

// qkv [B, S, 3, H, hd] -> q, k (rotated) and v as contiguous [B, H, S, hd]. cos/sin: [S, hd/2] fp32.
// `inverse`: rotate by -theta and write back into the qkv layout (the backward).
template <bool kBackward>
__global__ void __launch_bounds__(256) rope_qkv_kernel(__nv_bfloat16* qkv, HeadMatrix q, HeadMatrix k, HeadMatrix v,
                                                       const float* cos_t, const float* sin_t, int B, int S, int H, int hd) {
  const int units = hd >> 3;  // 8 values = 4 rotation pairs per unit
  const size_t total = static_cast<size_t>(B) * S * H * units;
  for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int u = static_cast<int>(idx % units);
    size_t rest = idx / units;
    const int h = static_cast<int>(rest % H); rest /= H;
    const int s = static_cast<int>(rest % S);
    const int b = static_cast<int>(rest / S);
    const size_t in_base = ((static_cast<size_t>(b) * S + s) * 3 * H + h) * hd + static_cast<size_t>(u) * 8;
    auto at = [&](const HeadMatrix& m) {
      return reinterpret_cast<int4*>(static_cast<__nv_bfloat16*>(m.data) + b * m.batch + h * m.head + s * m.row + u * 8);
    };
    const float4 c = *reinterpret_cast<const float4*>(cos_t + static_cast<size_t>(s) * (hd >> 1) + u * 4);
    const float4 sn = *reinterpret_cast<const float4*>(sin_t + static_cast<size_t>(s) * (hd >> 1) + u * 4);
    const float cs[4] = {c.x, c.y, c.z, c.w};
    const float ss[4] = {kBackward ? -sn.x : sn.x, kBackward ? -sn.y : sn.y, kBackward ? -sn.z : sn.z,
                         kBackward ? -sn.w : sn.w};
#pragma unroll
    for (int part = 0; part < 2; ++part) {  // q then k
      int4* rot = at(part == 0 ? q : k);
      const size_t in_off = in_base + static_cast<size_t>(part) * H * hd;
      const int4 raw = kBackward ? *rot
                                 : *reinterpret_cast<const int4*>(qkv + in_off);
      const uint32_t wds[4] = {(uint32_t)raw.x, (uint32_t)raw.y, (uint32_t)raw.z, (uint32_t)raw.w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x1 = bf_lo(wds[e]), x2 = bf_hi(wds[e]);
        o[e] = bf_pack(x1 * cs[e] - x2 * ss[e], x1 * ss[e] + x2 * cs[e]);
      }
      const int4 res = make_int4(o[0], o[1], o[2], o[3]);
      if (kBackward) *reinterpret_cast<int4*>(qkv + in_off) = res;
      else *rot = res;
    }
    const size_t v_off = in_base + static_cast<size_t>(2) * H * hd;
    if (kBackward) *reinterpret_cast<int4*>(qkv + v_off) = *at(v);
    else *at(v) = *reinterpret_cast<const int4*>(qkv + v_off);
  }
}

// 2^x, subnormal results flushed to zero: a term below 2^-126 is nothing beside the largest, which is 1.
__device__ __forceinline__ float exp2_term(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Cross-entropy of bf16 logits, one CTA per row: loss[row] = logsumexp(row) - row[target]; lse is kept for the backward.
// Bound by the read of the logits as long as enough of it is in flight and the exponentials are all that a value costs beside two or three
// other instructions: four 16-byte loads a thread, one rescaling of the sum for their 32 values, subtraction, scaling and sum two values an
// instruction, the maximum on pairs of bf16. 8192 x 32000: 112 us with one load and one rescaling at a time, 103 us with four, 92 us like this
// (5.2e8 bytes: 82 us at the measured copy rate).
__global__ void __launch_bounds__(256) cross_entropy_fwd_kernel(const __nv_bfloat16* logits, const int64_t* targets,
                                                                float* loss, float* lse_out, int cols) {
  constexpr int kAhead = 4;
  constexpr float kLog2e = 1.4426950408889634f;
  __shared__ float s_m[8], s_s[8];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int4* lr = reinterpret_cast<const int4*>(logits + static_cast<size_t>(row) * cols);
  const int units = cols >> 3;
  const f32x2 log2e = make_f32x2(kLog2e, kLog2e);
  float m = -FLT_MAX, sum = 0.0f;  // online softmax: sum of exp(v - m); finite, so that a batch of -inf adds nothing
  for (int u0 = threadIdx.x; u0 < units; u0 += kAhead * 256) {
    int4 raw[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)  // (past the end the first once more: no larger a maximum, and left out of the sum)
      raw[k] = lr[u0 + k * 256 < units ? u0 + k * 256 : u0];
    __nv_bfloat162 top = *reinterpret_cast<const __nv_bfloat162*>(&raw[0].x);
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw[k]);
#pragma unroll
      for (int e = 0; e < 4; ++e) top = __hmax2(top, pairs[e]);
    }
    const float mx = fmaxf(m, fmaxf(__low2float(top), __high2float(top)));
    const f32x2 less = make_f32x2(-mx, -mx);
    f32x2 add = make_f32x2(sum * exp2_term((m - mx) * kLog2e), 0.0f);
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      if (u0 + k * 256 >= units) break;
      const uint32_t wds[4] = {(uint32_t)raw[k].x, (uint32_t)raw[k].y, (uint32_t)raw[k].z, (uint32_t)raw[k].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float lo, hi;
        split_f32x2(mul2(add2(make_f32x2(bf_lo(wds[e]), bf_hi(wds[e])), less), log2e), &lo, &hi);
        add = add2(add, make_f32x2(exp2_term(lo), exp2_term(hi)));
      }
    }
    float even, odd;
    split_f32x2(add, &even, &odd);
    sum = even + odd;
    m = mx;
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, sum, o);
    const float nm = fmaxf(m, om);
    sum = (nm == -INFINITY) ? 0.0f : sum * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  if (lane == 0) { s_m[warp] = m; s_s[warp] = sum; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float fm = s_m[0], fs = s_s[0];
    for (int i = 1; i < 8; ++i) {
      const float nm = fmaxf(fm, s_m[i]);
      fs = (nm == -INFINITY) ? 0.0f : fs * __expf(fm - nm) + s_s[i] * __expf(s_m[i] - nm);
      fm = nm;
    }
    const float lse = fm + __logf(fs);
    lse_out[row] = lse;
    loss[row] = lse - __bfloat162float(logits[static_cast<size_t>(row) * cols + targets[row]]);
  }
}

// dlogits = (softmax - onehot(target)) * scale, bf16.
__global__ void __launch_bounds__(256) cross_entropy_bwd_kernel(const __nv_bfloat16* logits, const int64_t* targets,
                                                                const float* lse, const float* grad_scale,
                                                                __nv_bfloat16* dlogits, int cols) {
  const int row = blockIdx.x;
  const int4* lr = reinterpret_cast<const int4*>(logits + static_cast<size_t>(row) * cols);
  int4* dr = reinterpret_cast<int4*>(dlogits + static_cast<size_t>(row) * cols);
  const float l = lse[row], scale = *grad_scale;
  const int target = static_cast<int>(targets[row]);
  const int units = cols >> 3;
  for (int u = threadIdx.x; u < units; u += blockDim.x) {
    const int4 raw = lr[u];
    const uint32_t wds[4] = {(uint32_t)raw.x, (uint32_t)raw.y, (uint32_t)raw.z, (uint32_t)raw.w};
    float p[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) { p[2 * e] = __expf(bf_lo(wds[e]) - l); p[2 * e + 1] = __expf(bf_hi(wds[e]) - l); }
    const int t = target - u * 8;
    if (t >= 0 && t < 8) p[t] -= 1.0f;
    dr[u] = make_int4(bf_pack(p[0] * scale, p[1] * scale), bf_pack(p[2] * scale, p[3] * scale),
                      bf_pack(p[4] * scale, p[5] * scale), bf_pack(p[6] * scale, p[7] * scale));
  }
}

// act = silu(gate) * up for gu = [gate | up] (two contiguous halves of `ffn` columns per row), eight columns a thread.
__global__ void __launch_bounds__(256) dense_swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* act,
                                                               size_t units, int ffn_units) {
  for (size_t u = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; u < units;
       u += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = u / ffn_units, c = u - row * ffn_units;
    const int4 g = reinterpret_cast<const int4*>(gu)[row * 2 * ffn_units + c];
    const int4 v = reinterpret_cast<const int4*>(gu)[row * 2 * ffn_units + ffn_units + c];
    const uint32_t gw[4] = {(uint32_t)g.x, (uint32_t)g.y, (uint32_t)g.z, (uint32_t)g.w};
    const uint32_t vw[4] = {(uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float g0 = bf_lo(gw[e]), g1 = bf_hi(gw[e]);
      o[e] = bf_pack(g0 * __fdividef(1.0f, 1.0f + __expf(-g0)) * bf_lo(vw[e]),
                     g1 * __fdividef(1.0f, 1.0f + __expf(-g1)) * bf_hi(vw[e]));
    }
    reinterpret_cast<int4*>(act)[u] = make_int4(o[0], o[1], o[2], o[3]);
  }
}

// d_gu = [d_act * up * silu'(gate) | d_act * silu(gate)].
__global__ void __launch_bounds__(256) dense_swiglu_bwd_kernel(const __nv_bfloat16* gu, const __nv_bfloat16* d_act,
                                                               __nv_bfloat16* d_gu, size_t units, int ffn_units) {
  for (size_t u = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; u < units;
       u += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = u / ffn_units, c = u - row * ffn_units;
    const size_t gi = row * 2 * ffn_units + c, vi = gi + ffn_units;
    const int4 g = reinterpret_cast<const int4*>(gu)[gi];
    const int4 v = reinterpret_cast<const int4*>(gu)[vi];
    const int4 d = reinterpret_cast<const int4*>(d_act)[u];
    const uint32_t gw[4] = {(uint32_t)g.x, (uint32_t)g.y, (uint32_t)g.z, (uint32_t)g.w};
    const uint32_t vw[4] = {(uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w};
    const uint32_t dw[4] = {(uint32_t)d.x, (uint32_t)d.y, (uint32_t)d.z, (uint32_t)d.w};
    uint32_t og[4], ov[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float dg[2], dv[2];
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        const float gt = z ? bf_hi(gw[e]) : bf_lo(gw[e]);
        const float up = z ? bf_hi(vw[e]) : bf_lo(vw[e]);
        const float da = z ? bf_hi(dw[e]) : bf_lo(dw[e]);
        const float sig = __fdividef(1.0f, 1.0f + __expf(-gt));
        const float sl = gt * sig;
        dg[z] = da * up * (sig + sl * (1.0f - sig));
        dv[z] = da * sl;
      }
      og[e] = bf_pack(dg[0], dg[1]);
      ov[e] = bf_pack(dv[0], dv[1]);
    }
    reinterpret_cast<int4*>(d_gu)[gi] = make_int4(og[0], og[1], og[2], og[3]);
    reinterpret_cast<int4*>(d_gu)[vi] = make_int4(ov[0], ov[1], ov[2], ov[3]);
  }
}

}  // namespace

// Calls `f` with the smallest instantiated number of units per lane that holds a row.
template <typename F>
static void for_norm_units(int cols, F&& f) {
  const int per_lane = ((cols >> 3) + 31) >> 5;
  if (per_lane <= 1) f(std::integral_constant<int, 1>{});
  else if (per_lane == 2) f(std::integral_constant<int, 2>{});
  else if (per_lane == 3) f(std::integral_constant<int, 3>{});
  else if (per_lane == 4) f(std::integral_constant<int, 4>{});
  else f(std::integral_constant<int, kMaxNormUnits>{});
}

void launch_add_rms_norm_fwd(const void* x, const void* delta, const void* w, void* s_out, void* y, float* rstd,
                             int rows, int cols, float eps, cudaStream_t stream) {
  int grid = (rows + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
  if (grid < 1) grid = 1;
  for_norm_units(cols, [&](auto units) {
    add_rms_norm_fwd_kernel<decltype(units)::value><<<grid, kNormThreads, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(delta),
        static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(s_out), static_cast<__nv_bfloat16*>(y), rstd,
        rows, cols, eps);
  });
}

int add_rms_norm_bwd_blocks(int rows) {
  int grid = (rows + 7) / 8;
  if (grid > 148 * 2) grid = 148 * 2;
  return grid < 1 ? 1 : grid;
}

void launch_add_rms_norm_bwd(const void* dy, const void* ds_in, const void* s, const void* w, const float* rstd,
                             void* ds_out, float* dw_partial, void* dw, int rows, int cols, cudaStream_t stream) {
  const int grid = add_rms_norm_bwd_blocks(rows);
  const size_t smem = static_cast<size_t>(kNormThreads / 32) * cols * sizeof(float);
  for_norm_units(cols, [&](auto units) {
    constexpr int kUnits = decltype(units)::value;
    // (64 KB at 2048 columns: above the default limit)
    static const cudaError_t configured = cudaFuncSetAttribute(
        add_rms_norm_bwd_kernel<kUnits>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUnits * 8192);
    (void)configured;
    add_rms_norm_bwd_kernel<kUnits><<<grid, kNormThreads, smem, stream>>>(
        static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(ds_in),
        static_cast<const __nv_bfloat16*>(s), static_cast<const __nv_bfloat16*>(w), rstd,
        static_cast<__nv_bfloat16*>(ds_out), dw_partial, rows, cols);
  });
  norm_dw_kernel<<<(cols + 31) / 32, 256, 0, stream>>>(dw_partial, grid, cols, static_cast<__nv_bfloat16*>(dw));
}

void launch_rope_qkv(void* qkv, HeadMatrix q, HeadMatrix k, HeadMatrix v, const float* cos_t, const float* sin_t, int B, int S, int H,
                     int hd, bool backward, cudaStream_t stream) {
  const size_t total = static_cast<size_t>(B) * S * H * (hd >> 3);
  int grid = static_cast<int>((total + 255) / 256);
  if (grid > 148 * 16) grid = 148 * 16;
  if (grid < 1) grid = 1;
  if (backward)
    rope_qkv_kernel<true><<<grid, 256, 0, stream>>>(static_cast<__nv_bfloat16*>(qkv), q, k, v, cos_t, sin_t, B, S, H, hd);
  else
    rope_qkv_kernel<false><<<grid, 256, 0, stream>>>(static_cast<__nv_bfloat16*>(qkv), q, k, v, cos_t, sin_t, B, S, H, hd);
}

void launch_cross_entropy_fwd(const void* logits, const int64_t* targets, float* loss, float* lse, int rows, int cols,
                              cudaStream_t stream) {
  cross_entropy_fwd_kernel<<<rows, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), targets, loss, lse,
                                                     cols);
}

void launch_cross_entropy_bwd(const void* logits, const int64_t* targets, const float* lse, const float* grad_scale,
                              void* dlogits, int rows, int cols, cudaStream_t stream) {
  cross_entropy_bwd_kernel<<<rows, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), targets, lse,
                                                     grad_scale, static_cast<__nv_bfloat16*>(dlogits), cols);
}

void launch_dense_swiglu(const void* gu, const void* d_act, void* out, int rows, int ffn, bool backward,
                         cudaStream_t stream) {
  const size_t units = static_cast<size_t>(rows) * (ffn >> 3);
  if (units == 0) return;
  int grid = static_cast<int>((units + 255) / 256);
  if (grid > 148 * 16) grid = 148 * 16;
  if (backward)
    dense_swiglu_bwd_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(gu),
                                                      static_cast<const __nv_bfloat16*>(d_act),
                                                      static_cast<__nv_bfloat16*>(out), units, ffn >> 3);
  else
    dense_swiglu_fwd_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(gu),
                                                      static_cast<__nv_bfloat16*>(out), units, ffn >> 3);
}

}  // namespace cem
