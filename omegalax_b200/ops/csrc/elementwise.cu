// Memory-bound kernels (K4, K5, K13, K14 and the softmax half of K6).  Every kernel moves
// 16-byte vectors where the layout allows it and does its arithmetic in fp32.
#include "host_utils.h"
#include "sm100_common.cuh"

namespace ob {

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = 0.f;
  for (int i = 0; i < nw; ++i) r += red[i];
  return r;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = -INFINITY;
  for (int i = 0; i < nw; ++i) r = fmaxf(r, red[i]);
  return r;
}

// ------------------------------------------------------------------ RMSNorm (K4)
// y = x * rsqrt(mean(x^2) + eps) * (w or 1+w).  One CTA per row, D % 8 == 0.
template <bool kOnePlus>
__global__ void rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                   bf16* __restrict__ y, float* __restrict__ rstd_out, int D,
                                   float eps) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * D);
  const int nv = D >> 3;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) prefetch_l2(reinterpret_cast<const uint4*>(w) + i);
  grid_begin();
  float ss = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 q = xr[i];
    uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16(u[j]);
      ss += f.x * f.x + f.y * f.y;
    }
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / (float)D + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + row * D);
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 q = xr[i], ww = wr[i], o;
    uint32_t u[4] = {q.x, q.y, q.z, q.w}, wu[4] = {ww.x, ww.y, ww.z, ww.w}, ou[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16(u[j]), g = unpack_bf16(wu[j]);
      if (kOnePlus) { g.x += 1.f; g.y += 1.f; }
      ou[j] = pack_bf16(f.x * rstd * g.x, f.y * rstd * g.y);
    }
    o.x = ou[0]; o.y = ou[1]; o.z = ou[2]; o.w = ou[3];
    yr[i] = o;
  }
}

// dx = rstd * (dy*w - x * rstd^2 * mean(dy*w*x));  dw += sum_rows dy * x * rstd.
// A CTA walks rows blockIdx.x, +gridDim.x, ... with the next row's loads in flight and its dw partial in registers
// (D <= blockDim.x * 8 * kMaxVec).  The partials of a cluster of eight meet in shared memory before they
// leave as one coalesced addition per column: 592 CTAs that added element by element queued 4736 deep on
// every 32 bytes of dw, which took longer than the rows.  In us, before and after: 999 rows of 1024 47.7, 5.3;
// 4096 of 2048 101.6, 14.5; 8192 of 4096 90.7, 47.3 (201 MB: 4.3 TB/s).
constexpr int kRmsCluster = 8;

template <bool kOnePlus, int kMaxVec>
__global__ void __cluster_dims__(kRmsCluster, 1, 1) __launch_bounds__(256)
rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                   const float* __restrict__ rstd_in, bf16* __restrict__ dx, float* __restrict__ dw, int M, int D, float eps) {
  __shared__ float red[32];
  extern __shared__ __align__(16) float dw_sm[];      // [D]
  const int nv = D >> 3;
  float dwacc[kMaxVec][8];
  uint4 ww[kMaxVec], q[kMaxVec], g[kMaxVec], qn[kMaxVec], gn[kMaxVec];
  const uint4 none = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int a = 0; a < kMaxVec; ++a) {
    const int i = threadIdx.x + a * blockDim.x;
    ww[a] = i < nv ? reinterpret_cast<const uint4*>(w)[i] : none;
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[a][j] = 0.f;
  }
  float rstd_n = 0.f;
  auto fetch = [&](long long row) {
    if (row < M && rstd_in) rstd_n = rstd_in[row];
#pragma unroll
    for (int a = 0; a < kMaxVec; ++a) {
      const int i = threadIdx.x + a * blockDim.x;
      const bool in = row < M && i < nv;
      qn[a] = in ? reinterpret_cast<const uint4*>(x + row * D)[i] : none;
      gn[a] = in ? reinterpret_cast<const uint4*>(dy + row * D)[i] : none;
    }
  };
  fetch(blockIdx.x);
  for (long long row = blockIdx.x; row < M; row += gridDim.x) {
    float rstd = rstd_n;
#pragma unroll
    for (int a = 0; a < kMaxVec; ++a) {
      q[a] = qn[a];
      g[a] = gn[a];
    }
    fetch(row + gridDim.x);
    if (!rstd_in) {
      float ss = 0.f;
#pragma unroll
      for (int a = 0; a < kMaxVec; ++a) {
        const uint32_t u[4] = {q[a].x, q[a].y, q[a].z, q[a].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 f = unpack_bf16(u[j]);
          ss += f.x * f.x + f.y * f.y;
        }
      }
      ss = block_sum(ss, red);
      rstd = rsqrtf(ss / (float)D + eps);
    }
    float dot = 0.f;
#pragma unroll
    for (int a = 0; a < kMaxVec; ++a) {
      const uint32_t u[4] = {q[a].x, q[a].y, q[a].z, q[a].w}, gu[4] = {g[a].x, g[a].y, g[a].z, g[a].w},
                     wu[4] = {ww[a].x, ww[a].y, ww[a].z, ww[a].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 xf = unpack_bf16(u[j]), gf = unpack_bf16(gu[j]), wf = unpack_bf16(wu[j]);
        if (kOnePlus) { wf.x += 1.f; wf.y += 1.f; }
        dot += gf.x * wf.x * xf.x + gf.y * wf.y * xf.y;
        dwacc[a][2 * j] += gf.x * xf.x * rstd;
        dwacc[a][2 * j + 1] += gf.y * xf.y * rstd;
      }
    }
    dot = block_sum(dot, red);
    const float c = dot * rstd * rstd * rstd / (float)D;
    uint4* dxr = reinterpret_cast<uint4*>(dx + row * D);
#pragma unroll
    for (int a = 0; a < kMaxVec; ++a) {
      const int i = threadIdx.x + a * blockDim.x;
      if (i < nv) {
        const uint32_t u[4] = {q[a].x, q[a].y, q[a].z, q[a].w}, gu[4] = {g[a].x, g[a].y, g[a].z, g[a].w},
                       wu[4] = {ww[a].x, ww[a].y, ww[a].z, ww[a].w};
        uint32_t ou[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 xf = unpack_bf16(u[j]), gf = unpack_bf16(gu[j]), wf = unpack_bf16(wu[j]);
          if (kOnePlus) { wf.x += 1.f; wf.y += 1.f; }
          ou[j] = pack_bf16(gf.x * wf.x * rstd - xf.x * c, gf.y * wf.y * rstd - xf.y * c);
        }
        dxr[i] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
      }
    }
  }
  if (dw) {      // the same for every CTA of the cluster
#pragma unroll
    for (int a = 0; a < kMaxVec; ++a) {
      const int i = threadIdx.x + a * blockDim.x;
      if (i < nv) {
        float4* d = reinterpret_cast<float4*>(dw_sm + i * 8);
        d[0] = make_float4(dwacc[a][0], dwacc[a][1], dwacc[a][2], dwacc[a][3]);
        d[1] = make_float4(dwacc[a][4], dwacc[a][5], dwacc[a][6], dwacc[a][7]);
      }
    }
    cluster_sync_all();
    const uint32_t base = smem_u32(dw_sm);
    for (int c = cluster_ctarank() * blockDim.x + threadIdx.x; c < D; c += kRmsCluster * blockDim.x) {
      float t = 0.f;
#pragma unroll
      for (int r = 0; r < kRmsCluster; ++r) {
        float v;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(mapa_shared(base + c * 4, r)) : "memory");
        t += v;
      }
      atomicAdd(dw + c, t);
    }
    cluster_sync_all();      // nobody leaves while its partial may still be read
  }
}

// ------------------------------------------------------------------ SwiGLU (K5)
// gu is [M, 2F] = [gate | up];  act = silu(gate) * up.
// rows (may be null): a device count of the rows that matter, the first ones.
__global__ void swiglu_fwd_kernel(const bf16* __restrict__ gu, bf16* __restrict__ act, const int* __restrict__ rows, long long M,
                                  int F) {
  grid_begin();
  if (rows) M = min(M, (long long)*rows);
  const int fv = F >> 3;
  const long long total = M * fv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    long long m = idx / fv;
    int c = (int)(idx - m * fv);
    const uint4 g = reinterpret_cast<const uint4*>(gu + m * 2 * F)[c];
    const uint4 u = reinterpret_cast<const uint4*>(gu + m * 2 * F + F)[c];
    uint32_t ga[4] = {g.x, g.y, g.z, g.w}, ua[4] = {u.x, u.y, u.z, u.w}, oa[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 gf = unpack_bf16(ga[j]), uf = unpack_bf16(ua[j]);
      float a = gf.x / (1.f + __expf(-gf.x)) * uf.x;
      float b = gf.y / (1.f + __expf(-gf.y)) * uf.y;
      oa[j] = pack_bf16(a, b);
    }
    uint4 o; o.x = oa[0]; o.y = oa[1]; o.z = oa[2]; o.w = oa[3];
    reinterpret_cast<uint4*>(act + m * F)[c] = o;
  }
}

// dgu = [dact * up * dsilu(gate) | dact * silu(gate)]; optionally also re-emits act.
// dgu may be gu itself (no __restrict__ on the two): every thread reads its eight gate and up
// values before it writes the gradients to the same places, and no other thread touches them.
__global__ void swiglu_bwd_kernel(const bf16* gu, const bf16* __restrict__ dact, bf16* dgu,
                                  bf16* __restrict__ act_out, const int* __restrict__ rows, long long M, int F) {
  if (rows) M = min(M, (long long)*rows);
  const int fv = F >> 3;
  const long long total = M * fv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    long long m = idx / fv;
    int c = (int)(idx - m * fv);
    const uint4 g = reinterpret_cast<const uint4*>(gu + m * 2 * F)[c];
    const uint4 u = reinterpret_cast<const uint4*>(gu + m * 2 * F + F)[c];
    const uint4 d = reinterpret_cast<const uint4*>(dact + m * F)[c];
    uint32_t ga[4] = {g.x, g.y, g.z, g.w}, ua[4] = {u.x, u.y, u.z, u.w},
             da[4] = {d.x, d.y, d.z, d.w}, dg[4], du[4], ao[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 gf = unpack_bf16(ga[j]), uf = unpack_bf16(ua[j]), df = unpack_bf16(da[j]);
      float s0 = 1.f / (1.f + __expf(-gf.x)), s1 = 1.f / (1.f + __expf(-gf.y));
      float si0 = gf.x * s0, si1 = gf.y * s1;
      dg[j] = pack_bf16(df.x * uf.x * s0 * (1.f + gf.x * (1.f - s0)),
                        df.y * uf.y * s1 * (1.f + gf.y * (1.f - s1)));
      du[j] = pack_bf16(df.x * si0, df.y * si1);
      ao[j] = pack_bf16(si0 * uf.x, si1 * uf.y);
    }
    uint4 o; o.x = dg[0]; o.y = dg[1]; o.z = dg[2]; o.w = dg[3];
    reinterpret_cast<uint4*>(dgu + m * 2 * F)[c] = o;
    o.x = du[0]; o.y = du[1]; o.z = du[2]; o.w = du[3];
    reinterpret_cast<uint4*>(dgu + m * 2 * F + F)[c] = o;
    if (act_out) {
      o.x = ao[0]; o.y = ao[1]; o.z = ao[2]; o.w = ao[3];
      reinterpret_cast<uint4*>(act_out + m * F)[c] = o;
    }
  }
}

// ------------------------------------------------------------------ QK-RMSNorm + RoPE
// qkv: [M, (H+2G)*K] (q heads, then k heads, then v heads).  For every q and k head:
// per-head RMSNorm over K with weight (qw / kw, or 1+w), then rotate-half RoPE on the
// first `rot` channels using cos/sin tables [M, rot/2] (fp32).  Outputs q_out [M,H,K],
// k_out [M,G,K].  One warp per (row, head).
template <bool kOnePlus>
__global__ void qknorm_rope_fwd_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ qw,
                                       const bf16* __restrict__ kw, const float* __restrict__ cosT,
                                       const float* __restrict__ sinT, bf16* __restrict__ q_out,
                                       bf16* __restrict__ k_out, long long M, int H, int G, int K,
                                       int rot, float eps, int q_in_stride_heads) {
  const int lane = threadIdx.x & 31;
  const long long wid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int HG = H + G;
  if (wid >= M * HG) return;
  const long long m = wid / HG;
  const int h = (int)(wid - m * HG);
  const bool is_q = h < H;
  // q heads may be interleaved with a per-head gate (q_in_stride_heads = 2 for gated attention)
  const long long in_off = is_q ? (long long)h * K * q_in_stride_heads
                                : (long long)H * K * q_in_stride_heads + (long long)(h - H) * K;
  const long long row_stride = (long long)H * K * q_in_stride_heads + 2ll * G * K;
  const bf16* src = qkv + m * row_stride + in_off;
  const bf16* w = is_q ? qw : kw;
  bf16* dst = is_q ? q_out + (m * H + h) * K : k_out + (m * G + (h - H)) * K;
  float ss = 0.f;
  for (int i = lane; i < K; i += 32) {
    float v = __bfloat162float(src[i]);
    ss += v * v;
  }
  ss = warp_sum(ss);
  const float rstd = w ? rsqrtf(ss / (float)K + eps) : 1.f;
  const int half = rot >> 1;
  const float* cr = cosT + m * half;
  const float* sr = sinT + m * half;
  for (int i = lane; i < half; i += 32) {
    float w1 = 1.f, w2 = 1.f;
    if (w) {
      w1 = __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f);
      w2 = __bfloat162float(w[i + half]) + (kOnePlus ? 1.f : 0.f);
    }
    // normalised values are rounded to bf16 before the rotation, as the module-level
    // composition (norm then rope, both in model dtype) does
    float x1 = __bfloat162float(__float2bfloat16(__bfloat162float(src[i]) * rstd * w1));
    float x2 = __bfloat162float(__float2bfloat16(__bfloat162float(src[i + half]) * rstd * w2));
    float c = cr[i], s = sr[i];
    dst[i] = __float2bfloat16(x1 * c - x2 * s);
    dst[i + half] = __float2bfloat16(x2 * c + x1 * s);
  }
  for (int i = rot + lane; i < K; i += 32) {
    float wv = w ? __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f) : 1.f;
    dst[i] = __float2bfloat16(__bfloat162float(src[i]) * rstd * wv);
  }
}

// Backward: dq_rot/dk_rot -> un-rotate -> per-head RMSNorm backward -> the q and k slices of dqkv
// [M, (H+2G)*K]; dqw / dkw accumulate with fp32 atomics.  v and gate slices: dv, dgate (null: zeros).
template <bool kOnePlus>
__global__ void qknorm_rope_bwd_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ qw,
                                       const bf16* __restrict__ kw, const float* __restrict__ cosT,
                                       const float* __restrict__ sinT,
                                       const bf16* __restrict__ dq_rot,
                                       const bf16* __restrict__ dk_rot, const bf16* __restrict__ dv,
                                       const bf16* __restrict__ dgate, bf16* __restrict__ dqkv,
                                       float* __restrict__ dqw, float* __restrict__ dkw,
                                       long long M, int H, int G, int K, int rot, float eps,
                                       int q_in_stride_heads, int rows_per_block) {
  extern __shared__ float dw_sm[];  // [2][K] per-CTA partial of dqw, dkw
  for (int i = threadIdx.x; i < 2 * K; i += blockDim.x) dw_sm[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int QH = H * q_in_stride_heads, HT = QH + 2 * G;
  const int half = rot >> 1;
  const long long m0 = (long long)blockIdx.x * rows_per_block;
  const long long m1 = min(M, m0 + rows_per_block);
  for (long long item = m0 * HT + warp; item < m1 * HT; item += nwarps) {
    const long long m = item / HT;
    const int part = (int)(item - m * HT);
    const bool is_q = part < QH;
    const int h = is_q ? part / q_in_stride_heads : part - QH + H;
    const bf16* src = qkv + item * K;
    bf16* ddst = dqkv + item * K;
    if (is_q ? part % q_in_stride_heads != 0 : part >= QH + G) {
      const bf16* from = is_q ? dgate : dv;
      if (from) from += (is_q ? m * H + h : m * G + (part - QH - G)) * K;
      for (int i = lane; i < K; i += 32) ddst[i] = from ? from[i] : __float2bfloat16(0.f);
      continue;
    }
    const bf16* w = is_q ? qw : kw;
    const bf16* dsrc = is_q ? dq_rot + (m * H + h) * K : dk_rot + (m * G + (h - H)) * K;
    float* dws = dw_sm + (is_q ? 0 : K);
    const float* cr = cosT + m * half;
    const float* sr = sinT + m * half;
    float ss = 0.f;
    for (int i = lane; i < K; i += 32) {
      float v = __bfloat162float(src[i]);
      ss += v * v;
    }
    ss = warp_sum(ss);
    const float rstd = w ? rsqrtf(ss / (float)K + eps) : 1.f;
    // pass 1: gradient w.r.t. the normalised value (dn) and dot = sum dn * w * x
    float dot = 0.f;
    for (int i = lane; i < half; i += 32) {
      float c = cr[i], s = sr[i];
      float d1 = __bfloat162float(dsrc[i]), d2 = __bfloat162float(dsrc[i + half]);
      float dn1 = d1 * c + d2 * s, dn2 = d2 * c - d1 * s;
      float x1 = __bfloat162float(src[i]), x2 = __bfloat162float(src[i + half]);
      float w1 = 1.f, w2 = 1.f;
      if (w) {
        w1 = __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f);
        w2 = __bfloat162float(w[i + half]) + (kOnePlus ? 1.f : 0.f);
        atomicAdd(dws + i, dn1 * x1 * rstd);
        atomicAdd(dws + i + half, dn2 * x2 * rstd);
      }
      dot += dn1 * w1 * x1 + dn2 * w2 * x2;
    }
    for (int i = rot + lane; i < K; i += 32) {
      float dn = __bfloat162float(dsrc[i]);
      float xv = __bfloat162float(src[i]);
      float wv = 1.f;
      if (w) {
        wv = __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f);
        atomicAdd(dws + i, dn * xv * rstd);
      }
      dot += dn * wv * xv;
    }
    dot = warp_sum(dot);
    const float cc = w ? dot * rstd * rstd * rstd / (float)K : 0.f;
    for (int i = lane; i < half; i += 32) {
      float c = cr[i], s = sr[i];
      float d1 = __bfloat162float(dsrc[i]), d2 = __bfloat162float(dsrc[i + half]);
      float dn1 = d1 * c + d2 * s, dn2 = d2 * c - d1 * s;
      float x1 = __bfloat162float(src[i]), x2 = __bfloat162float(src[i + half]);
      float w1 = 1.f, w2 = 1.f;
      if (w) {
        w1 = __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f);
        w2 = __bfloat162float(w[i + half]) + (kOnePlus ? 1.f : 0.f);
      }
      ddst[i] = __float2bfloat16(dn1 * w1 * rstd - x1 * cc);
      ddst[i + half] = __float2bfloat16(dn2 * w2 * rstd - x2 * cc);
    }
    for (int i = rot + lane; i < K; i += 32) {
      float dn = __bfloat162float(dsrc[i]);
      float xv = __bfloat162float(src[i]);
      float wv = w ? __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f) : 1.f;
      ddst[i] = __float2bfloat16(dn * wv * rstd - xv * cc);
    }
  }
  __syncthreads();
  if (qw && dqw)
    for (int i = threadIdx.x; i < K; i += blockDim.x) atomicAdd(dqw + i, dw_sm[i]);
  if (kw && dkw)
    for (int i = threadIdx.x; i < K; i += blockDim.x) atomicAdd(dkw + i, dw_sm[K + i]);
}

// The same for heads of 16 L channels, L = 4, 8, 16, rot % 16 == 0, everything on 16-byte boundaries: L lanes have a head, each
// two vectors of eight channels.  The first rot / 16 of them hold both partners of their rotations (channels 8 j ... and rot / 2 + 8 j
// ...), the others 16 that are not rotated, so every head is read once in 16-byte accesses.  Bound by HBM.  With 4-byte accesses, a
// warp per head, and v and gate left to zero filling, copies and an addition (100 us more), in us from launch to end, L2 flushed, before
// and now, forward and backward: 8192 rows, 32 heads on 8 of 128 76 and 104, 56 and 91; 3001 of 32 on 2 of 256, rot 64, with gates 64 and
// 356, 42 and 104; 999 of 16 on 8 of 128 26 and 30, 19 and 22.  (The order of head_sum costs 3 us forward at 8192 rows, nothing backward.)
struct HeadLane {
  int a, b;         // first channels of the lane's vectors
  bool turns;
  __device__ __forceinline__ HeadLane(int j, int rot) : turns(16 * j < rot) {
    a = turns ? 8 * j : 16 * j;
    b = turns ? (rot >> 1) + 8 * j : a + 8;
  }
};
__device__ __forceinline__ void unpack8(uint4 q, float* v) {
  const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = unpack_bf16(u[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* v) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
// Sums over a head of products of a lane's channel pairs u (2 u, 2 u + 1 of both vectors), in the order of a warp whose 32 lanes have a pair
// each (heads of 128): halves of the pairs' lanes first, then the pairs of a lane.  Rounding of the normed values to bf16 hangs on the
// last bit of this sum, and a model's gradients on that; this order is the one that its tolerances were measured with.  The four pairs
// change hands on the way, so it takes 3 + log2 L shuffles.
template <int L>
__device__ __forceinline__ float head_sum(const float (&p)[4]) {
  const bool high = threadIdx.x & (L / 2), odd = threadIdx.x & (L / 4);
  const float x0 = (high ? p[2] : p[0]) + __shfl_xor_sync(0xffffffffu, high ? p[0] : p[2], L / 2);
  const float x1 = (high ? p[3] : p[1]) + __shfl_xor_sync(0xffffffffu, high ? p[1] : p[3], L / 2);
  float s = (odd ? x1 : x0) + __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, L / 4);
#pragma unroll
  for (int o = L / 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  s += __shfl_xor_sync(0xffffffffu, s, L / 2);
  return s + __shfl_xor_sync(0xffffffffu, s, L / 4);
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16(x)); }
// weights (1 without one) and the row's cosines and sines of a lane
template <bool kOnePlus>
__device__ __forceinline__ void head_factors(const bf16* w, const float* cosT, const float* sinT, long long m, int rot, const HeadLane& h,
                                             float* wa, float* wb, float* c, float* sn) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    wa[i] = wb[i] = c[i] = 1.f;
    sn[i] = 0.f;
  }
  if (w) {
    unpack8(*reinterpret_cast<const uint4*>(w + h.a), wa);
    unpack8(*reinterpret_cast<const uint4*>(w + h.b), wb);
    if (kOnePlus) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        wa[i] += 1.f;
        wb[i] += 1.f;
      }
    }
  }
  if (h.turns) {
    const float4 *cp = reinterpret_cast<const float4*>(cosT + m * (rot >> 1) + h.a), *sp = reinterpret_cast<const float4*>(sinT + m * (rot >> 1) + h.a);
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    sn[0] = s0.x; sn[1] = s0.y; sn[2] = s0.z; sn[3] = s0.w; sn[4] = s1.x; sn[5] = s1.y; sn[6] = s1.z; sn[7] = s1.w;
  }
}

// (a, b) turned by the angle (sign 1) or back (-1) in separate products and sums, as the plain operations on heads without a norm round
// (vision towers: a single flipped bit of a bf16 head shows in the gradients of the whole model).
__device__ __forceinline__ void turn_apart(float* a, float* b, const float* c, const float* sn, float sign) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x1 = a[i], x2 = b[i], s = sign * sn[i];
    a[i] = __fsub_rn(__fmul_rn(x1, c[i]), __fmul_rn(x2, s));
    b[i] = __fadd_rn(__fmul_rn(x2, c[i]), __fmul_rn(x1, s));
  }
}

template <int L, bool kOnePlus>
__global__ void __launch_bounds__(256)
qknorm_rope_fwd_vec_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ qw, const bf16* __restrict__ kw,
                           const float* __restrict__ cosT, const float* __restrict__ sinT, bf16* __restrict__ q_out,
                           bf16* __restrict__ k_out, long long M, int H, int G, int rot, float eps, int q_in_stride_heads) {
  constexpr int K = 16 * L;
  const HeadLane at(threadIdx.x % L, rot);
  const int HG = H + G;
  const long long item = (blockIdx.x * 256ll + threadIdx.x) / L;
  const bool live = item < M * HG;      // the shuffles want every lane
  const long long m = live ? item / HG : 0;
  const int h = live ? (int)(item - m * HG) : 0;
  const bool is_q = h < H;
  const bf16* src = qkv + (m * ((long long)H * q_in_stride_heads + 2 * G) +
                           (is_q ? (long long)h * q_in_stride_heads : (long long)H * q_in_stride_heads + h - H)) * K;
  const bf16* w = is_q ? qw : kw;
  float a[8], b[8], wa[8], wb[8], c[8], sn[8], squares[4];
  unpack8(*reinterpret_cast<const uint4*>(src + at.a), a);
  unpack8(*reinterpret_cast<const uint4*>(src + at.b), b);
  head_factors<kOnePlus>(w, cosT, sinT, m, rot, at, wa, wb, c, sn);
#pragma unroll
  for (int i = 0; i < 8; i += 2) squares[i / 2] = a[i] * a[i] + a[i + 1] * a[i + 1] + b[i] * b[i] + b[i + 1] * b[i + 1];
  const float ss = head_sum<L>(squares);
  if (!live) return;
  if (w) {
    const float rstd = rsqrtf(ss / (float)K + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float x1 = bf16r(a[i] * rstd * wa[i]), x2 = bf16r(b[i] * rstd * wb[i]);
      a[i] = x1 * c[i] - x2 * sn[i];
      b[i] = x2 * c[i] + x1 * sn[i];
    }
  } else {
    turn_apart(a, b, c, sn, 1.f);
  }
  bf16* dst = is_q ? q_out + (m * H + h) * K : k_out + (m * G + (h - H)) * K;
  *reinterpret_cast<uint4*>(dst + at.a) = pack8(a);
  *reinterpret_cast<uint4*>(dst + at.b) = pack8(b);
}

// All heads of a row of dqkv: gate and v heads are copies of dgate [M,H,K] and dv [M,G,K] (null: zeros).
template <int L, bool kOnePlus>
__global__ void __launch_bounds__(256)
qknorm_rope_bwd_vec_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ qw, const bf16* __restrict__ kw,
                           const float* __restrict__ cosT, const float* __restrict__ sinT, const bf16* __restrict__ dq_rot,
                           const bf16* __restrict__ dk_rot, const bf16* __restrict__ dv, const bf16* __restrict__ dgate,
                           bf16* __restrict__ dqkv, float* __restrict__ dqw, float* __restrict__ dkw, long long M, int H, int G, int rot,
                           float eps, int q_in_stride_heads) {
  constexpr int K = 16 * L;
  __shared__ float red[8][2 * K];
  const HeadLane at(threadIdx.x % L, rot);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int QH = H * q_in_stride_heads, HT = QH + 2 * G;
  float gq[16] = {}, gk[16] = {};
  const long long items = M * HT, step = gridDim.x * (256ll / L);
  for (long long first = blockIdx.x * (256ll / L) + warp * (32 / L); first < items; first += step) {
    const long long item = first + lane / L;
    const bool live = item < items;
    const long long m = live ? item / HT : 0;
    const int h = live ? (int)(item - m * HT) : 0;
    bf16* ddst = dqkv + (m * HT + h) * K;
    const bool is_q = h < QH, norm = live && (is_q ? h % q_in_stride_heads == 0 : h < QH + G);
    float squares[4] = {}, dots[4] = {}, a[8], b[8], n1[8], n2[8], wa[8], wb[8];
    const bf16* w = is_q ? qw : kw;
    if (norm) {
      const bf16* src = qkv + (m * HT + h) * K;
      const bf16* dsrc = is_q ? dq_rot + (m * H + h / q_in_stride_heads) * K : dk_rot + (m * G + (h - QH)) * K;
      float c[8], sn[8], da[8], db[8];
      unpack8(*reinterpret_cast<const uint4*>(src + at.a), a);
      unpack8(*reinterpret_cast<const uint4*>(src + at.b), b);
      unpack8(*reinterpret_cast<const uint4*>(dsrc + at.a), da);
      unpack8(*reinterpret_cast<const uint4*>(dsrc + at.b), db);
      head_factors<kOnePlus>(w, cosT, sinT, m, rot, at, wa, wb, c, sn);
      if (w) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {      // un-rotate: gradient of the normalised, weighted values
          n1[i] = da[i] * c[i] + db[i] * sn[i];
          n2[i] = db[i] * c[i] - da[i] * sn[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          n1[i] = da[i];
          n2[i] = db[i];
        }
        turn_apart(n1, n2, c, sn, -1.f);
      }
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        squares[i / 2] = a[i] * a[i] + a[i + 1] * a[i + 1] + b[i] * b[i] + b[i + 1] * b[i + 1];
        dots[i / 2] = n1[i] * wa[i] * a[i] + n1[i + 1] * wa[i + 1] * a[i + 1] + n2[i] * wb[i] * b[i] + n2[i + 1] * wb[i + 1] * b[i + 1];
      }
    } else if (live) {
      const bf16* from = is_q ? dgate : dv;
      if (from) from += is_q ? (m * H + h / q_in_stride_heads) * K : (m * G + (h - QH - G)) * K;
      const uint4 zero = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(ddst + at.a) = from ? *reinterpret_cast<const uint4*>(from + at.a) : zero;
      *reinterpret_cast<uint4*>(ddst + at.b) = from ? *reinterpret_cast<const uint4*>(from + at.b) : zero;
    }
    const float ss = head_sum<L>(squares), dot = head_sum<L>(dots);
    if (!norm) continue;
    if (w) {
      const float rstd = rsqrtf(ss / (float)K + eps);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (is_q) {
          gq[i] = fmaf(n1[i] * a[i], rstd, gq[i]);
          gq[8 + i] = fmaf(n2[i] * b[i], rstd, gq[8 + i]);
        } else {
          gk[i] = fmaf(n1[i] * a[i], rstd, gk[i]);
          gk[8 + i] = fmaf(n2[i] * b[i], rstd, gk[8 + i]);
        }
      }
      const float cc = dot * rstd * rstd * rstd / (float)K;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        n1[i] = n1[i] * wa[i] * rstd - a[i] * cc;
        n2[i] = n2[i] * wb[i] * rstd - b[i] * cc;
      }
    }
    *reinterpret_cast<uint4*>(ddst + at.a) = pack8(n1);
    *reinterpret_cast<uint4*>(ddst + at.b) = pack8(n2);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 16; ++i) {      // the heads of a warp
#pragma unroll
    for (int o = L; o < 32; o <<= 1) {
      gq[i] += __shfl_xor_sync(0xffffffffu, gq[i], o);
      gk[i] += __shfl_xor_sync(0xffffffffu, gk[i], o);
    }
    if (lane < L) {
      const int ch = i < 8 ? at.a + i : at.b + i - 8;
      red[warp][ch] = gq[i];
      red[warp][K + ch] = gk[i];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * K; i += 256) {
    float sacc = 0.f;
#pragma unroll
    for (int wi = 0; wi < 8; ++wi) sacc += red[wi][i];
    if (i < K) { if (qw && dqw) atomicAdd(dqw + i, sacc); }
    else if (kw && dkw) atomicAdd(dkw + i - K, sacc);
  }
}

// ------------------------------------------------------------------ sums over rows
// out[c] = scale * sum_m x[m, c], fp32 sums, in a fixed order.  A cluster of CTAs has 64 columns, each CTA a share of the rows; a
// thread adds eight columns of every 32nd row, four loads in flight, and the CTAs' sums meet in shared memory.  Bias gradients
// and mean router probabilities have few columns, to which a reduction per column gives few CTAs: bf16 3136 x 1024, 3136 x 4096, 784 x 4096,
// fp32 3001 x 32, 4096 x 128 in us from launch to end, L2 flushed: the library's reduction 26, 33, 44, 39, 22, this 21, 23, 17, 18, 19 (a
// launch that does nothing: 14 to 20).
__device__ __forceinline__ void row8(const bf16* p, float* v) { unpack8(*reinterpret_cast<const uint4*>(p), v); }
__device__ __forceinline__ void row8(const float* p, float* v) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void put(bf16* p, float v) { *p = __float2bfloat16(v); }
__device__ __forceinline__ void put(float* p, float v) { *p = v; }
template <typename T>
__global__ void __launch_bounds__(256) column_sum_kernel(const T* __restrict__ x, T* __restrict__ out, long long M, int N, float scale) {
  __shared__ float red[32][66];
  __shared__ float part[64];
  grid_begin();
  const int ctas = gridDim.x, rank = blockIdx.x, tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  const int c = blockIdx.y * 64 + tx * 8;
  float acc[8] = {};
  if (c < N) {
    const long long step = 32ll * ctas;
    long long m = rank * 32 + ty;
    for (; m + 3 * step < M; m += 4 * step) {
      float v[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) row8(x + (m + u * step) * N + c, v[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += v[u][i];
    }
    for (; m < M; m += step) {
      float v[8];
      row8(x + m * N + c, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[ty][tx * 8 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < 64) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 32; ++r) s += red[r][threadIdx.x];
    part[threadIdx.x] = s;
  }
  __syncthreads();
  cluster_sync_all();
  if (rank == 0 && threadIdx.x < 64) {
    float s = 0.f;
    for (int r = 0; r < ctas; ++r) {
      float t;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t) : "r"(mapa_shared(smem_u32(&part[threadIdx.x]), r)) : "memory");
      s += t;
    }
    const int col = blockIdx.y * 64 + threadIdx.x;
    if (col < N) put(out + col, s * scale);
  }
  __syncthreads();
  cluster_sync_all();      // nobody leaves while its sums may still be read
}

// ------------------------------------------------------------------ sigmoid output gate
// out[m,h,:] = o[m,h,:] * sigmoid(gate[m,h,:]) (gated attention of Qwen3.5: every query head of the
// fused projection is followed by a gate head, so the gate is a strided view of that buffer).
// o / out / dout / d_o / d_gate are dense [M, H, Kd]; the gate has its own row and head strides.
__global__ void sigmoid_gate_fwd_kernel(const bf16* __restrict__ o, const bf16* __restrict__ gate, bf16* __restrict__ out,
                                        long long M, int H, int Kd, long long g_row, long long g_head) {
  const int kv = Kd >> 3;
  const long long total = M * H * kv;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(t % kv);
    const long long mh = t / kv;
    const int h = (int)(mh % H);
    const long long m = mh / H;
    const uint4 a = reinterpret_cast<const uint4*>(o)[t];
    const uint4 gq = *reinterpret_cast<const uint4*>(gate + m * g_row + h * g_head + c * 8);
    const uint32_t au[4] = {a.x, a.y, a.z, a.w}, gu[4] = {gq.x, gq.y, gq.z, gq.w};
    uint32_t r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16(au[j]), g = unpack_bf16(gu[j]);
      r[j] = pack_bf16(x.x / (1.f + __expf(-g.x)), x.y / (1.f + __expf(-g.y)));
    }
    reinterpret_cast<uint4*>(out)[t] = make_uint4(r[0], r[1], r[2], r[3]);
  }
}

__global__ void sigmoid_gate_bwd_kernel(const bf16* __restrict__ o, const bf16* __restrict__ gate,
                                        const bf16* __restrict__ dout, bf16* __restrict__ d_o, bf16* __restrict__ d_gate,
                                        long long M, int H, int Kd, long long g_row, long long g_head) {
  const int kv = Kd >> 3;
  const long long total = M * H * kv;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(t % kv);
    const long long mh = t / kv;
    const int h = (int)(mh % H);
    const long long m = mh / H;
    const uint4 a = reinterpret_cast<const uint4*>(o)[t];
    const uint4 d = reinterpret_cast<const uint4*>(dout)[t];
    const uint4 gq = *reinterpret_cast<const uint4*>(gate + m * g_row + h * g_head + c * 8);
    const uint32_t au[4] = {a.x, a.y, a.z, a.w}, du[4] = {d.x, d.y, d.z, d.w}, gu[4] = {gq.x, gq.y, gq.z, gq.w};
    uint32_t ro[4], rg[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16(au[j]), dy = unpack_bf16(du[j]), g = unpack_bf16(gu[j]);
      const float s0 = 1.f / (1.f + __expf(-g.x)), s1 = 1.f / (1.f + __expf(-g.y));
      ro[j] = pack_bf16(dy.x * s0, dy.y * s1);
      rg[j] = pack_bf16(dy.x * x.x * s0 * (1.f - s0), dy.y * x.y * s1 * (1.f - s1));
    }
    reinterpret_cast<uint4*>(d_o)[t] = make_uint4(ro[0], ro[1], ro[2], ro[3]);
    reinterpret_cast<uint4*>(d_gate)[t] = make_uint4(rg[0], rg[1], rg[2], rg[3]);
  }
}

// ------------------------------------------------------------------ softmax cross-entropy
// One CTA per row of a bf16 logits chunk [R, V] (pitch ld).  Adds mask*nll to loss_sum and
// overwrites the row with dlogits = (softmax - onehot) * mask * (*grad_scale).
__global__ void ce_fwd_bwd_kernel(bf16* __restrict__ logits, long long ld, int V,
                                  const int* __restrict__ targets, const float* __restrict__ mask,
                                  const float* __restrict__ grad_scale,
                                  float* __restrict__ loss_sum, float* __restrict__ lse_out,
                                  int write_grad) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  bf16* lr = logits + row * ld;
  const float mk = mask ? mask[row] : 1.f;
  const int tgt = targets[row];
  const int nv = V >> 3;  // V % 8 == 0
  const uint4* lv = reinterpret_cast<const uint4*>(lr);
  float mx = -INFINITY, sm = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 q = lv[i];
    uint32_t u[4] = {q.x, q.y, q.z, q.w};
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = unpack_bf16(u[j]);
      f[2 * j] = t.x; f[2 * j + 1] = t.y;
    }
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    if (lm > mx) {
      sm *= __expf(mx - lm);
      mx = lm;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sm += __expf(f[j] - mx);
  }
  const float gmx = block_max(mx, red);
  sm *= (mx == -INFINITY) ? 0.f : __expf(mx - gmx);
  const float gsum = block_sum(sm, red);
  const float lse = gmx + logf(gsum);
  if (threadIdx.x == 0) {
    float tl = (tgt >= 0 && tgt < V) ? __bfloat162float(lr[tgt]) : 0.f;
    if (mk != 0.f) atomicAdd(loss_sum, (lse - tl) * mk);
    if (lse_out) lse_out[row] = lse;
  }
  if (!write_grad) return;
  __syncthreads();
  const float gs = mk * (grad_scale ? *grad_scale : 1.f);
  uint4* ov = reinterpret_cast<uint4*>(lr);
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 q = lv[i], o;
    uint32_t u[4] = {q.x, q.y, q.z, q.w}, ou[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = unpack_bf16(u[j]);
      int c0 = i * 8 + 2 * j;
      float p0 = __expf(t.x - lse) - (c0 == tgt ? 1.f : 0.f);
      float p1 = __expf(t.y - lse) - (c0 + 1 == tgt ? 1.f : 0.f);
      ou[j] = pack_bf16(p0 * gs, p1 * gs);
    }
    o.x = ou[0]; o.y = ou[1]; o.z = ou[2]; o.w = ou[3];
    ov[i] = o;
  }
}

// Log-sum-exp and loss of a logits chunk from the per-tile statistics that the logits GEMM wrote
// in its epilogue (fp32 maximum and sum of exponentials per row and 256-column tile, fp32 target
// logit per row): one warp per row.  lse_out feeds the gradient pass over the bf16 logits.
__global__ void ce_finish_kernel(const float2* __restrict__ stats, int n_tiles, const float* __restrict__ tgt_logit,
                                 const float* __restrict__ mask, float* __restrict__ loss_sum,
                                 float* __restrict__ lse_out, long long R, const int* __restrict__ rows_dev,
                                 int rows_off) {
  const long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= R || (rows_dev && row >= __ldg(rows_dev) - rows_off)) return;
  const float2* sp = stats + row * n_tiles;
  float mx = -INFINITY, sm = 0.f;
  for (int i = lane; i < n_tiles; i += 32) {
    const float2 t = sp[i];
    if (t.x > mx) {
      sm *= __expf(mx - t.x);
      mx = t.x;
    }
    if (t.x != -INFINITY) sm += t.y * __expf(t.x - mx);
  }
  const float gmx = warp_max(mx);
  sm *= (mx == -INFINITY) ? 0.f : __expf(mx - gmx);
  const float gsum = warp_sum(sm);
  if (lane == 0) {
    const float lse = gmx + logf(gsum);
    lse_out[row] = lse;
    const float mk = mask ? mask[row] : 1.f;
    if (mk != 0.f) atomicAdd(loss_sum, (lse - tgt_logit[row]) * mk);
  }
}

// Vocabulary-parallel variant, two passes around an all-reduce of the row statistics.  This GPU
// holds the logits of vocabulary ids [v0, v0 + V).  Pass 1: row maximum, sum of exp(x - max) and
// the target's logit (zero when another GPU owns the target).  Pass 2 (after the caller has
// combined the statistics into the global log-sum-exp): overwrite with dlogits.
__global__ void ce_vp_stats_kernel(const bf16* __restrict__ logits, long long ld, int V, int v0,
                                   const int* __restrict__ targets, float* __restrict__ max_out,
                                   float* __restrict__ sum_out, float* __restrict__ tgt_out) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const bf16* lr = logits + row * ld;
  const int nv = V >> 3;
  const uint4* lv = reinterpret_cast<const uint4*>(lr);
  float mx = -INFINITY, sm = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 q = lv[i];
    uint32_t u[4] = {q.x, q.y, q.z, q.w};
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = unpack_bf16(u[j]);
      f[2 * j] = t.x; f[2 * j + 1] = t.y;
    }
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    if (lm > mx) {
      sm *= __expf(mx - lm);
      mx = lm;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sm += __expf(f[j] - mx);
  }
  const float gmx = block_max(mx, red);
  sm *= (mx == -INFINITY) ? 0.f : __expf(mx - gmx);
  const float gsum = block_sum(sm, red);
  if (threadIdx.x == 0) {
    const int t = targets[row] - v0;
    max_out[row] = gmx;
    sum_out[row] = gsum;
    tgt_out[row] = (t >= 0 && t < V) ? __bfloat162float(lr[t]) : 0.f;
  }
}

__global__ void ce_vp_grad_kernel(bf16* __restrict__ logits, long long ld, int V, int v0,
                                  const int* __restrict__ targets, const float* __restrict__ lse_in,
                                  const float* __restrict__ mask, const float* __restrict__ grad_scale) {
  const long long row = blockIdx.x;
  bf16* lr = logits + row * ld;
  const int tgt = targets[row] - v0;
  const float lse = lse_in[row];
  const float gs = (mask ? mask[row] : 1.f) * (grad_scale ? *grad_scale : 1.f);
  const int nv = V >> 3;
  uint4* ov = reinterpret_cast<uint4*>(lr);
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 q = ov[i], o;
    uint32_t u[4] = {q.x, q.y, q.z, q.w}, ou[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = unpack_bf16(u[j]);
      int c0 = i * 8 + 2 * j;
      float p0 = __expf(t.x - lse) - (c0 == tgt ? 1.f : 0.f);
      float p1 = __expf(t.y - lse) - (c0 + 1 == tgt ? 1.f : 0.f);
      ou[j] = pack_bf16(p0 * gs, p1 * gs);
    }
    o.x = ou[0]; o.y = ou[1]; o.z = ou[2]; o.w = ou[3];
    ov[i] = o;
  }
}

// Supervised rows only.  A conversation's prompt and padding carry no loss, and a row without loss needs
// none of the head's three products, so the rows with a mask other than zero are numbered here, in order,
// and gathered.  One CTA: the scan is serial over tiles of 1024 rows (1.5 us each), next to products of
// milliseconds.  rows[c] is the row of number c (-1 past the count), place[row] its number or -1.
__global__ void __launch_bounds__(1024) ce_count_kernel(const float* __restrict__ mask, const int* __restrict__ targets,
                                                        long long M, int* __restrict__ rows, int* __restrict__ place,
                                                        int* __restrict__ tgt_out, float* __restrict__ mask_out,
                                                        int* __restrict__ count) {
  __shared__ int part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (long long r0 = 0; r0 < M; r0 += 1024) {
    const long long r = r0 + threadIdx.x;
    const float mk = r < M ? mask[r] : 0.f;
    const bool on = mk != 0.f;
    const unsigned votes = __ballot_sync(0xffffffffu, on);
    if (lane == 0) part[warp] = __popc(votes);
    __syncthreads();
    int before = base, total = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += part[w];
      total += part[w];
    }
    const int c = before + __popc(votes & ((1u << lane) - 1));
    if (r < M) place[r] = on ? c : -1;
    if (on) {
      rows[c] = (int)r;
      tgt_out[c] = targets[r];
      mask_out[c] = mk;
    }
    base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = base;
  for (long long c = base + threadIdx.x; c < M; c += 1024) {
    rows[c] = -1;
    tgt_out[c] = -1;
    mask_out[c] = 0.f;
  }
}

// dlogits are rounded to bf16, and the largest of a row, (p - 1) times the loss's scale, has nearly the same value
// in every row: the rounding of the scale would be an error of one sign in all gradients (5e-4 at 2440 rows).
// So dlogits carry the scale's power of two only; the rest, in [1, 2), meets both gradients in fp32: the weight's as it
// leaves the accumulator, the hidden rows' when they go back to their places.

// Hidden rows in that order; the reduction of the weight gradient runs in blocks of 64 rows, so the rows
// after the last one are zeroed that far.
__global__ void ce_gather_kernel(const bf16* __restrict__ h, const int* __restrict__ rows, const int* __restrict__ count,
                                 bf16* __restrict__ out, long long M, int D) {
  const int dv = D >> 3;
  const long long n = *count, end = min((n + 63) / 64 * 64, M);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < end * dv; t += (long long)gridDim.x * blockDim.x) {
    const long long c = t / dv;
    const int i = (int)(t - c * dv);
    reinterpret_cast<uint4*>(out + c * D)[i] =
        c < n ? reinterpret_cast<const uint4*>(h + (long long)rows[c] * D)[i] : make_uint4(0, 0, 0, 0);
  }
}

// Gradient rows back in their places, times the upstream gradient; zero where there was no loss.
__global__ void ce_scatter_kernel(const float* __restrict__ dh, const int* __restrict__ place, const float* __restrict__ g,
                                  const float* __restrict__ scale, bf16* __restrict__ out, long long M, int D) {
  const int dv = D >> 3;
  const float gs = *g * scale_rest(*scale);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < M * dv; t += (long long)gridDim.x * blockDim.x) {
    const long long r = t / dv;
    const int i = (int)(t - r * dv);
    const int c = place[r];
    uint4 o = make_uint4(0, 0, 0, 0);
    if (c >= 0) {
      const float4* s = reinterpret_cast<const float4*>(dh + (long long)c * D) + 2 * i;
      const float4 a = s[0], b = s[1];
      o.x = pack_bf16(a.x * gs, a.y * gs); o.y = pack_bf16(a.z * gs, a.w * gs);
      o.z = pack_bf16(b.x * gs, b.y * gs); o.w = pack_bf16(b.z * gs, b.w * gs);
    }
    reinterpret_cast<uint4*>(out + r * D)[i] = o;
  }
}

// ce_vp_grad_kernel over counted rows: logits -> dlogits in place, zeros up to the next multiple of 64 rows.
__global__ void ce_counted_grad_kernel(bf16* __restrict__ logits, long long ld, int V, const int* __restrict__ targets,
                                       const float* __restrict__ lse_in, const float* __restrict__ mask,
                                       const float* __restrict__ grad_scale, const int* __restrict__ rows_dev, int rows_off) {
  const int row = blockIdx.x, n = __ldg(rows_dev) - rows_off;
  if (row >= (n + 63) / 64 * 64 || n <= 0) return;
  uint4* ov = reinterpret_cast<uint4*>(logits + (long long)row * ld);
  const int nv = V >> 3;
  if (row >= n) {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) ov[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  const int tgt = targets[row];
  const float lse = lse_in[row];
  const float gs = mask[row] * scale_pow2(*grad_scale);
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const uint4 q = ov[i];
    const uint32_t u[4] = {q.x, q.y, q.z, q.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = unpack_bf16(u[j]);
      const int c0 = i * 8 + 2 * j;
      const float p0 = __expf(t.x - lse) - (c0 == tgt ? 1.f : 0.f);
      const float p1 = __expf(t.y - lse) - (c0 + 1 == tgt ? 1.f : 0.f);
      o[j] = pack_bf16(p0 * gs, p1 * gs);
    }
    ov[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ------------------------------------------------------------------ embedding (K13)
__global__ void embedding_fwd_kernel(const int* __restrict__ ids, const bf16* __restrict__ table,
                                     bf16* __restrict__ out, long long M, int D) {
  grid_begin();
  const int dv = D >> 3;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < M * dv;
       idx += (long long)gridDim.x * blockDim.x) {
    long long m = idx / dv;
    int c = (int)(idx - m * dv);
    reinterpret_cast<uint4*>(out + m * D)[c] =
        reinterpret_cast<const uint4*>(table + (long long)ids[m] * D)[c];
  }
}
__global__ void embedding_bwd_kernel(const int* __restrict__ ids, const bf16* __restrict__ dy,
                                     float* __restrict__ dtable, long long M, int D, int row_lo,
                                     int row_hi) {
  const int dv = D >> 1;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < M * dv;
       idx += (long long)gridDim.x * blockDim.x) {
    long long m = idx / dv;
    int c = (int)(idx - m * dv);
    int id = ids[m];
    if (id < row_lo || id >= row_hi) continue;
    float2 f = unpack_bf16(reinterpret_cast<const uint32_t*>(dy + m * D)[c]);
    float* d = dtable + (long long)(id - row_lo) * D + 2 * c;
    atomicAdd(d, f.x);
    atomicAdd(d + 1, f.y);
  }
}

// ------------------------------------------------------------------ optimizer (K14)
// Sum of squares, and (used, may be null) a byte for every 128 elements: whether any of them is not zero.  A warp's eight loads of
// 512 bytes are eight of these blocks (with four the pass takes 3 % longer, with one 29 %; 7.1 TB/s).
__global__ void __launch_bounds__(256) sumsq_kernel(const float* __restrict__ g, long long n, float* __restrict__ out,
                                                    uint8_t* __restrict__ used) {
  __shared__ float red[32];
  float s = 0.f;
  constexpr int U = 8;
  const int lane = threadIdx.x & 31;
  const long long n4 = n >> 2, warps = (long long)gridDim.x * (blockDim.x >> 5);
  const float4* g4 = reinterpret_cast<const float4*>(g);
  for (long long b = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * U; b * 32 < n4; b += warps * U) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = (b + u) * 32 + lane;
      v[u] = i < n4 ? __ldcs(g4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    int any = 0;      // lane u: of block u
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s += v[u].x * v[u].x + v[u].y * v[u].y + v[u].z * v[u].z + v[u].w * v[u].w;
      const uint32_t bits = __float_as_uint(v[u].x) | __float_as_uint(v[u].y) | __float_as_uint(v[u].z) | __float_as_uint(v[u].w);
      const int is = __any_sync(0xffffffffu, bits != 0);
      if (lane == u) any = is;
    }
    if (used && lane < U) used[b + lane] = any ? 1 : 0;      // the buffer is a multiple of eight bytes
  }
  if (blockIdx.x == 0)
    for (long long i = (n4 << 2) + threadIdx.x; i < n; i += blockDim.x) s += g[i] * g[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// AdamW on a flat fp32 shard.  The clip coefficient is derived on the device from the
// already-reduced squared gradient norm so the host never synchronises:
//   g' = g * grad_mul * min(1, max_norm / (sqrt(norm_sq) * grad_mul + 1e-6))
// Writes the fp32 master, both moments, the bf16 compute copy, and zeroes the gradient.
// Bound by HBM (34 bytes a parameter: 1.63 G parameters 9.34 ms, 5.9 TB/s).  Where sumsq_kernel found 128 gradients zero (``used``, may be
// null) they are neither read nor cleared: rows of an embedding table whose token was not in the batch, experts without tokens.  ibc1 / ibc2 are the
// reciprocals of the bias corrections, rounded once from double precision on the host: one division per
// parameter is left instead of three.
struct AdamArgs {
  float lr, b1, b2, eps, wd, ibc1, ibc2;
};

__device__ __forceinline__ void adam_one(const AdamArgs& a, float mul, float& p, float& m, float& v, float g) {
  const float gr = g * mul;
  m = a.b1 * m + (1.f - a.b1) * gr;
  v = a.b2 * v + (1.f - a.b2) * gr * gr;
  p = p - a.lr * ((m * a.ibc1) / (sqrtf(v * a.ibc2) + a.eps) + a.wd * p);
}

// A thread has two groups of four parameters in flight, 128 bytes of loads before any arithmetic.
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                                                    float* __restrict__ g, bf16* __restrict__ p16, long long n, AdamArgs a,
                                                    float grad_mul, const float* __restrict__ norm_sq, float max_norm,
                                                    int zero_grad, const uint8_t* __restrict__ used) {
  float mul = grad_mul;
  if (norm_sq && max_norm > 0.f) {
    float nrm = sqrtf(*norm_sq) * grad_mul;
    mul *= fminf(1.f, max_norm / (nrm + 1e-6f));
  }
  constexpr int U = 2;
  const long long n4 = n >> 2, step = (long long)gridDim.x * (256 * U);
  float4 *p4 = reinterpret_cast<float4*>(p), *m4 = reinterpret_cast<float4*>(m), *v4 = reinterpret_cast<float4*>(v),
         *g4 = reinterpret_cast<float4*>(g);
  for (long long i0 = blockIdx.x * (long long)(256 * U) + threadIdx.x; i0 < n4; i0 += step) {
    float4 pp[U], mm[U], vv[U], gg[U];
    bool any[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + 256 * u;
      any[u] = i < n4 && (!used || __ldg(used + (i >> 5)));      // the same for a whole warp
      if (i < n4) {
        pp[u] = __ldcs(p4 + i); mm[u] = __ldcs(m4 + i); vv[u] = __ldcs(v4 + i);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) gg[u] = any[u] ? __ldcs(g4 + i0 + 256 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + 256 * u;
      if (i >= n4) break;
      adam_one(a, mul, pp[u].x, mm[u].x, vv[u].x, gg[u].x);
      adam_one(a, mul, pp[u].y, mm[u].y, vv[u].y, gg[u].y);
      adam_one(a, mul, pp[u].z, mm[u].z, vv[u].z, gg[u].z);
      adam_one(a, mul, pp[u].w, mm[u].w, vv[u].w, gg[u].w);
      __stcs(p4 + i, pp[u]);
      __stcs(m4 + i, mm[u]);
      __stcs(v4 + i, vv[u]);
      if (zero_grad && any[u]) __stcs(g4 + i, make_float4(0.f, 0.f, 0.f, 0.f));
      if (p16) __stcs(reinterpret_cast<uint2*>(p16) + i, make_uint2(pack_bf16(pp[u].x, pp[u].y), pack_bf16(pp[u].z, pp[u].w)));
    }
  }
  if (blockIdx.x == 0) {
    for (long long i = (n4 << 2) + threadIdx.x; i < n; i += blockDim.x) {
      adam_one(a, mul, p[i], m[i], v[i], g[i]);
      if (zero_grad) g[i] = 0.f;
      if (p16) p16[i] = __float2bfloat16(p[i]);
    }
  }
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ src, bf16* __restrict__ dst,
                                     long long n) {
  const long long n4 = n >> 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4;
       i += (long long)gridDim.x * blockDim.x) {
    float4 v = reinterpret_cast<const float4*>(src)[i];
    uint2 o;
    o.x = pack_bf16(v.x, v.y);
    o.y = pack_bf16(v.z, v.w);
    reinterpret_cast<uint2*>(dst)[i] = o;
  }
  if (blockIdx.x == 0)
    for (long long i = (n4 << 2) + threadIdx.x; i < n; i += blockDim.x)
      dst[i] = __float2bfloat16(src[i]);
}

// bf16 [R, C] -> [C, R] through a padded shared-memory tile.
__global__ void transpose_bf16_kernel(const bf16* __restrict__ src, bf16* __restrict__ dst, int R,
                                      int C, long long lds, long long ldd) {
  __shared__ bf16 tile[64][66];
  const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    int r = r0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      int c = c0 + j;
      tile[i][j] = (r < R && c < C) ? src[(long long)r * lds + c] : __float2bfloat16(0.f);
    }
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    int c = c0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      int r = r0 + j;
      if (r < R && c < C) dst[(long long)c * ldd + r] = tile[j][i];
    }
  }
}

// Flush helper for benchmarks: touch a buffer larger than L2.
__global__ void fill_u32_kernel(uint32_t* p, long long n, uint32_t v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    p[i] = v;
}

static inline int grid_for(long long work, int threads) {
  long long b = (work + threads - 1) / threads;
  long long cap = (long long)num_sms() * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

// Embedding gradient with the table's rows spread over the GPUs (rows_per_rank consecutive rows on
// each): every token's gradient row is added into the owner's fp32 shard over NVLink.  A warp
// covers 64 consecutive columns of one token (256 contiguous bytes) per step.
struct EmbPeerPtrs {
  float* p[8];
};
__global__ void embedding_bwd_peer_kernel(const int* __restrict__ ids, const bf16* __restrict__ dy, EmbPeerPtrs dst,
                                          long long M, int D, int rows_per_rank, int world) {
  const int dv = D >> 1;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < M * dv;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long m = idx / dv;
    const int c = (int)(idx - m * dv);
    const int id = ids[m];
    const int owner = id / rows_per_rank;
    if (id < 0 || owner >= world) continue;
    const float2 f = unpack_bf16(reinterpret_cast<const uint32_t*>(dy + m * D)[c]);
    float* d = dst.p[owner] + (long long)(id - owner * rows_per_rank) * D + 2 * c;
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(d), "f"(f.x), "f"(f.y) : "memory");
  }
}

}  // namespace ob

using namespace ob;

extern "C" {

int ob_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, long long M, int D,
                   float eps, int one_plus, cudaStream_t s) {
  if (D % 8) return 6001;
  if (M <= 0) return 0;
  int threads = D >= 2048 ? 256 : 128;
  if (one_plus)
    OB_LAUNCH(rmsnorm_fwd_kernel<true>, (unsigned)M, threads, 0, s, (const bf16*)x, (const bf16*)w,
                                                             (bf16*)y, rstd, D, eps);
  else
    OB_LAUNCH(rmsnorm_fwd_kernel<false>, (unsigned)M, threads, 0, s, (const bf16*)x, (const bf16*)w,
                                                              (bf16*)y, rstd, D, eps);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                   float* dw, long long M, int D, float eps, int one_plus, cudaStream_t s) {
  if (D % 8) return 6001;
  if (M <= 0) return 0;
  const int threads = 256;
  const int nv = D / 8;
  int need = (nv + threads - 1) / threads;
  // three CTAs per SM, in whole clusters
  const long long want = (M + kRmsCluster - 1) / kRmsCluster, most = (long long)num_sms() * 3 / kRmsCluster;
  const int grid = (int)(want < most ? want : most) * kRmsCluster;
#define OB_RB(OP, MV)                                                                           \
  OB_ENSURE_DYN_SMEM((rmsnorm_bwd_kernel<OP, MV>), MV * threads * 32);                           \
  rmsnorm_bwd_kernel<OP, MV><<<grid, threads, D * 4, s>>>((const bf16*)dy, (const bf16*)x,      \
                                                          (const bf16*)w, rstd, (bf16*)dx, dw,  \
                                                          (int)M, D, eps)
  if (need <= 1) { if (one_plus) { OB_RB(true, 1); } else { OB_RB(false, 1); } }
  else if (need <= 2) { if (one_plus) { OB_RB(true, 2); } else { OB_RB(false, 2); } }
  else if (need <= 4) { if (one_plus) { OB_RB(true, 4); } else { OB_RB(false, 4); } }
  else return 6004;
#undef OB_RB
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_swiglu_fwd(const void* gu, void* act, const int* rows, long long M, int F, cudaStream_t s) {
  if (F % 8) return 6001;
  if (M <= 0) return 0;
  OB_LAUNCH(swiglu_fwd_kernel, grid_for(M * (F / 8), 256), 256, 0, s, (const bf16*)gu, (bf16*)act, rows, M, F);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_swiglu_bwd(const void* gu, const void* dact, void* dgu, void* act_out, const int* rows, long long M, int F,
                  cudaStream_t s) {
  if (F % 8) return 6001;
  if (M <= 0) return 0;
  swiglu_bwd_kernel<<<grid_for(M * (F / 8), 256), 256, 0, s>>>(
      (const bf16*)gu, (const bf16*)dact, (bf16*)dgu, (bf16*)act_out, rows, M, F);
  OB_CHECK_LAUNCH();
  return 0;
}

// x [M,N] bf16 or fp32 -> out [N] of the same type: scale * sums over the rows.  N % 8 == 0, 16-byte aligned rows.
int ob_column_sum(const void* x, void* out, long long M, int N, int is_bf16, float scale, cudaStream_t s) {
  if (M < 0 || N <= 0 || (N & 7)) return 6001;
  if ((uintptr_t)x & 15) return 6002;
  const int tiles = (N + 63) / 64;
  if (tiles > 65535) return 6005;
  int ctas = 1;      // about two waves of four on an SM, as long as a thread has a few rows
  while (ctas < 8 && tiles * ctas < 4 * num_sms() && M > 128ll * ctas) ctas *= 2;
  const dim3 grid(ctas, tiles);
  const cudaError_t e = is_bf16 ? launch(column_sum_kernel<bf16>, grid, dim3(256), 0, s, ctas, (const bf16*)x, (bf16*)out, M, N, scale)
                                : launch(column_sum_kernel<float>, grid, dim3(256), 0, s, ctas, (const float*)x, (float*)out, M, N, scale);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return 1000 + (int)e;
  }
  return 0;
}

// Sizes and alignment of the vector kernels: their L, or 0.
static int qknorm_lanes(int K, int rot, const void* const* ptrs, int n) {
  uintptr_t any = 0;
  for (int i = 0; i < n; ++i) any |= (uintptr_t)ptrs[i];
  return (K == 64 || K == 128 || K == 256) && rot >= 0 && rot <= K && !(rot & 15) && !(any & 15) ? K / 16 : 0;
}

int ob_qknorm_rope_fwd(const void* qkv, const void* qw, const void* kw, const float* cosT,
                       const float* sinT, void* q_out, void* k_out, long long M, int H, int G,
                       int K, int rot, float eps, int one_plus, int q_stride_heads,
                       cudaStream_t s) {
  if (M <= 0) return 0;
  const void* ptrs[] = {qkv, qw, kw, cosT, sinT, q_out, k_out};
  const int lanes = qknorm_lanes(K, rot, ptrs, 7);
  const int threads = 256;
#define OB_QKNORM_FWD(kern, blocks, ...)                                                                                       \
  kern<<<(unsigned)(blocks), threads, 0, s>>>((const bf16*)qkv, (const bf16*)qw, (const bf16*)kw, cosT, sinT, (bf16*)q_out, \
                                              (bf16*)k_out, M, H, G, __VA_ARGS__)
#define OB_QKNORM_FWD_VEC(L)                                                                                                     \
  if (lanes == L) {                                                                                                              \
    const long long blocks = (M * (H + G) * L + threads - 1) / threads;                                                          \
    if (one_plus) OB_QKNORM_FWD((qknorm_rope_fwd_vec_kernel<L, true>), blocks, rot, eps, q_stride_heads);                        \
    else OB_QKNORM_FWD((qknorm_rope_fwd_vec_kernel<L, false>), blocks, rot, eps, q_stride_heads);                                \
  }
  OB_QKNORM_FWD_VEC(4) else OB_QKNORM_FWD_VEC(8) else OB_QKNORM_FWD_VEC(16) else {
    const long long blocks = (M * (H + G) * 32 + threads - 1) / threads;
    if (one_plus) OB_QKNORM_FWD(qknorm_rope_fwd_kernel<true>, blocks, K, rot, eps, q_stride_heads);
    else OB_QKNORM_FWD(qknorm_rope_fwd_kernel<false>, blocks, K, rot, eps, q_stride_heads);
  }
  OB_CHECK_LAUNCH();
  return 0;
}

// dqkv of all heads; dv [M,G,K] and dgate [M,H,K] (q_stride_heads 2) are copied to their places, null: zeros.
int ob_qknorm_rope_bwd(const void* qkv, const void* qw, const void* kw, const float* cosT,
                       const float* sinT, const void* dq_rot, const void* dk_rot, const void* dv, const void* dgate, void* dqkv,
                       float* dqw, float* dkw, long long M, int H, int G, int K, int rot,
                       float eps, int one_plus, int q_stride_heads, cudaStream_t s) {
  if (M <= 0) return 0;
  const int threads = 256;
  const void* ptrs[] = {qkv, qw, kw, cosT, sinT, dq_rot, dk_rot, dv, dgate, dqkv};
  const int lanes = qknorm_lanes(K, rot, ptrs, 10);
#define OB_QKNORM_BWD_VEC(L, P)                                                                                                    \
  qknorm_rope_bwd_vec_kernel<L, P><<<(unsigned)min(((long long)M * (H * q_stride_heads + 2 * G) * L + 255) / 256, (long long)num_sms() * 8), \
                                     threads, 0, s>>>((const bf16*)qkv, (const bf16*)qw, (const bf16*)kw, cosT, sinT,           \
                                                      (const bf16*)dq_rot, (const bf16*)dk_rot, (const bf16*)dv, (const bf16*)dgate, \
                                                      (bf16*)dqkv, dqw, dkw, M, H, G, rot, eps, q_stride_heads)
  if (lanes == 4) { if (one_plus) OB_QKNORM_BWD_VEC(4, true); else OB_QKNORM_BWD_VEC(4, false); }
  else if (lanes == 8) { if (one_plus) OB_QKNORM_BWD_VEC(8, true); else OB_QKNORM_BWD_VEC(8, false); }
  else if (lanes == 16) { if (one_plus) OB_QKNORM_BWD_VEC(16, true); else OB_QKNORM_BWD_VEC(16, false); }
  if (lanes) {
    OB_CHECK_LAUNCH();
    return 0;
  }
  const int rows_per_block = 16;
  long long blocks = (M + rows_per_block - 1) / rows_per_block;
  size_t sm = 2 * K * sizeof(float);
  if (one_plus)
    qknorm_rope_bwd_kernel<true><<<(unsigned)blocks, threads, sm, s>>>(
        (const bf16*)qkv, (const bf16*)qw, (const bf16*)kw, cosT, sinT, (const bf16*)dq_rot,
        (const bf16*)dk_rot, (const bf16*)dv, (const bf16*)dgate, (bf16*)dqkv, dqw, dkw, M, H, G, K, rot, eps, q_stride_heads,
        rows_per_block);
  else
    qknorm_rope_bwd_kernel<false><<<(unsigned)blocks, threads, sm, s>>>(
        (const bf16*)qkv, (const bf16*)qw, (const bf16*)kw, cosT, sinT, (const bf16*)dq_rot,
        (const bf16*)dk_rot, (const bf16*)dv, (const bf16*)dgate, (bf16*)dqkv, dqw, dkw, M, H, G, K, rot, eps, q_stride_heads,
        rows_per_block);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_fwd_bwd(void* logits, long long ld, long long R, int V, const int* targets,
                  const float* mask, const float* grad_scale, float* loss_sum, float* lse_out,
                  int write_grad, cudaStream_t s) {
  if (V % 8 || ld % 8) return 6001;
  if (R <= 0) return 0;
  ce_fwd_bwd_kernel<<<(unsigned)R, 512, 0, s>>>((bf16*)logits, ld, V, targets, mask, grad_scale,
                                                loss_sum, lse_out, write_grad);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_sigmoid_gate_fwd(const void* o, const void* gate, void* out, long long M, int H, int Kd, long long g_row,
                        long long g_head, cudaStream_t s) {
  if (Kd % 8 || g_row % 8 || g_head % 8 || (((uintptr_t)gate | (uintptr_t)o | (uintptr_t)out) & 15)) return 6001;
  if (M <= 0) return 0;
  sigmoid_gate_fwd_kernel<<<grid_for(M * H * (Kd / 8), 256), 256, 0, s>>>((const bf16*)o, (const bf16*)gate, (bf16*)out,
                                                                          M, H, Kd, g_row, g_head);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_sigmoid_gate_bwd(const void* o, const void* gate, const void* dout, void* d_o, void* d_gate, long long M, int H,
                        int Kd, long long g_row, long long g_head, cudaStream_t s) {
  if (Kd % 8 || g_row % 8 || g_head % 8 || (((uintptr_t)gate | (uintptr_t)o | (uintptr_t)dout) & 15)) return 6001;
  if (M <= 0) return 0;
  sigmoid_gate_bwd_kernel<<<grid_for(M * H * (Kd / 8), 256), 256, 0, s>>>(
      (const bf16*)o, (const bf16*)gate, (const bf16*)dout, (bf16*)d_o, (bf16*)d_gate, M, H, Kd, g_row, g_head);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_finish(const void* stats, int n_tiles, const float* tgt_logit, const float* mask, float* loss_sum,
                 float* lse_out, long long R, const int* rows_dev, int rows_off, cudaStream_t s) {
  if (R <= 0) return 0;
  ce_finish_kernel<<<grid_for(R * 32, 256), 256, 0, s>>>((const float2*)stats, n_tiles, tgt_logit, mask, loss_sum,
                                                         lse_out, R, rows_dev, rows_off);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_count(const float* mask, const int* targets, long long M, int* rows, int* place, int* tgt_out, float* mask_out,
                int* count, cudaStream_t s) {
  ce_count_kernel<<<1, 1024, 0, s>>>(mask, targets, M, rows, place, tgt_out, mask_out, count);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_gather(const void* h, const int* rows, const int* count, void* out, long long M, int D, cudaStream_t s) {
  if (D % 8) return 6001;
  if (((uintptr_t)h | (uintptr_t)out) & 15) return 6002;
  if (M <= 0) return 0;
  ce_gather_kernel<<<grid_for(M * (D / 8), 256), 256, 0, s>>>((const bf16*)h, rows, count, (bf16*)out, M, D);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_scatter(const float* dh, const int* place, const float* g, const float* scale, void* out, long long M, int D,
                  cudaStream_t s) {
  if (D % 8) return 6001;
  if (M <= 0) return 0;
  ce_scatter_kernel<<<grid_for(M * (D / 8), 256), 256, 0, s>>>(dh, place, g, scale, (bf16*)out, M, D);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_counted_grad(void* logits, long long R, int V, long long ld, const int* targets, const float* lse, const float* mask,
                       const float* grad_scale, const int* rows_dev, int rows_off, cudaStream_t s) {
  if (V % 8 || ld % 8) return 6001;
  if (R <= 0) return 0;
  ce_counted_grad_kernel<<<(unsigned)R, 512, 0, s>>>((bf16*)logits, ld, V, targets, lse, mask, grad_scale, rows_dev, rows_off);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_vp_stats(const void* logits, long long R, int V, long long ld, int v0, const int* targets, float* mx,
                   float* sm, float* tg, cudaStream_t s) {
  if (V % 8 || ld % 8) return 6001;
  if (R <= 0) return 0;
  ce_vp_stats_kernel<<<(unsigned)R, 512, 0, s>>>((const bf16*)logits, ld, V, v0, targets, mx, sm, tg);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_ce_vp_grad(void* logits, long long R, int V, long long ld, int v0, const int* targets, const float* lse,
                  const float* mask, const float* grad_scale, cudaStream_t s) {
  if (V % 8 || ld % 8) return 6001;
  if (R <= 0) return 0;
  ce_vp_grad_kernel<<<(unsigned)R, 512, 0, s>>>((bf16*)logits, ld, V, v0, targets, lse, mask, grad_scale);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_embedding_fwd(const int* ids, const void* table, void* out, long long M, int D,
                     cudaStream_t s) {
  if (D % 8) return 6001;
  if (M <= 0) return 0;
  OB_LAUNCH(embedding_fwd_kernel, grid_for(M * (D / 8), 256), 256, 0, s, ids, (const bf16*)table,
                                                                  (bf16*)out, M, D);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_embedding_bwd(const int* ids, const void* dy, float* dtable, long long M, int D, int row_lo,
                     int row_hi, cudaStream_t s) {
  if (D % 2) return 6001;
  if (M <= 0) return 0;
  embedding_bwd_kernel<<<grid_for(M * (D / 2), 256), 256, 0, s>>>(ids, (const bf16*)dy, dtable, M,
                                                                  D, row_lo, row_hi);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_embedding_bwd_peer(const int* ids, const void* dy, void* const* dst_ptrs, int world, int rows_per_rank,
                          long long M, int D, cudaStream_t s) {
  if (D % 2 || world > 8 || rows_per_rank <= 0) return 6001;
  if (M <= 0) return 0;
  EmbPeerPtrs d = {};
  for (int i = 0; i < world; ++i) d.p[i] = (float*)dst_ptrs[i];
  embedding_bwd_peer_kernel<<<grid_for(M * (D / 2), 256), 256, 0, s>>>(ids, (const bf16*)dy, d, M, D, rows_per_rank,
                                                                       world);
  OB_CHECK_LAUNCH();
  return 0;
}

// used (may be null): uint8 [ceil(n / 1024) * 8], one for every 128 elements
int ob_sumsq(const float* g, long long n, float* out, uint8_t* used, cudaStream_t s) {
  if (n <= 0) return 0;
  if (((uintptr_t)g) & 15) return 6002;
  const long long blocks = n / (4 * 8 * 256) + 1, cap = (long long)num_sms() * 32;
  sumsq_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, s>>>(g, n, out, used);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_adamw(float* p, float* m, float* v, float* g, void* p16, long long n, float lr, float b1,
             float b2, float eps, float wd, double bc1, double bc2, float grad_mul,
             const float* norm_sq, float max_norm, int zero_grad, const uint8_t* used, cudaStream_t s) {
  if (n <= 0) return 0;
  if ((((uintptr_t)p) | ((uintptr_t)m) | ((uintptr_t)v) | ((uintptr_t)g)) & 15) return 6002;
  if (p16 && (((uintptr_t)p16) & 7)) return 6002;
  const AdamArgs a = {lr, b1, b2, eps, wd, (float)(1.0 / bc1), (float)(1.0 / bc2)};
  adamw_kernel<<<grid_for(n / 8 + 1, 256), 256, 0, s>>>(p, m, v, g, (bf16*)p16, n, a, grad_mul, norm_sq, max_norm, zero_grad, used);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_cast_f32_bf16(const float* src, void* dst, long long n, cudaStream_t s) {
  if (n <= 0) return 0;
  if ((((uintptr_t)src) & 15) || (((uintptr_t)dst) & 7)) return 6002;
  cast_f32_bf16_kernel<<<grid_for(n / 4 + 1, 256), 256, 0, s>>>(src, (bf16*)dst, n);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_transpose_bf16(const void* src, void* dst, int R, int C, long long lds, long long ldd,
                      cudaStream_t s) {
  if (R <= 0 || C <= 0) return 0;
  dim3 grid((C + 63) / 64, (R + 63) / 64), block(32, 8);
  transpose_bf16_kernel<<<grid, block, 0, s>>>((const bf16*)src, (bf16*)dst, R, C, lds, ldd);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_l2_flush(void* buf, long long bytes, cudaStream_t s) {
  fill_u32_kernel<<<num_sms() * 8, 256, 0, s>>>((uint32_t*)buf, bytes / 4, 0u);
  OB_CHECK_LAUNCH();
  return 0;
}

}  // extern "C"
