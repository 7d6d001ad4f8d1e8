// Rows on their way into the gated delta rule and out of it.
//
// The rule works in fp32 on sequences padded to whole chunks, its neighbours in bf16 on the real rows.  As separate operations (split,
// casts, l2 norms, scales, padding, sigmoid, softplus, and the same backward) the way there and back passed 20 times over 50 to
// 100 MB.  Here each way is one pass, bound by HBM: 3001 rows, 16 key heads, 64 of 128, in 40 us (222 MB: 5.5 TB/s), the gradients
// back 42, casts behind the rule 22 and 28; a training step of four such layers' width, three with the rule, 31.3 -> 30.0 ms.
#include "host_utils.h"
#include "serve_common.cuh"
#include "sm100_common.cuh"

namespace ob {

struct GdnRowArgs {
  const bf16* mixed;       // [B*T, C]: Hk q heads of 128, Hk k heads, H v heads of U
  const bf16 *b, *a;       // [B*T, H]
  const float *neg_a, *dt; // [H]: g = neg_a * softplus(a + dt)
  float *q, *k, *v;        // [B*Tp, Hk, 128] twice, [B*Tp, H*U]; their gradients in the backward pass
  float *g, *beta;         // [B*Tp, H]; likewise
  bf16 *dmixed, *db, *da;
  float *da32, *dneg;      // [B*T, H]: gradient of a before rounding, and of neg_a by row
  int T, Tp, Hk, H, V;
  float scale, eps;
};

// One CTA of eight warps per padded row; a warp takes q and k heads, 4 channels a lane.
__global__ void __launch_bounds__(256) gdn_rows_in_kernel(const GdnRowArgs p) {
  const long long row = blockIdx.x;
  const int t = (int)(row % p.Tp), lane = threadIdx.x & 31;
  const bool real = t < p.T;
  const long long src = row / p.Tp * p.T + t;
  const bf16* x = p.mixed + src * (2 * p.Hk * 128 + p.V);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int h = threadIdx.x >> 5; h < 2 * p.Hk; h += 8) {
    float4 f = real ? load4(x + h * 128 + lane * 4) : zero;
    const float r = rsqrtf(warp_sum(f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w) + p.eps);
    const float s = h < p.Hk ? p.scale : 1.f;
    f.x = f.x * r * s; f.y = f.y * r * s; f.z = f.z * r * s; f.w = f.w * r * s;
    store4((h < p.Hk ? p.q + (row * p.Hk + h) * 128 : p.k + (row * p.Hk + h - p.Hk) * 128) + lane * 4, f);
  }
  x += 2 * p.Hk * 128;
  for (int i = threadIdx.x * 8; i < p.V; i += 2048) {
    float f[8] = {};
    if (real) load8(x + i, f);
    store8(p.v + row * p.V + i, f);
  }
  for (int h = threadIdx.x; h < p.H; h += 256) {
    float g = 0.f, be = 0.f;
    if (real) {
      const float y = __bfloat162float(p.a[src * p.H + h]) + p.dt[h];
      g = p.neg_a[h] * (y > 20.f ? y : log1pf(expf(y)));
      be = 1.f / (1.f + expf(-__bfloat162float(p.b[src * p.H + h])));
    }
    p.g[row * p.H + h] = g;
    p.beta[row * p.H + h] = be;
  }
}

// One CTA per real row.
__global__ void __launch_bounds__(256) gdn_rows_in_bwd_kernel(const GdnRowArgs p) {
  const long long src = blockIdx.x, row = src / p.T * p.Tp + src % p.T;
  const int lane = threadIdx.x & 31, C = 2 * p.Hk * 128 + p.V;
  const bf16* x = p.mixed + src * C;
  bf16* dx = p.dmixed + src * C;
  for (int h = threadIdx.x >> 5; h < 2 * p.Hk; h += 8) {
    const float4 f = load4(x + h * 128 + lane * 4);
    float4 d = load4((h < p.Hk ? p.q + (row * p.Hk + h) * 128 : p.k + (row * p.Hk + h - p.Hk) * 128) + lane * 4);
    const float s = h < p.Hk ? p.scale : 1.f;
    d.x *= s; d.y *= s; d.z *= s; d.w *= s;
    const float r = rsqrtf(warp_sum(f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w) + p.eps);
    const float m = warp_sum(f.x * d.x + f.y * d.y + f.z * d.z + f.w * d.w) * r * r;
    store4(dx + h * 128 + lane * 4, make_float4(r * (d.x - f.x * m), r * (d.y - f.y * m), r * (d.z - f.z * m), r * (d.w - f.w * m)));
  }
  dx += 2 * p.Hk * 128;
  for (int i = threadIdx.x * 8; i < p.V; i += 2048) {
    float f[8];
    load8(p.v + row * p.V + i, f);
    store8(dx + i, f);
  }
  for (int h = threadIdx.x; h < p.H; h += 256) {
    const long long at = src * p.H + h;
    const float y = __bfloat162float(p.a[at]) + p.dt[h], e = expf(y), dg = p.g[row * p.H + h];
    const float be = 1.f / (1.f + expf(-__bfloat162float(p.b[at])));
    const float da = dg * p.neg_a[h] * (y > 20.f ? 1.f : e / (1.f + e));
    p.da32[at] = da;
    p.da[at] = __float2bfloat16(da);
    p.dneg[at] = dg * (y > 20.f ? y : log1pf(e));
    p.db[at] = __float2bfloat16(p.beta[row * p.H + h] * be * (1.f - be));
  }
}

// kPad: x bf16 [B, T, W] -> y fp32 [B, Tp, W], zeros past T.  Otherwise back.  W % 8 == 0.
template <bool kPad>
__global__ void __launch_bounds__(256) gdn_rows_cast_kernel(const void* __restrict__ x, void* __restrict__ y, int T, int Tp, int W) {
  const long long row = blockIdx.x;
  const int out = kPad ? Tp : T, t = (int)(row % out);
  const long long src = row / out * (kPad ? T : Tp) + t;
  for (int i = threadIdx.x * 8; i < W; i += 2048) {
    float f[8] = {};
    if (kPad) {
      if (t < T) load8((const bf16*)x + src * W + i, f);
      store8((float*)y + row * W + i, f);
    } else {
      load8((const float*)x + src * W + i, f);
      store8((bf16*)y + row * W + i, f);
    }
  }
}

static int gdn_rows_args(GdnRowArgs& a, int B, int T, int Tp, int Hk, int H, int V) {
  if (B <= 0 || T <= 0 || Tp < T || Hk <= 0 || H <= 0 || V <= 0 || (V & 7) || (long long)B * Tp > 0x7fffffff) return 6005;
  a.T = T; a.Tp = Tp; a.Hk = Hk; a.H = H; a.V = V;
  return 0;
}

}  // namespace ob

using namespace ob;

extern "C" {

int ob_gdn_rows_in(const void* mixed, const void* b, const void* a, const float* neg_a, const float* dt, float* q, float* k, float* v,
                   float* g, float* beta, int B, int T, int Tp, int Hk, int H, int V, float scale, float eps, cudaStream_t s) {
  GdnRowArgs p = {};
  const int e = gdn_rows_args(p, B, T, Tp, Hk, H, V);
  if (e) return e;
  if (((uintptr_t)mixed | (uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) return 6002;
  p.mixed = (const bf16*)mixed; p.b = (const bf16*)b; p.a = (const bf16*)a; p.neg_a = neg_a; p.dt = dt;
  p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.scale = scale; p.eps = eps;
  gdn_rows_in_kernel<<<(unsigned)(B * Tp), 256, 0, s>>>(p);
  OB_CHECK_LAUNCH();
  return 0;
}

// dq, dk, dv, dg, dbeta: gradients of what ob_gdn_rows_in gave
int ob_gdn_rows_in_bwd(const void* mixed, const void* b, const void* a, const float* neg_a, const float* dt, const float* dq,
                       const float* dk, const float* dv, const float* dg, const float* dbeta, void* dmixed, void* db, void* da,
                       float* da32, float* dneg, int B, int T, int Tp, int Hk, int H, int V, float scale, float eps, cudaStream_t s) {
  GdnRowArgs p = {};
  const int e = gdn_rows_args(p, B, T, Tp, Hk, H, V);
  if (e) return e;
  if (((uintptr_t)mixed | (uintptr_t)dq | (uintptr_t)dk | (uintptr_t)dv | (uintptr_t)dmixed) & 15) return 6002;
  p.mixed = (const bf16*)mixed; p.b = (const bf16*)b; p.a = (const bf16*)a; p.neg_a = neg_a; p.dt = dt;
  p.q = const_cast<float*>(dq); p.k = const_cast<float*>(dk); p.v = const_cast<float*>(dv);
  p.g = const_cast<float*>(dg); p.beta = const_cast<float*>(dbeta);
  p.dmixed = (bf16*)dmixed; p.db = (bf16*)db; p.da = (bf16*)da; p.da32 = da32; p.dneg = dneg; p.scale = scale; p.eps = eps;
  gdn_rows_in_bwd_kernel<<<(unsigned)(B * T), 256, 0, s>>>(p);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_gdn_rows_cast(const void* x, void* y, int B, int T, int Tp, int W, int pad, cudaStream_t s) {
  if (B <= 0 || T <= 0 || Tp < T || W <= 0 || (W & 7) || (long long)B * Tp > 0x7fffffff) return 6005;
  if (((uintptr_t)x | (uintptr_t)y) & 15) return 6002;
  if (pad) gdn_rows_cast_kernel<true><<<(unsigned)(B * Tp), 256, 0, s>>>(x, y, T, Tp, W);
  else gdn_rows_cast_kernel<false><<<(unsigned)(B * T), 256, 0, s>>>(x, y, T, Tp, W);
  OB_CHECK_LAUNCH();
  return 0;
}

}  // extern "C"
