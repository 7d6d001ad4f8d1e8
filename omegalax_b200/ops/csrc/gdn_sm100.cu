// K7a: chunked gated delta rule (GatedDeltaNet core), forward and backward, fp32 throughout
// (the reference keeps this recurrence in fp32: omegalax/models/qwen3_5/deltanet.py:68-70).
//
// Per (batch, value head) the state S [A=128, U] is carried through the sequence in chunks of
// 64 tokens.  With gamma = cumsum(g) inside the chunk, a_i = exp(gamma_i), b_j = exp(gamma_C - gamma_j),
// D_ij = exp(gamma_i - gamma_j):
//     L_ij = beta_i (k_i . k_j) D_ij  (i > j)        P_ij = (q_i . k_j) D_ij  (i >= j)
//     r_i  = beta_i (v_i - a_i (k S)_i)              n = (I + L)^-1 r
//     o_i  = a_i (q S)_i + sum_j P_ij n_j            S'  = a_C S + sum_j b_j k_j n_j^T
// and backward, from the chunk-start states and the rows n that the forward saved,
//     dn = P^T do + b (k dS')        dr = (I + L)^-T dn        dL = -dr n^T     dP = do n^T
//     dS = a_C dS' + sum_i a_i q_i do_i^T - sum_i beta_i a_i k_i dr_i^T
// and everything else by the product rule.
//
// Only S and dS tie the chunks together, so what does not need them leaves the walk:
//   gdn_prep_kernel    all chunks at once: (I + L)^-1 and P (backward: their transposes, P, and (k k^T) D)
//   gdn_fwd_kernel     the walk: k S and q S, r, n, o, S'
//   gdn_dstate_kernel  the walk back: dn, dr, dS (saved per chunk)
//   gdn_grad_kernel    all chunks at once: dq, dk, dg, dbeta
// The walks take 128 of 148 SMs at 64 heads of 128 (one CTA per head and 64 value channels); with everything in
// them they took 34 and 91 us a chunk, now 16 and 16.  One layer of 3008 tokens, 64 heads on 16: 1.61 -> 0.87 ms forward (prep 0.13),
// 4.73 -> 2.46 backward (prep 0.16, walk 0.77, gradients 1.50); the multiply-adds keep 50 to 57 % of the fp32 pipes busy, the
// operands 65 % of the shared-memory ports.  Distance from 64 bits at eight shapes: no larger than with the substitution on r and dn.
//
// Products run on packed fp32 pairs (two multiply-adds an instruction, fma.rn.f32x2): operands stored along the reduction give pairs of
// partial sums for even and odd elements (mm_k), outputs whose columns are consecutive in one operand pairs of columns
// (mm_n).  Tiles lie in shared memory with row strides = 4 mod 32 words: 128-bit reads along rows are free of conflicts.  The walks load
// a chunk ahead with cp.async.  Quantities that sum over the slices of U and over the value heads of a key head (dq, dk,
// dg, dbeta) are accumulated with reductions in global memory.
#include "host_utils.h"
#include "sm100_common.cuh"

namespace ob {

constexpr int GC = 64;          // chunk length
constexpr int GA = 128;         // key head dim
constexpr int BU = 64;          // value channels of a CTA
constexpr int LDA_ = GA + 4;    // row stride of [.][128] tiles
constexpr int LDC_ = GC + 4;    // of [.][64] tiles
constexpr int kTileA = GC * LDA_, kTileC = GC * LDC_;

struct GdnArgs {
  const float* q;       // [B,T,Hk,A]  (L2-normalised, q pre-scaled)
  const float* k;       // [B,T,Hk,A]
  const float* v;       // [B,T,H,U]
  const float* g;       // [B,T,H]   log decay (<= 0)
  const float* beta;    // [B,T,H]
  const float* s0;      // [B,H,A,U] or null: state (backward: gradient of the state) that the walk starts from
  float* s1;            // [B,H,A,U] or null: where it ends
  float* carry;         // [B,H,U,A]: between two ranges of chunks of one walk
  float* o;             // [B,T,H,U]
  float* n;             // [B,T,H,U] solved rows (saved for the backward) or null
  float* states;        // [B,H,J,U,A] chunk-start states or null
  // work buffers of the chunks j0 ... j1 - 1, [B,H,j1-j0,64,64]
  float *inv, *pm;      // (I + L)^-1 and P; transposed for the backward walk
  float *kd, *pr;       // backward: (k k^T) D, and P as it is
  float* dstate;        // backward: [B,H,j1-j0,U,A] gradients of the chunk-end states
  const float* d_o;     // [B,T,H,U]
  float* dq;            // [B,T,Hk,A]  accumulated (zero-initialised by the caller)
  float* dk;            // [B,T,Hk,A]  accumulated
  float* dv;            // [B,T,H,U]: dr between the walk and gdn_grad_kernel, which makes beta dr of it
  float* dg;            // [B,T,H]     accumulated
  float* dbeta;         // [B,T,H]     accumulated
  int B, T, H, Hk, U;   // T is a multiple of 64
  int j0, j1, first, last;      // this range of chunks; whether the walk starts, ends with it
};

// ------------------------------------------------------------------------------------------------ products
// A thread (ty, tx) of 16 x 16 owns rows 4 ty ... + 3 and either columns tx + 16 d (mm_k) or 64 (d / 4) + 4 tx + d % 4 (mm_n).
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t both(float x) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
  return d;
}
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
  return (uint64_t)__float_as_uint(lo) | ((uint64_t)__float_as_uint(hi) << 32);
}

// acc[c][d] (+)= sum_k A[4 ty + c][k] B[tx + 16 d][k], both row-major along k
template <int K>
__device__ __forceinline__ void mm_k(float (&acc)[4][4], const float* __restrict__ A, int lda, const float* __restrict__ Bm, int ldb,
                                     int ty, int tx) {
  uint64_t p[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) p[c][d] = pair2(acc[c][d], 0.f);
  const float *ap = A + 4 * ty * lda, *bp = Bm + tx * ldb;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = *reinterpret_cast<const ulonglong2*>(ap + c * lda + k);
#pragma unroll
    for (int d = 0; d < 4; ++d) b[d] = *reinterpret_cast<const ulonglong2*>(bp + 16 * d * ldb + k);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        p[c][d] = fma2(a[c].x, b[d].x, p[c][d]);
        p[c][d] = fma2(a[c].y, b[d].y, p[c][d]);
      }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) acc[c][d] = lo2(p[c][d]) + hi2(p[c][d]);
}

// the same for two left operands against one right operand
template <int K>
__device__ __forceinline__ void mm_k2(float (&acc0)[4][4], float (&acc1)[4][4], const float* __restrict__ A0, const float* __restrict__ A1,
                                      int lda, const float* __restrict__ Bm, int ldb, int ty, int tx) {
  uint64_t p[2][4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) p[0][c][d] = p[1][c][d] = 0;
  const float *ap = A0 + 4 * ty * lda, *aq = A1 + 4 * ty * lda, *bp = Bm + tx * ldb;
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    ulonglong2 a[2][4], b[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      a[0][c] = *reinterpret_cast<const ulonglong2*>(ap + c * lda + k);
      a[1][c] = *reinterpret_cast<const ulonglong2*>(aq + c * lda + k);
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) b[d] = *reinterpret_cast<const ulonglong2*>(bp + 16 * d * ldb + k);
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          p[e][c][d] = fma2(a[e][c].x, b[d].x, p[e][c][d]);
          p[e][c][d] = fma2(a[e][c].y, b[d].y, p[e][c][d]);
        }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      acc0[c][d] = lo2(p[0][c][d]) + hi2(p[0][c][d]);
      acc1[c][d] = lo2(p[1][c][d]) + hi2(p[1][c][d]);
    }
}

// acc[c][e] (pairs of columns 64 (e / 2) + 4 tx + 2 (e % 2)) += sum_k A[4 ty + c][k] B[k][columns]; kAT: A is stored [k][row]
template <int K, bool kAT>
__device__ __forceinline__ void mm_n(uint64_t (&acc)[4][4], const float* __restrict__ A, int lda, const float* __restrict__ Bm, int ldb,
                                     int ty, int tx) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float a[4][4];      // [row][k]
    if (kAT) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const float4 t = *reinterpret_cast<const float4*>(A + (k + kk) * lda + 4 * ty);
        a[0][kk] = t.x; a[1][kk] = t.y; a[2][kk] = t.z; a[3][kk] = t.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 t = *reinterpret_cast<const float4*>(A + (4 * ty + c) * lda + k);
        a[c][0] = t.x; a[c][1] = t.y; a[c][2] = t.z; a[c][3] = t.w;
      }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const float* bp = Bm + (k + kk) * ldb + 4 * tx;
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(bp), b1 = *reinterpret_cast<const ulonglong2*>(bp + 64);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint64_t x = both(a[c][kk]);
        acc[c][0] = fma2(x, b0.x, acc[c][0]);
        acc[c][1] = fma2(x, b0.y, acc[c][1]);
        acc[c][2] = fma2(x, b1.x, acc[c][2]);
        acc[c][3] = fma2(x, b1.y, acc[c][3]);
      }
    }
  }
}

__device__ __forceinline__ void zero(float (&acc)[4][4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) acc[c][d] = 0.f;
}
__device__ __forceinline__ void zero(uint64_t (&acc)[4][4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) acc[c][d] = 0;
}

// sum over the 16 lanes that share ty (a half warp)
__device__ __forceinline__ float half_warp_sum(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// ------------------------------------------------------------------------------------------------ tiles
__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 64 rows of 128 floats (any pitch), 64 x 64 dense tiles, 64 x 64 of a wider matrix; 256 threads
__device__ __forceinline__ void copy_rows128(float* dst, const float* src, long long pitch, int tid) {
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int i = tid + 256 * it, r = i >> 5, c = (i & 31) * 4;
    copy16(dst + r * LDA_ + c, src + r * pitch + c);
  }
}
__device__ __forceinline__ void copy_rows64(float* dst, const float* src, long long pitch, int tid) {
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int i = tid + 256 * it, r = i >> 4, c = (i & 15) * 4;
    copy16(dst + r * LDC_ + c, src + r * pitch + c);
  }
}
// state tile [64 u][128 a] from / to [U, A] (its own layout) or [A, U] (the callers')
__device__ __forceinline__ void load_state(float* dst, const float* ua, const float* au, int U, int tid) {
  for (int i = tid; i < BU * GA; i += 256) {
    if (ua) dst[(i >> 7) * LDA_ + (i & 127)] = ua[i];
    else dst[(i & 63) * LDA_ + (i >> 6)] = au ? au[(long long)(i >> 6) * U + (i & 63)] : 0.f;
  }
}
__device__ __forceinline__ void store_state(float* ua, float* au, const float* src, int U, int tid) {
  if (ua) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int i = tid + 256 * it, r = i >> 5, c = (i & 31) * 4;
      *reinterpret_cast<float4*>(ua + r * GA + c) = *reinterpret_cast<const float4*>(src + r * LDA_ + c);
    }
  }
  if (au)
    for (int i = tid; i < BU * GA; i += 256) au[(long long)(i >> 6) * U + (i & 63)] = src[(i & 63) * LDA_ + (i >> 6)];
}

// gamma (inclusive cumsum of g), a = exp(gamma), b = exp(gamma_last - gamma) of a chunk; lane l of one warp brings g of tokens 2 l, 2 l + 1
__device__ __forceinline__ void chunk_scalars(float x0, float x1, float* gam, float* a, float* b, int lane) {
  float s = x0 + x1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += t;
  }
  const float g1 = s, g0 = s - x1;
  const float last = __shfl_sync(0xffffffffu, s, 31);
  gam[2 * lane] = g0; gam[2 * lane + 1] = g1;
  a[2 * lane] = expf(g0); a[2 * lane + 1] = expf(g1);
  b[2 * lane] = expf(last - g0); b[2 * lane + 1] = expf(last - g1);
}

// ------------------------------------------------------------------------------------------------ what needs no state
// CTA = (chunk, key head, batch), for up to four of its value heads at a time.  k k^T and q k^T once for all of them; the inverse of
// I + L by forward substitution on unit vectors, a column a thread (64 threads a head).
template <bool kBwd>
__global__ void __launch_bounds__(256) gdn_prep_kernel(GdnArgs p) {
  extern __shared__ __align__(16) float gsm[];
  float *k_s = gsm, *q_s = gsm + kTileA;      // then the L of four heads in their place
  __shared__ float gam[4][GC], ex[4][2][GC], beta[4][GC];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int rep = p.H / p.Hk, Jn = p.j1 - p.j0, jn = blockIdx.x % Jn, j = p.j0 + jn, hk = blockIdx.x / Jn % p.Hk, b = blockIdx.x / Jn / p.Hk;
  const long long row0 = (long long)b * p.T + (long long)j * GC;
  copy_rows128(k_s, p.k + (row0 * p.Hk + hk) * GA, (long long)p.Hk * GA, tid);
  copy_rows128(q_s, p.q + (row0 * p.Hk + hk) * GA, (long long)p.Hk * GA, tid);
  copies_commit();
  copies_wait<0>();
  __syncthreads();
  float kk[4][4], qk[4][4];
  mm_k2<GA>(kk, qk, k_s, q_s, LDA_, k_s, LDA_, ty, tx);
  for (int h0 = 0; h0 < rep; h0 += 4) {
    const int nh = min(4, rep - h0);
    __syncthreads();      // k and q are read, or the heads before are done with their L
    if (tid < 32 * nh) {
      const int w = tid >> 5, lane = tid & 31, h = hk * rep + h0 + w;
      const float *gp = p.g + (row0 + 2 * lane) * p.H + h, *bp = p.beta + (row0 + 2 * lane) * p.H + h;
      chunk_scalars(gp[0], gp[p.H], gam[w], ex[w][0], ex[w][1], lane);
      beta[w][2 * lane] = bp[0];
      beta[w][2 * lane + 1] = bp[p.H];
    }
    __syncthreads();
    for (int w = 0; w < nh; ++w) {
      float* L = gsm + w * kTileC;
      const long long at = (((long long)b * p.H + hk * rep + h0 + w) * Jn + jn) * (GC * GC);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = 4 * ty + c;
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const int jj = tx + 16 * d;
          const float D = i >= jj ? expf(gam[w][i] - gam[w][jj]) : 0.f;
          const float kd = i > jj ? kk[c][d] * D : 0.f, pv = qk[c][d] * D;
          L[i * LDC_ + jj] = beta[w][i] * kd;
          (kBwd ? p.pr : p.pm)[at + i * GC + jj] = pv;
          if (kBwd) {
            p.kd[at + i * GC + jj] = kd;
            p.pm[at + jj * GC + i] = pv;
          }
        }
      }
    }
    __syncthreads();
    const int w = tid >> 6, col = tid & 63;
    if (w < nh) {
      const float* L = gsm + w * kTileC;
      float x[GC];
#pragma unroll
      for (int i = 0; i < GC; ++i) {
        float s = i == col ? 1.f : 0.f;
#pragma unroll
        for (int q4 = 0; q4 < (i + 3) / 4; ++q4) {
          const float4 l = *reinterpret_cast<const float4*>(L + i * LDC_ + 4 * q4);
          if (4 * q4 + 0 < i) s = fmaf(-l.x, x[4 * q4 + 0], s);
          if (4 * q4 + 1 < i) s = fmaf(-l.y, x[4 * q4 + 1], s);
          if (4 * q4 + 2 < i) s = fmaf(-l.z, x[4 * q4 + 2], s);
          if (4 * q4 + 3 < i) s = fmaf(-l.w, x[4 * q4 + 3], s);
        }
        x[i] = s;
      }
      float* out = p.inv + (((long long)b * p.H + hk * rep + h0 + w) * Jn + jn) * (GC * GC);
      if (kBwd) {
#pragma unroll
        for (int i = 0; i < GC; i += 4) *reinterpret_cast<float4*>(out + col * GC + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < GC; ++i) out[i * GC + col] = x[i];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ the walk forward
// CTA = (batch, value head, 64 value channels).  The state and every [64 tokens][64 channels] quantity lie transposed, channel by channel.
__global__ void __launch_bounds__(256, 1) gdn_fwd_kernel(GdnArgs p) {
  extern __shared__ __align__(16) float gsm[];
  float* St = gsm;                      // [64 u][128 a]
  float* kb = St + kTileA;              // two chunks of k
  float* q_s = kb + 2 * kTileA;
  float* inv = q_s + kTileA;            // [64 i][64 j]
  float* pm = inv + kTileC;
  float* rt = pm + kTileC;              // [64 u][64 i]
  float* nt = rt + kTileC;
  float* nb = nt + kTileC;              // b_j n_j
  float* sc = nb + kTileC;              // two chunks of {gamma, a, b, beta}[64]
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, lane = tid & 31;
  const int NS = p.U / BU, bh = blockIdx.x / NS, u0 = blockIdx.x % NS * BU;
  const int b = bh / p.H, h = bh % p.H, hk = h / (p.H / p.Hk), U = p.U, J = p.T / GC, Jn = p.j1 - p.j0;
  const long long qk_pitch = (long long)p.Hk * GA, v_pitch = (long long)p.H * U;
  auto row = [&](int j) { return (long long)b * p.T + (long long)j * GC; };
  auto tile = [&](const float* base, int j) { return base + ((long long)bh * Jn + (j - p.j0)) * (GC * GC); };
  float g0 = 0.f, g1 = 0.f, be0 = 0.f, be1 = 0.f, v[4][4];
  auto fetch_scalars = [&](int j) {
    if (tid < 32) {
      const long long at = (row(j) + 2 * lane) * p.H + h;
      g0 = p.g[at]; g1 = p.g[at + p.H];
      be0 = p.beta[at]; be1 = p.beta[at + p.H];
    }
  };
  auto put_scalars = [&](int j) {
    if (tid < 32) {
      float* s = sc + (j & 1) * 4 * GC;
      chunk_scalars(g0, g1, s, s + GC, s + 2 * GC, lane);
      s[3 * GC + 2 * lane] = be0;
      s[3 * GC + 2 * lane + 1] = be1;
    }
  };
  auto fetch_v = [&](int j) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int d = 0; d < 4; ++d) v[c][d] = p.v[(row(j) + 4 * ty + c) * v_pitch + (long long)h * U + u0 + tx + 16 * d];
  };

  // Copies are committed in the order k, q, inv, P of every chunk, one group each, so two groups may be on their way
  // wherever one of them is needed.
  const int j0 = p.j0;
  copy_rows128(kb + (j0 & 1) * kTileA, p.k + (row(j0) * p.Hk + hk) * GA, qk_pitch, tid);
  copies_commit();
  copy_rows128(q_s, p.q + (row(j0) * p.Hk + hk) * GA, qk_pitch, tid);
  copies_commit();
  copy_rows64(inv, tile(p.inv, j0), GC, tid);
  copies_commit();
  copy_rows64(pm, tile(p.pm, j0), GC, tid);
  copies_commit();
  load_state(St, p.first ? nullptr : p.carry + ((long long)bh * U + u0) * GA, p.s0 ? p.s0 + (long long)bh * GA * U + u0 : nullptr, U, tid);
  fetch_scalars(j0);
  put_scalars(j0);
  fetch_v(j0);

  for (int j = j0; j < p.j1; ++j) {
    const bool more = j + 1 < p.j1;
    float *k_s = kb + (j & 1) * kTileA, *s = sc + (j & 1) * 4 * GC;
    const float *a_s = s + GC, *b_s = s + 2 * GC, *beta_s = s + 3 * GC;
    copies_wait<2>();      // k and q of this chunk
    __syncthreads();
    if (more) {
      copy_rows128(kb + (~j & 1) * kTileA, p.k + (row(j + 1) * p.Hk + hk) * GA, qk_pitch, tid);
      fetch_scalars(j + 1);
    }
    copies_commit();
    if (p.states) store_state(p.states + (((long long)bh * J + j) * U + u0) * GA, nullptr, St, U, tid);

    float w[4][4], o[4][4];
    mm_k2<GA>(w, o, k_s, q_s, LDA_, St, LDA_, ty, tx);
    float ai[4], bi[4], be[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      ai[c] = a_s[4 * ty + c];
      bi[c] = b_s[4 * ty + c];
      be[c] = beta_s[4 * ty + c];
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      float r[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        r[c] = be[c] * (v[c][d] - ai[c] * w[c][d]);
        o[c][d] *= ai[c];
      }
      *reinterpret_cast<float4*>(rt + (tx + 16 * d) * LDC_ + 4 * ty) = make_float4(r[0], r[1], r[2], r[3]);
    }
    copies_wait<2>();      // the inverse
    __syncthreads();
    if (more) {
      copy_rows128(q_s, p.q + (row(j + 1) * p.Hk + hk) * GA, qk_pitch, tid);
      put_scalars(j + 1);
      fetch_v(j + 1);
    }
    copies_commit();
    float n[4][4];
    zero(n);
    mm_k<GC>(n, inv, LDC_, rt, LDC_, ty, tx);
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      *reinterpret_cast<float4*>(nt + (tx + 16 * d) * LDC_ + 4 * ty) = make_float4(n[0][d], n[1][d], n[2][d], n[3][d]);
      *reinterpret_cast<float4*>(nb + (tx + 16 * d) * LDC_ + 4 * ty) =
          make_float4(n[0][d] * bi[0], n[1][d] * bi[1], n[2][d] * bi[2], n[3][d] * bi[3]);
    }
    const long long out = (row(j) + 4 * ty) * v_pitch + (long long)h * U + u0 + tx;
    if (p.n) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int d = 0; d < 4; ++d) p.n[out + c * v_pitch + 16 * d] = n[c][d];
    }
    copies_wait<2>();      // P
    __syncthreads();
    if (more) copy_rows64(inv, tile(p.inv, j + 1), GC, tid);
    copies_commit();
    mm_k<GC>(o, pm, LDC_, nt, LDC_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int d = 0; d < 4; ++d) p.o[out + c * v_pitch + 16 * d] = o[c][d];
    uint64_t ds[4][4];
    zero(ds);
    mm_n<GC, false>(ds, nb, LDC_, k_s, LDA_, ty, tx);
    const float aC = a_s[GC - 1];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float4* x = reinterpret_cast<float4*>(St + (4 * ty + c) * LDA_ + 64 * e + 4 * tx);
        const float4 t = *x;
        *x = make_float4(fmaf(aC, t.x, lo2(ds[c][2 * e])), fmaf(aC, t.y, hi2(ds[c][2 * e])), fmaf(aC, t.z, lo2(ds[c][2 * e + 1])),
                         fmaf(aC, t.w, hi2(ds[c][2 * e + 1])));
      }
    __syncthreads();
    if (more) copy_rows64(pm, tile(p.pm, j + 1), GC, tid);
    copies_commit();
  }
  if (!p.last) store_state(p.carry + ((long long)bh * U + u0) * GA, nullptr, St, U, tid);
  else if (p.s1) store_state(nullptr, p.s1 + (long long)bh * GA * U + u0, St, U, tid);
}

// ------------------------------------------------------------------------------------------------ the walk back
__global__ void __launch_bounds__(256, 1) gdn_dstate_kernel(GdnArgs p) {
  extern __shared__ __align__(16) float gsm[];
  float* dSt = gsm;                     // [64 u][128 a] gradient of the chunk-end state
  float* kb = dSt + kTileA;             // two chunks of k
  float* q_s = kb + 2 * kTileA;
  float* inv = q_s + kTileA;            // transposed: [64 j][64 i]
  float* pm = inv + kTileC;             // P transposed
  float* dot = pm + kTileC;             // [64 u][64 i] do, then -beta a dr
  float* adot = dot + kTileC;           // a do
  float* dnt = adot + kTileC;
  float* sc = dnt + kTileC;             // two chunks of {gamma, a, b, beta}[64]
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, lane = tid & 31;
  const int NS = p.U / BU, bh = blockIdx.x / NS, u0 = blockIdx.x % NS * BU;
  const int b = bh / p.H, h = bh % p.H, hk = h / (p.H / p.Hk), U = p.U, Jn = p.j1 - p.j0;
  const long long qk_pitch = (long long)p.Hk * GA, v_pitch = (long long)p.H * U;
  auto row = [&](int j) { return (long long)b * p.T + (long long)j * GC; };
  auto tile = [&](const float* base, int j) { return base + ((long long)bh * Jn + (j - p.j0)) * (GC * GC); };
  float g0 = 0.f, g1 = 0.f, be0 = 0.f, be1 = 0.f, dO[4][4];
  auto fetch_scalars = [&](int j) {
    if (tid < 32) {
      const long long at = (row(j) + 2 * lane) * p.H + h;
      g0 = p.g[at]; g1 = p.g[at + p.H];
      be0 = p.beta[at]; be1 = p.beta[at + p.H];
    }
  };
  auto put_scalars = [&](int j) {
    if (tid < 32) {
      float* s = sc + (j & 1) * 4 * GC;
      chunk_scalars(g0, g1, s, s + GC, s + 2 * GC, lane);
      s[3 * GC + 2 * lane] = be0;
      s[3 * GC + 2 * lane + 1] = be1;
    }
  };
  auto fetch_do = [&](int j) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int d = 0; d < 4; ++d) dO[c][d] = p.d_o[(row(j) + 4 * ty + c) * v_pitch + (long long)h * U + u0 + tx + 16 * d];
  };

  // committed in the order k, P, inverse, q of every chunk
  const int je = p.j1 - 1;
  copy_rows128(kb + (je & 1) * kTileA, p.k + (row(je) * p.Hk + hk) * GA, qk_pitch, tid);
  copies_commit();
  copy_rows64(pm, tile(p.pm, je), GC, tid);
  copies_commit();
  copy_rows64(inv, tile(p.inv, je), GC, tid);
  copies_commit();
  copy_rows128(q_s, p.q + (row(je) * p.Hk + hk) * GA, qk_pitch, tid);
  copies_commit();
  load_state(dSt, p.first ? nullptr : p.carry + ((long long)bh * U + u0) * GA, p.s0 ? p.s0 + (long long)bh * GA * U + u0 : nullptr, U, tid);
  fetch_scalars(je);
  put_scalars(je);
  fetch_do(je);
  __syncthreads();      // the scalars

  for (int j = je; j >= p.j0; --j) {
    const bool more = j > p.j0;
    float *k_s = kb + (j & 1) * kTileA, *s = sc + (j & 1) * 4 * GC;
    const float *a_s = s + GC, *b_s = s + 2 * GC, *beta_s = s + 3 * GC;
    float ai[4], bi[4], be[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      ai[c] = a_s[4 * ty + c];
      bi[c] = b_s[4 * ty + c];
      be[c] = beta_s[4 * ty + c];
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      *reinterpret_cast<float4*>(dot + (tx + 16 * d) * LDC_ + 4 * ty) = make_float4(dO[0][d], dO[1][d], dO[2][d], dO[3][d]);
      *reinterpret_cast<float4*>(adot + (tx + 16 * d) * LDC_ + 4 * ty) =
          make_float4(dO[0][d] * ai[0], dO[1][d] * ai[1], dO[2][d] * ai[2], dO[3][d] * ai[3]);
    }
    copies_wait<2>();      // k and P of this chunk
    __syncthreads();
    if (more) {
      copy_rows128(kb + (~j & 1) * kTileA, p.k + (row(j - 1) * p.Hk + hk) * GA, qk_pitch, tid);
      fetch_scalars(j - 1);
      fetch_do(j - 1);
    }
    copies_commit();
    store_state(p.dstate + (((long long)bh * Jn + (j - p.j0)) * U + u0) * GA, nullptr, dSt, U, tid);
    float dn[4][4];
    zero(dn);
    mm_k<GA>(dn, k_s, LDA_, dSt, LDA_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int d = 0; d < 4; ++d) dn[c][d] *= bi[c];
    mm_k<GC>(dn, pm, LDC_, dot, LDC_, ty, tx);
#pragma unroll
    for (int d = 0; d < 4; ++d)
      *reinterpret_cast<float4*>(dnt + (tx + 16 * d) * LDC_ + 4 * ty) = make_float4(dn[0][d], dn[1][d], dn[2][d], dn[3][d]);
    copies_wait<2>();      // the inverse
    __syncthreads();
    if (more) copy_rows64(pm, tile(p.pm, j - 1), GC, tid);
    copies_commit();
    float dr[4][4];
    zero(dr);
    mm_k<GC>(dr, inv, LDC_, dnt, LDC_, ty, tx);
    const long long out = (row(j) + 4 * ty) * v_pitch + (long long)h * U + u0 + tx;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int d = 0; d < 4; ++d) p.dv[out + c * v_pitch + 16 * d] = dr[c][d];
#pragma unroll
    for (int d = 0; d < 4; ++d)
      *reinterpret_cast<float4*>(dot + (tx + 16 * d) * LDC_ + 4 * ty) =
          make_float4(-be[0] * ai[0] * dr[0][d], -be[1] * ai[1] * dr[1][d], -be[2] * ai[2] * dr[2][d], -be[3] * ai[3] * dr[3][d]);
    copies_wait<2>();      // q
    __syncthreads();
    if (more) {
      copy_rows64(inv, tile(p.inv, j - 1), GC, tid);
      put_scalars(j - 1);
    }
    copies_commit();
    uint64_t ds[4][4];
    zero(ds);
    mm_n<GC, false>(ds, adot, LDC_, q_s, LDA_, ty, tx);
    mm_n<GC, false>(ds, dot, LDC_, k_s, LDA_, ty, tx);
    const float aC = a_s[GC - 1];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float4* x = reinterpret_cast<float4*>(dSt + (4 * ty + c) * LDA_ + 64 * e + 4 * tx);
        const float4 t = *x;
        *x = make_float4(fmaf(aC, t.x, lo2(ds[c][2 * e])), fmaf(aC, t.y, hi2(ds[c][2 * e])), fmaf(aC, t.z, lo2(ds[c][2 * e + 1])),
                         fmaf(aC, t.w, hi2(ds[c][2 * e + 1])));
      }
    __syncthreads();
    if (more) copy_rows128(q_s, p.q + (row(j - 1) * p.Hk + hk) * GA, qk_pitch, tid);
    copies_commit();
  }
  if (!p.last) store_state(p.carry + ((long long)bh * U + u0) * GA, nullptr, dSt, U, tid);
  else if (p.s1) store_state(nullptr, p.s1 + (long long)bh * GA * U + u0, dSt, U, tid);
}

// ------------------------------------------------------------------------------------------------ gradients of a chunk
// CTA = (chunk of a head, 64 value channels).
__global__ void __launch_bounds__(256, 1) gdn_grad_kernel(GdnArgs p) {
  extern __shared__ __align__(16) float gsm[];
  float* St = gsm;                      // [64 u][128 a] chunk-start state
  float* dSt = St + kTileA;             // gradient of the chunk-end state
  float* k_s = dSt + kTileA;
  float* q_s = k_s + kTileA;
  float* n_s = q_s + kTileA;            // [64 i][64 u]
  float* do_s = n_s + kTileC;
  float* dr_s = do_s + kTileC;
  float* M_s = dr_s + kTileC;           // sym(dKK)
  float* Q_s = M_s + kTileC;            // dQK
  float* sc = Q_s + kTileC;
  float *gam_s = sc, *a_s = sc + GC, *b_s = sc + 2 * GC, *beta_s = sc + 3 * GC, *dgam_s = sc + 4 * GC, *dbeta_s = sc + 5 * GC;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int NS = p.U / BU, Jn = p.j1 - p.j0, u0 = blockIdx.x % NS * BU, jn = blockIdx.x / NS % Jn, bh = blockIdx.x / NS / Jn;
  const int b = bh / p.H, h = bh % p.H, hk = h / (p.H / p.Hk), U = p.U, J = p.T / GC, j = p.j0 + jn;
  const long long row0 = (long long)b * p.T + (long long)j * GC, v_pitch = (long long)p.H * U;
  const long long vat = row0 * v_pitch + (long long)h * U + u0, mat = ((long long)bh * Jn + jn) * (GC * GC);
  copy_rows64(n_s, p.n + vat, v_pitch, tid);
  copy_rows64(do_s, p.d_o + vat, v_pitch, tid);
  copy_rows64(dr_s, p.dv + vat, v_pitch, tid);
  copies_commit();
  copy_rows128(k_s, p.k + (row0 * p.Hk + hk) * GA, (long long)p.Hk * GA, tid);
  copy_rows128(St, p.states + (((long long)bh * J + j) * U + u0) * GA, GA, tid);
  copies_commit();
  copy_rows128(q_s, p.q + (row0 * p.Hk + hk) * GA, (long long)p.Hk * GA, tid);
  copy_rows128(dSt, p.dstate + (((long long)bh * Jn + jn) * U + u0) * GA, GA, tid);
  copies_commit();
  float kd[4][4], pv[4][4], vv[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const int i = 4 * ty + c, jj = tx + 16 * d;
      kd[c][d] = p.kd[mat + i * GC + jj];
      pv[c][d] = p.pr[mat + i * GC + jj];
      vv[c][d] = p.v[vat + i * v_pitch + jj];
    }
  if (tid < 32) {
    const long long at = (row0 + 2 * tid) * p.H + h;
    chunk_scalars(p.g[at], p.g[at + p.H], gam_s, a_s, b_s, tid);
    beta_s[2 * tid] = p.beta[at];
    beta_s[2 * tid + 1] = p.beta[at + p.H];
  }
  if (tid >= 64 && tid < 128) {
    dgam_s[tid - 64] = 0.f;
    dbeta_s[tid - 64] = 0.f;
  }
  copies_wait<2>();
  __syncthreads();

  {  // dP = do n^T, dL = -dr n^T; decay and beta gradients; dQK, sym(dKK)
    float dp[4][4], dl[4][4];
    mm_k2<BU>(dp, dl, do_s, dr_s, LDC_, n_s, LDC_, ty, tx);
    float colE[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = 4 * ty + c;
      const float bi = beta_s[i];
      float rowE = 0.f, rowB = 0.f;
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const int jj = tx + 16 * d;
        const float D = (i >= jj) ? expf(gam_s[i] - gam_s[jj]) : 0.f;
        const float dL = -dl[c][d];
        Q_s[i * LDC_ + jj] = dp[c][d] * D;                 // dQK (zero above the diagonal)
        float E = 0.f;
        if (i > jj) {
          rowB = fmaf(dL, kd[c][d], rowB);
          E = dL * bi * kd[c][d] + dp[c][d] * pv[c][d];
          const float dKK = dL * bi * D;
          M_s[i * LDC_ + jj] = dKK;
          M_s[jj * LDC_ + i] = dKK;
        } else if (i == jj) {
          M_s[i * LDC_ + jj] = 0.f;
        }
        rowE += E;
        colE[d] += E;
      }
      rowE = half_warp_sum(rowE);
      rowB = half_warp_sum(rowB);
      if (tx == 0) {
        atomicAdd(dgam_s + i, rowE);
        atomicAdd(dbeta_s + i, rowB);
      }
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const float e = colE[d] + __shfl_xor_sync(0xffffffffu, colE[d], 16);
      if ((tid & 16) == 0) atomicAdd(dgam_s + tx + 16 * d, -e);
    }
  }
  copies_wait<1>();
  __syncthreads();
  {  // dbeta from r = beta (v - a W), W = k S
    float w[4][4];
    zero(w);
    mm_k<GA>(w, k_s, LDA_, St, LDA_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = 4 * ty + c;
      float s = 0.f;
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const float dr = dr_s[i * LDC_ + tx + 16 * d];
        s = fmaf(dr, vv[c][d] - a_s[i] * w[c][d], s);
        p.dv[vat + i * v_pitch + tx + 16 * d] = beta_s[i] * dr;
      }
      s = half_warp_sum(s);
      if (tx == 0) atomicAdd(dbeta_s + i, s);
    }
  }
  copies_wait<0>();
  __syncthreads();
  // rows of the chunk x 128 channels; this thread's columns 4 tx ... + 3 and 64 + 4 tx ... + 3
  auto row_dot = [&](const uint64_t (&t)[4], const float* x) {
    const float4 x0 = *reinterpret_cast<const float4*>(x + 4 * tx), x1 = *reinterpret_cast<const float4*>(x + 64 + 4 * tx);
    float s = x0.x * lo2(t[0]) + x0.y * hi2(t[0]) + x0.z * lo2(t[1]) + x0.w * hi2(t[1]);
    s += x1.x * lo2(t[2]) + x1.y * hi2(t[2]) + x1.z * lo2(t[3]) + x1.w * hi2(t[3]);
    return half_warp_sum(s);
  };
  auto scale_row = [&](uint64_t (&t)[4], float f) {
#pragma unroll
    for (int e = 0; e < 4; ++e) t[e] = pair2(lo2(t[e]) * f, hi2(t[e]) * f);
  };
  auto add_row = [&](float* dst, const uint64_t (&t)[4]) {
    red_add_v4(dst + 4 * tx, lo2(t[0]), hi2(t[0]), lo2(t[1]), hi2(t[1]));
    red_add_v4(dst + 64 + 4 * tx, lo2(t[2]), hi2(t[2]), lo2(t[3]), hi2(t[3]));
  };
  {  // dq_i = a_i S do_i + sum_j dQK_ij k_j
    uint64_t t[4][4];
    zero(t);
    mm_n<BU, false>(t, do_s, LDC_, St, LDA_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = 4 * ty + c;
      scale_row(t[c], a_s[i]);
      const float dot = row_dot(t[c], q_s + i * LDA_);      // d gamma_i += a_i do_i . (q S)_i
      if (tx == 0) atomicAdd(dgam_s + i, dot);
    }
    mm_n<GC, false>(t, Q_s, LDC_, k_s, LDA_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c) add_row(p.dq + ((row0 + 4 * ty + c) * p.Hk + hk) * GA, t[c]);
  }
  {  // dk_i = -beta_i a_i S dr_i + b_i dS' n_i + sum_j sym(dKK)_ij k_j + sum_i' dQK_i'i q_i'
    uint64_t t[4][4], t2[4][4];
    zero(t);
    zero(t2);
    mm_n<BU, false>(t, dr_s, LDC_, St, LDA_, ty, tx);
    mm_n<BU, false>(t2, n_s, LDC_, dSt, LDA_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = 4 * ty + c;
      scale_row(t[c], -beta_s[i] * a_s[i]);
      scale_row(t2[c], b_s[i]);
      const float dot1 = row_dot(t[c], k_s + i * LDA_);      // d gamma_i += dW_i . W_i
      const float dot2 = row_dot(t2[c], k_s + i * LDA_);     // b_i db_i
      if (tx == 0) {
        atomicAdd(dgam_s + i, dot1 - dot2);
        atomicAdd(dgam_s + GC - 1, dot2);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) t[c][e] = pair2(lo2(t[c][e]) + lo2(t2[c][e]), hi2(t[c][e]) + hi2(t2[c][e]));
    }
    mm_n<GC, false>(t, M_s, LDC_, k_s, LDA_, ty, tx);
    mm_n<GC, true>(t, Q_s, LDC_, q_s, LDA_, ty, tx);
#pragma unroll
    for (int c = 0; c < 4; ++c) add_row(p.dk + ((row0 + 4 * ty + c) * p.Hk + hk) * GA, t[c]);
  }
  {  // d gamma_C += a_C <S, dS'>
    float part = 0.f;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int i = tid + 256 * it, at = (i >> 5) * LDA_ + (i & 31) * 4;
      const float4 x = *reinterpret_cast<const float4*>(St + at), y = *reinterpret_cast<const float4*>(dSt + at);
      part += (x.x * y.x + x.y * y.y) + (x.z * y.z + x.w * y.w);
    }
    part = warp_sum(part);
    if ((tid & 31) == 0) atomicAdd(dgam_s + GC - 1, a_s[GC - 1] * part);
  }
  __syncthreads();
  // dg_t = sum_{i >= t} d gamma_i; partial over this slice of U
  if (tid < GC) {
    float s = 0.f;
    for (int i = tid; i < GC; ++i) s += dgam_s[i];
    atomicAdd(p.dg + (row0 + tid) * p.H + h, s);
    atomicAdd(p.dbeta + (row0 + tid) * p.H + h, dbeta_s[tid]);
  }
}

}  // namespace ob

using namespace ob;

namespace {
constexpr int kPrepSmem = 4 * (4 * kTileC > 2 * kTileA ? 4 * kTileC : 2 * kTileA);
constexpr int kWalkSmem = 4 * (4 * kTileA + 5 * kTileC + 2 * 4 * GC);
constexpr int kGradSmem = 4 * (4 * kTileA + 5 * kTileC + 6 * GC);
static_assert(kWalkSmem <= 227 * 1024 && kGradSmem <= 227 * 1024, "shared memory");

int check_shape(int B, int T, int H, int Hk, int A, int U, int j0, int j1) {
  if (A != GA) return 6101;
  if (U % 64 || U <= 0) return 6102;
  if (T % GC || T <= 0) return 6103;
  if (Hk <= 0 || H % Hk) return 6104;
  if (B <= 0) return 6105;
  if (j0 < 0 || j1 > T / GC || j0 >= j1) return 6106;
  if ((long long)B * H * (U / BU) * (j1 - j0) > 0x7fffffff) return 6105;
  return 0;
}
}  // namespace

extern "C" {

// Chunks j0 ... j1 - 1 of a walk (all ranges of a walk one after the other, first to last).  q,k [B,T,Hk,128] fp32; v [B,T,H,U]; g,beta
// [B,T,H]; s0/s_final [B,H,128,U] optional; n_out [B,T,H,U] and states [B,H,T/64,U,128] optional (needed by the backward).  Work
// buffers: inv, pm [B,H,j1-j0,64,64]; carry [B,H,U,128] with more than one range.
int ob_gdn_fwd(const float* q, const float* k, const float* v, const float* g, const float* beta, const float* s0, float* o,
               float* n_out, float* states, float* s_final, float* inv, float* pm, float* carry, int B, int T, int H, int Hk, int A,
               int U, int j0, int j1, cudaStream_t stream) {
  if (int e = check_shape(B, T, H, Hk, A, U, j0, j1)) return e;
  GdnArgs p{};
  p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.s0 = s0; p.s1 = s_final; p.carry = carry;
  p.o = o; p.n = n_out; p.states = states; p.inv = inv; p.pm = pm;
  p.B = B; p.T = T; p.H = H; p.Hk = Hk; p.U = U;
  p.j0 = j0; p.j1 = j1; p.first = j0 == 0; p.last = j1 == T / GC;
  if (!carry && !(p.first && p.last)) return 6106;
  OB_ENSURE_DYN_SMEM(gdn_prep_kernel<false>, kPrepSmem);
  OB_ENSURE_DYN_SMEM(gdn_fwd_kernel, kWalkSmem);
  gdn_prep_kernel<false><<<B * Hk * (j1 - j0), 256, kPrepSmem, stream>>>(p);
  OB_CHECK_LAUNCH();
  gdn_fwd_kernel<<<B * H * (U / BU), 256, kWalkSmem, stream>>>(p);
  OB_CHECK_LAUNCH();
  return 0;
}

// The same ranges from the last chunk to the first.  dq, dk, dg, dbeta are accumulated into: the caller zero-fills them.  Work buffers: inv, pm,
// kd, pr [B,H,j1-j0,64,64]; dstate [B,H,j1-j0,U,128]; carry as above.
int ob_gdn_bwd(const float* q, const float* k, const float* v, const float* g, const float* beta, const float* n_out,
               const float* states, const float* d_o, const float* d_sfinal, float* dq, float* dk, float* dv, float* dg, float* dbeta,
               float* ds0, float* inv, float* pm, float* kd, float* pr, float* dstate, float* carry, int B, int T, int H,
               int Hk, int A, int U, int j0, int j1, cudaStream_t stream) {
  if (int e = check_shape(B, T, H, Hk, A, U, j0, j1)) return e;
  GdnArgs p{};
  p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.s0 = d_sfinal; p.s1 = ds0; p.carry = carry;
  p.n = const_cast<float*>(n_out); p.states = const_cast<float*>(states); p.d_o = d_o;
  p.inv = inv; p.pm = pm; p.kd = kd; p.pr = pr; p.dstate = dstate;
  p.dq = dq; p.dk = dk; p.dv = dv; p.dg = dg; p.dbeta = dbeta;
  p.B = B; p.T = T; p.H = H; p.Hk = Hk; p.U = U;
  p.j0 = j0; p.j1 = j1; p.first = j1 == T / GC; p.last = j0 == 0;
  if (!carry && !(p.first && p.last)) return 6106;
  OB_ENSURE_DYN_SMEM(gdn_prep_kernel<true>, kPrepSmem);
  OB_ENSURE_DYN_SMEM(gdn_dstate_kernel, kWalkSmem);
  OB_ENSURE_DYN_SMEM(gdn_grad_kernel, kGradSmem);
  gdn_prep_kernel<true><<<B * Hk * (j1 - j0), 256, kPrepSmem, stream>>>(p);
  OB_CHECK_LAUNCH();
  gdn_dstate_kernel<<<B * H * (U / BU), 256, kWalkSmem, stream>>>(p);
  OB_CHECK_LAUNCH();
  gdn_grad_kernel<<<B * H * (U / BU) * (j1 - j0), 256, kGradSmem, stream>>>(p);
  OB_CHECK_LAUNCH();
  return 0;
}

}  // extern "C"
