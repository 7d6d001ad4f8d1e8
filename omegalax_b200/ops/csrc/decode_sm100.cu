// K8: decode-time attention over a paged KV cache.
//
// Cache layout: k_pages / v_pages [num_pages, page_size, G, HD] (bf16); block_table [B, max_blocks]
// maps the logical block j of sequence b to a physical page; seq_lens [B] counts the tokens
// already stored (padding never enters the cache, so every sequence has its own length).
//
//  decode_append_kernel   per new token: per-head RMSNorm of q and k (optional), rotate-half RoPE
//                         at the token's own position, q -> q_out, k and v -> their page slot.
//  decode_attn_kernel     one CTA per (sequence, kv head, KV split): the R = H/G query heads of
//                         the group share every K/V row that is read (GQA grouping), online
//                         softmax in fp32, partial (m, l, o) per split.
//  decode_combine_kernel  merges the splits.
// Decode is bound by reading the cache once, so these are CUDA-core kernels built around 16-byte
// loads; the tensor cores are not involved.
#include "host_utils.h"
#include "sm100_common.cuh"

namespace ob {

// one warp per (token, head) of the fused [q heads | k heads | v heads] projection
template <bool kOnePlus>
__global__ void decode_append_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ qw,
                                     const bf16* __restrict__ kw, const int* __restrict__ positions,
                                     const int* __restrict__ seq_of_token, const int* __restrict__ slot_of_token,
                                     const int* __restrict__ block_table, int max_blocks, int page_size,
                                     bf16* __restrict__ q_out, bf16* __restrict__ k_pages,
                                     bf16* __restrict__ v_pages, long long ntok, int H, int G, int HD, int rot,
                                     float theta, float eps) {
  grid_begin();
  const int lane = threadIdx.x & 31;
  const long long wid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int HH = H + 2 * G;
  if (wid >= ntok * HH) return;
  const long long t = wid / HH;
  const int h = (int)(wid - t * HH);
  const bf16* src = qkv + t * (long long)HH * HD + (long long)h * HD;
  const int b = seq_of_token[t];
  const int slot = slot_of_token[t];                 // index of this token inside its sequence
  const int page = block_table[(long long)b * max_blocks + slot / page_size];
  const long long cache_row = ((long long)page * page_size + slot % page_size) * G;
  if (h >= H + G) {                                   // value head: plain copy
    bf16* dst = v_pages + (cache_row + (h - H - G)) * HD;
    for (int i = lane; i < HD; i += 32) dst[i] = src[i];
    return;
  }
  const bool is_q = h < H;
  const bf16* w = is_q ? qw : kw;
  bf16* dst = is_q ? q_out + (t * H + h) * HD : k_pages + (cache_row + (h - H)) * HD;
  float ss = 0.f;
  for (int i = lane; i < HD; i += 32) {
    float v = __bfloat162float(src[i]);
    ss += v * v;
  }
  ss = warp_sum(ss);
  const float rstd = w ? rsqrtf(ss / (float)HD + eps) : 1.f;
  const int half = rot >> 1;
  const float pos = (float)positions[t];
  for (int i = lane; i < half; i += 32) {
    float w1 = 1.f, w2 = 1.f;
    if (w) {
      w1 = __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f);
      w2 = __bfloat162float(w[i + half]) + (kOnePlus ? 1.f : 0.f);
    }
    float x1 = __bfloat162float(__float2bfloat16(__bfloat162float(src[i]) * rstd * w1));
    float x2 = __bfloat162float(__float2bfloat16(__bfloat162float(src[i + half]) * rstd * w2));
    float inv = __powf(theta, -(float)(2 * i) / (float)rot);
    float s, c;
    sincosf(pos * inv, &s, &c);
    dst[i] = __float2bfloat16(x1 * c - x2 * s);
    dst[i + half] = __float2bfloat16(x2 * c + x1 * s);
  }
  for (int i = rot + lane; i < HD; i += 32) {
    float wv = w ? __bfloat162float(w[i]) + (kOnePlus ? 1.f : 0.f) : 1.f;
    dst[i] = __float2bfloat16(__bfloat162float(src[i]) * rstd * wv);
  }
}

// Keys and values of a prompt into their pages: row n of k and v (W channels, any pitch) to cache row rows[n].  blockIdx.y: 0 k, 1 v.
// Four 16-byte groups of a thread are in flight.  8192 rows of 1024 channels, keys and values, L2 flushed: 17.4 us (67 MB: 3.9 TB/s),
// where two indexed copies and one to close the gaps of v took 78.8.
__global__ void __launch_bounds__(256)
kv_store_kernel(const bf16* __restrict__ k, const bf16* __restrict__ v, long long ldk, long long ldv,
                const int* __restrict__ rows, bf16* __restrict__ k_pages, bf16* __restrict__ v_pages, long long N, int W) {
  constexpr int U = 4;
  const bf16* src = blockIdx.y ? v : k;
  bf16* dst = blockIdx.y ? v_pages : k_pages;
  const long long ld = blockIdx.y ? ldv : ldk;
  const int wv = W >> 3;
  const long long total = N * wv, i0 = blockIdx.x * (256ll * U) + threadIdx.x;
  uint4 x[U];
  long long at[U];
#pragma unroll
  for (int t = 0; t < U; ++t) {
    const long long i = i0 + t * 256;
    if (i < total) {
      const long long n = i / wv;
      const int c = (int)(i - n * wv) * 8;
      x[t] = *reinterpret_cast<const uint4*>(src + n * ld + c);
      at[t] = (long long)rows[n] * W + c;
    }
  }
#pragma unroll
  for (int t = 0; t < U; ++t)
    if (i0 + t * 256 < total) *reinterpret_cast<uint4*>(dst + at[t]) = x[t];
}

// Sums of V values over the 16 lanes of a half-warp: lane hl ends with value hl * V / 16 (V a power of two up to
// 16).  Exchanging halves takes V - 1 + log2(16 / V) shuffles where a butterfly per value takes 4 V.
template <int V>
__device__ __forceinline__ float transpose_sum16(float (&v)[V], int hl) {
  int mask = 8;
#pragma unroll
  for (int n = V / 2; n > 0; n >>= 1, mask >>= 1) {
    const bool up = hl & mask;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
    }
  }
#pragma unroll
  for (; mask > 0; mask >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], mask);
  return v[0];
}

constexpr int kDecodeStages = 3, kDecodeRing = kDecodeStages * 8 * 128 * 16;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// grid (B, G, splits); 128 threads = 8 half-warps; a half-warp takes four keys at a time, the CTA 32 in a row.
// HD = 128: each lane owns 8 consecutive channels (one 16-byte load per K and V row).
// R <= 8 query heads per kv head share every row that is read.
// Rows arrive through a ring of three stages in shared memory, filled by cp.async two iterations ahead; a lane reads
// back only what it copied itself, so no barrier is involved, and 32 KB a CTA are in flight while it computes.
// With registers in place of the ring a warp computed only when its loads had come back.
// Next to the bytes instructions are the bound, so the 4 R scores of a half-warp are summed by
// transposing: a lane ends with one score (two for R 8), takes its exponential alone and hands it round, and the
// running maximum moves once in four keys.  Everything stays fp32.  32 sequences of 2048 tokens, 32 heads on 8:
// 69 us, from 143 (268 MB: 3.9 TB/s).
template <int HD, int R>
__global__ void __launch_bounds__(128, R <= 4 ? 4 : 2)
decode_attn_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k_pages, const bf16* __restrict__ v_pages,
                   const int* __restrict__ block_table, const int* __restrict__ seq_lens, int max_blocks,
                   int page_size, int G, int splits, float scale, float* __restrict__ part_o,
                   float* __restrict__ part_ml) {
  grid_begin();
  static_assert(HD == 128, "one half-warp covers a 128-channel row");
  constexpr int C = 8;    // channels per lane
  constexpr int NW = 8;   // half-warps per CTA
  constexpr int U = 4;    // keys of a half-warp and iteration
  constexpr int V = R < 4 ? 4 * R : 16;        // scores summed together
  constexpr int S = 4 * R / V;                 // times (2 for R 8: keys 0, 1 and keys 2, 3)
  constexpr int KV = U / S;                    // keys of one sum
  const int b = blockIdx.x, g = blockIdx.y, sp = blockIdx.z;
  const int sub = threadIdx.x >> 4, hl = threadIdx.x & 15;
  const int H = G * R;
  const int len = seq_lens[b];
  const int per = (len + splits - 1) / splits;
  const int k_lo = sp * per, k_hi = min(len, k_lo + per);
  float qv[R][C];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint4 u = *reinterpret_cast<const uint4*>(q + ((long long)b * H + g * R + r) * HD + hl * C);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 t = unpack_bf16(w[c]);
      qv[r][2 * c] = t.x * scale; qv[r][2 * c + 1] = t.y * scale;
    }
  }
  // value i of a sum is (key i / R, head i % R); this lane's is mine
  const int mine = hl * V / 16, my_r = mine % R, my_u = mine / R;
  float m = -INFINITY, l = 0.f, o[R][C];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) o[r][c] = 0.f;
  extern __shared__ __align__(16) uint4 ring[];      // [stage][K rows, V rows of the four keys][thread]
  const int iters = (k_hi - k_lo + NW * U - 1) / (NW * U);
  const int* table = block_table + (long long)b * max_blocks;
  int page[U];       // of the iteration that is fetched next
  auto look_up = [&](int it) {
#pragma unroll
    for (int u = 0; u < U; ++u) page[u] = __ldg(table + min(k_lo + (it * U + u) * NW + sub, k_hi - 1) / page_size);
  };
  auto fetch = [&](int it) {
    const uint32_t dst = smem_u32(ring + (it % kDecodeStages) * 2 * U * 128 + threadIdx.x);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = k_lo + (it * U + u) * NW + sub, sc = min(s, k_hi - 1);      // past the end: zeros
      const long long row = (((long long)page[u] * page_size + sc % page_size) * G + g) * HD + hl * C;
      cp_async16(dst + u * 2048, k_pages + row, s < k_hi);
      cp_async16(dst + (U + u) * 2048, v_pages + row, s < k_hi);
    }
  };
  if (iters > 0) look_up(0);
#pragma unroll
  for (int i = 0; i < kDecodeStages - 1; ++i) {
    if (i < iters) {
      fetch(i);
      look_up(i + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int it = 0; it < iters; ++it) {   // uniform trip count: the shuffles below need all lanes
    const int s0 = k_lo + it * NW * U;
    if (it + kDecodeStages - 1 < iters) {
      fetch(it + kDecodeStages - 1);
      look_up(it + kDecodeStages);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group %0;" ::"n"(kDecodeStages - 1) : "memory");
    const uint4* ku = ring + (it % kDecodeStages) * 2 * U * 128 + threadIdx.x;
    const uint4* vu = ku + U * 128;
    float d[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      float v[V];
#pragma unroll
      for (int t = 0; t < KV; ++t) {
        const uint4 x = ku[(j * KV + t) * 128];
        const uint32_t kw[4] = {x.x, x.y, x.z, x.w};
        float kv[C];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 a = unpack_bf16(kw[c]);
          kv[2 * c] = a.x; kv[2 * c + 1] = a.y;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float a = 0.f;
#pragma unroll
          for (int c = 0; c < C; ++c) a = fmaf(qv[r][c], kv[c], a);
          v[t * R + r] = a;
        }
      }
      d[j] = transpose_sum16<V>(v, hl);
      if (s0 + (j * KV + my_u) * NW + sub >= k_hi) d[j] = -INFINITY;
    }
    // maximum of this head over the four keys
    float mn = d[0];
#pragma unroll
    for (int j = 1; j < S; ++j) mn = fmaxf(mn, d[j]);
#pragma unroll
    for (int x = 16 / KV; x < 16; x <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, x));
    mn = fmaxf(mn, m);
    const bool any = mn != -INFINITY;
    const float a = any ? __expf(m - mn) : 1.f;
    float p[S];
    l *= a;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      p[j] = any ? __expf(d[j] - mn) : 0.f;
      l += p[j];
    }
    m = mn;
    if (__any_sync(0xffffffffu, a != 1.f)) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float ar = __shfl_sync(0xffffffffu, a, r * (16 / V), 16);
#pragma unroll
        for (int c = 0; c < C; ++c) o[r][c] *= ar;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 y = vu[u * 128];
      const uint32_t vw[4] = {y.x, y.y, y.z, y.w};
      float vv[C];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 t = unpack_bf16(vw[c]);
        vv[2 * c] = t.x; vv[2 * c + 1] = t.y;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float pr = __shfl_sync(0xffffffffu, p[u / KV], ((u % KV) * R + r) * (16 / V), 16);
#pragma unroll
        for (int c = 0; c < C; ++c) o[r][c] = fmaf(pr, vv[c], o[r][c]);
      }
    }
  }
#pragma unroll
  for (int x = 16 / KV; x < 16; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
  // merge the eight half-warps through shared memory
  __shared__ float sm_m[NW][R], sm_l[NW][R];
  static_assert(NW * R * HD * 4 <= kDecodeRing, "the partial outputs reuse the ring");
  float(*sm_o)[R][HD] = reinterpret_cast<float(*)[R][HD]>(ring);
  __syncthreads();      // all warps are done with their rows
  if (hl % (16 / V) == 0 && my_u == 0) { sm_m[sub][my_r] = m; sm_l[sub][my_r] = l; }
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int c = 0; c < C; c += 4)
      *reinterpret_cast<float4*>(&sm_o[sub][r][hl * C + c]) = make_float4(o[r][c], o[r][c + 1], o[r][c + 2], o[r][c + 3]);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int c = threadIdx.x;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; ++w) mm = fmaxf(mm, sm_m[w][r]);
    float ll = 0.f, oo = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float a = (sm_m[w][r] == -INFINITY) ? 0.f : __expf(sm_m[w][r] - mm);
      ll += sm_l[w][r] * a;
      oo += sm_o[w][r][c] * a;
    }
    const long long base = (((long long)b * H + g * R + r) * splits + sp);
    part_o[base * HD + c] = oo;
    if (c == 0) { part_ml[base * 2] = mm; part_ml[base * 2 + 1] = ll; }
  }
}

// One CTA per head: the weights of the splits once, a lane each, then every channel's sum with its loads independent.
__global__ void __launch_bounds__(128) decode_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                             bf16* __restrict__ out, int splits, int HD) {
  grid_begin();
  __shared__ float w[64], sm[2];      // weights of the first 64 splits, maximum and denominator
  const long long bh = blockIdx.x;
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + bh * splits;
  if (threadIdx.x < 32) {
    float mm = -INFINITY, ll = 0.f;
    for (int s = threadIdx.x; s < splits; s += 32) mm = fmaxf(mm, ml[s].x);
    mm = warp_max(mm);
    for (int s = threadIdx.x; s < splits; s += 32) {
      const float2 t = ml[s];
      const float ws = t.x == -INFINITY ? 0.f : __expf(t.x - mm);
      ll += t.y * ws;
      if (s < 64) w[s] = ws;
    }
    ll = warp_sum(ll);
    if (threadIdx.x == 0) { sm[0] = mm; sm[1] = ll; }
  }
  __syncthreads();
  const float mm = sm[0], ll = sm[1];
  for (int c = threadIdx.x; c < HD; c += blockDim.x) {
    const float* src = part_o + bh * splits * HD + c;
    float oo = 0.f;
#pragma unroll 8
    for (int s = 0; s < min(splits, 64); ++s) oo += src[(long long)s * HD] * w[s];
    for (int s = 64; s < splits; ++s) oo += ml[s].x == -INFINITY ? 0.f : src[(long long)s * HD] * __expf(ml[s].x - mm);
    out[bh * HD + c] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
  }
}

}  // namespace ob

using namespace ob;

extern "C" {

int ob_decode_append(const void* qkv, const void* qw, const void* kw, const int* positions,
                     const int* seq_of_token, const int* slot_of_token, const int* block_table, int max_blocks,
                     int page_size, void* q_out, void* k_pages, void* v_pages, long long ntok, int H, int G,
                     int HD, int rot, float theta, float eps, int one_plus, cudaStream_t s) {
  if (ntok <= 0) return 0;
  long long warps = ntok * (H + 2 * G);
  long long blocks = (warps * 32 + 255) / 256;
  if (one_plus)
    OB_LAUNCH(decode_append_kernel<true>, (unsigned)blocks, 256, 0, s, 
        (const bf16*)qkv, (const bf16*)qw, (const bf16*)kw, positions, seq_of_token, slot_of_token, block_table,
        max_blocks, page_size, (bf16*)q_out, (bf16*)k_pages, (bf16*)v_pages, ntok, H, G, HD, rot, theta, eps);
  else
    OB_LAUNCH(decode_append_kernel<false>, (unsigned)blocks, 256, 0, s, 
        (const bf16*)qkv, (const bf16*)qw, (const bf16*)kw, positions, seq_of_token, slot_of_token, block_table,
        max_blocks, page_size, (bf16*)q_out, (bf16*)k_pages, (bf16*)v_pages, ntok, H, G, HD, rot, theta, eps);
  OB_CHECK_LAUNCH();
  return 0;
}

int ob_kv_store(const void* k, const void* v, long long ldk, long long ldv, const int* rows, void* k_pages, void* v_pages,
                long long N, int W, cudaStream_t s) {
  if (N <= 0 || W <= 0) return 0;
  if ((W & 7) || (ldk & 7) || (ldv & 7)) return 6001;
  if (((uintptr_t)k | (uintptr_t)v | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) return 6002;
  const long long blocks = (N * (W / 8) + 1023) / 1024;
  if (blocks > 0x7fffffff) return 6005;
  kv_store_kernel<<<dim3((unsigned)blocks, 2), 256, 0, s>>>((const bf16*)k, (const bf16*)v, ldk, ldv, rows, (bf16*)k_pages,
                                                            (bf16*)v_pages, N, W);
  OB_CHECK_LAUNCH();
  return 0;
}

// q [B,H,HD] -> out [B,H,HD]; part_o fp32 [B*H*splits*HD], part_ml fp32 [B*H*splits*2] scratch.
int ob_decode_attn(const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                   const int* seq_lens, int B, int H, int G, int HD, int max_blocks, int page_size, int splits,
                   float scale, float* part_o, float* part_ml, void* out, cudaStream_t s) {
  if (B <= 0) return 0;
  if (HD != 128 || H % G) return 6005;
  const int R = H / G;
  dim3 grid(B, G, splits);
#define OB_DA(RR)                                                                                         \
  OB_ENSURE_DYN_SMEM((decode_attn_kernel<128, RR>), kDecodeRing);                                          \
  OB_LAUNCH((decode_attn_kernel<128, RR>), grid, 128, kDecodeRing, s, (const bf16*)q, (const bf16*)k_pages, (const bf16*)v_pages, \
                                                    block_table, seq_lens, max_blocks, page_size, G, splits,   \
                                                    scale, part_o, part_ml)
  if (R == 1) { OB_DA(1); } else if (R == 2) { OB_DA(2); } else if (R == 4) { OB_DA(4); } else if (R == 8) { OB_DA(8); }
  else return 6005;
#undef OB_DA
  OB_CHECK_LAUNCH();
  OB_LAUNCH(decode_combine_kernel, (unsigned)(B * H), 128, 0, s, part_o, part_ml, (bf16*)out, splits, HD);
  OB_CHECK_LAUNCH();
  return 0;
}

}  // extern "C"
