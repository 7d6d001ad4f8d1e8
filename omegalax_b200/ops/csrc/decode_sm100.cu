// K8: decode-time attention over a paged KV cache.
//
// Cache layout: k_pages / v_pages [num_pages, page_size, G, HD] (bf16); block_table [B, max_blocks]
// maps the logical block j of sequence b to a physical page; seq_lens [B] counts the tokens
// already stored (padding never enters the cache, so every sequence has its own length).
//
//  decode_append_kernel   per new token: per-head RMSNorm of q and k (optional), rotate-half RoPE
//                         at the token's own position, q -> q_out, k and v -> their page slot.
//  decode_rows_kernel     attention of the R = H/G query heads of a group over its rows, split over the keys (decode_rows.cuh)
//  kv_store_kernel        keys and values of a prompt.
#include "decode_rows.cuh"

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
  if (R != 1 && R != 2 && R != 4 && R != 8) return 6005;
  DecodeRowsArgs a = {};
  a.q = (const bf16*)q; a.ldq = (long long)H * HD;
  a.k = (const bf16*)k_pages; a.v = (const bf16*)v_pages; a.pitch = (long long)G * HD; a.head = HD;
  a.table = block_table; a.len = seq_lens; a.max_blocks = max_blocks; a.page_size = page_size;
  a.part_o = part_o; a.part_ml = part_ml; a.out = (bf16*)out;
  a.H = H; a.G = G; a.splits = splits; a.scale = scale;
  return launch_decode_rows(a, B, s);
}

}  // extern "C"
