// Decode attention of grouped heads of 128 channels over paged rows: one query row per sequence, up to eight query
// heads (R) on a key head, keys and values bf16 anywhere in a row of fixed pitch.
//
// The cache is read once and little else is moved, so the bound is HBM as long as a key costs few instructions.
// On CUDA cores it cost about 50 a warp and key row (products, unpacking, sums over lanes).  Here it costs 7: mma.sync
// tiles with the heads as rows.  Their eight spare rows carry precision instead of padding: a probability p enters as three bf16
// terms hi + mid + lo (24 bits, all of an fp32 mantissa), hi in row r and mid in row r + 8 of one product, lo in row r of a
// second, so a lane splits its own values and no shuffle is involved.  Queries, keys and values are bf16 in memory and enter
// exactly; scores, maxima, sums and outputs are fp32.  (A term that is zero makes a NaN of an infinite value, so sums that are none while
// their denominators are numbers look at the values again.)
//
// In us, before and now, alone: 32 sequences of 2048 tokens, 32 heads on 8 70.9 48.0 (268 MB: 5.6 TB/s); one of 4096 13.6 11.0; 8 of
// 4096, 32 heads on 4 34.0 19.7; 64 of 300, 16 on 8 23.4 18.1; 64 of one token, 16 on 16 9.0 6.8; Difedra's windowed
// heads, 64 of 1000, 32 on 4 46.0 28.1.  Distance from 64 bits the same to six digits.
//
// A warp walks groups of 16 keys by itself (no CTA barrier before the end) with a ring of three groups in shared memory, filled by
// cp.async two groups ahead: 17 KB a warp in flight, eight warps per SM.  Rows of 272 bytes keep ldmatrix free
// of bank conflicts.
#pragma once
#include "host_utils.h"
#include "sm100_common.cuh"

namespace ob {

struct DecodeRowsArgs {
  const bf16* q;             // head h of sequence b: q + b * ldq + h * 128
  const bf16 *k, *v;         // key head g of cache row r: k + r * pitch + g * head
  const int* table;          // [B, max_blocks]
  const int* len;            // [B] visible tokens, 0: none
  const bf16* sink;          // [H] or null: a score per head that enters the denominator without a value
  float *part_o, *part_ml;   // [B, H, splits, 128], [B, H, splits, 2]: with more than one split
  bf16* out;                 // [B, H, 128]
  long long ldq, pitch;
  int head, H, G, max_blocks, page_size, splits, window;
  float scale;
};

namespace drows {
constexpr int kGroup = 16, kStages = 3;
constexpr int kRow = 272;                              // bytes of a staged row: 256 and one 16-byte bank group
constexpr int kStage = 2 * kGroup * kRow;              // keys, then values
constexpr int kWarpRing = kStages * kStage;

__device__ __forceinline__ void ldsm(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The upper 16 bits of two values as a bf16 pair, and what they leave: cutting (not rounding) makes the three terms
// exact, x = hi + mid + lo, for every finite x.
__device__ __forceinline__ uint32_t cut_pair(float& x, float& y) {
  const uint32_t a = __float_as_uint(x) & 0xffff0000u, b = __float_as_uint(y) & 0xffff0000u;
  x -= __uint_as_float(a);
  y -= __uint_as_float(b);
  return (a >> 16) | b;
}
}  // namespace drows

// grid: key heads x splits x sequences, flat.  Key head fastest, as the heads of a token lie side by side.
template <int kWarps>
static __global__ void __launch_bounds__(32 * kWarps, 8 / kWarps) decode_rows_kernel(const DecodeRowsArgs p) {
  using namespace drows;
  extern __shared__ __align__(128) uint8_t ring[];
  const int R = p.H / p.G;
  const int g = blockIdx.x % p.G, sp = blockIdx.x / p.G % p.splits, b = blockIdx.x / p.G / p.splits;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hr = lane >> 2, tq = lane & 3;
  const int len = p.len[b], first = p.window > 0 ? max(0, len - p.window) : 0, n = len - first;
  const int groups = (n + kGroup - 1) / kGroup, per = (groups + p.splits - 1) / p.splits;
  const int g_lo = min(sp * per, groups) + warp, g_hi = min(sp * per + per, groups);
  const int iters = g_hi > g_lo ? (g_hi - g_lo + kWarps - 1) / kWarps : 0;      // of this warp

  const int* table = p.table + (long long)b * p.max_blocks;
  const bf16* src = (lane < 16 ? p.k : p.v) + (long long)g * p.head + (lane & 15) * 8;
  const uint32_t mine = smem_u32(ring) + warp * kWarpRing;
  const uint32_t dst = mine + (lane >> 4) * (kGroup * kRow) + (lane & 15) * 16;
  auto look_up = [&](int it) {      // cache row of key lane % 16 of a group
    const int t = min((g_lo + it * kWarps) * kGroup + (lane & 15), n - 1) + first;
    return __ldg(table + t / p.page_size) * p.page_size + t % p.page_size;
  };
  auto fetch = [&](int it, int rows) {
    const int left = n - (g_lo + it * kWarps) * kGroup;      // keys past the end become zeros
    const uint32_t d = dst + (it % kStages) * kStage;
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      const long long r = __shfl_sync(0xffffffffu, rows, i);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + i * kRow), "l"(src + r * p.pitch), "r"(i < left ? 16 : 0)
                   : "memory");
    }
  };
  // The kernel before this one stores each sequence's newest key at most: groups without it are fetched at once.
  bool begun = false;
  int rows = iters > 0 ? look_up(0) : 0;
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) {
    if (i < iters) {
      if (!begun && (g_lo + i * kWarps + 1) * kGroup >= n) {
        grid_begin();
        begun = true;
      }
      fetch(i, rows);
      rows = look_up(i + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (!begun) grid_begin();

  uint32_t qa[8][2];      // queries as the row operand: row hr, channels 16 ks + 2 tq and + 8
  {
    const bf16* q = p.q + (long long)b * p.ldq + (long long)(g * R + hr) * 128 + tq * 2;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks)
#pragma unroll
      for (int e = 0; e < 2; ++e) qa[ks][e] = hr < R ? *reinterpret_cast<const uint32_t*>(q + ks * 16 + e * 8) : 0u;
  }
  float m = -INFINITY, l = 0.f, o[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) o[i][c] = 0.f;
  const uint32_t ka = mine + (lane & 7) * kRow + (lane >> 3) * 16;                                   // 8 keys x 32 channels
  const uint32_t va = mine + (kGroup + (lane & 15)) * kRow + (lane >> 4) * 16;                       // 16 keys x 16 channels

  for (int it = 0; it < iters; ++it) {
    if (it + kStages - 1 < iters) {
      fetch(it + kStages - 1, rows);
      rows = look_up(it + kStages);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
    __syncwarp();
    const uint32_t st = (it % kStages) * kStage;
    float s[2][2][4] = {};      // [block of 8 keys][even, odd k-steps]
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) {
        uint32_t kb[4];
        ldsm(kb, ka + st + j * 8 * kRow + k2 * 64);
        mma(s[j][0], qa[2 * k2][0], 0u, qa[2 * k2][1], 0u, kb[0], kb[1]);
        mma(s[j][1], qa[2 * k2 + 1][0], 0u, qa[2 * k2 + 1][1], 0u, kb[2], kb[3]);
      }
    // this lane: head hr, keys 8 j + 2 tq + c
    const int left = n - (g_lo + it * kWarps) * kGroup;
    float x[2][2], mn = m;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        x[j][c] = j * 8 + tq * 2 + c < left ? (s[j][0][c] + s[j][1][c]) * p.scale : -INFINITY;
        mn = fmaxf(mn, x[j][c]);
      }
    mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
    mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
    const bool any = mn != -INFINITY;
    const float a = any ? __expf(m - mn) : 1.f;
    m = mn;
    l *= a;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        x[j][c] = any ? __expf(x[j][c] - mn) : 0.f;
        l += x[j][c];
      }
    if (__any_sync(0xffffffffu, a != 1.f)) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[i][c] *= a;
    }
    uint32_t pt[3][2];
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int j = 0; j < 2; ++j) pt[t][j] = cut_pair(x[j][0], x[j][1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t vb[4];
      ldsm_t(vb, va + st + i * 32);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        mma(o[2 * i + e], pt[0][0], pt[1][0], pt[0][1], pt[1][1], vb[2 * e], vb[2 * e + 1]);
        mma(o[2 * i + e], pt[2][0], 0u, pt[2][1], 0u, vb[2 * e], vb[2 * e + 1]);
      }
    }
    __syncwarp();      // the stage is free for the fetch of the next round
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);

  // merge the warps through shared memory
  __shared__ float sm_m[kWarps][8], sm_l[kWarps][8];
  float(*sm_o)[8][128] = reinterpret_cast<float(*)[8][128]>(ring);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (tq == 0) {
    sm_m[warp][hr] = m;
    sm_l[warp][hr] = l;
  }
  if (hr < R) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      *reinterpret_cast<float2*>(&sm_o[warp][hr][i * 8 + tq * 2]) = make_float2(o[i][0] + o[i][2], o[i][1] + o[i][3]);
  }
  __syncthreads();
  auto merge = [&](int r, int c, float& mm, float& ll, float& oo) {
    mm = -INFINITY;
    ll = oo = 0.f;
    if (p.splits == 1 && p.sink) {
      mm = __bfloat162float(p.sink[g * R + r]);
      ll = 1.f;
    }
    const float m0 = mm;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, sm_m[w][r]);
    if (ll != 0.f) ll = __expf(m0 - mm);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float e = sm_m[w][r] == -INFINITY ? 0.f : __expf(sm_m[w][r] - mm);
      ll += sm_l[w][r] * e;
      oo += sm_o[w][r][c] * e;
    }
  };
  bool none = false;
  for (int i = threadIdx.x; i < R * 128; i += 32 * kWarps) {
    const int r = i >> 7, c = i & 127;
    const long long bh = (long long)b * p.H + g * R + r;
    float mm, ll, oo;
    merge(r, c, mm, ll, oo);
    none |= oo != oo;
    if (p.splits == 1) {
      p.out[bh * 128 + c] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
    } else {
      const long long at = bh * p.splits + sp;
      p.part_o[at * 128 + c] = oo;
      if (c == 0) *reinterpret_cast<float2*>(p.part_ml + at * 2) = make_float2(mm, ll);
    }
  }
  // Infinite values of one sign among this CTA's keys: apart from the loop above, whose iterations overlap without it (0.6 us), and with the CTA's
  // keys worked out anew, so that nothing is kept for it through the walk.
  if (none) {
    unsigned cta;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta) : : "memory");
    const int split = cta / p.G % p.splits, seq = cta / p.G / p.splits, end = p.len[seq];
    const int begin = p.window > 0 ? max(0, end - p.window) : 0;
    const int share = ((end - begin + kGroup - 1) / kGroup + p.splits - 1) / p.splits * kGroup;
    const int* pages = p.table + (long long)seq * p.max_blocks;
#pragma unroll 1
    for (int i = threadIdx.x; i < R * 128; i += 32 * kWarps) {
      const int r = i >> 7, c = i & 127;
      const long long bh = (long long)b * p.H + g * R + r;
      float mm, ll, oo;
      merge(r, c, mm, ll, oo);
      if (oo == oo || ll != ll) continue;
      bool up = false, down = false, nan = false;
#pragma unroll 1
      for (int key = begin + split * share; key < min(end, begin + split * share + share); ++key) {
        const long long row = (long long)pages[key / p.page_size] * p.page_size + key % p.page_size;
        const float v = __bfloat162float(p.v[row * p.pitch + (long long)g * p.head + c]);
        up |= v == INFINITY;
        down |= v == -INFINITY;
        nan |= v != v;
      }
      if (up == down || nan) continue;
      const float x = up ? INFINITY : -INFINITY;
      if (p.splits == 1) p.out[bh * 128 + c] = __float2bfloat16(x);
      else p.part_o[(bh * p.splits + sp) * 128 + c] = x;
    }
  }
}

// One CTA per head: the weights of the splits once, a lane each, then every channel's sum with its loads independent.
static __global__ void __launch_bounds__(128) decode_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                             const bf16* __restrict__ sink, bf16* __restrict__ out, int H,
                                                             int splits) {
  grid_begin();
  __shared__ float w[64], sm[2];      // weights of the first 64 splits, maximum and denominator
  const long long bh = blockIdx.x;
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + bh * splits;
  if (threadIdx.x < 32) {
    const float s0 = sink ? __bfloat162float(sink[bh % H]) : -INFINITY;
    float mm = s0, ll = 0.f;
    for (int s = threadIdx.x; s < splits; s += 32) mm = fmaxf(mm, ml[s].x);
    mm = warp_max(mm);
    for (int s = threadIdx.x; s < splits; s += 32) {
      const float2 t = ml[s];
      const float ws = t.x == -INFINITY ? 0.f : __expf(t.x - mm);
      ll += t.y * ws;
      if (s < 64) w[s] = ws;
    }
    ll = warp_sum(ll);
    if (threadIdx.x == 0) {
      sm[0] = mm;
      sm[1] = ll + (s0 == -INFINITY ? 0.f : __expf(s0 - mm));
    }
  }
  __syncthreads();
  const int c = threadIdx.x;
  const float mm = sm[0], ll = sm[1], *src = part_o + bh * splits * 128 + c;
  float oo = 0.f;
#pragma unroll 8
  for (int s = 0; s < min(splits, 64); ++s) oo += src[(long long)s * 128] * w[s];
  for (int s = 64; s < splits; ++s) oo += ml[s].x == -INFINITY ? 0.f : src[(long long)s * 128] * __expf(ml[s].x - mm);
  out[bh * 128 + c] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
}

// 1 <= H / G <= 8, 1 <= splits; channels contiguous, everything in multiples of 8 channels on 16-byte boundaries
static int launch_decode_rows(const DecodeRowsArgs& a, int B, cudaStream_t s) {
  if (a.G <= 0 || a.H % a.G || a.H / a.G > 8 || a.H < a.G || a.splits < 1) return 6005;
  if ((a.pitch | a.head | a.ldq) & 7) return 6001;
  if (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v) & 15) return 6002;
  const long long ctas = (long long)B * a.G * a.splits;
  if (ctas > 0x7fffffff || (long long)B * a.H > 0x7fffffff) return 6005;
  // four warps share the keys while that leaves no CTA waiting; more CTAs of two warps fill the SMs more evenly
  if (ctas <= 2 * num_sms()) {
    OB_ENSURE_DYN_SMEM(decode_rows_kernel<4>, 4 * drows::kWarpRing);
    OB_LAUNCH(decode_rows_kernel<4>, (unsigned)ctas, 128, 4 * drows::kWarpRing, s, a);
  } else {
    OB_ENSURE_DYN_SMEM(decode_rows_kernel<2>, 2 * drows::kWarpRing);
    OB_LAUNCH(decode_rows_kernel<2>, (unsigned)ctas, 64, 2 * drows::kWarpRing, s, a);
  }
  OB_CHECK_LAUNCH();
  if (a.splits > 1) {
    OB_LAUNCH(decode_combine_kernel, (unsigned)(B * a.H), 128, 0, s, a.part_o, a.part_ml, a.sink, a.out, a.H, a.splits);
    OB_CHECK_LAUNCH();
  }
  return 0;
}

}  // namespace ob
