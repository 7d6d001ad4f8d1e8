// Routed experts of serving decoders, forward only: the router's weight scales an expert's input and the
// outputs of a token's experts are summed into its fp32 residual row.
//
// Prompts sort (token, slot) pairs by expert (moe_route_sm100.cu), gather the scaled rows, run the
// grouped tcgen05 GEMM (or, for fp32 and sizes it cannot address, expert_rows_any_kernel) and sum.
// Few pairs per expert (decoding, short prompts) have a plan of their own, without padding, and kernels that stream each used
// expert's weights once past the pairs routed to it.
#include "host_utils.h"
#include "serve_common.cuh"

namespace ob {

// ------------------------------------------------------------------------------------------------ row movement
// xs[dest[p]] = w[p] * h[p / k]
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) moe_gather_kernel(const T* __restrict__ h, const float* __restrict__ w,
                                                         const int* __restrict__ dest, T* __restrict__ xs, int k, int D,
                                                         int max_rows) {
  const long long pr = blockIdx.x;
  const int d = dest[pr];
  if (d < 0 || d >= max_rows) return;
  const T* src = h + pr / k * D;
  T* dst = xs + (long long)d * D;
  const float a = w[pr];
  if (VEC) {
    for (int i = threadIdx.x * 8; i < D; i += 1024) {
      float v[8];
      load8(src + i, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] *= a;
      store8(dst + i, v);
    }
  } else {
    for (int i = threadIdx.x; i < D; i += 128) dst[i] = from_f<T>(to_f(src[i]) * a);
  }
}

// x[m] += sum over the k slots of y[dest[m * k + j]] (dest null: row m * k + j)
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) moe_sum_kernel(const T* __restrict__ y, const int* __restrict__ dest,
                                                      float* __restrict__ x, int k, int D, int max_rows) {
  grid_begin();
  const long long m = blockIdx.y;
  const int i = (blockIdx.x * 256 + threadIdx.x) * (VEC ? 4 : 1);
  if (i >= D) return;
  float* o = x + m * D + i;
  float4 acc = VEC ? load4(o) : make_float4(o[0], 0.f, 0.f, 0.f);
  for (int j = 0; j < k; ++j) {
    const long long r = dest ? dest[m * k + j] : m * k + j;
    if (r < 0 || r >= max_rows) continue;
    const T* s = y + r * D + i;
    if (VEC) {
      const float4 v = load4(s);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    } else {
      acc.x += to_f(s[0]);
    }
  }
  if (VEC) store4(o, acc);
  else o[0] = acc.x;
}

// ------------------------------------------------------------------------------------------------ any-size grouped product
// C[r, :N] = A[r, :K] W[e]^T for the rows r of [offsets[e], offsets[e + 1]); 64 x 64 tiles, fp32 arithmetic.
// CTA = (column block, expert, every gridDim.z-th row block).
template <typename T, typename O>
__global__ void __launch_bounds__(256) expert_rows_any_kernel(const T* __restrict__ A, const T* __restrict__ W,
                                                              O* __restrict__ C, const int* __restrict__ offsets, int N,
                                                              int K, int max_rows) {
  __shared__ __align__(16) float sa[16][68], sb[16][68];
  const int e = blockIdx.y, n0 = blockIdx.x * 64;
  const int lo = offsets[e], hi = min(offsets[e + 1], max_rows);
  const T* w = W + (long long)e * N * K;
  const int tr = threadIdx.x >> 4, tc = threadIdx.x & 15;
  for (int m0 = lo + blockIdx.z * 64; m0 < hi; m0 += gridDim.z * 64) {
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += 16) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = tr + 16 * i, k = k0 + tc;
        sa[tc][r] = m0 + r < hi && k < K ? to_f(A[(long long)(m0 + r) * K + k]) : 0.f;
        sb[tc][r] = n0 + r < N && k < K ? to_f(w[(long long)(n0 + r) * K + k]) : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        const float4 a = load4(&sa[kk][tr * 4]), b = load4(&sb[kk][tc * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = m0 + tr * 4 + i, n = n0 + tc * 4 + j;
        if (r < hi && n < N) C[(long long)r * N + n] = from_f<O>(acc[i][j]);
      }
  }
}

// ------------------------------------------------------------------------------------------------ few pairs
// Pairs in the order of their experts, and units: at most `cap` consecutive pairs of one expert.
//   order [P]  pairs by expert (in any order within one: a pair's results do not depend on its place)
//   unit [2 * max]  first place in the order, expert << 8 | pairs - 1;  count: number of units
// One CTA; pairs whose id is not in 0 ... E - 1 belong to no unit and add nothing: their rows of y [P, D] become zeros.
constexpr int kPlanExperts = 8192;      // counted in shared memory; more of them in `wide` [E]

__global__ void __launch_bounds__(1024) expert_units_kernel(const int* __restrict__ idx, int P, int E, int cap, int* __restrict__ order,
                                                            int* __restrict__ unit, int* __restrict__ count, int* wide, float* __restrict__ y, int D) {
  extern __shared__ int near[];
  __shared__ int part[2][32];
  int* hist = wide ? wide : near;      // [E] pairs, then the next free place
  grid_begin();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < E; e += 1024) hist[e] = 0;
  __syncthreads();
  for (int i = tid; i < P; i += 1024)
    if ((unsigned)idx[i] < (unsigned)E) atomicAdd(hist + idx[i], 1);
  __syncthreads();
  // places and units before the experts of this thread: inclusive sums over the threads, less its own
  const int per = (E + 1023) / 1024, lo = tid * per, hi = min(lo + per, E);
  int np = 0, nu = 0;
  for (int e = lo; e < hi; ++e) {
    np += hist[e];
    nu += (hist[e] + cap - 1) / cap;
  }
  int sp = np, su = nu;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const int x = __shfl_up_sync(0xffffffffu, sp, o), y = __shfl_up_sync(0xffffffffu, su, o);
    if (lane >= o) { sp += x; su += y; }
  }
  if (lane == 31) { part[0][warp] = sp; part[1][warp] = su; }
  __syncthreads();
  if (warp == 0) {
    int x = part[0][lane], y = part[1][lane];
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int a = __shfl_up_sync(0xffffffffu, x, o), b = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) { x += a; y += b; }
    }
    part[0][lane] = x;
    part[1][lane] = y;
    if (lane == 31) *count = y;
  }
  __syncthreads();
  sp += (warp ? part[0][warp - 1] : 0) - np;
  su += (warp ? part[1][warp - 1] : 0) - nu;
  for (int e = lo; e < hi; ++e) {
    const int n = hist[e];
    hist[e] = sp;
    for (int f = 0; f < n; f += cap, ++su) {
      unit[2 * su] = sp + f;
      unit[2 * su + 1] = e << 8 | (min(cap, n - f) - 1);
    }
    sp += n;
  }
  __syncthreads();
  for (int i = tid; i < P; i += 1024) {
    if ((unsigned)idx[i] < (unsigned)E) {
      order[atomicAdd(hist + idx[i], 1)] = i;
    } else {
      for (int d = 0; d < D; ++d) y[(long long)i * D + d] = 0.f;
    }
  }
}

// xs[place] = h[order[place] / k]; one warp per row, D % 8 == 0.  Places past the pairs that have an expert hold no pair.
__global__ void __launch_bounds__(256) expert_rows_kernel(const bf16* __restrict__ h, const int* __restrict__ idx, const int* __restrict__ order,
                                                          bf16* __restrict__ xs, int P, int E, int k, int D) {
  grid_begin();
  const int place = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (place >= P) return;
  const int pr = order[place];
  if ((unsigned)pr >= (unsigned)P || (unsigned)idx[pr] >= (unsigned)E) return;
  const uint4* src = reinterpret_cast<const uint4*>(h + (long long)(pr / k) * D);
  uint4* dst = reinterpret_cast<uint4*>(xs + (long long)place * D);
#pragma unroll 4
  for (int i = lane; i < D / 8; i += 32) dst[i] = src[i];
}

// The used experts' weights stream past their pairs: 128 rows of W on the M side of the MMA, the NB (16 ... 128) pairs of a unit on
// its N side.  Persistent, one CTA per SM with about 200 KB of tiles in flight across its tasks (unit x 128 rows), so that only the first
// tile of a CTA waits for memory; accumulators alternate between two ranges of TMEM.  kUp: 64 features' gate rows and their up
// rows are one tile; out = silu(s g) (s u) in the order of the pairs, s the weight of the pair (the products are linear in the
// input, so its scale is applied to them).  Otherwise out[pair] = fp32 rows.
// Bound by reading the weights (128 experts of 768, width 2048, 8 per token: 1.21 GB, 184 us).  In us, whole experts with plan and sum, a
// CTA per 16 rows that looked for its pairs before and now, 64 tokens: 255, 209 (5.8 TB/s); against padded
// tiles, 500 tokens: 300, 239; 1000: 311, 287; 2000: 370, 443, where calls go to the tiles (64 pairs per expert are the line).
// Roles (192 threads): warp 0 TMA, warp 1 TMEM and MMA, warps 2 ... 5 empty the accumulators.  Every wait is bounded.
struct ExpertArgs {
  const int *unit, *count, *order;
  const float* weight;
  void* out;
  int rows, K;      // rows of the output, length of the reduction
  int* status;
};

template <int NB>
struct ExpertSmem {
  static constexpr int kABytes = 128 * 64 * 2, kStageBytes = kABytes + NB * 128;
  static constexpr int kStages = 200 * 1024 / kStageBytes;
  static constexpr int kPairOff = kStages * kStageBytes;      // up products on their way to the warps with the gates
  static constexpr int kBarOff = kPairOff + 2 * 16 * 64 * 4;
  static constexpr int kTotal = kBarOff + 512 + 1024;
};

template <int NB, bool kUp>
__global__ void __launch_bounds__(192, 1) experts_few_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                                                             const ExpertArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  using L = ExpertSmem<NB>;
  constexpr int kSt = L::kStages, kCols = 2 * NB < 32 ? 32 : 2 * NB, kPanel = kUp ? 64 : 128;
  uint64_t* full = (uint64_t*)(smem + L::kBarOff);
  uint64_t *empty = full + kSt, *tfull = empty + kSt, *tempty = tfull + 2;
  uint32_t* tmem_slot = (uint32_t*)(tempty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    for (int i = 0; i < kSt; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_begin();
  const int units = *p.count, panels = (p.rows + kPanel - 1) / kPanel, tasks = units * panels;
  const int kblocks = (p.K + 63) / 64;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tasks && ok; t += gridDim.x) {
        const int u = t % units, r0 = t / units * kPanel;      // panels of one expert's units side by side: read once
        const int first = p.unit[2 * u], e = p.unit[2 * u + 1] >> 8;
        const int w0 = (kUp ? 2 * e : e) * p.rows + r0;
        for (int k = 0; k < kblocks; ++k) {
          ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status, OB_ERR_WAIT_EMPTY);
          if (!ok) break;
          uint8_t* sw = smem + stage * L::kStageBytes;
          mbar_expect_tx(&full[stage], L::kStageBytes);
          if (kUp) {
            tma_load_2d(sw, &tmW, &full[stage], k * 64, w0);
            tma_load_2d(sw + L::kABytes / 2, &tmW, &full[stage], k * 64, w0 + p.rows);
          } else {
            tma_load_2d(sw, &tmW, &full[stage], k * 64, w0);
          }
          tma_load_2d(sw + L::kABytes, &tmX, &full[stage], k * 64, first);
          if (++stage == kSt) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, NB, 0, 0);
      int stage = 0, buf = 0;
      uint32_t phase = 0, tphase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tasks && ok; t += gridDim.x) {
        ok = mbar_wait(&tempty[buf], tphase ^ 1, abort_flag, p.status, OB_ERR_WAIT_TMEM_EMPTY);
        if (!ok) break;
        tc_fence_after();
        for (int k = 0; k < kblocks; ++k) {
          ok = mbar_wait(&full[stage], phase, abort_flag, p.status, OB_ERR_WAIT_FULL);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + stage * L::kStageBytes), sx = sw + L::kABytes;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_ss(tmem_base + buf * NB, make_smem_desc(sw + j * 32, 16, 1024), make_smem_desc(sx + j * 32, 16, 1024), idesc,
                    (k | j) ? 1u : 0u);
          umma_commit(&empty[stage]);
          if (++stage == kSt) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        umma_commit(&tfull[buf]);
        if (buf) tphase ^= 1;
        buf ^= 1;
      }
    }
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;      // TMEM lane = row of the tile
    float* pair = (float*)(smem + L::kPairOff);             // [2][16 pairs][64 features]
    int buf = 0, pb = 0;
    uint32_t tphase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tasks && ok; t += gridDim.x) {
      const int u = t % units, r = t / units * kPanel + (kUp ? row & 63 : row);
      const int first = p.unit[2 * u], n = (p.unit[2 * u + 1] & 255) + 1;
      ok = mbar_wait(&tfull[buf], tphase, abort_flag, p.status, OB_ERR_WAIT_TMEM_FULL);
      if (kUp) ok = named_bar_and(1, 128, ok);      // the exchange below takes all four warps
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + buf * NB + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < n; c += 16) {
        uint32_t v[16];
        tmem_ld16(taddr + c, v);
        const int my = c + (lane & 15) < n ? p.order[first + c + (lane & 15)] : 0;      // a lane knows one pair
        const float mw = kUp ? p.weight[my] : 0.f;
        tmem_ld_wait();
        if (kUp) {
          float* x = pair + pb * 16 * 64;
          pb ^= 1;
          if (quad >= 2) {
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i * 64 + (row & 63)] = __uint_as_float(v[i]);
          }
          named_bar_and(1, 128, true);      // a buffer is written again two rounds later, past the next barrier
          if (quad < 2) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float s = __shfl_sync(0xffffffffu, mw, i);
              if (c + i < n && r < p.rows)
                ((bf16*)p.out)[(long long)(first + c + i) * p.rows + r] =
                    __float2bfloat16(silu_f(__uint_as_float(v[i]) * s) * (x[i * 64 + row] * s));
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int pr = __shfl_sync(0xffffffffu, my, i);
            if (c + i < n && r < p.rows) ((float*)p.out)[(long long)pr * p.rows + r] = __uint_as_float(v[i]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
      if (buf) tphase ^= 1;
      buf ^= 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {   // copies that may still be in flight land before shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kCols);
  }
}

template <int NB, bool kUp>
static int launch_experts(const void* X, const void* W, const ExpertArgs& a, int P, int E, cudaStream_t s) {
  CUtensorMap tmW, tmX;
  int e = make_tmap_2d(&tmX, X, P, a.K, a.K, NB, 64);
  if (e) return 2000 + e;
  e = make_tmap_2d(&tmW, W, (uint64_t)E * (kUp ? 2 : 1) * a.rows, a.K, a.K, kUp ? 64 : 128, 64);
  if (e) return 3000 + e;
  auto kern = experts_few_kernel<NB, kUp>;
  OB_ENSURE_DYN_SMEM(kern, ExpertSmem<NB>::kTotal);
  const long long most = (long long)P * ((a.rows + (kUp ? 63 : 127)) / (kUp ? 64 : 128));      // no more tasks than that
  const unsigned grid = (unsigned)(most < num_sms() ? most : num_sms());
  (void)launch(kern, dim3(grid), dim3(192), ExpertSmem<NB>::kTotal, s, 0, tmW, tmX, a);
  OB_CHECK_LAUNCH();
  return 0;
}

}  // namespace ob

using namespace ob;

extern "C" {

// h T [M, D], w fp32 [P], dest [P] (P = M * k) -> xs T [max_rows, D]
int ob_moe_gather(const void* h, const float* w, const int* dest, void* xs, long long P, int k, int D, int max_rows, int fp32,
                  cudaStream_t s) {
  if (P <= 0) return 0;
  if (k <= 0) return 6005;
  const bool vec = D % 8 == 0 && !((((uintptr_t)h) | ((uintptr_t)xs)) & 15);
#define OB_GATHER(T, V) moe_gather_kernel<T, V><<<(unsigned)P, 128, 0, s>>>((const T*)h, w, dest, (T*)xs, k, D, max_rows)
  if (fp32) { if (vec) OB_GATHER(float, true); else OB_GATHER(float, false); }
  else { if (vec) OB_GATHER(bf16, true); else OB_GATHER(bf16, false); }
#undef OB_GATHER
  OB_CHECK_LAUNCH();
  return 0;
}

// x fp32 [M, D] += the k rows of y (bf16 or fp32) of every token
int ob_moe_sum(const void* y, const int* dest, float* x, int M, int k, int D, int max_rows, int y_fp32, cudaStream_t s) {
  const bool vec = D % 4 == 0 && !((((uintptr_t)y) | ((uintptr_t)x)) & 15);
  for (int m0 = 0; m0 < M; m0 += 65535) {      // gridDim.y limit
    const int n = M - m0 < 65535 ? M - m0 : 65535;
    const dim3 grid((D + (vec ? 1023 : 255)) / (vec ? 1024 : 256), n);
    const int* d = dest ? dest + (long long)m0 * k : nullptr;
    const long long skip = dest ? 0 : (long long)m0 * k;
    float* xo = x + (long long)m0 * D;
    const int rows = max_rows - (int)skip;
#define OB_SUM(T, V) OB_LAUNCH((moe_sum_kernel<T, V>), grid, 256, 0, s, (const T*)y + skip * D, d, xo, k, D, rows)
    if (y_fp32) { if (vec) OB_SUM(float, true); else OB_SUM(float, false); }
    else { if (vec) OB_SUM(bf16, true); else OB_SUM(bf16, false); }
#undef OB_SUM
    OB_CHECK_LAUNCH();
  }
  return 0;
}

// C T [max_rows, N] = rows of A T [max_rows, K], grouped by offsets [E + 1], times W T [E, N, K]
int ob_expert_rows_any(const void* A, const void* W, void* C, const int* offsets, int E, int N, int K, int max_rows, int fp32,
                       cudaStream_t s) {
  if (max_rows <= 0) return 0;
  if (E <= 0 || E > 65535) return 6001;
  const int blocks = (max_rows + 64 * E - 1) / (64 * E);      // row blocks of an average expert
  const dim3 grid((N + 63) / 64, E, blocks < 1 ? 1 : blocks > 64 ? 64 : blocks);
  if (fp32) expert_rows_any_kernel<float, float><<<grid, 256, 0, s>>>((const float*)A, (const float*)W, (float*)C, offsets, N, K, max_rows);
  else expert_rows_any_kernel<bf16, bf16><<<grid, 256, 0, s>>>((const bf16*)A, (const bf16*)W, (bf16*)C, offsets, N, K, max_rows);
  OB_CHECK_LAUNCH();
  return 0;
}

// Experts of P = M * k pairs, bf16, for few pairs per expert: h [M, D], idx / weight [P], gate_up [E, 2F, D], down [E, D, F];
// scratch xs [P, D], act [P, F] bf16, plan int32 [1 + 3 * P], and E more with over 8192 experts; y fp32 [P, D].  D, F multiples of 8.
// cap: pairs of a unit (16, 32, 64 or 128).
int ob_experts_few(const void* h, const int* idx, const float* weight, const void* gate_up, const void* down, void* xs, void* act,
                   int* plan, float* y, int P, int k, int E, int D, int F, int cap, int* status, cudaStream_t s) {
  if (P <= 0) return 0;
  if (k <= 0 || E <= 0 || E > 65535 || D <= 0 || F <= 0 || (long long)E * 2 * (D > F ? D : F) > 0x7fffffff) return 6005;
  if ((D & 7) || (F & 7)) return 6001;
  if ((((uintptr_t)h) | ((uintptr_t)gate_up) | ((uintptr_t)down) | ((uintptr_t)act) | ((uintptr_t)xs)) & 15) return 6002;
  int *count = plan, *order = plan + 1, *unit = order + P;
  const bool wide = E > kPlanExperts;
  OB_LAUNCH(expert_units_kernel, 1, 1024, wide ? 0 : E * 4, s, idx, P, E, cap, order, unit, count, wide ? unit + 2 * (size_t)P : (int*)nullptr,
            y, D);
  OB_CHECK_LAUNCH();
  OB_LAUNCH(expert_rows_kernel, (unsigned)((P + 7) / 8), 256, 0, s, (const bf16*)h, idx, (const int*)order, (bf16*)xs, P, E, k, D);
  OB_CHECK_LAUNCH();
  const ExpertArgs up = {unit, count, order, weight, act, F, D, status}, dn = {unit, count, order, weight, y, D, F, status};
#define OB_EXPERTS(NB)                                              \
  do {                                                              \
    const int e = launch_experts<NB, true>(xs, gate_up, up, P, E, s); \
    if (e) return e;                                                \
    return launch_experts<NB, false>(act, down, dn, P, E, s);       \
  } while (0)
  if (cap == 16) OB_EXPERTS(16);
  if (cap == 32) OB_EXPERTS(32);
  if (cap == 64) OB_EXPERTS(64);
  if (cap == 128) OB_EXPERTS(128);
#undef OB_EXPERTS
  return 6005;
}

}  // extern "C"
