// Products of few rows: C[M,N] = X[M,K] W[N,K]^T, where streaming W is what takes the time.
//
// The 128 x 128 tiles of gemm_sm100.cu put the rows of X on the 128 lanes of the tensor core and give every
// output column panel to one CTA: a projection of one decoded token (N 4096) runs on 32 of 148 SMs, with
// 64 KB in flight on each, and multiplies 127 rows of padding.  Here the roles are swapped: 128 rows of W
// are the M side of the MMA, NB (16 .. 128) rows of X its N side.  The reduction of a panel is cut over a cluster
// of up to eight CTAs, whose partial sums meet in shared memory: every CTA sums, in the order of the ranks
// (fp32, no atomics, no workspace), and stores its share of the rows.  Two CTAs per SM, each with a ring of about
// 100 KB, so that one streams while the other starts or drains.  One row, N 24576, K 4096: 5.3 TB/s (37.6 us, against
// 67.1 on 256 x 256 tiles); N 4096: 3.3 TB/s (10.3 us, against 27.2), where launch, first loads and the
// cluster's sum are most of it.
//
// Roles per CTA (192 threads): warp 0 TMA producer, warp 1 TMEM allocation and MMA, warps 2..5 move the
// accumulator to shared memory; all warps sum and store.  Every wait is bounded.
#include "gemm_common.cuh"
#include "host_utils.h"

namespace ob {

struct FewArgs {
  int M, N, K;
  int k_per_split;         // multiple of 64
  void* C;
  long long ldc;
  int out_mode;            // 0 bf16, 1 fp32, 2 fp32 accumulate
  const bf16* residual;
  long long ldr;
  const bf16* bias;
  int vec;                 // C (and residual) rows take 4-element accesses
  int* status;
  // in a decode step (ob_gemm_step)
  const bf16 *X, *norm_w;  // kNorm: rows of X, weights of the norm that they pass on their way to shared memory
  const float* squares;    // kNorm: [M, K / 128] sums of squares of X by panels of 128 columns
  float* squares_out;      // or null: the same of C
  long long ldx;
  float eps;
  int act;                 // 1: W is [gate | up], C = silu(gate) * up, N / 2 columns; 2: C = max(., 0)^2
  int ahead;               // W may be read while the kernel before still runs
};

template <int NB>
struct FewSmem {
  static constexpr int kABytes = 128 * BK * 2;
  static constexpr int kStageBytes = kABytes + NB * BK * 2;
  static constexpr int kStages = NB <= 16 ? 6 : NB <= 32 ? 5 : NB <= 64 ? 4 : 3;
  static constexpr int kRing = kStages * kStageBytes;
  static constexpr int kBarOff = kRing;
  static constexpr int kTotal = kBarOff + 128 + 1024;
  static_assert(NB * 128 * 4 <= kRing, "the partial sums reuse the ring");
  static_assert(2 * (kTotal + 1024) <= 228 * 1024, "two CTAs per SM");
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr)
               : "memory");
  return v;
}

// One stage's rows of X (NB x 64), normalised: 128 threads, 16 bytes of NB / 16 rows each, in the layout that TMA would
// leave (128-byte rows, 16-byte groups exchanged by the row's last three bits).  Loads run kAhead stages ahead, since a stage of
// weights passes in 0.5 us and a load takes one (two ahead, 32 rows: 47 us for N 24576, K 4096, four: 40).
template <int NB>
__device__ __forceinline__ void few_norm_rows(const FewArgs& p, uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar,
                                              volatile int* abort_flag, int m0, int k_begin, int k_end) {
  using L = FewSmem<NB>;
  constexpr int kR = NB / 16, kAhead = NB == 16 ? 6 : 4;
  const int t = threadIdx.x - 64, r0 = t >> 3, c = t & 7, n = (k_end - k_begin) / BK;
  const bf16* w = p.norm_w + k_begin + c * 8;
  uint4 wq[kAhead], xq[kAhead][kR];
  auto load = [&](int j, int i) {
    if (i >= n) return;
    wq[j] = *reinterpret_cast<const uint4*>(w + i * BK);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int m = m0 + r0 + 16 * r;
      xq[j][r] = m < p.M ? *reinterpret_cast<const uint4*>(p.X + m * p.ldx + k_begin + c * 8 + i * BK) : make_uint4(0, 0, 0, 0);
    }
  };
#pragma unroll
  for (int j = 0; j < kAhead; ++j) load(j, j);
  float rstd[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) {      // the eight threads of a row
    const int m = min(m0 + r0 + 16 * r, p.M - 1), parts = p.K >> 7;
    float s = 0.f;
    for (int i = c; i < parts; i += 8) s += p.squares[(long long)m * parts + i];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    rstd[r] = rsqrtf(s / (float)p.K + p.eps);
  }
  int stage = 0;
  uint32_t phase = 0;
  for (int i0 = 0; i0 < n; i0 += kAhead) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (i0 + j >= n) break;
      if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, OB_ERR_WAIT_EMPTY)) return;
      uint8_t* sx = smem + stage * L::kStageBytes + L::kABytes;
      const uint32_t g[4] = {wq[j].x, wq[j].y, wq[j].z, wq[j].w};
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const uint32_t u[4] = {xq[j][r].x, xq[j][r].y, xq[j][r].z, xq[j][r].w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = unpack_bf16(u[e]), y = unpack_bf16(g[e]);
          o[e] = pack_bf16(x.x * rstd[r] * y.x, x.y * rstd[r] * y.y);
        }
        const int row = r0 + 16 * r;
        *reinterpret_cast<uint4*>(sx + row * 128 + ((c ^ (row & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
      }
      load(j, i0 + j + kAhead);
      fence_proxy_async_smem();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(&full_bar[stage]);
      if (++stage == L::kStages) {
        stage = 0;
        phase ^= 1;
      }
    }
  }
}

template <int NB, bool kNorm>
__global__ void __launch_bounds__(kGemmThreads, 2)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const FewArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  using L = FewSmem<NB>;
  constexpr int kSt = L::kStages;
  constexpr int kCols = NB < 32 ? 32 : NB;     // TMEM columns, a power of two from 32
  uint64_t* full_bar = (uint64_t*)(smem + L::kBarOff);
  uint64_t* empty_bar = full_bar + kSt;
  uint64_t* done_bar = empty_bar + kSt;
  uint32_t* tmem_slot = (uint32_t*)(done_bar + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = (int)gridDim.x, rank = (int)blockIdx.x;    // the cluster spans the x dimension
  const int n0 = blockIdx.y * (p.act == 1 ? 64 : 128), m0 = blockIdx.z * NB;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  const int k_begin = rank * p.k_per_split, k_end = min(p.K, k_begin + p.k_per_split);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSt; ++i) {
      mbar_init(&full_bar[i], kNorm ? 5 : 1);      // the copies, and the four warps that bring X
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(done_bar, 1);
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

  if (warp == 0) {
    if (lane == 0) {
      auto load_w = [&](int stage, int k0) {
        uint8_t* sw = smem + stage * L::kStageBytes;
        mbar_expect_tx(&full_bar[stage], kNorm ? L::kABytes : L::kStageBytes);
        tma_load_2d(sw, &tmW, &full_bar[stage], k0, n0);
        if (p.act == 1) tma_load_2d(sw + L::kABytes / 2, &tmW, &full_bar[stage], k0, p.N / 2 + n0);
      };
      // The weights of the first stages are on their way while the kernel before, which gives X, still runs: parameters, that is.
      // Weights that the call itself made (padded, of another type) may come from that very kernel.
      if (!p.ahead) grid_begin();
      const int ahead = min(kSt, (k_end - k_begin + BK - 1) / BK);
      for (int i = 0; i < ahead; ++i) load_w(i, k_begin + i * BK);
      if (p.ahead) grid_begin();
      for (int i = 0; i < ahead && !kNorm; ++i)
        tma_load_2d(smem + i * L::kStageBytes + L::kABytes, &tmX, &full_bar[i], k_begin + i * BK, m0);
      int stage = ahead == kSt ? 0 : ahead;
      uint32_t phase = ahead == kSt;
      for (int k0 = k_begin + ahead * BK; k0 < k_end; k0 += BK) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, OB_ERR_WAIT_EMPTY)) break;
        load_w(stage, k0);
        if (!kNorm) tma_load_2d(smem + stage * L::kStageBytes + L::kABytes, &tmX, &full_bar[stage], k0, m0);
        if (++stage == kSt) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, NB, 0, 0);
      int stage = 0;
      uint32_t phase = 0, accumulate = 0;
      bool ok = true;
      for (int k0 = k_begin; k0 < k_end; k0 += BK) {
        ok = mbar_wait(&full_bar[stage], phase, abort_flag, p.status, OB_ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * L::kStageBytes), sx = sw + L::kABytes;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          umma_ss(tmem_base, make_smem_desc(sw + k * 32, 16, 1024), make_smem_desc(sx + k * 32, 16, 1024), idesc, accumulate);
          accumulate = 1;
        }
        umma_commit(&empty_bar[stage]);
        if (++stage == kSt) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) umma_commit(done_bar);
    }
  } else {
    // accumulator -> partial sums [NB][128] over the ring, which nothing reads or writes any more: a lane is an
    // output column, so a warp's stores cover 128 consecutive bytes
    float* part = reinterpret_cast<float*>(smem);
    const int quad = warp & 3;
    if constexpr (kNorm) {
      grid_wait();
      few_norm_rows<NB>(p, smem, full_bar, empty_bar, abort_flag, m0, k_begin, k_end);
    }
    if (mbar_wait(done_bar, 0, abort_flag, p.status, OB_ERR_WAIT_TMEM_FULL)) {
      __syncwarp();
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < NB; c += 16) {
        uint32_t v[16];
        tmem_ld16(taddr + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) part[(c + i) * 128 + quad * 32 + lane] = __uint_as_float(v[i]);
      }
      tc_fence_before();
    }
  }
  grid_wait();            // the threads that read the residual below
  __syncwarp();
  cluster_sync_all();     // every partial sum of the cluster is in place
  if (!*abort_flag) {
    const int col = n0 + 4 * lane, ncol = min(4, p.N - col);
    const uint32_t mine = smem_u32(smem) + lane * 16;
    // rows of this CTA: rank, rank + splits, ...
    for (int m = rank + splits * warp; m < NB && m0 + m < p.M; m += splits * (kGemmThreads / 32)) {
      float4 s = ld_cluster_v4(mapa_shared(mine + m * 512, 0));
      for (int r = 1; r < splits; ++r) {
        const float4 t = ld_cluster_v4(mapa_shared(mine + m * 512, r));
        s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
      }
      float v[4] = {s.x, s.y, s.z, s.w};
      const long long row = m0 + m;
      if (p.act == 1) {      // lanes 0..15 gate, 16..31 up, rounded as products of their own would be
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[i] = __bfloat162float(__float2bfloat16(v[i]));
          const float u = __shfl_down_sync(0xffffffffu, v[i], 16);
          v[i] = v[i] / (1.f + __expf(-v[i])) * u;
        }
        if (lane < 16)
          *reinterpret_cast<uint2*>((bf16*)p.C + row * p.ldc + col) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
        continue;
      }
      if (ncol <= 0) continue;
      if (p.act == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[i] = fmaxf(__bfloat162float(__float2bfloat16(v[i])), 0.f);
          v[i] *= v[i];
        }
      }
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i) if (i < ncol) v[i] += __bfloat162float(p.bias[col + i]);
      }
      if (p.residual) {
        const bf16* rp = p.residual + row * p.ldr + col;
        if (p.vec && ncol == 4) {
          const uint2 q = *reinterpret_cast<const uint2*>(rp);
          const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y);
          v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y;
        } else {
          for (int i = 0; i < ncol; ++i) v[i] += __bfloat162float(rp[i]);
        }
      }
      if (p.out_mode == 0) {
        bf16* cp = (bf16*)p.C + row * p.ldc + col;
        if (p.squares_out) {      // N % 128 == 0: all lanes are here
          const float2 a = unpack_bf16(pack_bf16(v[0], v[1])), b = unpack_bf16(pack_bf16(v[2], v[3]));
          const float ss = warp_sum(a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y);
          if (lane == 0) p.squares_out[row * (p.N >> 7) + blockIdx.y] = ss;
        }
        if (p.vec && ncol == 4) *reinterpret_cast<uint2*>(cp) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
        else for (int i = 0; i < ncol; ++i) cp[i] = __float2bfloat16(v[i]);
      } else {
        float* cp = (float*)p.C + row * p.ldc + col;
        if (p.vec && ncol == 4) {
          float4 o = make_float4(v[0], v[1], v[2], v[3]);
          if (p.out_mode == 2) {
            const float4 c = *reinterpret_cast<const float4*>(cp);
            o.x += c.x; o.y += c.y; o.z += c.z; o.w += c.w;
          }
          *reinterpret_cast<float4*>(cp) = o;
        } else {
          for (int i = 0; i < ncol; ++i) cp[i] = v[i] + (p.out_mode == 2 ? cp[i] : 0.f);
        }
      }
    }
  } else {   // copies that may still be in flight land before shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) __nanosleep(1000);
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();     // nobody leaves while a partner may still read its sums
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kCols);
  }
}

// CTAs per panel: as many as the SMs take in one wave of two, with slices of at least four k-blocks (six where they are no power
// of two).  The more of the panel's weights wait in the rings when X arrives, the better, but clusters of more than two do not
// fill the last 46 of the 296 places, since the SMs of a GPC are no whole number of them (four: the last 40).  In a chain with
// norms, in us by CTAs per panel: N 6144, K 4096, M 1 2: 15.5, 4: 14.0, 5: 13.1, 6: 18.0; N 10240, M 64 2: 23.4, 3: 21.8, 4: 27.9;
// N 4096, K 12288, M 32 4: 27.1, 7: 25.7, 8: 33.8; N 24576 1: 37.6, 2: 39.3.  Short slices lose: N 9216, K 1024, M 32 2: 9.6, 3: 10.5.
static int few_splits(long long panels, int kblocks) {
  for (int s = 8; s > 1; --s) {
    const bool two = (s & (s - 1)) == 0;
    if (panels * s <= (s == 2 ? 2 * num_sms() : 2 * num_sms() - (s == 4 ? 40 : 46)) && kblocks / s >= (two ? 4 : 6)) return s;
  }
  return 1;
}

template <int NB, bool kNorm = false>
static int launch_few(const void* X, const void* W, FewArgs a, long long ldx, long long ldw, int splits, cudaStream_t stream) {
  CUtensorMap tmW, tmX;
  int e = make_tmap_2d(&tmX, X, a.M, a.K, ldx, NB, BK);
  if (e) return 2000 + e;
  e = make_tmap_2d(&tmW, W, a.N, a.K, ldw, a.act == 1 ? 64 : 128, BK);
  if (e) return 3000 + e;
  auto kern = gemm_few_kernel<NB, kNorm>;
  OB_ENSURE_DYN_SMEM(kern, FewSmem<NB>::kTotal);
  const int panels = (a.N + 127) / 128, mblocks = (a.M + NB - 1) / NB, kblocks = (a.K + BK - 1) / BK;
  if (panels > 65535 || mblocks > 65535) return 6005;
  if (splits <= 0) splits = few_splits((long long)panels * mblocks, kblocks);
  if (splits > 8) return 6005;
  const int per = (kblocks + splits - 1) / splits;
  splits = (kblocks + per - 1) / per;     // every CTA has a slice
  a.k_per_split = per * BK;
  const cudaError_t ce = launch(kern, dim3(splits, panels, mblocks), dim3(kGemmThreads), FewSmem<NB>::kTotal, stream, splits,
                                tmW, tmX, a);
  if (ce != cudaSuccess) {
    (void)cudaGetLastError();
    return 1000 + (int)ce;
  }
  return 0;
}

}  // namespace ob

using namespace ob;

namespace {
constexpr int kReadAhead = 4;
}

extern "C" {

// Launches of this thread that support it overlap with the kernel before them (1) or not (0).
int ob_overlap_launches(int on) {
  overlapped_launches() = on != 0;
  return 0;
}

// C[M,N] (+)= X[M,K] W[N,K]^T (+ bias, residual): contract of ob_gemm_bf16 with K-major operands.  out_mode + kReadAhead: no kernel
// of an overlapped sequence writes W.
// splits: CTAs per column panel (at most 8, fewer where the reduction has fewer slices; 0 chooses).
int ob_gemm_few(const void* X, const void* W, void* C, const void* residual, int M, int N, int K, long long ldx, long long ldw,
                long long ldc, long long ldr, int out_mode, const void* bias, int splits, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  FewArgs a = {};
  if (out_mode & kReadAhead) {
    a.ahead = 1;
    out_mode -= kReadAhead;
  }
  if (K <= 0 || out_mode < 0 || out_mode > 2) return 6005;
  if ((ldx & 7) || (ldw & 7)) return 6001;
  if ((((uintptr_t)X) & 15) || (((uintptr_t)W) & 15)) return 6002;
  a.M = M; a.N = N; a.K = K;
  a.C = C; a.ldc = ldc; a.out_mode = out_mode;
  a.residual = (const bf16*)residual; a.ldr = ldr;
  a.bias = (const bf16*)bias;
  a.vec = !(ldc & 3) && !((uintptr_t)C & (out_mode ? 15 : 7)) && (!residual || (!(ldr & 3) && !((uintptr_t)residual & 7)));
  a.status = status;
#define OB_FEW(NB) return launch_few<NB>(X, W, a, ldx, ldw, splits, stream)
  if (M <= 16) OB_FEW(16);
  if (M <= 32) OB_FEW(32);
  if (M <= 64) OB_FEW(64);
  OB_FEW(128);
#undef OB_FEW
}

// The same for the rows of a decode step, with what stands beside its products (each was a launch of 3 to 5 us in a chain
// where every kernel waits for the one before: 8 layers of 4096 channels, one sequence of 4096 tokens 1001 -> 957 us, 32 of 2048
// 1440 -> 1412; a norm and its product of N 24576, 32 rows, with the activation 42.5 -> 40.0, the product alone 37.6).
// norm_w with squares [M, K / 128] (sums of squares of X by panels of 128 columns; eps): X passes an RMS norm on its way, M <= 32.
// squares_out [M, N / 128] or null: the same sums of C as stored.  act 1: W is [gate | up], C [M, N / 2] = silu(gate) * up of
// the rounded products; 2: C = max(., 0)^2 of them; + kReadAhead as above.  Rounding and order are those of ob_rmsnorm_fwd and ob_swiglu_fwd but for the order of a sum of squares.
int ob_gemm_step(const void* X, const void* W, void* C, const void* residual, int M, int N, int K, long long ldx, long long ldw,
                 long long ldc, long long ldr, const void* norm_w, const float* squares, float eps, float* squares_out, int act,
                 int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return 6005;
  if ((ldx & 7) || (ldw & 7)) return 6001;
  if ((((uintptr_t)X) & 15) || (((uintptr_t)W) & 15)) return 6002;
  FewArgs a = {};
  if (act & kReadAhead) {
    a.ahead = 1;
    act -= kReadAhead;
  }
  a.M = M; a.N = N; a.K = K;
  a.C = C; a.ldc = ldc;
  a.residual = (const bf16*)residual; a.ldr = ldr;
  a.vec = !(ldc & 3) && !((uintptr_t)C & 7) && (!residual || (!(ldr & 3) && !((uintptr_t)residual & 7)));
  a.X = (const bf16*)X; a.ldx = ldx;
  a.norm_w = (const bf16*)norm_w; a.squares = squares; a.eps = eps;
  a.squares_out = squares_out;
  a.act = act;
  a.status = status;
  if (act < 0 || act > 2 || (act && (residual || squares_out)) || (act == 1 && ((N & 127) || !a.vec))) return 6005;
  if (squares_out && (N & 127)) return 6005;
  if (norm_w) {
    if (M > 32 || !squares || (K & 127) || ((uintptr_t)norm_w & 15)) return 6005;
    if (M <= 16) return launch_few<16, true>(X, W, a, ldx, ldw, 0, stream);
    return launch_few<32, true>(X, W, a, ldx, ldw, 0, stream);
  }
  if (M <= 16) return launch_few<16>(X, W, a, ldx, ldw, 0, stream);
  if (M <= 32) return launch_few<32>(X, W, a, ldx, ldw, 0, stream);
  if (M <= 64) return launch_few<64>(X, W, a, ldx, ldw, 0, stream);
  return launch_few<128>(X, W, a, ldx, ldw, 0, stream);
}

}  // extern "C"
