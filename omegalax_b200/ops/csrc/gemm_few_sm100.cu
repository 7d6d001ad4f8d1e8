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

template <int NB>
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
  const int n0 = blockIdx.y * 128, m0 = blockIdx.z * NB;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  const int k_begin = rank * p.k_per_split, k_end = min(p.K, k_begin + p.k_per_split);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSt; ++i) {
      mbar_init(&full_bar[i], 1);
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
      // the weights of the first stages are on their way while the kernel before, which gives X, still runs
      const int ahead = min(kSt, (k_end - k_begin + BK - 1) / BK);
      for (int i = 0; i < ahead; ++i) {
        mbar_expect_tx(&full_bar[i], L::kStageBytes);
        tma_load_2d(smem + i * L::kStageBytes, &tmW, &full_bar[i], k_begin + i * BK, n0);
      }
      grid_begin();
      for (int i = 0; i < ahead; ++i)
        tma_load_2d(smem + i * L::kStageBytes + L::kABytes, &tmX, &full_bar[i], k_begin + i * BK, m0);
      int stage = ahead == kSt ? 0 : ahead;
      uint32_t phase = ahead == kSt;
      for (int k0 = k_begin + ahead * BK; k0 < k_end; k0 += BK) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, OB_ERR_WAIT_EMPTY)) break;
        uint8_t* sw = smem + stage * L::kStageBytes;
        mbar_expect_tx(&full_bar[stage], L::kStageBytes);
        tma_load_2d(sw, &tmW, &full_bar[stage], k0, n0);
        tma_load_2d(sw + L::kABytes, &tmX, &full_bar[stage], k0, m0);
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
      if (ncol <= 0) continue;
      float v[4] = {s.x, s.y, s.z, s.w};
      const long long row = m0 + m;
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

template <int NB>
static int launch_few(const void* X, const void* W, FewArgs a, long long ldx, long long ldw, int splits, cudaStream_t stream) {
  CUtensorMap tmW, tmX;
  int e = make_tmap_2d(&tmX, X, a.M, a.K, ldx, NB, BK);
  if (e) return 2000 + e;
  e = make_tmap_2d(&tmW, W, a.N, a.K, ldw, 128, BK);
  if (e) return 3000 + e;
  auto kern = gemm_few_kernel<NB>;
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

extern "C" {

// Launches of this thread that support it overlap with the kernel before them (1) or not (0).  The caller sees to it that no
// kernel of the sequence writes what the one after it reads as weights.
int ob_overlap_launches(int on) {
  overlapped_launches() = on != 0;
  return 0;
}

// C[M,N] (+)= X[M,K] W[N,K]^T (+ bias, residual): contract of ob_gemm_bf16 with K-major operands.
// splits: CTAs per column panel (at most 8, fewer where the reduction has fewer slices; 0 chooses).
int ob_gemm_few(const void* X, const void* W, void* C, const void* residual, int M, int N, int K, long long ldx, long long ldw,
                long long ldc, long long ldr, int out_mode, const void* bias, int splits, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || out_mode < 0 || out_mode > 2) return 6005;
  if ((ldx & 7) || (ldw & 7)) return 6001;
  if ((((uintptr_t)X) & 15) || (((uintptr_t)W) & 15)) return 6002;
  FewArgs a = {};
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

}  // extern "C"
