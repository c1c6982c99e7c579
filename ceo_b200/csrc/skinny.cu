// See skinny.cuh for the design.  Warp 0 is the TMA producer, warp 1 issues the MMAs, warps
// 2..5 (one TMEM lane quadrant each) move the accumulator to shared memory, where the cluster's
// partial sums are added and written out.
#include <atomic>

#include "common/ptx.cuh"
#include "common/tmap.h"
#include "common/util.cuh"
#include "include/ceo_kernels.h"
#include "skinny.cuh"

namespace ceo {

constexpr int SK_THREADS = 192;
constexpr int SK_BK = 64;
constexpr int SK_W_BYTES = SK_ROWS * SK_BK * 2;  // 16 KB
constexpr int SK_STATUS = 0x534B;

struct SkinnyKernelArgs {
  void* C;
  const bf16* residual;
  bf16* act;
  long long ldc, ldr, ldact;
  int M, N, num_kb;
  int out_f32;
  float alpha;
  int w_early;
  int* status;
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}

template <int NB, int STG>
__global__ void __launch_bounds__(SK_THREADS)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA,
                   const SkinnyKernelArgs p) {
  constexpr int A_BYTES = NB * SK_BK * 2, STAGE = SK_W_BYTES + A_BYTES;
  constexpr uint32_t COLS = NB < 32 ? 32 : NB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STG * STAGE);
  uint64_t* empty = full + STG;
  uint64_t* done = empty + STG;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = static_cast<int>(gridDim.x), rank = static_cast<int>(blockIdx.x);
  const int n0 = static_cast<int>(blockIdx.y) * SK_ROWS;
  const int kb0 = static_cast<int>(static_cast<long long>(rank) * p.num_kb / S);
  const int kb1 = static_cast<int>(static_cast<long long>(rank + 1) * p.num_kb / S);
  const int nkb = kb1 - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STG; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
    // the first weight tiles leave before anything else: nothing below is on their path
    if (p.w_early) {
      const int pre = nkb < STG ? nkb : STG;
      for (int i = 0; i < pre; ++i) {
        mbar_arrive_expect_tx(&full[i], STAGE);
        tma_load_2d(smem + i * STAGE, &tmW, &full[i], (kb0 + i) * SK_BK, n0);
      }
      for (int i = pre; i < nkb; ++i) tma_prefetch_2d(&tmW, (kb0 + i) * SK_BK, n0);
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // every CTA of the grid that follows may become resident now (its TMEM request cannot starve
  // this grid's: the trigger counts once every CTA here has its columns)
  pdl_trigger();
  pdl_wait();

  float* part = reinterpret_cast<float*>(smem);  // [M][128], once the ring is drained
  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        const int s = i % STG;
        if (i >= STG && !mbar_wait(&empty[s], ((i / STG) - 1) & 1)) {
          ok = false;
          break;
        }
        uint8_t* st = smem + s * STAGE;
        if (!p.w_early || i >= STG) {
          mbar_arrive_expect_tx(&full[s], STAGE);
          tma_load_2d(st, &tmW, &full[s], (kb0 + i) * SK_BK, n0);
        }
        tma_load_2d(st + SK_W_BYTES, &tmA, &full[s], (kb0 + i) * SK_BK, 0);
      }
      if (!ok) {
        if (p.status) atomicCAS(p.status, 0, SK_STATUS);
        for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight land first
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(SK_ROWS, NB, 0, 0);
      const uint64_t wd0 = umma_smem_desc(smem_u32(smem), 16, 1024);
      const uint64_t ad0 = umma_smem_desc(smem_u32(smem) + SK_W_BYTES, 16, 1024);
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        const int s = i % STG;
        if (!mbar_wait(&full[s], (i / STG) & 1)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t off = static_cast<uint64_t>(s) * (STAGE >> 4);
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k)
          umma_f16(tmem, wd0 + off + 2 * k, ad0 + off + 2 * k, idesc, (i | k) ? 1u : 0u);
        if (i + STG < nkb) umma_commit(&empty[s]);
      }
      if (ok) umma_commit(done);
      else if (p.status) atomicCAS(p.status, 0, SK_STATUS);
    }
  } else {
    const int quad = warp & 3;
    const bool ok = mbar_wait(done, 0);
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, 0, SK_STATUS);
    tc_fence_after();
    if (ok) {
      // all MMAs have read their operands: the ring becomes the partial-sum tile
#pragma unroll 1
      for (int c = 0; c < static_cast<int>(COLS); c += 32) {
        if (c >= p.M) break;
        uint32_t v[32];
        tmem_ld_32x32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c + j < p.M) part[(c + j) * SK_ROWS + quad * 32 + lane] = __uint_as_float(v[j]);
      }
    }
    tc_fence_before();
  }
  // partial sums of the whole cluster are in place
  __syncwarp();
  if (S > 1) cluster_sync_all();
  else __syncthreads();

  // rank r finishes columns [r * 128 / S, (r + 1) * 128 / S) of the tile, four at a time
  const int qpr = SK_ROWS / 4 / S;  // quads per row of this rank
  const uint32_t part_addr = smem_u32(part);
  for (int q = threadIdx.x; q < qpr * p.M; q += SK_THREADS) {
    const int m = q / qpr, nl = rank * (SK_ROWS / S) + (q - m * qpr) * 4;
    const int n = n0 + nl;
    if (n >= p.N) continue;
    const uint32_t off = part_addr + (m * SK_ROWS + nl) * 4;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < S; ++r) {
      const float4 x = ld_cluster_f4(off, r);
      f.x += x.x; f.y += x.y; f.z += x.z; f.w += x.w;
    }
    f.x *= p.alpha; f.y *= p.alpha; f.z *= p.alpha; f.w *= p.alpha;
    if (p.residual) {
      const uint2 u = *reinterpret_cast<const uint2*>(p.residual + m * p.ldr + n);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(&u.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const bf162*>(&u.y));
      f.x += a.x; f.y += a.y; f.z += b.x; f.w += b.y;
    }
    if (p.act) {
      const float a0 = f.x / (1.f + __expf(-f.x)) * f.y;
      const float a1 = f.z / (1.f + __expf(-f.z)) * f.w;
      *reinterpret_cast<bf162*>(p.act + m * p.ldact + (n >> 1)) = __floats2bfloat162_rn(a0, a1);
    }
    if (p.C) {
      if (p.out_f32) {
        *reinterpret_cast<float4*>(static_cast<float*>(p.C) + m * p.ldc + n) = f;
      } else {
        uint2 o;
        *reinterpret_cast<bf162*>(&o.x) = __floats2bfloat162_rn(f.x, f.y);
        *reinterpret_cast<bf162*>(&o.y) = __floats2bfloat162_rn(f.z, f.w);
        *reinterpret_cast<uint2*>(static_cast<bf16*>(p.C) + m * p.ldc + n) = o;
      }
    }
  }
  // the loop above leaves its lanes at different times, and both the cluster barrier and the
  // TMEM release below are warp-aligned instructions
  __syncwarp();
  // no CTA leaves while another one may still read its partial sums
  if (S > 1) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, COLS);
  }
}

template <int NB, int STG>
static cudaError_t skinny_launch(const CUtensorMap& tw, const CUtensorMap& ta,
                                 const SkinnyKernelArgs& p, int S, int tiles, cudaStream_t stream) {
  constexpr int SMEM = STG * (SK_W_BYTES + NB * SK_BK * 2) + 1024 + 256;
  static_assert(STG * (SK_W_BYTES + NB * SK_BK * 2) >= NB * SK_ROWS * 4, "partial sums fit the ring");
  int dev = 0;
  cudaError_t e0 = cudaGetDevice(&dev);
  if (e0 != cudaSuccess) return e0;
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev >= 64 || !(configured.load(std::memory_order_relaxed) & bit)) {
    e0 = cudaFuncSetAttribute(skinny_gemm_kernel<NB, STG>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e0 != cudaSuccess) return e0;
    configured.fetch_or(bit, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S, tiles, 1);
  cfg.blockDim = dim3(SK_THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  int na = 0;
  at[na].id = cudaLaunchAttributeClusterDimension;
  at[na].val.clusterDim.x = S;
  at[na].val.clusterDim.y = 1;
  at[na].val.clusterDim.z = 1;
  ++na;
  if (p.w_early) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, skinny_gemm_kernel<NB, STG>, tw, ta, p);
}

bool skinny_ok(const SkinnyArgs& a) {
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.A) | reinterpret_cast<uintptr_t>(a.W);
  if (a.M < 1 || a.M > 128 || (al & 15) || (a.lda & 7) || (a.ldw & 7) || a.lda < a.K ||
      a.ldw < a.K || (a.N & 3))
    return false;
  if (a.C && ((reinterpret_cast<uintptr_t>(a.C) & (a.out_f32 ? 15 : 7)) || (a.ldc & 3))) return false;
  if (a.residual && ((reinterpret_cast<uintptr_t>(a.residual) & 7) || (a.ldr & 3))) return false;
  if (a.act && ((reinterpret_cast<uintptr_t>(a.act) & 3) || (a.ldact & 1))) return false;
  return (a.N + SK_ROWS - 1) / SK_ROWS <= 65535;
}

int skinny_gemm(const SkinnyArgs& a, cudaStream_t stream) {
  const int nb = a.M <= 16 ? 16 : a.M <= 32 ? 32 : a.M <= 64 ? 64 : 128;
  CUtensorMap tw, ta;
  if (encode_tmap_2d_bf16(&ta, a.A, a.K, a.M, a.lda, nb)) return -3;
  if (encode_tmap_2d_bf16(&tw, a.W, a.K, a.N, a.ldw, SK_ROWS)) return -4;
  SkinnyKernelArgs p;
  p.C = a.C;
  p.residual = static_cast<const bf16*>(a.residual);
  p.act = static_cast<bf16*>(a.act);
  p.ldc = a.ldc;
  p.ldr = a.ldr;
  p.ldact = a.ldact;
  p.M = a.M;
  p.N = a.N;
  p.num_kb = (a.K + SK_BK - 1) / SK_BK;
  p.out_f32 = a.out_f32;
  p.alpha = a.alpha;
  p.w_early = a.w_early;
  p.status = a.status;
  const int tiles = (a.N + SK_ROWS - 1) / SK_ROWS;
  // the deepest cut of K that still fits two CTAs per SM (296) and leaves each two k-blocks:
  // every SM then has weights in flight, and no second wave starts
  int S = 1;
  while (S < 8 && tiles * S * 2 <= 296 && p.num_kb / (S * 2) >= 2) S *= 2;
  cudaError_t e;
  if (nb == 16) e = skinny_launch<16, 6>(tw, ta, p, S, tiles, stream);
  else if (nb == 32) e = skinny_launch<32, 5>(tw, ta, p, S, tiles, stream);
  else if (nb == 64) e = skinny_launch<64, 4>(tw, ta, p, S, tiles, stream);
  else e = skinny_launch<128, 3>(tw, ta, p, S, tiles, stream);
  return static_cast<int>(e);
}

}  // namespace ceo

// See ceo_set_wait_limit.
extern "C" int ceo_skinny_set_wait_limit(unsigned int iterations) {
  return ceo::set_wait_limit_override(iterations);
}
