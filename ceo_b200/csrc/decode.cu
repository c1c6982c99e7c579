// Token-by-token inference: a few rows (the next token of every running sequence, or the
// tokens of a prompt) through the whole model in one host call.
//
// Such a pass moves every weight once (2.4 GB for the 1.3B model) and computes next to nothing,
// so what counts is that memory never idles: the host loop below launches every kernel of the
// pass as a programmatic dependent of the one before it, each GEMM requests its weights while
// its predecessor still runs (skinny.cuh), and the recurrence asks L2 for its states the same
// way.  Only activations wait for the previous kernel.  The chain is safe because the first
// kernel (the embedding gather) is an ordinary launch: everything the stream held before is
// complete, and no kernel of the chain writes a weight.
//
// Per step, layers from Python -> this loop: 1.3B, one sequence, 11.7 -> 0.96 ms; 340M, 40
// sequences, 11.8 -> 0.92 ms; 7B, 7 sequences, 15.9 -> 3.46 ms (4.1 TB/s).
#include "common/ptx.cuh"
#include "common/sigmoid.cuh"
#include "common/util.cuh"
#include "include/ceo_kernels.h"
#include "skinny.cuh"

namespace ceo {

__device__ __forceinline__ void dec_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dec_pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Activations of the chain: the kernel before may still be writing them when this one is already
// resident, so they are no read-only data (`const __restrict__` or __ldg would say so, and such
// loads may move across the wait).  These loads are neither moved nor non-coherent.
__device__ __forceinline__ uint4 ld_act16(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ float ld_act(const bf16* p) {
  uint16_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return __uint_as_float(static_cast<uint32_t>(v) << 16);
}

// ------------------------------------------------------------------- embedding
__global__ void __launch_bounds__(128)
decode_embed_kernel(const long long* __restrict__ ids, const bf16* __restrict__ table,
                    bf16* __restrict__ h, int D, long long vocab) {
  dec_pdl_trigger();
  const long long id = ids[blockIdx.x];
  const uint4* s = reinterpret_cast<const uint4*>(table + id * D);
  uint4* o = reinterpret_cast<uint4*>(h + static_cast<long long>(blockIdx.x) * D);
  const bool ok = id >= 0 && id < vocab;  // out-of-range ids give a zero row
  for (int c = threadIdx.x; c < (D >> 3); c += 128) o[c] = ok ? s[c] : make_uint4(0, 0, 0, 0);
}

// --------------------------------------------------------------------- RMSNorm
constexpr int DN_THREADS = 256;
constexpr int DN_MAXV = 4;  // 8-element vectors per thread: D <= 8192
__global__ void __launch_bounds__(DN_THREADS)
decode_rmsnorm_kernel(const bf16* x, const bf16* __restrict__ w, bf16* y, int D, float eps) {
  __shared__ float red[33];
  const int nv = D >> 3;
  dec_pdl_trigger();
  uint4 wp[DN_MAXV];
#pragma unroll
  for (int i = 0; i < DN_MAXV; ++i) {
    const int c = threadIdx.x + i * DN_THREADS;
    if (c < nv) wp[i] = reinterpret_cast<const uint4*>(w)[c];
  }
  dec_pdl_wait();
  const bf16* xr = x + static_cast<long long>(blockIdx.x) * D;
  uint4 xp[DN_MAXV];
#pragma unroll
  for (int i = 0; i < DN_MAXV; ++i) {
    const int c = threadIdx.x + i * DN_THREADS;
    if (c < nv) xp[i] = ld_act16(xr + c * 8);
  }
  float v[DN_MAXV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < DN_MAXV; ++i) {
    const int c = threadIdx.x + i * DN_THREADS;
    if (c < nv) {
      unpack8(xp[i], v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += v[i][j] * v[i][j];
    }
  }
  ss = block_reduce_sum(ss, red);
  const float rs = rsqrtf(ss / D + eps);
#pragma unroll
  for (int i = 0; i < DN_MAXV; ++i) {
    const int c = threadIdx.x + i * DN_THREADS;
    if (c < nv) {
      float wv[8], o[8];
      unpack8(wp[i], wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = v[i][j] * rs * wv[j];
      reinterpret_cast<uint4*>(y + static_cast<long long>(blockIdx.x) * D)[c] = pack8(o);
    }
  }
}

// ------------------------------------------------------------- delta-rule recurrence
// One CTA per (sequence, head, 32 value columns), walking the T tokens of the call with its
// D x 32 slice of the fp32 state in registers: value columns never meet, so four lanes share a
// column (D / 4 rows each) and two shuffles finish a sum.  One pass over the old state gives
// both S^T k and S^T q; with u = v - S^T k the new read-out is S^T q + alpha (k.q) u, so the
// update itself is off the token's critical path.  q and k are normalised (and rounded to
// bf16, as the chunked path rounds them) for 16 tokens at a time into shared memory.
// Bound by latency at one sequence (64 CTAs for 16 heads of 128) and by the states' traffic,
// 8 D^2 bytes per head and call, from about 8 sequences on.
constexpr int DR_TOK = 16;
template <int D>
__global__ void __launch_bounds__(128)
decode_delta_kernel(const bf16* proj, long long ldp, int P, int H,
                    const float* __restrict__ beta_scalar, int normalize, float* state, bf16* o,
                    int T) {
  constexpr int RT = D / 4;  // state rows per thread
  __shared__ __align__(16) float ks[DR_TOK][D], qs[DR_TOK][D];
  __shared__ float vs[DR_TOK][32], al[DR_TOK], kq[DR_TOK];
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane >> 3, col = blockIdx.x * 32 + warp * 8 + (lane & 7);
  float* sp = state + (static_cast<long long>(bh) * D) * D + col;
  // row i * 4 + j of this thread is state row 16 i + 4 rg + j: the four lanes of a column then
  // read 64 consecutive bytes of k and q
  if ((threadIdx.x & 7) == 0) {
#pragma unroll
    for (int i = 0; i < RT / 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(sp + static_cast<long long>(16 * i + 4 * rg + j) * D));
  }
  dec_pdl_trigger();
  dec_pdl_wait();
  float s[RT];
#pragma unroll
  for (int i = 0; i < RT / 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      s[4 * i + j] = sp[static_cast<long long>(16 * i + 4 * rg + j) * D];
  const int hd = H * D;
  for (int t0 = 0; t0 < T; t0 += DR_TOK) {
    const int nt = T - t0 < DR_TOK ? T - t0 : DR_TOK;
    if (t0) __syncthreads();  // the previous tokens' rows have been read
    for (int t = warp; t < nt; t += 4) {
      const bf16* row = proj + (static_cast<long long>(b) * T + t0 + t) * ldp + h * D;
      constexpr int E = D / 32;
      float qv[E], kv[E], sq = 0.f, sk = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        qv[e] = ld_act(row + lane + 32 * e);
        kv[e] = P == 3 ? ld_act(row + hd + lane + 32 * e) : qv[e];
        sq += qv[e] * qv[e];
        sk += kv[e] * kv[e];
      }
      vs[t][lane] = ld_act(row + (P - 1) * hd + blockIdx.x * 32 + lane);
      const float bl = beta_scalar ? beta_scalar[0] : ld_act(row + P * hd - h * D + h);
      sq = warp_reduce_sum(sq);
      sk = warp_reduce_sum(sk);
      const float iq = normalize ? rsqrtf(sq + 1e-6f) : 1.f;
      const float ik = normalize ? rsqrtf(sk + 1e-6f) : 1.f;
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float qr = __bfloat162float(__float2bfloat16(qv[e] * iq));
        const float kr = __bfloat162float(__float2bfloat16(kv[e] * ik));
        qs[t][lane + 32 * e] = qr;
        ks[t][lane + 32 * e] = kr;
        dot += qr * kr;
      }
      dot = warp_reduce_sum(dot);
      if (lane == 0) {
        const float beta = beta_scalar ? bl : sigmoid_f32(bl);
        al[t] = normalize ? -expm1f(-beta) : efla_coeff(beta, sk);
        kq[t] = dot;
      }
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      float u0 = 0.f, u1 = 0.f, w0 = 0.f, w1 = 0.f;
      float kr[RT];
#pragma unroll
      for (int i = 0; i < RT / 4; ++i) {
        const float4 k4 = *reinterpret_cast<const float4*>(&ks[t][16 * i + 4 * rg]);
        const float4 q4 = *reinterpret_cast<const float4*>(&qs[t][16 * i + 4 * rg]);
        kr[4 * i] = k4.x; kr[4 * i + 1] = k4.y; kr[4 * i + 2] = k4.z; kr[4 * i + 3] = k4.w;
        u0 += s[4 * i] * k4.x + s[4 * i + 1] * k4.y;
        u1 += s[4 * i + 2] * k4.z + s[4 * i + 3] * k4.w;
        w0 += s[4 * i] * q4.x + s[4 * i + 1] * q4.y;
        w1 += s[4 * i + 2] * q4.z + s[4 * i + 3] * q4.w;
      }
      float u = u0 + u1, w = w0 + w1;
      u += __shfl_xor_sync(0xffffffffu, u, 8);
      w += __shfl_xor_sync(0xffffffffu, w, 8);
      u += __shfl_xor_sync(0xffffffffu, u, 16);
      w += __shfl_xor_sync(0xffffffffu, w, 16);
      const float g = al[t] * (vs[t][warp * 8 + (lane & 7)] - u);
#pragma unroll
      for (int i = 0; i < RT; ++i) s[i] += kr[i] * g;
      if (rg == 0)
        o[(static_cast<long long>(b) * T + t0 + t) * hd + h * D + col] =
            __float2bfloat16(w + kq[t] * g);
    }
  }
#pragma unroll
  for (int i = 0; i < RT / 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      sp[static_cast<long long>(16 * i + 4 * rg + j) * D] = s[4 * i + j];
}

template <typename... KA, typename... A>
static cudaError_t launch_pdl(void (*kern)(KA...), dim3 grid, int threads, cudaStream_t stream,
                              A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...);
}

}  // namespace ceo
using namespace ceo;

// Per layer of `layers` (host array of 8 pointers): ln1.weight, w_qkv, w_o, ln2.weight, w_up
// (gate and up rows interleaved), w_down, state (fp32 [B][H][D][D], updated in place), scalar
// beta (fp32, or null: beta logits ride in the projection).
extern "C" int ceo_decode_tokens(const long long* ids, const void* table, long long vocab,
                                 void* const* layers, int n_layers, const void* final_norm,
                                 const void* head, float* logits, void* ws, int B, int T, int hidden,
                                 int H, int D, int P, int n_proj, int F, int normalize, float eps,
                                 int* status, cudaStream_t stream) {
  const int M = B * T, hd = H * D;
  if (B < 1 || T < 1 || M > 128 || (B > 1 && T > 1) || (D != 64 && D != 128) || (hidden & 7) ||
      hidden > 8192 || (P != 2 && P != 3) || (F & 31) || (n_proj & 7) || H < 1 ||
      static_cast<long long>(B) * H > 65535 || (vocab & 3) || n_layers < 1)
    return -5;
  // workspace: h, normed rows, projection, read-out, activation; each part rounded up to 256 bytes
  bf16* h = static_cast<bf16*>(ws);
  bf16* nrm = h + (static_cast<long long>(M) * hidden + 127) / 128 * 128;
  bf16* proj = nrm + (static_cast<long long>(M) * hidden + 127) / 128 * 128;
  bf16* o = proj + (static_cast<long long>(M) * n_proj + 127) / 128 * 128;
  bf16* act = o + (static_cast<long long>(M) * hd + 127) / 128 * 128;
  decode_embed_kernel<<<M, 128, 0, stream>>>(ids, static_cast<const bf16*>(table), h, hidden, vocab);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);
  auto gemm = [&](const void* A, int K, const void* W, int N, int rows, void* C, int f32,
                  const void* res, void* a_out) -> int {
    SkinnyArgs g = {};
    g.A = A; g.W = W; g.C = C; g.residual = res; g.act = a_out;
    g.lda = K; g.ldw = K; g.ldc = N; g.ldr = N; g.ldact = N / 2;
    g.M = rows; g.N = N; g.K = K;
    g.out_f32 = f32;
    g.alpha = 1.f;
    g.w_early = 1;
    g.status = status;
    return skinny_ok(g) ? skinny_gemm(g, stream) : -2;
  };
  for (int l = 0; l < n_layers; ++l) {
    void* const* L = layers + 8 * l;
    int rc;
    e = launch_pdl(decode_rmsnorm_kernel, dim3(M), DN_THREADS, stream, h,
                   static_cast<const bf16*>(L[0]), nrm, hidden, eps);
    if (e != cudaSuccess) return static_cast<int>(e);
    if ((rc = gemm(nrm, hidden, L[1], n_proj, M, proj, 0, nullptr, nullptr))) return rc;
    const dim3 dg(D / 32, B * H);
    if (D == 128)
      e = launch_pdl(decode_delta_kernel<128>, dg, 128, stream, proj,
                     static_cast<long long>(n_proj), P, H, static_cast<const float*>(L[7]),
                     normalize, static_cast<float*>(L[6]), o, T);
    else
      e = launch_pdl(decode_delta_kernel<64>, dg, 128, stream, proj,
                     static_cast<long long>(n_proj), P, H, static_cast<const float*>(L[7]),
                     normalize, static_cast<float*>(L[6]), o, T);
    if (e != cudaSuccess) return static_cast<int>(e);
    if ((rc = gemm(o, hd, L[2], hidden, M, h, 0, h, nullptr))) return rc;
    e = launch_pdl(decode_rmsnorm_kernel, dim3(M), DN_THREADS, stream, h,
                   static_cast<const bf16*>(L[3]), nrm, hidden, eps);
    if (e != cudaSuccess) return static_cast<int>(e);
    if ((rc = gemm(nrm, hidden, L[4], 2 * F, M, nullptr, 0, nullptr, act))) return rc;
    if ((rc = gemm(act, F, L[5], hidden, M, h, 0, h, nullptr))) return rc;
  }
  if (!logits) return 0;
  // the head reads the last token of every sequence (all rows when T = 1)
  const bf16* hl = h + (T > 1 ? static_cast<long long>(T - 1) * hidden : 0);
  e = launch_pdl(decode_rmsnorm_kernel, dim3(B), DN_THREADS, stream, hl,
                 static_cast<const bf16*>(final_norm), nrm, hidden, eps);
  if (e != cudaSuccess) return static_cast<int>(e);
  return gemm(nrm, hidden, head, static_cast<int>(vocab), B, logits, 1, nullptr, nullptr);
}
