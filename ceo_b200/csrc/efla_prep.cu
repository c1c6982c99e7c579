// q / k normalisation, the coefficient alpha and the sigmoid of the beta logits around the EFLA
// kernels (efla.cu), forward and backward.  Bound by memory.
//
// A unit of its own because its sigmoid must be CUDA's accurate one (common/sigmoid.cuh): a beta
// that differs in its last bit from sigmoid() in fp32 moves a bf16 rounding somewhere in the
// first layer, and after 24 layers of the 1.3B model a gradient by 1 % (256 tokens).  The accurate
// exponential costs nothing here: one lane of eight or sixteen evaluates it, between two loads.
#include "common/sigmoid.cuh"
#include "common/util.cuh"
#include "include/ceo_kernels.h"

namespace ceo {

// D / 8 lanes share one (token, head) row, eight elements (one 16-byte access) each, so a
// warp covers 32 / (D / 8) rows at a time.
template <int LPR>
__device__ __forceinline__ float group_reduce_sum(float v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// A warp takes U * RPW consecutive (token, head) rows per iteration and requests all of their
// 16-byte pieces before it uses any (2 U loads in flight per lane forward, 4 U backward): with
// one row group in flight per warp these kernels ran at half the memory bandwidth.
// rows * H < 2^31 (checked on the host), so row ids divide as 32-bit integers.
template <int D>
__global__ void __launch_bounds__(256)
efla_prep_fwd_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k,
                     const float* __restrict__ beta, int beta_scalar, bf16* __restrict__ qn,
                     bf16* __restrict__ kn, float* __restrict__ rq, float* __restrict__ rk,
                     float* __restrict__ alpha, long long rows, int H, long long qs, long long ks,
                     int normalize, const bf16* __restrict__ logits, long long ls,
                     float* __restrict__ beta_out) {
  constexpr int LPR = D / 8, RPW = 32 / LPR, U = 4;
  const int lane = threadIdx.x & 31, sub = lane % LPR, rw = lane / LPR;
  const unsigned wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned nw = (gridDim.x * blockDim.x) >> 5;
  const unsigned total = static_cast<unsigned>(rows * H);
  for (unsigned id0 = wid * (RPW * U); id0 < total; id0 += nw * (RPW * U)) {
    uint4 qp[U], kp[U];
    float bl[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned id = id0 + u * RPW + rw;
      const unsigned idc = id < total ? id : 0;
      const unsigned tok = idc / static_cast<unsigned>(H), h = idc - tok * H;
      bl[u] = logits ? __bfloat162float(logits[tok * ls + h]) : beta_scalar ? beta[0] : beta[idc];
      qp[u] = *reinterpret_cast<const uint4*>(q + tok * qs + h * D + sub * 8);
      kp[u] = *reinterpret_cast<const uint4*>(k + tok * ks + h * D + sub * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned id = id0 + u * RPW + rw;
      float qv[8], kv[8];
      unpack8(qp[u], qv);
      unpack8(kp[u], kv);
      float sq = 0.f, sk = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        sq += qv[e] * qv[e];
        sk += kv[e] * kv[e];
      }
      sq = group_reduce_sum<LPR>(sq);
      sk = group_reduce_sum<LPR>(sk);
      const float iq = normalize ? rsqrtf(sq + 1e-6f) : 1.f;
      const float ik = normalize ? rsqrtf(sk + 1e-6f) : 1.f;
      if (id >= total) continue;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        qv[e] *= iq;
        kv[e] *= ik;
      }
      *reinterpret_cast<uint4*>(qn + static_cast<long long>(id) * D + sub * 8) = pack8(qv);
      *reinterpret_cast<uint4*>(kn + static_cast<long long>(id) * D + sub * 8) = pack8(kv);
      if (sub == 0) {
        float b = bl[u];
        if (logits) {
          b = sigmoid_f32(b);
          if (beta_out) beta_out[id] = b;
        }
        rq[id] = iq;
        rk[id] = ik;
        alpha[id] = normalize ? -expm1f(-b) : efla_coeff(b, sk);
      }
    }
  }
}

// dq = iq (dqn - qn (qn.dqn)),  same for k (normalize); d(beta) = d(alpha) * exp(-beta*lam);
// without normalisation dk += d(alpha) * dc/dlam * 2k.
template <int D>
__global__ void __launch_bounds__(256)
efla_prep_bwd_kernel(const bf16* __restrict__ dqn, const bf16* __restrict__ dkn,
                     const bf16* __restrict__ qn, const bf16* __restrict__ kn,
                     const float* __restrict__ rq, const float* __restrict__ rk,
                     const float* __restrict__ beta, int beta_scalar,
                     const float* __restrict__ dalpha, bf16* __restrict__ dq,
                     bf16* __restrict__ dk, float* __restrict__ dbeta, long long rows, int H,
                     long long dqs, long long dks, int normalize, bf16* __restrict__ dlogits,
                     long long dls, int pad) {
  constexpr int LPR = D / 8, RPW = 32 / LPR, U = 2;
  const int lane = threadIdx.x & 31, sub = lane % LPR, rw = lane / LPR;
  const unsigned wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned nw = (gridDim.x * blockDim.x) >> 5;
  const unsigned total = static_cast<unsigned>(rows * H);
  for (unsigned id0 = wid * (RPW * U); id0 < total; id0 += nw * (RPW * U)) {
    uint4 qp[U], kp[U], gqp[U], gkp[U];
    float bb[U], daa[U], iqq[U], ikk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned id = id0 + u * RPW + rw;
      const unsigned idc = id < total ? id : 0;
      const long long o = static_cast<long long>(idc) * D + sub * 8;
      qp[u] = *reinterpret_cast<const uint4*>(qn + o);
      kp[u] = *reinterpret_cast<const uint4*>(kn + o);
      gqp[u] = *reinterpret_cast<const uint4*>(dqn + o);
      gkp[u] = *reinterpret_cast<const uint4*>(dkn + o);
      bb[u] = beta_scalar ? beta[0] : beta[idc];
      daa[u] = dalpha[idc];
      iqq[u] = rq[idc];
      ikk[u] = rk[idc];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned id = id0 + u * RPW + rw;
      float qv[8], kv[8], gq[8], gk[8];
      unpack8(qp[u], qv);
      unpack8(kp[u], kv);
      unpack8(gqp[u], gq);
      unpack8(gkp[u], gk);
      float dq_dot = 0.f, dk_dot = 0.f, sk = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        dq_dot += qv[e] * gq[e];
        dk_dot += kv[e] * gk[e];
        sk += kv[e] * kv[e];
      }
      dq_dot = group_reduce_sum<LPR>(dq_dot);
      dk_dot = group_reduce_sum<LPR>(dk_dot);
      sk = group_reduce_sum<LPR>(sk);
      if (id >= total) continue;
      const float b = bb[u], da = daa[u];
      float kcoef = 0.f, db;
      if (normalize) {
        db = da * __expf(-b);
      } else {
        const float lam = sk;
        const float ex = __expf(-b * lam);
        db = da * ex;
        float dcdl;
        if (lam <= 1e-6f) dcdl = -0.5f * b * b + b * b * b * lam * (1.f / 3.f);
        else dcdl = (b * lam * ex + expm1f(-b * lam)) / (lam * lam);
        kcoef = 2.f * da * dcdl;
      }
      const float iq = iqq[u], ik = ikk[u];
      float oq[8], ok[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (normalize) {
          oq[e] = iq * (gq[e] - qv[e] * dq_dot);
          ok[e] = ik * (gk[e] - kv[e] * dk_dot);
        } else {
          oq[e] = gq[e];
          ok[e] = gk[e] + kcoef * kv[e];
        }
      }
      const unsigned tok = id / static_cast<unsigned>(H), h = id - tok * H;
      *reinterpret_cast<uint4*>(dq + tok * dqs + h * D + sub * 8) = pack8(oq);
      *reinterpret_cast<uint4*>(dk + tok * dks + h * D + sub * 8) = pack8(ok);
      if (dlogits) {
        // beta = sigmoid(logit); the projection's padding columns get a zero gradient
        if (sub == 0) dlogits[tok * dls + h] = __float2bfloat16(db * b * (1.f - b));
        if (h == H - 1)
          for (int c = sub; c < pad; c += LPR) dlogits[tok * dls + H + c] = __float2bfloat16(0.f);
      } else if (sub == 0) {
        dbeta[id] = db;
      }
    }
  }
}

}  // namespace ceo
using namespace ceo;

static int prep_fwd_run(const void* q, const void* k, const float* beta, int beta_scalar, void* qn,
                        void* kn, float* rq, float* rk, float* alpha, long long rows, int H, int D,
                        long long q_stride, long long k_stride, int normalize, const void* logits,
                        long long logit_stride, float* beta_out, cudaStream_t stream) {
  if (rows <= 0 || H <= 0 || (D != 64 && D != 128) || rows * H >= (1LL << 31)) return -5;
  if (((q_stride | k_stride) & 7) ||
      ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
        reinterpret_cast<uintptr_t>(qn) | reinterpret_cast<uintptr_t>(kn)) & 15))
    return -2;  // rows move as 16-byte accesses
  const int grid = grid_for(rows * H, 8 * 4 * (D == 64 ? 4 : 2), 148 * 4);  // one resident wave
  auto kern = D == 64 ? efla_prep_fwd_kernel<64> : efla_prep_fwd_kernel<128>;
  kern<<<grid, 256, 0, stream>>>(static_cast<const bf16*>(q), static_cast<const bf16*>(k), beta,
                                 beta_scalar, static_cast<bf16*>(qn), static_cast<bf16*>(kn), rq,
                                 rk, alpha, rows, H, q_stride, k_stride, normalize,
                                 static_cast<const bf16*>(logits), logit_stride, beta_out);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int ceo_efla_prep_fwd(const void* q, const void* k, const float* beta, int beta_scalar,
                                 void* qn, void* kn, float* rq, float* rk, float* alpha,
                                 long long rows, int H, int D, long long q_stride,
                                 long long k_stride, int normalize, cudaStream_t stream) {
  return prep_fwd_run(q, k, beta, beta_scalar, qn, kn, rq, rk, alpha, rows, H, D, q_stride,
                      k_stride, normalize, nullptr, 0, nullptr, stream);
}

extern "C" int ceo_efla_prep_fwd_logits(const void* q, const void* k, const void* logits,
                                        long long logit_stride, float* beta, void* qn, void* kn,
                                        float* rq, float* rk, float* alpha, long long rows, int H,
                                        int D, long long q_stride, long long k_stride,
                                        int normalize, cudaStream_t stream) {
  if (!logits) return -5;
  return prep_fwd_run(q, k, nullptr, 0, qn, kn, rq, rk, alpha, rows, H, D, q_stride, k_stride,
                      normalize, logits, logit_stride, beta, stream);
}

static int prep_bwd_run(const void* dqn, const void* dkn, const void* qn, const void* kn,
                        const float* rq, const float* rk, const float* beta, int beta_scalar,
                        const float* dalpha, void* dq, void* dk, float* dbeta, long long rows,
                        int H, int D, long long dq_stride, long long dk_stride, int normalize,
                        void* dlogits, long long dlogit_stride, int pad, cudaStream_t stream) {
  if (rows <= 0 || H <= 0 || (D != 64 && D != 128) || rows * H >= (1LL << 31)) return -5;
  if (((dq_stride | dk_stride) & 7) ||
      ((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) |
        reinterpret_cast<uintptr_t>(dqn) | reinterpret_cast<uintptr_t>(dkn) |
        reinterpret_cast<uintptr_t>(qn) | reinterpret_cast<uintptr_t>(kn)) & 15))
    return -2;  // rows move as 16-byte accesses
  const int grid = grid_for(rows * H, 8 * 2 * (D == 64 ? 4 : 2), 148 * 3);  // one resident wave
  auto kern = D == 64 ? efla_prep_bwd_kernel<64> : efla_prep_bwd_kernel<128>;
  kern<<<grid, 256, 0, stream>>>(static_cast<const bf16*>(dqn), static_cast<const bf16*>(dkn),
                                 static_cast<const bf16*>(qn), static_cast<const bf16*>(kn), rq, rk,
                                 beta, beta_scalar, dalpha, static_cast<bf16*>(dq),
                                 static_cast<bf16*>(dk), dbeta, rows, H, dq_stride, dk_stride,
                                 normalize, static_cast<bf16*>(dlogits), dlogit_stride, pad);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int ceo_efla_prep_bwd(const void* dqn, const void* dkn, const void* qn, const void* kn,
                                 const float* rq, const float* rk, const float* beta,
                                 int beta_scalar, const float* dalpha, void* dq, void* dk,
                                 float* dbeta, long long rows, int H, int D, long long dq_stride,
                                 long long dk_stride, int normalize, cudaStream_t stream) {
  return prep_bwd_run(dqn, dkn, qn, kn, rq, rk, beta, beta_scalar, dalpha, dq, dk, dbeta, rows, H,
                      D, dq_stride, dk_stride, normalize, nullptr, 0, 0, stream);
}

extern "C" int ceo_efla_prep_bwd_logits(const void* dqn, const void* dkn, const void* qn,
                                        const void* kn, const float* rq, const float* rk,
                                        const float* beta, const float* dalpha, void* dq, void* dk,
                                        void* dlogits, long long dlogit_stride, int pad,
                                        long long rows, int H, int D, long long dq_stride,
                                        long long dk_stride, int normalize, cudaStream_t stream) {
  if (!dlogits || pad < 0 || dlogit_stride < H + pad) return -5;
  return prep_bwd_run(dqn, dkn, qn, kn, rq, rk, beta, 0, dalpha, dq, dk, nullptr, rows, H, D,
                      dq_stride, dk_stride, normalize, dlogits, dlogit_stride, pad, stream);
}
