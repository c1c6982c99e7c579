// Inference over whole sequences (prefill, evaluation): every block's kernels launched from one
// host call.  The kernels are the training path's; what goes is the host's share (about 28 us a
// launch through autograd, 12 launches a layer) and what only a backward pass reads: the
// gate / up tensor, the 64 x 64 inverses, the saved activations of all layers.
#include "common/util.cuh"
#include "include/ceo_kernels.h"

using namespace ceo;

// Per layer of `layers` (host array of 9 pointers): ln1.weight, w_qkv, w_o, ln2.weight, w_up,
// w_down, scalar beta (fp32) or null, s0 (fp32 [B][H][D][D]) or null, s_final.
extern "C" int ceo_forward_tokens(const long long* ids, const void* table, long long vocab,
                                  void* const* layers, int n_layers, const void* final_norm,
                                  void* out, void* ws, long long ws_bytes,
                                  const unsigned char* resets, int B, int T, int hidden, int H,
                                  int D, int P, int n_proj, int F, int normalize, float eps,
                                  int* status, cudaStream_t stream) {
  const long long rows = static_cast<long long>(B) * T;
  if (B < 1 || T < 1 || (T & 63) || rows > 0x7fffffffLL || n_layers < 1 || (P != 2 && P != 3))
    return -5;
  const int M = static_cast<int>(rows), hd = H * D, n = T / 64;
  const int segs = ceo_efla_fwd_segments(B, T, H, D);
  if (segs < 1) return -5;
  const long long states_b = static_cast<long long>(B) * H * n * D * D * 2;
  const long long seg_b = segs > 1 ? 3LL * B * H * segs * D * D * 4 : 0;
  uint8_t* base = static_cast<uint8_t*>(ws);
  long long used = 0;
  auto take = [&](long long bytes) {
    void* p = base + used;
    used += (bytes + 255) / 256 * 256;
    return p;
  };
  void* h = take(rows * hidden * 2);
  void* nrm = take(rows * hidden * 2);
  void* proj = take(rows * n_proj * 2);
  void* qn = take(rows * hd * 2);
  void* kn = P == 3 ? take(rows * hd * 2) : qn;
  float* rq = static_cast<float*>(take(rows * H * 4));
  float* rk = static_cast<float*>(take(rows * H * 4));
  float* alpha = static_cast<float*>(take(rows * H * 4));
  void* w = take(rows * hd * 2);
  void* up = take(rows * hd * 2);
  void* o = take(rows * hd * 2);
  void* states = take(states_b);
  void* act = take(rows * F * 2);
  float* seg_ws = static_cast<float*>(take(seg_b));
  if (used > ws_bytes) return -5;

  int rc = ceo_embedding_fwd(ids, table, h, rows, hidden, vocab, nullptr, stream);
  for (int l = 0; l < n_layers && !rc; ++l) {
    void* const* L = layers + 9 * l;
    if ((rc = ceo_rmsnorm_fwd(h, nullptr, L[0], nrm, nullptr, rq, M, hidden, eps, stream))) break;
    if ((rc = ceo_gemm_bf16(nrm, L[1], proj, M, n_proj, hidden, hidden, hidden, n_proj, 0, 0, 1, 0,
                            0, 0, 0, 0, 1.f, nullptr, nullptr, 0, 0, status, 0, stream)))
      break;
    const uint8_t* pp = static_cast<const uint8_t*>(proj);
    const void* k = P == 3 ? pp + 2LL * hd : pp;
    rc = L[6] ? ceo_efla_prep_fwd(pp, k, static_cast<const float*>(L[6]), 1, qn, kn, rq, rk, alpha,
                                  rows, H, D, n_proj, n_proj, normalize, stream)
              : ceo_efla_prep_fwd_logits(pp, k, pp + 2LL * P * hd, n_proj, nullptr, qn, kn, rq, rk,
                                         alpha, rows, H, D, n_proj, n_proj, normalize, stream);
    if (rc) break;
    if ((rc = ceo_efla_fwd_seg(qn, kn, pp + 2LL * (P - 1) * hd, alpha,
                               static_cast<const float*>(L[7]), w, up, states, nullptr, o,
                               static_cast<float*>(L[8]), resets, segs, seg_ws, B, T, H, D, hd, hd,
                               n_proj, status, stream)))
      break;
    if ((rc = ceo_gemm_bf16(o, L[2], h, M, hidden, hd, hd, hd, hidden, 0, 0, 1, 0, 0, 0, 0, 0, 1.f,
                            nullptr, h, hidden, 0, status, 0, stream)))
      break;
    if ((rc = ceo_rmsnorm_fwd(h, nullptr, L[3], nrm, nullptr, rq, M, hidden, eps, stream))) break;
    if ((rc = ceo_gemm_bf16_swiglu(nrm, L[4], nullptr, M, 2 * F, hidden, hidden, hidden, 2 * F, 0, 0,
                                   1.f, 1, act, F, status, stream)))
      break;
    rc = ceo_gemm_bf16(act, L[5], h, M, hidden, F, F, F, hidden, 0, 0, 1, 0, 0, 0, 0, 0, 1.f,
                       nullptr, h, hidden, 0, status, 0, stream);
  }
  if (!rc) rc = ceo_rmsnorm_fwd(h, nullptr, final_norm, out, nullptr, rq, M, hidden, eps, stream);
  return rc;
}
