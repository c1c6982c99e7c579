// GEMM for a handful of rows: C[M,N] = A[M,K] W[N,K]^T with M <= 128 (one token per running
// sequence, or the tokens of a prompt).  Such a product reads W once and does next to no
// arithmetic: it is bound by how soon and how evenly W is requested from memory.
//
// * Roles are swapped: 128 rows of W are the M side of tcgen05.mma and the few rows of A its N
//   side (16 / 32 / 64 / 128 columns), so a tile costs 128 x K weights whatever M is.  The
//   128 x 256 tiles of gemm_tcgen05.cu hand a 2048 x 2048 weight to 8 of 148 SMs.
// * K is cut over the CTAs of a cluster (1, 2, 4 or 8): their fp32 partial sums meet in
//   distributed shared memory in rank order, so results do not depend on timing.
// * About 100 KB of shared memory per CTA, so two are resident: the weights of the NEXT launch
//   are requested while this one drains.  With `w_early` (the caller vouches that no kernel of
//   the running chain writes W) the launch is a programmatic dependent one: its weight tiles go
//   into the ring, and the rest of its slice into L2, before griddepcontrol.wait; only A waits.
//
// Alone, one after the other, the 97 products of a 1.3B decode step (2.4 GB of weights, one row)
// take 0.97 ms; chained, with norms and recurrence between them, 0.96 ms (2.5 TB/s).  What bounds
// the chain is the hop between two dependent launches (0.96 ms over 171 of them, 5.6 us), not the
// weights.
// Tried and dropped: normalising A inside this kernel (49 launches fewer, but the hop grows: 40
// rows 0.92 -> 1.28 ms a step) and several blocks of 128 rows (576 x 2048 x 2048 20.5 -> 22.6 us).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace ceo {

constexpr int SK_ROWS = 128;  // rows of W per tile

struct SkinnyArgs {
  const void* A;        // bf16 [M][K], row stride lda
  const void* W;        // bf16 [N][K], row stride ldw
  void* C;              // bf16 or fp32 [M][N], row stride ldc; may be null with `act`
  const void* residual; // bf16 [M][N] or null
  void* act;            // bf16 [M][N/2]: silu(even column) * odd column, or null
  long long lda, ldw, ldc, ldr, ldact;
  int M, N, K;
  int out_f32;
  float alpha;
  int w_early;
  int* status;
};

// True when the kernel takes the shape (the caller keeps its general path otherwise).
bool skinny_ok(const SkinnyArgs& a);
// 0, a negative argument code, or a cudaError_t.
int skinny_gemm(const SkinnyArgs& a, cudaStream_t stream);

}  // namespace ceo
