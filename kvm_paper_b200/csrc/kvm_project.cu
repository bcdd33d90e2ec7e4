// Linear layers over a handful of rows (decode tokens): y[m, n] = sum_k x[m, k] * w[n, k] for up to 64 rows of x and
// several weight matrices at once.
//
// Bound by reading the weights once (33 MB around a 2048-wide mixer: 5 us at the copy bandwidth) and by launches, so all
// layers that read the same input are one launch, and all of it is in flight at once: a CTA takes 16 weight rows, its
// eight warps an eighth of k each, so that a 2048-wide layer is one resident wave of CTAs whose loads are all issued before
// the first is used.  Warp-level MMAs with the weight rows on M and the input rows on N.  The order of k inside a 32-wide
// slice is permuted alike in both operands (thread t of a quad holds k = 8t .. 8t+7), so that fragments are loaded
// straight from global memory with 16-byte accesses.  Sums: fp32, warps in order, rounded once to bf16.
// Measured, B200, 8 rows x 2048 -> 6256 + 2048 columns: see the table of the design notes.
#include "kvm_common.cuh"

namespace kvm {

namespace {

constexpr int kProjWarps = 8;

// NT: tiles of 8 input rows
template <int NT>
__global__ void __launch_bounds__(kProjWarps * 32)
kvm_project_kernel(const __grid_constant__ ProjectArgs a) {
  __shared__ float red[kProjWarps][16][NT * 8 + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // the CTA's layer and its 16 rows of that layer's weights
  int part = 0, tile = blockIdx.x, col0 = 0;
  while (part + 1 < a.n_parts && tile >= (a.rows[part] + 15) / 16) {
    tile -= (a.rows[part] + 15) / 16;
    col0 += a.rows[part];
    ++part;
  }
  const int n_rows = a.rows[part], r0 = tile * 16;
  const bf16* w_lo = a.weight[part] + (size_t)min(r0 + g, n_rows - 1) * a.K + t * 8;  // rows past the end repeat the last one
  const bf16* w_hi = a.weight[part] + (size_t)min(r0 + g + 8, n_rows - 1) * a.K + t * 8;
  const bf16* xp[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xp[n] = a.x + (size_t)min(n * 8 + g, a.M - 1) * a.x_stride + t * 8;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const int slices = a.K / 32, per = (slices + kProjWarps - 1) / kProjWarps;
  const int s_end = min(slices, (warp + 1) * per);
  constexpr int kAhead = NT <= 2 ? 8 : 4;  // slices whose loads are issued together
  for (int s0 = warp * per; s0 < s_end; s0 += kAhead) {
    uint4 wl[kAhead], wh[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (s0 + i < s_end) {
        wl[i] = __ldcs(reinterpret_cast<const uint4*>(w_lo + (s0 + i) * 32));
        wh[i] = __ldcs(reinterpret_cast<const uint4*>(w_hi + (s0 + i) * 32));
      }
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (s0 + i < s_end) {
        const uint32_t a0[4] = {wl[i].x, wh[i].x, wl[i].y, wh[i].y}, a1[4] = {wl[i].z, wh[i].z, wl[i].w, wh[i].w};
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint4 x = *reinterpret_cast<const uint4*>(xp[n] + (s0 + i) * 32);
          mma_bf16_16816(acc[n], a0, x.x, x.y);
          mma_bf16_16816(acc[n], a1, x.z, x.w);
        }
      }
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    red[warp][g][n * 8 + t * 2] = acc[n][0];
    red[warp][g][n * 8 + t * 2 + 1] = acc[n][1];
    red[warp][g + 8][n * 8 + t * 2] = acc[n][2];
    red[warp][g + 8][n * 8 + t * 2 + 1] = acc[n][3];
  }
  __syncthreads();
  for (int e = tid; e < 16 * a.M; e += kProjWarps * 32) {  // consecutive threads: consecutive columns of one output row
    const int r = e & 15, m = e >> 4;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kProjWarps; ++w) s += red[w][r][m];
    if (r0 + r < n_rows) a.out[(size_t)m * a.out_stride + col0 + r0 + r] = __float2bfloat16_rn(s);
  }
}

}  // namespace

cudaError_t launch_project(const ProjectArgs& a, cudaStream_t stream) {
  int ctas = 0;
  for (int i = 0; i < a.n_parts; ++i) ctas += (a.rows[i] + 15) / 16;
  if (a.M <= 8) kvm_project_kernel<1><<<ctas, kProjWarps * 32, 0, stream>>>(a);
  else if (a.M <= 16) kvm_project_kernel<2><<<ctas, kProjWarps * 32, 0, stream>>>(a);
  else if (a.M <= 32) kvm_project_kernel<4><<<ctas, kProjWarps * 32, 0, stream>>>(a);
  else kvm_project_kernel<8><<<ctas, kProjWarps * 32, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace kvm
