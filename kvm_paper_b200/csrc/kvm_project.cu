// Linear layers over few rows (decode tokens, short prompts): y[m, n] = sum_k x[m, k] * w[n, k] for up to 128 rows of x and
// several weight matrices at once.
//
// Bound by reading the weights once (33 MB around a 2048-wide mixer: 5 us at the copy bandwidth) and by launches, so all
// layers that read the same input are one launch, and all of it is in flight at once: a CTA takes 16 weight rows, its
// eight warps an eighth of k each, so that a 2048-wide layer is one resident wave of CTAs whose loads are all issued before
// the first is used.  Warp-level MMAs with the weight rows on M and the input rows on N.  The order of k inside a 32-wide
// slice is permuted alike in both operands (thread t of a quad holds k = 8t .. 8t+7), so that fragments are loaded
// straight from global memory with 16-byte accesses.  Sums: fp32, warps in order, rounded once to bf16.
// More than 64 rows take a second layer of CTAs (the weights then come from L2).  The first loads of the weights are issued
// before the wait for the previous kernel, whose results are only the input rows.
#include "kvm_pdl.cuh"

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
  const int m0 = blockIdx.y * NT * 8;
  const bf16* xp[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xp[n] = a.x + (size_t)min(m0 + n * 8 + g, a.M - 1) * a.x_stride + t * 8;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const int slices = a.K / 32, per = (slices + kProjWarps - 1) / kProjWarps;
  const int s_end = min(slices, (warp + 1) * per);
  constexpr int kAhead = NT <= 2 ? 8 : 4;  // slices whose loads are issued together
  pdl_trigger();
  bool waited = false;
  for (int s0 = warp * per; s0 < s_end; s0 += kAhead) {
    uint4 wl[kAhead], wh[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (s0 + i < s_end) {
        wl[i] = __ldg(reinterpret_cast<const uint4*>(w_lo + (s0 + i) * 32));
        wh[i] = __ldg(reinterpret_cast<const uint4*>(w_hi + (s0 + i) * 32));
      }
    }
    if (!waited) {
      pdl_wait();
      waited = true;
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
  if (!waited) pdl_wait();  // (a warp without a share of k: nothing is written ahead of the previous kernel's end)
  for (int e = tid; e < 16 * min(NT * 8, a.M - m0); e += kProjWarps * 32) {  // consecutive threads: consecutive columns of an output row
    const int r = e & 15, m = e >> 4;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kProjWarps; ++w) s += red[w][r][m];
    if (r0 + r < n_rows) a.out[(size_t)(m0 + m) * a.out_stride + col0 + r0 + r] = __float2bfloat16_rn(s);
  }
}

}  // namespace

cudaError_t launch_project(const ProjectArgs& a, cudaStream_t stream, bool pdl) {
  int ctas = 0;
  for (int i = 0; i < a.n_parts; ++i) ctas += (a.rows[i] + 15) / 16;
  const int nt = a.M <= 8 ? 1 : a.M <= 16 ? 2 : a.M <= 32 ? 4 : 8;
  auto kern = nt == 1 ? kvm_project_kernel<1> : nt == 2 ? kvm_project_kernel<2> : nt == 4 ? kvm_project_kernel<4> : kvm_project_kernel<8>;
  return launch_pdl(kern, dim3(ctas, (a.M + nt * 8 - 1) / (nt * 8)), dim3(kProjWarps * 32), 0, stream, pdl, a);
}

}  // namespace kvm
