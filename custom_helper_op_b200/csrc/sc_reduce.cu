// Sum of the per-CTA partial filter gradients ("slabs") of the manifold convolution, in a fixed order (deterministic).
#include "sc_entry.h"

namespace chop {
namespace {

// A block owns 32 consecutive elements; its warps each add every RED_WARPS-th slab with coalesced 128-byte reads, four in
// flight, then the warp sums are added in warp order.  The slabs are tens of KB apart, so every load is a separate L2 / DRAM
// access: 592 slabs of 16x16 channels take 5.2 us (9 us with 8 warps a block, 35 us with one thread per element).
constexpr int RED_WARPS = 32;

// Slab element [tap][k][n] goes to filter_grad[tap][k][n] (TR: to filter_grad[taps-1-tap][n][k], the transposed
// convolution's order); element taps*KC*NC is the default-value gradient (null: not wanted).
template <bool TR>
__global__ void __launch_bounds__(32 * RED_WARPS) slab_reduce(const float* part, int nparts, int taps, int KC, int NC,
                                                              float* filter_grad, float* default_grad) {
  __shared__ float sm[RED_WARPS][32];
  const long long n_el = (long long)taps * KC * NC;
  const size_t stride = (size_t)n_el + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long e = (long long)blockIdx.x * 32 + lane;
  float s = 0.f;
  if (e <= n_el) {
    const float* col = part + e;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    int p = warp;
    for (; p + 3 * RED_WARPS < nparts; p += 4 * RED_WARPS) {
      const float a0 = col[(size_t)p * stride], a1 = col[(size_t)(p + RED_WARPS) * stride],
                  a2 = col[(size_t)(p + 2 * RED_WARPS) * stride], a3 = col[(size_t)(p + 3 * RED_WARPS) * stride];
      s0 += a0; s1 += a1; s2 += a2; s3 += a3;
    }
    for (; p < nparts; p += RED_WARPS) s0 += col[(size_t)p * stride];
    s = (s0 + s1) + (s2 + s3);
  }
  sm[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e <= n_el) {
    float t = sm[0][lane];
#pragma unroll
    for (int w = 1; w < RED_WARPS; ++w) t += sm[w][lane];
    if (e == n_el) {
      if (default_grad) *default_grad = t;
    } else if (!TR) {
      filter_grad[e] = t;
    } else {
      const int n = (int)(e % NC), k = (int)((e / NC) % KC), tap = (int)(e / ((long long)NC * KC));
      filter_grad[((long long)(taps - 1 - tap) * NC + n) * KC + k] = t;
    }
  }
}

}  // namespace

int sc_slab_reduce(const float* part, int nparts, int taps, int KC, int NC, bool transposed, float* filter_grad,
                   float* default_grad, cudaStream_t st) {
  const unsigned blocks = (unsigned)(((long long)taps * KC * NC + 1 + 31) / 32);
  if (transposed)
    slab_reduce<true><<<blocks, 32 * RED_WARPS, 0, st>>>(part, nparts, taps, KC, NC, filter_grad, default_grad);
  else
    slab_reduce<false><<<blocks, 32 * RED_WARPS, 0, st>>>(part, nparts, taps, KC, NC, filter_grad, default_grad);
  return (int)cudaGetLastError();
}

}  // namespace chop
