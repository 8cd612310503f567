// CostVolumeV2 forward with eight channels: a lane per VOXEL, MEAN (fused arithmetic) and MIN (unfused, exact).
//
// With two lanes per pixel (cv2_fwd_tuned) a footprint was dropped every two planes, and with a lane per pixel and the planes in
// its registers (as in cv2_wide.cuh) every store, depth hypothesis and validity count of a warp lay a cost slab (D * groups floats)
// from the next lane's: 32 lines a request, half of all that the L1 looked up.  Here the lanes of a warp are PB consecutive planes
// of 32/PB neighbouring pixels: stores are whole runs of a slab, the corners of neighbouring pixels and planes share their
// lines, a lane holds one voxel's sums (48 registers, 40 warps an SM) and nothing passes through shared memory.
// Bound: issue (77 % of the slots at 1152x1536x8, bfloat16 MEAN; widening and paired blends) and the L1 behind it (68 % of its data pipe, four
// gathers per voxel and view; a warp waits for them half of the time).  Four views, planes 1 / 8 apart, us before and now:
//   bfloat16 MEAN, 8 groups  1152x1536x8 419 / 425, 364 / 408; 288x384x48 184 / 189, 131 / 134
//   bfloat16 MIN,  8 groups  1152x1536x8 607 / 645, 530 / 515; 288x384x48 213 / 227, 176 / 174
//   float32  MEAN, 8 groups  288x384x48 193 / 212, 144 / 184; 1152x1536x8 561 / 612, 514 / 560; where it is the slower one: v2_vox_fwd
// PB = 4 against 2, bfloat16, 8 groups: 378 / 450 and 400 / 428 at 1152x1536x8, 143 / 146 and 157 / 157 at 288x384x48; 2 groups 335 / 410
// and 336 / 353; float32 at 288x384x64, one view 104 and 135 (eight planes: 774 and 683).  Eight planes of four pixels 383 / 561.
// Two or four voxels per lane (the cameras fetched once for them): 406 / 550, 454 / 631.  With 16 and 32 channels (two and four
// lanes per voxel) the kernels that keep the footprint are faster (288x384x48, C = 16, four groups: 204, 259 us).
#pragma once
#include "cv_fwd.cuh"
#include "cv_packed.cuh"

namespace chop {

// A lane's eight consecutive channels of one texel, widened to pairs on use.  WIDE: 32 bytes in one load where the type has as many
// (two 16-byte loads of a warp's texels touch every line twice), which need addresses that are multiples of 32.
template <typename T, bool WIDE = false>
struct Ch8;
template <bool WIDE>
struct Ch8<__nv_bfloat16, WIDE> {
  uint4 r;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { r = __ldg(reinterpret_cast<const uint4*>(p)); }
  __device__ __forceinline__ unsigned word(int k) const { return k == 0 ? r.x : k == 1 ? r.y : k == 2 ? r.z : r.w; }
  __device__ __forceinline__ float one(int k) const { return __uint_as_float(k & 1 ? word(k / 2) & 0xffff0000u : word(k / 2) << 16); }
  __device__ __forceinline__ pk2 get(int k) const {
    const unsigned w = word(k);
    return pk_make(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
};
template <bool WIDE>
struct Ch8<float, WIDE> {
  pk2 r[4];
  __device__ __forceinline__ void load(const float* p) {
    if constexpr (WIDE) {
      asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r[0]), "=l"(r[1]), "=l"(r[2]), "=l"(r[3]) : "l"(p));
    } else {
      PkLoad<float>::ld(p, r[0], r[1]);
      PkLoad<float>::ld(p + 4, r[2], r[3]);
    }
  }
  __device__ __forceinline__ pk2 get(int k) const { return r[k]; }
  __device__ __forceinline__ float one(int k) const {
    float lo, hi;
    pk_split(r[k / 2], lo, hi);
    return k & 1 ? hi : lo;
  }
};
// acc + lo(a)*lo(b) + hi(a)*hi(b) of two bfloat16 pairs
__device__ __forceinline__ float dot2_bf16(unsigned a, unsigned b, float acc) { return fma_hi_bf16(a, b, fma_lo_bf16(a, b, acc)); }

// PB planes by 32/PB neighbouring pixels per warp: a lane is a voxel.
constexpr int VOX_CTAS = 10;   // 128-thread CTAs per SM, 48 registers
constexpr int VOX_MIN_CTAS = 8;
template <typename T, int SUB, int PB, bool MIN, bool WIDE>
__global__ void __launch_bounds__(128, MIN ? VOX_MIN_CTAS : VOX_CTAS) cv2_fwd_vox(const CvArgs a, const unsigned nitems, const unsigned ndb) {
  constexpr int C = 8, PX = 32 / PB;
  constexpr int NG = C / SUB;                        // groups per voxel
  constexpr int NA = SUB == 4 ? 2 : 4;               // paired accumulators
  constexpr bool DOT = sizeof(T) == 2 && SUB == 4;   // products with the reference before the blend
  const int lane = threadIdx.x & 31, b = blockIdx.y;
  const unsigned item = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= nitems) return;
  const unsigned pg = item / ndb, hw = (unsigned)a.H * a.W;
  const unsigned pu = pg * PX + lane / PB;
  const int du = a.d_begin + (int)(item - pg * ndb) * PB + lane % PB;
  const bool live = pu < hw && du < a.d_end;
  const unsigned p = min(pu, hw - 1), h = p / (unsigned)a.W;
  const int d = min(du, a.d_end - 1), N = a.N;
  float x = (float)(p - h * a.W), y = (float)h;
  if (a.half_centor) {
    x = xadd(x, 0.5f);
    y = xadd(y, 0.5f);
  }
  const size_t pix = (size_t)b * hw + p;
  const float depth = __ldcs(static_cast<const float*>(a.depth) + pix * a.D + d);
  Ch8<T, WIDE> ref;
  ref.load(static_cast<const T*>(a.ref) + pix * C);
  pk2 acc[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) acc[k] = 0ull;
  const T* src = static_cast<const T*>(a.src);
  const long long rowc = (long long)a.Ws * C;
  int used = 0;
  float best[NG];                                    // MIN: the largest group correlation and its view (v2:179-180, :221-224)
  int arg[NG];
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    best[g] = 1.175494351e-38f;
    arg[g] = -1;
  }

  for (int n = 0; n < N; ++n) {
    const float* Rm = static_cast<const float*>(a.Rs) + (size_t)(b * N + n) * 9;   // warp-uniform hits
    const float* tv = static_cast<const float*>(a.Ts) + (size_t)(b * N + n) * 3;
    Coef<float> cf;
    cf.zc = xadd(xadd(xmul(__ldg(Rm + 6), x), xmul(__ldg(Rm + 7), y)), __ldg(Rm + 8));
    cf.wc = xadd(xadd(xmul(__ldg(Rm + 0), x), xmul(__ldg(Rm + 1), y)), __ldg(Rm + 2));
    cf.hc = xadd(xadd(xmul(__ldg(Rm + 3), x), xmul(__ldg(Rm + 4), y)), __ldg(Rm + 5));
    cf.t0 = __ldg(tv + 0);
    cf.t1 = __ldg(tv + 1);
    cf.t2 = __ldg(tv + 2);
    int fh, fw;
    float dh, dw, gh, gw;
    const bool seen = project_rcp<false>(cf, depth, a, fh, fw, dh, dw, gh, gw);
    auto add = [&]() {
      Ch8<T, WIDE> x00, x01, x10, x11;
      const T* q = src + (size_t)((fh - FLOOR_BIAS + a.Hs * (n + N * b)) * a.Ws + (fw - FLOOR_BIAS)) * C;
      x00.load(q);
      x01.load(q + C);
      x10.load(q + rowc);
      x11.load(q + rowc + C);
      float w00, w01, w11, w10;
      if constexpr (MIN) {                           // unfused, in the reference's order: cost and arg index are exact
        bilinear_weights(dh, dw, w00, w01, w11, w10);
        float val[C], gs[NG];
#pragma unroll
        for (int k = 0; k < C; ++k) {
          const float s = xadd(xadd(xadd(xmul(w00, x00.one(k)), xmul(w01, x01.one(k))), xmul(w11, x11.one(k))), xmul(w10, x10.one(k)));
          val[k] = xmul(s, ref.one(k));              // v2:213-216
        }
        in_lane_groups_t<float, C, SUB, true>(val, gs);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          if (best[g] < gs[g]) {                     // the first view wins a tie
            best[g] = gs[g];
            arg[g] = n;
          }
        }
        return;
      }
      bilinear_weights_fast(dh, dw, w00, w01, w11, w10);
      const pk2 p00 = pk_make(w00, w00), p01 = pk_make(w01, w01), p10 = pk_make(w10, w10), p11 = pk_make(w11, w11);
      if constexpr (DOT) {
        auto dots = [&](const Ch8<T, WIDE>& t) {           // both groups' products with the reference pixel
          return pk_make(dot2_bf16(t.word(1), ref.word(1), dot2_bf16(t.word(0), ref.word(0), 0.0f)),
                         dot2_bf16(t.word(3), ref.word(3), dot2_bf16(t.word(2), ref.word(2), 0.0f)));
        };
        acc[0] = pk_fma(p11, dots(x11), pk_fma(p10, dots(x10), pk_fma(p01, dots(x01), pk_fma(p00, dots(x00), acc[0]))));
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const pk2 s = pk_fma(p11, x11.get(k), pk_fma(p10, x10.get(k), pk_fma(p01, x01.get(k), pk_mul(p00, x00.get(k)))));
          const int g = SUB == 4 ? k / 2 : k;
          acc[g] = pk_fma(s, ref.get(k), acc[g]);    // sum_c sample*ref (v2:118-120)
        }
      }
    };
    used += seen;
    if (__all_sync(0xffffffffu, seen)) add();
    else if (seen) add();
  }

  if (!live) return;
  const size_t v = pix * a.D + d;
  if constexpr (MIN) {
    store_stream<float, NG>(static_cast<float*>(a.cost) + v * NG, best);
    store_stream<int, NG>(a.mask + v * NG, arg);
    return;
  }
  __stcs(a.mask + v, used);
  const float inv = used > 0 ? 1.0f / (float)used : 0.0f;   // v2:128-133
  float o[NG];
  if constexpr (DOT) {
    pk_split(acc[0], o[0], o[1]);
    o[0] *= inv;
    o[1] *= inv;
  } else {
#pragma unroll
    for (int g = 0; g < NA; ++g) {
      float lo, hi;
      pk_split(acc[g], lo, hi);
      if constexpr (SUB == 1) {
        o[2 * g] = lo * inv;
        o[2 * g + 1] = hi * inv;
      } else {
        o[g] = (lo + hi) * inv;
      }
    }
  }
  store_stream<float, NG>(static_cast<float*>(a.cost) + v * NG, o);
}

template <typename T, int SUB, int PB, bool MIN, bool WIDE = false>
inline int v2_vox_go(const CvArgs& a, cudaStream_t st) {
  constexpr bool W = WIDE && sizeof(T) == 4;
  if (((reinterpret_cast<size_t>(a.ref) | reinterpret_cast<size_t>(a.src)) & (W ? 31 : 15)) != 0) return -4;
  const int px = 32 / PB, ndb = (a.d_end - a.d_begin + PB - 1) / PB;
  const long long items = ((long long)a.H * a.W + px - 1) / px * ndb;
  if (items >= (1LL << 31) - 4 || a.B > 65535) return -4;
  cv2_fwd_vox<T, SUB, PB, MIN, W><<<dim3((unsigned)((items + 3) / 4), a.B), 128, 0, st>>>(a, (unsigned)items, (unsigned)ndb);
  return (int)cudaGetLastError();
}
// C = 8, aligned features, cost and mask; -4: not one of the cases, or one where two lanes per pixel (cv_tuned.cuh) are the faster kernel.
// us of that kernel against this one, on the inputs of an inference program (smooth depths, cameras around the scene), planes 1 / 8 apart:
//   * Four planes a warp, MEAN and MIN with one channel per group, from 16 planes on where few lanes idle.  576x768x16, float32 MEAN,
//     1 view 108 / 118 : 89 / 110, 4 views 270 / 294 : 212 / 294 (two planes 261 / 276); MIN 301 / 327 : 242 / 303.  1152x1536x8 bfloat16
//     MEAN 421 / 425 : 367 / 409 (two planes, elsewhere measured: 383 / 419).
//   * One channel per group, one view, planes that four do not divide or fewer than 16: float32 MEAN 576x768x18 106 / 114 : 116 / 129,
//     x19 113 / 121 : 136 / 149, 1152x1536x8 234 / 247 : 227 / 263; MIN 576x768x18 129 / 142 : 151 / 162, bfloat16 122 / 130 : 147 / 147.
//   * Two views, the same: MIN 1152x1536x9 403 / 429 : 445 / 475, bfloat16 399 / 413 : 431 / 414; 576x768x18 191 / 207 : 204 / 215, but
//     288x384x50 132 / 139 : 128 / 132.  float32 MEAN 576x768x19 179 / 192 : 187 / 206, 1152x1536x9 376 / 398 : 363 / 407, x18 no difference.
//   * 32-byte loads where they were the faster ones: with four channels per group (288x384x48, 4 views, 8 planes apart 186 -> 176), in MIN
//     with two and four (1152x1536x8 606 -> 506), and with one and two in MEAN where the source features are larger than L2, so that a line
//     fetched twice is the dearer thing: 1152x1536x8, 4 views, 16 bytes 496 / 627, 32 bytes 518 / 561 (two lanes per pixel 563 / 614), two
//     channels per group 457 / 582, 483 / 517 (524 / 577); smaller 288x384x48 144 / 184, 164 / 187; two 164 / 187, 175 / 183.
//     In MIN with one channel per group the 64 registers do not hold their aligned groups (581 -> 686).
// What is left: MEAN and MIN with one channel per group and planes 8 apart lose up to 7 % where they gain as much or more at 1 apart
// (float32, 4 views, MIN 576x768x19 335 / 358 : 310 / 383, MEAN 576x768x32 530 / 583 : 409 / 597).
template <typename T>
inline int v2_vox_fwd(const CvArgs& a, bool min, cudaStream_t st) {
  if (a.C != 8 || ((reinterpret_cast<size_t>(a.cost) | reinterpret_cast<size_t>(a.mask)) & 15) != 0) return -4;
  const int sub = a.C / a.G, nd = a.d_end - a.d_begin;
  const int nd4 = (nd + 3) / 4 * 4;
  if (min) {
    if (sub == 1) {
      if (nd >= 16 && nd == nd4) return v2_vox_go<T, 1, 4, true>(a, st);
      if (a.N == 1 || (a.N == 2 && nd != nd4 && nd < 32)) return -4;
      return nd >= 16 && 16 * nd4 <= 17 * nd ? v2_vox_go<T, 1, 4, true>(a, st) : v2_vox_go<T, 1, 2, true>(a, st);
    }
    return sub == 2 ? v2_vox_go<T, 2, 2, true, true>(a, st) : sub == 4 ? v2_vox_go<T, 4, 2, true, true>(a, st) : -4;
  }
  const bool far = sizeof(T) == 4 && (long long)a.N * a.Hs * a.Ws * 32 > 126LL << 20 &&
                   ((reinterpret_cast<size_t>(a.ref) | reinterpret_cast<size_t>(a.src)) & 31) == 0;
  if (sub == 1) {
    if (nd == nd4 && (sizeof(T) == 2 || nd >= 16)) return v2_vox_go<T, 1, 4, false>(a, st);
    if (sizeof(T) == 4 && (a.N == 1 || (a.N == 2 && nd % 2 != 0))) return -4;
    return far ? v2_vox_go<T, 1, 2, false, true>(a, st) : v2_vox_go<T, 1, 2, false>(a, st);
  }
  if (sub == 2) return far ? v2_vox_go<T, 2, 2, false, true>(a, st) : v2_vox_go<T, 2, 2, false>(a, st);
  return sub == 4 ? v2_vox_go<T, 4, 2, false, true>(a, st) : -4;
}

}  // namespace chop
