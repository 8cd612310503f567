// CostVolumeV2 forward with eight channels: a lane per VOXEL, MEAN (fused arithmetic) and MIN (unfused, exact).
//
// With two lanes per pixel (cv2_fwd_tuned) a footprint was dropped every two planes, and with a lane per pixel and the planes in
// its registers (as in cv2_wide.cuh) every store, depth hypothesis and validity count of a warp lay a cost slab (D * groups floats)
// from the next lane's: 32 lines a request, half of all that the L1 looked up.  Here the lanes of a warp are PB consecutive planes
// of 32/PB neighbouring pixels: stores are whole runs of a slab, the corners of neighbouring pixels and planes share their
// lines, a lane holds one voxel's sums (48 registers, 40 warps an SM) and nothing passes through shared memory.
// Bound: L1 (gather) and the widening.  Four views, planes 1 / 8 apart, us before and now:
//   bfloat16 MEAN, 8 groups  1152x1536x8 437 / 442, 371 / 447; 288x384x48 193 / 198, 138 / 144; 2 groups 385 / 407, 332 / 352; 166 / 176, 127 / 131
//   bfloat16 MIN,  8 groups  1152x1536x8 632 / 662, 527 / 529; 2 groups 554 / 582, 403 / 404
//   float32  MEAN, 8 groups  288x384x48 205 / 223, 158 / 207; 1152x1536x8 569 / 613, 516 / 610; where it is the slower one: v2_vox_fwd
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
// 32-byte loads: everywhere but in MIN with one channel per group, whose 64 registers do not hold their aligned groups (1152x1536x8, four
// views, planes 1 / 8 apart: 581 / 717 us without, 686 / 790 with)
template <int SUB, bool MIN>
constexpr bool VOX_WIDE = !(MIN && SUB == 1);

template <typename T, int SUB, int PB, bool MIN>
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
  constexpr bool WIDE = VOX_WIDE<SUB, MIN>;
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

template <typename T, int SUB, int PB, bool MIN>
inline int v2_vox_go(const CvArgs& a, cudaStream_t st) {
  const int px = 32 / PB, ndb = (a.d_end - a.d_begin + PB - 1) / PB;
  const long long items = ((long long)a.H * a.W + px - 1) / px * ndb;
  if (items >= (1LL << 31) - 4 || a.B > 65535) return -4;
  cv2_fwd_vox<T, SUB, PB, MIN><<<dim3((unsigned)((items + 3) / 4), a.B), 128, 0, st>>>(a, (unsigned)items, (unsigned)ndb);
  return (int)cudaGetLastError();
}
// C = 8, aligned features (float32 MEAN, and MIN with two or four channels per group: to 32 bytes), cost and mask; -4: not one of the cases.
// us at 1152x1536x8 / 576x768x16 (12 where noted), planes 1, 3 and 8 apart, kernels before (two lanes per pixel) against this one:
//   float32 MEAN 8 groups, 1 view  225 229 239 : 239 237 243 / 108 110 116 : 98 98 102 (12: 83 84 88 : 90 90 93)
//                          4 views 569 591 613 : 516 548 610 / 273 284 296 : 262 266 296 with two planes, 237 258 317 with four
//                2 groups, 4 views 494 516 539 : 440 468 514 / 247 258 273 : 225 233 261 (16-byte loads 446 504 594 / 229 243 286)
//   float32 MIN  8 groups, 1 view  274 281 291 : 300 306 321 / 133 135 141 : 120 119 124; 4 views 629 654 680 : 581 639 717 / 305 315 329 : 241 268 360
//   bfloat16 MEAN 8 groups, 4 views 426 428 428 : 364 399 463 with four planes, 383 391 419 with two / 221 224 224 : 177 181 217, 190 192 204
//   bfloat16 MIN 8 groups, 1 view  261 265 273 : 294 286 280 / 123 125 129 : 123 120 118 (12: 100 101 104 : 108 106 107)
// How far a plane moves a footprint is not known here: four planes where they lie close by in most uses of so many planes and views.
template <typename T>
inline int v2_vox_fwd(const CvArgs& a, bool min, cudaStream_t st) {
  const int sub = a.C / a.G;
  const size_t feat = sizeof(T) == 4 && !(min && sub == 1) ? 31 : 15;
  if (a.C != 8 || ((reinterpret_cast<size_t>(a.ref) | reinterpret_cast<size_t>(a.src)) & feat) != 0 ||
      ((reinterpret_cast<size_t>(a.cost) | reinterpret_cast<size_t>(a.mask)) & 15) != 0)
    return -4;
  const int nd = a.d_end - a.d_begin;
  if (min) {
    if (sub == 1) return nd >= 16 ? v2_vox_go<T, 1, 4, true>(a, st) : a.N > 1 ? v2_vox_go<T, 1, 2, true>(a, st) : -4;
    return sub == 2 ? v2_vox_go<T, 2, 2, true>(a, st) : sub == 4 ? v2_vox_go<T, 4, 2, true>(a, st) : -4;
  }
  if (sub == 1) {
    const bool four = sizeof(T) == 2 || (nd >= 16 && (a.N <= 2 || nd >= 32));
    if (nd % 4 == 0 && four) return v2_vox_go<T, 1, 4, false>(a, st);
    return sizeof(T) == 2 || a.N > 1 ? v2_vox_go<T, 1, 2, false>(a, st) : -4;
  }
  return sub == 2 ? v2_vox_go<T, 2, 2, false>(a, st) : sub == 4 ? v2_vox_go<T, 4, 2, false>(a, st) : -4;
}

}  // namespace chop
