// CostVolumeV2 forward (MEAN, fused arithmetic), eight channels per lane.
//
// cv2_fwd_tuned gives a lane four channels and caches the footprint along the planes.  At the cascade's depth spacings the
// footprint moves on every second plane or oftener, so what counts is the price of a fetch.  Here a lane fetches 16 bytes of
// bfloat16 per corner (half the loads, addresses and record reads per channel), blends with the four bilinear weights and
// takes the products with the reference pixel at once, in pairs.  There is no cache and no test per plane: where every lane
// sees the block's planes (the usual case) the loads of several planes are in flight together.
// Bound: latency of the gathers behind the unpacking (32 of 128 instructions).  Four views, 576x768x32, C = 16, eight groups:
// 648 -> 571 us (780 -> 602 with planes eight times as far apart).  Eight channels are cv2_vox.cuh's.
//
// Float32 features double the fetch, and with few groups per channel the cached form (a plane costs its GROUPS only) stays
// ahead while the footprint rests (C = 32, eight groups, planes 1 apart: 251 us against 328).  Where it is chosen otherwise:
// v2_wide_fwd.
#pragma once
#include "cv2_vox.cuh"

namespace chop {

template <int C, int SUB>
struct V2Wide {
  static constexpr int LG = C / 8, G = 32 / LG;
  static constexpr int PB = 4;                       // planes per block: at most 32 accumulator registers
  static constexpr int BLOCKS = 5;                   // CTAs per SM
  static constexpr int PL = PB / LG;                 // planes that a lane projects
  // A lane owns whole pixels, so a small image has too few warps even with one block of planes each.  From so many on this is
  // the faster kernel; us here : with four channels per lane, four views (replayed from a graph):
  //   C = 16, 16 / 8       48x60x24 1080 warps 7.6 : 7.0 / 7.3 : 6.4, 64x80x16 1280 8.3 : 10.3 / 7.7 : 9.3
  //   C = 32, 32           48x60x8   720 warps 6.4 : 7.6 (nothing smaller measured)
  static constexpr int MIN_WARPS = 148 * (C == 16 ? 8 : 4);
  static constexpr size_t smem_per_warp = (size_t)PB * G * 16;
};

template <typename T, int C, int SUB>
__global__ void __launch_bounds__(128, V2Wide<C, SUB>::BLOCKS) cv2_fwd_wide(const CvArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef V2Wide<C, SUB> Cf;
  constexpr int LG = Cf::LG, G = Cf::G, PB = Cf::PB, PL = Cf::PL;
  constexpr int NG = 8 / SUB;              // groups per lane
  constexpr int GR = C / SUB;              // groups per voxel
  constexpr int NA = 4;                    // paired accumulators per plane
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int li = lane & (LG - 1);
  const int g = lane / LG;

  const long long item = (long long)blockIdx.x * 4 + wib;
  if (item >= (long long)a.npb * a.nchunks) return;
  const int chunk_id = (int)(item / a.npb);
  const int pb = (int)(item - (long long)chunk_id * a.npb);
  const long long pix0 = (long long)pb * G;
  const bool pvalid = pix0 + g < a.npix;
  const unsigned pix = (unsigned)(pvalid ? pix0 + g : a.npix - 1);
  const int dlo = a.d_begin + chunk_id * a.chunk;
  const int dhi = min(a.d_end, dlo + a.chunk);
  const int N = a.N;
  const int D = a.D;
  float4* rec = reinterpret_cast<float4*>(smem_raw + (size_t)wib * Cf::smem_per_warp) + g;   // [PB][G] {texel, dw, dh, -}

  const unsigned w = pix % (unsigned)a.W, tt = pix / (unsigned)a.W;
  const unsigned h = tt % (unsigned)a.H;
  const int b = (int)(tt / (unsigned)a.H);
  float x = (float)w, y = (float)h;
  if (a.half_centor) {
    x = xadd(x, 0.5f);
    y = xadd(y, 0.5f);
  }
  const T* src_lane = static_cast<const T*>(a.src) + li * 8;
  pk2 ref[4];
  {
    Ch8<T> r;
    r.load(static_cast<const T*>(a.ref) + (size_t)pix * C + li * 8);
#pragma unroll
    for (int k = 0; k < 4; ++k) ref[k] = r.get(k);
  }
  const float* dgrid = static_cast<const float*>(a.depth) + (size_t)pix * D;
  float* out = static_cast<float*>(a.cost) + ((size_t)pix * D + dlo) * GR + li * NG;
  const long long rowc = (long long)a.Ws * C;

  for (int dblk = dlo; dblk < dhi; dblk += PB, out += PB * GR) {
    float depth[PL];
    int used[PL];
#pragma unroll
    for (int p = 0; p < PL; ++p) {
      depth[p] = __ldg(dgrid + min(dblk + p * LG + li, dhi - 1));
      used[p] = 0;
    }
    pk2 acc[PB][NA];
#pragma unroll
    for (int j = 0; j < PB; ++j)
#pragma unroll
      for (int k = 0; k < NA; ++k) acc[j][k] = 0ull;

    for (int n = 0; n < N; ++n) {
      Coef<float> cf;   // recomputed per block and view: the camera loads are warp-uniform hits
      {
        const float* Rm = static_cast<const float*>(a.Rs) + (size_t)(b * N + n) * 9;
        const float* tv = static_cast<const float*>(a.Ts) + (size_t)(b * N + n) * 3;
        cf.zc = xadd(xadd(xmul(__ldg(Rm + 6), x), xmul(__ldg(Rm + 7), y)), __ldg(Rm + 8));
        cf.wc = xadd(xadd(xmul(__ldg(Rm + 0), x), xmul(__ldg(Rm + 1), y)), __ldg(Rm + 2));
        cf.hc = xadd(xadd(xmul(__ldg(Rm + 3), x), xmul(__ldg(Rm + 4), y)), __ldg(Rm + 5));
        cf.t0 = __ldg(tv + 0);
        cf.t1 = __ldg(tv + 1);
        cf.t2 = __ldg(tv + 2);
        cf.row0 = a.Hs * (n + N * b);
      }
      int tex[PL];
      float dw[PL], dh[PL];
      bool all_seen = true;
#pragma unroll
      for (int p = 0; p < PL; ++p) {
        int fh, fw;
        float gh, gw;
        const bool seen = project_rcp<false>(cf, depth[p], a, fh, fw, dh[p], dw[p], gh, gw);
        tex[p] = seen ? (fh - FLOOR_BIAS + cf.row0) * a.Ws + (fw - FLOOR_BIAS) : -1;
        used[p] += seen;
        all_seen &= seen;
      }
      __syncwarp();
#pragma unroll
      for (int p = 0; p < PL; ++p) rec[(p * LG + li) * G] = make_float4(__int_as_float(tex[p]), dw[p], dh[p], 0.0f);
      __syncwarp();
      auto record = [&](int j, int& t, float& fw, float& fh) {
        const float4 r = rec[j * G];
        t = __float_as_int(r.x); fw = r.y; fh = r.z;
      };
      auto plane = [&](int j, int t, float fw, float fh) {
        Ch8<T> x00, x01, x10, x11;
        const T* p = src_lane + (size_t)t * C;
        x00.load(p);
        x01.load(p + C);
        x10.load(p + rowc);
        x11.load(p + rowc + C);
        float w00, w01, w11, w10;
        bilinear_weights_fast(fh, fw, w00, w01, w11, w10);
        const pk2 p00 = pk_make(w00, w00), p01 = pk_make(w01, w01), p10 = pk_make(w10, w10), p11 = pk_make(w11, w11);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const pk2 s = pk_fma(p11, x11.get(k), pk_fma(p10, x10.get(k), pk_fma(p01, x01.get(k), pk_mul(p00, x00.get(k)))));
          acc[j][k] = pk_fma(s, ref[k], acc[j][k]);   // sum_c sample*ref (v2:118-120)
        }
      };
      if (__all_sync(0xffffffffu, all_seen)) {
#pragma unroll
        for (int j = 0; j < PB; ++j) {
          int t;
          float fw, fh;
          record(j, t, fw, fh);
          plane(j, t, fw, fh);
        }
      } else {
#pragma unroll
        for (int j = 0; j < PB; ++j) {
          int t;
          float fw, fh;
          record(j, t, fw, fh);
          if (t >= 0) plane(j, t, fw, fh);
        }
      }
    }

#pragma unroll
    for (int p = 0; p < PL; ++p) {
      const int d = dblk + p * LG + li;
      if (pvalid && d < dhi) __stcs(a.mask + (size_t)pix * D + d, used[p]);
    }
#pragma unroll
    for (int j = 0; j < PB; ++j) {
      const int u = __shfl_sync(0xffffffffu, used[j / LG], g * LG + j % LG);
      const float inv = u > 0 ? 1.0f / (float)u : 0.0f;   // v2:128-133
      float o[NG];
#pragma unroll
      for (int q = 0; q < NA; ++q) {
        float lo, hi;
        pk_split(acc[j][q], lo, hi);
        if constexpr (SUB == 1) {
          o[2 * q] = lo * inv;
          o[2 * q + 1] = hi * inv;
        } else {
          o[q] = (lo + hi) * inv;
        }
      }
      if (pvalid && dblk + j < dhi) store_stream<float, NG>(out + j * GR, o);
    }
  }
}

template <int C, int SUB>
inline int v2_wide_go(const CvArgs& a0, cudaStream_t st) {
  typedef V2Wide<C, SUB> Cf;
  CvArgs a = a0;
  a.npb = (int)((a.npix + Cf::G - 1) / Cf::G);
  const int drange = a.d_end - a.d_begin;
  // by all planes, not those of this call: a depth range takes the kernel that the whole volume takes
  if ((long long)a.npb * ((a.D + Cf::PB - 1) / Cf::PB) < Cf::MIN_WARPS) return -4;
  int chunk = (a.chunk + Cf::PB - 1) / Cf::PB * Cf::PB;
  // a warp has twice the pixels that the caller's plan assumed: shorter chunks until the GPU is filled
  while (chunk > Cf::PB && (long long)a.npb * ((drange + chunk - 1) / chunk) < 148LL * 20 * 2)
    chunk = (chunk / 2 + Cf::PB - 1) / Cf::PB * Cf::PB;
  a.chunk = chunk;
  a.nchunks = (drange + chunk - 1) / chunk;
  const long long items = (long long)a.npb * a.nchunks;
  cv2_fwd_wide<__nv_bfloat16, C, SUB><<<(unsigned)((items + 3) / 4), 128, Cf::smem_per_warp * 4, st>>>(a);
  return (int)cudaGetLastError();
}

// Source views from which on the wide kernel is the faster one.  A view costs it less, a voxel more: a lane owns whole
// pixels, so a warp's stores are 32-byte pieces a cost slab (D * groups floats) apart, and the more planes the wider apart.
// Measured at 1, 2, 3, 4 and 6 views, 8 to 64 planes, depths 1 and 8 apart (the footprint rests / moves), us of this kernel
// against four channels per lane:
//   C = 16, 16 groups: 16 planes, 1 view 173 : 141 / 172 : 158, 2 views 223 : 225 / 227 : 260; 64 planes, 2 views
//                      238 : 195 / 245 : 244, 3 views 283 : 256 / 291 : 322
//   C = 16, 8 groups:  16 planes, 1 view 123 : 121 / 125 : 139; 32 planes, 1 view 74 : 64 / 74 : 71, 2 views 101 : 96 / 106 : 119
//   C = 32, 32 groups: 16 planes, 1 view 215 : 223 / 225 : 279; 64 planes, 1 view 213 : 176 / 217 : 217, 2 views 291 : 266 / 303 : 358
inline int v2_wide_views(int C, int sub, int D) {
  const int n = D <= 8 ? 1 : D <= 16 ? 2 : 3;
  return C == 16 && sub == 1 ? n : n > 1 ? n - 1 : 1;
}

// bfloat16, 16-byte aligned features and cost; -4: not one of the cases
inline int v2_wide_fwd(const CvArgs& a, cudaStream_t st) {
  if (((reinterpret_cast<size_t>(a.ref) | reinterpret_cast<size_t>(a.src) | reinterpret_cast<size_t>(a.cost)) & 15) != 0) return -4;
  const int sub = a.C / a.G;
  if (a.N < v2_wide_views(a.C, sub, a.D)) return -4;
  if (a.C == 16) return sub == 1 ? v2_wide_go<16, 1>(a, st) : sub == 2 ? v2_wide_go<16, 2>(a, st) : -4;
  if (a.C == 32 && sub == 1) return v2_wide_go<32, 1>(a, st);
  return -4;
}

}  // namespace chop
