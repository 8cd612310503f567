// Register-tiled CUDA-core manifold convolution for float32 data (the reference's own dtype) and for bfloat16 storage
// with float32 accumulation where the tensor-core kernels do not apply (8 channels, other filter sizes, dilation):
// forward, gather-form image gradient, transposed forward and filter gradient, any filter size / stride / dilation,
// 8, 16 or 32 channels on either side.
//
// The shape-agnostic one-thread-per-output-element kernels of sc_simt.cu remain the fallback (other channel counts,
// float64, filters whose weights do not fit in shared memory).
#include "cv_packed.cuh"
#include "sc_common.cuh"
#include "sc_entry.h"
#include "smem_grant.h"

namespace chop {
namespace {

// Storage type T: float, or bfloat16 widened to float on load and rounded on store (float32 accumulation).
template <typename T> struct TileIo;
template <> struct TileIo<float> {
  static __device__ __forceinline__ float ld1(const float* p) { return __ldg(p); }
  static __device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
  static __device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
  }
};
template <> struct TileIo<__nv_bfloat16> {
  static __device__ __forceinline__ float ld1(const __nv_bfloat16* p) { return ScIo<__nv_bfloat16>::ld(p); }
  static __device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
  }
  static __device__ __forceinline__ void st4(__nv_bfloat16* p, float a, float b, float c, float d) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
  }
};

// FORM 0: forward - voxels of the output grid gather the input grid (sc_tap); weights w[t][ci][co].
// FORM 1: gather form - voxels of the fine grid gather the coarse grid (sc_tap_t); the gathered tensor has Cout
//         channels, the produced one Cin, weights flipped: w'[t][co][ci] = filter[taps-1-t][ci][co].
//
// The gathered channels are split over lanes: LK = KCH/4 neighbouring lanes share a voxel, each holding four of its
// channels, and a thread accumulates RT voxels x all NCH produced channels over its quarter of the reduction; the lanes'
// partial sums are added once per voxel, after all taps.  So one warp-wide 16-byte load covers whole channel vectors of
// 32/LK voxels (one thread per voxel touched 32 cache lines per load and was bound by the L1: 83 % busy), and every
// 16-byte weight load (LK addresses per warp, padded to different banks) feeds 4*RT multiply-adds, issued two at a time
// (fma.rn.f32x2).  Which voxel a tap reads is worked out once per CTA and tile into a shared table, and the next tap's
// values are requested before the present tap's arithmetic.
// Bound: the FMA pipe.  189x251x7, 16 -> 16 channels, 3x3x3, float32: 142 us forward (235
// before), 147 us image gradient (287); the FMA pipe is 55 % busy, the rest is splatting the gathered values and latency.
template <int KCH, int NCH>
struct TileCfg {
  static constexpr int LK = KCH / 4;                  // lanes per voxel
  static constexpr int RPW = 32 / LK;                 // voxels per warp-wide load
  static constexpr int RT = NCH <= 16 ? 4 : 2;        // loads (voxels per thread) in flight: 4*RT*NCH/4 accumulators
  static constexpr int VPC = 4 * RPW * RT;            // voxels per CTA (four warps)
  static constexpr int WROW = 4 * NCH + 4;            // floats of a lane's four weight rows, padded by 16 bytes
};

// Source voxels of the taps of filter column (fr, fc) for voxel (b, r, c, dz): tab[fz*step] = voxel index or -1.
template <int FORM>
__device__ __forceinline__ void tile_column(const ScArgs& a, const int4 vx, int fr, int fc, int* tab, int step) {
  const bool s1 = a.sr == 1 && a.sc == 1 && a.sd == 1;
  if (!s1) {   // strides: the plain index functions
    for (int fz = 0; fz < a.fd; ++fz)
      tab[fz * step] = (int)(FORM == 0 ? sc_tap(a, vx.x, vx.y, vx.z, vx.w, fr, fc, fz) : sc_tap_t(a, vx.x, vx.y, vx.z, vx.w, fr, fc, fz));
    return;
  }
  const int pr = FORM == 0 ? a.pr : (a.fh - 1) * a.dr - a.pr, pc = FORM == 0 ? a.pc : (a.fw - 1) * a.dc - a.pc;
  const int pd = FORM == 0 ? a.pd : (a.fd - 1) * a.dd - a.pd;
  const int orow = vx.y - pr + fr * a.dr, ocol = vx.z - pc + fc * a.dc;
  const bool in = !oob(orow, a.H) && !oob(ocol, a.W);
  const int pix = in ? (vx.x * a.H + orow) * a.W + ocol : 0;
  const int d = vx.w + __ldg(a.base_plane + (vx.x * a.H + vx.y) * a.W + vx.z) - __ldg(a.base_plane + pix) - pd;
  for (int fz = 0; fz < a.fd; ++fz) {
    const int ind = d + fz * a.dd;
    tab[fz * step] = in && !oob(ind, a.D) ? pix * a.D + ind : -1;
  }
}

template <typename T, int KCH, int NCH, int FORM>
__global__ void __launch_bounds__(128, 4) sc_tile_kernel(const ScArgs a, const int nvox, const int ntiles) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef TileCfg<KCH, NCH> Cf;
  constexpr int LK = Cf::LK, RPW = Cf::RPW, RT = Cf::RT, VPC = Cf::VPC, WROW = Cf::WROW;
  const int taps = a.fh * a.fw * a.fd;
  float* ws = reinterpret_cast<float*>(smem_raw);                         // [taps][LK][WROW]
  int4* vox = reinterpret_cast<int4*>(ws + (size_t)taps * LK * WROW);      // [VPC] batch (-1: none), row, column, depth
  int* outv = reinterpret_cast<int*>(vox + VPC);                           // [VPC] produced voxel
  int* tab = outv + VPC;                                                   // [taps][VPC] gathered voxel, -1 padding, -2 none
  const T* flt = static_cast<const T*>(a.filters);
  for (int e = threadIdx.x; e < taps * KCH * NCH; e += 128) {
    const int n = e % NCH, k = (e / NCH) % KCH, t = e / (NCH * KCH);
    ws[((size_t)t * LK + k / 4) * WROW + (k % 4) * NCH + n] =
        FORM == 0 ? TileIo<T>::ld1(flt + e) : TileIo<T>::ld1(flt + ((size_t)(taps - 1 - t) * NCH + n) * KCH + k);
  }
  const T* src = static_cast<const T*>(FORM == 0 ? a.images : a.out_grad);
  T* dst = static_cast<T*>(FORM == 0 ? a.output : a.images_grad);
  const float pad = a.pad_zero ? 0.f : TileIo<T>::ld1(static_cast<const T*>(a.default_value));
  const float4 pad4 = make_float4(pad, pad, pad, pad);
  const bool classes = FORM == 1 && (a.sr > 1 || a.sc > 1);
  TileClass cl;
  cl.k = 0;
  cl.begin = 0;
  if (classes) class_open<VPC>(a, cl);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q = lane % LK, row0 = warp * RPW * RT + lane / LK;   // this thread's voxels: row0 + i*RPW
  const T* src_lane = src + q * 4;

  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (classes)
      while (tile >= cl.end) {
        ++cl.k;
        cl.begin = cl.end;
        class_open<VPC>(a, cl);
      }
    __syncthreads();   // the previous tile's tables have been read
    for (int e = threadIdx.x; e < VPC; e += 128) {
      int4 x = make_int4(-1, 0, 0, 0);
      int o = -1;
      if (classes) {   // voxels of one (row, column) residue class: whole taps of a tile are empty and skipped
        unsigned u = (unsigned)(tile - cl.begin) * VPC + e;
        if (u < (unsigned)a.B * cl.hc * cl.wc * a.D) {
          x.w = (int)(u % (unsigned)a.D); u /= (unsigned)a.D;
          x.z = (int)(u % (unsigned)cl.wc) * a.sc + cl.pc; u /= (unsigned)cl.wc;
          x.y = (int)(u % (unsigned)cl.hc) * a.sr + cl.pr;
          x.x = (int)(u / (unsigned)cl.hc);
          o = ((x.x * a.H + x.y) * a.W + x.z) * a.D + x.w;
        }
      } else {
        const int d1 = FORM == 0 ? a.oD : a.D, d2 = FORM == 0 ? a.oW : a.W, d3 = FORM == 0 ? a.oH : a.H;
        unsigned u = (unsigned)tile * VPC + e;
        if (u < (unsigned)nvox) {
          o = (int)u;
          x.w = (int)(u % (unsigned)d1); u /= (unsigned)d1;
          x.z = (int)(u % (unsigned)d2); u /= (unsigned)d2;
          x.y = (int)(u % (unsigned)d3);
          x.x = (int)(u / (unsigned)d3);
        }
      }
      vox[e] = x;
      outv[e] = o;
    }
    __syncthreads();
    const int ncols = a.fh * a.fw;
    for (int e = threadIdx.x; e < VPC * ncols; e += 128) {
      const int col = e / VPC, v = e % VPC;
      const int4 x = vox[v];
      int* t = tab + col * a.fd * VPC + v;
      if (x.x < 0) {
        for (int fz = 0; fz < a.fd; ++fz) t[fz * VPC] = -2;
      } else {
        tile_column<FORM>(a, x, col / a.fw, col % a.fw, t, VPC);
      }
    }
    __syncthreads();

    pk2 acc[RT][NCH / 2];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int n = 0; n < NCH / 2; ++n) acc[i][n] = 0ull;
    // two sets of values in turn: one tap's arithmetic runs while the next tap's loads are in flight
    auto request = [&](float4 (&x)[RT], int t) -> bool {   // false: no voxel of the warp has this tap
      bool live = pad != 0.f;
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int at = tab[t * VPC + row0 + i * RPW];
        x[i] = at == -1 ? pad4 : make_float4(0.f, 0.f, 0.f, 0.f);
        if (at >= 0) x[i] = TileIo<T>::ld4(src_lane + (size_t)at * KCH);
        live |= at >= 0;
      }
      return __any_sync(0xffffffffu, live);
    };
    auto multiply = [&](const float4 (&x)[RT], int t) {
      const float* wt = ws + (t * LK + q) * WROW;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        pk2 x2[RT];
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          const float v = kk == 0 ? x[i].x : kk == 1 ? x[i].y : kk == 2 ? x[i].z : x[i].w;
          x2[i] = pk_make(v, v);
        }
#pragma unroll
        for (int n4 = 0; n4 < NCH / 4; ++n4) {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(wt + kk * NCH + n4 * 4);
#pragma unroll
          for (int i = 0; i < RT; ++i) {
            pk_fma_to(acc[i][n4 * 2], x2[i], w.x);
            pk_fma_to(acc[i][n4 * 2 + 1], x2[i], w.y);
          }
        }
      }
    };
    float4 xa[RT], xb[RT];
    bool la = request(xa, 0), lb = false;
    for (int t = 0; t < taps; t += 2) {
      if (t + 1 < taps) lb = request(xb, t + 1);
      if (la) multiply(xa, t);
      if (t + 1 >= taps) break;
      if (t + 2 < taps) la = request(xa, t + 2);
      if (lb) multiply(xb, t + 1);
    }

    // add the LK lanes' partial sums; lane q keeps values q*M/LK .. of the M = RT*NCH (voxel, channel) sums
    constexpr int M = RT * NCH;
    float v[M];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int n = 0; n < NCH / 2; ++n) pk_split(acc[i][n], v[i * NCH + 2 * n], v[i * NCH + 2 * n + 1]);
#pragma unroll
    for (int s = LK / 2, half = M / 2; s >= 1; s >>= 1, half >>= 1) {
      const bool hi = (q & s) != 0;
#pragma unroll
      for (int e = 0; e < M / 2; ++e) {
        if (e < half) {
          const float keep = hi ? v[e + half] : v[e];
          const float send = hi ? v[e] : v[e + half];
          v[e] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
      }
    }
    constexpr int MINE = M / LK;
#pragma unroll
    for (int e = 0; e < MINE; e += 4) {
      const int at = q * MINE + e;
      const int o = outv[row0 + (at / NCH) * RPW];
      if (o >= 0) TileIo<T>::st4(dst + (size_t)o * NCH + at % NCH, v[e], v[e + 1], v[e + 2], v[e + 3]);
    }
  }
}

// Filter gradient, float32: dW[tap][k][n] = sum over voxels of gathered(voxel, tap)[k] * upstream(voxel)[n].
// A CTA owns a contiguous slice of the voxels and the whole [taps*KCH][NCH] result: thread q holds four consecutive
// gathered channels of one tap times NT upstream channels in registers (4*NT accumulators in pairs), so a voxel costs one
// 16-byte load of the gathered values, NT/4 warp-uniform 16-byte loads of the upstream row from shared memory and
// 2*NT paired FMAs.  Tap indices and upstream rows of WT voxels are staged per step.  Per-CTA slabs are summed in a fixed
// order by sc_slab_reduce (deterministic).  TR = transposed convolution: the voxels are those of the fine grid,
// the gathered tensor is the coarse input (Cout channels), the upstream one has Cin channels, and the reduction
// writes element [tap][co][ci] to filter_grad[taps-1-tap][ci][co].
constexpr int WT = 32;   // voxels per staging step

template <typename T, int KCH, int NCH, bool TR>
__global__ void __launch_bounds__(256) sc_wgrad_tile_kernel(const ScArgs a, const int vox_per_cta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT = NCH < 16 ? NCH : 16;                   // upstream channels per sweep
  const int taps = a.fh * a.fw * a.fd;
  const int K4 = taps * KCH / 4;                            // threads with work
  float* gt = reinterpret_cast<float*>(smem_raw);                         // [WT][NCH]
  int4* vox = reinterpret_cast<int4*>(gt + WT * NCH);                     // [WT]: b, row, column, depth of a staged voxel
  int* tapidx = reinterpret_cast<int*>(vox + WT);                         // [taps][WT] gathered voxel or -1
  float* wsum = reinterpret_cast<float*>(tapidx + (size_t)WT * taps);      // [taps][NCH], dynamic_default only
  float* red = wsum + (size_t)taps * NCH;                                 // [blockDim]
  const T* img = static_cast<const T*>(a.images);
  const T* og = static_cast<const T*>(a.out_grad);
  const bool dyn = !TR && a.dynamic_default;
  if (dyn) {
    const T* flt = static_cast<const T*>(a.filters);
    for (int e = threadIdx.x; e < taps * NCH; e += blockDim.x) {
      const int n = e % NCH, t = e / NCH;
      float s = 0.f;
      for (int k = 0; k < KCH; ++k) s += TileIo<T>::ld1(flt + ((size_t)t * KCH + k) * NCH + n);
      wsum[e] = s;
    }
  }
  const float defv = TileIo<T>::ld1(static_cast<const T*>(a.default_value));
  const float4 pad4 = make_float4(defv, defv, defv, defv);
  const long long nvox = TR ? a.nvox_in : a.nvox_out;
  const int d1 = TR ? a.D : a.oD, d2 = TR ? a.W : a.oW, d3 = TR ? a.H : a.oH;
  const long long v0 = (long long)blockIdx.x * vox_per_cta;
  const long long v1 = min(nvox, v0 + vox_per_cta);
  const int q = threadIdx.x;
  const bool active = q < K4;
  const int my_tap = active ? (q * 4) / KCH : 0;
  const int my_k = active ? (q * 4) % KCH : 0;
  const size_t slab = (size_t)taps * KCH * NCH + 1;
  float* part = static_cast<float*>(a.workspace) + (size_t)blockIdx.x * slab;
  float dacc = 0.f;

  for (int n0 = 0; n0 < NCH; n0 += NT) {
    pk2 acc[4][NT / 2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int n = 0; n < NT / 2; ++n) acc[i][n] = 0ull;
    for (long long vt = v0; vt < v1; vt += WT) {
      const int tm = (int)min((long long)WT, v1 - vt);
      __syncthreads();
      // voxel coordinates once per voxel (the 64-bit divisions are the expensive part), then the tap table
      if (threadIdx.x < tm) {
        unsigned v = (unsigned)(vt + threadIdx.x);   // 31-bit voxel counts
        const int dz = (int)(v % (unsigned)d1); v /= (unsigned)d1;
        const int cc = (int)(v % (unsigned)d2); v /= (unsigned)d2;
        vox[threadIdx.x] = make_int4((int)(v / (unsigned)d3), (int)(v % (unsigned)d3), cc, dz);
      }
      for (int e = threadIdx.x; e < tm * NCH; e += blockDim.x) gt[e] = TileIo<T>::ld1(og + vt * NCH + e);
      __syncthreads();
      for (int e = threadIdx.x; e < WT * a.fh * a.fw; e += blockDim.x) {
        const int col = e / WT, m = e % WT;
        if (m < tm) tile_column<TR ? 1 : 0>(a, vox[m], col / a.fw, col % a.fw, tapidx + col * a.fd * WT + m, WT);
      }
      __syncthreads();
      if (active) {
        // four voxels per step: their gathered loads are issued together, then 4 x 4 x NT FMAs
        for (int m0 = 0; m0 < tm; m0 += 4) {
          int at[4];
          float4 x[4];
          *reinterpret_cast<int4*>(at) = *reinterpret_cast<const int4*>(tapidx + my_tap * WT + m0);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (m0 + u >= tm) at[u] = -2;   // no voxel
#pragma unroll
          for (int u = 0; u < 4; ++u)
            x[u] = at[u] >= 0 ? TileIo<T>::ld4(img + (size_t)at[u] * KCH + my_k)
                              : (at[u] == -1 ? pad4 : make_float4(0.f, 0.f, 0.f, 0.f));
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (m0 + u >= tm) break;
            const ulonglong2* g4 = reinterpret_cast<const ulonglong2*>(gt + (m0 + u) * NCH + n0);
            const pk2 xs[4] = {pk_make(x[u].x, x[u].x), pk_make(x[u].y, x[u].y), pk_make(x[u].z, x[u].z), pk_make(x[u].w, x[u].w)};
#pragma unroll
            for (int n4 = 0; n4 < NT / 4; ++n4) {
              const ulonglong2 g = g4[n4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                pk_fma_to(acc[i][n4 * 2], xs[i], g.x);
                pk_fma_to(acc[i][n4 * 2 + 1], xs[i], g.y);
              }
            }
            if (dyn && at[u] == -1 && my_k == 0) {
              // d(default) collects (sum over input channels of the filter) . out_grad over the padded taps
              // (sparse_conv3d_fast_fixed_param_op_gpu.cu.cc:273-277); one thread per tap does it
              const float* ws = wsum + my_tap * NCH + n0;
              const float* gr = gt + (m0 + u) * NCH + n0;
#pragma unroll
              for (int n = 0; n < NT; ++n) dacc = fmaf(ws[n], gr[n], dacc);
            }
          }
        }
      }
    }
    if (active) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float* o = part + ((size_t)my_tap * KCH + my_k + i) * NCH + n0;
#pragma unroll
        for (int n = 0; n < NT / 2; ++n) pk_split(acc[i][n], o[2 * n], o[2 * n + 1]);
      }
    }
  }
  __syncthreads();
  red[threadIdx.x] = dacc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[slab - 1] = red[0];
}

template <typename T, int KCH, int NCH, bool TR>
int launch_wgrad(const ScArgs& a, int nparts, cudaStream_t st) {
  const int taps = a.fh * a.fw * a.fd;
  const int K4 = taps * KCH / 4;
  int threads = 64;   // a power of two (the block sum of the default-value gradient halves the block repeatedly)
  while (threads < K4) threads <<= 1;
  if (threads > 256) return -4;
  const long long nvox = TR ? a.nvox_in : a.nvox_out;
  if (nparts > (nvox + WT - 1) / WT) nparts = (int)((nvox + WT - 1) / WT);
  const int vox_per_cta = (int)((nvox + nparts - 1) / nparts);
  nparts = (int)((nvox + vox_per_cta - 1) / vox_per_cta);   // every launched CTA owns at least one voxel and writes its slab
  const size_t smem = (size_t)WT * NCH * 4 + WT * sizeof(int4) + (size_t)WT * taps * 4 + ((size_t)taps * NCH + threads) * 4;
  auto k = sc_wgrad_tile_kernel<T, KCH, NCH, TR>;
  if (int e = grant_smem(k, smem)) return e;
  k<<<nparts, threads, smem, st>>>(a, vox_per_cta);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  return sc_slab_reduce(static_cast<const float*>(a.workspace), nparts, taps, KCH, NCH, TR, static_cast<float*>(a.filter_grad),
                        TR ? nullptr : static_cast<float*>(a.default_grad), st);
}

template <typename T, bool TR>
int dispatch_wgrad(const ScArgs& a, int nparts, cudaStream_t st) {
  const int kch = TR ? a.Cout : a.Cin, nch = TR ? a.Cin : a.Cout;
#define CHOP_TILE_CASE(K, N) \
  if (kch == K && nch == N) return launch_wgrad<T, K, N, TR>(a, nparts, st);
  CHOP_TILE_CASE(8, 8) CHOP_TILE_CASE(8, 16) CHOP_TILE_CASE(8, 32) CHOP_TILE_CASE(16, 8) CHOP_TILE_CASE(16, 16)
  CHOP_TILE_CASE(16, 32) CHOP_TILE_CASE(32, 8) CHOP_TILE_CASE(32, 16) CHOP_TILE_CASE(32, 32)
#undef CHOP_TILE_CASE
  return -4;
}

template <typename T, int KCH, int NCH, int FORM>
int launch(const ScArgs& a, cudaStream_t st) {
  typedef TileCfg<KCH, NCH> Cf;
  const int taps = a.fh * a.fw * a.fd;
  const size_t smem = (size_t)taps * Cf::LK * Cf::WROW * 4 + (size_t)Cf::VPC * (sizeof(int4) + 4) + (size_t)Cf::VPC * taps * 4;
  auto k = sc_tile_kernel<T, KCH, NCH, FORM>;
  if (int e = grant_smem(k, smem)) return e;
  const long long nvox = FORM == 0 ? a.nvox_out : a.nvox_in;
  long long ntiles = (nvox + Cf::VPC - 1) / Cf::VPC;
  if (FORM == 1 && (a.sr > 1 || a.sc > 1)) ntiles = class_tiles(a, Cf::VPC);
  // weights are staged per CTA: as many CTAs as are resident, each walking its tiles
  int per_sm = (int)((size_t)220 * 1024 / (smem + 1024));
  if (per_sm > 4) per_sm = 4;
  if (per_sm < 1) per_sm = 1;
  const long long blocks = ntiles < 148LL * per_sm ? ntiles : 148LL * per_sm;
  k<<<(unsigned)blocks, 128, smem, st>>>(a, (int)nvox, (int)ntiles);
  return (int)cudaGetLastError();
}

template <typename T, int FORM>
int dispatch(const ScArgs& a, cudaStream_t st) {
  const int kch = FORM == 0 ? a.Cin : a.Cout, nch = FORM == 0 ? a.Cout : a.Cin;
#define CHOP_TILE_CASE(K, N) \
  if (kch == K && nch == N) return launch<T, K, N, FORM>(a, st);
  CHOP_TILE_CASE(8, 8) CHOP_TILE_CASE(8, 16) CHOP_TILE_CASE(8, 32) CHOP_TILE_CASE(16, 8) CHOP_TILE_CASE(16, 16)
  CHOP_TILE_CASE(16, 32) CHOP_TILE_CASE(32, 8) CHOP_TILE_CASE(32, 16) CHOP_TILE_CASE(32, 32)
#undef CHOP_TILE_CASE
  return -4;
}

}  // namespace

// float32 or bfloat16 data, both channel counts in {8,16,32}, weights and tap table within an SM's shared memory (either
// form), 31-bit voxel indices, 16-byte aligned tensors (checked by the caller)
bool sc_tile_supported(int dtype, const ScArgs& a) {
  if (dtype != 0 && dtype != 2) return false;
  const size_t taps = (size_t)a.fh * a.fw * a.fd;
  const int c[2] = {a.Cin, a.Cout};
  for (int i = 0; i < 2; ++i) {
    const int k = c[i], n = c[1 - i];
    if (k != 8 && k != 16 && k != 32) return false;
    const size_t vpc = 4 * (size_t)(128 / k) * (n <= 16 ? 4 : 2);
    if (taps * (k / 4) * (4 * n + 4) * 4 + vpc * (20 + taps * 4) > 220 * 1024) return false;
  }
  return a.nvox_in < (1LL << 31) - 4096 && a.nvox_out < (1LL << 31) - 4096;
}

// the filter gradient additionally needs taps * (gathered channels) / 4 <= 256 threads
bool sc_tile_wgrad_supported(int dtype, const ScArgs& a, bool transposed) {
  if (!sc_tile_supported(dtype, a)) return false;
  return (long long)a.fh * a.fw * a.fd * (transposed ? a.Cout : a.Cin) / 4 <= 256;
}
int sc_tile_wgrad_launch(int dtype, const ScArgs& a, int nparts, cudaStream_t st) {
  return dtype == 0 ? dispatch_wgrad<float, false>(a, nparts, st) : dispatch_wgrad<__nv_bfloat16, false>(a, nparts, st);
}
int sc_tile_twgrad_launch(int dtype, const ScArgs& a, int nparts, cudaStream_t st) {
  return dtype == 0 ? dispatch_wgrad<float, true>(a, nparts, st) : dispatch_wgrad<__nv_bfloat16, true>(a, nparts, st);
}

int sc_tile_fwd_launch(int dtype, const ScArgs& a, cudaStream_t st) {
  return dtype == 0 ? dispatch<float, 0>(a, st) : dispatch<__nv_bfloat16, 0>(a, st);
}
// gather form: a.out_grad = the coarse tensor (Cout channels), a.images_grad = the fine result (Cin channels);
// a.pad_zero selects the image gradient (1) or the transposed forward (0)
int sc_tile_gather_launch(int dtype, const ScArgs& a, cudaStream_t st) {
  return dtype == 0 ? dispatch<float, 1>(a, st) : dispatch<__nv_bfloat16, 1>(a, st);
}

}  // namespace chop
