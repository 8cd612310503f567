// Stride-1 3x3x3 manifold convolution of float32 data on the CUDA cores, in runs of planes: forward, image gradient and
// transposed forward, 8, 16 or 32 channels on either side.
//
// As in sc_tile.cu the gathered channels are split over lanes - LK = KCH/4 neighbouring lanes share an item, each holding
// four channels of it, and their sums are added once at the end - but an item is a RUN of TZ consecutive planes of one pixel,
// not a voxel.  The three depth taps of a filter column read the same neighbour pixel at consecutive planes, so a run loads
// TZ + 2 rows per column where single voxels load 3*TZ, and every row then feeds up to three planes from its registers.
// Nothing is looked up per tap: one (first voxel, shift) pair per item and column, in a table that each warp fills for
// itself, so that after the weights are staged no warp waits for another.
// Bound: shared memory returns 128 bytes a cycle, so a 16-byte weight load occupies it for the four cycles that its eight paired
// multiply-adds take (load-store data pipe 75 % busy, FMA pipe 63).  189x251x7, float32, us before (sc_tile.cu) and now:
// 8 -> 8 channels 66, 49; 8 -> 16 104, 73; 16 -> 8 99, 78; 16 -> 16 150, 127; 32 -> 32 683, 447; scalar instead of paired 156.
#include "cv_packed.cuh"
#include "sc_common.cuh"
#include "sc_entry.h"
#include "smem_grant.h"

namespace chop {
namespace {

constexpr int RUN_WARPS = 4, RUN_OCC = 3;   // 168 registers: two columns' rows and 64 sums (four CTAs of 128: 127 -> 158 us)
template <int KCH, int NCH, int TZ>
struct RunCfg {
  static constexpr int LK = KCH / 4;                  // lanes per item
  static constexpr int IPW = 32 / LK;                 // items per warp
  static constexpr int NT = NCH < 16 ? NCH : 16;      // produced channels per thread; 32 are produced by two CTAs
  static constexpr int WROW = 4 * NT + 4;             // floats of a lane's four weight rows, padded by 16 bytes
  static constexpr size_t WBYTES = (size_t)27 * LK * WROW * 4;
  static constexpr size_t SMEM = WBYTES + (size_t)RUN_WARPS * IPW * 9 * sizeof(int2);
};

// FWD: weights w[t][ci][co], otherwise flipped and swapped, w'[t][co][ci] = filter[26 - t][ci][co], over a.out_grad.
template <int KCH, int NCH, int TZ, bool FWD>
__global__ void __launch_bounds__(32 * RUN_WARPS, RUN_OCC) sc_run_kernel(const __grid_constant__ ScArgs a, const int nz, const unsigned nitems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef RunCfg<KCH, NCH, TZ> Cf;
  constexpr int LK = Cf::LK, IPW = Cf::IPW, NT = Cf::NT, WROW = Cf::WROW;
  float* ws = reinterpret_cast<float*>(smem_raw);                          // [27][LK][WROW]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int2* tab = reinterpret_cast<int2*>(smem_raw + Cf::WBYTES) + warp * IPW * 9;   // [9][IPW] first voxel (-1: padding), shift
  const int n0 = NCH > NT ? blockIdx.y * NT : 0;
  const float* flt = static_cast<const float*>(a.filters);
  for (int e = threadIdx.x; e < 27 * KCH * NT; e += 32 * RUN_WARPS) {
    int t, k, n;
    if (FWD) {
      n = e % NT; k = e / NT % KCH; t = e / (NT * KCH);
    } else {
      k = e % KCH; n = e / KCH % NT; t = e / (NT * KCH);
    }
    ws[(size_t)(t * LK + k / 4) * WROW + (k % 4) * NT + n] =
        __ldg(FWD ? flt + ((size_t)t * KCH + k) * NCH + n0 + n : flt + ((size_t)(26 - t) * NCH + n0 + n) * KCH + k);
  }
  __syncthreads();
  const float pad = a.pad_zero ? 0.f : __ldg(static_cast<const float*>(a.default_value));
  const float4 pad4 = make_float4(pad, pad, pad, pad);
  const int q = lane % LK, it = lane / LK;
  const float* src = static_cast<const float*>(FWD ? a.images : a.out_grad) + q * 4;
  float* dst = static_cast<float*>(FWD ? a.output : a.images_grad) + n0;
  const int H = a.H, W = a.W, D = a.D;
  const unsigned step = gridDim.x * RUN_WARPS * IPW;

  for (unsigned first = (blockIdx.x * RUN_WARPS + warp) * IPW; first < nitems; first += step) {
    __syncwarp();
    for (int e = lane; e < IPW * 9; e += 32) {
      const unsigned item = first + e % IPW;
      const int col = e / IPW;
      int2 ent = make_int2(-1, 0);
      if (item < nitems) {
        const unsigned pix = item / (unsigned)nz;
        const int c = (int)(pix % (unsigned)W), r = (int)(pix / (unsigned)W % (unsigned)H);
        const int orow = r - 1 + col / 3, ocol = c - 1 + col % 3;
        if (!oob(orow, H) && !oob(ocol, W)) {
          const unsigned np = pix + (col / 3 - 1) * W + (col % 3 - 1);
          ent = make_int2((int)(np * D), __ldg(a.base_plane + pix) - __ldg(a.base_plane + np));
        }
      }
      tab[col * IPW + e % IPW] = ent;
    }
    __syncwarp();
    const unsigned item = first + it;
    const bool live = item < nitems;
    const int pix = live ? (int)(item / (unsigned)nz) : 0;
    const int z0 = live ? (int)(item % (unsigned)nz) * TZ : 0;             // first plane of the run

    pk2 acc[TZ][NT / 2];
#pragma unroll
    for (int j = 0; j < TZ; ++j)
#pragma unroll
      for (int n = 0; n < NT / 2; ++n) acc[j][n] = 0ull;
    float4 x[TZ + 2], y[TZ + 2];
    auto request = [&](float4 (&v)[TZ + 2], int col) {
      const int2 e = tab[col * IPW + it];
      const int plane = z0 - 1 + e.y;
      const float* p = src + ((long long)e.x + plane) * KCH;               // dereferenced for planes of the band only
#pragma unroll
      for (int r = 0; r < TZ + 2; ++r) {
        v[r] = pad4;
        if (e.x >= 0 && !oob(plane + r, D)) v[r] = __ldg(reinterpret_cast<const float4*>(p + r * KCH));
      }
    };
    auto multiply = [&](const float4 (&v)[TZ + 2], int col) {
      const float* wc = ws + (size_t)(col * 3 * LK + q) * WROW;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        pk2 x2[TZ + 2];
#pragma unroll
        for (int r = 0; r < TZ + 2; ++r) {
          const float s = kk == 0 ? v[r].x : kk == 1 ? v[r].y : kk == 2 ? v[r].z : v[r].w;
          x2[r] = pk_make(s, s);
        }
#pragma unroll
        for (int fz = 0; fz < 3; ++fz) {
#pragma unroll
          for (int n4 = 0; n4 < NT / 4; ++n4) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(wc + fz * LK * WROW + kk * NT + n4 * 4);
#pragma unroll
            for (int j = 0; j < TZ; ++j) {
              pk_fma_to(acc[j][n4 * 2], x2[j + fz], w.x);
              pk_fma_to(acc[j][n4 * 2 + 1], x2[j + fz], w.y);
            }
          }
        }
      }
    };
    request(x, 0);
#pragma unroll 1
    for (int col = 0; col < 8; col += 2) {   // two sets of rows in turn: one column's arithmetic covers the next one's loads
      request(y, col + 1);
      multiply(x, col);
      request(x, col + 2);
      multiply(y, col + 1);
    }
    multiply(x, 8);

    // add the LK lanes' partial sums; lane q keeps values q*M/LK .. of the M = TZ*NT (plane, channel) sums
    constexpr int M = TZ * NT;
    float v[M];
#pragma unroll
    for (int j = 0; j < TZ; ++j)
#pragma unroll
      for (int n = 0; n < NT / 2; ++n) pk_split(acc[j][n], v[j * NT + 2 * n], v[j * NT + 2 * n + 1]);
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
    constexpr int MINE = M / LK, VW = MINE % 4 == 0 ? 4 : 2;
    static_assert(MINE % 2 == 0, "vector stores");
#pragma unroll
    for (int e = 0; e < MINE; e += VW) {
      const int at = q * MINE + e, z = z0 + at / NT;
      float* o = dst + ((size_t)pix * D + z) * NCH + at % NT;
      if (live && z < D) {
        if constexpr (VW == 4) *reinterpret_cast<float4*>(o) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
        else *reinterpret_cast<float2*>(o) = make_float2(v[e], v[e + 1]);
      }
    }
  }
}

template <int KCH, int NCH, int TZ, bool FWD>
int launch_tz(const ScArgs& a, cudaStream_t st) {
  typedef RunCfg<KCH, NCH, TZ> Cf;
  auto k = sc_run_kernel<KCH, NCH, TZ, FWD>;
  if (int e = grant_smem(k, Cf::SMEM)) return e;
  const int nz = (a.D + TZ - 1) / TZ;
  const unsigned nitems = (unsigned)((long long)a.B * a.H * a.W * nz);     // at most as many as voxels
  int per_sm = (int)((size_t)224 * 1024 / (Cf::SMEM + 1024));
  if (per_sm > RUN_OCC) per_sm = RUN_OCC;
  const unsigned split = NCH / Cf::NT;
  const unsigned slots = 148u * per_sm / split, need = (nitems + RUN_WARPS * Cf::IPW - 1) / (RUN_WARPS * Cf::IPW);
  k<<<dim3(need < slots ? need : slots, split), 32 * RUN_WARPS, Cf::SMEM, st>>>(a, nz, nitems);
  return (int)cudaGetLastError();
}
template <int KCH, int NCH, bool FWD>
int launch_run(const ScArgs& a, cudaStream_t st) {
  // runs of four planes, of three where those leave fewer planes of the last run empty
  if ((a.D + 2) / 3 * 3 < (a.D + 3) / 4 * 4 && KCH < 32) return launch_tz<KCH, NCH, KCH < 32 ? 3 : 4, FWD>(a, st);
  return launch_tz<KCH, NCH, 4, FWD>(a, st);
}

// Filter gradient of the same convolution: dW[fr,fc,fz][k][n] = sum over voxels of gathered[k] * upstream[n].
// A thread holds four gathered and eight upstream channels of the THREE depth taps of one filter column, 96 sums in pairs, and
// walks the planes of a pixel: the neighbour's row of one plane meets the upstream rows of three, so a plane costs it one 16-byte
// load of gathered values and two (warp-uniform but for the channels) of upstream ones for 48 paired multiply-adds, where a
// thread per tap loads five for 32.  288 threads are 9 columns x the channel blocks x as many groups as that leaves room for, each
// with pixels of its own; their sums are added in shared memory in a fixed order and sc_slab_reduce adds the CTAs'.
// The upstream rows of the next pixels are copied while the present ones are multiplied.
// Bound: issue and latency at three warps a scheduler (158 registers: issue 51 %, FMA pipe 58 %, stalls on dependent arithmetic, on the
// gathered rows and on the FMA pipe in equal parts).  189x251x7, float32, 3x3x3, the filter gradient and its
// reduction, us before (sc_tile.cu) and now: 16 -> 16 channels 215, 140; 8 -> 8 95, 48; 32 -> 32 670, 570.  Four upstream channels per
// thread and two CTAs of nine warps 205, 288 threads 170.  Error against float64 (2-norm), 60x80x17: 16 -> 16 channels 2.39e-7
// before, 1.87e-7 now; 32 -> 32 3.11e-7, 1.93e-7; 256x320x17 8.5e-7, 2.1e-7; 1.20e-6, 2.8e-7.
constexpr int WG_THR = 384;   // twelve warps, three to a scheduler; 288 left one with three and three with two
constexpr int WG_CHAIN = 64;    // planes after which a thread's sums go to its group's table, which keeps the chains of additions short
                                // (fewer where a thread has fewer than 128: half of them)
template <int KCH, int NCH>
struct WgRun {
  static constexpr int QK = KCH / 4, QN = NCH / 8;    // channel blocks
  static constexpr int TPG = 9 * QK * QN, GROUPS = WG_THR / TPG;
  static constexpr int SUMS = 27 * KCH * NCH;
  static constexpr size_t TABLE = (size_t)GROUPS * SUMS * 4;
  // two buffers of upstream rows and (first voxel, shift) per pixel and column, behind the groups' tables
  static size_t stage(int px, int D) { return (size_t)px * D * NCH * 4 + (size_t)px * 9 * sizeof(int2); }
  static int pixels(int D) {                          // per stage: whole rounds of the groups, about 24 KB
    int r = (int)(24 * 1024 / stage(GROUPS, D));
    return GROUPS * (r < 1 ? 1 : r > 8 ? 8 : r);
  }
  static size_t smem(int D) { return TABLE + 2 * ((stage(pixels(D), D) + 15) / 16 * 16); }
};

template <int KCH, int NCH>
__global__ void __launch_bounds__(WG_THR, 1) sc_wgrad_run_kernel(const __grid_constant__ ScArgs a, const int px, const int stage_bytes,
                                                                 const unsigned pix_per_cta, const int chain_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef WgRun<KCH, NCH> Cf;
  const int D = a.D, H = a.H, W = a.W, tid = threadIdx.x;
  const unsigned npix = (unsigned)a.B * H * W;
  const unsigned p0 = blockIdx.x * pix_per_cta, p1 = min(npix, p0 + pix_per_cta);
  const float* og = static_cast<const float*>(a.out_grad);
  auto rows_of = [&](int buf) { return reinterpret_cast<float*>(smem_raw + Cf::TABLE + (size_t)buf * stage_bytes); };
  auto tab_of = [&](int buf) { return reinterpret_cast<int2*>(smem_raw + Cf::TABLE + (size_t)buf * stage_bytes + (size_t)px * D * NCH * 4); };
  auto fetch = [&](unsigned first, int buf) {         // px pixels from `first` on
    const int n = (int)min((unsigned)px, p1 - first);
    float* rows = rows_of(buf);
    const float* from = og + (size_t)first * D * NCH;
    for (int e = tid * 4; e < n * D * NCH; e += WG_THR * 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(rows + e)), "l"(from + e) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    int2* tab = tab_of(buf);
    for (int e = tid; e < n * 9; e += WG_THR) {
      const unsigned pix = first + e / 9;
      const int col = e % 9, c = (int)(pix % (unsigned)W), r = (int)(pix / (unsigned)W % (unsigned)H);
      const int orow = r - 1 + col / 3, ocol = c - 1 + col % 3;
      int2 ent = make_int2(-1, 0);
      if (!oob(orow, H) && !oob(ocol, W)) {
        const unsigned np = pix + (col / 3 - 1) * W + (col % 3 - 1);
        ent = make_int2((int)(np * D), __ldg(a.base_plane + pix) - __ldg(a.base_plane + np));
      }
      tab[e] = ent;
    }
  };
  // lanes: channel blocks fastest, so that a warp's loads of gathered rows are whole rows
  const int group = tid / Cf::TPG, t = tid % Cf::TPG;
  const int qk = t % Cf::QK, qn = t / Cf::QK % Cf::QN, col = t / (Cf::QK * Cf::QN);
  const float pad = __ldg(static_cast<const float*>(a.default_value));
  const float4 pad4 = make_float4(pad, pad, pad, pad);
  const float* img = static_cast<const float*>(a.images) + qk * 4;
  constexpr int NN = 8;
  pk2 acc[3][4][NN / 2];
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int n = 0; n < NN / 2; ++n) acc[f][k][n] = 0ull;

  // table of a group: [3*4*NN/2 pairs][TPG threads]
  pk2* mine = reinterpret_cast<pk2*>(smem_raw) + (size_t)group * (12 * NN / 2) * Cf::TPG + t;
  bool written = false;
  auto put = [&]() {
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int n = 0; n < NN / 2; ++n) {
          pk2* o = mine + ((f * 4 + k) * (NN / 2) + n) * Cf::TPG;
          *o = written ? pk_add(*o, acc[f][k][n]) : acc[f][k][n];
          acc[f][k][n] = 0ull;
        }
    written = true;
  };
  const bool active = group < Cf::GROUPS;
  int buf = 0, chain = 0;
  if (p0 < p1) fetch(p0, 0);
  for (unsigned first = p0; first < p1; first += px, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                  // this stage has landed; the other one has been read
    if (first + px < p1) fetch(first + px, buf ^ 1);
    const int n = (int)min((unsigned)px, p1 - first);
    for (int i = active ? group : n; i < n; i += Cf::GROUPS) {
      if (chain >= chain_max) {
        put();
        chain = 0;
      }
      chain += D;
      const int2 e = tab_of(buf)[i * 9 + col];
      const ulonglong2* g = reinterpret_cast<const ulonglong2*>(rows_of(buf) + (size_t)i * D * NCH + qn * NN);
      auto row = [&](int plane) {                     // gathered row of a plane of the neighbour, or padding
        float4 v = pad4;
        if (e.x >= 0 && !oob(plane, D)) v = __ldg(reinterpret_cast<const float4*>(img + (size_t)(e.x + plane) * KCH));
        return v;
      };
      const int s = e.y;                              // plane z of the pixel is plane z + s of the neighbour
      pk2 x[3][4];
      auto splat = [](pk2 (&o)[4], const float4& v) {
        o[0] = pk_make(v.x, v.x);
        o[1] = pk_make(v.y, v.y);
        o[2] = pk_make(v.z, v.z);
        o[3] = pk_make(v.w, v.w);
      };
      auto plane = [&](const pk2 (&lo)[4], const pk2 (&mid)[4], const pk2 (&hi)[4], int z) {
        pk2 gs[NN / 2];
#pragma unroll
        for (int n = 0; n < NN / 4; ++n) {
          const ulonglong2 v = g[z * (NCH / 4) + n];
          gs[2 * n] = v.x;
          gs[2 * n + 1] = v.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int n = 0; n < NN / 2; ++n) {
            pk_fma_to(acc[0][k][n], lo[k], gs[n]);
            pk_fma_to(acc[1][k][n], mid[k], gs[n]);
            pk_fma_to(acc[2][k][n], hi[k], gs[n]);
          }
      };
      splat(x[0], row(s - 1));
      splat(x[1], row(s));
      float4 n0 = row(s + 1), n1 = row(s + 2), n2 = row(s + 3);   // requested three planes ahead
      for (int z = 0; z < D; z += 3) {
        splat(x[2], n0);
        n0 = row(z + s + 4);
        plane(x[0], x[1], x[2], z);
        if (z + 1 < D) {
          splat(x[0], n1);
          n1 = row(z + s + 5);
          plane(x[1], x[2], x[0], z + 1);
        }
        if (z + 2 < D) {
          splat(x[1], n2);
          n2 = row(z + s + 6);
          plane(x[2], x[0], x[1], z + 2);
        }
      }
    }
  }
  if (active) put();
  __syncthreads();
  // the groups' sums, in order
  float* part = static_cast<float*>(a.workspace) + (size_t)blockIdx.x * (Cf::SUMS + 1);
  const float* table = reinterpret_cast<const float*>(smem_raw);
  for (int e = tid; e < Cf::SUMS; e += WG_THR) {
    const int n = e % NCH, k = e / NCH % KCH, tap = e / (NCH * KCH);
    const int pair = ((tap % 3) * 4 + k % 4) * (NN / 2) + n % NN / 2, th = (tap / 3 * Cf::QN + n / NN) * Cf::QK + k / 4;
    float v = 0.f;
    for (int gr = 0; gr < Cf::GROUPS; ++gr) v += table[(((size_t)gr * (12 * NN / 2) + pair) * Cf::TPG + th) * 2 + n % 2];
    part[e] = v;
  }
  if (tid == 0) part[Cf::SUMS] = 0.f;                 // the default value's gradient: not asked for
}

template <int KCH, int NCH>
int launch_wgrad(const ScArgs& a, int nparts, cudaStream_t st) {
  typedef WgRun<KCH, NCH> Cf;
  auto k = sc_wgrad_run_kernel<KCH, NCH>;
  const int px = Cf::pixels(a.D);
  const size_t smem = Cf::smem(a.D), stage = (Cf::stage(px, a.D) + 15) / 16 * 16;
  if (int e = grant_smem(k, smem)) return e;
  const unsigned npix = (unsigned)a.B * a.H * a.W;
  if (nparts > 148) nparts = 148;                     // one CTA per SM
  const unsigned rounds = (npix + Cf::GROUPS - 1) / Cf::GROUPS;   // whole rounds of the groups
  if ((unsigned)nparts > rounds) nparts = (int)rounds;
  const unsigned per = (rounds + nparts - 1) / nparts * Cf::GROUPS;
  nparts = (int)((npix + per - 1) / per);             // every CTA owns at least one pixel and writes its slab
  // a small problem has short chains anyway: half of a thread's planes (32 instead of 64 costs 12 us at 189x251x7)
  const long long half = (long long)per / Cf::GROUPS * a.D / 2;
  k<<<nparts, WG_THR, smem, st>>>(a, px, (int)stage, per, half < WG_CHAIN ? (int)half : WG_CHAIN);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  return sc_slab_reduce(static_cast<const float*>(a.workspace), nparts, 27, KCH, NCH, false, static_cast<float*>(a.filter_grad),
                        static_cast<float*>(a.default_grad), st);
}

}  // namespace

// Runs that leave up to a third of their planes empty are still the faster ones (sc_tile.cu at 120x150x5, two runs of four planes:
// 32 -> 32 channels 202 us there, 190 here, 32 -> 8 60 and 64).
bool sc_run_supported(int dtype, const ScArgs& a, int gathered) {
  auto ok = [](int c) { return c == 8 || c == 16 || c == 32; };
  const int in4 = (a.D + 3) / 4 * 4, in3 = (a.D + 2) / 3 * 3, planes = gathered < 32 && in3 < in4 ? in3 : in4;
  return dtype == 0 && a.fh == 3 && a.fw == 3 && a.fd == 3 && a.dr == 1 && a.dc == 1 && a.dd == 1 && a.sr == 1 && a.sc == 1 &&
         a.sd == 1 && ok(a.Cin) && ok(a.Cout) && a.nvox_in < (1LL << 31) - 4096 && 2 * planes <= 3 * a.D;
}

int sc_run_launch(const ScArgs& a, bool dgrad, cudaStream_t st) {
  const int in = dgrad ? a.Cout : a.Cin, out = dgrad ? a.Cin : a.Cout;
  if (sc_band_f32_better(a, in, out)) return sc_band_f32_launch(a, dgrad, st);
#define CHOP_CASE(K, N) if (in == K && out == N) return dgrad ? launch_run<K, N, false>(a, st) : launch_run<K, N, true>(a, st);
  CHOP_CASE(8, 8) CHOP_CASE(8, 16) CHOP_CASE(8, 32) CHOP_CASE(16, 8) CHOP_CASE(16, 16) CHOP_CASE(16, 32) CHOP_CASE(32, 8)
  CHOP_CASE(32, 16) CHOP_CASE(32, 32)
#undef CHOP_CASE
  return -4;
}

namespace {
size_t wgrad_run_smem(int k, int n, int D) {
#define CHOP_CASE(K, N) if (k == K && n == N) return WgRun<K, N>::smem(D);
  CHOP_CASE(8, 8) CHOP_CASE(8, 16) CHOP_CASE(8, 32) CHOP_CASE(16, 8) CHOP_CASE(16, 16) CHOP_CASE(16, 32) CHOP_CASE(32, 8)
  CHOP_CASE(32, 16) CHOP_CASE(32, 32)
#undef CHOP_CASE
  return (size_t)-1;   // other channel counts
}
}  // namespace
// Filter gradient; a.images and a.out_grad 16-byte aligned, nparts slabs of 27*Cin*Cout + 1 floats in the workspace.  Bands whose
// stages do not fit beside the groups' tables (8 -> 8 channels: more than 57 planes) take sc_tile.cu's.
bool sc_run_wgrad_supported(int dtype, const ScArgs& a) {
  return dtype == 0 && a.fh == 3 && a.fw == 3 && a.fd == 3 && a.dr == 1 && a.dc == 1 && a.dd == 1 && a.sr == 1 && a.sc == 1 &&
         a.sd == 1 && !a.dynamic_default && a.D <= 64 && wgrad_run_smem(a.Cin, a.Cout, a.D) <= 220 * 1024 &&
         a.nvox_in < (1LL << 31) - 4096;
}
int sc_run_wgrad_launch(const ScArgs& a, int nparts, cudaStream_t st) {
#define CHOP_CASE(K, N) if (a.Cin == K && a.Cout == N) return launch_wgrad<K, N>(a, nparts, st);
  CHOP_CASE(8, 8) CHOP_CASE(8, 16) CHOP_CASE(8, 32) CHOP_CASE(16, 8) CHOP_CASE(16, 16) CHOP_CASE(16, 32) CHOP_CASE(32, 8)
  CHOP_CASE(32, 16) CHOP_CASE(32, 32)
#undef CHOP_CASE
  return -4;
}

}  // namespace chop
